// Which maps the corridor kernel serves, by width and length: winding corridors of
// squares (two triangles each), `width` squares wide.
#include <cstdio>
#include <cstring>
#include <map>
#include <vector>

#include "internal.h"

using namespace gmapf_b200;

// free squares of a grid as a navmesh
static std::vector<gmapf_node> squares(const std::vector<std::vector<char>>& open) {
    std::vector<gmapf_node> out;
    std::map<std::pair<int, int>, int> first;  // square -> its lower triangle
    const int h = (int)open.size(), w = (int)open[0].size();
    for (int y = 0; y < h; y++)
        for (int x = 0; x < w; x++)
            if (open[y][x]) {
                first[{y, x}] = (int)out.size();
                for (int up = 0; up < 2; up++) {
                    gmapf_node n;
                    std::memset(&n, 0, sizeof(n));
                    n.P1 = {(float)x, (float)y};
                    n.P2 = up ? gmapf_v2{(float)x + 1, (float)y + 1} : gmapf_v2{(float)x + 1, (float)y};
                    n.P3 = up ? gmapf_v2{(float)x, (float)y + 1} : gmapf_v2{(float)x + 1, (float)y + 1};
                    out.push_back(n);
                }
            }
    for (const auto& s : first) {
        const int y = s.first.first, x = s.first.second, i = s.second;
        auto at = [&](int yy, int xx, int up) {
            const auto f = first.find({yy, xx});
            return f == first.end() ? -1 : f->second + up;
        };
        // lower: below and right; upper: above and left
        const int nb[2][3] = {{i + 1, at(y - 1, x, 1), at(y, x + 1, 1)}, {i, at(y + 1, x, 0), at(y, x - 1, 0)}};
        for (int up = 0; up < 2; up++) {
            int k = 0;
            for (int j : nb[up])
                if (j >= 0) out[i + up].NeibsIdx[k++] = j;
            while (k < 3) out[i + up].NeibsIdx[k++] = -1;
        }
    }
    return out;
}

static std::vector<std::vector<char>> winding(int width, int length, int rows) {
    std::vector<std::vector<char>> open(rows * (width + 1) - 1, std::vector<char>(length, 0));
    for (int r = 0; r < rows; r++) {
        for (int j = 0; j < width; j++) std::fill(open[r * (width + 1) + j].begin(), open[r * (width + 1) + j].end(), 1);
        if (r + 1 < rows)
            for (int j = 0; j < width; j++) open[r * (width + 1) + width][r % 2 == 0 ? length - 1 - j : j] = 1;
    }
    return open;
}

static int bad = 0;

static Corridors measure(const std::vector<gmapf_node>& nodes) {
    HostMap m;
    build_host_map(nodes.data(), (int)nodes.size(), m);
    SceneInfo si{};
    si.n = m.n;
    return measure_corridors(m, {si});
}

static void expect(const char* what, const std::vector<gmapf_node>& nodes, const std::vector<int>& served) {
    const Corridors c = measure(nodes);
    for (int T : {2, 4, 8, 16, 32}) {
        bool want = false;
        for (int t : served) want = want || t == T;
        if (corridor_kernel_serves(c, T) != want) {
            bad++;
            std::printf("%s, T=%d: %d levels, %.2f loops per level\n", what, T, c.levels, c.loops);
        }
    }
}

// two maps in one, cut off from one another
static std::vector<gmapf_node> both(std::vector<gmapf_node> a, const std::vector<gmapf_node>& b) {
    const int base = (int)a.size();
    for (gmapf_node n : b) {
        for (int& k : n.NeibsIdx)
            if (k >= 0) k += base;
        a.push_back(n);
    }
    return a;
}

int main() {
    const auto open = squares(std::vector<std::vector<char>>(60, std::vector<char>(60, 1)));
    const auto patch = squares(std::vector<std::vector<char>>(3, std::vector<char>(3, 1)));
    const auto lane = squares(winding(1, 50, 1)), lanes = squares(winding(1, 160, 24));
    expect("open ground", open, {});
    expect("a lane, then open ground", both(lane, open), {});
    expect("a patch and a lane, then open ground", both(both(patch, lane), open), {});
    expect("a patch, then long lanes", both(patch, lanes), {2, 4, 8, 16, 32});
    expect("open ground, then long lanes", both(open, lanes), {2, 4, 8, 16, 32});
    expect("long lanes, then a patch", both(lanes, patch), {2, 4, 8, 16, 32});
    expect("1 wide", squares(winding(1, 160, 24)), {2, 4, 8, 16, 32});
    expect("2 wide", squares(winding(2, 160, 12)), {8, 16, 32});
    expect("3 wide", squares(winding(3, 160, 8)), {16, 32});
    expect("4 wide", squares(winding(4, 160, 6)), {32});
    expect("5 wide", squares(winding(5, 160, 5)), {});
    expect("8 wide", squares(winding(8, 160, 4)), {});
    expect("12 wide", squares(winding(12, 160, 2)), {});
    expect("1 wide, 800 triangles", squares(winding(1, 400, 1)), {8, 16, 32});
    expect("1 wide, 100 triangles", squares(winding(1, 50, 1)), {16, 32});
    expect("1 wide, 50 triangles", squares(winding(1, 25, 1)), {});
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
