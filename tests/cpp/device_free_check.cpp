// What a start set is gone after device_free: a failed start leaves its context
// restartable with other options, and the next start allocates only what those
// ask for (no GPU needed: nothing here was allocated).
#include <cstdio>

#include "internal.h"

using namespace gmapf_b200;

int main() {
    static char buf[64];
    Context c;
    Device& d = c.dev;
    d.device = 3;
    d.order_hist = reinterpret_cast<int*>(buf);
    d.lm = reinterpret_cast<unsigned short*>(buf);
    d.lm_count = 8;
    d.lm_max = 700;
    d.req_sorted = d.breq = d.breq_sorted = reinterpret_cast<int4*>(buf);
    d.req_keys = d.breq_keys = reinterpret_cast<int2*>(buf);
    d.breq_cap = 64;
    d.bstarts = d.bpaths = reinterpret_cast<int*>(buf);
    d.bio_cap = 64;
    d.bpaths_cap = 64;
    d.waypoints = reinterpret_cast<float2*>(buf);
    d.clearance = true;
    d.agent_scene = d.scene_abase = d.scene_P = d.scene_first = reinterpret_cast<int*>(buf);
    d.erow = reinterpret_cast<EdgeRow*>(buf);
    d.third = reinterpret_cast<EdgeHalf*>(buf);
    d.corridors.levels = 300;
    d.corridors.loops = 0.5f;
    d.form = FORM_LOG_GLOBAL;
    d.full_pad = true;
    d.slots = d.rec_cap = d.log_cap = d.gbm_cap = 64;
    device_free(c);
    int bad = 0;
#define GONE(f) \
    if (d.f != Device{}.f) bad++, std::printf("%s is left set\n", #f)
    GONE(order_hist);
    GONE(lm);
    GONE(lm_count);
    GONE(lm_max);
    GONE(req_sorted);
    GONE(req_keys);
    GONE(breq);
    GONE(breq_sorted);
    GONE(breq_keys);
    GONE(breq_cap);
    GONE(bstarts);
    GONE(bpaths);
    GONE(bio_cap);
    GONE(bpaths_cap);
    GONE(waypoints);
    GONE(clearance);
    GONE(agent_scene);
    GONE(scene_abase);
    GONE(scene_P);
    GONE(scene_first);
    GONE(erow);
    GONE(third);
    GONE(corridors.levels);
    GONE(corridors.loops);
    GONE(form);
    GONE(full_pad);
    GONE(slots);
    GONE(rec_cap);
    GONE(log_cap);
    GONE(gbm_cap);
    if (d.device != 3) bad++, std::printf("the device id is lost\n");
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
