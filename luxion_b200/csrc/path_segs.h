// path_segs.h -- which of a launch's (lane, bounce) segments the whole-path kernel (paths.cu) takes.
//
// Every block of a launch works this out for itself from the lanes' counters, at its own start,
// and all of them have to find the same although block 0 marks the lanes meanwhile. A lane that an
// earlier launch has finished may still be among the segments: the job engine keeps a wave in
// flight until the host has counted it through its bounces, and new waves start beside it.
#pragma once

#include "device_scene.h"

#ifdef __CUDACC__
#define LUX_SEG_FN __host__ __device__ inline
#else
#define LUX_SEG_FN inline
#endif

namespace lux {

struct PathSegs {
    int first[kMaxSegs + 1];  // paths of segment k: [first[k], first[k + 1]) of the launch's list
    int lane;                 // the lane whose cursor and error word serve the launch: the first taken
};

// The cursor is that of a lane the launch takes: a lane is taken once in its wave's life, so its
// cursor is still at the zero the wave started with. Any other lane's may have served before, and
// the paths it has counted off would be skipped.
LUX_SEG_FN PathSegs path_segments(const WaveCounters* ctr, const Segs& G) {
    PathSegs s;
    s.lane = G.lane[0];
    s.first[0] = 0;
    bool any = false;
    for (int k = 0; k < kMaxSegs; ++k) {
        int t = 0;
        if (k < G.n) {
            const WaveCounters* c = ctr + G.lane[k];
            const int f = *(volatile const int*)&c->finished;  // this launch sets bounce + 1
            if (f == 0 || f == G.bounce[k] + 1) {
                t = *(volatile const int*)&c->count[G.bounce[k]];
                if (!any) s.lane = G.lane[k];
                any = true;
            }
        }
        s.first[k + 1] = s.first[k] + t;
    }
    return s;
}

// Marks segment k's lane, so that the wavefront launches that follow find it finished. The mark of
// an earlier launch stays: overwritten by this launch's, it would let a block that starts later
// count the lane's paths again.
LUX_SEG_FN void mark_segment(WaveCounters* ctr, const Segs& G, int k) {
    WaveCounters* c = ctr + G.lane[k];
    if (*(volatile int*)&c->finished == 0) c->finished = G.bounce[k] + 1;
}

}  // namespace lux
