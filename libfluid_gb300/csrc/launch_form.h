// How a layout's sort and neighbour passes are launched.  The choice decides not
// only which builds run but what lies in the neighbour words (how long lists may
// get, which copies of the positions are kept and where), so a pass reads them
// rightly only if it runs in the form of the passes that wrote them.  The engine
// therefore decides once, when layout and parameters are brought up to date,
// captures its graphs again when the decision changed, and hands the same form to
// every launch, captured or not.
#pragma once
#include <stdint.h>
#include "sph_types.h"

namespace sph {

struct LaunchForm {
    uint32_t lanes = 1u;        // lanes per particle of the neighbour passes (WideShared)
    bool density_wide = false;  // the density pass's too (not with skin words)
    bool half = true;           // candidate positions in half precision (HalfScan)
    bool dense = false;         // position and density once more for the normal pass
    bool one_wave = false;      // the launch fits the GPU at 80 registers
    bool operator==(const LaunchForm& o) const {
        return lanes == o.lanes && density_wide == o.density_wide && half == o.half && dense == o.dense &&
               one_wave == o.one_wave;
    }
    bool operator!=(const LaunchForm& o) const { return !(*this == o); }
};

// ntiles tiles of `tile` threads on a GPU of `sms` SMs; crowded: SPH_CROWDED_NBRS
// neighbours or more on average; skin: some scene runs a per-substep XSPH pass;
// tension: some scene runs the normal pass.
//
// The lanes go by the tiles' threads and not by their particles: blocks are
// launched for all of a tile, and those without particles are what a batch of many
// tiny scenes then spends its time on.  Substep with eight lanes and with one, us:
// 4,800 scenes of one particle 102 and 51, 600 of sixteen 35 and 27, 388 of 36 43
// and 37, 138 of 36 31 and 34, 8 of 1,728 33 and 41; with four lanes and with
// one: 312 of 64 (39,936 threads) 41 and 35, 160 of 125 (20,480) 37 and 39.
inline LaunchForm launch_form(uint32_t ntiles, uint32_t tile, bool persistent, uint32_t variant, bool crowded,
                              bool skin, bool tension, uint32_t sms) {
    LaunchForm f;
    const uint64_t threads = (uint64_t)ntiles * tile;
    if ((variant & SPH_VARIANT_DENSITY_SPLIT) != 0u && !persistent) {
        if (threads <= (crowded ? SPH_CROWDED8_MAX : SPH_WIDE8_MAX)) f.lanes = 8u;
        else if (threads <= SPH_DENSITY_SPLIT_MAX) f.lanes = 4u;
    }
    f.density_wide = f.lanes > 1u && !skin;
    f.half = f.lanes == 1u && !skin;
    f.dense = f.half && tension;   // (long lists and skin words leave no room)
    f.one_wave = !persistent && threads <= (uint64_t)SPH_ONE_WAVE_THREADS * sms;
    return f;
}

}  // namespace sph
