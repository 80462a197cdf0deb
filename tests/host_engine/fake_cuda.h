// The engine (csrc/engine.cpp) on the host: the CUDA runtime calls it makes work
// on host memory, a captured graph is a list of recorded calls, and every launch
// only notes what it was given.  For tests of what the engine launches, in which
// form and after which failures; nothing is computed.
#pragma once
#include <functional>
#include <set>
#include <vector>
#include "engine.h"

namespace fake {

// What the passes of one substep have to agree on.
struct Key {
    sph::LaunchForm form;
    uint32_t skin = 0, tension = 0, block = 0, ntiles = 0;
    const void *tiles = nullptr, *mask = nullptr;
    size_t stride = 0;
    bool operator==(const Key& o) const {
        return form == o.form && skin == o.skin && tension == o.tension && block == o.block && ntiles == o.ntiles &&
               tiles == o.tiles && mask == o.mask && stride == o.stride;
    }
};

struct State {
    Key sorted, written;           // the last sort's and density pass's
    uint64_t substeps = 0, mixed = 0;   // force passes; passes whose key was not that of the pass before
    std::set<uint32_t> lanes;      // lanes that force passes ran with
    std::set<uint32_t> crowded;    // scenes (by their first slot) that have a cell of too many particles
    std::function<void()> after_force;     // called after each force pass
    std::vector<uint32_t> sorts;   // tiles of each sort
    size_t pinned_limit = ~(size_t)0;      // larger pinned allocations fail
    size_t pinned = 0;                     // bytes pinned now
    int fail_from = -1, fail_count = 0;    // device allocations from the fail_from-th on fail, fail_count of them
    uint64_t mallocs = 0;                  // device allocations asked for
    uint64_t bad_arrays = 0;               // launches given an array that is freed, null or too short
    cudaError_t last_error = cudaSuccess;
    uint64_t null_writes = 0;      // packs and unsorts into a null or unknown buffer
};
extern State st;
// Velocity that an unsort writes for every component.
constexpr float kVelocity = 7.0f;
constexpr float kPosition = 3.0f;

}  // namespace fake
