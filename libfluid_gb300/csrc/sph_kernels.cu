// sm_103a kernels of the WCSPH substep.
//
// One substep (the body of FluidSystem::advance, fluidsystem.cu:301-398) is:
//   [k_hash: only when no force pass hashed the state] -> scan (one pass)
//   -> k_scatter -> k_rank_gather
//   -> k_density (+ the previous substep's XSPH update) -> [k_normals]
//   -> k_force_integrate [-> k_xsph, for scenes that do not defer XSPH]
// Every kernel is scene-aware: a launch covers the tiles of all live scenes,
// so the plain step is the batched step with one scene.
//
// State buffers (float4 per particle, slots indexed by the arena):
//   P0,V0,A0  state between substeps (P0.w = density of the last substep)
//   V2, okey  post-integration velocity and cell of the last substep, for a
//             scene whose XSPH update is pending (pend[scene] != 0)
//   G, A1     state gathered into cell order: G holds two float4 per slot,
//             P0 and the velocity (with a pending update, its w lane holds
//             the gathered okey bits)
//   X         the gathered positions again for the density pass's candidate
//             scan, four slots at a time: their x, their y, their z, 48 bytes
//             in all, or with one thread per particle cell-relative halves, 32
//             bytes (HalfScan); they lie in rows of the neighbour words that the
//             density pass does not write
//   D         position and density again for the normal pass, in such rows too
//   R         neighbour record per sorted slot, 32 bytes, written by the
//             density pass: (x, y, z, rho) and (velocity with the pending
//             XSPH update applied, pressure)
//   C2        squared sound speed per sorted slot
//   N         surface normals, w: C2 again (only when a scene has surface tension)
#include <cfloat>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <type_traits>
#include "sph_types.h"
#include "sph_device.cuh"
#include "sph_kernels.h"

namespace sph {

// Adds the lanes in `mask` to their cells' counts and, with `sums`, to the sums
// of the scan tiles (kScanTileCells cells) they lie in, from which every block of
// the scan finds its own prefix.  Returns the lane's provisional slot in its
// cell.  Equal cells share one atomic; the cells of a warp in cell order nearly
// always lie in one tile and share that one too.
__device__ __forceinline__ uint32_t count_cell(unsigned mask, uint32_t cell, uint32_t* __restrict__ count,
                                               uint32_t* __restrict__ sums) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned peers = __match_any_sync(mask, cell);
    const int leader = __ffs(peers) - 1;
    if (sums) {
        const uint32_t tile = cell / kScanTileCells;
        const int first = __ffs(mask) - 1;
        const uint32_t t0 = __shfl_sync(mask, tile, first);
        const bool one_tile = __all_sync(mask, tile == t0);
        if ((int)lane == (one_tile ? first : leader))
            atomicAdd(sums + tile, (uint32_t)__popc(one_tile ? mask : peers));
    }
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(&count[cell], (uint32_t)__popc(peers));
    base = __shfl_sync(mask, base, leader);
    return base + (uint32_t)__popc(peers & ((1u << lane) - 1u));
}

// ---------------------------------------------------------------------------
// Spatial hash + cell counts (hash.cu:10-27 and the fill at
// fluidsystem.cu:304-306).  Equal keys inside a warp are combined with
// __match_any_sync so one atomic serves each group; the slot a particle gets
// inside its cell is provisional (atomic order) and is made stable by
// k_rank_gather.  For a scene with a pending XSPH update, a particle whose
// cell differs from the one recorded by the last force pass gets the
// SPH_OKEY_MOVED flag there (the density pass's fast adjacency test).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SPH_TILE) k_hash(const DevParams* __restrict__ params,
                                                   const DevScene* __restrict__ scenes,
                                                   const uint4* __restrict__ tiles,
                                                   const float4* __restrict__ P, uint32_t* __restrict__ count,
                                                   uint32_t* __restrict__ key, uint32_t* __restrict__ slot,
                                                   const uint32_t* __restrict__ pend, uint32_t* __restrict__ okey,
                                                   uint32_t* __restrict__ status) {
    const uint4 t = tiles[blockIdx.x];
    const unsigned lanes = __ballot_sync(0xffffffffu, threadIdx.x < t.z);
    if (threadIdx.x >= t.z) return;
    const uint32_t i = t.y + threadIdx.x;
    const DevScene sc = scenes[t.x];
    const DevParams& pp = params[t.x];
    const float4 p = P[i];
    const int3 gc = grid_of(pp, p.x, p.y, p.z);
    const bool inside = grid_inside(pp, gc);
    const uint32_t local = inside ? (uint32_t)gc.x + (uint32_t)gc.y * pp.gx + (uint32_t)gc.z * pp.gxy : pp.ncells;
    if (__ldg(pend + t.x) != 0u) {
        const uint32_t o = okey[i];
        if (o != SPH_OKEY_NULL && (!inside || (o & ~SPH_OKEY_MOVED) != pack_cell(gc))) okey[i] = o | SPH_OKEY_MOVED;
    }
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) atomicOr(status, SPH_STATUS_NONFINITE);
    key[i] = local;
    slot[i] = count_cell(lanes, sc.cell_base + local, count, nullptr);
}

// ---------------------------------------------------------------------------
// Exclusive scan of cell counts -> cell starts (fluidsystem.cu:316), 4096
// counts per tile, in three forms: the substep's (k_scan_tiles), whose tile
// sums the hash made; one pass over any range (k_scan_single); and reduce,
// scan, down-sweep over caller's memory (launch_scan_raw).
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
static_assert(SCAN_TILE == (int)kScanTileCells, "scan tile size");

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (unsigned)o) v += u;
    }
    return v;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t* __restrict__ in, uint32_t n,
                                                              uint32_t* __restrict__ sums) {
    const uint32_t base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t idx = base + k;
        if (idx < n) s += in[idx];
    }
    __shared__ uint32_t red[SCAN_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t w = (threadIdx.x < SCAN_THREADS / 32) ? red[threadIdx.x] : 0u;
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (threadIdx.x == 0) sums[blockIdx.x] = w;
    }
}

// Single block: exclusive scan of up to kScanRawMaxTiles tile sums, in place.
__global__ void __launch_bounds__(1024) k_scan_top(uint32_t* __restrict__ sums, uint32_t nt) {
    constexpr int ITEMS = 32;
    static_assert(ITEMS * 1024 == (int)kScanRawMaxTiles, "k_scan_top capacity");
    uint32_t v[ITEMS];
    const uint32_t base = threadIdx.x * ITEMS;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        v[k] = (base + k < nt) ? sums[base + k] : 0u;
        s += v[k];
    }
    __shared__ uint32_t warp_tot[32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t inc = warp_incl_scan(s);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = warp_tot[lane];
        const uint32_t wi = warp_incl_scan(w);
        warp_tot[lane] = wi - w;
    }
    __syncthreads();
    uint32_t run = warp_tot[warp] + inc - s;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (base + k < nt) sums[base + k] = run;
        run += v[k];
    }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(const uint32_t* __restrict__ in, uint32_t n,
                                                            const uint32_t* __restrict__ sums,
                                                            uint32_t* __restrict__ out) {
    const uint32_t base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t idx = base + k;
        v[k] = (idx < n) ? in[idx] : 0u;
        s += v[k];
    }
    __shared__ uint32_t warp_tot[SCAN_THREADS / 32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t inc = warp_incl_scan(s);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = (lane < SCAN_THREADS / 32) ? warp_tot[lane] : 0u;
        const uint32_t wi = warp_incl_scan(w);
        if (lane < SCAN_THREADS / 32) warp_tot[lane] = wi - w;
    }
    __syncthreads();
    uint32_t run = sums[blockIdx.x] + warp_tot[warp] + inc - s;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const uint32_t idx = base + k;
        if (idx < n) out[idx] = run;
        run += v[k];
        if (idx + 1 == n) out[n] = run;   // total after the last cell
    }
}

// Single-pass form of the same scan, for a range whose tile sums nobody made (one
// scene's cells, when a single scene of many is read): decoupled
// look-back (Merrill and Garland, "Single-pass Parallel Prefix Scan with
// Decoupled Look-back", NVIDIA technical report NVR-2016-002).  Each tile
// publishes its aggregate, then adds the aggregates of the tiles before it
// until it meets one that has published its inclusive prefix, and publishes
// its own.  A descriptor is one 64-bit word (flag << 32 | value), so flag and
// value are read together.  desc[0] hands out tile numbers in the order the
// blocks start, so every tile waited on belongs to a block that is already
// running and waits only on tiles before it; the waits are bounded all the
// same (SPH_STATUS_SCAN_TIMEOUT, the outputs are then invalid).
//
// With `zero` set the kernel also leaves every count it read at zero (as
// k_scan_tiles does).
constexpr unsigned long long SCAN_AGG = 1ull << 32;
constexpr unsigned long long SCAN_PRE = 2ull << 32;
constexpr uint32_t SCAN_SPIN_LIMIT = 1u << 22;   // the default limit (StepArgs.scan_spin_limit = 0)

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_single(uint32_t* __restrict__ in, uint32_t n,
                                                              unsigned long long* __restrict__ desc,
                                                              uint32_t* __restrict__ out,
                                                              uint32_t* __restrict__ status, uint32_t zero,
                                                              uint32_t spin_limit, uint32_t vec_ok) {
    __shared__ uint32_t s_tile, s_prefix, s_total;
    __shared__ uint32_t warp_tot[SCAN_THREADS / 32];
    if (threadIdx.x == 0) s_tile = atomicAdd(reinterpret_cast<unsigned int*>(desc), 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    // 16 counts in four 128-bit accesses, when `in` and `out` are 16-byte
    // aligned (a scene's own range may start anywhere)
    const bool whole = vec_ok && base + SCAN_ITEMS <= n;
    uint32_t v[SCAN_ITEMS];
    // each count is read (and, with `zero`, cleared at the end) by this thread alone
    if (whole) {
        const uint4* p4 = reinterpret_cast<const uint4*>(in + base);
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / 4; ++q) {
            const uint4 w = p4[q];
            v[4 * q] = w.x; v[4 * q + 1] = w.y; v[4 * q + 2] = w.z; v[4 * q + 3] = w.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) v[k] = (base + k < n) ? in[base + k] : 0u;
    }
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) s += v[k];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t inc = warp_incl_scan(s);
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = (lane < SCAN_THREADS / 32) ? warp_tot[lane] : 0u;
        const uint32_t wi = warp_incl_scan(w);
        if (lane < SCAN_THREADS / 32) warp_tot[lane] = wi - w;
        if (lane == 31) s_total = wi;
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t agg = s_total;
        uint32_t excl = 0;
        if (tile == 0) {
            if (lane == 0) st_relaxed_u64(desc + 1, SCAN_PRE | agg);
        } else {
            if (lane == 0) st_relaxed_u64(desc + 1 + tile, SCAN_AGG | agg);
            int j = (int)tile - 1;   // lane l reads tile j - l
            for (;;) {
                const int idx = j - (int)lane;
                unsigned long long d = SCAN_PRE;   // before tile 0: an empty prefix
                if (idx >= 0) {
                    uint32_t spins = 0;
                    d = ld_relaxed_u64(desc + 1 + idx);
                    while ((d >> 32) == 0ull) {
                        if (++spins > spin_limit) {
                            atomicOr(status, SPH_STATUS_SCAN_TIMEOUT);
                            d = SCAN_PRE;
                            break;
                        }
                        __nanosleep(32);
                        d = ld_relaxed_u64(desc + 1 + idx);
                    }
                }
                const unsigned pre = __ballot_sync(0xffffffffu, (d >> 32) == 2ull);
                const int stop = pre ? __ffs(pre) - 1 : 31;   // lanes 0..stop contribute
                uint32_t val = ((int)lane <= stop) ? (uint32_t)d : 0u;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
                excl += val;
                if (pre) break;
                j -= 32;
            }
            if (lane == 0) st_relaxed_u64(desc + 1 + tile, SCAN_PRE | (excl + agg));
        }
        if (lane == 0) s_prefix = excl;
    }
    __syncthreads();
    uint32_t run = s_prefix + warp_tot[warp] + inc - s;
    if (whole) {
        uint4* o4 = reinterpret_cast<uint4*>(out + base);
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS / 4; ++q) {
            uint4 w;
            w.x = run; run += v[4 * q];
            w.y = run; run += v[4 * q + 1];
            w.z = run; run += v[4 * q + 2];
            w.w = run; run += v[4 * q + 3];
            o4[q] = w;
        }
        if (base + SCAN_ITEMS == n) out[n] = run;   // total after the last cell
        if (zero) {
            uint4* z4 = reinterpret_cast<uint4*>(in + base);
#pragma unroll
            for (int q = 0; q < SCAN_ITEMS / 4; ++q) z4[q] = make_uint4(0u, 0u, 0u, 0u);
        }
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            const uint32_t idx = base + k;
            if (idx < n) out[idx] = run;
            run += v[k];
            if (idx + 1 == n) out[n] = run;
            if (zero && idx < n) in[idx] = 0u;
        }
    }
}

// The substep's scan.  A tile's prefix is the sum of the tiles before it, which
// the hash counted (count_cell) and every block reads for itself.  No block
// waits for another and no descriptors are cleared: against the look-back the
// substep of the 1M dam break (489 tiles) went from 379 to 372 us and that of
// 1,728 particles from 27 to 25 us.  Lanes take fours of cells side by side, so
// that a warp's loads and stores cover whole lines (13.0 -> 9.7 us by events around
// the pass at 1M, against 16 cells in a row per lane).  The sums' reads grow with the square of the
// tiles, so from SPH_SCAN_SUM_TILES on (67 million cells; 0.1 ms of reads beside
// 0.1 ms of scan) the look-back takes over.  The counts are left at zero: the next substep's hash (fused into
// the force pass) adds into them, which otherwise needs a memset of the whole
// array; k_scatter clears the sums.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(uint32_t* __restrict__ in, uint32_t n,
                                                             const uint32_t* __restrict__ sums,
                                                             uint32_t* __restrict__ out) {
    constexpr uint32_t kFours = SCAN_ITEMS / 4u;
    __shared__ uint32_t warp_tot[SCAN_THREADS / 32], warp_pre[SCAN_THREADS / 32];
    const uint32_t tile = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // a warp's lanes take fours side by side, kFours times
    const uint32_t base = tile * SCAN_TILE + warp * (32u * SCAN_ITEMS) + 4u * lane;
    uint4 v[kFours];
#pragma unroll
    for (uint32_t q = 0u; q < kFours; ++q) {
        const uint32_t c = base + 128u * q;
        if (c + 4u <= n) {
            v[q] = *reinterpret_cast<const uint4*>(in + c);
        } else {
            v[q].x = c < n ? in[c] : 0u;
            v[q].y = c + 1u < n ? in[c + 1u] : 0u;
            v[q].z = c + 2u < n ? in[c + 2u] : 0u;
            v[q].w = 0u;
        }
    }
    uint32_t pre = 0u;
    for (uint32_t i = threadIdx.x; i < tile; i += SCAN_THREADS) pre += __ldg(sums + i);
    uint32_t run[kFours], tot = 0u;   // cells before each four in the warp
#pragma unroll
    for (uint32_t q = 0u; q < kFours; ++q) {
        const uint32_t s = v[q].x + v[q].y + v[q].z + v[q].w, inc = warp_incl_scan(s);
        run[q] = tot + inc - s;
        tot += __shfl_sync(0xffffffffu, inc, 31);
    }
    pre = __reduce_add_sync(0xffffffffu, pre);
    if (lane == 0u) {
        warp_tot[warp] = tot;
        warp_pre[warp] = pre;
    }
    __syncthreads();
    uint32_t before = 0u;
#pragma unroll
    for (uint32_t w = 0u; w < SCAN_THREADS / 32u; ++w) before += warp_pre[w] + (w < warp ? warp_tot[w] : 0u);
#pragma unroll
    for (uint32_t q = 0u; q < kFours; ++q) {
        const uint32_t c = base + 128u * q;
        uint4 o;
        o.x = before + run[q];
        o.y = o.x + v[q].x;
        o.z = o.y + v[q].y;
        o.w = o.z + v[q].z;
        if (c + 4u <= n) {
            *reinterpret_cast<uint4*>(out + c) = o;
            *reinterpret_cast<uint4*>(in + c) = make_uint4(0u, 0u, 0u, 0u);
            if (c + 4u == n) out[n] = o.w + v[q].w;   // total after the last cell
        } else if (c < n) {
            out[c] = o.x;
            in[c] = 0u;
            if (c + 1u < n) { out[c + 1u] = o.y; in[c + 1u] = 0u; }
            if (c + 2u < n) { out[c + 2u] = o.z; in[c + 2u] = 0u; }
            out[n] = c + 1u == n ? o.y : c + 2u == n ? o.z : o.w;
        }
    }
}

// The cell starts are invalid once a wait of the scan ran out, and the cell
// order is incomplete once the rank pass met a cell of more than
// SPH_MAX_CELL_OCC particles (it writes no slot of that cell): every pass
// that indexes with them returns at once, and the step reports SPH_ETIMEOUT
// or SPH_ECELL with the particles as they were before the failed substep.
// Each block tests once, at its start; only the rank pass raises a bit this
// tests while later passes could see it, and its output is dropped anyway.
__device__ __forceinline__ bool step_failed(const uint32_t* status) {
    return (__ldcg(status) & (SPH_STATUS_SCAN_TIMEOUT | SPH_STATUS_CELL_OVERFLOW)) != 0u;
}

// ---------------------------------------------------------------------------
// Scatter: provisional slot of each particle in cell order.  The scan's tile
// sums (nsums of them) are left at zero for the next hash.
// A thread's chain of loads (tile, scene, key, start) is all there is to it, so
// a block takes kScatterTiles tiles and has their loads in flight together: with
// one, two, four and eight tiles the sort (this and the rank pass) of 1M
// particles took 33.0, 30.6, 28.7 and 31.2 us, of 8M 212, 189, 178 and 187.
// ---------------------------------------------------------------------------
constexpr uint32_t kScatterTiles = 4u;
__global__ void __launch_bounds__(SPH_TILE) k_scatter(const DevScene* __restrict__ scenes,
                                                      const uint4* __restrict__ tiles, uint32_t ntiles,
                                                      const uint32_t* __restrict__ start,
                                                      const uint32_t* __restrict__ key,
                                                      const uint32_t* __restrict__ slot,
                                                      uint32_t* __restrict__ tmp, uint32_t* __restrict__ sums,
                                                      uint32_t nsums,
                                                      const uint32_t* __restrict__ status) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nsums; i += gridDim.x * blockDim.x) sums[i] = 0u;
    if (step_failed(status)) return;
    bool on[kScatterTiles];
    uint32_t i[kScatterTiles], c[kScatterTiles], to[kScatterTiles];
#pragma unroll
    for (uint32_t q = 0u; q < kScatterTiles; ++q) {
        const uint32_t b = blockIdx.x * kScatterTiles + q;
        const uint4 t = b < ntiles ? tiles[b] : make_uint4(0u, 0u, 0u, 0u);
        on[q] = threadIdx.x < t.z;
        i[q] = t.y + threadIdx.x;
        c[q] = to[q] = 0u;
        if (on[q]) {
            const DevScene sc = scenes[t.x];
            c[q] = sc.cell_base + key[i[q]];
            to[q] = sc.part_base - __ldg(start + sc.cell_base) + slot[i[q]];
        }
    }
#pragma unroll
    for (uint32_t q = 0u; q < kScatterTiles; ++q)
        if (on[q]) to[q] += __ldg(start + c[q]);
#pragma unroll
    for (uint32_t q = 0u; q < kScatterTiles; ++q)
        if (on[q]) tmp[to[q]] = i[q];
}

// ---------------------------------------------------------------------------
// Stable rank inside the cell + gather into cell order.  thrust::sort_by_key
// over u32 keys (fluidsystem.cu:309-313) is a stable radix sort: within a cell
// particles keep their current order.  Each sorted slot's final position is
// the cell start plus the number of cell members with a smaller current
// index, which reproduces that permutation exactly.
// A scene whose last XSPH update is still pending (pend[scene] != 0) has its
// post-integration velocities in V2 and its previous cells in okey: those
// are gathered (the density pass applies the XSPH update); otherwise V0.
// ---------------------------------------------------------------------------
// Where slot f's x lies in the per-axis copies (its y 4, its z 8 floats further).
__device__ __forceinline__ size_t axes_index(uint32_t f) { return 12 * (size_t)(f / 4u) + (f & 3u); }

// The same for HalfScan: a position in its cell's terms, in half precision.  x is
// kept modulo four cells, in [-2, 2), twice: from cell 0 and from cell 2, so that
// any three neighbouring cells lie in order in one of the two; y and z as their
// place in the cell, in [-1/2, 1/2).  Four slots to 32 bytes: x, x from cell 2, y, z.
__device__ __forceinline__ size_t half_index(uint32_t f) { return 16 * (size_t)(f / 4u) + (f & 3u); }
__device__ __forceinline__ void half_axes(__half* H, uint32_t f, const float4& p, float inv_cell) {
    const float ux = p.x * inv_cell, uy = p.y * inv_cell, uz = p.z * inv_cell;
    const float cx = floorf(ux);
    const int c = __float2int_rz(cx);
    H += half_index(f);
    H[0] = __float2half_rn((ux - cx) + (float)((c & 3) - 2));
    H[4] = __float2half_rn((ux - cx) + (float)(((c + 2) & 3) - 2));
    H[8] = __float2half_rn((uy - floorf(uy)) - 0.5f);
    H[12] = __float2half_rn((uz - floorf(uz)) - 0.5f);
}

template <bool HALF>
__global__ void __launch_bounds__(SPH_TILE) k_rank_gather(const DevParams* __restrict__ params,
                                                          const DevScene* __restrict__ scenes,
                                                          const uint4* __restrict__ tiles,
                                                          const uint32_t* __restrict__ start,
                                                          const uint32_t* __restrict__ key,
                                                          const uint32_t* __restrict__ tmp,
                                                          const float4* __restrict__ P0,
                                                          const float4* __restrict__ V0,
                                                          const float4* __restrict__ A0,
                                                          const float4* __restrict__ V2,
                                                          const uint32_t* __restrict__ okey,
                                                          const uint32_t* __restrict__ pend,
                                                          float4* __restrict__ G, float* __restrict__ X,
                                                          float4* __restrict__ A1,
                                                          uint32_t* __restrict__ perm,
                                                          uint32_t* __restrict__ status) {
    if (step_failed(status)) return;
    const uint4 t = tiles[blockIdx.x];
    if (threadIdx.x >= t.z) return;
    const uint32_t g = t.y + threadIdx.x;
    const DevScene sc = scenes[t.x];
    const bool pending = __ldg(pend + t.x) != 0u;
    const uint32_t i = tmp[g];
    const uint32_t s0 = __ldg(start + sc.cell_base);
    const uint32_t c = sc.cell_base + __ldg(key + i);
    const uint32_t b = sc.part_base + (__ldg(start + c) - s0);
    const uint32_t e = sc.part_base + (__ldg(start + c + 1) - s0);
    if (e - b > SPH_MAX_CELL_OCC) {
        atomicOr(status, SPH_STATUS_CELL_OVERFLOW);
        return;
    }
    uint32_t rank = 0;
    for (uint32_t m = b; m < e; ++m) rank += (__ldg(tmp + m) < i) ? 1u : 0u;
    const uint32_t f = b + rank;
    perm[f] = i;
    const float4 p = P0[i];
    if (HALF) {
        half_axes(reinterpret_cast<__half*>(X), f, p, params[t.x].inv_cell);
    } else {
        float* xf = X + axes_index(f);
        xf[0] = p.x;
        xf[4] = p.y;
        xf[8] = p.z;
    }
    float4 v = pending ? V2[i] : V0[i];
    // the cell of the last substep travels with the velocity (w lane) to the
    // density pass's XSPH update, which loads both together
    if (pending) v.w = __uint_as_float(__ldg(okey + i));
    st_float4_pair(G + 2 * (size_t)f, p, v);
    A1[f] = A0[i];
}

// ---------------------------------------------------------------------------
// Density + Tait EOS (computeDensity, fluidphysics.cu:8-84), in two phases.
//
// Phase 1 scans the candidates of the 27 cells with the distance test alone,
// 32 at a time, and appends those within h (j != i), and with HalfScan a few
// just beyond, to the particle's
// neighbour list in shared memory (NbrList).  Phase 2 walks that list, does
// the kernel arithmetic for the pairs (about one candidate in six), so a warp
// does not run it on every candidate that any of its lanes accepts, and
// stores the list for the normal and force passes.  Coincident pairs
// (r^2 <= eps) stay in the list: the density sum and XSPH take them, the other
// passes drop them with their own r^2 > eps test, and all drop those beyond h.  Neighbours past the list's
// end are found again by testing the remaining candidates (walk_tail).  Both
// forms visit neighbours in the same order (rows z outer, then y, then slots,
// the row's cells x ascending); the reference's loop runs the cells x outer
// and z inner (fluidphysics.cu:29-33), the same terms in another order.
//
// With SKIN, phase 1 also records the candidates within the skin radius, one
// word per row of up to 32 candidates (SPH_MASK_SKIN).
//
// Deferred XSPH.  For a scene whose previous substep ended without its XSPH
// update (pend[scene] != 0), G holds that substep's post-integration
// positions (w = its densities) and its post-integration velocities with, in
// their w lane, the cells the particles were sorted into then (okey bits).  The reference's update
// (correctVelocityXSPH, fluidphysics.cu:355-409) sums over pairs with
// r^2 <= h^2 at these positions whose previous cells are adjacent (its cell
// lists were those of the previous sort); every such pair is within h now, so
// phase 2 meets all of them, and the previous-cell test keeps exactly the
// reference's pairs.  The poly6 weight is the one the density sum uses.  The
// corrected velocity goes to the record R, which the force pass reads; without
// a pending update it is G's.
//
// The record.  Position, density, velocity and pressure of a neighbour sit in 32
// bytes, one sector, fetched by one 256-bit load; the squared sound speed comes
// from C2, or with surface tension from the normal's w lane, and 1/rho^2 is
// formed per pair (rcp_exact).  Against separate gathers of position, (rho, p,
// c^2, 1/rho^2) and velocity (48 bytes in three requests) the force pass of the
// 1M dam break went from 230 to 196 us, before the neighbour lists.
// ---------------------------------------------------------------------------
// Neighbour loads in flight per list step, as many as the registers hold.  Where
// occupancy decides: density two (239.5 against 246.5 us with one, 1M dam break),
// force one (two measured the same at 64 registers, where they spill), normals
// four with 48 registers (502 us for 8M particles; two with 48 507, two with 56
// 533, four with 64 539).  FEW: launches of one wave (SPH_ONE_WAVE_THREADS).
template <bool FEW> constexpr int kDensityDepth = FEW ? 4 : 2;
template <int MINB> constexpr int kForceDepth = MINB <= 3 ? 2 : 1;
constexpr int kNormalsDepth = 4;
// Phase 1's distance test: four candidates at a time from the per-axis copies,
// aligned to four slots (the up to three before a row's start and after its end
// are tested too and masked out: no loop for the ragged ends), with the packed
// FP32 instructions of sm_100-class GPUs (add/mul/fma.rn.f32x2): each component
// is rounded exactly as the scalar operation, so r^2 (dot3's fusion order) is
// the same to the bit.  Two neighbouring floats of one axis are the register
// pair that these instructions take; positions of four floats each would be
// taken apart with two moves per pair and axis, and cost 64 instead of 48 bytes
// of L1 bandwidth, the other limit of this pass (238 -> 206 us on the 1M dam
// break, 1.80 -> 1.55 ms on the 8M scene, with one thread per particle; HalfScan
// has taken its place there).
// A candidate's bit is the sign of r^2 - h2n, h2n the float after h^2 (the sign
// of a rounded difference is that of the exact one, so the test is r^2 <= h^2
// to the bit), shifted into the word: the first candidate ends in its highest
// bit.
template <bool SKIN>
struct CandidateScan {
    float2 mx, my, mz, nh2, ns2;
    __device__ __forceinline__ CandidateScan(float px, float py, float pz, float h2, float skin2)
        : mx(make_float2(-px, -px)), my(make_float2(-py, -py)), mz(make_float2(-pz, -pz)) {
        const float nh = -__uint_as_float(__float_as_uint(h2) + 1u), ns = -__uint_as_float(__float_as_uint(skin2) + 1u);
        nh2 = make_float2(nh, nh);
        ns2 = make_float2(ns, ns);
    }
    static __device__ __forceinline__ void shift_in(const float2& x, uint32_t& m) {
        m = __funnelshift_l(__float_as_uint(x.x), m, 1);
        m = __funnelshift_l(__float_as_uint(x.y), m, 1);
    }
    __device__ __forceinline__ void visit2(const float2& x, const float2& y, const float2& z, uint32_t& dm,
                                           uint32_t& sm) const {
        const float2 dx = __fadd2_rn(x, mx), dy = __fadd2_rn(y, my), dz = __fadd2_rn(z, mz);
        const float2 rr = __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
        shift_in(__fadd2_rn(rr, nh2), dm);
        if (SKIN) shift_in(__fadd2_rn(rr, ns2), sm);
    }
    __device__ __forceinline__ void visit4(const float4& x, const float4& y, const float4& z, uint32_t& dm,
                                           uint32_t& sm) const {
        visit2(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y), dm, sm);
        visit2(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w), dm, sm);
    }
};

// The same test in half precision, which finds every candidate within h and one
// in a hundred or so beyond (DevParams::near2); whoever uses the list tests each
// pair exactly.  A candidate is 6 bytes to load instead of 12: each lane's bytes
// pass through the L1 pipe, however many lanes load the same ones, and that pipe
// was busy 80% of the pass, 43% of it with the scan's loads.  Density pass 205 ->
// 185 us (1M dam break), 1.550 -> 1.386 ms (8M tension scene), 71 -> 59 us
// (250,000 particles); the force pass tests pairs it did not before, 145 -> 147
// us and 1.331 -> 1.350 ms.  With several lanes per particle the loads are shared
// out and the longer lists would cost more than they save.
struct HalfScan {
    __half2 nx, ny, nz, nt;   // minus the particle's place in the row's terms; minus the threshold
    float fy, fz;             // its place in its cell
    uint32_t copy;            // which x it compares with: from cell 0 or from cell 2
    __device__ __forceinline__ HalfScan(const DevParams& P, const float4& p, const int3& g) {
        const float fx = p.x * P.inv_cell - (float)g.x;
        fy = p.y * P.inv_cell - (float)g.y;
        fz = p.z * P.inv_cell - (float)g.z;
        // cells g.x - 1 to g.x + 1 in order: g.x is the second or third of the four
        const bool second = ((g.x - 1) & 2) != 0;
        copy = second ? 1u : 0u;
        nx = __float2half2_rn(-(fx + (float)(((g.x + (second ? 2 : 0)) & 3) - 2)));
        nt = __half2half2(__float2half_rd(-P.near2));
        ny = nz = nt;
    }
    // Row r = 3 (1 + its z - the particle's) + 1 + its y - the particle's.
    __device__ __forceinline__ void row(int r) {
        ny = __float2half2_rn((float)(r % 3) - 0.5f - fy);
        nz = __float2half2_rn((float)(r / 3) - 0.5f - fz);
    }
    static __device__ __forceinline__ uint32_t bits(const __half2& x) {
        return *reinterpret_cast<const uint32_t*>(&x);
    }
    static __device__ __forceinline__ __half2 half2(uint32_t x) { return *reinterpret_cast<const __half2*>(&x); }
    // r^2 - threshold of two candidates: negative where near
    __device__ __forceinline__ uint32_t two(uint32_t x, uint32_t y, uint32_t z) const {
        const __half2 dx = __hadd2(half2(x), nx), dy = __hadd2(half2(y), ny), dz = __hadd2(half2(z), nz);
        return bits(__hfma2(dz, dz, __hfma2(dy, dy, __hfma2(dx, dx, nt))));
    }
    // A four's hits into the low bits of m: the signs spread over a byte each, then
    // minus one times minus 8, 4, 2, 1.
    __device__ __forceinline__ void visit4(const uint2& x, const uint4& yz, uint32_t& m) const {
        const uint32_t a = two(x.x, yz.x, yz.z), b = two(x.y, yz.y, yz.w);
        uint32_t s;
        asm("prmt.b32 %0, %1, %2, 0xFDB9;" : "=r"(s) : "r"(a), "r"(b));
        m = (uint32_t)__dp4a((int)s, (int)0xFFFEFCF8, (int)(m << 4));
    }
};

// Candidates from slot `from` on, in row order; f(j) tests the distance.  The
// density pass's: walk_tail there costs its list's loop registers (180 -> 207 us at
// 1M).
template <class F>
__device__ __forceinline__ void walk_rows(const DevParams& P, const uint32_t* __restrict__ start, uint32_t cell_base,
                                          uint32_t delta, int3 g, uint32_t from, F&& f) {
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
        uint32_t jb, je;
        if (!row_range(P, start, cell_base, delta, g, r, jb, je)) continue;
        for (uint32_t j = max(jb, from); j < je; ++j) f(j);
    }
}
// The same without k, in the normal and force passes: those that the candidate scan
// finds (HalfScan with `half_x`, else CandidateScan, of X's positions), 32 tested
// before the first is visited: visiting each candidate to test it runs the pair
// arithmetic on almost every one, as one lane in 32 that accepts is enough.  f(j)
// tests the distance itself.  66,560 particles compressed until most lists end
// early: substep 185 -> 151 us; 64,000 of 260 neighbours with an XSPH pass per
// substep (lists of 56, positions as floats) 1057 -> 865, 250,000 2266 -> 1992.
template <class F>
__device__ __forceinline__ void walk_tail(const DevParams& P, const uint32_t* __restrict__ start, uint32_t cell_base,
                                          uint32_t delta, int3 g, const float4& p, uint32_t k, uint32_t from,
                                          const float* __restrict__ X, bool half_x, F&& f) {
    HalfScan half(P, p, g);
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
        uint32_t jb, je;
        if (!row_range(P, start, cell_base, delta, g, r, jb, je)) continue;
        jb = max(jb, from);
        half.row(r);
#pragma unroll 1
        for (uint32_t c = jb & ~3u; c < je; c += 32u) {
            const uint32_t left = je - c, nq = (min(left, 32u) + 3u) / 4u;
            uint32_t dm = 0u;
            if (half_x) {
                const uint2* hp = reinterpret_cast<const uint2*>(X) + 4 * (size_t)(c / 4u);
                for (uint32_t q = 0u; q < nq; ++q, hp += 4)
                    half.visit4(__ldg(hp + half.copy), __ldg(reinterpret_cast<const uint4*>(hp + 2)), dm);
            } else {
                const CandidateScan<false> scan(p.x, p.y, p.z, P.h2, P.h2);
                const float4* xp = reinterpret_cast<const float4*>(X) + 3 * (size_t)(c / 4u);
                uint32_t none = 0u;
#pragma unroll 1
                for (uint32_t q = 0u; q < nq; ++q, xp += 3)
                    scan.visit4(__ldg(xp), __ldg(xp + 1), __ldg(xp + 2), dm, none);
            }
            uint32_t bits = dm << (32u - 4u * nq);
            if (left < 32u) bits &= ~(~0u >> left);
            if (c < jb) bits &= ~0u >> (jb - c);
            if (k - c < 32u) bits &= ~(0x80000000u >> (k - c));
            while (bits) {
                const uint32_t b = (uint32_t)__clz(bits);
                bits &= ~(0x80000000u >> b);
                f(c + b);
            }
        }
    }
}

// A particle outside the grid: no density, its velocity kept.
__device__ __forceinline__ void density_outside(uint32_t k, const float4& p, const float4& v, float* C2, float4* R,
                                                uint32_t* nbr_out, float4* D = nullptr) {
    C2[k] = 0.f;
    if (D) D[k] = make_float4(p.x, p.y, p.z, 0.f);
    st_float4_pair(R + 2 * (size_t)k, make_float4(p.x, p.y, p.z, 0.f), make_float4(v.x, v.y, v.z, 0.f));
    if (nbr_out) nbr_out[k] = 0;
}
// The density, its equation of state and the record of slot k from the pair
// sums (with xs, XSPH's too).
__device__ __forceinline__ void density_finish(const DevParams& pp, uint32_t k, float sum, bool xs, float ax, float ay,
                                               float az, const float4& p, float4 vi, float* C2, float4* R,
                                               float4* D = nullptr) {
    const float d = fabsf(sdf(pp, p.x, p.y, p.z));
    float corr = sum;
    if (d < pp.h) corr = fmaf(pp.rest_density, 1.0f - boundary_density(pp, d), corr);
    const float rho = (sum == 0.0f) ? pp.rest_density : corr;
    const float ratio = corr * pp.inv_rest_density;
    const float prs = (corr == 0.0f) ? 0.0f : pp.eos_k * (powf(ratio, pp.gamma) - 1.0f);
    C2[k] = pp.gas_constant * powf(ratio, pp.gamma - 1.0f);
    if (xs) {
        vi.x = fmaf(pp.xsph, ax, vi.x);
        vi.y = fmaf(pp.xsph, ay, vi.y);
        vi.z = fmaf(pp.xsph, az, vi.z);
    }
    st_float4_pair(R + 2 * (size_t)k, make_float4(p.x, p.y, p.z, rho), make_float4(vi.x, vi.y, vi.z, prs));
    if (D) D[k] = make_float4(p.x, p.y, p.z, rho);
}

// Registers: with 56 nine blocks of 128 threads share an SM (as many as the lists
// in shared memory allow beside L1), with 64 eight, and a few values spill either
// way.  Loads of three fours in flight with 56, of four with 64: 180 and 185 us
// (1M dam break), 1.334 and 1.387 ms (8M tension scene), 59.6 and 59.2 us (250,000
// particles); four with 56 183 us and 1.361 ms, three with 64 194 us and 1.439 ms,
// 72 (no spills) 192 us, 48 225 us.  FEW: SPH_ONE_WAVE_THREADS.
template <bool SKIN, bool FEW>
__global__ void __maxnreg__(FEW ? 80 : SKIN ? 64 : 56)
k_density(const DevParams* __restrict__ params,
                                                      const DevScene* __restrict__ scenes,
                                                      const uint4* __restrict__ tiles,
                                                      const uint32_t* __restrict__ start,
                                                      const float4* __restrict__ G, const float* __restrict__ X,
                                                      float* __restrict__ C2,
                                                      uint32_t* __restrict__ mask, size_t mask_stride,
                                                      const uint32_t* __restrict__ pend, float4* __restrict__ R,
                                                      float4* __restrict__ D, uint32_t* __restrict__ nbr_out,
                                                      uint32_t ntiles,
                                                      uint32_t* __restrict__ tile_ctr,
                                                      const uint32_t* __restrict__ status) {
  extern __shared__ uint32_t s_list[];
  if (step_failed(status)) return;
  for_each_tile<1>(tiles, ntiles, tile_ctr, [&](const uint4 t) {
    if (threadIdx.x >= t.z) return;
    const uint32_t k = t.y + threadIdx.x;
    const DevScene sc = scenes[t.x];
    const DevParams& pp = params[t.x];
    // phase 1 needs the position alone; the rest of the particle's state is
    // loaded after it (registers)
    float4 p, vi;
    if (SKIN) {
        const float* xk = X + axes_index(k);
        p = make_float4(xk[0], xk[4], xk[8], 0.f);
    } else {
        p = G[2 * (size_t)k];
    }
    const int3 g = grid_of(pp, p.x, p.y, p.z);
    if (!grid_inside(pp, g)) {
        ld_float4_pair(G + 2 * (size_t)k, p, vi);
        density_outside(k, p, vi, C2, R, nbr_out, D);
        return;
    }
    const uint32_t delta = sc.part_base - __ldg(start + sc.cell_base);
    // the skin-radius words serve only the per-substep XSPH pass
    const float h2 = pp.h2, skin2 = SKIN ? pp.skin2 : pp.h2, eps = pp.eps;
    // row starts in a column per thread, list words in a row per thread
    uint32_t* rows = s_list + threadIdx.x;
    const uint32_t rs = blockDim.x;
    uint8_t* list = reinterpret_cast<uint8_t*>(s_list + SPH_NBR_ROWS * rs + threadIdx.x * SPH_NBR_LIST_WORDS);
    NbrHeader hd;
    constexpr uint32_t kCap = SKIN ? SPH_NBR_CAP_SKIN : SPH_NBR_CAP;

    // ---- phase 1: distance test of every candidate ----
    // (CandidateScan; HalfScan without the skin words)
    const CandidateScan<SKIN> scan(p.x, p.y, p.z, h2, skin2);
    HalfScan half(pp, p, g);
    // The row ranges of this thread, loaded together (18 independent loads):
    // starts into the row table, lengths (at most 255 kept: a longer row is
    // cut short as any above 128 is) packed into bytes.
    constexpr int kRows = 9;
    uint32_t lens[(kRows + 3) / 4] = {};
#pragma unroll
    for (int rr = 0; rr < kRows; ++rr) {
        uint32_t jb0, je0;
        if (row_range(pp, start, sc.cell_base, delta, g, rr, jb0, je0)) {
            rows[rr * rs] = jb0;
            lens[rr / 4] |= min(je0 - jb0, 255u) << (8 * (rr % 4));
        }
    }
    uint32_t nrows = 0u;   // rows with a neighbour so far: their starts move to the front of the table
#pragma unroll 1
    for (int rr = 0; rr < kRows; ++rr) {
        const uint32_t len = (lens[0] & 255u);
#pragma unroll
        for (int q = 0; q < (kRows + 3) / 4; ++q)
            lens[q] = (lens[q] >> 8) | (q + 1 < (kRows + 3) / 4 ? lens[q + 1] << 24 : 0u);
        if (len == 0u) continue;
        const uint32_t jb0 = rows[rr * rs];
        if (len > SPH_NBR_MAX_ROW) {   // its offsets do not fit: the list ends here
            hd.over = true;
            if (SKIN) continue;   // later rows still get their skin words
            break;
        }
        if (!SKIN) half.row(rr);
        bool first = true;
        const uint32_t mis = jb0 & 3u, alen = len + mis;   // from the aligned slot on
        uint32_t c0 = 0u, skw = 0u;                        // offset of the chunk there
        do {
            const uint32_t cb = jb0 - mis + c0, clen = min(alen - c0, 32u);
            const float4* xp = reinterpret_cast<const float4*>(X) + 3 * (size_t)(cb / 4u);
            uint32_t dm = 0u, sm = 0u;
            const uint32_t nq = (clen + 3u) / 4u;
            uint32_t q = 0u;
            if constexpr (!SKIN) {
                const uint2* hp = reinterpret_cast<const uint2*>(X) + 4 * (size_t)(cb / 4u);
                const uint2* hx = hp + half.copy;
                // (at rest density a row is six fours or seven)
                auto fours = [&](auto count) {
                    constexpr uint32_t n = decltype(count)::value;
                    for (; q + n <= nq; q += n) {
                        uint2 x[n];
                        uint4 yz[n];
#pragma unroll
                        for (uint32_t i = 0u; i < n; ++i) {
                            x[i] = __ldg(hx + 4 * i);
                            yz[i] = __ldg(reinterpret_cast<const uint4*>(hp + 4 * i + 2));
                        }
                        hx += 4 * n;
                        hp += 4 * n;
#pragma unroll
                        for (uint32_t i = 0u; i < n; ++i) half.visit4(x[i], yz[i], dm);
                    }
                };
                if constexpr (FEW) {
                    fours(std::integral_constant<uint32_t, 4u>());
                    fours(std::integral_constant<uint32_t, 2u>());
                    fours(std::integral_constant<uint32_t, 1u>());
                } else {
                    fours(std::integral_constant<uint32_t, 3u>());
                    for (; q < nq; ++q, hx += 4, hp += 4)
                        half.visit4(__ldg(hx), __ldg(reinterpret_cast<const uint4*>(hp + 2)), dm);
                }
            } else {
                for (; q + 2u <= nq; q += 2u) {
                    const float4 x0 = __ldg(xp), y0 = __ldg(xp + 1), z0 = __ldg(xp + 2);
                    const float4 x1 = __ldg(xp + 3), y1 = __ldg(xp + 4), z1 = __ldg(xp + 5);
                    xp += 6;
                    scan.visit4(x0, y0, z0, dm, sm);
                    scan.visit4(x1, y1, z1, dm, sm);
                }
                if (q < nq) scan.visit4(__ldg(xp), __ldg(xp + 1), __ldg(xp + 2), dm, sm);
            }
            // candidate cb + b in bit 31 - b, those outside the row and the
            // particle itself left out
            const uint32_t so = k - cb;
            uint32_t in = ~0u << (32u - clen);
            if (c0 == 0u) in &= ~0u >> mis;
            if (so < 32u) in &= ~(0x80000000u >> so);
            uint32_t bits = (dm << (32u - 4u * nq)) & in;
            if (SKIN) {
                const uint32_t v = __brev((sm << (32u - 4u * nq)) & in);
                if (c0 == 0u) skw = v >> mis;
                else if (mis != 0u) skw |= v << (32u - mis);   // (rows of up to 32: at most two chunks)
            }
            if (hd.n + (uint32_t)__popc(bits) > kCap) hd.over = true;
            if (bits && !hd.over) {
                int b = __clz(bits);
                if (first) {
                    first = false;
                    rows[nrows++ * rs] = jb0;
                    hd.live |= 1u << rr;
                    bits &= ~(0x80000000u >> b);
                    list[hd.n++] = (uint8_t)(c0 - mis + b + SPH_NBR_NEW_ROW);
                }
                while (bits) {
                    b = __clz(bits);
                    bits &= ~(0x80000000u >> b);
                    list[hd.n++] = (uint8_t)(c0 - mis + b);
                }
            }
            c0 += 32u;
        } while (c0 < alen && (SKIN || !hd.over));
        if (SKIN && len <= 32u) mask[(size_t)(SPH_MASK_SKIN + rr) * mask_stride + k] = skw;
        if (!SKIN && hd.over) break;
    }

    // the last word's padding: offset 0 of the current row (read, not used)
    for (uint32_t m = hd.n; m & 3u; ++m) list[m] = 0;
    mask[k] = hd.pack();

    // ---- phase 2: the density pairs, in candidate order ----
    ld_float4_pair(G + 2 * (size_t)k, p, vi);
    const float h = pp.h, mass = pp.mass, c6 = pp.poly6, two_m = pp.two_mass;
    float sum = 0.0f;
    uint32_t cnt = 0;
    // deferred XSPH of the previous substep (only for particles that had a cell then)
    const uint32_t oi = (__ldg(pend + t.x) != 0u) ? __float_as_uint(vi.w) : SPH_OKEY_NULL;
    const bool xs = oi != SPH_OKEY_NULL;
    // XSPH sums: x and y packed (f32x2), z alone
    float2 axy = make_float2(0.f, 0.f);
    float az = 0.f;
    const float2 mvixy = make_float2(-vi.x, -vi.y);
    // position with the previous density, and the XSPH operands (velocity, and
    // the last cell in the w lane): one 256-bit load
    struct Nbr { float4 q, v; };
    auto load = [&](uint32_t j) {
        Nbr n;
        ld_float4_pair(G + 2 * (size_t)j, n.q, n.v);
        return n;
    };
    auto use = [&](const Nbr& n) {
        const float4 q = n.q, vj = n.v;
        const uint32_t oj = __float_as_uint(vj.w);
        const float2 dxy = __fadd2_rn(make_float2(p.x, p.y), make_float2(-q.x, -q.y));
        const float dx = dxy.x, dy = dxy.y, dz = p.z - q.z;
        const float rr = dot3(dx, dy, dz, dx, dy, dz);
        // the exact test: HalfScan's lists hold pairs just beyond h too, and past the
        // list's end every candidate comes here
        if (rr <= h2) {
            const float w = poly6_r2(rr, h, h2, c6);
            sum = fmaf(mass, w, sum);
            cnt++;
            if (xs) {
                const float rs = p.w + q.w;   // the previous substep's densities
                if (rs > eps && cells_adjacent_fast(oi, oj)) {
                    const float coeff = w * div_approx(two_m, rs);
                    axy = __ffma2_rn(make_float2(coeff, coeff), __fadd2_rn(make_float2(vj.x, vj.y), mvixy), axy);
                    az = fmaf(coeff, vj.z - vi.z, az);
                }
            }
        }
    };
    const uint32_t* words = reinterpret_cast<const uint32_t*>(list);
    NbrRows table(rows, rs);
    uint32_t last = 0u;
    for (uint32_t m = 0; m < hd.n; m += 4u) {
        const uint32_t w = words[m >> 2];
        mask[(size_t)(SPH_NBR_LIST + (m >> 2)) * mask_stride + k] = w;
        last = visit_word<kDensityDepth<FEW>>(w, hd.n - m, table, load, use);
    }
    if (hd.over)
        walk_rows(pp, start, sc.cell_base, delta, g, hd.n ? last + 1u : 0u,
                  [&](uint32_t j) { if (j != k) use(load(j)); });
    density_finish(pp, k, sum, xs, axy.x, axy.y, az, p, vi, C2, R, D);
    if (nbr_out) nbr_out[k] = cnt;
  });
}

// Several lanes per particle (WideShared), for launches of few particles.
template <int LANES>
__global__ void __launch_bounds__(kWideBlock, 7)
k_density_wide(const DevParams* __restrict__ params, const DevScene* __restrict__ scenes,
               const uint4* __restrict__ tiles, const uint32_t* __restrict__ start, const float4* __restrict__ G,
               const float* __restrict__ X, float* __restrict__ C2, uint32_t* __restrict__ mask,
               size_t mask_stride, const uint32_t* __restrict__ pend, float4* __restrict__ R,
               uint32_t* __restrict__ nbr_out, const uint32_t* __restrict__ status) {
  extern __shared__ uint4 s_dyn[];
  if (step_failed(status)) return;
  for_each_tile<LANES>(tiles, 0u, nullptr, [&](const uint4 t) {
    // every lane stays to the end of phase 2
    const uint32_t li = tile_particle<LANES>();
    const bool act = li < t.z;
    uint32_t k = t.y + (act ? li : 0u);
    const DevScene sc = scenes[t.x];
    const DevParams& pp = params[t.x];
    const bool pending = __ldg(pend + t.x) != 0u;
    float4 p, vi;
    ld_float4_pair(G + 2 * (size_t)k, p, vi);
    const int3 g = grid_of(pp, p.x, p.y, p.z);
    const bool work = act && grid_inside(pp, g);
    if (act && !work) density_outside(k, p, vi, C2, R, nbr_out);   // (the same by every lane)
    const uint32_t delta = sc.part_base - __ldg(start + sc.cell_base);
    const float h2 = pp.h2, h = pp.h, eps = pp.eps;
    const WideLanes<LANES> wl;
    WideShared<LANES>& ws = reinterpret_cast<WideShared<LANES>*>(s_dyn)[threadIdx.x / LANES];

    // ---- phase 1: the lanes test up to 32 candidates of a row, four at a time ----
    wide_ranges(pp, start, sc.cell_base, delta, g, work, wl, ws);
    const CandidateScan<false> scan(p.x, p.y, p.z, h2, h2);
    using Chunk = WideChunk<LANES>;
    auto fetch = [&](int r, uint32_t c) {
        const uint32_t jb0 = ws.jb[r];
        Chunk f;
        f.fetch(X, wl, (jb0 & ~3u) + c, jb0 + ws.len[r]);
        return f;
    };
    // The hits of a row's chunk c.
    auto step = [&](int r, uint32_t c, const Chunk& f) {
        const uint32_t jb0 = ws.jb[r], len = ws.len[r], first = (jb0 & ~3u) + 32u * c;
        const uint32_t w = f.hits(scan, wl, first, jb0, jb0 + len, k);
        if (wl.l == 0u && len <= SPH_NBR_MAX_ROW && first < jb0 + len) ws.words[r][c] = w;
        return (uint32_t)__popc(w);
    };
    // The list's rows: it ends before the first that does not fit.
    NbrHeader hd;
    uint32_t at[(8 + LANES) / LANES] = {};   // where this lane's rows begin in the list
    auto row_done = [&](int r, uint32_t hits) {
        hd.over = hd.over || ws.len[r] > SPH_NBR_MAX_ROW || hd.n + hits > SPH_NBR_CAP_WIDE;
        if (hd.over) return;
        if (wl.l == (uint32_t)(r % LANES)) at[r / LANES] = hd.n;
        if (hits) hd.live |= 1u << r;
        hd.n += hits;
    };
#pragma unroll
    for (int z = 0; z < 9; z += 3) {
        if (z != 0 && __all_sync(~0u, hd.over || !work)) break;   // (wide_tail tests the rest)
        const Chunk q[3] = {fetch(z, 0u), fetch(z + 1, 0u), fetch(z + 2, 0u)};   // loaded together
#pragma unroll
        for (int y = 0; y < 3; ++y) {
            const int r = z + y;
            uint32_t hits = step(r, 0u, q[y]);
            const uint32_t len = ws.len[r];
            const uint32_t most = __reduce_max_sync(~0u, len <= SPH_NBR_MAX_ROW ? len + (ws.jb[r] & 3u) : 0u);
            for (uint32_t c = 1u; 32u * c < most; ++c) hits += step(r, c, fetch(r, 32u * c));
            row_done(r, hits);
        }
    }
    __syncwarp();
    // Each lane writes its rows' bytes.
#pragma unroll
    for (uint32_t i = 0u; i < (8u + LANES) / LANES; ++i) {
        const uint32_t r = wl.l + LANES * i;
        if (r < 9u && ((hd.live >> r) & 1u)) {
            const uint32_t jb0 = ws.jb[r], mis = jb0 & 3u;
            ws.rows[__popc(hd.live & ((1u << r) - 1u))] = jb0;
            uint32_t pos = at[i], flag = SPH_NBR_NEW_ROW;
            for (uint32_t c = 0u; 32u * c < ws.len[r] + mis; ++c) {
                uint32_t bits = ws.words[r][c];
                while (bits) {
                    const uint32_t b = (uint32_t)__clz(bits);
                    bits &= ~(0x80000000u >> b);
                    ws.list[pos++] = (uint8_t)(32u * c + b - mis + flag);
                    flag = 0u;
                }
            }
        }
    }
    if (wl.l < ((0u - hd.n) & 3u)) ws.list[hd.n + wl.l] = 0;
    __syncwarp();
    if (work) {
        if (wl.l == 0u) mask[k] = hd.pack();
        for (uint32_t w = wl.l; 4u * w < hd.n; w += LANES)
            mask[(size_t)(SPH_NBR_LIST + w) * mask_stride + k] = reinterpret_cast<const uint32_t*>(ws.list)[w];
    }

    // ---- phase 2 ----
    // Terms: w, the XSPH coefficient, the velocity difference, and the mass.  Lane 0
    // sums w times the mass, lanes 1 to 3 the coefficient times a component, each in
    // list order: the sums one thread forms, to the bit.
    uint32_t cnt = 0u;
    const uint32_t oi = pending ? __float_as_uint(vi.w) : SPH_OKEY_NULL;
    const bool xs = oi != SPH_OKEY_NULL;
    float acc = 0.0f;
    const float c6 = pp.poly6, two_m = pp.two_mass;
    ws.terms[5][wl.l] = pp.mass;
    const float* scale = ws.terms[wl.l == 0u ? 0 : 1];
    const float* value = ws.terms[wl.l == 0u ? 5 : 1 + min(wl.l, 3u)];
    struct Nbr { float4 q, v; };
    auto load = [&](uint32_t j) {
        Nbr n;
        ld_float4_pair(G + 2 * (size_t)j, n.q, n.v);
        return n;
    };
    auto term = [&](const Nbr& n, uint32_t j, bool on) {
        float w = 0.f, c = 0.f;
        float3 dv = make_float3(0.f, 0.f, 0.f);
        const float dx = p.x - n.q.x, dy = p.y - n.q.y, dz = p.z - n.q.z;
        const float rr = dot3(dx, dy, dz, dx, dy, dz);
        on = on && rr <= h2 && j != k;
        if (on) {
            w = poly6_r2(rr, h, h2, c6);
            const float rs = p.w + n.q.w;   // the previous substep's densities
            if (xs && rs > eps && cells_adjacent_fast(oi, __float_as_uint(n.v.w))) {
                c = w * div_approx(two_m, rs);
                dv = make_float3(n.v.x - vi.x, n.v.y - vi.y, n.v.z - vi.z);
            }
        }
        cnt += (uint32_t)__popc(wl.ballot(on));
        ws.terms[0][wl.l] = w;
        ws.terms[1][wl.l] = c;
        ws.terms[2][wl.l] = dv.x;
        ws.terms[3][wl.l] = dv.y;
        ws.terms[4][wl.l] = dv.z;
    };
    auto add = [&]() { acc = wide_sum<LANES>(scale, value, acc); };
    const uint32_t last = wide_list(wl, ws, work ? hd.n : 0u, load, term, add);
    wide_tail(wl, ws, work && hd.over, hd.n ? last + 1u : 0u, k, X, scan, load, term, add);

    // ---- the rest is one thread's work per particle: the block's first threads ----
    if (wl.l < 4u) ws.terms[0][wl.l] = acc;
    if (wl.l == 0u) ws.words[0][0] = work ? cnt : SPH_OKEY_NULL;
    if (!wide_handover<LANES>(t, k)) return;
    const WideShared<LANES>& mine = reinterpret_cast<WideShared<LANES>*>(s_dyn)[threadIdx.x];
    const float* sums = mine.terms[0];
    cnt = mine.words[0][0];
    if (cnt == SPH_OKEY_NULL) return;   // outside the grid
    ld_float4_pair(G + 2 * (size_t)k, p, vi);
    density_finish(pp, k, sums[0], pending && __float_as_uint(vi.w) != SPH_OKEY_NULL, sums[1], sums[2], sums[3], p, vi,
                   C2, R);
    if (nbr_out) nbr_out[k] = cnt;
  });
}

// ---------------------------------------------------------------------------
// Surface normals (computeNormals, fluidphysics.cu:154-210).  Only launched
// for scenes with surface tension: with sigma == 0 the normals enter the
// force only through sigma * (...), which is exactly zero.  Neighbours come
// from the density pass's list, as in the force pass.  LANES > 1: several lanes
// per particle (WideShared).
//
// A gather takes the L1 pipe a cycle for each 128-byte line its lanes touch, and
// the pass little else.  D holds position and density 16 bytes a slot where
// there is room for it (eight neighbours to a line): 528 us for 8M particles,
// 622 from the records (dstride 2), for 2.5 us of the density pass, which writes
// it.
// ---------------------------------------------------------------------------
template <int LANES, bool FEW = false>
__global__ void __maxnreg__(LANES > 1 ? 40 : FEW ? 64 : 48) k_normals(const DevParams* __restrict__ params,
                                                      const DevScene* __restrict__ scenes,
                                                      const uint4* __restrict__ tiles,
                                                      const uint32_t* __restrict__ start,
                                                      const float4* __restrict__ D, uint32_t dstride,
                                                      const float* __restrict__ C2, const float* __restrict__ X,
                                                      bool half_x,
                                                      const uint32_t* __restrict__ mask, size_t mask_stride,
                                                      float4* __restrict__ N, uint32_t ntiles,
                                                      uint32_t* __restrict__ tile_ctr,
                                                      const uint32_t* __restrict__ status) {
  if (step_failed(status)) return;
  extern __shared__ uint4 s_dyn[];
  for_each_tile<LANES>(tiles, ntiles, tile_ctr, [&](const uint4 t) {
    const DevParams& pp = params[t.x];
    if (!(pp.flags & 1u)) return;
    const uint32_t li = tile_particle<LANES>();
    if (LANES == 1 && li >= t.z) return;
    const bool act = li < t.z;
    const uint32_t k = t.y + (act ? li : 0u);
    const DevScene sc = scenes[t.x];
    const WideEarly early = wide_early<LANES>(mask, mask_stride, k);
    const float4 p = D[dstride * (size_t)k];
    const int3 g = grid_of(pp, p.x, p.y, p.z);
    const bool work = act && grid_inside(pp, g);
    if (act && !work) {
        N[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (LANES == 1) return;
    }
    const uint32_t delta = sc.part_base - __ldg(start + sc.cell_base);
    // x and y packed (f32x2, rounded per component as the scalar operations), z alone
    float2 sxy = make_float2(0.f, 0.f);
    float sz = 0.f;
    const float2 pxy = make_float2(p.x, p.y);
    // m gradPoly6(r) rvec / (rho_j r) = m c (h^2 - r^2)^2 rvec / rho_j: the
    // factor r of gradPoly6 cancels the 1/r; h^2 - r^2 is formed from the
    // rounded root r as gradPoly6 forms it (it cancels near r = h)
    const float mc = pp.mass * pp.grad_poly6;
    const float h2 = pp.h2, eps = pp.eps, h = pp.h;
    auto load = [&](uint32_t j) { return __ldg(D + dstride * (size_t)j); };   // w = rho_j
    // the pair's factor of rvec
    auto grad = [&](float r2, float rhoj) {
        const float r = sqrt_exact(r2, rsqrt_approx(r2));
        const float x = fmaf(-r, r, h2);
        return (r >= h) ? 0.0f : div_approx(mc * (x * x), rhoj);
    };
    if constexpr (LANES > 1) {
        const WideLanes<LANES> wl;
        WideShared<LANES>& ws = reinterpret_cast<WideShared<LANES>*>(s_dyn)[threadIdx.x / LANES];
        float acc = 0.f;   // lanes 0 to 2: the sum's components
        const float* value = ws.terms[1 + min(wl.l, 2u)];
        wide_neighbours(
            pp, start, sc.cell_base, delta, g, mask, mask_stride, k, work, early, wl, ws, X,
            CandidateScan<false>(p.x, p.y, p.z, h2, h2), load,
            [&](const float4& q, uint32_t, bool on) {
                const float rx = p.x - q.x, ry = p.y - q.y, rz = p.z - q.z;
                const float r2 = dot3(rx, ry, rz, rx, ry, rz);
                on = on && r2 <= h2 && r2 > eps && q.w > eps;
                float s = 0.f;
                if (on) s = grad(r2, q.w);
                ws.terms[0][wl.l] = s;
                ws.terms[1][wl.l] = on ? rx : 0.f;
                ws.terms[2][wl.l] = on ? ry : 0.f;
                ws.terms[3][wl.l] = on ? rz : 0.f;
            },
            [&]() { acc = wide_sum<LANES>(ws.terms[0], value, acc); });
        sxy = make_float2(wl.get(acc, 0), wl.get(acc, 1));
        sz = wl.get(acc, 2);
        if (!work || wl.l != 0u) return;
    } else {
        auto pair = [&](const float4& q) {
            const float2 rxy = __fadd2_rn(pxy, make_float2(-q.x, -q.y));
            const float rx = rxy.x, ry = rxy.y, rz = p.z - q.z;
            const float r2 = dot3(rx, ry, rz, rx, ry, rz);
            if (r2 <= h2 && r2 > eps && q.w > eps) {
                const float s = grad(r2, q.w);
                sxy = __ffma2_rn(make_float2(s, s), rxy, sxy);
                sz = fmaf(s, rz, sz);
            }
        };
        walk_neighbours<kNormalsDepth>(
            pp, start, sc.cell_base, delta, g, mask, mask_stride, k,
            reinterpret_cast<uint32_t*>(s_dyn) + threadIdx.x, blockDim.x, load,
            pair,
            [&](uint32_t from) {
                walk_tail(pp, start, sc.cell_base, delta, g, p, k, from, X, half_x,
                          [&](uint32_t j) { pair(load(j)); });
            });
    }
    // w: the squared sound speed, so that the force pass gathers it with the normal
    N[k] = make_float4(pp.h * sxy.x, pp.h * sxy.y, pp.h * sz, C2[k]);
  });
}

// ---------------------------------------------------------------------------
// Forces (computeAllForces, fluidphysics.cu:215-352) fused with the leapfrog
// integrator and box boundary (LeapfrogIntegratorOperator,
// fluidintegrator.cu:11-70).  Reads cell-order state (the density pass's
// records R, C2, A1, N), writes the integrated state to P0 (w =
// density), V2,
// A0, each particle's cell to okey, and the next substep's hash of the new
// positions (key, slot, cell counts), so that substep needs no hash pass.
// The integrator sums the
// force buffers in the reference's order, which after the swapped arguments
// at fluidsystem.cu:352-364 is ((pressure + tension) + viscosity) + adhesion.
// ---------------------------------------------------------------------------
// Every operation and its rounding are those of the plain formulas in
// fluidphysics.cu (as the oracle writes them), whatever form computes it: a
// particle that rests against a wall takes the contact branch or not by its
// last bit, so results stay comparable over many substeps only if all of them
// agree to the bit.  Leaving the constant factors to the end of the sums and
// h - r as (h^2 - r^2)/(h + r) measured 139 against 145 us (1M dam break) and
// 1.22 against 1.33 ms (8M tension scene), but moved such particles.
//
// Short forms.  The pair loop takes 1/rho^2 from rcp_exact, its quotient from
// div_approx, and multiplies the viscosity of a pair that does not approach by zero.
// Where rho^2 or a product leaves the normal numbers, or a sound speed is infinite,
// these give NaN or an infinity where the plain formulas mostly do not; only a rho^2
// above 2^126 gives 0 instead of its reciprocal, which no sum shows unless the
// particle's own density or the rest density is that large too.  A particle of such
// sums or densities adds up its pressure and viscosity again (plain_pairs), with
// sums of the plain formulas.  Substep 355.0 -> 355.5 us (1M dam break), 67.8 -> 68.6
// (82,484 particles), 3387 -> 3376 (8M): pairs need no test.  With one per pair the
// force pass of the 8M scene took 1406 instead of 1370 us, with a division behind a
// branch 1495, and with two loops and a word from the density pass that chooses
// between them the substep of 82,484 particles 69.2.
constexpr float kShortFormDensity = 0x1p40f;
__device__ __forceinline__ void plain_pairs(const DevParams& P, const uint32_t* __restrict__ start, uint32_t cell_base,
                                            uint32_t delta, int3 g, uint32_t k, const float4* __restrict__ R,
                                            const float* __restrict__ C2, float3& fp, float3& fv) {
    float4 pi, vi;
    ld_float4_pair(R + 2 * (size_t)k, pi, vi);
    const float csi = C2[k], ri2 = pi.w * pi.w;
    fp = fv = make_float3(0.f, 0.f, 0.f);
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
        uint32_t j, je;
        if (!row_range(P, start, cell_base, delta, g, r, j, je)) continue;
#pragma unroll 1
        for (; j < je; ++j) {
            float4 pj, vj;
            ld_float4_pair(R + 2 * (size_t)j, pj, vj);
            const float rx = pj.x - pi.x, ry = pj.y - pi.y, rz = pj.z - pi.z;
            const float r2 = dot3(rx, ry, rz, rx, ry, rz);
            if (!(r2 <= P.h2 && r2 > FLT_MIN && pj.w > FLT_MIN) || j == k) continue;
            const float d = sqrtf(r2);
            const float ux = dot3(vj.x - vi.x, vj.y - vi.y, vj.z - vi.z, rx, ry, rz);
            const float Pv = __fdividef((-P.viscosity * (csi + C2[j])) * (P.h * ux), (r2 + P.visc_eps) * (pi.w + pj.w));
            const float mid = vj.w / ri2 + vi.w / (pj.w * pj.w);
            const float mp = mid + (ux < 0.0f ? Pv : 0.0f);
            const float sr = (P.mass * ((P.grad_spiky * (P.h - d)) * (P.h - d))) * rsqrt_approx(r2);
            const float cx = sr * rx, cy = sr * ry, cz = sr * rz;
            fp.x = fmaf(cx, mid, fp.x); fp.y = fmaf(cy, mid, fp.y); fp.z = fmaf(cz, mid, fp.z);
            fv.x = fmaf(cx, mp, fv.x); fv.y = fmaf(cy, mp, fv.y); fv.z = fmaf(cz, mp, fv.z);
        }
    }
}

// TENSION = false is the build for launches where no scene has surface
// tension (the tension terms are then compiled out).  MINB is the register
// budget as resident blocks of 256 threads per SM: 3 (80 registers, no
// spills) or 4 (64 registers, more warps per SM, a few spilled values in the
// tension build).
// LANES > 1: several lanes per particle through the pair sums (WideShared), then
// one.
template <bool TENSION, int MINB, int LANES = 1>
__global__ void __launch_bounds__(LANES > 1 ? kWideBlock : SPH_TILE, MINB)
k_force_integrate(const DevParams* __restrict__ params,
                                                              const DevScene* __restrict__ scenes,
                                                              const uint4* __restrict__ tiles,
                                                              const uint32_t* __restrict__ start,
                                                              const float4* __restrict__ R,
                                                              const float* __restrict__ C2,
                                                              const float4* __restrict__ A1,
                                                              const float4* __restrict__ N,
                                                              const float* __restrict__ X, bool half_x,
                                                              const uint32_t* __restrict__ mask, size_t mask_stride,
                                                              float4* __restrict__ P0, float4* __restrict__ V2,
                                                              float4* __restrict__ A0, uint32_t* __restrict__ maxdisp,
                                                              uint32_t* __restrict__ okey, uint32_t* __restrict__ pend,
                                                              uint32_t* __restrict__ count,
                                                              uint32_t* __restrict__ sums,
                                                              uint32_t* __restrict__ key,
                                                              uint32_t* __restrict__ slot, uint32_t* __restrict__ status,
                                                              float4* __restrict__ dbg_forces, uint32_t ntiles,
                                                              uint32_t* __restrict__ tile_ctr) {
  if (step_failed(status)) return;
  extern __shared__ uint4 s_dyn[];
  for_each_tile<LANES>(tiles, ntiles, tile_ctr, [&](const uint4 t) {
    const uint32_t li = tile_particle<LANES>();
    const bool act = li < t.z;
    // lanes that integrate a particle of this tile (taken before any divergence)
    unsigned lanes = __ballot_sync(0xffffffffu, act);
    if (LANES == 1 && !act) return;
    uint32_t k = t.y + (act ? li : 0u);
    const DevScene sc = scenes[t.x];
    const DevParams& pp = params[t.x];
    // the scene's XSPH update is now pending (applied by the next density
    // pass, or by k_xsph right after this pass)
    if (threadIdx.x == 0) pend[t.x] = 1u;
    const WideEarly early = wide_early<LANES>(mask, mask_stride, k);
    if (LANES > 1 && threadIdx.x < kWideBlock / LANES && blockIdx.x * (kWideBlock / LANES) + threadIdx.x < t.z)
        prefetch_l1(A1 + t.y + blockIdx.x * (kWideBlock / LANES) + threadIdx.x);
    float4 pi, vi;
    ld_float4_pair(R + 2 * (size_t)k, pi, vi);
    int3 g = grid_of(pp, pi.x, pi.y, pi.z);
    const bool tension = TENSION && (pp.flags & 1u) != 0u;
    bool inside = grid_inside(pp, g);
    float fpx = 0.f, fpy = 0.f, fpz = 0.f;   // pressure
    float fvx = 0.f, fvy = 0.f, fvz = 0.f;   // "viscosity" (pressure re-added)
    float ftx = 0.f, fty = 0.f, ftz = 0.f;   // tension
    float fax = 0.f, fay = 0.f, faz = 0.f;   // adhesion
    const uint32_t delta = sc.part_base - __ldg(start + sc.cell_base);
    float4 ni = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tension && inside) ni = N[k];
    const float ri = pi.w, pri = vi.w, csi = C2[k], inv_ri2 = 1.0f / (ri * ri);
    // 2 rho0 / (rho_i + rho_i) of the tension sum (fluidphysics.cu:293), once per particle
    const float tden = (2.0f * pp.rest_density) / (ri + ri);
    // per-scene constants of the pair loop, held in registers
    const float h2 = pp.h2, hh = pp.h, visc_eps = pp.visc_eps, visc = -pp.viscosity;
    const float mass = pp.mass, gsp = pp.grad_spiky;
    const float sm = -pp.surface_tension * mass;
    const Cohesion coh(pp);
    // One pair: neighbour j with its record, and its normal with the squared
    // sound speed.  press(mid, mp, c) takes the pressure and viscosity terms'
    // scales and the spiky gradient along rvec; tens(t) the tension term.  The test
    // r^2 <= h^2 decides what counts: lists hold pairs just beyond h too (HalfScan),
    // and what is found past their end may lie there as well.
    // r is the correctly rounded root: h - r cancels, and pairs at r ~ h must see
    // the reference's r; 1/r and the quotients only scale (approximate).  At
    // r = h the gradient and the cohesion vanish with h - r.  j == k has r^2 = 0
    // and drops out with the coincident pairs.
    auto pair = [&](const float4& pj, const float4& vj, const float4& nj, auto&& press, auto&& tens) {
        const float rx = pj.x - pi.x, ry = pj.y - pi.y, rz = pj.z - pi.z;
        const float r2 = dot3(rx, ry, rz, rx, ry, rz);
        if (r2 <= h2 && r2 > FLT_MIN && pj.w > FLT_MIN) {
            const float inv_r = rsqrt_approx(r2), r = sqrt_exact(r2, inv_r);
            // artificial viscosity -visc (cs_i + cs_j) mu / (rho_i + rho_j),
            // mu = h ux / (r^2 + 0.01 h^2), only for approaching pairs (ux < 0)
            const float ux = fminf(dot3(vj.x - vi.x, vj.y - vi.y, vj.z - vi.z, rx, ry, rz), 0.0f);
            const float Pi = div_approx((visc * (csi + nj.w)) * (hh * ux), (r2 + visc_eps) * (ri + pj.w));
            const float mid = vj.w * inv_ri2 + pri * rcp_exact(pj.w * pj.w);
            const float hr = hh - r;
            const float sr = (mass * ((gsp * hr) * hr)) * inv_r;
            press(mid, mid + Pi, make_float3(sr * rx, sr * ry, sr * rz));
            if (tension) {
                // Akinci cohesion + curvature (fluidphysics.cu:291-293).  With
                // sigma == 0 the tension force is sigma * (finite sum) = 0, so
                // the term is skipped.
                const float sc2 = (-mass * mass) * coh(r, hr) * inv_r;
                tens(make_float3(sc2 * rx + sm * (ni.x - nj.x), sc2 * ry + sm * (ni.y - nj.y),
                                 sc2 * rz + sm * (ni.z - nj.z)));
            }
        }
    };
    struct Nbr { float4 p, v, n; };
    auto load = [&](uint32_t j) {
        Nbr r;
        ld_float4_pair(R + 2 * (size_t)j, r.p, r.v);
        r.n = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tension) r.n = __ldg(N + j);
        else r.n.w = __ldg(C2 + j);
        return r;
    };
    if constexpr (LANES > 1) {
        // Terms: the two scales, the gradient, then the tension and its factor.
        // Lanes 0 to 2 sum one component each, in list order.
        const WideLanes<LANES> wl;
        WideShared<LANES>& ws = reinterpret_cast<WideShared<LANES>*>(s_dyn)[threadIdx.x / LANES];
        const uint32_t axis = min(wl.l, 2u);
        float sum_p = 0.f, sum_v = 0.f, sum_t = 0.f;
        wide_neighbours(
            pp, start, sc.cell_base, delta, g, mask, mask_stride, k, act && inside, early, wl, ws, X,
            CandidateScan<false>(pi.x, pi.y, pi.z, h2, h2), load,
            [&](const Nbr& r, uint32_t, bool on) {
                float o[9] = {};   // (zeros for lanes without a pair, the tension's factor too: it may be infinite)
                if (on)
                    pair(r.p, r.v, r.n,
                         [&](float mid, float mp, const float3& c) {
                             o[0] = mid; o[1] = mp; o[2] = c.x; o[3] = c.y; o[4] = c.z;
                         },
                         [&](const float3& t) { o[5] = t.x; o[6] = t.y; o[7] = t.z; o[8] = tden; });
#pragma unroll
                for (int c = 0; c < (TENSION ? 9 : 5); ++c) ws.terms[c][wl.l] = o[c];
            },
            [&]() {
                sum_p = wide_sum<LANES>(ws.terms[0], ws.terms[2u + axis], sum_p);
                sum_v = wide_sum<LANES>(ws.terms[1], ws.terms[2u + axis], sum_v);
                if (tension) sum_t = wide_sum<LANES>(ws.terms[8], ws.terms[5u + axis], sum_t);
            });
        // the rest is one thread's work per particle: the block's first threads
        ws.terms[0][wl.l] = sum_p;
        ws.terms[1][wl.l] = sum_v;
        ws.terms[2][wl.l] = sum_t;
        if (!wide_handover<LANES>(t, k)) return;
        lanes = ~0u >> (32u - min(kWideBlock / LANES, t.z - blockIdx.x * (kWideBlock / LANES)));
        const WideShared<LANES>& w = reinterpret_cast<WideShared<LANES>*>(s_dyn)[threadIdx.x];
        fpx = w.terms[0][0]; fpy = w.terms[0][1]; fpz = w.terms[0][2];
        fvx = w.terms[1][0]; fvy = w.terms[1][1]; fvz = w.terms[1][2];
        ftx = w.terms[2][0]; fty = w.terms[2][1]; ftz = w.terms[2][2];
        ld_float4_pair(R + 2 * (size_t)k, pi, vi);
        g = grid_of(pp, pi.x, pi.y, pi.z);
        inside = grid_inside(pp, g);
    } else if (inside) {
        auto visit = [&](const Nbr& r) {
            pair(r.p, r.v, r.n,
                 [&](float mid, float mp, const float3& c) {
                     fpx = fmaf(c.x, mid, fpx); fpy = fmaf(c.y, mid, fpy); fpz = fmaf(c.z, mid, fpz);
                     fvx = fmaf(c.x, mp, fvx); fvy = fmaf(c.y, mp, fvy); fvz = fmaf(c.z, mp, fvz);
                 },
                 [&](const float3& t) {
                     ftx = fmaf(tden, t.x, ftx); fty = fmaf(tden, t.y, fty); ftz = fmaf(tden, t.z, ftz);
                 });
        };
        walk_neighbours<kForceDepth<MINB>>(
            pp, start, sc.cell_base, delta, g, mask, mask_stride, k,
            reinterpret_cast<uint32_t*>(s_dyn) + threadIdx.x, blockDim.x, load,
            visit, [&](uint32_t from) {
                walk_tail(pp, start, sc.cell_base, delta, g, pi, k, from, X, half_x,
                          [&](uint32_t j) { visit(load(j)); });
            });
    }
    if (inside) {
        if (!(fabsf(fvx) + fabsf(fvy) + fabsf(fvz) <= FLT_MAX && fmaxf(pi.w, pp.rest_density) <= kShortFormDensity)) {
            float3 fp, fv;
            plain_pairs(pp, start, sc.cell_base, delta, g, k, R, C2, fp, fv);
            fpx = fp.x; fpy = fp.y; fpz = fp.z;
            fvx = fv.x; fvy = fv.y; fvz = fv.z;
        }
        fvx = pp.viscosity * fvx; fvy = pp.viscosity * fvy; fvz = pp.viscosity * fvz;
        ftx = pp.surface_tension * ftx; fty = pp.surface_tension * fty; ftz = pp.surface_tension * ftz;
        const float z = -fminf(sdf(pp, pi.x, pi.y, pi.z), 0.0f) * 0.25f * pp.inv_particle_size;
        if (z < 1.0f) {
            const float3 nb = sdf_normal(pp, pi.x, pi.y, pi.z);
            const float denom = 1.0f / powf(1.0f - z, 3.0f);
            const float a = pp.adhesion * pi.w * pp.inv_rest_density * denom;
            fax = a * nb.x; fay = a * nb.y; faz = a * nb.z;
        }
    }
    if (dbg_forces) {
        dbg_forces[4 * (size_t)k + 0] = make_float4(fpx, fpy, fpz, 0.f);
        dbg_forces[4 * (size_t)k + 1] = make_float4(ftx, fty, ftz, 0.f);
        dbg_forces[4 * (size_t)k + 2] = make_float4(fax, fay, faz, 0.f);
        dbg_forces[4 * (size_t)k + 3] = make_float4(fvx, fvy, fvz, 0.f);
    }
    // ---- leapfrog integrator + boundary ----
    const float4 ai = A1[k];
    const float Fx = ((fpx + ftx) + fvx) + fax;
    const float Fy = ((fpy + fty) + fvy) + fay;
    const float Fz = ((fpz + ftz) + fvz) + faz;
    float anx = fmaf(Fx, pp.mass, pp.grav_x), any = fmaf(Fy, pp.mass, pp.grav_y), anz = fmaf(Fz, pp.mass, pp.grav_z);
    float sq = dot3(anx, any, anz, anx, any, anz);
    if (sq > pp.acc_limit2) {
        const float s = pp.acc_limit / sqrtf(sq);
        anx = anx * s; any = any * s; anz = anz * s;
    }
    float px = pi.x + fmaf(vi.x, pp.dt, (0.5f * ai.x) * pp.dtdt);
    float py = pi.y + fmaf(vi.y, pp.dt, (0.5f * ai.y) * pp.dtdt);
    float pz = pi.z + fmaf(vi.z, pp.dt, (0.5f * ai.z) * pp.dtdt);
    float vx = fmaf(0.5f * (ai.x + anx), pp.dt, vi.x);
    float vy = fmaf(0.5f * (ai.y + any), pp.dt, vi.y);
    float vz = fmaf(0.5f * (ai.z + anz), pp.dt, vi.z);
    sq = dot3(vx, vy, vz, vx, vy, vz);
    if (sq > pp.vel_limit2) {
        const float s = pp.vel_limit / sqrtf(sq);
        vx = vx * s; vy = vy * s; vz = vz * s;
    }
    const float d = sdf(pp, px, py, pz);
    if (d > -pp.particle_size) {
        const float3 nb = sdf_normal(pp, px, py, pz);
        const float s = -(d + pp.particle_size);
        px = fmaf(s, nb.x, px); py = fmaf(s, nb.y, py); pz = fmaf(s, nb.z, pz);
        const float kk = (1.0f + pp.vdamp) * dot3(nb.x, nb.y, nb.z, vx, vy, vz);
        vx = fmaf(-kk, nb.x, vx); vy = fmaf(-kk, nb.y, vy); vz = fmaf(-kk, nb.z, vz);
    }
    P0[k] = make_float4(px, py, pz, pi.w);
    V2[k] = make_float4(vx, vy, vz, 0.f);
    A0[k] = make_float4(anx, any, anz, 0.f);
    // The next substep's hash (k_hash's work, on the position just written):
    // its cell key, a provisional slot from the cell count (made stable by
    // the rank pass) and the non-finite check.  The cell XSPH's cell lists
    // use is recorded with SPH_OKEY_MOVED when the particle leaves it.
    const int3 gn = grid_of(pp, px, py, pz);
    const bool inside_new = grid_inside(pp, gn);
    if (!(isfinite(px) && isfinite(py) && isfinite(pz))) atomicOr(status, SPH_STATUS_NONFINITE);
    const uint32_t local = inside_new ? (uint32_t)gn.x + (uint32_t)gn.y * pp.gx + (uint32_t)gn.z * pp.gxy : pp.ncells;
    key[k] = local;
    slot[k] = count_cell(lanes, sc.cell_base + local, count, sums);
    okey[k] = grid_inside(pp, g)
                  ? (pack_cell(g) | ((inside_new && pack_cell(gn) == pack_cell(g)) ? 0u : SPH_OKEY_MOVED))
                  : SPH_OKEY_NULL;
    // largest displacement of the substep in units of h (squared), for XSPH's
    // use of the neighbour masks; NaN compares above every finite value
    const float ddx = px - pi.x, ddy = py - pi.y, ddz = pz - pi.z;
    const float d2 = dot3(ddx, ddy, ddz, ddx, ddy, ddz) * pp.inv_h2;
    const uint32_t bits = (d2 != d2) ? 0x7fffffffu : __float_as_uint(d2);
    if (maxdisp) {   // only scenes with a per-substep XSPH pass use the skin masks
        const uint32_t wmax = __reduce_max_sync(lanes, bits);
        if ((threadIdx.x & 31u) == (uint32_t)(__ffs(lanes) - 1)) atomicMax(maxdisp, wmax);
    }
  });
}

// One XSPH pair term (fluidphysics.cu:392-401).
__device__ __forceinline__ void xsph_pair(const float4* __restrict__ P0, const float4* __restrict__ V2, uint32_t j,
                                          uint32_t k, const float4& pi, const float4& vi, float h2, float h, float c6,
                                          float two_m, float eps, float& sx, float& sy, float& sz) {
    const float4 q = __ldg(P0 + j);
    const float4 vj = __ldg(V2 + j);   // issued with the position: most candidates are neighbours
    const float dx = pi.x - q.x, dy = pi.y - q.y, dz = pi.z - q.z;
    const float rr = dot3(dx, dy, dz, dx, dy, dz);
    const float rs = pi.w + q.w;
    if (rr <= h2 && rs > eps && j != k) {
        const float r = sqrtf(rr);
        const float x = fmaf(-r, r, h2);
        const float w = (r >= h) ? 0.0f : c6 * (x * x * x);
        const float coeff = w * __fdividef(two_m, rs);
        sx = fmaf(coeff, vj.x - vi.x, sx);
        sy = fmaf(coeff, vj.y - vi.y, sy);
        sz = fmaf(coeff, vj.z - vi.z, sz);
    }
}

// ---------------------------------------------------------------------------
// XSPH velocity smoothing (correctVelocityXSPH, fluidphysics.cu:355-409):
// post-integration positions, this substep's cell lists and densities.  The
// reference updates velocities in place while neighbours read them (a race);
// here reads see V2 and the result goes to V0 (Jacobi).
// ---------------------------------------------------------------------------
// WALK selects the candidate walk: 0 one loop flattened across the rows, 1 one
// loop per (y,z) row; both visit the same candidates in the same order.  (The
// row-table walk of the force pass measured slower here, 72 registers against
// 54: the pair term is too light to pay for the table.)
// (no __launch_bounds__: with it ptxas caps this kernel at 48 registers and spills)
template <int WALK>
__global__ void k_xsph(const DevParams* __restrict__ params,
                                                   const DevScene* __restrict__ scenes,
                                                   const uint4* __restrict__ tiles,
                                                   const uint32_t* __restrict__ start,
                                                   const float4* __restrict__ G,
                                                   const float4* __restrict__ P0,
                                                   const float4* __restrict__ V2,
                                                   const uint32_t* __restrict__ mask, size_t mask_stride,
                                                   const uint32_t* __restrict__ maxdisp, float4* __restrict__ V0,
                                                   uint32_t* __restrict__ pend, uint32_t ntiles,
                                                   uint32_t* __restrict__ tile_ctr,
                                                   const uint32_t* __restrict__ status) {
  if (step_failed(status)) return;
  for_each_tile<1>(tiles, ntiles, tile_ctr, [&](const uint4 t) {
    if (threadIdx.x >= t.z) return;
    const uint32_t k = t.y + threadIdx.x;
    const DevScene sc = scenes[t.x];
    const DevParams& pp = params[t.x];
    if (pp.flags & SPH_FLAG_DEFER_XSPH) return;   // the next density pass applies it
    if (threadIdx.x == 0) pend[t.x] = 0u;         // the update is applied here
    const float4 vi = V2[k];
    const float4 old = G[2 * (size_t)k];   // the cell this particle was sorted into
    const int3 g = grid_of(pp, old.x, old.y, old.z);
    if (!grid_inside(pp, g)) {
        V0[k] = vi;
        return;
    }
    const float4 pi = P0[k];    // post-integration position, w = density
    const uint32_t delta = sc.part_base - __ldg(start + sc.cell_base);
    const float h2 = pp.h2, h = pp.h, c6 = pp.poly6, two_m = pp.two_mass, eps = pp.eps;
    float sx = 0.f, sy = 0.f, sz = 0.f;
    // The masks hold every candidate within (1 + skin) h at the old
    // positions; a pair can close to h after the move only if the particles
    // moved less than skin*h/2 each, which the force pass recorded.
    uint32_t j;
    const bool masked = __uint_as_float(__ldg(maxdisp)) <= pp.xsph_disp_limit2;
    const uint32_t* skin = mask + SPH_MASK_SKIN * mask_stride;
    if (WALK == 1) {
        auto visit = [&](uint32_t jj) { xsph_pair(P0, V2, jj, k, pi, vi, h2, h, c6, two_m, eps, sx, sy, sz); };
        if (masked) for_masked(pp, start, sc.cell_base, delta, g, skin, mask_stride, k, visit);
        else for_candidates(pp, start, sc.cell_base, delta, g, visit);
    } else if (masked) {
        MaskWalk walk(pp, start, sc.cell_base, delta, g, skin, mask_stride, k);
        while (walk.next(j)) xsph_pair(P0, V2, j, k, pi, vi, h2, h, c6, two_m, eps, sx, sy, sz);
    } else {
        RangeWalk walk(pp, start, sc.cell_base, delta, g);
        while (walk.next(j)) xsph_pair(P0, V2, j, k, pi, vi, h2, h, c6, two_m, eps, sx, sy, sz);
    }
    V0[k] = make_float4(fmaf(pp.xsph, sx, vi.x), fmaf(pp.xsph, sy, vi.y), fmaf(pp.xsph, sz, vi.z), 0.f);
  });
}

// ---------------------------------------------------------------------------
// The velocities of a density pass (in R, cell order) back in the state order
// of the substep before it (slot perm[f]): the export of a scene whose XSPH
// update was pending (packed xyz into `out`, particle perm[f] - base), and its
// materialisation into the state (V0, clearing the scene's pending flag).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SPH_TILE) k_unsort_vel(const uint4* __restrict__ tiles,
                                                         const uint32_t* __restrict__ perm,
                                                         const float4* __restrict__ R, uint32_t base,
                                                         float* __restrict__ out, float4* __restrict__ V0,
                                                         uint32_t* __restrict__ pend,
                                                         const uint32_t* __restrict__ status,
                                                         uint32_t* __restrict__ gate, uint32_t n,
                                                         uint32_t* __restrict__ status_out) {
    const uint4 t = tiles[blockIdx.x];
    if (status_out && blockIdx.x == 0 && threadIdx.x == 0) *status_out = __ldcg(status);
    // the status word of a force pass run ahead (launch_unsort_vel): it
    // starts failed, so that pass does nothing, when the prefix reported an error
    if (gate && blockIdx.x == 0 && threadIdx.x == 0) *gate = __ldcg(status) != 0u ? SPH_STATUS_SCAN_TIMEOUT : 0u;
    // a failed prefix leaves perm incomplete (the host reports its error)
    if (step_failed(status)) return;
    if (pend && blockIdx.x == 0 && threadIdx.x == 0) pend[t.x] = 0u;
    if (threadIdx.x >= t.z) return;
    const uint32_t f = t.y + threadIdx.x;
    const uint32_t i = __ldg(perm + f);
    if (i - base >= n) return;   // every slot of the scene, once, after a complete prefix
    const float4 r = R[2 * (size_t)f + 1];
    const float4 v = make_float4(r.x, r.y, r.z, 0.f);
    if (out) {
        const size_t o = 3 * (size_t)(i - base);
        out[o] = v.x;
        out[o + 1] = v.y;
        out[o + 2] = v.z;
    }
    if (V0) V0[i] = v;
}

// ---------------------------------------------------------------------------
// Undo a force pass run ahead of the step that takes it: the state before it
// is what the prefix gathered (G, A1; G holds the post-integration
// velocities of a scene whose XSPH update is pending, with its previous cells
// in the w lane), scattered back to the slots it came from.  The force pass
// writes no array the prefix wrote, so the prefix stays valid.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SPH_TILE) k_undo_ahead(const uint4* __restrict__ tiles,
                                                         const uint32_t* __restrict__ perm,
                                                         const float4* __restrict__ G,
                                                         const float4* __restrict__ A1, float4* __restrict__ P0,
                                                         float4* __restrict__ V2, float4* __restrict__ A0,
                                                         uint32_t* __restrict__ okey) {
    const uint4 t = tiles[blockIdx.x];
    if (threadIdx.x >= t.z) return;
    const uint32_t f = t.y + threadIdx.x;
    const uint32_t i = __ldg(perm + f);
    float4 p, v;
    ld_float4_pair(G + 2 * (size_t)f, p, v);
    P0[i] = p;
    V2[i] = make_float4(v.x, v.y, v.z, 0.f);
    A0[i] = A1[f];
    okey[i] = __float_as_uint(v.w);
}

// ---------------------------------------------------------------------------
// Host<->device layout helpers and the lattice generator.
// ---------------------------------------------------------------------------
__global__ void k_unpack_state(const float* __restrict__ pos, const float* __restrict__ vel, uint32_t n,
                               uint32_t base, float4* __restrict__ P0, float4* __restrict__ V0,
                               float4* __restrict__ A0, float* __restrict__ C2,
                               float4* __restrict__ R) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t s = base + i;
    P0[s] = make_float4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], 0.f);
    V0[s] = vel ? make_float4(vel[3 * i], vel[3 * i + 1], vel[3 * i + 2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    A0[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    C2[s] = 0.f;
    R[2 * (size_t)s].w = 0.f;
    R[2 * (size_t)s + 1].w = 0.f;
}

// Overwrite positions of slots [base, base+n) keeping the rest of the state
// (createFluidBlock writes m_Points element by element, fluidsystem.cu:119-123).
__global__ void k_set_positions(const float* __restrict__ pos, uint32_t n, uint32_t base, float4* __restrict__ P0) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 old = P0[base + i];
    P0[base + i] = make_float4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], old.w);
}

// Export: positions, density colour (DensityColourOperator, fluidutil.cu:67-80)
// and velocities, packed xyz.
__global__ void k_pack_state(const float4* __restrict__ P0, const float4* __restrict__ V0, uint32_t n,
                             uint32_t base, float inv_rest_density, float* __restrict__ pos,
                             float* __restrict__ colour, float* __restrict__ vel) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = P0[base + i];
    const float4 v = V0[base + i];
    if (pos) { pos[3 * i] = p.x; pos[3 * i + 1] = p.y; pos[3 * i + 2] = p.z; }
    if (vel) { vel[3 * i] = v.x; vel[3 * i + 1] = v.y; vel[3 * i + 2] = v.z; }
    if (colour) {
        const float ratio = p.w * inv_rest_density;
        float r = 1.0f, gg = 0.0f, b = 0.0f;
        if (ratio < 1.0f) { r = 0.0f; gg = ratio; b = 1.0f - ratio; }
        else if (ratio < 2.0f) { r = ratio - 1.0f; gg = 2.0f - ratio; b = 0.0f; }
        colour[3 * i] = r; colour[3 * i + 1] = gg; colour[3 * i + 2] = b;
    }
}

// Lattice block with seeded jitter; site (ix,iy,iz) -> particle
// (ix*ny + iy)*nz + iz.  Coordinate: lo + (i + 0.5)*spacing + (2u-1)*jitter.
__global__ void k_lattice(LatticeSpec spec, uint32_t base, float4* __restrict__ P0, float4* __restrict__ V0,
                          float4* __restrict__ A0, float* __restrict__ C2,
                               float4* __restrict__ R) {
    const uint32_t n = spec.nx * spec.ny * spec.nz;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t iz = i % spec.nz, iy = (i / spec.nz) % spec.ny, ix = i / (spec.nz * spec.ny);
    const uint32_t idx[3] = {ix, iy, iz};
    float c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float u = uniform01(spec.seed, 3ull * i + a);
        const float j = (2.0f * u - 1.0f) * spec.jitter;
        c[a] = (spec.lo[a] + ((float)idx[a] + 0.5f) * spec.spacing) + j;
    }
    const uint32_t s = base + i;
    P0[s] = make_float4(c[0], c[1], c[2], 0.f);
    V0[s] = make_float4(spec.vel[0], spec.vel[1], spec.vel[2], 0.f);
    A0[s] = make_float4(0.f, 0.f, 0.f, 0.f);
    C2[s] = 0.f;
    R[2 * (size_t)s].w = 0.f;
    R[2 * (size_t)s + 1].w = 0.f;
}

// Sorted hash for the debug tap: key of the particle now at each slot, with
// the NULL bucket reported as NULL_HASH (m_Hash after the sort).
__global__ void k_sorted_keys(const DevParams* __restrict__ params, const float4* __restrict__ G, uint32_t n,
                              uint32_t base, uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // the cell of the position gathered into slot i by the last sort: the key
    // it was sorted by (the key array itself may already hold the next
    // substep's keys, written by the force pass)
    const float4 p = G[2 * (size_t)(base + i)];
    const uint32_t k = cell_of(*params, p.x, p.y, p.z);
    out[i] = (k == params->ncells) ? SPH_NULL_HASH : k;
}

// ---------------------------------------------------------------------------
// Tile table of a layout: one block per scene writes that scene's tiles
// (scene, first slot, count) from its slot range, starting at tile_first[s].
// The host computes only the per-scene offsets, so a membership change of
// the served form costs O(scenes) on the host instead of O(tiles).
// ---------------------------------------------------------------------------
__global__ void k_build_tiles(const DevScene* __restrict__ scenes, const uint32_t* __restrict__ tile_first,
                              uint32_t tile, uint4* __restrict__ tiles) {
    const uint32_t s = blockIdx.x;
    const DevScene sc = scenes[s];
    const uint32_t first = tile_first[s];
    const uint32_t cnt = (sc.n + tile - 1u) / tile;
    for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
        const uint32_t f = i * tile;
        tiles[first + i] = make_uint4(s, sc.part_base + f, min(tile, sc.n - f), 0u);
    }
}

// ---------------------------------------------------------------------------
// Launch wrappers.
// ---------------------------------------------------------------------------
cudaError_t launch_build_tiles(const DevScene* scenes, const uint32_t* tile_first, uint32_t nscenes, uint32_t tile,
                               uint4* tiles, cudaStream_t st) {
    if (nscenes == 0) return cudaSuccess;
    k_build_tiles<<<nscenes, 128, 0, st>>>(scenes, tile_first, tile, tiles);
    return cudaGetLastError();
}
static uint32_t scan_tiles(uint32_t cells) { return (cells + SCAN_TILE - 1) / SCAN_TILE; }
cudaError_t launch_hash(const StepArgs& a, cudaStream_t st) {
    k_hash<<<a.ntiles, a.block, 0, st>>>(a.params, a.scenes, a.tiles, a.P0, a.count, a.key, a.slot, a.pend, a.okey,
                                         a.status);
    // an unsorted state's warps are spread over the tiles: their sums from the counts
    k_scan_reduce<<<scan_tiles(a.total_cells), SCAN_THREADS, 0, st>>>(a.count, a.total_cells, a.sums);
    return cudaGetLastError();
}
static inline uint32_t* ctr(const StepArgs& a, int k) { return a.tile_ctr ? a.tile_ctr + k : nullptr; }

// Kernels with row starts or neighbour lists in shared memory: left to itself
// the driver may give them the largest shared-memory carveout and shrink L1,
// which holds the neighbour gathers.  Ask for the smallest carveout that still
// fits the blocks that registers allow on an SM (SPH_*_CARVEOUT_PCT).
cudaError_t init_kernel_attributes() {
    struct { const void* f; int pct; } fns[] = {
        {(const void*)k_force_integrate<true, 3>, SPH_ROWS_CARVEOUT_PCT},
        {(const void*)k_force_integrate<true, 4>, SPH_ROWS_CARVEOUT_PCT},
        {(const void*)k_force_integrate<false, 3>, SPH_ROWS_CARVEOUT_PCT},
        {(const void*)k_force_integrate<false, 4>, SPH_ROWS_CARVEOUT_PCT},
        {(const void*)k_normals<1, false>, SPH_ROWS_CARVEOUT_PCT},
        {(const void*)k_normals<1, true>, SPH_ROWS_CARVEOUT_PCT},
        {(const void*)k_density<false, false>, SPH_LIST_CARVEOUT_PCT},
        {(const void*)k_density<false, true>, SPH_LIST_CARVEOUT_PCT},
        {(const void*)k_density<true, false>, SPH_LIST_CARVEOUT_PCT}};
    for (const auto& x : fns) {
        const cudaError_t e = cudaFuncSetAttribute(x.f, cudaFuncAttributePreferredSharedMemoryCarveout, x.pct);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Whether this scan covers every scene's cells and consumes the counts: the
// tile sums are then this scan's, and cleared after it.
static bool whole_scan(const StepArgs& a) { return a.scan_cells == 0u && a.scan_zeroes_counts != 0u; }

// a.scan_sums holds at least nt + 2 64-bit words: the tile counter, then one
// look-back descriptor per tile; they start at zero.  With scan_withhold the
// counter starts at 1 instead: the blocks take tiles 1..nt, no block takes
// tile 0, and every wait that reaches tile 0 runs out after scan_spin_limit
// polls (the test of the timeout path).  Tile nt covers no cell (its first
// cell is past n), so it reads and writes no count or start, and its
// descriptor is word nt + 1.
cudaError_t launch_scan(const StepArgs& a, cudaStream_t st) {
    const uint32_t n = a.scan_cells ? a.scan_cells : a.total_cells;
    if (n == 0) return cudaErrorInvalidValue;
    if (whole_scan(a) && scan_tiles(n) <= SPH_SCAN_SUM_TILES && !a.scan_spin_limit && !a.scan_withhold) {
        // (the test controls are the look-back's)
        k_scan_tiles<<<scan_tiles(n), SCAN_THREADS, 0, st>>>(a.count, n, a.sums, a.start);
        return cudaGetLastError();
    }
    uint32_t* counts = a.count + a.scan_first;
    uint32_t* starts = a.start + a.scan_first;
    const uint32_t vec_ok = ((reinterpret_cast<uintptr_t>(counts) | reinterpret_cast<uintptr_t>(starts)) & 15u) == 0u;
    const uint32_t nt = (n + SCAN_TILE - 1) / SCAN_TILE;
    unsigned long long* desc = reinterpret_cast<unsigned long long*>(a.scan_sums);
    cudaError_t e = cudaMemsetAsync(desc, 0, (size_t)(nt + 2) * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    if (a.scan_withhold) {
        e = cudaMemsetAsync(desc, 1, 1, st);   // the counter's low byte: the next tile handed out is 1
        if (e != cudaSuccess) return e;
    }
    const uint32_t limit = a.scan_spin_limit ? a.scan_spin_limit : SCAN_SPIN_LIMIT;
    k_scan_single<<<nt, SCAN_THREADS, 0, st>>>(counts, n, desc, starts, a.status, a.scan_zeroes_counts, limit,
                                                 vec_ok);
    return cudaGetLastError();
}
cudaError_t launch_scan_raw(const uint32_t* counts, uint32_t n, uint32_t* tile_sums, uint32_t* starts,
                            cudaStream_t st) {
    const uint32_t nt = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (n == 0 || nt > kScanRawMaxTiles) return cudaErrorInvalidValue;
    k_scan_reduce<<<nt, SCAN_THREADS, 0, st>>>(counts, n, tile_sums);
    k_scan_top<<<1, 1024, 0, st>>>(tile_sums, nt);
    k_scan_down<<<nt, SCAN_THREADS, 0, st>>>(counts, n, tile_sums, starts);
    return cudaGetLastError();
}
// The per-axis positions lie in three neighbour-word rows that the density pass
// does not write: past the list, or where a skin pass needs the rows after it, in
// the list's last three (which is then shorter).
static float* axes(const StepArgs& a) {
    return reinterpret_cast<float*>(a.mask + (a.skin_masks ? SPH_AXIS_ROWS_SKIN : SPH_AXIS_ROWS) * a.mask_stride);
}
cudaError_t launch_sort(const StepArgs& a, cudaStream_t st) {
    k_scatter<<<(a.ntiles + kScatterTiles - 1u) / kScatterTiles, a.block, 0, st>>>(
        a.scenes, a.tiles, a.ntiles, a.start, a.key, a.slot, a.tmp, a.sums,
        whole_scan(a) ? scan_tiles(a.total_cells) : 0u, a.status);
    auto rank = a.form.half ? k_rank_gather<true> : k_rank_gather<false>;
    rank<<<a.ntiles, a.block, 0, st>>>(a.params, a.scenes, a.tiles, a.start, a.key, a.tmp, a.P0, a.V0, a.A0, a.V2,
                                                a.okey, a.pend, a.G, axes(a), a.A1, a.perm, a.status);
    return cudaGetLastError();
}
static dim3 wide_grid(const StepArgs& a, int lanes) {
    return dim3((a.block * (uint32_t)lanes + kWideBlock - 1u) / kWideBlock, a.ntiles);
}
static size_t wide_smem(int lanes) {
    return kWideBlock / lanes * (lanes == 8 ? sizeof(WideShared<8>) : sizeof(WideShared<4>));
}
// Position and density once more, 16 bytes a slot.
static float4* dense(const StepArgs& a) {
    if (!a.form.dense) return nullptr;
    return reinterpret_cast<float4*>(a.mask + SPH_DENSE_ROWS * a.mask_stride);
}
cudaError_t launch_density(const StepArgs& a, cudaStream_t st) {
    const int l = (int)a.form.lanes;
    if (a.form.density_wide) {
        auto kern = l == 8 ? k_density_wide<8> : k_density_wide<4>;
        kern<<<wide_grid(a, l), kWideBlock, wide_smem(l), st>>>(a.params, a.scenes, a.tiles, a.start, a.G, axes(a),
                                                               a.C2, a.mask, a.mask_stride, a.pend, a.R, a.dbg_nbr,
                                                               a.status);
        return cudaGetLastError();
    }
    const size_t smem = (size_t)SPH_NBR_SMEM_WORDS * a.block * sizeof(uint32_t);
    auto kern = a.skin_masks ? k_density<true, false> : a.form.one_wave ? k_density<false, true> : k_density<false, false>;
    kern<<<a.grid_nbr, a.block, smem, st>>>(a.params, a.scenes, a.tiles, a.start, a.G, axes(a), a.C2, a.mask,
                                            a.mask_stride, a.pend, a.R, dense(a), a.dbg_nbr, a.ntiles, ctr(a, 0),
                                            a.status);
    return cudaGetLastError();
}
cudaError_t launch_unsort_vel(const StepArgs& a, uint32_t first_tile, uint32_t ntiles, uint32_t base, uint32_t n,
                              float* out, float4* V0, bool clear_pending, cudaStream_t st, uint32_t* gate,
                              uint32_t* status_out) {
    if (ntiles == 0) return cudaSuccess;
    k_unsort_vel<<<ntiles, a.block, 0, st>>>(a.tiles + first_tile, a.perm, a.R, base, out, V0,
                                             clear_pending ? a.pend : nullptr, a.status, gate, n, status_out);
    return cudaGetLastError();
}
cudaError_t launch_undo_ahead(const StepArgs& a, uint32_t first_tile, uint32_t ntiles, cudaStream_t st) {
    if (ntiles == 0) return cudaSuccess;
    k_undo_ahead<<<ntiles, a.block, 0, st>>>(a.tiles + first_tile, a.perm, a.G, a.A1, a.P0, a.V2, a.A0,
                                             a.okey);
    return cudaGetLastError();
}
static size_t rows_smem(const StepArgs& a) { return (size_t)SPH_NBR_ROWS * a.block * sizeof(uint32_t); }
cudaError_t launch_normals(const StepArgs& a, cudaStream_t st) {
    const int l = (int)a.form.lanes;
    auto kern = l == 8   ? k_normals<8>
                : l == 4 ? k_normals<4>
                         : a.form.one_wave ? k_normals<1, true> : k_normals<1, false>;
    const float4* D = dense(a);
    kern<<<l > 1 ? wide_grid(a, l) : dim3(a.grid_nbr), l > 1 ? kWideBlock : a.block,
           l > 1 ? wide_smem(l) : rows_smem(a), st>>>(a.params, a.scenes, a.tiles, a.start, D ? D : a.R, D ? 1u : 2u, a.C2, axes(a),
                                                         a.form.half, a.mask,
                                                         a.mask_stride, a.N, a.ntiles, ctr(a, 1), a.status);
    return cudaGetLastError();
}
cudaError_t launch_force(const StepArgs& a, cudaStream_t st) {
    const bool occ = (a.variant & SPH_VARIANT_FORCE_OCC) != 0u && !a.form.one_wave;
    const int l = (int)a.form.lanes;
    auto kern = l == 8   ? (a.any_tension ? k_force_integrate<true, 5, 8> : k_force_integrate<false, 6, 8>)
                : l == 4 ? (a.any_tension ? k_force_integrate<true, 5, 4> : k_force_integrate<false, 7, 4>)
                : a.any_tension ? (occ ? k_force_integrate<true, 4> : k_force_integrate<true, 3>)
                                : (occ ? k_force_integrate<false, 4> : k_force_integrate<false, 3>);
    kern<<<l > 1 ? wide_grid(a, l) : dim3(a.grid_nbr), l > 1 ? kWideBlock : a.block,
           l > 1 ? wide_smem(l) : rows_smem(a), st>>>(
                                                    a.params, a.scenes, a.tiles, a.start, a.R, a.C2, a.A1, a.N,
                                                    axes(a), a.form.half, a.mask, a.mask_stride, a.P0, a.V2, a.A0,
                                                    a.skin_masks ? a.maxdisp : nullptr, a.okey, a.pend, a.count, a.sums,
                                                    a.key, a.slot, a.status, a.dbg_forces, a.ntiles, ctr(a, 2));
    return cudaGetLastError();
}
cudaError_t launch_xsph(const StepArgs& a, cudaStream_t st) {
    auto kern = (a.variant & SPH_VARIANT_XSPH_ROWS) ? k_xsph<1> : k_xsph<0>;
    kern<<<a.grid_nbr, a.block, 0, st>>>(a.params, a.scenes, a.tiles, a.start, a.G, a.P0, a.V2, a.mask,
                                         a.mask_stride, a.maxdisp, a.V0, a.pend, a.ntiles, ctr(a, 3), a.status);
    return cudaGetLastError();
}
cudaError_t launch_unpack(const float* pos, const float* vel, uint32_t n, uint32_t base, float4* P0, float4* V0,
                          float4* A0, float* C2, float4* R, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_unpack_state<<<(n + 255) / 256, 256, 0, st>>>(pos, vel, n, base, P0, V0, A0, C2, R);
    return cudaGetLastError();
}
cudaError_t launch_set_positions(const float* pos, uint32_t n, uint32_t base, float4* P0, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_set_positions<<<(n + 255) / 256, 256, 0, st>>>(pos, n, base, P0);
    return cudaGetLastError();
}
cudaError_t launch_pack(const float4* P0, const float4* V0, uint32_t n, uint32_t base, float inv_rest_density,
                        float* pos, float* colour, float* vel, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_pack_state<<<(n + 255) / 256, 256, 0, st>>>(P0, V0, n, base, inv_rest_density, pos, colour, vel);
    return cudaGetLastError();
}
cudaError_t launch_lattice(const LatticeSpec& spec, uint32_t base, float4* P0, float4* V0, float4* A0, float* C2,
                           float4* R, cudaStream_t st) {
    const uint32_t n = spec.nx * spec.ny * spec.nz;
    if (n == 0) return cudaSuccess;
    k_lattice<<<(n + 255) / 256, 256, 0, st>>>(spec, base, P0, V0, A0, C2, R);
    return cudaGetLastError();
}
cudaError_t launch_sorted_keys(const DevParams* params, const float4* G, uint32_t n, uint32_t base,
                               uint32_t* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_sorted_keys<<<(n + 255) / 256, 256, 0, st>>>(params, G, n, base, out);
    return cudaGetLastError();
}

}  // namespace sph
