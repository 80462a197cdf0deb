#include "fake_cuda.h"
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>

namespace fake {
State st;

using Op = std::function<void()>;
static std::vector<Op>* capture = nullptr;
static void run(Op op) {
    if (capture) capture->push_back(std::move(op));
    else op();
}
static std::map<const char*, size_t> blocks;   // live allocations
static cudaError_t take(void** p, size_t n) {
    *p = std::calloc(n ? n : 1, 1);
    blocks[(const char*)*p] = n;
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
static cudaError_t give(void* p) {
    blocks.erase((const char*)p);
    std::free(p);
    return cudaSuccess;
}
// `n` bytes from p on lie inside one live allocation
static bool inside(const void* p, size_t n) {
    auto it = blocks.upper_bound((const char*)p);
    if (it == blocks.begin()) return false;
    --it;
    return (const char*)p + n <= it->first + it->second;
}
static void fill(float* p, size_t n, float v) {
    if (!inside(p, n * sizeof(float))) { ++st.null_writes; return; }
    for (size_t i = 0; i < n; ++i) p[i] = v;
}
static cudaError_t last() {
    const cudaError_t e = st.last_error;
    st.last_error = cudaSuccess;
    return e;
}
static Key key(const sph::StepArgs& a) {
    Key k;
    k.form = a.form;
    k.skin = a.skin_masks;
    k.tension = a.any_tension;
    k.block = a.block;
    k.ntiles = a.ntiles;
    k.tiles = a.tiles;
    k.mask = a.mask;
    k.stride = a.mask_stride;
    return k;
}
// Every array that the substep's passes index, for the slots and cells they reach.
static void check(const sph::StepArgs& a) {
    bool ok = inside(a.tiles, a.ntiles * sizeof(uint4)) && inside(a.status, 4);
    size_t slots = 0, scenes = 0;
    for (uint32_t i = 0; ok && i < a.ntiles; ++i) {
        slots = std::max<size_t>(slots, a.tiles[i].y + a.tiles[i].z);
        scenes = std::max<size_t>(scenes, a.tiles[i].x + 1u);
    }
    for (const void* p : {(const void*)a.P0, (const void*)a.V0, (const void*)a.A0, (const void*)a.A1,
                          (const void*)a.V2, (const void*)a.N})
        ok = ok && inside(p, slots * sizeof(float4));
    for (const void* p : {(const void*)a.G, (const void*)a.R}) ok = ok && inside(p, 2 * slots * sizeof(float4));
    for (const void* p : {(const void*)a.okey, (const void*)a.key, (const void*)a.slot, (const void*)a.perm,
                          (const void*)a.C2})
        ok = ok && inside(p, slots * sizeof(uint32_t));
    ok = ok && a.mask_stride >= slots && inside(a.mask, SPH_MASK_ROWS * a.mask_stride * sizeof(uint32_t)) &&
         inside(a.count, a.total_cells * sizeof(uint32_t)) && inside(a.start, (a.total_cells + 1) * sizeof(uint32_t)) &&
         inside(a.sums, (a.total_cells + 4095) / 4096 * sizeof(uint32_t)) &&
         inside(a.scan_sums, ((a.total_cells + 4095) / 4096 + 2) * sizeof(uint64_t)) &&
         inside(a.params, scenes * sizeof(DevParams)) && inside(a.scenes, scenes * sizeof(DevScene)) &&
         inside(a.pend, scenes * sizeof(uint32_t)) &&
         (!a.dbg_nbr || inside(a.dbg_nbr, slots * sizeof(uint32_t))) &&
         (!a.dbg_forces || inside(a.dbg_forces, 4 * slots * sizeof(float4)));
    if (!ok) ++st.bad_arrays;
}
static bool failed(const uint32_t* s) { return (*s & (SPH_STATUS_SCAN_TIMEOUT | SPH_STATUS_CELL_OVERFLOW)) != 0u; }
}  // namespace fake

using fake::give;
using fake::run;
using fake::take;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return fake::last(); }
cudaError_t cudaMalloc(void** p, size_t n) {
    const long k = (long)fake::st.mallocs++;
    if (fake::st.fail_from >= 0 && k >= fake::st.fail_from && k < (long)fake::st.fail_from + fake::st.fail_count)
        return fake::st.last_error = cudaErrorMemoryAllocation;
    return take(p, n);
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    if (n > fake::st.pinned_limit) {
        *p = nullptr;
        return fake::st.last_error = cudaErrorMemoryAllocation;
    }
    fake::st.pinned += n;
    return take(p, n);
}
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeHost(void* p) {
    fake::st.pinned -= fake::blocks[(const char*)p];
    return give(p);
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    run([=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    run([=] { std::memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return take((void**)s, 1); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return give(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return take((void**)e, 1); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return take((void**)e, 1); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return give(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
// a graph is its list of recorded calls
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    fake::capture = new std::vector<fake::Op>;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = reinterpret_cast<cudaGraph_t>(fake::capture);
    fake::capture = nullptr;
    return cudaSuccess;
}
static std::vector<fake::Op>* ops(void* g) { return reinterpret_cast<std::vector<fake::Op>*>(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(new std::vector<fake::Op>(*ops(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t e, cudaGraph_t g, cudaGraphExecUpdateResultInfo*) {
    *ops(e) = *ops(g);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    for (auto& op : *ops(e)) op();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete ops(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete ops(e); return cudaSuccess; }
}

namespace sph {
using fake::st;

cudaError_t init_kernel_attributes() { return cudaSuccess; }
cudaError_t launch_build_tiles(const DevScene* scenes, const uint32_t* tile_first, uint32_t nscenes, uint32_t tile,
                               uint4* tiles, cudaStream_t) {
    for (uint32_t s = 0; s < nscenes; ++s)
        for (uint32_t i = 0, f = 0; f < scenes[s].n; ++i, f += tile)
            tiles[tile_first[s] + i] = make_uint4(s, scenes[s].part_base + f, std::min(tile, scenes[s].n - f), 0u);
    return fake::last();
}
cudaError_t launch_hash(const StepArgs& a, cudaStream_t) {
    run([a] { fake::check(a); });
    return fake::last();
}
cudaError_t launch_scan(const StepArgs&, cudaStream_t) { return fake::last(); }
cudaError_t launch_sort(const StepArgs& a, cudaStream_t) {
    run([a] {
        fake::check(a);
        if (fake::failed(a.status)) return;
        st.sorted = fake::key(a);
        st.sorts.push_back(a.ntiles);
        for (uint32_t i = 0; i < a.ntiles; ++i)
            if (st.crowded.count(a.scenes[a.tiles[i].x].part_base)) *a.status |= SPH_STATUS_CELL_OVERFLOW;
    });
    return fake::last();
}
cudaError_t launch_density(const StepArgs& a, cudaStream_t) {
    run([a] {
        fake::check(a);
        if (fake::failed(a.status)) return;
        if (!(st.sorted == fake::key(a))) ++st.mixed;
        st.written = fake::key(a);
    });
    return fake::last();
}
cudaError_t launch_normals(const StepArgs& a, cudaStream_t) {
    run([a] { if (!fake::failed(a.status) && !(st.written == fake::key(a))) ++st.mixed; });
    return fake::last();
}
cudaError_t launch_force(const StepArgs& a, cudaStream_t) {
    run([a] {
        fake::check(a);
        if (fake::failed(a.status)) return;
        ++st.substeps;
        st.lanes.insert(a.form.lanes);
        if (!(st.written == fake::key(a))) ++st.mixed;
        if (st.after_force) st.after_force();
    });
    return fake::last();
}
cudaError_t launch_xsph(const StepArgs&, cudaStream_t) { return fake::last(); }
cudaError_t launch_unsort_vel(const StepArgs& a, uint32_t, uint32_t ntiles, uint32_t, uint32_t n, float* out, float4*,
                              bool, cudaStream_t, uint32_t* gate, uint32_t* status_out) {
    if (ntiles == 0) return cudaSuccess;
    run([=] {
        if (status_out) *status_out = *a.status;
        if (gate) *gate = *a.status ? SPH_STATUS_SCAN_TIMEOUT : 0u;
        if (!fake::failed(a.status) && out) fake::fill(out, 3 * (size_t)n, fake::kVelocity);
    });
    return fake::last();
}
cudaError_t launch_undo_ahead(const StepArgs&, uint32_t, uint32_t, cudaStream_t) { return fake::last(); }
cudaError_t launch_unpack(const float*, const float*, uint32_t, uint32_t, float4*, float4*, float4*, float*, float4*,
                          cudaStream_t) { return fake::last(); }
cudaError_t launch_set_positions(const float*, uint32_t, uint32_t, float4*, cudaStream_t) { return fake::last(); }
cudaError_t launch_pack(const float4*, const float4*, uint32_t n, uint32_t, float, float* pos, float* colour,
                        float* vel, cudaStream_t) {
    run([=] {
        if (pos) fake::fill(pos, 3 * (size_t)n, fake::kPosition);
        if (colour) fake::fill(colour, 3 * (size_t)n, fake::kPosition);
        if (vel) fake::fill(vel, 3 * (size_t)n, fake::kVelocity);
    });
    return fake::last();
}
cudaError_t launch_lattice(const LatticeSpec&, uint32_t, float4*, float4*, float4*, float*, float4*, cudaStream_t) {
    return fake::last();
}
cudaError_t launch_sorted_keys(const DevParams*, const float4*, uint32_t, uint32_t, uint32_t*, cudaStream_t) {
    return fake::last();
}
}  // namespace sph
