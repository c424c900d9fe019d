// host_runtime.cpp — the CUDA runtime calls that mms_api.cu makes, and stand-ins
// of the kernels it launches, in host memory: the library's host side then runs
// without a device.  It counts device memory, holds it to a limit, and notes a
// launch or a copy that is handed memory already given back (tests/
// test_host_memory.py).  Steps only count; no field changes.
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>
#include <functional>
#include <map>
#include <mutex>
#include <vector>

#include "mms_internal.h"
#include "sites.h"

using namespace mms;

namespace {

std::mutex mu;
std::map<const char *, size_t> live;  // device allocations
size_t held = 0, limit = (size_t)1 << 40, total = (size_t)1 << 40;
std::atomic<long long> stale{0};  // uses of memory that is not allocated
std::atomic<long long> launched{0};  // graph launches
thread_local cudaError_t last = cudaSuccess;

struct Graph {
    std::vector<std::function<void()>> work;
};
thread_local Graph *capturing = nullptr;

bool valid(const void *p)
{
    if (!p) return true;
    std::lock_guard<std::mutex> lock(mu);
    auto it = live.upper_bound((const char *)p);
    if (it == live.begin()) return false;
    --it;
    return (const char *)p < it->first + it->second;
}

void use(std::initializer_list<const void *> ptrs)
{
    for (const void *p : ptrs)
        if (!valid(p)) stale++;
}

// now, or as part of the graph being captured
template <typename F>
int enqueue(F &&f)
{
    if (capturing) capturing->work.emplace_back(f);
    else f();
    return 1;
}

void step(const DevPtrs &d)
{
    use({d.ce, d.cl[0], d.cl[1], d.fs[0], d.fs[1], d.gr, d.ctl, d.tm.chg, d.tm.act, d.rec_flags});
    if (valid(d.ctl) && !d.ctl->stall) d.ctl->timestep++;
}

}  // namespace

// ------------------------------------------------------------ test controls
extern "C" {
size_t host_runtime_held() { return held; }
void host_runtime_limit(size_t bytes) { limit = bytes; }
void host_runtime_total(size_t bytes) { total = bytes; }
long long host_runtime_stale() { return stale; }
long long host_runtime_graph_launches() { return launched; }
}

// ------------------------------------------------------------------- runtime
extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    std::lock_guard<std::mutex> lock(mu);
    *p = nullptr;
    if (held + n > limit) return last = cudaErrorMemoryAllocation;
    char *q = (char *)aligned_alloc(256, (n + 255) / 256 * 256);
    live[q] = n;
    held += n;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> lock(mu);
    auto it = live.find((char *)p);
    if (it == live.end()) return last = cudaErrorInvalidValue;
    held -= it->second;
    live.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = limit - held; *t = total; return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->totalGlobalMem = total;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    if ((k == cudaMemcpyHostToDevice || k == cudaMemcpyDeviceToDevice) && !valid(d)) { stale++; return cudaSuccess; }
    if ((k == cudaMemcpyDeviceToHost || k == cudaMemcpyDeviceToDevice) && !valid(s)) { stale++; return cudaSuccess; }
    if (k != cudaMemcpyDeviceToDevice) std::memcpy(d, s, n);  // (no field's values matter here)
    return cudaSuccess;
}
cudaError_t cudaMemcpyPeerAsync(void *d, int, const void *s, int, size_t n, cudaStream_t)
{
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t)
{
    for (size_t r = 0; r < h; r++) std::memcpy((char *)d + r * dp, (const char *)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
    if (!valid(d)) { stale++; return cudaSuccess; }
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    capturing = new Graph();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g)
{
    *g = (cudaGraph_t)capturing;
    capturing = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long)
{
    *x = (cudaGraphExec_t) new Graph(*(Graph *)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph *)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete (Graph *)x; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t)
{
    launched++;
    for (auto &f : ((Graph *)x)->work) f();
    return cudaSuccess;
}
}

// ------------------------------------------------------- kernels' stand-ins
namespace mms {
int launch_step(const KernelArgs &a, const TmaHolder &, int, void *, int, Profiler *, bool)
{
    const DevPtrs d = a.d;
    return enqueue([d] { step(d); });
}
void tile_geometry(KernelArgs &a, const TmaHolder &t)
{
    TileMap &m = a.d.tm;
    m.wsh = t.cpt == 2 ? 6 : 5;
    m.zc = t.zc > 0 ? t.zc : 4;
    m.nx = (a.g.gx + (1 << m.wsh) - 1) >> m.wsh;
    m.ny = (a.g.gy + 7) / 8;
    m.nz = (a.g.gz + m.zc - 1) / m.zc;
    m.n = m.nx * m.ny * m.nz;
}
int stencil_default_cpt(const Geo &) { return 1; }
void tile_map_max(const Geo &g, long long *tiles, long long *edges)
{
    *tiles = (long long)((g.gx + 31) / 32) * ((g.gy + 7) / 8) * g.gz;
    *edges = (g.gx + 31) / 32 + (g.gy + 7) / 8 + g.gz;
}
int make_tma(const KernelArgs &, int, TmaHolder &out) { return out.ok = 1; }
int launch_stencil(const KernelArgs &a, const TmaHolder &, int, void *)
{
    use({a.d.ce, a.d.gr});
    return 1;
}
int launch_curv(const KernelArgs &a, int, void *)
{
    const void *c = a.d.curv;
    return enqueue([c] { use({c}); });
}
int launch_slab_phase(const KernelArgs &, const TmaHolder &, int, void *, int, int) { return 1; }
size_t batch_item_bytes() { return sizeof(DevPtrs); }
long long fill_batch_item(void *dst, const KernelArgs &a, const TmaHolder &, long long, unsigned char *)
{
    std::memcpy(dst, (const void *)&a.d, sizeof a.d);
    return a.d.tm.n;
}
void batch_prepare(int, int) {}
int launch_stencil_batch(const void *items, int n, long long, int, int, const unsigned char *act, void *)
{
    return enqueue([=] {
        use({items, act});
        if (valid(items))
            for (int i = 0; i < n; i++) step(((const DevPtrs *)items)[i]);
    });
}
int batch_blocks(const KernelArgs &, int) { return 1; }
int launch_small_batch(int, const void *items, const int *begin, int, int, int, void *)
{
    return enqueue([=] { use({items, begin}); });
}
int am_default_rows(const Geo &) { return 128; }
int launch_am_halo_fill(const KernelArgs &, const AmParams &, double *o, void *) { use({o}); return 1; }
int am_tc_prepare() { return 0; }
long long am_ximg_size(int, int, int) { return 1; }
int launch_temp_am(const KernelArgs &a, const AmParams &, int, void *, Profiler *, int)
{
    const void *t = a.d.am_tab;
    return enqueue([t] { use({t}); });
}
int launch_reduce(const KernelArgs &, int, int, double *o, void *, double *) { *o = 0; return 1; }
long long stencil_parts(const KernelArgs &, const TmaHolder &) { return 0; }
long long stencil_parts_max(const Geo &g) { return (long long)g.gx * g.gy * g.gz / 256 + 64; }
int launch_fold_fs(const KernelArgs &, long long, void *, double *) { return 1; }
int launch_fold_fs_out(const KernelArgs &, long long, void *, double *, void *) { return 1; }
int launch_fill_temperature(const KernelArgs &, double *o, void *) { use({o}); return 1; }
int launch_compute_d(const KernelArgs &, int, double *o, void *) { use({o}); return 1; }
int launch_repack(void *d, long long, const void *s, long long, int, long long, void *) { use({d, s}); return 1; }
int launch_mask_captured(const KernelArgs &, void *d, int, void *) { use({d}); return 1; }
int launch_convert(const KernelArgs &, int, int, int, double *d, void *) { use({d}); return 1; }
int launch_convert_ref(const KernelArgs &, int, int, int, double *d, void *) { use({d}); return 1; }
int adj_nblocks(const Geo &g) { return (int)(((long long)g.gx * g.gy * g.gz + 255) / 256); }
int launch_replay(const Geo &, const Phys &, int, const void *const x0[3], void *const x1[3], const unsigned char *f,
                  const double *c, unsigned long long, void *)
{
    use({x0[0], x0[1], x0[2], x1[0], x1[1], x1[2], f, c});
    return 1;
}
int launch_adj_step(const Geo &, const Phys &, int, const void *const x0[3], const void *ce1, const unsigned char *f,
                    const double *c, const void *const l1[3], void *const l0[3], double *part, unsigned long long, void *)
{
    use({x0[0], x0[1], x0[2], ce1, f, c, l1[0], l1[1], l1[2], l0[0], l0[1], l0[2], part});
    return 1;
}
int launch_adj_fold(const Geo &, const double *part, double *grad, void *)
{
    use({part, grad});
    if (valid(grad)) std::memset(grad, 0, ADJ_SLOTS * sizeof(double));
    return 1;
}
int launch_adj_terminal(const Geo &, int, double, const void *ce, const double *target, void *lce, void *lcl, void *lfs,
                        double *part, double *loss, void *)
{
    use({ce, target, lce, lcl, lfs, part, loss});
    if (valid(loss)) *loss = 0;
    return 1;
}
int site_draw_device(const SiteDrawArgs &, const std::vector<double> &, const std::vector<double> &,
                     const std::vector<long long> &, const std::vector<float> &, std::vector<long long> &,
                     std::vector<float> &, std::vector<int> &, std::string &)
{
    return 0;
}
}  // namespace mms
