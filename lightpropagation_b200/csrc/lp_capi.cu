// lp_capi.cu -- C ABI of liblpcuda.so (declared in include/lpcuda.h).
//
// Host side of the drop-in for the reference launcher
// (src/Simulation/CalculatePropagation.cpp): setters copy their inputs, lp_run
// uploads what changed, launches the persistent transport kernel once for the
// whole photon budget (the reference loops over 6400-photon launches,
// CalculatePropagation.cpp:1446-1451) and accumulates fixed-point tallies on the
// device.  No exceptions cross the ABI; errors are int codes plus a message.
#include <cuda_runtime.h>
#include <cub/device/device_scan.cuh>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "../../include/lpcuda.h"
#include "lp_bvh.hpp"
#include "lp_kernel.cuh"

namespace lp {
int smem_bytes(int nodes_smem, int tris_smem);
cudaError_t launch_transport_fast(const KParams &P, int grid, int smem, cudaStream_t s);
cudaError_t transport_occupancy_fast(int smem, int *blocks_per_sm);
cudaError_t launch_transport_exact(const KParams &P, int grid, int smem, cudaStream_t s);
cudaError_t transport_occupancy_exact(int smem, int *blocks_per_sm);
cudaError_t transport_occupancy_fast_grad(int smem, int *blocks_per_sm);
cudaError_t transport_occupancy_exact_grad(int smem, int *blocks_per_sm);
cudaError_t launch_query(const KParams &P, int smem, int64_t n, const float *orig, const float *dir,
                         const int32_t *ref, const float *tmax, int32_t *id_out, float *t_out,
                         cudaStream_t s);
cudaError_t launch_philox(const uint32_t *ctr, const uint32_t *key, int64_t n, uint32_t *out,
                          cudaStream_t s);
cudaError_t launch_exact_ops(int op, int64_t n, const float *a, const float *b, float *out, cudaStream_t s);
cudaError_t launch_cell_lists(const KParams &P, int n_tri, float h, float eps, uint32_t *count, const uint32_t *start,
                              int32_t *refs, cudaStream_t s);
cudaError_t launch_cell_words(const KParams &P, float m, const uint32_t *count, const uint32_t *start, bool lists,
                              uint8_t *gap, float *d2, uint32_t *word, cudaStream_t s);
cudaError_t launch_interleave(const float4 *soa, int64_t n, float4 *out, cudaStream_t s);
cudaError_t launch_fold(unsigned long long *dst, unsigned long long *part, int copies, int64_t n, int64_t images,
                        cudaStream_t s);
double fma_peak_tflops(int num_sms);
double red_peak_per_s(int num_sms);
int block_size();
}  // namespace lp

using lp::KParams;
using lp::Medium;

namespace {

thread_local std::string g_thread_error;

// An NVTX range over a phase of the host path (mesh build, upload, cell grid, launch,
// wait, readback), seen by profilers on the context's timeline; the counterpart of the
// reference's per-launch OpenCL profiling events (CalculatePropagation.cpp:1229, 1544-1548).
struct Phase {
    explicit Phase(const char *name) { nvtxRangePushA(name); }
    ~Phase() { nvtxRangePop(); }
    Phase(const Phase &) = delete;
    Phase &operator=(const Phase &) = delete;
};

// Allocation-failure injection (lp_debug_fail_allocation): the allocation that brings the
// countdown from 0 to -1 reports cudaErrorMemoryAllocation without allocating.
std::atomic<int64_t> g_alloc_countdown{-1};
// Launch-failure injection (lp_debug_fail_launch), the same for the transport, batch and fold
// launches: cudaErrorLaunchOutOfResources without launching.
std::atomic<int64_t> g_launch_countdown{-1};

bool counted_down(std::atomic<int64_t> &countdown)
{
    int64_t v = countdown.load();
    while (v >= 0) {
        if (countdown.compare_exchange_weak(v, v - 1)) return v == 0;
    }
    return false;
}
bool injected_alloc_failure() { return counted_down(g_alloc_countdown); }

template <class Launch>
cudaError_t launch_unless_injected(Launch launch)
{
    return counted_down(g_launch_countdown) ? cudaErrorLaunchOutOfResources : launch();
}

template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaError_t ensure(size_t count)
    {
        if (count <= n && p) return cudaSuccess;
        release();
        if (injected_alloc_failure()) return cudaErrorMemoryAllocation;
        cudaError_t e = cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
        if (e != cudaSuccess) {
            p = nullptr;
            return e;
        }
        n = count;
        return cudaSuccess;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
};

// Page-locked host memory, so that the tally copies run at the link's speed rather than
// through the driver's staging buffer.  size() is the last resize; the allocation grows.
template <class T>
struct HostBuf {
    T *p = nullptr;
    size_t n = 0, cap = 0;
    cudaError_t resize(size_t count)
    {
        if (count > cap) {
            if (p) cudaFreeHost(p);
            p = nullptr;
            cap = n = 0;
            if (injected_alloc_failure()) return cudaErrorMemoryAllocation;
            cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&p), count * sizeof(T), cudaHostAllocPortable);
            if (e != cudaSuccess) {
                p = nullptr;
                return e;
            }
            cap = count;
        }
        n = count;
        return cudaSuccess;
    }
    T *data() { return p; }
    size_t size() const { return n; }
    bool empty() const { return n == 0; }
    HostBuf() = default;
    HostBuf(const HostBuf &) = delete;
    HostBuf &operator=(const HostBuf &) = delete;
    ~HostBuf()
    {
        if (p) cudaFreeHost(p);
    }
};

// Ring signals and their derivatives formed from the device sums (see KParams::grad).
struct GradOut {
    std::vector<double> signal, signal_se, mua, mus, mua_se, mus_se;
};

// det: [D][2] fixed-point (sum s, sum s^2); gsum: [D][R][5]; N photons; per-photon values
// are 0 for photons not scored, so each standard error is that of a mean over N.
void form_gradient(const uint64_t *det, const double *gsum, double N, double factor, const float *nmuasg, int D,
                   int R, GradOut &o)
{
    o.signal.assign((size_t)D, 0.0);
    o.signal_se.assign((size_t)D, 0.0);
    o.mua.assign((size_t)D * R, 0.0);
    o.mus.assign((size_t)D * R, 0.0);
    o.mua_se.assign((size_t)D * R, 0.0);
    o.mus_se.assign((size_t)D * R, 0.0);
    auto se = [N](double sx, double sxx) {
        return N > 1 ? std::sqrt(std::max(sxx / N - (sx / N) * (sx / N), 0.0) / N) : 0.0;
    };
    const double f = factor;
    for (int d = 0; d < D && N > 0; ++d) {
        const double s1 = (double)det[2 * d] / LP_FIX_ONE, s2 = (double)det[2 * d + 1] / LP_FIX_ONE;
        o.signal[d] = s1 / N;
        o.signal_se[d] = se(s1, s2);
        if (!gsum) continue;
        for (int r = 0; r < R; ++r) {
            const double *g = gsum + 5 * ((size_t)d * R + r);
            const double A = g[0], B = g[1], AA = g[2], BB = g[3], AB = g[4];
            const size_t i = (size_t)d * R + r;
            o.mua[i] = -A / f / N;
            o.mua_se[i] = se(-A / f, AA / (f * f));
            const double mus = (double)nmuasg[4 * r + 2];
            if (mus > 0.0) {
                const double sx = B / mus - A / f;
                const double sxx = BB / (mus * mus) + AA / (f * f) - 2.0 * AB / (mus * f);
                o.mus[i] = sx / N;
                o.mus_se[i] = se(sx, sxx);
            }
        }
    }
}

void fill_gradient(const GradOut &o, int D, int R, int64_t n, lp_gradient *out)
{
    out->n_det = D;
    out->n_media = R;
    out->n_photons = n;
    out->signal = o.signal.data();
    out->signal_se = o.signal_se.data();
    out->d_mua = o.mua.data();
    out->d_mus = o.mus.data();
    out->d_mua_se = o.mua_se.data();
    out->d_mus_se = o.mus_se.data();
}

}  // namespace

struct lp_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::string err;
    int num_sms = 148;
    // inputs
    bool have_mesh = false, have_media = false, have_source = false, have_grid = false;
    bool mesh_dirty = false, media_dirty = false, tally_dirty = true;
    int64_t n_tri = 0;
    int32_t max_region = 0;   // largest region id referenced by the mesh
    uint64_t mesh_gen = 0;    // counts the meshes and cell grids put on the device
    lp::Bvh bvh;
    std::vector<float4> tri_attr;
    std::vector<float> nmuasg;
    int32_t n_media = 0;
    float p_start[3] = {0, 0, 0}, v_start[3] = {0, 0, 1}, ep0xyz[12] = {0};
    float dimensions[3] = {1, 1, 1}, det_grid[6] = {1, 1, 1, 1, 1, 1};
    int32_t fetal_id = 1;
    float chance = 0.1f, w_th = 1e-4f, factor = 1.0f;
    uint64_t seed = 0x4C50;
    uint32_t compat = LP_COMPAT_ALL;
    bool exact = false;   // reference-order arithmetic (lp_set_arithmetic)
    int64_t max_steps = 100000000;
    int32_t vox_n[3] = {0, 0, 0};
    float vox_d[3] = {1, 1, 1};
    int32_t n_rbins = 0;
    float rbin_dr = 1.0f;
    std::vector<float> det_r;
    int64_t exit_cap = 0;
    float fiber_radius = 0.0f, fiber_na = 0.0f;
    lp_geometry geo{};
    // device buffers
    DevBuf<float4> node_a, node_b, node_c, tri, attr;
    DevBuf<int4> node_d;
    DevBuf<Medium> media;
    DevBuf<unsigned long long> sft, rtd, rz, vox, rbins, region, det, counters, work;
    DevBuf<unsigned long long> rz_part;   // copies of rz (KParams::rz_part), zero between launches
    bool rz_pending = false;              // but for deposits that are still to be folded (fold_rz)
    DevBuf<float> exit_rec;
    // safety grid (lp_set_safety_grid)
    // shared memory per block for staged BVH nodes and triangles: 8 KB stages a small mesh whole,
    // and on a large one the L1 left over (the cell grid, lists, triangles) is worth more than
    // the staged top of the tree (64 KB measured 1.2 % slower on the 202,500-triangle abdomen)
    int smem_budget = 8 * 1024;
    int64_t grid_max_cells = int64_t(1) << 24;
    bool grid_dirty = true;
    bool cell_lists = true;
    DevBuf<uint32_t> cell_word;
    DevBuf<int32_t> cell_refs;
    int64_t n_cell_refs = 0;
    float g_origin[3] = {0, 0, 0}, g_h = 0, g_unit = 0, g_eps = 0, g_step_eps = 0, g_push = 0;
    // lists hold the triangles touching each cell widened by cell_margin cells on every side
    // by default half a cell, or three quarters where the triangles are large (build_safety_grid)
    float cell_margin = 0.5f;
    bool margin_set = false;   // lp_set_cell_margin
    float grid_margin = 0.5f;  // the built grid's
    bool agg_tallies = false;   // lp_set_tally_aggregation
    int32_t g_n[3] = {0, 0, 0};
    float grid_ms = 0;
    // differentiation (lp_set_gradient / lp_forward / lp_backward)
    bool grad_on = false;
    DevBuf<double> grad;                  // [kMaxDet][kGradRegions][5], see KParams::grad
    std::vector<double> h_grad;
    GradOut gout;
    // host copies of tallies
    HostBuf<uint64_t> h_sft, h_rtd, h_rz, h_vox, h_rbins, h_region, h_det;
    float last_ms = 0.0f;
    bool launched = false;
    // statistics
    int64_t h2d_bytes = 0, d2h_bytes = 0;
    int32_t st_nodes_smem = 0, st_tris_smem = 0, st_smem = 0, st_per_sm = 0, st_grid = 0;
};

namespace {

int fail(lp_ctx *c, int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    g_thread_error = buf;
    return code;
}

int cuda_fail(lp_ctx *c, cudaError_t e, const char *what)
{
    cudaGetLastError();   // reported here: a later launch must not take it for its own
    return fail(c, e == cudaErrorMemoryAllocation ? LP_ERR_NOMEM : LP_ERR_CUDA, "%s: %s", what,
                cudaGetErrorString(e));
}

#define LP_CUDA(ctx, call)                                   \
    do {                                                     \
        cudaError_t _e = (call);                             \
        if (_e != cudaSuccess) return cuda_fail(ctx, _e, #call); \
    } while (0)

void geometry_of(const float dims[3], const float dg[6], lp_geometry &g)
{
    // CalculatePropagation::InitLogVectors (CP.cpp:127-131): float divisions, int casts
    g.dimx = (int32_t)(dims[0] / dg[0]);
    g.dimy = (int32_t)(dims[1] / dg[1]);
    g.dimz = (int32_t)(dims[2] / dg[2]);
    g.dimAlpha = (int32_t)(90 / dg[5]);
    g.dimR = (int32_t)std::ceil(std::sqrt(std::pow((double)(g.dimx / 2), 2) + std::pow((double)(g.dimy / 2), 2)));
    g.sft_nx = 2 * (g.dimx / 2) + 1;
    g.sft_ny = 2 * (g.dimy / 2) + 1;
    g.rz_nr = 2 * g.dimR + 1;
    g.rz_nz = g.dimz + 1;
    const float hx = (float)g.dimx / 2, hy = (float)g.dimy / 2;
    g.kernel_dimR = (int32_t)std::ceil(std::sqrt(std::pow(hx, 2.0f) + std::pow(hy, 2.0f)));
}

inline float normf3(float v[3])
{
    float l = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (l != 0.0f) {
        v[0] = v[0] / l;
        v[1] = v[1] / l;
        v[2] = v[2] / l;
    }
    return l;
}

int64_t n_vox(const lp_ctx *c)
{
    return c->vox_n[0] > 0 ? (int64_t)c->vox_n[0] * c->vox_n[1] * c->vox_n[2] : 0;
}

// Copies of an r-z image of n values for the deposits of a launch.  Every scatter event
// adds to its cell of the r-z image, and as all photons start at one point, a few cells
// near it take most of the adds: the L2 works them off one after the other.  On the curved
// abdomen at 660 nm (3e6 photons, 1.2 MB image, the step as it was then) one copy took
// 400 ms, two 277, four 217 and eight or more 216; without the deposits it was 215.
// Sixteen leave room for a faster step.  The limit keeps the copies of one image within a
// quarter of the L2 (a larger image has finer cells, so fewer adds to each).  The instances of
// a batch launch run side by side, each with an image of its own, and share out the sixteen:
// together they can be twice the L2 (eight images of 16 MB).
int rz_copies(size_t n, size_t images = 1)
{
    size_t k = 16;
    while (k > 1 && (k * n * 8 > (size_t(32) << 20) || k * images > 16)) k /= 2;
    return (int)k;
}

size_t rz_values(const lp_ctx *c) { return (size_t)c->geo.rz_nr * c->geo.rz_nz * 2; }

int alloc_tallies(lp_ctx *c)
{
    const lp_geometry &g = c->geo;
    LP_CUDA(c, c->sft.ensure((size_t)g.sft_nx * g.sft_ny * 3));
    LP_CUDA(c, c->rtd.ensure((size_t)g.dimR * g.dimAlpha * 3));
    LP_CUDA(c, c->rz.ensure(rz_values(c)));
    const int copies = rz_copies(rz_values(c));
    if (copies > 1) {
        LP_CUDA(c, c->rz_part.ensure(rz_values(c) * copies));
        LP_CUDA(c, cudaMemsetAsync(c->rz_part.p, 0, rz_values(c) * copies * 8, c->stream));
    }
    c->rz_pending = false;
    LP_CUDA(c, c->vox.ensure((size_t)std::max<int64_t>(n_vox(c), 1)));
    LP_CUDA(c, c->rbins.ensure((size_t)std::max(c->n_rbins, 1) * 2));
    LP_CUDA(c, c->region.ensure(lp::kMaxMedia));
    LP_CUDA(c, c->det.ensure((size_t)lp::kMaxDet * 2));
    LP_CUDA(c, c->counters.ensure(LP_NCOUNTERS));
    LP_CUDA(c, c->work.ensure(1));
    LP_CUDA(c, c->grad.ensure((size_t)lp::kMaxDet * lp::kGradRegions * 5));
    return LP_OK;
}

// Adds the deposits in the copies of the r-z image to it: after the launches of every run, the
// ones that did start when a later one failed included, and once more where the tallies are
// read if that launch failed too.
cudaError_t fold_rz(lp_ctx *c)
{
    if (!c->rz_pending) return cudaSuccess;
    const int copies = rz_copies(rz_values(c));
    cudaError_t e = cudaSetDevice(c->device);   // the reading calls need no device of their own
    if (e != cudaSuccess) return e;
    e = launch_unless_injected([&] {
        return lp::launch_fold(c->rz.p, c->rz_part.p, copies, (int64_t)rz_values(c), 1, c->stream);
    });
    if (e == cudaSuccess) c->rz_pending = false;
    return e;
}

// Drops deposits that are still to be folded, before the tallies are set to something else.
cudaError_t clear_rz_copies(lp_ctx *c)
{
    if (!c->rz_pending) return cudaSuccess;
    const cudaError_t e =
        cudaMemsetAsync(c->rz_part.p, 0, rz_values(c) * rz_copies(rz_values(c)) * 8, c->stream);
    if (e == cudaSuccess) c->rz_pending = false;
    return e;
}

int zero_tallies(lp_ctx *c)
{
    const lp_geometry &g = c->geo;
    cudaStream_t s = c->stream;
    LP_CUDA(c, clear_rz_copies(c));
    LP_CUDA(c, cudaMemsetAsync(c->sft.p, 0, (size_t)g.sft_nx * g.sft_ny * 3 * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->rtd.p, 0, (size_t)g.dimR * g.dimAlpha * 3 * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->rz.p, 0, (size_t)g.rz_nr * g.rz_nz * 2 * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->vox.p, 0, (size_t)std::max<int64_t>(n_vox(c), 1) * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->rbins.p, 0, (size_t)std::max(c->n_rbins, 1) * 2 * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->region.p, 0, lp::kMaxMedia * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->det.p, 0, lp::kMaxDet * 2 * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->counters.p, 0, LP_NCOUNTERS * 8, s));
    LP_CUDA(c, cudaMemsetAsync(c->grad.p, 0, (size_t)lp::kMaxDet * lp::kGradRegions * 5 * 8, s));
    return LP_OK;
}

int upload_mesh(lp_ctx *c)
{
    Phase phase("lp mesh upload");
    if (!c->mesh_dirty) return LP_OK;
    const lp::Bvh &b = c->bvh;
    const size_t nn = b.node_a.size(), nt = b.tri_a.size();
    ++c->mesh_gen;
    LP_CUDA(c, c->node_a.ensure(nn));
    LP_CUDA(c, c->node_b.ensure(nn));
    LP_CUDA(c, c->node_c.ensure(nn));
    LP_CUDA(c, c->node_d.ensure(nn));
    LP_CUDA(c, c->tri.ensure(3 * nt));
    DevBuf<float4> soa;   // the three arrays of the host tree, put together per triangle on the device
    LP_CUDA(c, soa.ensure(3 * nt));
    LP_CUDA(c, c->attr.ensure(nt));
    cudaStream_t s = c->stream;
    LP_CUDA(c, cudaMemcpyAsync(c->node_a.p, b.node_a.data(), nn * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->node_b.p, b.node_b.data(), nn * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->node_c.p, b.node_c.data(), nn * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->node_d.p, b.node_d.data(), nn * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(soa.p, b.tri_a.data(), nt * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(soa.p + nt, b.tri_b.data(), nt * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(soa.p + 2 * nt, b.tri_c.data(), nt * 16, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, lp::launch_interleave(soa.p, (int64_t)nt, c->tri.p, s));
    LP_CUDA(c, cudaMemcpyAsync(c->attr.p, c->tri_attr.data(), nt * 16, cudaMemcpyHostToDevice, s));
    c->h2d_bytes += (int64_t)(nn * 64 + nt * 64);
    c->mesh_dirty = false;
    return LP_OK;
}

// Device media records (with the derived factors of the fast mode) from (n, mua, mus, g).
void media_table(const float *nmuasg, int n_media, std::vector<Medium> &m)
{
    m.assign((size_t)n_media, Medium{});
    for (int i = 0; i < n_media; ++i) {
        const float *q = &nmuasg[4 * i];
        m[i].n = q[0];
        m[i].mua = q[1];
        m[i].mus = q[2];
        m[i].g = q[3];
        m[i].mut = q[1] + q[2];
        m[i].alb = q[1] / (q[1] + q[2]);
        m[i].kind = (q[1] > 0.0f && q[2] > 0.0f ? lp::kAbsorbs : 0u) |
                    (q[1] == 0.0f && q[2] == 0.0f ? lp::kAmbient : 0u) |
                    lp::plain_div_of(q[1], q[1] + q[2], q[3]);
        m[i].inv_mut = (q[1] + q[2]) > 0.0f ? 1.0f / (q[1] + q[2]) : 0.0f;
        m[i].inv_mua = q[1] > 0.0f ? 1.0f / q[1] : 0.0f;
        const float g = q[3];
        m[i].hg_a = 1.0f - g * g;
        m[i].hg_b = 1.0f - g;
        m[i].hg_c = 2.0f * g;
        m[i].hg_d = 1.0f + g * g;
        m[i].hg_inv2g = g != 0.0f ? 1.0f / (2.0f * g) : 0.0f;
    }
}

int upload_media(lp_ctx *c)
{
    if (!c->media_dirty) return LP_OK;
    std::vector<Medium> m;
    media_table(c->nmuasg.data(), c->n_media, m);
    LP_CUDA(c, c->media.ensure(lp::kMaxMedia));
    LP_CUDA(c, cudaMemcpyAsync(c->media.p, m.data(), m.size() * sizeof(Medium), cudaMemcpyHostToDevice,
                               c->stream));
    c->h2d_bytes += (int64_t)(m.size() * sizeof(Medium));
    c->media_dirty = false;
    return LP_OK;
}

int build_safety_grid(lp_ctx *c);

int upload(lp_ctx *c)
{
    if (!c->have_mesh || !c->have_media || !c->have_source || !c->have_grid)
        return fail(c, LP_ERR_STATE, "lp_run: mesh, media, source and tally grid must be set first");
    if (c->max_region >= c->n_media)
        return fail(c, LP_ERR_INVALID, "lp_run: mesh references region %d but only %d regions are set",
                    c->max_region, c->n_media);
    LP_CUDA(c, cudaSetDevice(c->device));
    int r = upload_mesh(c);
    if (r) return r;
    r = upload_media(c);
    if (r) return r;
    if (c->tally_dirty) {
        r = alloc_tallies(c);
        if (r) return r;
        r = zero_tallies(c);
        if (r) return r;
        c->tally_dirty = false;
    }
    if (c->exit_cap > 0) LP_CUDA(c, c->exit_rec.ensure((size_t)c->exit_cap * 8));
    if (c->grid_dirty) {
        r = build_safety_grid(c);
        if (r) return r;
    }
    return LP_OK;
}

float rspecular(const float *nm, int n_media)
{
    // Rspecular (MCLightPropagation.cl:273-299)
    if (n_media < 2) return 0.0f;
    float r1, r2, temp;
    const float n1 = nm[0], n2 = nm[4], mua1 = nm[5], mus1 = nm[6];
    temp = (n1 - n2) / (n1 + n2);
    r1 = temp * temp;
    if (mua1 == 0.0f && mus1 == 0.0f && n_media > 2) {
        const float n3 = nm[8];
        temp = (n2 - n3) / (n2 + n3);
        r2 = temp * temp;
        r1 = r1 + (1 - r1) * (1 - r1) * r2 / (1 - r1 * r2);
    }
    return r1;
}

void fill_params(lp_ctx *c, KParams &P, int64_t first, int64_t n, int nodes_smem, int tris_smem)
{
    std::memset(&P, 0, sizeof P);
    P.node_a = c->node_a.p; P.node_b = c->node_b.p; P.node_c = c->node_c.p; P.node_d = c->node_d.p;
    P.tri = c->tri.p; P.tri_attr = c->attr.p;
    P.n_nodes = (int32_t)c->bvh.node_a.size();
    P.n_tri = (int32_t)c->n_tri;
    P.nodes_smem = nodes_smem;
    P.tris_smem = tris_smem;
    P.media = c->media.p;
    P.n_media = c->n_media;
    P.p0x = c->p_start[0]; P.p0y = c->p_start[1]; P.p0z = c->p_start[2];
    P.v0x = c->v_start[0]; P.v0y = c->v_start[1]; P.v0z = c->v_start[2];
    P.poix = c->ep0xyz[0]; P.poiy = c->ep0xyz[1]; P.poiz = c->ep0xyz[2];
    float ex[3] = {c->ep0xyz[3], c->ep0xyz[4], c->ep0xyz[5]};
    float ey[3] = {c->ep0xyz[6], c->ep0xyz[7], c->ep0xyz[8]};
    float ez[3] = {c->ep0xyz[9], c->ep0xyz[10], c->ep0xyz[11]};
    P.ezx = ez[0]; P.ezy = ez[1]; P.ezz = ez[2];
    normf3(ex); normf3(ey); normf3(ez);
    P.nxx = ex[0]; P.nxy = ex[1]; P.nxz = ex[2];
    P.nyx = ey[0]; P.nyy = ey[1]; P.nyz = ey[2];
    P.nzx = ez[0]; P.nzy = ez[1]; P.nzz = ez[2];
    P.Rsp = rspecular(c->nmuasg.data(), c->n_media);
    P.w0 = 1.0f - P.Rsp;
    P.exitScale = (c->compat & LP_COMPAT_EXIT_RSP) ? (1 - P.Rsp) : 1.0f;
    P.distMin = c->det_grid[2] * (float)c->geo.dimz / 2.0f;   // .cl:1351
    P.chance = c->chance;
    P.w_th = c->w_th;
    P.factor = c->factor;
    P.fetal_id = c->fetal_id;
    P.compat = c->compat;
    lp::set_keys(P, c->seed);
    P.stream = 0;
    P.first = first;
    P.n = n;
    P.step_cap = lp::step_cap_of(c->max_steps);
    const lp_geometry &g = c->geo;
    P.hx = g.dimx / 2; P.hy = g.dimy / 2; P.sft_nx = g.sft_nx;
    P.dimR = g.dimR; P.dimAlpha = g.dimAlpha; P.rz_nr = g.rz_nr; P.rz_nz = g.rz_nz;
    for (int i = 0; i < 6; ++i) P.dg[i] = c->det_grid[i];
    P.inv_dr = 1.0f / c->det_grid[3];
    P.inv_dz = 1.0f / c->det_grid[2];
    P.inv_vdx = 1.0f / c->vox_d[0];
    P.inv_vdy = 1.0f / c->vox_d[1];
    P.inv_vdz = 1.0f / c->vox_d[2];
    P.f_dimR = (float)g.dimR;
    P.half_vnx = 0.5f * (float)c->vox_n[0];
    P.half_vny = 0.5f * (float)c->vox_n[1];
    P.vox_on = c->vox_n[0] > 0 ? 1u : 0u;
    P.plain_div = lp::div_range(c->det_grid[2]) && lp::div_range(c->det_grid[3]) &&
                          (!P.vox_on || (lp::div_range(c->vox_d[0]) && lp::div_range(c->vox_d[1]) &&
                                         lp::div_range(c->vox_d[2])))
                      ? 0u
                      : 1u;
    P.sft = c->sft.p; P.rtd = c->rtd.p; P.rz = c->rz.p; P.vox = c->vox.p; P.rbins = c->rbins.p;
    P.region = c->region.p; P.det = c->det.p; P.counters = c->counters.p;
    const int copies = rz_copies(rz_values(c));
    P.rz_part = copies > 1 ? c->rz_part.p : c->rz.p;
    P.rz_stride = (int64_t)rz_values(c);
    P.rz_mask = (uint32_t)(copies - 1);
    P.vox_nx = c->vox_n[0]; P.vox_ny = c->vox_n[1]; P.vox_nz = c->vox_n[2];
    P.vox_dx = c->vox_d[0]; P.vox_dy = c->vox_d[1]; P.vox_dz = c->vox_d[2];
    P.n_rbins = c->n_rbins;
    P.rbin_dr = c->rbin_dr;
    P.n_det = (int32_t)(c->det_r.size() / 2);
    for (int k = 0; k < P.n_det; ++k) {
        P.det_lo[k] = c->det_r[2 * k];
        P.det_hi[k] = c->det_r[2 * k + 1];
    }
    P.src_type = (c->fiber_radius > 0.0f || c->fiber_na > 0.0f) ? 1 : 0;
    P.src_radius = c->fiber_radius;
    {
        // the query-only path runs without media: the cone is unused there
        const float n0 = c->nmuasg.empty() ? 1.0f : c->nmuasg[0];
        const float s = c->fiber_na / n0;
        P.src_cos_max = s < 1.0f ? std::sqrt(1.0f - s * s) : 0.0f;
    }
    P.exit_rec = c->exit_cap > 0 ? c->exit_rec.p : nullptr;
    P.exit_cap = c->exit_cap;
    P.grad = c->grad_on ? c->grad.p : nullptr;
    P.work = c->work.p;
    const bool grid = c->grid_max_cells > 0 && c->cell_word.p && !c->grid_dirty;
    P.cell_word = grid ? c->cell_word.p : nullptr;
    P.cell_refs = (grid && c->cell_lists && c->n_cell_refs > 0) ? c->cell_refs.p : nullptr;
    P.n_cell_refs = P.cell_refs ? c->n_cell_refs : 0;
    P.g_eps = c->g_eps;
    P.g_ox = c->g_origin[0];
    P.g_oy = c->g_origin[1];
    P.g_oz = c->g_origin[2];
    P.g_inv_h = c->g_h > 0 ? 1.0f / c->g_h : 0.0f;
    P.g_unit = c->g_unit;
    P.g_nx = grid ? c->g_n[0] : 0;
    P.g_ny = grid ? c->g_n[1] : 0;
    P.g_nz = grid ? c->g_n[2] : 0;
    P.g_h = c->g_h;
    P.g_margin = c->grid_margin * c->g_h;
    P.step_eps = c->g_step_eps;
    P.boundary_push = c->exact ? 0.0f : c->g_push;
    P.tri_eps = c->exact ? 0.0f : 2e-6f;
    P.agg_tallies = c->agg_tallies ? 1 : 0;
}

// Cell grid over the mesh bounds padded by one cell: cubic cells of size h chosen so
// the grid has at most grid_max_cells cells; distance bounds in units of h / 256.
//   1. cell_lists_kernel (count pass): per cell, the triangles touching it;
//   2. exclusive scan of the counts: each cell's first slot in cell_refs;
//   3. cell_lists_kernel (fill pass): the triangle indices;
//   4. launch_cell_words: the distance bounds of the empty cells, and one word per cell
//      (KParams::cell_word).
int build_safety_grid(lp_ctx *c)
{
    Phase phase("lp cell grid build");
    c->n_cell_refs = 0;
    ++c->mesh_gen;
    if (c->grid_max_cells <= 0 || c->n_tri == 0) {
        c->cell_word.release();
        c->cell_refs.release();
        c->grid_dirty = false;
        return LP_OK;
    }
    const lp::Bvh &b = c->bvh;
    double ext[3], vol = 1.0, scale = 0.0;
    for (int a = 0; a < 3; ++a) {
        ext[a] = std::max((double)b.hi[a] - b.lo[a], 1e-6);
        vol *= ext[a];
        scale = std::max({scale, ext[a], std::fabs((double)b.lo[a]), std::fabs((double)b.hi[a])});
    }
    double h = std::cbrt(vol / (double)c->grid_max_cells);
    h = std::max(h, 1e-6 * scale);
    int64_t cells = 0;
    for (int it = 0; it < 200; ++it) {
        cells = 1;
        for (int a = 0; a < 3; ++a) {
            c->g_n[a] = (int32_t)std::ceil(ext[a] / h) + 2;
            cells *= c->g_n[a];
        }
        if (cells <= c->grid_max_cells) break;
        h *= 1.05;
    }
    if (cells > c->grid_max_cells) return fail(c, LP_ERR_RANGE, "safety grid: cannot fit %lld cells", (long long)cells);
    c->g_h = (float)h;
    c->g_unit = (float)(h / 256.0);
    // list margin: far above the rounding of coordinates and of the ray/triangle test's
    // intersection point at this scale, far below any cell size
    c->g_eps = (float)(2e-5 * scale);
    // rounding of one position update p + s v: under 2 ulp of the largest coordinate per
    // component; 5e-7 * scale is about 4 ulp (2^-23 = 1.19e-7)
    c->g_step_eps = (float)(5e-7 * scale);
    for (int a = 0; a < 3; ++a) c->g_origin[a] = (float)(b.lo[a] - h);
    // scratch of the build, in one allocation: counts, offsets, bounds, row gaps, scan
    size_t tmp_bytes = 0;
    cudaStream_t s = c->stream;
    LP_CUDA(c, cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, (uint32_t *)nullptr, (uint32_t *)nullptr, cells, s));
    const size_t n_cells = ((size_t)cells + 255) & ~(size_t)255;
    LP_CUDA(c, c->cell_word.ensure((size_t)cells));
    DevBuf<unsigned char> scratch;
    LP_CUDA(c, scratch.ensure(n_cells * 13 + tmp_bytes));
    uint32_t *const count = reinterpret_cast<uint32_t *>(scratch.p), *const start = count + n_cells;
    float *const d2 = reinterpret_cast<float *>(start + n_cells);
    uint8_t *const gap = reinterpret_cast<uint8_t *>(d2 + n_cells);
    void *const scan_tmp = gap + n_cells;
    KParams P;
    std::memset(&P, 0, sizeof P);
    P.node_a = c->node_a.p; P.node_b = c->node_b.p; P.node_c = c->node_c.p; P.node_d = c->node_d.p;
    P.tri = c->tri.p;
    P.g_ox = c->g_origin[0]; P.g_oy = c->g_origin[1]; P.g_oz = c->g_origin[2];
    P.g_nx = c->g_n[0]; P.g_ny = c->g_n[1]; P.g_nz = c->g_n[2];
    P.g_unit = c->g_unit;
    P.g_inv_h = 1.0f / c->g_h;
    P.g_h = c->g_h;
    P.g_eps = c->g_eps;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    bool lists = false;
    const int nt = (int)c->bvh.tri_a.size();
    // A march stands still between a cell's faces without a margin, and its queries go to the
    // tree: 0 cells / a quarter, ms: slab 2e5 photons 51 / 33, abdomen 25,600 triangles 1e5 75 / 23,
    // 202,500 3e5 133 / 39, 2.25 M 1e5 72 / 32.
    c->grid_margin = std::max(c->cell_margin, 0.25f);
    // every list holds the triangles that touch its cell widened by the margin plus g_eps
    auto list_eps = [c]() { return c->grid_margin * c->g_h + c->g_eps; };
    // counts, their scan and the number of entries
    auto count_lists = [&](int64_t &total) {
        cudaError_t r = cudaMemsetAsync(count, 0, (size_t)cells * 4, s);
        if (r == cudaSuccess) r = lp::launch_cell_lists(P, nt, c->g_h, list_eps(), count, nullptr, nullptr, s);
        if (r != cudaSuccess || !c->cell_lists) return r;
        uint32_t last[2] = {0, 0};
        if ((r = cub::DeviceScan::ExclusiveSum(scan_tmp, tmp_bytes, count, start, cells, s)) == cudaSuccess &&
            (r = cudaMemcpyAsync(&last[0], start + cells - 1, 4, cudaMemcpyDeviceToHost, s)) == cudaSuccess &&
            (r = cudaMemcpyAsync(&last[1], count + cells - 1, 4, cudaMemcpyDeviceToHost, s)) == cudaSuccess)
            r = cudaStreamSynchronize(s);
        total = (int64_t)last[0] + last[1];
        return r;
    };
    int64_t total = 0;
    cudaError_t e = count_lists(total);
    // Triangles of many cells make short lists, which a wider margin lengthens by little while
    // the queries get fewer: slab (32 triangles), 1e6 photons, 98 -> 91 ms with three quarters
    // of a cell.  On the abdomen with 25,600 triangles (about 100 cells each) 71.6 -> 71.2, with
    // 202,500 (about 30) 73.2 -> 74.5.
    if (e == cudaSuccess && !c->margin_set && total >= 64 * (int64_t)nt && total <= (int64_t(1) << 22)) {
        c->grid_margin = 0.75f;
        e = count_lists(total);
    }
    // cells past 2^24 list entries are marked dense (BVH); beyond 2^28 lists are off
    if (e == cudaSuccess && total > 0 && total <= (int64_t(1) << 28)) {
        if ((e = c->cell_refs.ensure((size_t)total)) == cudaSuccess &&
            (e = cudaMemsetAsync(count, 0, (size_t)cells * 4, s)) == cudaSuccess &&
            (e = lp::launch_cell_lists(P, nt, c->g_h, list_eps(), count, start, c->cell_refs.p, s)) == cudaSuccess) {
            lists = true;
            c->n_cell_refs = total;
        }
    }
    if (e == cudaSuccess)
        e = lp::launch_cell_words(P, c->grid_margin, count, start, lists, gap, d2, c->cell_word.p, s);
    cudaEventRecord(e1, s);
    cudaEventSynchronize(e1);
    cudaEventElapsedTime(&c->grid_ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return cuda_fail(c, e, "cell grid");
    if (!lists) c->cell_refs.release();
    c->grid_dirty = false;   // a build that failed is tried again by the next run
    return LP_OK;
}

// shared-memory staging: as many top BVH levels and leading triangles as fit the budget
void smem_plan(const lp_ctx *c, int budget, int &nodes_smem, int &tris_smem)
{
    const int base = lp::smem_bytes(0, 0);
    int room = std::max(0, budget - base);
    const int nn = (int)c->bvh.node_a.size(), nt = (int)c->bvh.tri_a.size();
    nodes_smem = std::min(nn, room / 64);
    room -= nodes_smem * 64;
    tris_smem = std::min(nt, room / 48);
}

}  // namespace

// helpers shared with lp_noalloc.cu
namespace lp {
void set_thread_error(const char *msg) { g_thread_error = msg; }
float rspecular_of(const float *nmuasg, int n_media) { return rspecular(nmuasg, n_media); }
}  // namespace lp

// ============================================================ C ABI
extern "C" {

const char *lp_last_error(const lp_ctx *ctx)
{
    if (ctx) return ctx->err.c_str();
    return g_thread_error.c_str();
}

int lp_create(lp_ctx **out, int device)
{
    if (!out) return fail(nullptr, LP_ERR_INVALID, "lp_create: out is NULL");
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0)
        return fail(nullptr, LP_ERR_CUDA, "lp_create: no CUDA device (%s)", cudaGetErrorString(e));
    if (device < 0 || device >= n) return fail(nullptr, LP_ERR_INVALID, "lp_create: device %d of %d", device, n);
    lp_ctx *c = new (std::nothrow) lp_ctx;
    if (!c) return fail(nullptr, LP_ERR_NOMEM, "lp_create: out of host memory");
    c->device = device;
    if ((e = cudaSetDevice(device)) != cudaSuccess || (e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreate(&c->ev0)) != cudaSuccess || (e = cudaEventCreate(&c->ev1)) != cudaSuccess) {
        int r = cuda_fail(nullptr, e, "lp_create");
        delete c;
        return r;
    }
    cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
    *out = c;
    return LP_OK;
}

void lp_destroy(lp_ctx *c)
{
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    c->node_a.release(); c->node_b.release(); c->node_c.release(); c->node_d.release();
    c->tri.release(); c->attr.release();
    c->media.release();
    c->sft.release(); c->rtd.release(); c->rz.release(); c->vox.release(); c->rbins.release();
    c->region.release(); c->det.release(); c->counters.release(); c->work.release();
    c->exit_rec.release();
    c->cell_word.release();
    c->cell_refs.release();
    if (c->ev0) cudaEventDestroy(c->ev0);
    if (c->ev1) cudaEventDestroy(c->ev1);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

int lp_set_mesh(lp_ctx *c, int64_t n_tri, const float *tri, const float *nrm, const int32_t *med)
{
    Phase phase("lp BVH build");
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_mesh: ctx is NULL");
    if (n_tri <= 0 || !tri || !nrm || !med) return fail(c, LP_ERR_INVALID, "lp_set_mesh: empty mesh or NULL array");
    if (n_tri > (int64_t(1) << 27)) return fail(c, LP_ERR_RANGE, "lp_set_mesh: %lld triangles > 2^27", (long long)n_tri);
    for (int64_t i = 0; i < 2 * n_tri; ++i)
        if (med[i] < 0 || med[i] >= lp::kMaxMedia)
            return fail(c, LP_ERR_INVALID, "lp_set_mesh: region id %d of triangle %lld out of range", med[i],
                        (long long)(i / 2));
    try {
        lp::build_bvh(tri, n_tri, c->bvh);
    } catch (const std::bad_alloc &) {
        // the context holds no usable mesh until the next successful lp_set_mesh
        c->bvh = lp::Bvh();
        c->have_mesh = false;
        return fail(c, LP_ERR_NOMEM, "lp_set_mesh: out of host memory building the BVH of %lld triangles",
                    (long long)n_tri);
    }
    if (c->bvh.depth >= lp::kStackDepth) {
        c->have_mesh = false;
        return fail(c, LP_ERR_RANGE, "lp_set_mesh: BVH depth %d exceeds the traversal stack", c->bvh.depth);
    }
    c->tri_attr.resize((size_t)n_tri);
    for (int64_t i = 0; i < n_tri; ++i) {
        // nv = normalize(vload3(triID, normals)) (.cl:1489), done once here
        float v[3] = {nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2]};
        normf3(v);
        const int32_t ids = (med[2 * i] & 0xffff) | (med[2 * i + 1] << 16);
        float fb;
        std::memcpy(&fb, &ids, 4);
        c->tri_attr[i] = make_float4(v[0], v[1], v[2], fb);
    }
    c->n_tri = n_tri;
    {
        // boundary push of the production arithmetic: about 8 float ulps of the largest
        // coordinate of the mesh (2^-23 = 1.19e-7)
        double scale = 0.0;
        for (int a = 0; a < 3; ++a)
            scale = std::max({scale, std::fabs((double)c->bvh.lo[a]), std::fabs((double)c->bvh.hi[a])});
        c->g_push = (float)(1e-6 * scale);
    }
    c->max_region = 0;
    for (int64_t i = 0; i < 2 * n_tri; ++i) c->max_region = std::max(c->max_region, med[i]);
    c->have_mesh = true;
    c->mesh_dirty = true;
    c->grid_dirty = true;
    return LP_OK;
}

int lp_set_media(lp_ctx *c, int32_t n_media, const float *nmuasg)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_media: ctx is NULL");
    if (n_media < 1 || n_media > lp::kMaxMedia || !nmuasg)
        return fail(c, LP_ERR_RANGE, "lp_set_media: %d regions (1..%d supported)", n_media, lp::kMaxMedia);
    for (int i = 0; i < 4 * n_media; ++i)
        if (!std::isfinite(nmuasg[i])) return fail(c, LP_ERR_INVALID, "lp_set_media: non-finite value at %d", i);
    c->nmuasg.assign(nmuasg, nmuasg + 4 * n_media);
    c->n_media = n_media;
    c->have_media = true;
    c->media_dirty = true;
    return LP_OK;
}

int lp_set_source(lp_ctx *c, const float *p_start, const float *v_start, const int32_t *v_occ, int32_t k,
                  const float *ep0xyz)
{
    (void)v_occ;
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_source: ctx is NULL");
    if (!p_start || !v_start || k < 1 || !ep0xyz) return fail(c, LP_ERR_INVALID, "lp_set_source: missing input");
    std::memcpy(c->p_start, p_start, 12);
    std::memcpy(c->v_start, v_start, 12);
    std::memcpy(c->ep0xyz, ep0xyz, 48);
    c->have_source = true;
    return LP_OK;
}

int lp_set_fiber_source(lp_ctx *c, float radius, float na)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_fiber_source: ctx is NULL");
    if (!(radius >= 0.0f) || !(na >= 0.0f) || !(na < 1.0f))
        return fail(c, LP_ERR_INVALID, "lp_set_fiber_source: radius %g, NA %g", radius, na);
    c->fiber_radius = radius;
    c->fiber_na = na;
    return LP_OK;
}

int lp_set_tally_grid(lp_ctx *c, const float *dimensions, const float *det_grid, int32_t fetal_id)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_tally_grid: ctx is NULL");
    if (!dimensions || !det_grid) return fail(c, LP_ERR_INVALID, "lp_set_tally_grid: NULL input");
    for (int i = 0; i < 6; ++i)
        if (!(det_grid[i] > 0.0f)) return fail(c, LP_ERR_INVALID, "lp_set_tally_grid: grid step %d not positive", i);
    lp_geometry g;
    geometry_of(dimensions, det_grid, g);
    if (g.dimx < 0 || g.dimy < 0 || g.dimz < 0 || g.dimAlpha < 1 || g.dimR < 1 ||
        (int64_t)g.sft_nx * g.sft_ny > (int64_t(1) << 28) || (int64_t)g.rz_nr * g.rz_nz > (int64_t(1) << 28))
        return fail(c, LP_ERR_RANGE, "lp_set_tally_grid: image extents out of range");
    std::memcpy(c->dimensions, dimensions, 12);
    std::memcpy(c->det_grid, det_grid, 24);
    c->geo = g;
    c->fetal_id = fetal_id;
    c->have_grid = true;
    c->tally_dirty = true;
    return LP_OK;
}

int lp_set_params(lp_ctx *c, float chance, float w_threshold, float factor, uint64_t seed, uint32_t compat)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_params: ctx is NULL");
    if (!(chance > 0.0f && chance <= 1.0f)) return fail(c, LP_ERR_INVALID, "lp_set_params: chance %g", chance);
    if (!(w_threshold >= 0.0f) || !(factor > 0.0f)) return fail(c, LP_ERR_INVALID, "lp_set_params: bad threshold/factor");
    c->chance = chance;
    c->w_th = w_threshold;
    c->factor = factor;
    c->seed = seed;
    c->compat = compat & LP_COMPAT_ALL;
    return LP_OK;
}

int lp_set_extra_tallies(lp_ctx *c, const int32_t *vox_n, const float *vox_d, int32_t n_rbins, float rbin_dr,
                         int32_t n_det, const float *det_r)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_extra_tallies: ctx is NULL");
    if (n_det < 0 || n_det > lp::kMaxDet) return fail(c, LP_ERR_RANGE, "lp_set_extra_tallies: %d rings > %d", n_det, lp::kMaxDet);
    if (vox_n && vox_n[0] > 0) {
        if (!vox_d || vox_n[1] <= 0 || vox_n[2] <= 0 || !(vox_d[0] > 0) || !(vox_d[1] > 0) || !(vox_d[2] > 0))
            return fail(c, LP_ERR_INVALID, "lp_set_extra_tallies: bad voxel grid");
        if ((int64_t)vox_n[0] * vox_n[1] * vox_n[2] > (int64_t(1) << 31))
            return fail(c, LP_ERR_RANGE, "lp_set_extra_tallies: voxel grid too large");
        std::memcpy(c->vox_n, vox_n, 12);
        std::memcpy(c->vox_d, vox_d, 12);
    } else {
        c->vox_n[0] = c->vox_n[1] = c->vox_n[2] = 0;
    }
    if (n_rbins < 0 || (n_rbins > 0 && !(rbin_dr > 0))) return fail(c, LP_ERR_INVALID, "lp_set_extra_tallies: bad radial bins");
    c->n_rbins = n_rbins;
    c->rbin_dr = rbin_dr;
    c->det_r.assign(det_r ? det_r : (const float *)nullptr, det_r ? det_r + 2 * n_det : (const float *)nullptr);
    c->tally_dirty = true;
    return LP_OK;
}

int lp_set_arithmetic(lp_ctx *c, int exact)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_arithmetic: ctx is NULL");
    c->exact = exact != 0;
    return LP_OK;
}

int lp_set_tally_aggregation(lp_ctx *c, int enable)
{
    if (!c) return LP_ERR_INVALID;
    c->agg_tallies = enable != 0;
    return LP_OK;
}

int lp_set_cell_margin(lp_ctx *c, float cells)
{
    if (!c) return LP_ERR_INVALID;
    if (!(cells >= 0.0f && cells <= 4.0f)) return fail(c, LP_ERR_INVALID, "lp_set_cell_margin: %g cells", (double)cells);
    if (!c->margin_set || cells != c->cell_margin) {
        c->cell_margin = cells;
        c->margin_set = true;
        c->grid_dirty = true;
    }
    return LP_OK;
}

int lp_set_safety_grid(lp_ctx *c, int64_t max_cells)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_safety_grid: ctx is NULL");
    if (max_cells < 0 || max_cells > (int64_t(1) << 28)) return fail(c, LP_ERR_RANGE, "lp_set_safety_grid: %lld cells", (long long)max_cells);
    c->grid_max_cells = max_cells;
    c->grid_dirty = true;
    return LP_OK;
}

int lp_set_smem_budget(lp_ctx *c, int32_t bytes)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_smem_budget: ctx is NULL");
    if (bytes < lp::smem_bytes(0, 0) || bytes > 200 * 1024)
        return fail(c, LP_ERR_RANGE, "lp_set_smem_budget: %d bytes (%d..%d)", bytes, lp::smem_bytes(0, 0), 200 * 1024);
    c->smem_budget = bytes;
    return LP_OK;
}

int lp_set_gradient(lp_ctx *c, int enable)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_gradient: ctx is NULL");
    c->grad_on = enable != 0;
    return LP_OK;
}

int lp_get_gradient(lp_ctx *c, lp_gradient *out)
{
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_gradient: NULL argument");
    if (!c->grad.p || !c->counters.p || !c->det.p) return fail(c, LP_ERR_STATE, "lp_get_gradient: nothing has run");
    const int D = (int)c->det_r.size() / 2, R = c->n_media;
    if (R > lp::kGradRegions) return fail(c, LP_ERR_RANGE, "lp_get_gradient: %d regions (at most %d)", R,
                                          lp::kGradRegions);
    LP_CUDA(c, cudaSetDevice(c->device));
    std::vector<uint64_t> det((size_t)std::max(D, 1) * 2), cnt(LP_NCOUNTERS);
    c->h_grad.assign((size_t)std::max(D * R, 1) * 5, 0.0);
    cudaStream_t s = c->stream;
    if (D > 0) {
        LP_CUDA(c, cudaMemcpyAsync(c->h_grad.data(), c->grad.p, (size_t)D * R * 5 * 8, cudaMemcpyDeviceToHost, s));
        LP_CUDA(c, cudaMemcpyAsync(det.data(), c->det.p, (size_t)D * 2 * 8, cudaMemcpyDeviceToHost, s));
    }
    LP_CUDA(c, cudaMemcpyAsync(cnt.data(), c->counters.p, LP_NCOUNTERS * 8, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaStreamSynchronize(s));
    form_gradient(det.data(), c->h_grad.data(), (double)cnt[LP_C_PHOTONS], (double)c->factor, c->nmuasg.data(), D, R,
                  c->gout);
    fill_gradient(c->gout, D, R, (int64_t)cnt[LP_C_PHOTONS], out);
    c->d2h_bytes = (int64_t)(D * R * 5 + D * 2 + LP_NCOUNTERS) * 8;
    return LP_OK;
}

int lp_forward(lp_ctx *c, int64_t first, int64_t n, double *signal)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_forward: ctx is NULL");
    c->grad_on = true;
    int r = lp_zero_tallies(c);
    if (r) return r;
    if ((r = lp_run(c, first, n))) return r;
    lp_gradient g;
    if ((r = lp_get_gradient(c, &g))) return r;
    if (signal)
        for (int d = 0; d < g.n_det; ++d) signal[d] = g.signal[d];
    return LP_OK;
}

int lp_backward(lp_ctx *c, const double *grad_signal, double *grad_mua, double *grad_mus)
{
    if (!c || !grad_signal || !grad_mua || !grad_mus) return fail(c, LP_ERR_INVALID, "lp_backward: NULL argument");
    const int R = c->n_media, D = (int)c->gout.signal.size();
    if ((int64_t)c->gout.mua.size() != (int64_t)D * R) return fail(c, LP_ERR_STATE, "lp_backward: no lp_forward before");
    for (int r = 0; r < R; ++r) {
        double a = 0.0, b = 0.0;
        for (int d = 0; d < D; ++d) {
            a += grad_signal[d] * c->gout.mua[(size_t)d * R + r];
            b += grad_signal[d] * c->gout.mus[(size_t)d * R + r];
        }
        grad_mua[r] = a;
        grad_mus[r] = b;
    }
    return LP_OK;
}

int lp_set_cell_lists(lp_ctx *c, int enable)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_cell_lists: ctx is NULL");
    if ((enable != 0) != c->cell_lists) {
        c->cell_lists = enable != 0;
        c->grid_dirty = true;
    }
    return LP_OK;
}

int lp_set_max_steps(lp_ctx *c, int64_t max_steps)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_max_steps: ctx is NULL");
    c->max_steps = max_steps;
    return LP_OK;
}

int lp_set_exit_records(lp_ctx *c, int64_t capacity)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_set_exit_records: ctx is NULL");
    if (capacity < 0 || capacity > (int64_t(1) << 30)) return fail(c, LP_ERR_RANGE, "lp_set_exit_records: capacity");
    c->exit_cap = capacity;
    return LP_OK;
}

int lp_run_async(lp_ctx *c, int64_t first, int64_t n)
{
    Phase phase("lp transport launch");
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_run: ctx is NULL");
    if (n < 0 || first < 0) return fail(c, LP_ERR_INVALID, "lp_run: negative photon range");
    c->h2d_bytes = 0;
    int r = upload(c);
    if (r) return r;
    if (n == 0) return LP_OK;
    if (c->grad_on && c->n_media > lp::kGradRegions)
        return fail(c, LP_ERR_RANGE, "lp_run: differentiation supports at most %d regions (%d set)",
                    lp::kGradRegions, c->n_media);
    int nodes_smem, tris_smem;
    smem_plan(c, c->smem_budget, nodes_smem, tris_smem);
    const int smem = lp::smem_bytes(nodes_smem, tris_smem);
    int per_sm = 0;
    if (c->grad_on)
        LP_CUDA(c, c->exact ? lp::transport_occupancy_exact_grad(smem, &per_sm)
                            : lp::transport_occupancy_fast_grad(smem, &per_sm));
    else
        LP_CUDA(c, c->exact ? lp::transport_occupancy_exact(smem, &per_sm)
                            : lp::transport_occupancy_fast(smem, &per_sm));
    if (per_sm < 1) return fail(c, LP_ERR_CUDA, "lp_run: transport kernel does not fit on an SM");
    if (c->exit_cap > 0) LP_CUDA(c, cudaMemsetAsync(c->exit_rec.p, 0, (size_t)c->exit_cap * 32, c->stream));
    LP_CUDA(c, cudaEventRecord(c->ev0, c->stream));
    c->st_nodes_smem = nodes_smem;
    c->st_tris_smem = tris_smem;
    c->st_smem = smem;
    c->st_per_sm = per_sm;
    // The kernel indexes the photons of one launch with 32 bits: a longer range runs as
    // several launches in order (the same photon ids, so the same tallies).  Exit records
    // (at most 2^30 slots, indexed from the range's first photon) all come from the first.
    const bool copies = rz_copies(rz_values(c)) > 1;
    cudaError_t e = cudaSuccess;
    for (int64_t off = 0; off < n && e == cudaSuccess; off += lp::kMaxLaunchPhotons) {
        const int64_t m = std::min<int64_t>(n - off, lp::kMaxLaunchPhotons);
        KParams P;
        fill_params(c, P, first + off, m, nodes_smem, tris_smem);
        if (off > 0) {
            P.exit_rec = nullptr;
            P.exit_cap = 0;
        }
        int grid;
        lp::plan_launch(m, lp::block_size(), c->num_sms, per_sm, grid, P.lane_mask, P.few_blocks);
        c->st_grid = grid;
        c->h2d_bytes += (int64_t)sizeof(KParams);
        e = cudaMemsetAsync(c->work.p, 0, 8, c->stream);
        if (e == cudaSuccess)
            e = launch_unless_injected([&] {
                return c->exact ? lp::launch_transport_exact(P, grid, smem, c->stream)
                                : lp::launch_transport_fast(P, grid, smem, c->stream);
            });
        if (e == cudaSuccess) c->rz_pending = copies;
    }
    const cudaError_t folded = fold_rz(c);
    if (e == cudaSuccess) e = folded;
    if (e != cudaSuccess) return cuda_fail(c, e, "lp_run: launch");
    LP_CUDA(c, cudaEventRecord(c->ev1, c->stream));
    c->launched = true;
    return LP_OK;
}

int lp_sync(lp_ctx *c)
{
    Phase phase("lp transport wait");
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_sync: ctx is NULL");
    LP_CUDA(c, cudaStreamSynchronize(c->stream));
    if (c->launched) {
        LP_CUDA(c, cudaEventElapsedTime(&c->last_ms, c->ev0, c->ev1));
        c->launched = false;
    }
    return LP_OK;
}

int lp_run(lp_ctx *c, int64_t first, int64_t n)
{
    int r = lp_run_async(c, first, n);
    if (r) return r;
    return lp_sync(c);
}

int lp_zero_tallies(lp_ctx *c)
{
    if (!c) return fail(nullptr, LP_ERR_INVALID, "lp_zero_tallies: ctx is NULL");
    if (c->tally_dirty) return LP_OK;  // reallocated and zeroed on the next run
    int r = zero_tallies(c);
    if (r) return r;
    LP_CUDA(c, cudaStreamSynchronize(c->stream));
    return LP_OK;
}

int lp_get_geometry(lp_ctx *c, lp_geometry *out)
{
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_geometry: NULL argument");
    if (!c->have_grid) return fail(c, LP_ERR_STATE, "lp_get_geometry: tally grid not set");
    *out = c->geo;
    return LP_OK;
}

int lp_get_tallies(lp_ctx *c, lp_tallies *out)
{
    Phase phase("lp tally readback");
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_tallies: NULL argument");
    if (c->tally_dirty || !c->sft.p) return fail(c, LP_ERR_STATE, "lp_get_tallies: nothing has run");
    const lp_geometry &g = c->geo;
    LP_CUDA(c, c->h_sft.resize((size_t)g.sft_nx * g.sft_ny * 3));
    LP_CUDA(c, c->h_rtd.resize((size_t)g.dimR * g.dimAlpha * 3));
    LP_CUDA(c, c->h_rz.resize((size_t)g.rz_nr * g.rz_nz * 2));
    LP_CUDA(c, c->h_vox.resize((size_t)n_vox(c)));
    LP_CUDA(c, c->h_rbins.resize((size_t)c->n_rbins * 2));
    LP_CUDA(c, c->h_region.resize((size_t)c->n_media));
    LP_CUDA(c, c->h_det.resize(c->det_r.size()));
    LP_CUDA(c, fold_rz(c));
    cudaStream_t s = c->stream;
    LP_CUDA(c, cudaMemcpyAsync(c->h_sft.data(), c->sft.p, c->h_sft.size() * 8, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaMemcpyAsync(c->h_rtd.data(), c->rtd.p, c->h_rtd.size() * 8, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaMemcpyAsync(c->h_rz.data(), c->rz.p, c->h_rz.size() * 8, cudaMemcpyDeviceToHost, s));
    if (!c->h_vox.empty())
        LP_CUDA(c, cudaMemcpyAsync(c->h_vox.data(), c->vox.p, c->h_vox.size() * 8, cudaMemcpyDeviceToHost, s));
    if (!c->h_rbins.empty())
        LP_CUDA(c, cudaMemcpyAsync(c->h_rbins.data(), c->rbins.p, c->h_rbins.size() * 8, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaMemcpyAsync(c->h_region.data(), c->region.p, c->h_region.size() * 8, cudaMemcpyDeviceToHost, s));
    if (!c->h_det.empty())
        LP_CUDA(c, cudaMemcpyAsync(c->h_det.data(), c->det.p, c->h_det.size() * 8, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaMemcpyAsync(out->counters, c->counters.p, LP_NCOUNTERS * 8, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaStreamSynchronize(s));
    c->d2h_bytes = (int64_t)(c->h_sft.size() + c->h_rtd.size() + c->h_rz.size() + c->h_vox.size() +
                             c->h_rbins.size() + c->h_region.size() + c->h_det.size() + LP_NCOUNTERS) * 8;
    out->sft = c->h_sft.data();
    out->rtd = c->h_rtd.data();
    out->rz = c->h_rz.data();
    out->vox = c->h_vox.data();
    out->rbins = c->h_rbins.data();
    out->region = c->h_region.data();
    out->det = c->h_det.data();
    out->n_vox = (int64_t)c->h_vox.size();
    out->n_rbins = c->n_rbins;
    out->n_region = c->n_media;
    out->n_det = (int64_t)c->det_r.size() / 2;
    return LP_OK;
}

int lp_set_tallies(lp_ctx *c, const lp_tallies *in)
{
    if (!c || !in) return fail(c, LP_ERR_INVALID, "lp_set_tallies: NULL argument");
    if (!c->have_grid) return fail(c, LP_ERR_STATE, "lp_set_tallies: tally grid not set");
    const lp_geometry &g = c->geo;
    const int64_t D = (int64_t)c->det_r.size() / 2;
    if (in->n_vox != n_vox(c) || in->n_rbins != c->n_rbins || in->n_region != c->n_media || in->n_det != D)
        return fail(c, LP_ERR_INVALID,
                    "lp_set_tallies: layout differs from the context's (vox %lld/%lld, rbins %lld/%d, regions "
                    "%lld/%d, rings %lld/%lld)", (long long)in->n_vox, (long long)n_vox(c), (long long)in->n_rbins,
                    c->n_rbins, (long long)in->n_region, c->n_media, (long long)in->n_det, (long long)D);
    if (!in->sft || !in->rtd || !in->rz || !in->region || (in->n_vox && !in->vox) || (in->n_rbins && !in->rbins) ||
        (D && !in->det))
        return fail(c, LP_ERR_INVALID, "lp_set_tallies: NULL tally array");
    LP_CUDA(c, cudaSetDevice(c->device));
    if (c->tally_dirty) {
        int r = alloc_tallies(c);
        if (r) return r;
        r = zero_tallies(c);
        if (r) return r;
        c->tally_dirty = false;
    }
    LP_CUDA(c, clear_rz_copies(c));
    cudaStream_t s = c->stream;
    LP_CUDA(c, cudaMemcpyAsync(c->sft.p, in->sft, (size_t)g.sft_nx * g.sft_ny * 3 * 8, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->rtd.p, in->rtd, (size_t)g.dimR * g.dimAlpha * 3 * 8, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->rz.p, in->rz, (size_t)g.rz_nr * g.rz_nz * 2 * 8, cudaMemcpyHostToDevice, s));
    if (in->n_vox) LP_CUDA(c, cudaMemcpyAsync(c->vox.p, in->vox, (size_t)in->n_vox * 8, cudaMemcpyHostToDevice, s));
    if (in->n_rbins)
        LP_CUDA(c, cudaMemcpyAsync(c->rbins.p, in->rbins, (size_t)in->n_rbins * 2 * 8, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->region.p, in->region, (size_t)in->n_region * 8, cudaMemcpyHostToDevice, s));
    if (D) LP_CUDA(c, cudaMemcpyAsync(c->det.p, in->det, (size_t)D * 2 * 8, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(c->counters.p, in->counters, LP_NCOUNTERS * 8, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaStreamSynchronize(s));
    return LP_OK;
}

int lp_get_gradient_sums(lp_ctx *c, double *out, int64_t n)
{
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_gradient_sums: NULL argument");
    const int64_t want = (int64_t)(c->det_r.size() / 2) * c->n_media * 5;
    if (n != want) return fail(c, LP_ERR_INVALID, "lp_get_gradient_sums: %lld values, the layout has %lld",
                               (long long)n, (long long)want);
    if (!c->grad.p) return fail(c, LP_ERR_STATE, "lp_get_gradient_sums: nothing has run");
    if (n == 0) return LP_OK;
    LP_CUDA(c, cudaSetDevice(c->device));
    LP_CUDA(c, cudaMemcpyAsync(out, c->grad.p, (size_t)n * 8, cudaMemcpyDeviceToHost, c->stream));
    LP_CUDA(c, cudaStreamSynchronize(c->stream));
    return LP_OK;
}

int lp_set_gradient_sums(lp_ctx *c, const double *in, int64_t n)
{
    if (!c || !in) return fail(c, LP_ERR_INVALID, "lp_set_gradient_sums: NULL argument");
    const int64_t want = (int64_t)(c->det_r.size() / 2) * c->n_media * 5;
    if (n != want) return fail(c, LP_ERR_INVALID, "lp_set_gradient_sums: %lld values, the layout has %lld",
                               (long long)n, (long long)want);
    if (c->tally_dirty || !c->grad.p) return fail(c, LP_ERR_STATE, "lp_set_gradient_sums: set the tallies first");
    if (n == 0) return LP_OK;
    LP_CUDA(c, cudaSetDevice(c->device));
    LP_CUDA(c, cudaMemcpyAsync(c->grad.p, in, (size_t)n * 8, cudaMemcpyHostToDevice, c->stream));
    LP_CUDA(c, cudaStreamSynchronize(c->stream));
    return LP_OK;
}

int lp_get_exit_records(lp_ctx *c, float *out, int64_t n)
{
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_exit_records: NULL argument");
    if (n < 0 || n > c->exit_cap) return fail(c, LP_ERR_RANGE, "lp_get_exit_records: %lld > capacity", (long long)n);
    if (n == 0) return LP_OK;
    LP_CUDA(c, cudaMemcpyAsync(out, c->exit_rec.p, (size_t)n * 32, cudaMemcpyDeviceToHost, c->stream));
    LP_CUDA(c, cudaStreamSynchronize(c->stream));
    return LP_OK;
}

int lp_get_stats(lp_ctx *c, lp_stats *out)
{
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_stats: NULL argument");
    std::memset(out, 0, sizeof *out);
    out->n_tri = c->n_tri;
    out->n_nodes = (int64_t)c->bvh.node_a.size();
    out->bvh_depth = c->bvh.depth;
    out->nodes_smem = c->st_nodes_smem;
    out->tris_smem = c->st_tris_smem;
    out->smem_bytes = c->st_smem;
    out->blocks_per_sm = c->st_per_sm;
    out->grid = c->st_grid;
    out->block = lp::block_size();
    out->num_sms = c->num_sms;
    out->h2d_bytes = c->h2d_bytes;
    out->d2h_bytes = c->d2h_bytes;
    out->last_kernel_ms = c->last_ms;
    return LP_OK;
}

int lp_get_device_tallies(lp_ctx *c, lp_device_tallies *out)
{
    if (!c || !out) return fail(c, LP_ERR_INVALID, "lp_get_device_tallies: NULL argument");
    if (c->tally_dirty || !c->sft.p) return fail(c, LP_ERR_STATE, "lp_get_device_tallies: tallies not allocated yet");
    LP_CUDA(c, fold_rz(c));
    const lp_geometry &g = c->geo;
    out->sft = (uint64_t *)c->sft.p;
    out->rtd = (uint64_t *)c->rtd.p;
    out->rz = (uint64_t *)c->rz.p;
    out->vox = (uint64_t *)c->vox.p;
    out->rbins = (uint64_t *)c->rbins.p;
    out->region = (uint64_t *)c->region.p;
    out->det = (uint64_t *)c->det.p;
    out->counters = (uint64_t *)c->counters.p;
    out->n_sft = (int64_t)g.sft_nx * g.sft_ny * 3;
    out->n_rtd = (int64_t)g.dimR * g.dimAlpha * 3;
    out->n_rz = (int64_t)g.rz_nr * g.rz_nz * 2;
    out->n_vox = n_vox(c);
    out->n_rbins = (int64_t)c->n_rbins * 2;
    out->n_region = c->n_media;
    out->n_det = (int64_t)c->det_r.size();
    out->n_counters = LP_NCOUNTERS;
    out->stream = (void *)c->stream;
    out->grad = c->grad.p;
    out->n_grad = c->grad_on ? (int64_t)(c->det_r.size() / 2) * c->n_media * 5 : 0;
    return LP_OK;
}

int lp_fp32_peak(int device, double *tflops)
{
    if (!tflops) return fail(nullptr, LP_ERR_INVALID, "lp_fp32_peak: NULL argument");
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_fp32_peak");
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    *tflops = lp::fma_peak_tflops(sms);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_fp32_peak");
    return LP_OK;
}

int lp_debug_fail_allocation(int64_t after)
{
    g_alloc_countdown.store(after < 0 ? -1 : after);
    return LP_OK;
}

int lp_debug_fail_launch(int64_t after)
{
    g_launch_countdown.store(after < 0 ? -1 : after);
    return LP_OK;
}

int lp_l2_atomic_peak(int device, double *per_s)
{
    if (!per_s) return fail(nullptr, LP_ERR_INVALID, "lp_l2_atomic_peak: NULL argument");
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_l2_atomic_peak");
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    *per_s = lp::red_peak_per_s(sms);
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_l2_atomic_peak");
    return LP_OK;
}

int lp_last_kernel_ms(lp_ctx *c, float *ms)
{
    if (!c || !ms) return fail(c, LP_ERR_INVALID, "lp_last_kernel_ms: NULL argument");
    *ms = c->last_ms;
    return LP_OK;
}

int lp_query_triangles(lp_ctx *c, int64_t n, const float *orig, const float *dir, const int32_t *ref_tri,
                       const float *t_max, int32_t *id_out, float *t_out)
{
    if (!c || !orig || !dir || !ref_tri || !t_max || !id_out || !t_out)
        return fail(c, LP_ERR_INVALID, "lp_query_triangles: NULL argument");
    if (!c->have_mesh) return fail(c, LP_ERR_STATE, "lp_query_triangles: no mesh");
    if (n <= 0) return LP_OK;
    LP_CUDA(c, cudaSetDevice(c->device));
    int ur = upload_mesh(c);
    if (ur) return ur;
    if (c->grid_dirty && (ur = build_safety_grid(c))) return ur;
    DevBuf<float> o, d, tm, to;
    DevBuf<int32_t> rf, io;
    LP_CUDA(c, o.ensure((size_t)n * 3));
    LP_CUDA(c, d.ensure((size_t)n * 3));
    LP_CUDA(c, tm.ensure((size_t)n));
    LP_CUDA(c, to.ensure((size_t)n));
    LP_CUDA(c, rf.ensure((size_t)n));
    LP_CUDA(c, io.ensure((size_t)n));
    cudaStream_t s = c->stream;
    LP_CUDA(c, cudaMemcpyAsync(o.p, orig, (size_t)n * 12, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(d.p, dir, (size_t)n * 12, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(tm.p, t_max, (size_t)n * 4, cudaMemcpyHostToDevice, s));
    LP_CUDA(c, cudaMemcpyAsync(rf.p, ref_tri, (size_t)n * 4, cudaMemcpyHostToDevice, s));
    int nodes_smem, tris_smem;
    smem_plan(c, c->smem_budget, nodes_smem, tris_smem);
    KParams P;
    fill_params(c, P, 0, 0, nodes_smem, tris_smem);
    P.tri_eps = 0.0f;   // the reference's test: these queries are checked against its scan
    const int smem = lp::smem_bytes(nodes_smem, tris_smem);
    LP_CUDA(c, lp::launch_query(P, smem, n, o.p, d.p, rf.p, tm.p, io.p, to.p, s));
    LP_CUDA(c, cudaMemcpyAsync(id_out, io.p, (size_t)n * 4, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaMemcpyAsync(t_out, to.p, (size_t)n * 4, cudaMemcpyDeviceToHost, s));
    LP_CUDA(c, cudaStreamSynchronize(s));
    o.release(); d.release(); tm.release(); to.release(); rf.release(); io.release();
    return LP_OK;
}

int lp_exact_ops(int device, int32_t op, int64_t n, const float *a, const float *b, float *out)
{
    if (op < 0 || op > 2 || n < 0 || !a || !out || (op == 2 && !b))
        return fail(nullptr, LP_ERR_INVALID, "lp_exact_ops: bad argument");
    if (n == 0) return LP_OK;
    cudaError_t e = cudaSetDevice(device);
    DevBuf<float> da, db, dr;
    if (e == cudaSuccess) e = da.ensure((size_t)n);
    if (e == cudaSuccess) e = db.ensure((size_t)n);
    if (e == cudaSuccess) e = dr.ensure((size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(da.p, a, (size_t)n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && op == 2) e = cudaMemcpy(db.p, b, (size_t)n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = lp::launch_exact_ops(op, n, da.p, db.p, dr.p, 0);
    if (e == cudaSuccess) e = cudaMemcpy(out, dr.p, (size_t)n * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_exact_ops");
    return LP_OK;
}

int lp_philox_blocks(int device, const uint32_t *ctr, const uint32_t *key, int64_t n, uint32_t *out)
{
    if (!ctr || !key || !out || n < 0) return fail(nullptr, LP_ERR_INVALID, "lp_philox_blocks: bad argument");
    if (n == 0) return LP_OK;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_philox_blocks");
    DevBuf<uint32_t> b;
    if ((e = b.ensure((size_t)n * 4)) != cudaSuccess) return cuda_fail(nullptr, e, "lp_philox_blocks: alloc");
    e = lp::launch_philox(ctr, key, n, b.p, 0);
    if (e == cudaSuccess) e = cudaMemcpy(out, b.p, (size_t)n * 16, cudaMemcpyDeviceToHost);
    b.release();
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "lp_philox_blocks");
    return LP_OK;
}

}  // extern "C"

// ============================================================ batches
namespace lp {
cudaError_t launch_batch(int config, bool grad, const BatchParams &B, int grid, cudaStream_t s);
cudaError_t batch_occupancy(int config, bool grad, int *blocks_per_sm);
int batch_config_count();
int batch_config_info(int config, int *block, int *min_blocks, int *stack);
}  // namespace lp

struct lp_batch {
    int device = 0;
    int num_sms = 148;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::string err;
    std::vector<lp_ctx *> ctx;
    std::vector<lp_instance> inst;
    // elements of each tally per instance
    size_t n_sft = 0, n_rtd = 0, n_rz = 0, n_vox = 0, n_rbins = 0, n_det = 0;
    DevBuf<unsigned long long> sft, rtd, rz, vox, rbins, region, det, counters, claimed;
    DevBuf<double> grad;
    DevBuf<Medium> media;
    DevBuf<KParams> params;
    DevBuf<int64_t> cum;       // BatchParams::cum
    int64_t n_batch = 0;       // photons of the batch launch
    bool grad_on = false;
    int config = -1;
    int grid = 0;
    uint32_t lane_mask = 0xffffffffu;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    // Instances of at least plain_min photons (plain_min > 0) run as a persistent transport
    // launch of their own inside the graph, with their context's shared-memory plan; the
    // batch kernel sees them with no photons.  The batch kernel pays for its per-warp
    // instance switching on every photon, a launch of its own only once (its drain).  Equal
    // instances, shared / own, ms: abdomen 2 x 1e6 128 / 141, 2 x 3e6 351 / 342, 2 x 1e7 1136 /
    // 1049, 8 x 1e6 467 / 572, 8 x 3e6 1387 / 1374; slab 2 x 1e6 178 / 178, 2 x 3e6 503 / 472, 8 x
    // 1e6 665 / 713.  So they meet at 1e6 to 3e6 photons; the default is the callers' to raise.
    struct PlainLaunch {
        KParams P;
        int grid = 0, smem = 0;
    };
    int64_t plain_min = int64_t(1) << 20;
    std::vector<PlainLaunch> plain;
    DevBuf<unsigned long long> plain_work;
    // copies of the r-z images (KParams::rz_part), zero between launches: [instance][copy] of
    // the batch launch, and one set that the plain launches use in turn
    DevBuf<unsigned long long> rz_part, plain_rz_part;
    bool rz_pending = false;   // rz_part holds deposits of a launch whose fold failed
    // The r-z and voxel tallies (the atomic targets of every scatter event) of the
    // instances with a launch of their own sit in buffers of their own, like a context's: as
    // slices of the batch's large arrays the same launch measured up to 15 % slower (before the
    // r-z deposits went to copies).
    struct OwnTallies {
        DevBuf<unsigned long long> rz, vox;
    };
    std::vector<std::unique_ptr<OwnTallies>> own;
    std::vector<uint64_t> mesh_gen;   // lp_ctx::mesh_gen of each context in the parameters
    lp_geometry geo{};                // the tally layout that the buffers are for
    int32_t vox_dim[3] = {0, 0, 0};
    std::vector<unsigned long long *> rz_of, vox_of;   // per instance: where its r-z, voxel tallies are
    float last_ms = 0.0f;
    std::vector<uint64_t> h_sft, h_rtd, h_rz, h_vox, h_rbins, h_region, h_det, h_cnt;
    std::vector<double> h_grad;
    GradOut gout;
};

namespace {

int bfail(lp_batch *b, int code, const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (b) b->err = buf;
    g_thread_error = buf;
    return code;
}

#define LP_BCUDA(b, call)                                                        \
    do {                                                                         \
        cudaError_t _e = (call);                                                 \
        if (_e != cudaSuccess) {                                                 \
            cudaGetLastError(); /* as cuda_fail */                               \
            return bfail(b, LP_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(_e)); \
        }                                                                        \
    } while (0)

void drop_graph(lp_batch *b)
{
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

size_t grad_stride(const lp_batch *b) { return std::max<size_t>(b->n_det, 1) * lp::kBatchMedia * 5; }

// After a failure between the old and the new instances: buffers may have been replaced that
// the parameters on the device still point to, so the batch has no instances until the next
// lp_batch_set_instances.
void drop_instances(lp_batch *b)
{
    drop_graph(b);
    b->inst.clear();
    b->plain.clear();
}

// The tallies and parameters of I instances.
int alloc_instances(lp_batch *b, size_t I)
{
    const size_t J = std::max<size_t>(I, 1);
    LP_BCUDA(b, b->sft.ensure(J * b->n_sft));
    LP_BCUDA(b, b->rtd.ensure(J * b->n_rtd));
    LP_BCUDA(b, b->rz.ensure(J * b->n_rz));
    const int copies = rz_copies(b->n_rz, J);
    if (copies > 1) {
        LP_BCUDA(b, b->rz_part.ensure(J * copies * b->n_rz));
        LP_BCUDA(b, cudaMemsetAsync(b->rz_part.p, 0, J * copies * b->n_rz * 8, b->stream));
    }
    LP_BCUDA(b, b->vox.ensure(J * std::max<size_t>(b->n_vox, 1)));
    LP_BCUDA(b, b->rbins.ensure(J * std::max<size_t>(b->n_rbins, 1)));
    LP_BCUDA(b, b->region.ensure(J * lp::kBatchMedia));
    LP_BCUDA(b, b->det.ensure(J * std::max<size_t>(b->n_det, 1) * 2));
    LP_BCUDA(b, b->counters.ensure(J * LP_NCOUNTERS));
    LP_BCUDA(b, b->grad.ensure(J * grad_stride(b)));
    LP_BCUDA(b, b->claimed.ensure(J));
    LP_BCUDA(b, b->cum.ensure(J + 1));
    LP_BCUDA(b, b->media.ensure(J * lp::kBatchMedia));
    LP_BCUDA(b, b->params.ensure(J));
    return LP_OK;
}

// Per-instance parameters: the context's (mesh, source, tally layout, run parameters)
// with the instance's media, photon range and tally slices.
int fill_instances(lp_batch *b)
{
    const size_t I = b->inst.size();
    LP_BCUDA(b, cudaSetDevice(b->device));
    // the contexts may have been changed since lp_batch_create
    b->mesh_gen.assign(b->ctx.size(), 0);
    for (size_t k = 0; I > 0 && k < b->ctx.size(); ++k) {
        lp_ctx *c = b->ctx[k];
        if (!c->have_mesh || !c->have_source || !c->have_grid)
            return bfail(b, LP_ERR_STATE, "batch: context %d has no mesh, source or tally grid", (int)k);
        int r = upload_mesh(c);
        if (!r && c->grid_dirty) r = build_safety_grid(c);
        if (r) return bfail(b, r, "batch: context %d: %s", (int)k, c->err.c_str());
        if (std::memcmp(&c->geo, &b->geo, sizeof b->geo) != 0 || (size_t)c->n_rbins * 2 != b->n_rbins ||
            c->det_r.size() / 2 != b->n_det || std::memcmp(c->vox_n, b->vox_dim, sizeof b->vox_dim) != 0)
            return bfail(b, LP_ERR_STATE, "batch: the tally layout of context %d is not the one of lp_batch_create",
                         (int)k);
        b->mesh_gen[k] = c->mesh_gen;
    }
    for (size_t i = 0; i < I; ++i)
        if (b->ctx[b->inst[i].context]->max_region >= b->inst[i].n_media)
            return bfail(b, LP_ERR_INVALID, "batch: instance %d: mesh uses region %d", (int)i,
                         b->ctx[b->inst[i].context]->max_region);
    std::vector<KParams> P(I);
    std::vector<Medium> M(I * lp::kBatchMedia);
    b->plain.clear();
    b->rz_of.assign(I, nullptr);
    b->vox_of.assign(I, nullptr);
    for (size_t i = 0; i < I; ++i) {
        const lp_instance &in = b->inst[i];
        lp_ctx *c = b->ctx[in.context];
        KParams &p = P[i];
        fill_params(c, p, in.first, in.n_photons, 0, 0);
        std::vector<Medium> m;
        media_table(in.nmuasg, in.n_media, m);
        std::copy(m.begin(), m.end(), M.begin() + i * lp::kBatchMedia);
        p.media = b->media.p + i * lp::kBatchMedia;
        p.n_media = in.n_media;
        p.Rsp = rspecular(in.nmuasg, in.n_media);
        p.w0 = 1.0f - p.Rsp;
        p.exitScale = (c->compat & LP_COMPAT_EXIT_RSP) ? (1 - p.Rsp) : 1.0f;
        const float s = c->fiber_na / in.nmuasg[0];
        p.src_cos_max = s < 1.0f ? std::sqrt(1.0f - s * s) : 0.0f;
        p.sft = b->sft.p + i * b->n_sft;
        p.rtd = b->rtd.p + i * b->n_rtd;
        p.rz = b->rz.p + i * b->n_rz;
        p.vox = b->vox.p + i * std::max<size_t>(b->n_vox, 1);
        p.rbins = b->rbins.p + i * std::max<size_t>(b->n_rbins, 1);
        p.region = b->region.p + i * lp::kBatchMedia;
        p.det = b->det.p + i * std::max<size_t>(b->n_det, 1) * 2;
        p.counters = b->counters.p + i * LP_NCOUNTERS;
        p.grad = b->grad_on ? b->grad.p + i * grad_stride(b) : nullptr;
        p.exit_rec = nullptr;
        p.exit_cap = 0;
        p.work = nullptr;
        const int copies = rz_copies(b->n_rz, I), plain_copies = rz_copies(b->n_rz);
        p.rz_part = copies > 1 ? b->rz_part.p + i * copies * b->n_rz : p.rz;
        p.rz_stride = (int64_t)b->n_rz;
        p.rz_mask = (uint32_t)(copies - 1);
        if (b->plain_min > 0 && in.n_photons >= b->plain_min) {
            const size_t k = b->plain.size();
            if (b->own.size() <= k) b->own.push_back(std::unique_ptr<lp_batch::OwnTallies>(new lp_batch::OwnTallies));
            LP_BCUDA(b, b->own[k]->rz.ensure(std::max<size_t>(b->n_rz, 1)));
            LP_BCUDA(b, b->own[k]->vox.ensure(std::max<size_t>(b->n_vox, 1)));
            p.rz = b->own[k]->rz.p;
            p.vox = b->own[k]->vox.p;
            lp_batch::PlainLaunch L;
            L.P = p;
            if (plain_copies > 1 && !b->plain_rz_part.p) {
                LP_BCUDA(b, b->plain_rz_part.ensure(b->n_rz * plain_copies));
                LP_BCUDA(b, cudaMemsetAsync(b->plain_rz_part.p, 0, b->n_rz * plain_copies * 8, b->stream));
            }
            L.P.rz_part = plain_copies > 1 ? b->plain_rz_part.p : p.rz;
            L.P.rz_mask = (uint32_t)(plain_copies - 1);
            int ns = 0, ts = 0;
            smem_plan(c, c->smem_budget, ns, ts);
            L.P.nodes_smem = ns;
            L.P.tris_smem = ts;
            L.smem = lp::smem_bytes(ns, ts);
            b->plain.push_back(L);
            p.n = 0;
        }
        b->rz_of[i] = p.rz;
        b->vox_of[i] = p.vox;
    }
    b->own.resize(b->plain.size());
    if (!b->plain.empty()) {
        LP_BCUDA(b, b->plain_work.ensure(b->plain.size()));
        for (size_t k = 0; k < b->plain.size(); ++k) b->plain[k].P.work = b->plain_work.p + k;
    }
    std::vector<int64_t> cum(I + 1, 0);
    for (size_t i = 0; i < I; ++i) cum[i + 1] = cum[i] + P[i].n;
    // the graph's launch was planned for the photons it had then
    if (b->n_batch != cum[I]) drop_graph(b);
    b->n_batch = cum[I];
    if (I) {
        LP_BCUDA(b, cudaMemcpyAsync(b->cum.p, cum.data(), (I + 1) * 8, cudaMemcpyHostToDevice, b->stream));
        LP_BCUDA(b, cudaMemcpyAsync(b->params.p, P.data(), I * sizeof(KParams), cudaMemcpyHostToDevice, b->stream));
        LP_BCUDA(b, cudaMemcpyAsync(b->media.p, M.data(), M.size() * sizeof(Medium), cudaMemcpyHostToDevice,
                                    b->stream));
        LP_BCUDA(b, cudaStreamSynchronize(b->stream));
    }
    return LP_OK;
}

int upload_instances(lp_batch *b)
{
    const int r = fill_instances(b);
    if (r) drop_instances(b);
    return r;
}

// A context that got another mesh or cell grid since the parameters were formed has replaced
// what they point to: they are formed again.
int refresh_instances(lp_batch *b)
{
    bool same = true;
    for (size_t k = 0; k < b->ctx.size(); ++k) same = same && b->ctx[k]->mesh_gen == b->mesh_gen[k];
    if (same) return LP_OK;
    drop_graph(b);
    return upload_instances(b);
}

// Zero the tallies and claim counters of all instances (enqueued on the batch stream).
int enqueue_zero(lp_batch *b)
{
    const size_t I = b->inst.size();
    cudaStream_t s = b->stream;
    LP_BCUDA(b, cudaMemsetAsync(b->sft.p, 0, I * b->n_sft * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->rtd.p, 0, I * b->n_rtd * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->rz.p, 0, I * b->n_rz * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->vox.p, 0, I * std::max<size_t>(b->n_vox, 1) * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->rbins.p, 0, I * std::max<size_t>(b->n_rbins, 1) * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->region.p, 0, I * lp::kBatchMedia * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->det.p, 0, I * std::max<size_t>(b->n_det, 1) * 2 * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->counters.p, 0, I * LP_NCOUNTERS * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->grad.p, 0, I * grad_stride(b) * 8, s));
    LP_BCUDA(b, cudaMemsetAsync(b->claimed.p, 0, I * 8, s));
    if (!b->plain.empty()) LP_BCUDA(b, cudaMemsetAsync(b->plain_work.p, 0, b->plain.size() * 8, s));
    for (size_t k = 0; k < b->plain.size(); ++k) {
        LP_BCUDA(b, cudaMemsetAsync(b->own[k]->rz.p, 0, b->n_rz * 8, s));
        if (b->n_vox) LP_BCUDA(b, cudaMemsetAsync(b->own[k]->vox.p, 0, b->n_vox * 8, s));
    }
    return LP_OK;
}

// Grids of the plain launches: SMs x resident blocks of the transport kernel with each
// launch's shared memory (queried outside stream capture).
int prepare_plain(lp_batch *b)
{
    for (lp_batch::PlainLaunch &L : b->plain) {
        int per_sm = 0;
        LP_BCUDA(b, b->grad_on ? lp::transport_occupancy_fast_grad(L.smem, &per_sm)
                               : lp::transport_occupancy_fast(L.smem, &per_sm));
        if (per_sm < 1) return bfail(b, LP_ERR_CUDA, "batch: transport kernel does not fit on an SM");
        lp::plan_launch(L.P.n, lp::block_size(), b->num_sms, per_sm, L.grid, L.P.lane_mask, L.P.few_blocks);
    }
    return LP_OK;
}

int enqueue_plain(lp_batch *b)
{
    const int copies = rz_copies(b->n_rz);
    for (const lp_batch::PlainLaunch &L : b->plain) {
        LP_BCUDA(b, lp::launch_transport_fast(L.P, L.grid, L.smem, b->stream));
        if (copies > 1)
            LP_BCUDA(b, lp::launch_fold(L.P.rz, L.P.rz_part, copies, (int64_t)b->n_rz, 1, b->stream));
    }
    return LP_OK;
}

// Grid of the persistent launch: SMs x resident blocks of `config` (queried outside
// stream capture).
int prepare_grid(lp_batch *b, int config)
{
    int per_sm = 0;
    LP_BCUDA(b, lp::batch_occupancy(config, b->grad_on, &per_sm));
    if (per_sm < 1) return bfail(b, LP_ERR_CUDA, "batch configuration %d does not fit on an SM", config);
    int block, minb, stack;
    lp::batch_config_info(config, &block, &minb, &stack);
    uint32_t few;
    lp::plan_launch(b->n_batch, block, b->num_sms, per_sm, b->grid, b->lane_mask, few);
    return LP_OK;
}

int enqueue_launch(lp_batch *b, int config)
{
    lp::BatchParams B;
    B.inst = b->params.p;
    B.claimed = b->claimed.p;
    B.cum = b->cum.p;
    B.n_inst = (int32_t)b->inst.size();
    B.lane_mask = b->lane_mask;
    LP_BCUDA(b, launch_unless_injected([&] { return lp::launch_batch(config, b->grad_on, B, b->grid, b->stream); }));
    const int copies = rz_copies(b->n_rz, b->inst.size());
    if (copies > 1)
        LP_BCUDA(b, launch_unless_injected([&] {
            return lp::launch_fold(b->rz.p, b->rz_part.p, copies, (int64_t)b->n_rz, (int64_t)b->inst.size(), b->stream);
        }));
    return LP_OK;
}

bool config_eligible(const lp_batch *b, int config)
{
    int block, minb, stack;
    if (lp::batch_config_info(config, &block, &minb, &stack)) return false;
    for (const lp_ctx *c : b->ctx)
        if (c->bvh.depth >= stack) return false;
    return true;
}

int64_t total_photons(const std::vector<lp_instance> &v)
{
    int64_t t = 0;
    for (const lp_instance &i : v) t += i.n_photons;
    return t;
}

// Drops deposits that a failed fold left in the copies of the r-z images (every launch zeroes
// the tallies, so they belong to none).
int clear_rz_copies(lp_batch *b)
{
    if (!b->rz_pending) return LP_OK;
    LP_BCUDA(b, cudaMemsetAsync(b->rz_part.p, 0, b->rz_part.n * 8, b->stream));
    b->rz_pending = false;
    return LP_OK;
}

// One direct (ungraphed) launch of `config`; device milliseconds of the kernel.
int timed_launch(lp_batch *b, int config, float *ms)
{
    int r = prepare_grid(b, config);
    if (r) return r;
    if ((r = clear_rz_copies(b))) return r;
    if ((r = enqueue_zero(b))) return r;
    LP_BCUDA(b, cudaEventRecord(b->ev0, b->stream));
    b->rz_pending = true;
    if ((r = enqueue_launch(b, config))) return r;
    b->rz_pending = false;
    LP_BCUDA(b, cudaEventRecord(b->ev1, b->stream));
    LP_BCUDA(b, cudaEventSynchronize(b->ev1));
    LP_BCUDA(b, cudaEventElapsedTime(ms, b->ev0, b->ev1));
    return LP_OK;
}

// Times every eligible configuration on the instances as they are set: the fastest one's index
// and the nanoseconds per photon of each (-1: not eligible).
int time_configs(lp_batch *b, int &chosen, double *ns_per_photon)
{
    const double n_trial = (double)std::max<int64_t>(total_photons(b->inst), 1);
    double best_ns = 0.0;
    bool warmed = false;
    int r;
    for (int k = 0; k < lp::batch_config_count(); ++k) {
        double ns = -1.0;
        if (config_eligible(b, k)) {
            float ms = 0.0f;
            if (!warmed) {   // first launch of the process pays for module loading
                if ((r = timed_launch(b, k, &ms))) return r;
                warmed = true;
            }
            if ((r = timed_launch(b, k, &ms))) return r;
            ns = (double)ms * 1e6 / n_trial;
            if (chosen < 0 || ns < best_ns) {
                chosen = k;
                best_ns = ns;
            }
        }
        if (ns_per_photon) ns_per_photon[k] = ns;
    }
    return LP_OK;
}

int copy_counts(lp_batch *b)
{
    const size_t I = b->inst.size();
    b->h_det.resize(I * std::max<size_t>(b->n_det, 1) * 2);
    b->h_cnt.resize(I * LP_NCOUNTERS);
    LP_BCUDA(b, cudaMemcpyAsync(b->h_det.data(), b->det.p, b->h_det.size() * 8, cudaMemcpyDeviceToHost, b->stream));
    LP_BCUDA(b, cudaMemcpyAsync(b->h_cnt.data(), b->counters.p, b->h_cnt.size() * 8, cudaMemcpyDeviceToHost,
                                b->stream));
    LP_BCUDA(b, cudaStreamSynchronize(b->stream));
    return LP_OK;
}

}  // namespace

extern "C" {

int lp_batch_config_count(void) { return lp::batch_config_count(); }

int lp_batch_config_info(int32_t config, int32_t *block, int32_t *min_blocks, int32_t *stack)
{
    int a, m, s;
    if (!block || !min_blocks || !stack || lp::batch_config_info(config, &a, &m, &s))
        return fail(nullptr, LP_ERR_INVALID, "lp_batch_config_info: configuration %d", config);
    *block = a;
    *min_blocks = m;
    *stack = s;
    return LP_OK;
}

const char *lp_batch_last_error(const lp_batch *b)
{
    if (b) return b->err.c_str();
    return g_thread_error.c_str();
}

int lp_batch_create(lp_batch **out, int32_t n_ctx, lp_ctx *const *ctxs)
{
    if (!out || n_ctx < 1 || !ctxs) return fail(nullptr, LP_ERR_INVALID, "lp_batch_create: no contexts");
    *out = nullptr;
    for (int i = 0; i < n_ctx; ++i)
        if (!ctxs[i]) return fail(nullptr, LP_ERR_INVALID, "lp_batch_create: context %d is NULL", i);
    const lp_ctx *c0 = ctxs[0];
    for (int i = 0; i < n_ctx; ++i) {
        lp_ctx *c = ctxs[i];
        if (c->device != c0->device) return fail(nullptr, LP_ERR_INVALID, "lp_batch_create: contexts on two devices");
        int r = upload(c);
        if (r) return fail(nullptr, r, "lp_batch_create: context %d: %s", i, c->err.c_str());
        const lp_geometry &g = c->geo, &g0 = c0->geo;
        if (std::memcmp(&g, &g0, sizeof g) != 0 || c->n_rbins != c0->n_rbins || c->det_r != c0->det_r ||
            std::memcmp(c->vox_n, c0->vox_n, sizeof c->vox_n) != 0)
            return fail(nullptr, LP_ERR_INVALID, "lp_batch_create: context %d has another tally layout", i);
    }
    lp_batch *b = new lp_batch;
    b->device = c0->device;
    b->num_sms = c0->num_sms;
    b->ctx.assign(ctxs, ctxs + n_ctx);
    const lp_geometry &g = c0->geo;
    b->n_sft = (size_t)g.sft_nx * g.sft_ny * 3;
    b->n_rtd = (size_t)g.dimR * g.dimAlpha * 3;
    b->n_rz = (size_t)g.rz_nr * g.rz_nz * 2;
    b->n_vox = (size_t)n_vox(c0);
    b->geo = g;
    std::memcpy(b->vox_dim, c0->vox_n, sizeof b->vox_dim);
    b->n_rbins = (size_t)c0->n_rbins * 2;
    b->n_det = c0->det_r.size() / 2;
    cudaError_t e = cudaSetDevice(b->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreate(&b->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&b->ev1);
    if (e != cudaSuccess) {
        int r = cuda_fail(nullptr, e, "lp_batch_create");
        lp_batch_destroy(b);
        return r;
    }
    *out = b;
    return LP_OK;
}

void lp_batch_destroy(lp_batch *b)
{
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    drop_graph(b);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

int lp_batch_set_instances(lp_batch *b, int32_t n_inst, const lp_instance *in)
{
    if (!b || n_inst < 0 || (n_inst > 0 && !in)) return bfail(b, LP_ERR_INVALID, "lp_batch_set_instances: bad argument");
    for (int i = 0; i < n_inst; ++i) {
        const lp_instance &x = in[i];
        if (x.context < 0 || x.context >= (int)b->ctx.size())
            return bfail(b, LP_ERR_INVALID, "lp_batch_set_instances: instance %d: context %d", i, x.context);
        if (x.n_media < 1 || x.n_media > LP_BATCH_MAX_MEDIA)
            return bfail(b, LP_ERR_RANGE, "lp_batch_set_instances: instance %d: %d regions (1..%d)", i, x.n_media,
                         LP_BATCH_MAX_MEDIA);
        if (b->ctx[x.context]->max_region >= x.n_media)
            return bfail(b, LP_ERR_INVALID, "lp_batch_set_instances: instance %d: mesh uses region %d", i,
                         b->ctx[x.context]->max_region);
        if (x.n_photons < 0 || x.first < 0)
            return bfail(b, LP_ERR_INVALID, "lp_batch_set_instances: instance %d: negative photon range", i);
        if (x.n_photons > lp::kMaxLaunchPhotons)
            return bfail(b, LP_ERR_RANGE, "lp_batch_set_instances: instance %d: more than 2^31 photons", i);
        for (int k = 0; k < 4 * x.n_media; ++k)
            if (!std::isfinite(x.nmuasg[k]))
                return bfail(b, LP_ERR_INVALID, "lp_batch_set_instances: instance %d: non-finite media", i);
    }
    LP_BCUDA(b, cudaSetDevice(b->device));
    const size_t I = (size_t)n_inst;
    if (I != b->inst.size() || !b->params.p) {
        drop_graph(b);
        const int r = alloc_instances(b, I);
        if (r) {
            drop_instances(b);
            return r;
        }
    }
    b->inst.assign(in, in + n_inst);
    // the plain launches hold their parameters by value in the graph
    const bool had_plain = !b->plain.empty();
    const int r = upload_instances(b);
    if (had_plain || !b->plain.empty()) drop_graph(b);
    return r;
}

int lp_batch_set_plain_threshold(lp_batch *b, int64_t photons)
{
    if (!b) return fail(nullptr, LP_ERR_INVALID, "lp_batch_set_plain_threshold: batch is NULL");
    if (photons == b->plain_min) return LP_OK;
    b->plain_min = photons;
    drop_graph(b);
    if (b->inst.empty()) return LP_OK;
    LP_BCUDA(b, cudaSetDevice(b->device));
    return upload_instances(b);
}

int lp_batch_plain_count(const lp_batch *b, int32_t *count)
{
    if (!b || !count) return fail(nullptr, LP_ERR_INVALID, "lp_batch_plain_count: NULL argument");
    *count = (int32_t)b->plain.size();
    return LP_OK;
}

int lp_batch_set_gradient(lp_batch *b, int enable)
{
    if (!b) return fail(nullptr, LP_ERR_INVALID, "lp_batch_set_gradient: batch is NULL");
    if ((enable != 0) == b->grad_on) return LP_OK;
    b->grad_on = enable != 0;
    drop_graph(b);
    return upload_instances(b);
}

int lp_batch_set_config(lp_batch *b, int32_t config)
{
    if (!b) return fail(nullptr, LP_ERR_INVALID, "lp_batch_set_config: batch is NULL");
    if (config < -1 || config >= lp::batch_config_count())
        return bfail(b, LP_ERR_INVALID, "lp_batch_set_config: configuration %d", config);
    if (config >= 0 && !config_eligible(b, config))
        return bfail(b, LP_ERR_RANGE, "lp_batch_set_config: configuration %d: traversal stack below BVH depth", config);
    if (config != b->config) drop_graph(b);
    b->config = config;
    return LP_OK;
}

int lp_batch_autotune(lp_batch *b, int64_t photons, int32_t *best, double *ns_per_photon)
{
    if (!b) return fail(nullptr, LP_ERR_INVALID, "lp_batch_autotune: batch is NULL");
    if (b->inst.empty()) return bfail(b, LP_ERR_STATE, "lp_batch_autotune: no instances");
    LP_BCUDA(b, cudaSetDevice(b->device));
    const std::vector<lp_instance> saved = b->inst;
    const int64_t total = std::max<int64_t>(total_photons(saved), 1);
    const double scale = photons > 0 ? std::min(1.0, (double)photons / (double)total) : 1.0;
    std::vector<lp_instance> trial = saved;
    for (lp_instance &x : trial)
        if (x.n_photons > 0) x.n_photons = std::max<int64_t>(std::min<int64_t>(x.n_photons, 32), (int64_t)(x.n_photons * scale));
    int r = lp_batch_set_instances(b, (int32_t)trial.size(), trial.data());
    int chosen = -1;
    if (!r) r = time_configs(b, chosen, ns_per_photon);
    // the caller's budgets are put back whatever the trials came to
    const std::string err = b->err;
    const int back = lp_batch_set_instances(b, (int32_t)saved.size(), saved.data());
    if (r) return bfail(b, r, "%s", err.c_str());
    if (back) return back;
    if (chosen < 0) return bfail(b, LP_ERR_RANGE, "lp_batch_autotune: no configuration fits these meshes");
    drop_graph(b);
    b->config = chosen;
    if (best) *best = chosen;
    return LP_OK;
}

int lp_batch_run(lp_batch *b)
{
    Phase phase("lp batch graph launch");
    if (!b) return fail(nullptr, LP_ERR_INVALID, "lp_batch_run: batch is NULL");
    if (b->inst.empty()) return LP_OK;
    LP_BCUDA(b, cudaSetDevice(b->device));
    int r;
    if ((r = refresh_instances(b))) return r;
    if (b->config >= 0 && !config_eligible(b, b->config)) {   // a deeper tree since it was chosen
        drop_graph(b);
        b->config = -1;
    }
    if (b->config < 0) {
        int32_t best;
        if ((r = lp_batch_autotune(b, 4000000, &best, nullptr))) return r;
    }
    if (!b->exec) {
        // one graph: zero every instance's tallies and counters, the plain launches of
        // the large instances, then the persistent batch launch
        if ((r = prepare_grid(b, b->config))) return r;
        if ((r = prepare_plain(b))) return r;
        LP_BCUDA(b, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        r = enqueue_zero(b);
        if (!r) r = enqueue_plain(b);
        if (!r) r = enqueue_launch(b, b->config);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(b->stream, &g);
        if (r || e != cudaSuccess) {
            cudaGetLastError();   // as cuda_fail
            if (g) cudaGraphDestroy(g);
            return r ? r : bfail(b, LP_ERR_CUDA, "lp_batch_run: capture: %s", cudaGetErrorString(e));
        }
        b->graph = g;
        LP_BCUDA(b, cudaGraphInstantiate(&b->exec, b->graph, 0));
    }
    if ((r = clear_rz_copies(b))) return r;
    LP_BCUDA(b, cudaEventRecord(b->ev0, b->stream));
    LP_BCUDA(b, cudaGraphLaunch(b->exec, b->stream));
    LP_BCUDA(b, cudaEventRecord(b->ev1, b->stream));
    LP_BCUDA(b, cudaEventSynchronize(b->ev1));
    LP_BCUDA(b, cudaEventElapsedTime(&b->last_ms, b->ev0, b->ev1));
    return LP_OK;
}

int lp_batch_last_ms(const lp_batch *b, float *ms)
{
    if (!b || !ms) return fail(nullptr, LP_ERR_INVALID, "lp_batch_last_ms: NULL argument");
    *ms = b->last_ms;
    return LP_OK;
}

int lp_batch_ring_signals(lp_batch *b, double *signal, double *rel_err)
{
    if (!b || !signal) return fail(nullptr, LP_ERR_INVALID, "lp_batch_ring_signals: NULL argument");
    int r = copy_counts(b);
    if (r) return r;
    const size_t D = b->n_det, DD = std::max<size_t>(D, 1);
    for (size_t i = 0; i < b->inst.size(); ++i) {
        const double N = (double)b->h_cnt[i * LP_NCOUNTERS + LP_C_PHOTONS];
        for (size_t d = 0; d < D; ++d) {
            const double s1 = (double)b->h_det[(i * DD + d) * 2] / LP_FIX_ONE;
            const double s2 = (double)b->h_det[(i * DD + d) * 2 + 1] / LP_FIX_ONE;
            const double m = N > 0 ? s1 / N : 0.0;
            signal[i * D + d] = m;
            if (rel_err) {
                const double se = N > 1 ? std::sqrt(std::max(s2 / N - m * m, 0.0) / N) : 0.0;
                rel_err[i * D + d] = m > 0 ? se / m : INFINITY;
            }
        }
    }
    return LP_OK;
}

int lp_batch_get_tallies(lp_batch *b, int32_t i, lp_tallies *out)
{
    if (!b || !out) return fail(nullptr, LP_ERR_INVALID, "lp_batch_get_tallies: NULL argument");
    if (i < 0 || i >= (int32_t)b->inst.size()) return bfail(b, LP_ERR_INVALID, "lp_batch_get_tallies: instance %d", i);
    LP_BCUDA(b, cudaSetDevice(b->device));
    cudaStream_t s = b->stream;
    const size_t DD = std::max<size_t>(b->n_det, 1);
    b->h_sft.resize(b->n_sft);
    b->h_rtd.resize(b->n_rtd);
    b->h_rz.resize(b->n_rz);
    b->h_vox.resize(b->n_vox);
    b->h_rbins.resize(b->n_rbins);
    b->h_region.resize(lp::kBatchMedia);
    b->h_det.resize(DD * 2);
    LP_BCUDA(b, cudaMemcpyAsync(b->h_sft.data(), b->sft.p + i * b->n_sft, b->n_sft * 8, cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(b->h_rtd.data(), b->rtd.p + i * b->n_rtd, b->n_rtd * 8, cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(b->h_rz.data(), b->rz_of[i], b->n_rz * 8, cudaMemcpyDeviceToHost, s));
    if (b->n_vox)
        LP_BCUDA(b, cudaMemcpyAsync(b->h_vox.data(), b->vox_of[i], b->n_vox * 8, cudaMemcpyDeviceToHost, s));
    if (b->n_rbins)
        LP_BCUDA(b, cudaMemcpyAsync(b->h_rbins.data(), b->rbins.p + i * b->n_rbins, b->n_rbins * 8,
                                    cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(b->h_region.data(), b->region.p + (size_t)i * lp::kBatchMedia, lp::kBatchMedia * 8,
                                cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(b->h_det.data(), b->det.p + i * DD * 2, DD * 2 * 8, cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(out->counters, b->counters.p + (size_t)i * LP_NCOUNTERS, LP_NCOUNTERS * 8,
                                cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaStreamSynchronize(s));
    out->sft = b->h_sft.data();
    out->rtd = b->h_rtd.data();
    out->rz = b->h_rz.data();
    out->vox = b->h_vox.data();
    out->rbins = b->h_rbins.data();
    out->region = b->h_region.data();
    out->det = b->h_det.data();
    out->n_vox = (int64_t)b->n_vox;
    out->n_rbins = (int64_t)b->n_rbins / 2;
    out->n_region = b->inst[i].n_media;
    out->n_det = (int64_t)b->n_det;
    return LP_OK;
}

int lp_batch_get_gradient(lp_batch *b, int32_t i, lp_gradient *out)
{
    if (!b || !out) return fail(nullptr, LP_ERR_INVALID, "lp_batch_get_gradient: NULL argument");
    if (i < 0 || i >= (int32_t)b->inst.size()) return bfail(b, LP_ERR_INVALID, "lp_batch_get_gradient: instance %d", i);
    if (!b->grad_on) return bfail(b, LP_ERR_STATE, "lp_batch_get_gradient: differentiation is off");
    LP_BCUDA(b, cudaSetDevice(b->device));
    const lp_instance &in = b->inst[i];
    const int D = (int)b->n_det, R = in.n_media;
    const size_t DD = std::max<size_t>(b->n_det, 1);
    std::vector<uint64_t> det(DD * 2), cnt(LP_NCOUNTERS);
    b->h_grad.assign(grad_stride(b), 0.0);
    cudaStream_t s = b->stream;
    LP_BCUDA(b, cudaMemcpyAsync(b->h_grad.data(), b->grad.p + i * grad_stride(b), grad_stride(b) * 8,
                                cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(det.data(), b->det.p + i * DD * 2, DD * 2 * 8, cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaMemcpyAsync(cnt.data(), b->counters.p + (size_t)i * LP_NCOUNTERS, LP_NCOUNTERS * 8,
                                cudaMemcpyDeviceToHost, s));
    LP_BCUDA(b, cudaStreamSynchronize(s));
    form_gradient(det.data(), b->h_grad.data(), (double)cnt[LP_C_PHOTONS], (double)b->ctx[in.context]->factor,
                  in.nmuasg, D, R, b->gout);
    fill_gradient(b->gout, D, R, (int64_t)cnt[LP_C_PHOTONS], out);
    return LP_OK;
}

}  // extern "C"
