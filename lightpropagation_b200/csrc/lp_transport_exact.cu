// lp_transport_exact.cu -- reference-arithmetic instantiation of the transport kernel
// (Exact = true, compiled with --fmad=false), the BVH query kernel used to verify the
// traversal against the brute-force scan, and small utility kernels.
#include "lp_transport_impl.cuh"

namespace lp {

cudaError_t launch_transport_exact(const KParams &P, int grid, int smem, cudaStream_t s)
{
    return launch_transport_t<true>(P, grid, smem, s);
}

cudaError_t transport_occupancy_exact(int smem, int *blocks_per_sm)
{
    return transport_occupancy_t<true, false>(smem, blocks_per_sm);
}

// The transport of lp_run_noalloc: reference arithmetic, no cell grid, distance bounds from
// the mesh itself (P.mesh_eps set).
cudaError_t launch_transport_no_grid(const KParams &P, int grid, int smem, cudaStream_t s)
{
    if (P.few_blocks) return launch_instance<true, false, false, true, kFewBlocks>(P, grid, smem, s);
    return launch_instance<true, false, false, true, LP_TRANSPORT_MIN_BLOCKS>(P, grid, smem, s);
}

cudaError_t transport_occupancy_no_grid(int smem, int *blocks_per_sm)
{
    const cudaError_t e = allow_smem(transport_kernel<true, false, false, true>, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, transport_kernel<true, false, false, true>, kBlock,
                                                         smem);
}

cudaError_t transport_occupancy_exact_grad(int smem, int *blocks_per_sm)
{
    return transport_occupancy_t<true, true>(smem, blocks_per_sm);
}

__global__ void __launch_bounds__(kBlock) query_kernel(const __grid_constant__ KParams P, int64_t n,
                                                       const float *orig, const float *dir,
                                                       const int32_t *ref, const float *tmax,
                                                       int32_t *id_out, float *t_out)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ WarpQueue queues[kBlock / 32];
    const SmemLayout L = smem_layout(P.nodes_smem, P.tris_smem);
    const MeshView M = stage_mesh(P, smem, L);
    __shared__ MeshView shared_view;
    if (threadIdx.x == 0) shared_view = M;
    __syncthreads();
    // A march costs by the cell, a descent of a small tree little: on meshes below 2,048
    // triangles rays of more than n_tri / 16 cells go to the tree.  1e6 rays, march / tree, us:
    // slab (32 triangles) of 3 cells 139 / 96, of 34 517 / 159, unbounded 1221 / 237; abdomen of
    // 100 triangles, 3 cells 183 / 477, 40 753 / 638, unbounded 1178 / 766; of 1,600, 10 cells 319 /
    // 622, unbounded 1220 / 1208.
    const float march = P.n_tri < 2048 ? (float)P.n_tri * P.g_h * (1.0f / 16.0f) : 3.0e38f;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // warp-uniform trip count: the query is the whole warp's
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31u); w < n; w += stride) {
        const int64_t i = w + (threadIdx.x & 31u);
        const bool want = i < n;
        const int64_t q = want ? i : 0;
        const V3 p = v3(orig[3 * q], orig[3 * q + 1], orig[3 * q + 2]);
        const V3 v = v3(dir[3 * q], dir[3 * q + 1], dir[3 * q + 2]);
        float t, safe = 0.0f;
        bool used_bvh;
        const int id = warp_query(P, M, shared_view, queues[threadIdx.x >> 5], want, p, v, ref[q], tmax[q],
                                  tmax[q] > march ? kCellDense << 24 : query_word(P, p, v), t, safe, used_bvh);
        if (want) {
            id_out[i] = id;
            t_out[i] = t;
        }
    }
}

// out[3 i + k] = soa[k n + i], k < 3.
__global__ void __launch_bounds__(256) interleave_kernel(const float4 *soa, int64_t n, float4 *out)
{
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < 3 * n; x += (int64_t)gridDim.x * blockDim.x)
        out[x] = soa[(x % 3) * n + x / 3];
}

// dst[k][i] += the sum of part[k][0..copies)[i], and the copies are left at zero for the
// next launch.  k < images, i < n.  Bound by the bytes of the copies (HBM or L2).
__global__ void __launch_bounds__(256) fold_kernel(unsigned long long *dst, unsigned long long *part, int copies,
                                                   int64_t n, int64_t images)
{
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n * images;
         x += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long *const p = part + (x / n) * copies * n + x % n;
        unsigned long long sum = 0;
        for (int c = 0; c < copies; ++c) {
            const unsigned long long v = p[c * n];
            if (v) p[c * n] = 0;
            sum += v;
        }
        if (sum) dst[x] += sum;
    }
}

// op 0: sqrt_normal(a), 1: rcp_rn(a), 2: div_rn(a, b) with the reciprocal of rcp_rn.
__global__ void __launch_bounds__(256) exact_ops_kernel(int op, int64_t n, const float *a, const float *b, float *out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = op == 0 ? sqrt_normal(a[i]) : op == 1 ? rcp_rn(a[i]) : div_rn(a[i], b[i], rcp_rn(b[i]));
}

__global__ void philox_kernel(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0,
                              uint32_t k1, int64_t n, uint32_t *out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t a = c0, b = c1, c = c2 + (uint32_t)i, d = c3, r0[10], r1[10];
#pragma unroll
        for (int r = 0; r < 10; ++r) {
            r0[r] = philox_key0(k0, r);
            r1[r] = philox_key1(k1, r);
        }
        philox4x32_10(a, b, c, d, r0, r1);
        out[4 * i] = a; out[4 * i + 1] = b; out[4 * i + 2] = c; out[4 * i + 3] = d;
    }
}

// FP32 throughput probe: 8 independent FMA chains per thread.  2 flops per FMA.
__global__ void __launch_bounds__(256) fma_peak_kernel(float *out, int iters, float a, float b)
{
    float x0 = threadIdx.x * 1e-3f, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
    float x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            x0 = __fmaf_rn(x0, a, b); x1 = __fmaf_rn(x1, a, b); x2 = __fmaf_rn(x2, a, b); x3 = __fmaf_rn(x3, a, b);
            x4 = __fmaf_rn(x4, a, b); x5 = __fmaf_rn(x5, a, b); x6 = __fmaf_rn(x6, a, b); x7 = __fmaf_rn(x7, a, b);
        }
    }
    const float s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
    if (s == 1234.5f) out[0] = s;  // keeps the chains alive; practically never taken
}

// 64-bit atomic adds whose results are not used (reductions at the L2), each lane of a
// warp to its own pseudo-random slot of an L2-resident buffer: the access pattern of the
// transport kernel's absorption deposits.
__global__ void __launch_bounds__(256) red_peak_kernel(unsigned long long *buf, uint32_t mask, int iters)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t h = g * 0x9E3779B1u + 0x7F4A7C15u;
    for (int i = 0; i < iters; ++i) {
        h ^= h >> 15;
        h *= 0x2C1B3C6Du;
        h ^= h >> 12;
        atomicAdd(buf + (h & mask), 1ull);
    }
}

int smem_bytes(int nodes_smem, int tris_smem) { return smem_layout(nodes_smem, tris_smem).bytes; }

int block_size() { return kBlock; }

cudaError_t launch_query(const KParams &P, int smem, int64_t n, const float *orig, const float *dir,
                         const int32_t *ref, const float *tmax, int32_t *id_out, float *t_out,
                         cudaStream_t s)
{
    const cudaError_t e = allow_smem(query_kernel, smem);
    if (e != cudaSuccess) return e;
    // 2,048 threads per SM; half of them took a fifth longer for 1e6 rays
    int grid = (int)std::min<int64_t>((n + kBlock - 1) / kBlock, 148 * 16);
    if (grid < 1) grid = 1;
    query_kernel<<<grid, kBlock, smem, s>>>(P, n, orig, dir, ref, tmax, id_out, t_out);
    return cudaGetLastError();
}

cudaError_t launch_interleave(const float4 *soa, int64_t n, float4 *out, cudaStream_t s)
{
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((3 * n + 255) / 256, 148 * 8));
    interleave_kernel<<<grid, 256, 0, s>>>(soa, n, out);
    return cudaGetLastError();
}

cudaError_t launch_fold(unsigned long long *dst, unsigned long long *part, int copies, int64_t n, int64_t images,
                        cudaStream_t s)
{
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n * images + 255) / 256, 148 * 8));
    fold_kernel<<<grid, 256, 0, s>>>(dst, part, copies, n, images);
    return cudaGetLastError();
}

cudaError_t launch_exact_ops(int op, int64_t n, const float *a, const float *b, float *out, cudaStream_t s)
{
    exact_ops_kernel<<<(int)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(op, n, a, b, out);
    return cudaGetLastError();
}

cudaError_t launch_philox(const uint32_t *ctr, const uint32_t *key, int64_t n, uint32_t *out, cudaStream_t s)
{
    int grid = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
    if (grid < 1) grid = 1;
    philox_kernel<<<grid, 256, 0, s>>>(ctr[0], ctr[1], ctr[2], ctr[3], key[0], key[1], n, out);
    return cudaGetLastError();
}

double fma_peak_tflops(int num_sms)
{
    float *d = nullptr;
    if (cudaMalloc(&d, 16) != cudaSuccess) return 0.0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = num_sms * 8, threads = 256, iters = 4096;
    fma_peak_kernel<<<blocks, threads>>>(d, 64, 0.999f, 1e-3f);  // warm-up
    double best = 0.0;
    for (int r = 0; r < 3; ++r) {
        cudaEventRecord(e0);
        fma_peak_kernel<<<blocks, threads>>>(d, iters, 0.999f, 1e-3f);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
        if (ms > 0) best = std::max(best, flops / (ms * 1e-3) / 1e12);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(d);
    return best;
}

// Throughput of 64-bit atomic reductions to an L2-resident buffer (16 MB), in atomics/s.
double red_peak_per_s(int num_sms)
{
    const uint32_t slots = 1u << 21;   // 16 MB of uint64
    unsigned long long *d = nullptr;
    if (cudaMalloc(&d, (size_t)slots * 8) != cudaSuccess) return 0.0;
    cudaMemset(d, 0, (size_t)slots * 8);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = num_sms * 8, threads = 256, iters = 512;
    red_peak_kernel<<<blocks, threads>>>(d, slots - 1, 16);   // warm-up
    double best = 0.0;
    for (int r = 0; r < 3; ++r) {
        cudaEventRecord(e0);
        red_peak_kernel<<<blocks, threads>>>(d, slots - 1, iters);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        const double n = (double)iters * blocks * threads;
        if (ms > 0) best = std::max(best, n / (ms * 1e-3));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(d);
    return best;
}

}  // namespace lp
