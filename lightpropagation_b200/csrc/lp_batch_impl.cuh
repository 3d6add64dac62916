// lp_batch_impl.cuh -- one persistent launch over many transport instances.
//
// An instance is one complete transport problem: a mesh (BVH + cell grid), a table of
// optical properties, a photon budget and its own tallies, described by a KParams in
// device memory.  The reference runs one such problem per program run
// (CalculatePropagation::ExecKernel, CalculatePropagation.cpp:1389-1759); here a whole
// set of them -- meshes x wavelengths x optical-property draws with uneven budgets --
// runs in one launch, so the GPU drains once instead of once per problem.
//
// Work distribution: each warp is bound to one instance at a time and keeps a copy of
// its KParams, mesh view and media table in its own shared-memory slot.  The warps start
// spread over the instances in proportion to their photons, and lanes whose photon ended
// take new photon indices of their instance with one atomicAdd per warp refill on its
// claim counter.  When the instance has no unclaimed photons left, the warp finishes the
// photons it holds, adds its counters to the instance's, and binds the next instance that
// has some.  (A warp that changes its instance has to drain first, for as long as the
// longest of its photons; with every warp on the first unfinished instance, as it was,
// small instances drained each warp once per 32 photons.  Curved abdomen, 1e6 photons in
// 32 instances: 98 -> 70 ms; 4e5 in 8 differentiated: 46 -> 37 ms.)  A photon is
// traced by exactly the same device functions as in transport_kernel, with the same Philox
// counter (photon id, event, stream), so an instance's integer tallies equal those of a
// single-instance run bit for bit.
#pragma once
#include "lp_transport_impl.cuh"

namespace lp {

struct WarpSlot {
    KParams P;
    MeshView M;
    WarpQueue Q;
    WarpDraws W;
    Medium media[kBatchMedia];
};

__device__ __forceinline__ void warp_flush_counters(const KParams &P, const Counters &c, uint32_t photons,
                                                    unsigned lane)
{
    const uint32_t v[10] = {c.scatter(), c.boundary, c.query, c.roulette, c.rz_drop, c.vox_drop, photons, c.skip(),
                            c.bvh, 0u};
    const int slot[9] = {0, 1, 2, 3, 6, 7, 8, 10, 11};
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        unsigned long long x = v[i];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0 && x) atomicAdd(P.counters + slot[i], x);
    }
}

// Copy instance `i` into the warp's slot (all 32 lanes take part).
__device__ __forceinline__ void warp_load_slot(WarpSlot &S, const KParams *inst, int i, unsigned lane)
{
    const uint32_t *src = reinterpret_cast<const uint32_t *>(inst + i);
    uint32_t *dst = reinterpret_cast<uint32_t *>(&S.P);
    for (unsigned k = lane; k < sizeof(KParams) / 4; k += 32) dst[k] = __ldg(src + k);
    __syncwarp();
    const uint32_t *ms = reinterpret_cast<const uint32_t *>(S.P.media);
    uint32_t *md = reinterpret_cast<uint32_t *>(S.media);
    const unsigned words = (unsigned)S.P.n_media * (sizeof(Medium) / 4);
    for (unsigned k = lane; k < words; k += 32) md[k] = __ldg(ms + k);
    if (lane == 0) {
        MeshView &M = S.M;
        M.na = S.P.node_a; M.nb = S.P.node_b; M.nc = S.P.node_c; M.nd = S.P.node_d;
        M.tri = S.P.tri;
        M.s_na = M.s_nb = M.s_nc = nullptr;
        M.s_nd = nullptr;
        M.s_tri = nullptr;
        M.nodes_smem = 0;
        M.tris_smem = 0;
        M.n_nodes = S.P.n_nodes;
        M.n_tri = S.P.n_tri;
        M.dbg = S.P.counters ? S.P.counters + kBoundsCounter : nullptr;
        M.tri_eps = S.P.tri_eps;
    }
    __syncwarp();
}

__device__ __forceinline__ void zero_grad(GradAcc &ga, int n_media)
{
    for (int r = 0; r < n_media; ++r) {
        ga.L[r] = 0.0f;
        ga.k[r] = 0;
    }
}

// Claims photons of the first instance with unclaimed ones, looking from `from` on
// (cyclically): its index and the first claimed photon in `base`, or -1.  The whole warp.
__device__ __forceinline__ int claim_instance(const BatchParams &B, int from, unsigned lanes, unsigned lane,
                                              unsigned long long &base)
{
    for (int r = 0; r < B.n_inst; r += 32) {
        const int k = r + (int)lane;
        const int i = (from + k) % B.n_inst;
        const bool open = k < B.n_inst && __ldcg(B.claimed + i) < (unsigned long long)(B.cum[i + 1] - B.cum[i]);
        for (unsigned m = __ballot_sync(0xffffffffu, open); m; m &= m - 1) {
            const int c = __shfl_sync(0xffffffffu, i, __ffs(m) - 1);
            if (lane == 0) base = atomicAdd(B.claimed + c, (unsigned long long)lanes);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base < (unsigned long long)(B.cum[c + 1] - B.cum[c])) return c;
        }
    }
    return -1;
}

template <bool Exact, bool Grad, int BLOCK, int MINB, int STACK>
__global__ void __launch_bounds__(BLOCK, MINB) batch_kernel(const __grid_constant__ BatchParams B)
{
    extern __shared__ __align__(16) unsigned char smem[];
    WarpSlot *const slots = reinterpret_cast<WarpSlot *>(smem);
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    WarpSlot &S = slots[threadIdx.x >> 5];
    Counters cnt = {};
    uint32_t photons = 0;
    Photon ph;
    GradAcc ga;
    uint32_t next_draw = 0;
    ph.idx = ph.steps = 0;
    ph.curr = 0;
    bool alive = false;
    const unsigned lanes = __popc(B.lane_mask);
    int inst = -1, from;   // from: where the search for the next instance begins
    {
        // the instance that holds this warp's share of all photons
        const double w = (double)(blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5)) / (double)(gridDim.x * (BLOCK / 32));
        const int64_t x = (int64_t)(w * (double)B.cum[B.n_inst]);
        int lo = 0, hi = B.n_inst - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (B.cum[mid] <= x) lo = mid;
            else hi = mid - 1;
        }
        from = lo;
    }
    bool exhausted = true;   // the bound instance has no unclaimed photons (or none is bound)
    for (;;) {
        unsigned live = __ballot_sync(0xffffffffu, alive);
        if (live == 0 && exhausted) {
            // every lane is idle: close the instance, bind the next one with unclaimed photons
            if (inst >= 0) {
                warp_flush_counters(S.P, cnt, photons, lane);
                cnt = Counters{};
                photons = 0;
            }
            unsigned long long base = 0;
            const int next = claim_instance(B, from, lanes, lane, base);
            if (next < 0) break;
            from = next;
            __syncwarp();
            warp_load_slot(S, B.inst, next, lane);
            inst = next;
            const unsigned long long n = (unsigned long long)S.P.n;
            exhausted = base + lanes >= n;
            next_draw = 0;
            const unsigned long long idx = base + lane;
            if (lane < lanes && idx < n) {
                start_photon(S.P, ph, (uint32_t)idx);
                if (Grad) zero_grad(ga, S.P.n_media);
                alive = true;
            }
            live = __ballot_sync(0xffffffffu, alive);
        } else if (live != B.lane_mask && !exhausted) {
            const unsigned need = B.lane_mask & ~live;
            const int k = __popc(need);
            next_draw = 0;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(B.claimed + inst, (unsigned long long)k);
            base = __shfl_sync(0xffffffffu, base, 0);
            const unsigned long long n = (unsigned long long)S.P.n;
            if (base + (unsigned long long)k >= n) exhausted = true;
            if ((need >> lane) & 1u) {
                const unsigned long long idx = base + __popc(need & lt_mask);
                if (idx < n) {
                    start_photon(S.P, ph, (uint32_t)idx);
                    if (Grad) zero_grad(ga, S.P.n_media);
                    alive = true;
                }
            }
            live = __ballot_sync(0xffffffffu, alive);
        }
        const bool more = step_photon<Exact, Grad, STACK>(S.P, S.M, S.M, S.Q, S.media, S.P.region, S.P.counters, live,
                                                          alive, ph, cnt, &ga, S.W, next_draw, rz_copy_of(S.P));
        if (alive) {
            if (!more) {
                if (ph.region_acc) atomicAdd(S.P.region + ph.curr, ph.region_acc);
                if (Grad) {
                    ga.L[ph.curr] += ph.seg_len;
                    ga.k[ph.curr] += ph.seg_k;
                }
                finish_photon<Grad>(S.P, exit_state(ph), Grad ? &ga : nullptr);
                cnt.steps += ph.steps;
                photons++;
                alive = false;
            }
        }
    }
    if (inst >= 0) warp_flush_counters(S.P, cnt, photons, lane);
}

template <bool Exact, bool Grad, int BLOCK, int MINB, int STACK>
cudaError_t launch_batch_t(const BatchParams &B, int grid, cudaStream_t s)
{
    const int smem = BLOCK / 32 * (int)sizeof(WarpSlot);
    cudaError_t e = cudaFuncSetAttribute(batch_kernel<Exact, Grad, BLOCK, MINB, STACK>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    batch_kernel<Exact, Grad, BLOCK, MINB, STACK><<<grid, BLOCK, smem, s>>>(B);
    return cudaGetLastError();
}

template <bool Exact, bool Grad, int BLOCK, int MINB, int STACK>
cudaError_t batch_occupancy_t(int *blocks_per_sm)
{
    const int smem = BLOCK / 32 * (int)sizeof(WarpSlot);
    cudaError_t e = cudaFuncSetAttribute(batch_kernel<Exact, Grad, BLOCK, MINB, STACK>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, batch_kernel<Exact, Grad, BLOCK, MINB, STACK>,
                                                         BLOCK, smem);
}

}  // namespace lp
