// lp_kernel.cuh -- device-side data layout and helpers of the transport kernel.
//
// Arithmetic follows src/Simulation/MCLightPropagation.cl operation by operation
// (same operand order, IEEE division and square root, no contraction: the file is
// compiled with --fmad=false), so a photon that consumes the same random numbers
// follows the same trajectory as in the reference kernel up to the last-place
// differences of logf/cosf/acosf.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace lp {

constexpr int kMaxMedia = 64;
constexpr int kMaxDet = 32;
constexpr int kStackDepth = 64;
constexpr int kGradRegions = 8;      // regions a differentiated run may have
constexpr float kNoHit = 10000.0f;   // FindTriangleInPath's initial distance (.cl:1042)
// photons of one transport launch: the kernels index them with 32 bits
constexpr int64_t kMaxLaunchPhotons = int64_t(1) << 31;

// The factors of one step sit together: two 16-byte loads in the production arithmetic.
struct alignas(16) Medium {
    float inv_mut, alb, inv_mua;   // 1 / (mua + mus), mua / (mua + mus), 1 / mua (0 for mua <= 0)
    uint32_t kind;                 // kAbsorbs, kAmbient
    float hg_a, hg_b, hg_c, hg_d;  // 1-g^2, 1-g, 2g, 1+g^2
    float hg_inv2g, g, mua, mus;   // 1/(2g)
    float n, mut, pad_[2];         // mut = mua + mus
};
constexpr uint32_t kAbsorbs = 1u;  // mua > 0 && mus > 0  (Absorb, .cl:841-847)
constexpr uint32_t kAmbient = 2u;  // mua == 0 && mus == 0 (step = distance to boundary, .cl:1405-1410)
constexpr uint32_t kPlainDiv = 4u; // a divisor outside of div_range: the plain operator divides

// Divisors for which div_rn needs no care for overflow and underflow.
__host__ __device__ __forceinline__ bool div_range(float x) { return x >= 1e-12f && x <= 1e12f; }
// Those of a medium: mua, mut, 2 g and 1 - g + 2 g xi.
__host__ __device__ __forceinline__ uint32_t plain_div_of(float mua, float mut, float g)
{
    const float a = g < 0.0f ? -g : g;
    return div_range(mua) && div_range(mut) && (g == 0.0f || (a >= 1e-6f && 1.0f - a >= 1e-6f)) ? 0u : kPlainDiv;
}

struct KParams {
    // mesh (see lp_bvh.hpp)
    const float4 *node_a, *node_b, *node_c;
    const int4 *node_d;
    const float4 *tri;        // three per triangle in BVH order: tri_a, tri_b, tri_c of lp_bvh.hpp
    const float4 *tri_attr;   // by original index: unit normal, (inner | outer << 16) bits
    int32_t n_nodes, n_tri, nodes_smem, tris_smem;
    // media
    const Medium *media;
    int32_t n_media;
    // source and frame
    float p0x, p0y, p0z, v0x, v0y, v0z;
    float poix, poiy, poiz;
    float ezx, ezy, ezz;             // eZ as given (sign test of the axis override)
    float nxx, nxy, nxz, nyx, nyy, nyz, nzx, nzy, nzz;  // normalised eX, eY, eZ
    float Rsp, distMin, exitScale, w0;
    int32_t src_type;                // 0 pencil beam (reference), 1 fibre disk + cone
    float src_radius, src_cos_max;
    // run parameters
    float chance, w_th, factor;
    int32_t fetal_id;
    uint32_t compat;
    uint32_t key0[10], key1[10];     // Philox round keys (set_keys)
    uint32_t stream;
    uint32_t step_cap;               // steps after which a photon is stopped (step_cap_of)
    int64_t first, n;
    // reference tally layout
    int32_t hx, hy, sft_nx, dimR, dimAlpha, rz_nr, rz_nz;
    float dg[6];
    float inv_dr, inv_dz, inv_vdx, inv_vdy, inv_vdz;   // reciprocals for the fast mode
    float f_dimR, half_vnx, half_vny;                  // dimR, vox_nx / 2, vox_ny / 2
    uint32_t vox_on;                                   // 1 with a voxel grid
    uint32_t plain_div;                                // a bin width lies outside of div_range
    // tallies (fixed point, 2^32 per unit weight)
    unsigned long long *sft, *rtd, *rz, *vox, *rbins, *region, *det, *counters;
    // where the r-z deposits go: rz_mask + 1 (a power of two) copies of the image, each of
    // rz_stride values, one for every block index modulo their number; launch_fold adds
    // them to rz.  One copy: rz itself.
    unsigned long long *rz_part;
    int64_t rz_stride;
    uint32_t rz_mask;
    int32_t vox_nx, vox_ny, vox_nz;
    float vox_dx, vox_dy, vox_dz;
    int32_t n_rbins;
    float rbin_dr;
    int32_t n_det;
    float det_lo[kMaxDet], det_hi[kMaxDet];
    float *exit_rec;
    int64_t exit_cap;
    // differentiation (null: off): per (ring detector d, region r), over the photons
    // scored in ring d with surface weight s, the sums of a = s * L_r and b = s * k_r,
    // where L_r is the photon's path length and k_r its number of interactions in
    // region r: grad[5 * (d * n_media + r) + {0..4}] = sum a, sum b, sum a^2, sum b^2, sum a b
    double *grad;
    // cell grid over the mesh bounds (cubic cells of size 1 / g_inv_h), one word per cell:
    //   kCellEmpty set:   no triangle touches the cell; bits 0-15 hold a lower bound of
    //                     the distance from any point of the cell to the nearest
    //                     triangle, in units of g_unit
    //   kCellEmpty clear: bits 0-23 = first entry in cell_refs, bits 24-30 = number of
    //                     triangles touching the cell (kCellDense: too many, use the BVH)
    // cell_refs holds BVH-order triangle indices.  Null cell_word: BVH queries only.
    const uint32_t *cell_word;
    const int32_t *cell_refs;   // null: the words carry safety bounds only
    int64_t n_cell_refs;
    float g_ox, g_oy, g_oz, g_inv_h, g_unit, g_eps;
    int32_t g_nx, g_ny, g_nz;
    // a cell's list holds every triangle touching the cell widened by g_margin + g_eps on
    // every side; g_h is the cell edge; step_eps bounds the rounding of one position update
    float g_margin, g_h, step_eps;
    // a mesh without a grid whose scale only the device knows (lp_run_noalloc): the rounding
    // allowance of a distance bound and step_eps, in device memory; null: no bounds without a
    // grid
    const float *mesh_eps;
    // production arithmetic: distance a photon is moved off a face after a boundary event,
    // and the barycentric tolerance of the hit test (both 0 in the reference arithmetic)
    float boundary_push, tri_eps;
    // 1: absorption deposits are summed per cell across the warp before the atomic adds
    int32_t agg_tallies;
    // scratch: photon work counter
    unsigned long long *work;
    uint32_t lane_mask;   // lanes of a warp that carry photons (plan_launch)
    // host side: the kernel instance for 16 warps per SM runs (plan_launch)
    uint32_t few_blocks;
};

// Blocks of a transport launch and the lanes of a warp that carry photons.  A short run
// lasts as long as its longest photon (many times the mean), and a photon's step takes
// the longer the more others share its warp (each of them may have a query or a boundary
// event) and its SM.  So up to the lanes of 16 warps per SM the photons are spread evenly
// over those warps, and up to twice as many take turns on them.  Against full warps, 24 per
// SM (slab / curved abdomen at 660 nm): 1,000 photons 17.9 -> 12.2 / 15.3 -> 10.1 ms, 10,000
// 20.8 -> 16.6 / 20.3 -> 18.1, 30,000 25.0 -> 20.5 / 23.5 -> 20.1, 100,000 31.2 -> 29.6 / 28.6
// -> 27.3; at 300,000 more warps win on the slab (43.7 against 47.7) and lose on the abdomen
// (42.8 against 40.2).
// few: the launch has no more than those warps, so the kernel instance compiled for them runs
// (107 registers instead of 95): 30,000 slab photons 16.7 -> 15.7 ms, 50,000 on 25,600
// triangles 17.3 -> 16.4, 1e5 on the abdomen 23.7 -> 23.0.
inline void plan_launch(int64_t n, int block, int num_sms, int per_sm, int &grid, uint32_t &lane_mask, uint32_t &few)
{
    const int blocks = per_sm * block < 512 ? per_sm : 512 / block > 1 ? 512 / block : 1;
    const int64_t warps = (int64_t)num_sms * blocks * (block / 32);
    int64_t lanes = (n + warps - 1) / warps;
    lanes = lanes < 1 ? 1 : lanes > 32 ? 32 : lanes;
    lane_mask = lanes == 32 ? 0xffffffffu : (1u << lanes) - 1u;
    few = n <= 64 * warps ? 1u : 0u;
    grid = num_sms * (few ? blocks : per_sm);
}

// A batch: many instances (one KParams each) traced by one persistent launch.
constexpr int kBatchMedia = kGradRegions;   // regions per instance in a batch
struct BatchParams {
    const KParams *inst;             // [n_inst] per-instance parameters (device memory)
    unsigned long long *claimed;     // [n_inst] photon indices handed out so far
    const int64_t *cum;              // [n_inst + 1] photons of the instances before each
    int32_t n_inst;
    uint32_t lane_mask;              // lanes of a warp that carry photons (plan_launch)
};

// Bounds checks of the debug build (compiled with -DLP_DEBUG into liblpcuda_debug.so):
// an index outside its array is counted in the counter slot LP_C_BOUNDS (13) and the
// access is skipped, so a bad index is reported instead of reading or writing past an
// allocation.  The release build compiles every check to `true`.
constexpr int kBoundsCounter = 13;
__device__ __forceinline__ bool in_range_dbg(unsigned long long *dbg, long long i, long long n)
{
    const bool ok = i >= 0 && i < n;
    if (!ok && dbg) atomicAdd(dbg, 1ull);
    return ok;
}
#ifdef LP_DEBUG
#define LP_IN_RANGE(dbg, i, n) ::lp::in_range_dbg((dbg), (long long)(i), (long long)(n))
#else
#define LP_IN_RANGE(dbg, i, n) true
#endif


constexpr uint32_t kCellEmpty = 0x80000000u;
constexpr uint32_t kCellDense = 127u;
constexpr uint32_t kCellOutside = 0x00010000u;

// The cell word at p; points outside the grid (every point when there is none: g_nx = 0)
// read as an empty cell with bound 0 and kCellOutside set.  The grid has at most 2^28
// cells, so 32-bit indices do.
__device__ __forceinline__ uint32_t cell_at(const KParams &P, float px, float py, float pz)
{
    const int ix = (int)floorf((px - P.g_ox) * P.g_inv_h);
    const int iy = (int)floorf((py - P.g_oy) * P.g_inv_h);
    const int iz = (int)floorf((pz - P.g_oz) * P.g_inv_h);
    const bool in = ((unsigned)ix < (unsigned)P.g_nx) & ((unsigned)iy < (unsigned)P.g_ny) &
                    ((unsigned)iz < (unsigned)P.g_nz);
    uint32_t w = kCellEmpty | kCellOutside;
    if (in) w = __ldg(P.cell_word + ((iz * P.g_ny + iy) * P.g_nx + ix));
    return w;
}

// Distance from p to the nearest face of the cell containing it (0 outside the grid):
// the smallest of the fractional cell coordinates and their complements, times h.
__device__ __forceinline__ float cell_face_distance(const KParams &P, float px, float py, float pz)
{
    const float fx = (px - P.g_ox) * P.g_inv_h, fy = (py - P.g_oy) * P.g_inv_h, fz = (pz - P.g_oz) * P.g_inv_h;
    const float rx = fx - floorf(fx), ry = fy - floorf(fy), rz = fz - floorf(fz);
    const float d = fminf(fminf(fminf(rx, 1.0f - rx), fminf(ry, 1.0f - ry)), fminf(rz, 1.0f - rz));
    return fmaxf(d, 0.0f) * P.g_h;
}

// Conservative distance from p to the nearest triangle (0 near a surface).
__device__ __forceinline__ float safe_distance(const KParams &P, uint32_t word)
{
    return (word & kCellEmpty) ? (float)(word & 0xffffu) * P.g_unit : 0.0f;
}

// ----------------------------------------------------------------- Philox4x32-10
__host__ __device__ __forceinline__ uint32_t philox_key0(uint32_t k0, int round)
{
    return k0 + 0x9E3779B9u * (uint32_t)round;
}
__host__ __device__ __forceinline__ uint32_t philox_key1(uint32_t k1, int round)
{
    return k1 + 0xBB67AE85u * (uint32_t)round;
}

// k0, k1: the ten round keys.  Kept in the kernel's parameters, they are operands of the
// exclusive-ors instead of two additions a round; the 64-bit products give both halves of
// a product in one instruction.
__device__ __forceinline__ void philox4x32_10(uint32_t &c0, uint32_t &c1, uint32_t &c2, uint32_t &c3,
                                              const uint32_t *k0, const uint32_t *k1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0[r], n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1[r];
        c0 = n0;
        c1 = (uint32_t)p1;
        c2 = n2;
        c3 = (uint32_t)p0;
    }
}

// The seed's round keys.
__host__ __device__ inline void set_keys(KParams &P, uint64_t seed)
{
    for (int r = 0; r < 10; ++r) {
        P.key0[r] = philox_key0((uint32_t)seed, r);
        P.key1[r] = philox_key1((uint32_t)(seed >> 32), r);
    }
}

// max_steps (<= 0: none) as the kernel's 32-bit cap; a photon's steps are counted in 32 bits
__host__ __device__ inline uint32_t step_cap_of(int64_t max_steps)
{
    return max_steps <= 0 || max_steps > (int64_t)0xffffffff ? 0xffffffffu : (uint32_t)max_steps;
}

// ((x >> 8) | 1) * 2^-24, a uniform in (0, 1) that is never 0.  (x >> 8) | 1 is 2 k + 1
// with k = x >> 9, so the value is k 2^-23 + 2^-24: k goes into the mantissa of a float
// in [2^23, 2^24), and one exact fused multiply-add does the rest (no conversion).
__device__ __forceinline__ float uniform24(uint32_t x)
{
    return __fmaf_rn(__uint_as_float(0x4B000000u | (x >> 9)), 0x1.0p-23f, -0x1.fffffep-1f);
}

// One Philox block per event: counter (photon lo, photon hi, event, stream), key =
// seed.  Event 0 samples the source, loop iteration i is event i + 1.  The four words
// are the event's draw slots (step, Fresnel or polar angle, azimuth, roulette), each
// mapped to a uniform by uniform24.
struct EventRng {
    float u0, u1, u2, u3;
    __device__ __forceinline__ void draw(const KParams &P, uint32_t idx, uint32_t event)
    {
        const uint64_t pid = (uint64_t)(P.first + (int64_t)idx);
        uint32_t c0 = (uint32_t)pid, c1 = (uint32_t)(pid >> 32), c2 = event, c3 = P.stream;
        philox4x32_10(c0, c1, c2, c3, P.key0, P.key1);
        u0 = uniform24(c0);
        u1 = uniform24(c1);
        u2 = uniform24(c2);
        u3 = uniform24(c3);
    }
};

// ------------------------------------------------------------- small vectors
struct V3 { float x, y, z; };
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ float dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross3(V3 a, V3 b)
{
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ V3 scl3(float s, V3 a) { return v3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ V3 add3(V3 a, V3 b) { return v3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ V3 sub3(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
// normalize(): v / |v|, zero vector unchanged (OpenCL semantics)
__device__ __forceinline__ V3 norm3(V3 v)
{
    const float l = sqrtf(dot3(v, v));
    if (l == 0.0f) return v;
    return v3(v.x / l, v.y / l, v.z / l);
}
__device__ __forceinline__ float sign_cl(float x)
{
    if (x > 0.0f) return 1.0f;
    if (x < 0.0f) return -1.0f;
    if (x != x) return 0.0f;
    return x;
}
__device__ __forceinline__ unsigned long long fix32(float w)
{
    return (w > 0.0f) ? __float2ull_rn(w * 4294967296.0f) : 0ull;
}
__device__ __forceinline__ int trunc_sat(float q)
{
    if (q != q) return 0;
    if (q > 1e9f) return 1000000000;
    if (q < -1e9f) return -1000000000;
    return (int)q;
}
__device__ __forceinline__ int trunc_sat_d(double q)
{
    if (q != q) return 0;
    if (q > 1e9) return 1000000000;
    if (q < -1e9) return -1000000000;
    return (int)q;
}

// ------------------------------------------------------------- BVH query
// Nearest triangle along (p, v) with t in (0, bound] and t < 10000, excluding
// ref_tri; equal distances resolve to the lower original index.  Returns the
// original index or -1; *t_out = distance or 10000.
struct MeshView {
    const float4 *na, *nb, *nc;
    const int4 *nd;
    const float4 *tri;
    const float4 *s_na, *s_nb, *s_nc;
    const int4 *s_nd;
    const float4 *s_tri;
    int32_t nodes_smem, tris_smem;
    int32_t n_nodes, n_tri;          // array sizes for the debug build's bounds checks
    // barycentric tolerance of the hit test: 0 is the reference's test; a few 1e-6 (the
    // production arithmetic) lets neighbouring triangles overlap along their shared
    // edges, so no ray slips through the float gap between them
    float tri_eps;
    unsigned long long *dbg;         // its counter of skipped accesses (may be null)
};

// A triangle record in BVH order, 48 bytes in one piece (two sectors; three apart would be
// three).
struct TriRec {
    float4 a, b, c;
};
__device__ __forceinline__ TriRec load_tri(const float4 *tri, int j)
{
    return TriRec{__ldg(tri + 3 * j), __ldg(tri + 3 * j + 1), __ldg(tri + 3 * j + 2)};
}

// The reference's ray/triangle test (.cl:1047-1083) of the ray (p, v), with G = p - M,
// GE = G x E and t0 = GE . F already formed: true when the triangle is hit at t in
// (0, kNoHit) with t not above `limit` by more than the filter's margin.
__device__ __forceinline__ bool tri_hit(const MeshView &M, V3 E, V3 F, V3 G, V3 GE, float t0, V3 v, float limit,
                                        float &t_out)
{
    const V3 VF = cross3(v, F);
    float t = t0;
    const float w = dot3(VF, E);
    float k = dot3(VF, G);
    float l = dot3(GE, v);
    // Division-free filter, looser than the exact test below: t, k, l must share the
    // sign of w, |k| + |l| may not exceed |w| and |t| may not exceed limit * |w| (each
    // with a relative margin far above the rounding of the divided values).  Only
    // candidates that pass pay for the three IEEE divisions of the reference test.
    const float aw = fabsf(w);
    const float ek = M.tri_eps * aw;
    const bool sgn = (w > 0.0f) ? (t > 0.0f && k >= -ek && l >= -ek) : (t < 0.0f && k <= ek && l <= ek);
    if (!sgn || fabsf(k) + fabsf(l) > aw * (1.0001f + 3.0f * M.tri_eps) || fabsf(t) > limit * aw * 1.0001f)
        return false;
    t = t / w;
    k = k / w;
    l = l / w;
    t_out = t;
    return t > 0.0f && t < kNoHit && k >= -M.tri_eps && l >= -M.tri_eps && (k + l) < 1.0f + M.tri_eps;
}

__device__ __forceinline__ void test_tri(const MeshView &M, int j, V3 p, V3 v, int ref_tri, float &best,
                                         int &bid)
{
    if (!LP_IN_RANGE(M.dbg, j, M.n_tri)) return;
    TriRec T;
    if (j < M.tris_smem) T = TriRec{M.s_tri[3 * j], M.s_tri[3 * j + 1], M.s_tri[3 * j + 2]};
    else T = load_tri(M.tri, j);
    const int o = __float_as_int(T.c.y);
    if (o == ref_tri) return;
    const V3 E = v3(T.a.w, T.b.x, T.b.y), F = v3(T.b.z, T.b.w, T.c.x);
    const V3 G = sub3(p, v3(T.a.x, T.a.y, T.a.z));
    const V3 GE = cross3(G, E);
    float t;
    if (tri_hit(M, E, F, G, GE, dot3(GE, F), v, best, t) && (t < best || (t == best && o < bid))) {
        best = t;
        bid = o;
    }
}

// STACK: traversal stack entries; the host only runs a tree whose depth is below it.
template <int STACK = kStackDepth>
__device__ __noinline__ int query_nearest(const MeshView &M, V3 p, V3 v, int ref_tri, float bound,
                                             float &t_out)
{
    float best = fminf(bound, kNoHit);
    int bid = 0x7fffffff;
    const float ix = 1.0f / (fabsf(v.x) > 1e-30f ? v.x : copysignf(1e-30f, v.x));
    const float iy = 1.0f / (fabsf(v.y) > 1e-30f ? v.y : copysignf(1e-30f, v.y));
    const float iz = 1.0f / (fabsf(v.z) > 1e-30f ? v.z : copysignf(1e-30f, v.z));
    const float ox = p.x * ix, oy = p.y * iy, oz = p.z * iz;
    int stack[STACK];
    int sp = 0;
    int node = 0;
    for (;;) {
        float4 a, b, c;
        int4 d;
        if (!LP_IN_RANGE(M.dbg, node, M.n_nodes)) break;
        if (node < M.nodes_smem) {
            a = M.s_na[node]; b = M.s_nb[node]; c = M.s_nc[node]; d = M.s_nd[node];
        } else {
            a = __ldg(M.na + node); b = __ldg(M.nb + node); c = __ldg(M.nc + node); d = __ldg(M.nd + node);
        }
        // slab tests of both children against [0, best]
        float t0, t1, tn0, tf0, tn1, tf1;
        t0 = a.x * ix - ox; t1 = a.y * ix - ox;
        tn0 = fminf(t0, t1); tf0 = fmaxf(t0, t1);
        t0 = a.z * iy - oy; t1 = a.w * iy - oy;
        tn0 = fmaxf(tn0, fminf(t0, t1)); tf0 = fminf(tf0, fmaxf(t0, t1));
        t0 = c.x * iz - oz; t1 = c.y * iz - oz;
        tn0 = fmaxf(tn0, fminf(t0, t1)); tf0 = fminf(tf0, fmaxf(t0, t1));
        t0 = b.x * ix - ox; t1 = b.y * ix - ox;
        tn1 = fminf(t0, t1); tf1 = fmaxf(t0, t1);
        t0 = b.z * iy - oy; t1 = b.w * iy - oy;
        tn1 = fmaxf(tn1, fminf(t0, t1)); tf1 = fminf(tf1, fmaxf(t0, t1));
        t0 = c.z * iz - oz; t1 = c.w * iz - oz;
        tn1 = fmaxf(tn1, fminf(t0, t1)); tf1 = fminf(tf1, fmaxf(t0, t1));
        // widen the far end relative to best so rounding never culls a tie
        const float lim = best * 1.000001f + 1e-6f;
        bool h0 = fmaxf(tn0, 0.0f) <= fminf(tf0, lim);
        bool h1 = fmaxf(tn1, 0.0f) <= fminf(tf1, lim);
        if (h0 && d.x < 0) {
            const int e = ~d.x, f = e >> 3, cnt = (e & 7) + 1;
            for (int j = f; j < f + cnt; ++j) test_tri(M, j, p, v, ref_tri, best, bid);
            h0 = false;
        }
        if (h1 && d.y < 0) {
            const int e = ~d.y, f = e >> 3, cnt = (e & 7) + 1;
            for (int j = f; j < f + cnt; ++j) test_tri(M, j, p, v, ref_tri, best, bid);
            h1 = false;
        }
        if (h0 && h1) {
            const bool first0 = tn0 <= tn1;
            if (sp < STACK) stack[sp++] = first0 ? d.y : d.x;
            node = first0 ? d.x : d.y;
        } else if (h0) {
            node = d.x;
        } else if (h1) {
            node = d.y;
        } else {
            if (sp == 0) break;
            node = stack[--sp];
        }
    }
    if (bid == 0x7fffffff) {
        t_out = kNoHit;
        return -1;
    }
    t_out = best;
    return bid;
}

// The cell word that a query from p along v begins with (warp_query).  The march, its lists and
// the distance bounds take t for a distance, which holds for rays of at most unit length (a
// shorter one moves less far than t): a longer one is answered by the tree, as from a dense
// cell.  The allowance is that of a direction normalised in float (dot3 within 7e-7 of 1); the
// plane distances of tri_c allow for twice as much.
constexpr float kUnitDot = 1.000001f;
__device__ __forceinline__ uint32_t query_word(const KParams &P, V3 p, V3 v)
{
    return dot3(v, v) > kUnitDot ? kCellDense << 24 : cell_at(P, p.x, p.y, p.z);
}

// Per-warp shared memory of warp_query: the rays and results of up to kQueue queries,
// and the list segments of one pass.
constexpr int kQueue = 16;
struct WarpQueue {
    float4 ray0[kQueue], ray1[kQueue];     // (p, v.x), (v.y, v.z, bound, ref_tri as int bits)
    unsigned long long best[kQueue];       // (t as float bits) << 32 | original index
    uint32_t safe[kQueue];                 // distance bound as float bits (>= 0)
    uint32_t seg[kQueue];                  // query << 27 | (first list entry - first item + kSegBias)
};
constexpr uint32_t kSegBias = 4096;        // above kQueue * kCellDense, so a segment's word is not negative
constexpr uint32_t kNoTri = 0x7fffffffu;
constexpr int kMarchMax = 512;             // cells of one march; a longer one goes to the BVH

// Distance along the ray to the grid's box (0 inside, kNoHit when the ray misses it).
__device__ __forceinline__ float grid_entry(const KParams &P, V3 p, V3 v)
{
    float t0 = 0.0f, t1 = kNoHit;
    const float o[3] = {P.g_ox, P.g_oy, P.g_oz}, q[3] = {p.x, p.y, p.z}, d[3] = {v.x, v.y, v.z};
    const int n[3] = {P.g_nx, P.g_ny, P.g_nz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float lo = o[a] - q[a], hi = o[a] + (float)n[a] * P.g_h - q[a];
        if (fabsf(d[a]) > 1e-30f) {
            const float x = lo / d[a], y = hi / d[a];
            t0 = fmaxf(t0, fminf(x, y));
            t1 = fminf(t1, fmaxf(x, y));
        } else if (lo > 0.0f || hi < 0.0f) {
            t0 = kNoHit;
        }
    }
    return t0 <= t1 ? t0 : kNoHit;
}

// The warp's nearest-triangle queries over the cell lists; every lane calls it, those with
// `want` have a query: the nearest triangle along (p, v) with t in (0, bound] and
// t < kNoHit, ref_tri excluded, equal distances resolving to the lower original index.
// Returns its original index or -1 with t_out = kNoHit.  word: query_word (cell_at for a
// direction known to be of unit length).
//
// A query marches along its ray.  At distance s it stands in a cell (word: the cell at
// s = 0), d from the cell's faces:
//   * a listed cell: its list holds every triangle touching the cell widened by
//     g_margin + g_eps, so every triangle the ray can meet up to s + g_margin + d - g_eps;
//     it is tested, and the march goes on from 15/16 of that distance;
//   * an empty cell: no triangle lies within g_margin + d - g_eps, nor within the word's
//     bound; the march goes on from 15/16 of the larger;
//   * outside the grid: on to the grid's box, or the end when the ray does not meet it.
// It ends when s has passed the bound or the nearest hit so far.  Most queries are
// decided by the list they start in (bound <= g_margin + d - g_eps).  For those, and for
// starts in an empty cell, `safe` (coming in with a lower bound already known, the photon's
// carried one) is raised to a lower bound of the distance from p to every triangle: g_margin
// + d - g_eps for the unlisted ones (or the empty cell's bound, if larger), the distance to
// their plane for the listed ones, |(G x E) . F| / |E x F|
// less a bound of the rounding of that product (tri_c.z = 1 / |E x F|, tri_c.w = the
// rounding factor per unit |G|, see lp_bvh.hpp), 0 on a triangle (ref_tri >= 0).
// Dense cells, marches past kMarchMax cells or stuck (lists without a margin), and a mesh
// without lists go to the BVH (used_bvh).  Same test and tie-break everywhere, and the
// lists' margins are wider than the BVH's boxes, so the hit is the BVH's bit for bit.
//
// About a tenth of the lanes have a query on the same step, each with a list of its own
// length, so a loop per lane leaves the warp nearly empty.  Here the triangles of all the
// warp's lists form one sequence of items and the 32 lanes test 32 items at a time, each
// with the ray of the item's query read from shared memory; hits and distance bounds meet
// in shared memory by atomic minimum, which no order can change.
//
// M and SM are the same view: M's members are the kernel's parameters, SM is its copy in
// shared memory for the out-of-line BVH descent, which needs an address (that of M would
// move M to local memory, and its pointers would be loaded from there for every item).
template <int STACK = kStackDepth>
__device__ __forceinline__ int warp_query(const KParams &P, const MeshView &M, const MeshView &SM, WarpQueue &Q,
                                          bool want, V3 p, V3 v, int ref_tri, float bound, uint32_t word, float &t_out,
                                          float &safe, bool &used_bvh)
{
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    int tri = -1;
    t_out = kNoHit;
    bool bvh = want && !P.cell_refs;
    unsigned todo = __ballot_sync(0xffffffffu, want && !bvh);
    while (todo) {
        const int rank = __popc(todo & lt_mask);
        const bool mine = ((todo >> lane) & 1u) && rank < kQueue;
        float s = 0.0f, limit = fminf(bound, kNoHit);
        int cells = 0;
        bool own = false;
        uint32_t cnt = 0, off = 0;   // each query's next list
        if (mine) {
            // the cell it starts in
            const float reach = P.g_margin + cell_face_distance(P, p.x, p.y, p.z) - P.g_eps;
            Q.ray0[rank] = make_float4(p.x, p.y, p.z, v.x);
            Q.ray1[rank] = make_float4(v.y, v.z, limit, __int_as_float(ref_tri));
            Q.best[rank] = ((unsigned long long)__float_as_uint(limit) << 32) | kNoTri;
            Q.safe[rank] = __float_as_uint(ref_tri < 0 ? fmaxf(reach, 0.0f) : 0.0f);
            if (!(word & kCellEmpty)) {
                cnt = (word >> 24) & 127u;
                off = word & 0xffffffu;
                bvh = cnt == kCellDense;
                own = bound <= reach && !bvh;
                s = 0.9375f * reach;
                if (!bvh && !LP_IN_RANGE(M.dbg, (int64_t)off + cnt - 1, P.n_cell_refs)) {
                    cnt = 0;
                    Q.safe[rank] = 0u;
                }
                if (!own && !(reach > 0.125f * P.g_h)) bvh = true;
                if (bvh) cnt = 0;
            } else if (!(word & kCellOutside)) {
                // no triangle within g_margin + d - g_eps, nor within the word's bound
                const float clear = fmaxf(reach, safe_distance(P, word));
                safe = fmaxf(safe, clear);
                s = 0.9375f * clear;
            }
        }
        const bool march = mine && !own;
        const bool marching = __any_sync(0xffffffffu, march);
        for (;;) {
            if (marching) {
                while (march && !bvh && cnt == 0 && s <= limit) {
                    const V3 q = v3(p.x + s * v.x, p.y + s * v.y, p.z + s * v.z);
                    const uint32_t w = cell_at(P, q.x, q.y, q.z);
                    float reach = P.g_margin + cell_face_distance(P, q.x, q.y, q.z) - P.g_eps;
                    if (w & kCellEmpty) {
                        if (w & kCellOutside) {
                            // just inside the box: its outermost cells hold no triangle
                            const float t = grid_entry(P, q, v);
                            reach = t < kNoHit ? t + 0.25f * P.g_h : 4.0f * kNoHit;
                        } else {
                            reach = fmaxf(reach, safe_distance(P, w));
                        }
                    } else {
                        cnt = (w >> 24) & 127u;
                        off = w & 0xffffffu;
                        bvh = cnt == kCellDense;
                        if (!LP_IN_RANGE(M.dbg, (int64_t)off + cnt - 1, P.n_cell_refs)) cnt = 0;
                    }
                    s += 0.9375f * reach;
                    if (++cells > kMarchMax || !(reach > 0.125f * P.g_h)) bvh = true;
                    if (bvh) cnt = 0;
                }
            }
            const unsigned segs = __ballot_sync(0xffffffffu, cnt > 0);
            if (!segs) break;
            uint32_t end = cnt;   // items up to and including this lane's
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= (unsigned)o) end += x;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
            const uint32_t start = end - cnt;
            if (cnt) Q.seg[__popc(segs & lt_mask)] = ((uint32_t)rank << 27) | (off + kSegBias - start);
            __syncwarp();
            for (uint32_t r = 0; r < total; r += 32) {
                // the segment of item r + lane: the last one that starts at or before it
                const bool here = cnt && start >= r && start < r + 32u;
                const unsigned heads = __reduce_or_sync(0xffffffffu, here ? 1u << (start - r) : 0u);
                const int before = __popc(__ballot_sync(0xffffffffu, cnt && start < r));
                const uint32_t item = r + lane;
                if (item < total) {
                    const uint32_t sg = Q.seg[before + __popc(heads & (lt_mask | (1u << lane))) - 1];
                    const uint32_t k = sg >> 27;
                    const int j = __ldg(P.cell_refs + ((sg & 0x7ffffffu) - kSegBias + item));
                    if (LP_IN_RANGE(M.dbg, j, M.n_tri)) {
                        const TriRec T = load_tri(P.tri, j);
                        const float4 r0 = Q.ray0[k], r1 = Q.ray1[k];
                        const V3 E = v3(T.a.w, T.b.x, T.b.y), F = v3(T.b.z, T.b.w, T.c.x);
                        const V3 G = sub3(v3(r0.x, r0.y, r0.z), v3(T.a.x, T.a.y, T.a.z));
                        const V3 GE = cross3(G, E);
                        const float t0 = dot3(GE, F);
                        const float d = fabsf(t0) * T.c.z - T.c.w * (fabsf(G.x) + fabsf(G.y) + fabsf(G.z));
                        atomicMin(&Q.safe[k], __float_as_uint(fmaxf(d, 0.0f)));
                        // most triangles' planes lie beyond the step (d bounds the distance
                        // from below, rounding included): nothing to hit
                        const int o = __float_as_int(T.c.y);
                        float t;
                        if (d <= r1.z && o != __float_as_int(r1.w) &&
                            tri_hit(M, E, F, G, GE, t0, v3(r0.w, r1.x, r1.y), r1.z, t) && t <= r1.z)
                            atomicMin(&Q.best[k], ((unsigned long long)__float_as_uint(t) << 32) | (unsigned)o);
                    } else {
                        atomicMin(&Q.safe[k], 0u);
                    }
                }
            }
            __syncwarp();
            if (!marching) break;
            cnt = 0;
            if (march) limit = __uint_as_float((uint32_t)(Q.best[rank] >> 32));
        }
        if (mine && !bvh) {
            const unsigned long long b = Q.best[rank];
            if ((uint32_t)b != kNoTri) {
                tri = (int)(uint32_t)b;
                t_out = __uint_as_float((uint32_t)(b >> 32));
            }
            if (own) safe = fmaxf(safe, fmaxf(__uint_as_float(Q.safe[rank]) - P.g_eps, 0.0f));
        }
        __syncwarp();
        todo &= ~__ballot_sync(0xffffffffu, mine);
    }
    if (bvh) {
        float t;   // the address of t_out would keep it in local memory
        tri = query_nearest<STACK>(SM, p, v, ref_tri, bound, t);
        t_out = t;
    }
    used_bvh = bvh;
    return tri;
}

// Lower bound of the distance from p to the triangle (a, a + ab, a + ac): the closest point q
// by Voronoi regions of the vertices, edges and face (Ericson, Real-Time Collision Detection,
// 2005), then the smallest of the vertices' distances along p - q, which no point of the
// triangle falls short of.  With the right q that is |p - q|; on slivers (aspect ratios from a
// few hundred on) the weights of q are lost in the rounding, and |p - q| can be far above the
// distance, where this stays below it (to the rounding of one product).
__device__ __forceinline__ float triangle_clearance(V3 p, V3 a, V3 ab, V3 ac)
{
    const V3 ap = sub3(p, a), bp = sub3(ap, ab), cp = sub3(ap, ac);
    const float d1 = dot3(ab, ap), d2 = dot3(ac, ap);
    const float d3 = dot3(ab, bp), d4 = dot3(ac, bp);
    const float d5 = dot3(ab, cp), d6 = dot3(ac, cp);
    const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
    float u, w;   // q = a + u ab + w ac
    if (d1 <= 0.0f && d2 <= 0.0f) {
        u = w = 0.0f;
    } else if (d3 >= 0.0f && d4 <= d3) {
        u = 1.0f;
        w = 0.0f;
    } else if (vc <= 0.0f && d1 >= 0.0f && d3 <= 0.0f) {
        u = d1 / (d1 - d3);
        w = 0.0f;
    } else if (d6 >= 0.0f && d5 <= d6) {
        u = 0.0f;
        w = 1.0f;
    } else if (vb <= 0.0f && d2 >= 0.0f && d6 <= 0.0f) {
        u = 0.0f;
        w = d2 / (d2 - d6);
    } else if (va <= 0.0f && (d4 - d3) >= 0.0f && (d5 - d6) >= 0.0f) {
        w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
        u = 1.0f - w;
    } else {
        const float den = 1.0f / (va + vb + vc);
        u = vb * den;
        w = vc * den;
    }
    const V3 d = sub3(sub3(ap, scl3(u, ab)), scl3(w, ac));
    const float m = fminf(fminf(dot3(d, ap), dot3(d, bp)), dot3(d, cp)) * rsqrtf(dot3(d, d));
    return m > 0.0f ? m : 0.0f;   // 0 too where q is not a number
}

__device__ __forceinline__ float box_dist2(float lo_x, float hi_x, float lo_y, float hi_y, float lo_z, float hi_z,
                                           V3 p)
{
    const float dx = fmaxf(fmaxf(lo_x - p.x, 0.0f), p.x - hi_x);
    const float dy = fmaxf(fmaxf(lo_y - p.y, 0.0f), p.y - hi_y);
    const float dz = fmaxf(fmaxf(lo_z - p.z, 0.0f), p.z - hi_z);
    return dx * dx + dy * dy + dz * dz;
}

// Lower bound of the distance from p to every triangle (triangle_clearance), at most cap; 0
// once it would be below `useful`.
// lp_run_noalloc, 50,000 photons, with the closest points' distances as they were / the bounds /
// the bounds behind the test of the plane: slab in 512 triangles 618 / 670 / 474 ms, in 2,048
// 1,823 / 2,079 / 1,417, abdomen in 3,600 251 / 258 / 235.
static __device__ __noinline__ float mesh_clearance(const MeshView &M, V3 p, float cap, float useful)
{
    float best = cap;
    int stack[kStackDepth];
    int sp = 0, node = 0;
    for (;;) {
        if (!LP_IN_RANGE(M.dbg, node, M.n_nodes)) return 0.0f;
        float4 a, b, c;
        int4 d;
        if (node < M.nodes_smem) {
            a = M.s_na[node]; b = M.s_nb[node]; c = M.s_nc[node]; d = M.s_nd[node];
        } else {
            a = __ldg(M.na + node); b = __ldg(M.nb + node); c = __ldg(M.nc + node); d = __ldg(M.nd + node);
        }
        const float dist[2] = {box_dist2(a.x, a.y, a.z, a.w, c.x, c.y, p), box_dist2(b.x, b.y, b.z, b.w, c.z, c.w, p)};
        const int ref[2] = {d.x, d.y};
        bool open[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const bool near = dist[k] < best * best;
            open[k] = near && ref[k] >= 0;
            if (!near || ref[k] >= 0) continue;
            const int e = ~ref[k], f = e >> 3, cnt = (e & 7) + 1;
            for (int j = f; j < f + cnt; ++j) {
                if (!LP_IN_RANGE(M.dbg, j, M.n_tri)) return 0.0f;
                TriRec T;
                if (j < M.tris_smem) T = TriRec{M.s_tri[3 * j], M.s_tri[3 * j + 1], M.s_tri[3 * j + 2]};
                else T = load_tri(M.tri, j);
                const V3 a = v3(T.a.x, T.a.y, T.a.z), E = v3(T.a.w, T.b.x, T.b.y), F = v3(T.b.z, T.b.w, T.c.x);
                // its plane's distance (see warp_query) is a bound too: good enough when hardly
                // below what there is
                const V3 G = sub3(p, a);
                const float d = fabsf(dot3(cross3(G, E), F)) * T.c.z - T.c.w * (fabsf(G.x) + fabsf(G.y) + fabsf(G.z));
                best = fminf(best, d >= 0.98f * best ? d : triangle_clearance(p, a, E, F));
                if (best < useful) return 0.0f;
            }
        }
        if (open[0] && open[1]) {
            const bool first0 = dist[0] <= dist[1];
            if (sp < kStackDepth) stack[sp++] = first0 ? d.y : d.x;
            node = first0 ? d.x : d.y;
        } else if (open[0] || open[1]) {
            node = open[0] ? d.x : d.y;
        } else {
            if (sp == 0) break;
            node = stack[--sp];
        }
    }
    return best;
}

// The warp's nearest-triangle queries on a mesh without a grid (lp_run_noalloc), as
// warp_query.  `safe` is raised to a lower bound of the distance from p to every triangle, so
// that the next steps need no query.
//   * Up to kWholeMesh triangles the warp takes its queries one after the other, each lane
//     testing every 32nd triangle: nearest hit, and the distance to the triangles' planes
//     (see warp_query), both reduced over the warp.
//   * Larger meshes, and hits of the ray itself, go to the tree: first the distance to the
//     nearest triangle, looked for as far as 32 mean steps (`mean`), then the ray, where the
//     step can reach that far.  A search that finds less than two mean steps is given up; where
//     steps are long for the mesh most are.  So each such one in a row doubles the number of the
//     photon's queries that go without (`rest`: still to go in bits 0-7, last number in bits
//     8-15), and a photon begins with kRestFirst of them.  In a transparent medium (mean = 0)
//     every step goes to the next face and needs no bound.  Abdomen, 3,600 triangles, scattering
//     as usual (50,000 photons) / a tenth / a fiftieth (200,000): ray alone 739 / 229 / 67 ms,
//     search on every query 235 / 403 / 189, this rule 203 / 271 / 76.
// Slab (32 triangles), 50,000 photons in reference arithmetic: 186 ms with a descent on every
// step, 118 with the tree's bounds, 55 with the whole mesh.  256 triangles of an abdomen: 82 ms
// through the tree, 46 with the whole mesh, so kWholeMesh is on the safe side (400 of them: 114
// and 82).
constexpr int kWholeMesh = 256;
constexpr uint32_t kRestFirst = 31, kRestMost = 63;
template <int STACK = kStackDepth>
__device__ __forceinline__ int mesh_query(const KParams &P, const MeshView &SM, bool want, V3 p, V3 v, int ref_tri,
                                          float bound, float mean, float &t_out, float &safe, uint32_t &rest)
{
    const int lane = threadIdx.x & 31;
    const float eps = __ldg(P.mesh_eps);
    int tri = -1;
    t_out = kNoHit;
    const bool longer = dot3(v, v) > kUnitDot;   // than unit (query_word): no bound, the tree
    if (P.n_tri > kWholeMesh || __any_sync(0xffffffffu, want && longer)) {
        if (want) {
            bool ray = true;
            if (ref_tri < 0 && !longer && mean > 0.0f) {
                if (rest & 0xffu) {
                    --rest;
                } else {
                    const float clear = mesh_clearance(SM, p, fminf(32.0f * mean, kNoHit), 2.0f * mean) * 0.9999f - eps;
                    safe = fmaxf(safe, clear);
                    ray = !(bound < clear);
                    const uint32_t n = clear < 2.0f * mean ? min(2u * (rest >> 8) + 1u, kRestMost) : 0u;
                    rest = n << 8 | n;
                }
            }
            if (ray) tri = query_nearest<STACK>(SM, p, v, ref_tri, bound, t_out);
        }
        return tri;
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, want); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const V3 o = v3(__shfl_sync(0xffffffffu, p.x, src), __shfl_sync(0xffffffffu, p.y, src),
                        __shfl_sync(0xffffffffu, p.z, src));
        const V3 r = v3(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                        __shfl_sync(0xffffffffu, v.z, src));
        const int skip = __shfl_sync(0xffffffffu, ref_tri, src);
        float best = fminf(__shfl_sync(0xffffffffu, bound, src), kNoHit);
        float clear = 3.0e38f;
        int id = (int)kNoTri;
        for (int j = lane; j < P.n_tri; j += 32) {
            TriRec T;
            if (j < SM.tris_smem) T = TriRec{SM.s_tri[3 * j], SM.s_tri[3 * j + 1], SM.s_tri[3 * j + 2]};
            else T = load_tri(P.tri, j);
            const V3 E = v3(T.a.w, T.b.x, T.b.y), F = v3(T.b.z, T.b.w, T.c.x);
            const V3 G = sub3(o, v3(T.a.x, T.a.y, T.a.z));
            const V3 GE = cross3(G, E);
            const float t0 = dot3(GE, F);
            const float d = fabsf(t0) * T.c.z - T.c.w * (fabsf(G.x) + fabsf(G.y) + fabsf(G.z));
            clear = fminf(clear, fmaxf(d, 0.0f));
            const int i = __float_as_int(T.c.y);
            float t;
            if (d <= best && i != skip && tri_hit(SM, E, F, G, GE, t0, r, best, t) &&
                (t < best || (t == best && i < id))) {
                best = t;
                id = i;
            }
        }
        const uint32_t t_min = __reduce_min_sync(0xffffffffu, id != (int)kNoTri ? __float_as_uint(best) : 0x7f800000u);
        const uint32_t i_min = __reduce_min_sync(0xffffffffu, __float_as_uint(best) == t_min ? (uint32_t)id : kNoTri);
        const float c_min = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(clear)));
        if (lane == src) {
            if (i_min != kNoTri) {
                tri = (int)i_min;
                t_out = __uint_as_float(t_min);
            }
            if (ref_tri < 0) safe = fmaxf(safe, c_min - eps);
        }
    }
    return tri;
}

}  // namespace lp
