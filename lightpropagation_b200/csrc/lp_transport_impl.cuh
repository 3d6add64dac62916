// lp_transport_impl.cuh -- persistent photon-transport kernel for sm_100a.
//
// One CUDA thread carries one photon packet at a time, as one OpenCL work-item does
// in the reference (src/Simulation/MCLightPropagation.cl:1262-1606).  The grid is
// persistent: each warp refills the lanes whose photon has finished with new photon
// ids taken from a global counter, one atomicAdd per warp refill, so lanes stay busy
// until the photon budget is spent.  Photon i draws its random numbers from Philox
// blocks (key = seed, counter = (i, event, stream)), one per event, so results do not
// depend on which thread traced which photon, nor on whether its own lane drew the event or
// an idle one did some events ahead (next_draws).
//
// Per loop iteration (MCLightPropagation.cl:1375-1575), the warp's lanes together:
//   step length (.cl:1405-1442) -> nearest triangle within the step (replaces the O(T)
//   FindTriangleInPath, .cl:1037-1093; skipped by distance bounds, or answered by the
//   whole warp from the cell lists) -> boundary (TransmitOrReflect, .cl:921-1018) or
//   absorb + Henyey-Greenstein scatter + absorption tallies (.cl:1513-1537) -> roulette
//   (.cl:1539-1545).
// At the end of a photon its exit record (.cl:1583-1594) is binned on the device into
// the reference's SFT and RTd images (CalculatePropagation.cpp:1553-1626).
//
// What bounds it: the instructions of one step, 400 to 500 of them in one chain that
// branches on its own results.  A warp with one photon left issues one every 4 to 5
// cycles (fixed latencies and the special-function unit), so short runs and the ends of
// long ones wait for their longest photon; full warps (20 per SM at 96 registers) issue
// two cycles of three.  Hence the form of the step: selects instead of branches where both
// sides are a few operations, round keys and derived constants in the kernel's parameters,
// 32-bit indices, two 16-byte loads for a medium's factors, no counter that another one
// implies; no branch between the move and the deposits (square roots without a slow path,
// no test for a voxel grid), so that the chains of direction, tallies and the next cell
// word overlap; and random numbers drawn several events ahead once lanes are idle
// (next_draws); the lanes without a photon run along, and rare ends (roulette, step cap)
// share one branch.  One photon alone takes 0.65 us a step on the slab (1.20 before these),
// 0.73 on the curved abdomen (1.36; 0.60 and 0.67 without spills); slab, 1e6 photons, 114 -> 90 ms; abdomen at 660 nm,
// 3e6 photons, 201 -> 175 ms; 1e5 photons 40 -> 24 ms.
//
// Exact = true  keeps the reference's arithmetic operation by operation (compiled
//               with --fmad=false): a photon follows the oracle's trajectory for the
//               same random numbers up to last-place differences of logf/cosf/acosf.
// Exact = false (production) computes the same physics with fewer operations:
//               Henyey-Greenstein sampling with precomputed factors, the direction-
//               cosine update of Wang et al. (MCML, 1995) instead of two Rodrigues
//               rotations (same distribution: polar angle from HG, uniform azimuth),
//               vector refraction/reflection, reciprocal multiplies, explicit fused
//               multiply-adds.  No unit lets the compiler contract on its own, so a
//               device function gives the same bits in every kernel that inlines it.
#pragma once
#include <algorithm>
#include <mutex>

#include "lp_kernel.cuh"

namespace lp {

constexpr int kBlock = 128;
// Resident blocks per SM the single-instance kernel is compiled for (register budget
// 65536 / (kBlock x this)); the batched kernel's configurations are autotuned instead.  Five
// of 128 threads leave 96 registers, 20 warps per SM.  Slab 1e6 photons / curved abdomen 660
// nm 3e6 and 5e5, ms: 83.5 / 170 / 45.2; three of 256 (80 registers, 24 warps, spills) 86.2 /
// 173 / 49.0; eleven of 64 (88) 87.9 / 180 / 49.8.  Short runs use four (128, no spills).
#ifndef LP_TRANSPORT_MIN_BLOCKS
#define LP_TRANSPORT_MIN_BLOCKS 5
#endif
constexpr int kFewBlocks = 4;   // 16 warps, as plan_launch

struct Photon {
    float px, py, pz, vx, vy, vz;
    float w, unfin;          // unfin: residual step; the exit weight once the photon has left
    float absorbed;
    int32_t last_tri;        // face of the last boundary event, -1 before any: its normal is
                             // CalcAlphaOut's (.cl:1583), see photon_normal
    int32_t curr;
    uint32_t steps;
    uint32_t flags;          // see F_*, EXIT_SHIFT, AXIS_SHIFT
    unsigned long long region_acc;
    uint32_t idx;            // photon index within the launch: the photon id is P.first + idx
    float seg_len;           // differentiation: path length and interactions in the
    uint32_t seg_k;          // current region since the photon entered it
    float safe;              // lower bound of the distance from the position to any triangle
    uint32_t word;           // cell word at the position (cell_at); without a grid mesh_query's `rest`
};

// Per-photon, per-region path lengths and interaction counts of a differentiated run
// (thread-local, indexed by region id).
struct GradAcc {
    float L[kGradRegions];
    uint32_t k[kGradRegions];
};
// flags: bit 0 traversedFetalTissue, bit 1 the photon is on last_tri (refTri of the
// reference: no scattering since the boundary event), bits 2-3 exit kind, bits 4-5 the
// on-axis normal override at the last boundary (0 none, 1 +eZ, 2 -eZ, 3 zero vector).
// The reference's roulette flag is left out: it is clear only when the weight is 0.
enum : uint32_t { F_FETAL = 1u, F_ON_FACE = 2u, EXIT_SHIFT = 2, AXIS_SHIFT = 4 };
enum : uint32_t { EXIT_NONE = 0, EXIT_SURF = 1, EXIT_SURF_FETAL = 2, EXIT_TRANS = 3 };

// steps: of the finished photons.  Each step is a scatter or a boundary event, and has a
// query or skips it, so the other two counts follow.
struct Counters {
    uint32_t steps, boundary, query, roulette, rz_drop, vox_drop, bvh;
    __device__ __forceinline__ uint32_t scatter() const { return steps - boundary; }
    __device__ __forceinline__ uint32_t skip() const { return steps - query; }
};

// Rotate (.cl:697-708)
__device__ __forceinline__ V3 rotate(V3 vec, V3 axis, float c, float s)
{
    const float nDx = dot3(axis, vec);
    const V3 nXx = cross3(axis, vec);
    const V3 nXxXn = cross3(nXx, axis);
    return add3(add3(scl3(nDx, axis), scl3(c, nXxXn)), scl3(s, nXx));
}

// 1 / sqrt(x) of the special-function unit, for normal x (rsqrtf without its handling of
// denormals: the same bits).
__device__ __forceinline__ float rsqrt_normal(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The correctly rounded square root for x >= 1e-30, 0 from 0 to there: one Newton correction of
// x / sqrt(x) with fused multiply-adds (Markstein, IBM J. Res. Dev. 34, 1990).  Compared
// with sqrtf for every float from 1e-30 to 3e38.  Unlike sqrtf it has no branch to a slow
// path, which would cut the step's straight line of code.
__device__ __forceinline__ float sqrt_normal(float x)
{
    const float y = rsqrt_normal(x), s = x * y;
    const float r = __fmaf_rn(__fmaf_rn(-s, s, x), 0.5f * y, s);
    // one unsigned comparison for 0 <= x < 1e-30; negative x and NaN stay NaN, as sqrtf has them
    return __float_as_uint(x) < 0x0DA24260u ? 0.0f : r;
}

// 1 / b correctly rounded, for 2^-100 <= |b| <= 2^100: one Newton step from the
// special-function unit's reciprocal.  Compared with the division operator for every float
// of the range.
__device__ __forceinline__ float rcp_rn(float b)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return __fmaf_rn(y, __fmaf_rn(-b, y, 1.0f), y);
}

// a / b correctly rounded, y = 1 / b correctly rounded: Markstein's theorem (IBM J. Res. Dev.
// 34, 1990; the first correction brings the quotient within a unit, the second rounds it),
// compared with the division operator for 1.2e11 pairs.  For the reference arithmetic, whose
// step has 19 divisions, most by a constant of the run or three by the same length; the
// operator's slow path is a branch for each.  1e5 slab photons 48.4 -> 45.9 ms.
__device__ __forceinline__ float div_rn(float a, float b, float y)
{
    const float q0 = a * y;
    float q = __fmaf_rn(__fmaf_rn(-b, q0, a), y, q0);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return q0 == 0.0f ? q0 : q;
}

// norm3 of the reference arithmetic's scattering, bit for bit.
__device__ __forceinline__ V3 norm3_rn(V3 v)
{
    const float d = dot3(v, v);
    if (!(d >= 1e-20f && d <= 1e20f)) return norm3(v);
    const float l = sqrt_normal(d), y = rcp_rn(l);
    return v3(div_rn(v.x, l, y), div_rn(v.y, l, y), div_rn(v.z, l, y));
}

__device__ __forceinline__ V3 fast_norm(V3 v)
{
    const float r = rsqrt_normal(__fmaf_rn(v.x, v.x, __fmaf_rn(v.y, v.y, v.z * v.z)));
    return v3(v.x * r, v.y * r, v.z * r);
}

template <bool Exact>
__device__ __forceinline__ float hg_cos_theta(const Medium &m, float xi)
{
    float cosTheta;
    if (Exact) {
        // VScatter (.cl:625-634)
        const float g = m.g;
        const float den = 1.0f - g + 2.0f * g * xi;
        if (m.kind & kPlainDiv) {
            const float g1 = (1.0f - g * g) / den;
            cosTheta = (1.0f + g * g - g1 * g1) / (2.0f * g);
        } else {
            const float g1 = div_rn(1.0f - g * g, den, rcp_rn(den));
            cosTheta = div_rn(1.0f + g * g - g1 * g1, 2.0f * g, m.hg_inv2g);
        }
        if (g == 0.0f) cosTheta = 2.0f * xi - 1.0f;
    } else {
        // both cases and a select: the step loop pays more for a branch
        const float g1 = __fdividef(m.hg_a, __fmaf_rn(m.hg_c, xi, m.hg_b));
        cosTheta = __fmaf_rn(-g1, g1, m.hg_d) * m.hg_inv2g;
        if (m.hg_c == 0.0f) cosTheta = __fmaf_rn(2.0f, xi, -1.0f);
    }
    return fminf(fmaxf(cosTheta, -1.0f), 1.0f);
}

// Cosine and sine of the azimuth of the uniform xp.
template <bool Exact>
__device__ __forceinline__ void azimuth(float xp, float &cosPsi, float &sinPsi)
{
    if (Exact) {
        const float psi = 2.0f * 3.14159265358979323846f * xp;
        cosPsi = cosf(psi);
        sinPsi = sqrt_normal(1.0f - cosPsi * cosPsi);
        if (psi > 3.14159265358979323846f) sinPsi *= -1.0f;
    } else {
        sincospif(2.0f * xp, &sinPsi, &cosPsi);
    }
}

// What a step takes from its event's random numbers (EventRng): -log of the first, the
// second (polar angle or Fresnel), the azimuth of the third, the fourth (roulette).  None
// of it depends on the photon's state, only on its index and step number.
struct Draws {
    float neg_log, u1, cos_psi, sin_psi, u3;
};
template <bool Exact>
__device__ __forceinline__ Draws make_draws(const KParams &P, uint32_t idx, uint32_t event)
{
    EventRng rng;
    rng.draw(P, idx, event);
    Draws d;
    d.neg_log = -logf(rng.u0);
    d.u1 = rng.u1;
    azimuth<Exact>(rng.u2, d.cos_psi, d.sin_psi);
    d.u3 = rng.u3;
    return d;
}

// The warp's draws.  A warp of 17 to 32 photons draws one event for each, every lane its
// own.  With fewer photons the idle lanes draw the following events: each of k photons
// gets `span` lanes (the largest power of two with k span <= 32), the draws of its next
// `span` events go through shared memory, and the warp draws again when those are used
// up.  Philox, logarithm and azimuth are a quarter of a step's instructions; the end of a
// run, when each warp waits for its last photons, and short runs pay for them once in up
// to 32 steps.
struct WarpDraws {
    float v[5][32];
};
// next: the lane's next column of WarpDraws, plus 256 times the events drawn and not used
// yet (the same for the whole warp; below 256 the warp has to draw, 0 to begin with).
template <bool Exact>
__device__ __forceinline__ Draws next_draws(const KParams &P, WarpDraws &W, unsigned live, bool alive, uint32_t idx,
                                            uint32_t steps, uint32_t &next)
{
    Draws d;
    if (next < 256u) {
        const unsigned lane = threadIdx.x & 31u;
        const int span_log = __clz(max(__popc(live), 1) - 1) - 27;   // 5 for one photon (clz(0) = 32), 0 from 17 on
        uint32_t event = steps + 1u;
        next = 0;
        if (span_log > 0) {
            const unsigned rank = __popc(live & ((1u << lane) - 1u));
            next = (256u << span_log) + ((rank << span_log) & 31u);
            __syncwarp();
            if (alive) {
                W.v[0][rank] = __uint_as_float(idx);
                W.v[1][rank] = __uint_as_float(event);
            }
            __syncwarp();
            idx = __float_as_uint(W.v[0][lane >> span_log]);
            event = __float_as_uint(W.v[1][lane >> span_log]) + (lane & ((1u << span_log) - 1u));
            __syncwarp();
        }
        d = make_draws<Exact>(P, idx, event);
        if (span_log > 0) {
            W.v[0][lane] = d.neg_log;
            W.v[1][lane] = d.u1;
            W.v[2][lane] = d.cos_psi;
            W.v[3][lane] = d.sin_psi;
            W.v[4][lane] = d.u3;
            __syncwarp();
        }
    }
    // read and selected on every step: cheaper for the last photons than a branch (1000 slab
    // photons 10.5 -> 9.9 ms), and as good for full warps
    const uint32_t s = next & 31u;
    const bool shared = next >= 256u;
    const Draws e = {W.v[0][s], W.v[1][s], W.v[2][s], W.v[3][s], W.v[4][s]};
    next += shared ? 1u - 256u : 0u;
    d.neg_log = shared ? e.neg_log : d.neg_log;
    d.u1 = shared ? e.u1 : d.u1;
    d.cos_psi = shared ? e.cos_psi : d.cos_psi;
    d.sin_psi = shared ? e.sin_psi : d.sin_psi;
    d.u3 = shared ? e.u3 : d.u3;
    return d;
}

template <bool Exact>
__device__ __forceinline__ V3 scatter_direction(V3 v, const Medium &m, float xt, float cosPsi, float sinPsi)
{
    const float cosTheta = hg_cos_theta<Exact>(m, xt);
    if (Exact) {
        // VScatter (.cl:597-655): rotate by theta about e_rot _|_ v, then by psi about v
        V3 e_rot = v3(0.0f, 0.0f, 0.0f);
        if (v.z != 0.0f) {
            const float a = -(v.x + v.y);
            const float z = fabsf(v.z) > 1e-15f ? div_rn(a, v.z, rcp_rn(v.z)) : a / v.z;
            e_rot = v3(1.0f, 1.0f, z);
        } else if (v.y != 0.0f) {
            const float y = -(v.x) / (v.y);
            e_rot = v3(1.0f, y, 0.0f);
        } else if (v.x != 0.0f) {
            e_rot = v3(0.0f, 1.0f, 0.0f);
        }
        e_rot = norm3_rn(e_rot);
        const float sinTheta = sqrt_normal(1.0f - cosTheta * cosTheta);
        const V3 rot_theta = norm3_rn(rotate(v, e_rot, cosTheta, sinTheta));
        return norm3_rn(rotate(rot_theta, v, cosPsi, sinPsi));
    } else {
        // direction-cosine update (Wang, Jacques & Zheng, MCML 1995).  1 - uz^2 is taken
        // as ux^2 + uy^2 (|v| = 1), which keeps its precision near the z axis where the
        // difference form cancels; the axial case scatters about z with uz' = sign(uz) cos.
        const float sinTheta = sqrt_normal(fmaxf(0.0f, __fmaf_rn(-cosTheta, cosTheta, 1.0f)));
        const float uz2 = __fmaf_rn(v.x, v.x, v.y * v.y);
        const float it = rsqrt_normal(uz2);
        const float temp = uz2 * it;  // sqrt(1 - uz^2)
        const float st = sinTheta * it;
        const float ax = sinTheta * cosPsi;
        V3 r = v3(__fmaf_rn(st, __fmaf_rn(v.x * v.z, cosPsi, -v.y * sinPsi), v.x * cosTheta),
                  __fmaf_rn(st, __fmaf_rn(v.y * v.z, cosPsi, v.x * sinPsi), v.y * cosTheta),
                  __fmaf_rn(-ax, temp, v.z * cosTheta));
        // the axial case by selects (it and temp are not finite there): a branch costs more
        const bool axial = uz2 < 1e-20f;
        r.x = axial ? ax : r.x;
        r.y = axial ? sinTheta * sinPsi : r.y;
        r.z = axial ? (v.z > 0.0f ? cosTheta : -cosTheta) : r.z;
        return fast_norm(r);
    }
}

// GetFresnel (.cl:857-907)
__device__ __forceinline__ float fresnel(float n1, float n2, float cosIn)
{
    float r;
    if (n1 == n2) {
        r = 0.0f;
    } else if (fabsf(cosIn) == 1.0f) {
        r = (n1 - n2) / (n1 + n2);
        r *= r;
    } else if (cosIn == 0.0f) {
        r = 1.0f;
    } else {
        const float sinIn = sqrtf(1.0f - cosIn * cosIn);
        const float sinOut = n1 * sinIn / n2;
        if (sinOut >= 1.0f) {
            r = 1.0f;
        } else {
            const float cosOut = sqrtf(1.0f - sinOut * sinOut);
            const float cap = cosIn * cosOut - sinIn * sinOut;
            const float cam = cosIn * cosOut + sinIn * sinOut;
            const float sap = sinIn * cosOut + cosIn * sinOut;
            const float sam = sinIn * cosOut - cosIn * sinOut;
            r = 0.5f * (sam * sam) * ((cam * cam) + (cap * cap)) / ((sap * sap) * (cam * cam));
        }
    }
    return r;
}

// Sum of x over the lanes of grp (a __match_any_sync group, every lane of it calling),
// exact for x < 2^59: the three slices x[0:16], x[16:32], x[32:64] are reduced by
// redux.sync, and each slice's sum over at most 32 lanes fits in 32 bits.
__device__ __forceinline__ unsigned long long group_sum_u64(unsigned grp, unsigned long long x)
{
    if ((grp & (grp - 1u)) == 0u) return x;   // a group of one, as most are
    const unsigned a = __reduce_add_sync(grp, (unsigned)(x & 0xffffull));
    const unsigned b = __reduce_add_sync(grp, (unsigned)((x >> 16) & 0xffffull));
    const unsigned c = __reduce_add_sync(grp, (unsigned)(x >> 32));
    return (unsigned long long)a + ((unsigned long long)b << 16) + ((unsigned long long)c << 32);
}

__device__ __forceinline__ void add_fix(unsigned long long *a, float w)
{
    const unsigned long long f = fix32(w);
    if (f) atomicAdd(a, f);
}

// Differentiation: the photon scored surface weight s in ring d.  With path density
// prod_r mus_r^k_r exp(-(mua_r + mus_r) L_r / factor) times the albedo weights, the
// score's derivatives are s * (-L_r / factor) for mua_r and s * (k_r / mus_r - L_r / factor)
// for mus_r (perturbation Monte Carlo, Hayakawa et al., Opt. Lett. 26, 2001); the
// kernel accumulates the moments of s L_r and s k_r, the host forms the derivatives.
static __device__ __noinline__ void score_gradient(const KParams &P, const GradAcc &ga, int d, float s)
{
    double *g = P.grad + 5 * (int64_t)d * P.n_media;
    for (int r = 0; r < P.n_media; ++r) {
        const double a = (double)s * (double)ga.L[r];
        const double b = (double)s * (double)ga.k[r];
        if (a == 0.0 && b == 0.0) continue;
        atomicAdd(g + 5 * r + 0, a);
        atomicAdd(g + 5 * r + 1, b);
        atomicAdd(g + 5 * r + 2, a * a);
        atomicAdd(g + 5 * r + 3, b * b);
        atomicAdd(g + 5 * r + 4, a * b);
    }
}

// What an exit record needs of a photon, passed by value: a reference would take the
// photon's address out of the step loop, and every step would then store it to local
// memory.
struct ExitState {
    float px, py, pz, vx, vy, vz, exit_w;
    int32_t last_tri;
    uint32_t flags, idx;
};
__device__ __forceinline__ ExitState exit_state(const Photon &ph)
{
    return ExitState{ph.px, ph.py, ph.pz, ph.vx, ph.vy, ph.vz, ph.unfin, ph.last_tri, ph.flags, ph.idx};
}

// The normal of the photon's last boundary event as the transport used it: the face's unit
// normal, the on-axis override (sign * eZ), or (0, 0, -1) before any event (PhotonClass
// init, .cl:344-389).  Kept as the face index and two flag bits instead of three floats.
__device__ __forceinline__ V3 photon_normal(const KParams &P, const ExitState &ph)
{
    const uint32_t axis = (ph.flags >> AXIS_SHIFT) & 3u;
    if (axis) {
        const float sg = axis == 1u ? 1.0f : (axis == 2u ? -1.0f : 0.0f);
        return scl3(sg, v3(P.nzx, P.nzy, P.nzz));
    }
    if (ph.last_tri < 0) return v3(0.0f, 0.0f, -1.0f);
    const float4 at = __ldg(P.tri_attr + ph.last_tri);
    return v3(at.x, at.y, at.z);
}

// Exit record binning of CalculatePropagation.cpp:1553-1626 plus radial bins and rings.
template <bool Grad>
static __device__ __noinline__ void finish_photon(const KParams &P, const ExitState ph, const GradAcc *ga)
{
    const V3 v = v3(ph.vx, ph.vy, ph.vz), nv = photon_normal(P, ph);
    const float alpha = fabsf(acosf(dot3(v, nv)));
    const V3 d = v3(P.poix - ph.px, P.poiy - ph.py, P.poiz - ph.pz);
    const float radius = sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
    const V3 pr = v3(ph.px - P.poix, ph.py - P.poiy, ph.pz - P.poiz);
    const float cx = dot3(v3(P.nxx, P.nxy, P.nxz), pr);
    const float cy = dot3(v3(P.nyx, P.nyy, P.nyz), pr);
    const float cz = dot3(v3(P.nzx, P.nzy, P.nzz), pr);
    const uint32_t kind = (ph.flags >> EXIT_SHIFT) & 3u;
    const float s = (kind == EXIT_SURF || kind == EXIT_SURF_FETAL) ? ph.exit_w : 0.0f;
    const float f = (kind == EXIT_SURF_FETAL) ? ph.exit_w : 0.0f;
    const float t = (kind == EXIT_TRANS) ? ph.exit_w : 0.0f;
    const int64_t slot = (int64_t)ph.idx;
    if (P.exit_rec && slot >= 0 && slot < P.exit_cap) {
        float4 *r = reinterpret_cast<float4 *>(P.exit_rec + 8 * slot);
        r[0] = make_float4(cx, cy, cz, s);
        r[1] = make_float4(f, t, alpha, radius);
    }
    if (kind == EXIT_NONE) return;
    int x = trunc_sat(cx / P.dg[0]);
    int y = trunc_sat(cy / P.dg[1]);
    y = min(max(y, -P.hy), P.hy);
    x = min(max(x, -P.hx), P.hx);
    unsigned long long *c = P.sft + 3 * ((int64_t)(y + P.hy) * P.sft_nx + (x + P.hx));
    add_fix(c + 0, s);
    add_fix(c + 1, f);
    add_fix(c + 2, t);
    int ai = trunc_sat_d(((double)(alpha * 180.0f) / 3.14159265358979323846) / (double)P.dg[5]);
    int ri = trunc_sat(radius / P.dg[3]);
    if (ri > P.dimR - 1) ri = P.dimR - 1;
    else if (ri < 0) ri = 0;
    if (ai > P.dimAlpha - 1) ai = P.dimAlpha - 1;
    else if (ai < 0) ai = 0;
    unsigned long long *r = P.rtd + 3 * ((int64_t)ai * P.dimR + ri);
    add_fix(r + 0, s);
    add_fix(r + 1, f);
    add_fix(r + 2, t);
    const float rho = sqrtf(cx * cx + cy * cy);
    if (P.n_rbins > 0) {
        const int b = trunc_sat(rho / P.rbin_dr);
        if (b >= 0 && b < P.n_rbins) {
            add_fix(P.rbins + 2 * b, s);
            add_fix(P.rbins + 2 * b + 1, t);
        }
    }
    if (s > 0.0f) {
        for (int k = 0; k < P.n_det; ++k) {
            if (rho >= P.det_lo[k] && rho < P.det_hi[k]) {
                add_fix(P.det + 2 * k, s);
                add_fix(P.det + 2 * k + 1, s * s);
                if (Grad) score_gradient(P, *ga, k, s);
            }
        }
    }
}

__device__ __forceinline__ void start_photon(const KParams &P, Photon &ph, uint32_t idx)
{
    // PhotonClass::Init (.cl:344-389) with vStart[0] (.cl:429-467)
    ph.px = P.p0x; ph.py = P.p0y; ph.pz = P.p0z;
    ph.vx = P.v0x; ph.vy = P.v0y; ph.vz = P.v0z;
    if (P.src_type == 1) {
        // fibre source (no reference counterpart), event 0: disk of radius src_radius in
        // the (eX, eY) plane, direction uniform in solid angle within the cone about eZ
        EventRng rng;
        rng.draw(P, idx, 0u);
        const V3 ex = v3(P.nxx, P.nxy, P.nxz), ey = v3(P.nyx, P.nyy, P.nyz), ez = v3(P.nzx, P.nzy, P.nzz);
        const float r = P.src_radius * sqrtf(rng.u0);
        const float phi = 2.0f * 3.14159265358979323846f * rng.u1;
        const float cp = cosf(phi), sp = sinf(phi);
        const V3 p = add3(v3(ph.px, ph.py, ph.pz), add3(scl3(r * cp, ex), scl3(r * sp, ey)));
        ph.px = p.x; ph.py = p.y; ph.pz = p.z;
        const float ct = 1.0f - rng.u2 * (1.0f - P.src_cos_max);
        const float stt = sqrtf(1.0f - ct * ct);
        const float psi = 2.0f * 3.14159265358979323846f * rng.u3;
        const float cq = cosf(psi), sq = sinf(psi);
        const V3 v = norm3(add3(scl3(ct, ez), add3(scl3(stt * cq, ex), scl3(stt * sq, ey))));
        ph.vx = v.x; ph.vy = v.y; ph.vz = v.z;
    }
    ph.w = P.w0;
    ph.unfin = 0.0f;
    ph.absorbed = 0.0f;
    ph.last_tri = -1;
    ph.curr = 0;
    ph.steps = 0;
    ph.flags = 0;
    ph.region_acc = 0;
    ph.idx = idx;
    ph.seg_len = 0.0f;
    ph.seg_k = 0;
    ph.safe = 0.0f;
    // a source's direction is taken as given: one longer than unit is kept until the first
    // event, so its first step needs the tree (and no distance bound: a dense cell has none)
    ph.word = query_word(P, v3(ph.px, ph.py, ph.pz), v3(ph.vx, ph.vy, ph.vz));
}

// A boundary event (.cl:1443-1465 with TransmitOrReflect, .cl:921-1018): the photon moves
// thit to the face `tri` (-1: no face, it leaves the model), then is transmitted or
// reflected with probability from the Fresnel equations (xi against R).  Inline, although it
// runs about once per hundred steps: the photon goes in and comes back by value, and out of
// line that would be a copy of it through local memory.
template <bool Exact, bool Grad>
static __device__ __forceinline__ Photon boundary_event(const KParams &P, const Medium *s_media,
                                                     unsigned long long *s_region, unsigned long long *s_cnt,
                                                     Photon ph, GradAcc *ga, int tri, float thit, float step,
                                                     float xi)
{
    [[maybe_unused]] unsigned long long *const dbg = P.counters ? P.counters + kBoundsCounter : nullptr;
    const Medium m = s_media[ph.curr];
    const V3 v = v3(ph.vx, ph.vy, ph.vz);
    ph.safe = 0.0f;
    ph.px = ph.px + thit * ph.vx;
    ph.py = ph.py + thit * ph.vy;
    ph.pz = ph.pz + thit * ph.vz;
    ph.flags &= ~F_ON_FACE;
    if (tri < 0) {
        // the reference would read mediumIDs[-1] here; the photon leaves the model
        atomicAdd(s_cnt + 4, 1ull);
        ph.w = 0.0f;
    } else if (LP_IN_RANGE(dbg, tri, P.n_tri)) {
        const float4 at = __ldg(P.tri_attr + tri);
        const int ids = __float_as_int(at.w);
        const int inner = ids & 0xffff, outer = ids >> 16;
        V3 nv = v3(at.x, at.y, at.z);
        int nxt_id = (ph.curr == outer) ? inner : outer;
        // a photon whose region is neither side of the face it meets has passed through
        // another face unseen (a crack between triangles that the float test leaves)
        if (ph.curr != inner && ph.curr != outer) atomicAdd(s_cnt + 14, 1ull);
        if (!LP_IN_RANGE(dbg, nxt_id, P.n_media)) nxt_id = ph.curr;
        const Medium nx = s_media[nxt_id];
        uint32_t axis = 0u;
        if (P.compat & 0x2u) {
            if (fabsf(sqrtf(ph.px * ph.px + ph.py * ph.py)) < 0.01f) {
                const float sg = sign_cl(dot3(nv, v3(P.ezx, P.ezy, P.ezz)));
                nv = scl3(sg, v3(P.nzx, P.nzy, P.nzz));
                axis = sg > 0.0f ? 1u : (sg < 0.0f ? 2u : 3u);
            }
        }
        ph.last_tri = tri;
        ph.flags = (ph.flags & ~(3u << AXIS_SHIFT)) | (axis << AXIS_SHIFT);
        // TransmitOrReflect (.cl:921-1018)
        const float cosIn = dot3(nv, v);
        const float absCosIn = fabsf(cosIn);
        const float n1 = m.n, n2 = nx.n;
        float cos_crit = 0.0f;
        if (n1 > n2) cos_crit = sqrtf(1.0f - (n2 / n1) * (n2 / n1));
        float r;
        if (absCosIn <= cos_crit) r = 1.0f;
        else r = fresnel(n1, n2, (P.compat & 0x4u) ? cosIn : absCosIn);
        int newID;
        float muaNew, musNew;
        V3 vout;
        if (Exact) {
            const V3 e_y = norm3(cross3(nv, cross3(nv, v)));
            if (xi > r) {
                const float sinT = sqrtf(1.0f - cosIn * cosIn) * n1 / n2;
                float cosT = -sqrtf(1.0f - sinT * sinT);
                if (cosIn > 0.0f) cosT = fabsf(cosT);
                vout = norm3(sub3(scl3(cosT, nv), scl3(sinT, e_y)));
            } else {
                const float sinR = sqrtf(1.0f - cosIn * cosIn);
                const V3 t = norm3(add3(scl3(cosIn, nv), scl3(sinR, e_y)));
                vout = v3(-t.x, -t.y, -t.z);
            }
        } else {
            if (xi > r) {
                // v' = cosT n - sinT e_y with e_y = (n cosIn - v) / sinIn (unit n, v)
                const float s2 = fmaxf(0.0f, 1.0f - cosIn * cosIn);
                const float sinT = sqrtf(s2) * __fdividef(n1, n2);
                float cosT = sqrtf(fmaxf(0.0f, 1.0f - sinT * sinT));
                if (!(cosIn > 0.0f)) cosT = -cosT;
                const float k = s2 > 1e-12f ? sinT * rsqrtf(s2) : 0.0f;
                vout = fast_norm(v3(cosT * nv.x - k * (nv.x * cosIn - v.x), cosT * nv.y - k * (nv.y * cosIn - v.y),
                                    cosT * nv.z - k * (nv.z * cosIn - v.z)));
            } else {
                vout = fast_norm(v3(v.x - 2.0f * cosIn * nv.x, v.y - 2.0f * cosIn * nv.y,
                                    v.z - 2.0f * cosIn * nv.z));
            }
        }
        if (xi > r) {
            newID = (cosIn > 0.0f) ? outer : inner;
            muaNew = nx.mua;
            musNew = nx.mus;
        } else {
            newID = ph.curr;
            muaNew = m.mua;
            musNew = m.mus;
        }
        ph.vx = vout.x; ph.vy = vout.y; ph.vz = vout.z;
        if (!Exact) {
            // The hit point lies on the face's plane only to float rounding, on either
            // side.  On the wrong side, the next segment can cross a neighbouring face of
            // the same surface a rounding distance away (the face itself is excluded by
            // refTri): a spurious second boundary event, which in float happens to about
            // 2e-4 of the photons of a curved mesh and lets them leave the region they
            // are labelled with.  The production arithmetic moves the photon off the
            // plane, to the side it travels to, by a few rounding units of the scene's
            // coordinates and of the distance travelled.  (The reference-order
            // arithmetic keeps the reference's behaviour.)
            const float push = P.boundary_push + 1e-6f * thit;
            const float sp = (dot3(vout, nv) > 0.0f) ? push : -push;
            ph.px = __fmaf_rn(sp, nv.x, ph.px);
            ph.py = __fmaf_rn(sp, nv.y, ph.py);
            ph.pz = __fmaf_rn(sp, nv.z, ph.pz);
        }
        float exit_w = 0.0f;
        const bool leaves = muaNew == 0.0f || musNew == 0.0f;
        if (leaves) {
            const float dist = fabsf(dot3(v3(P.nzx, P.nzy, P.nzz),
                                          v3(ph.px - P.poix, ph.py - P.poiy, ph.pz - P.poiz)));
            uint32_t kind;
            if (dist > P.distMin) kind = EXIT_TRANS;
            else kind = (ph.flags & F_FETAL) ? EXIT_SURF_FETAL : EXIT_SURF;
            exit_w = ph.w * P.exitScale;
            ph.flags = (ph.flags & ~(3u << EXIT_SHIFT)) | (kind << EXIT_SHIFT);
            ph.w = 0.0f;
        }
        const int prev = ph.curr;
        ph.curr = newID;
        ph.flags |= F_ON_FACE;
        if (newID == P.fetal_id) ph.flags |= F_FETAL;
        ph.unfin = Exact ? (step - thit) * m.mut : fmaxf(step - thit, 0.0f) * m.mut;
        if (leaves) ph.unfin = exit_w;
        if (newID != prev) {
            if (ph.region_acc) atomicAdd(s_region + prev, ph.region_acc);
            ph.region_acc = 0;
            if (Grad) {
                ga->L[prev] += ph.seg_len + thit;
                ga->k[prev] += ph.seg_k;
                ph.seg_len = 0.0f;
                ph.seg_k = 0;
            }
        } else if (Grad) {
            ph.seg_len += thit;
        }
    } else {
        ph.w = 0.0f;   // debug build: a triangle index out of range ends the photon
    }
    return ph;
}

// The step a photon is on: its length and reach, and the distance bound at the position.
struct Pending {
    float step, reach, safe_here;
};

// The nearest triangle within the step's reach (-1: none) and its distance thit; updates
// the distance bound the query establishes.  Every lane of the warp calls it, the ones
// whose step needs a query with `want`.
template <int STACK, bool NoGrid>
__device__ __forceinline__ int query_step(const KParams &P, const MeshView &M, const MeshView &SM, WarpQueue &Q,
                                          const Medium *s_media, bool want, Photon &ph, Counters &cnt,
                                          Pending &pd, float &thit)
{
    thit = kNoHit;
    if (!__any_sync(0xffffffffu, want)) return -1;
    const bool ambient = want && (s_media[ph.curr].kind & kAmbient);
    bool used_bvh;
    if (NoGrid) {
        cnt.query += want ? 1u : 0u;
        cnt.bvh += want ? 1u : 0u;
        return mesh_query<STACK>(P, SM, want, v3(ph.px, ph.py, ph.pz), v3(ph.vx, ph.vy, ph.vz),
                                 (ph.flags & F_ON_FACE) ? ph.last_tri : -1, ambient ? kNoHit : pd.reach,
                                 ambient ? 0.0f : P.factor * s_media[ph.curr].inv_mut, thit, pd.safe_here, ph.word);
    }
    // an empty cell: pd.safe_here holds its bound, which the step exceeds; a listed cell
    // raises it from the planes of its triangles when its list decides the step
    const int tri = warp_query<STACK>(P, M, SM, Q, want, v3(ph.px, ph.py, ph.pz), v3(ph.vx, ph.vy, ph.vz),
                                      (ph.flags & F_ON_FACE) ? ph.last_tri : -1, ambient ? kNoHit : pd.reach, ph.word,
                                      thit, pd.safe_here, used_bvh);
    cnt.query += want ? 1u : 0u;
    cnt.bvh += used_bvh ? 1u : 0u;
    return tri;
}

// A scatter event: moves the photon by `step`, absorbs, scatters and adds the deposit to the
// tallies.  Agg: deposits summed per cell across the warp before the atomic adds.  rz_copy:
// first cell of the block's copy of the r-z image (rz_copy_of).
template <bool Exact, bool Grad, bool Agg, bool NoGrid>
__device__ __forceinline__ void scatter_event(const KParams &P, const Medium &m, unsigned long long *s_cnt, Photon &ph,
                                              Counters &cnt, float step, float safe_here, const Draws &d,
                                              uint32_t rz_copy)
{
    const V3 v = v3(ph.vx, ph.vy, ph.vz);
    ph.px = ph.px + step * ph.vx;
    ph.py = ph.py + step * ph.vy;
    ph.pz = ph.pz + step * ph.vz;
    // the next step's cell word: its load is in flight during the rest of this step
    if (!NoGrid) ph.word = cell_at(P, ph.px, ph.py, ph.pz);
    ph.flags &= ~F_ON_FACE;
    ph.safe = fmaxf(safe_here - step - (NoGrid ? __ldg(P.mesh_eps + 1) : P.step_eps), 0.0f);
    if (Grad) {
        ph.seg_len += step;
        ph.seg_k++;
    }
    const bool absorbs = (m.kind & kAbsorbs) != 0;
    ph.absorbed = absorbs ? ph.w * m.alb : ph.absorbed;
    ph.w = absorbs ? ph.w - ph.absorbed : ph.w;
    const V3 vn = scatter_direction<Exact>(v, m, d.u1, d.cos_psi, d.sin_psi);
    ph.vx = vn.x; ph.vy = vn.y; ph.vz = vn.z;
    const V3 pr = v3(ph.px - P.poix, ph.py - P.poiy, ph.pz - P.poiz);
    const float cx = dot3(v3(P.nxx, P.nxy, P.nxz), pr);
    const float cy = dot3(v3(P.nyx, P.nyy, P.nyz), pr);
    const float cz = dot3(v3(P.nzx, P.nzy, P.nzz), pr);
    const float dw = ph.absorbed;
    const unsigned long long fdw = fix32(dw);
    // r-z grid (RecordAbsorbtionRZ, .cl:254-271, with atomic adds and z rows)
    int row, col;
    if (Exact) {
        const float rad = sqrt_normal(cx * cx + cy * cy) * sign_cl(cx);
        row = (int)floorf(P.plain_div ? cz / P.dg[2] : div_rn(cz, P.dg[2], P.inv_dz));
        col = (int)floorf((P.plain_div ? rad / P.dg[3] : div_rn(rad, P.dg[3], P.inv_dr)) + P.f_dimR);
    } else {
        const float rad = copysignf(sqrt_normal(cx * cx + cy * cy), cx) * P.inv_dr;
        row = (int)floorf(cz * P.inv_dz);
        col = (int)floorf(rad + P.f_dimR);
    }
    const bool rz_in = ((unsigned)row < (unsigned)P.rz_nz) & ((unsigned)col < (unsigned)P.rz_nr);
    // inv_mua is 0 where mua is not positive
    unsigned long long fdm;
    if (!Exact) fdm = fix32(dw * m.inv_mua);
    else if (m.kind & kPlainDiv) fdm = m.mua > 0.0f ? fix32(dw / m.mua) : 0ull;
    else fdm = fix32(div_rn(dw, m.mua, m.inv_mua));
    int ix, iy, iz;
    if (Exact) {
        ix = (int)floorf((P.plain_div ? cx / P.vox_dx : div_rn(cx, P.vox_dx, P.inv_vdx)) + P.half_vnx);
        iy = (int)floorf((P.plain_div ? cy / P.vox_dy : div_rn(cy, P.vox_dy, P.inv_vdy)) + P.half_vny);
        iz = (int)floorf(P.plain_div ? cz / P.vox_dz : div_rn(cz, P.vox_dz, P.inv_vdz));
    } else {
        ix = (int)floorf(cx * P.inv_vdx + P.half_vnx);
        iy = (int)floorf(cy * P.inv_vdy + P.half_vny);
        iz = (int)floorf(cz * P.inv_vdz);
    }
    // never in without a voxel grid (vox_nx = 0), and then no drop either
    const bool vox_in = ((unsigned)ix < (unsigned)P.vox_nx) & ((unsigned)iy < (unsigned)P.vox_ny) &
                        ((unsigned)iz < (unsigned)P.vox_nz);
    const int vox_key = vox_in ? (iz * P.vox_ny + iy) * P.vox_nx + ix : -1;
    cnt.vox_drop += vox_in ? 0u : P.vox_on;
    cnt.rz_drop += rz_in ? 0u : 1u;
    const int rz_key = rz_in ? row * P.rz_nr + col : -1;
    unsigned long long *const rz = P.rz_part + 2 * (int64_t)rz_copy;
    if (Agg) {
        // warp-aggregated deposits: the lanes of this branch that hit the same cell
        // are matched, their fixed-point values summed exactly, and one leader per
        // cell issues the atomic add (integer sums: same tallies as the plain form)
        const unsigned lane = threadIdx.x & 31u;
        const unsigned act = __activemask();
        const unsigned g_rz = __match_any_sync(act, rz_key);
        if (rz_key >= 0) {
            const unsigned long long a = group_sum_u64(g_rz, fdw), b = group_sum_u64(g_rz, fdm);
            if (lane == (unsigned)(__ffs(g_rz) - 1)) {
                unsigned long long *c = rz + 2 * (int64_t)rz_key;
                if (a) atomicAdd(c, a);
                if (b) atomicAdd(c + 1, b);
                atomicAdd(s_cnt + 15, 1ull);   // leaders: 1 - leaders / deposits is the match rate
            }
        }
        const unsigned g_vox = __match_any_sync(act, vox_key);
        if (vox_key >= 0) {
            const unsigned long long a = group_sum_u64(g_vox, fdw);
            if (a && lane == (unsigned)(__ffs(g_vox) - 1)) atomicAdd(P.vox + vox_key, a);
        }
    } else {
        // a weight that rounds to 0 is rare, and adding it is cheaper than the test
        if (rz_key >= 0) {
            unsigned long long *c = rz + 2 * (int64_t)rz_key;
            atomicAdd(c, fdw);
            atomicAdd(c + 1, fdm);
        }
        if (vox_key >= 0) atomicAdd(P.vox + vox_key, fdw);
    }
    ph.region_acc += fdw;
}

__device__ __forceinline__ uint32_t rz_copy_of(const KParams &P)
{
    return (blockIdx.x & P.rz_mask) * (uint32_t)(P.rz_stride >> 1);
}

// One iteration of the reference's do-while loop (.cl:1388-1600) for the warp's photons
// (the whole warp calls it; `live` has the lanes with one, `alive` is the lane's bit): step
// length, query if the step may reach a triangle, boundary event or scatter event, roulette.
// Returns false when the lane's photon ends.  Lanes without a photon compute the step length
// too: a branch around it costs every step more.  (Letting the lanes whose step needs a
// query wait until several of a warp do, and running their queries together, measured
// slower on every batch size: the waiting lanes cost more steps than the shared queries
// save.)
template <bool Exact, bool Grad, int STACK = kStackDepth, bool Agg = false, bool NoGrid = false>
__device__ __forceinline__ bool step_photon(const KParams &P, const MeshView &M, const MeshView &SM, WarpQueue &Q,
                                            const Medium *s_media, unsigned long long *s_region,
                                            unsigned long long *s_cnt, unsigned live, bool alive, Photon &ph,
                                            Counters &cnt, GradAcc *ga, WarpDraws &W, uint32_t &next, uint32_t rz_copy)
{
    const Draws d = next_draws<Exact>(P, W, live, alive, ph.idx, ph.steps, next);
    [[maybe_unused]] unsigned long long *const dbg = P.counters ? P.counters + kBoundsCounter : nullptr;
    // debug build: a region id out of range ends the photon
    if (alive && !LP_IN_RANGE(dbg, ph.curr, P.n_media)) {
        ph.w = 0.0f;
        ph.curr = 0;
        alive = false;
    }
    const Medium &m = s_media[ph.curr];
    const bool ambient = (m.kind & kAmbient) != 0;
    // the residual of a step cut short by a boundary, or a new step
    Pending pd;
    const float optical = (ph.unfin == 0.0f) ? d.neg_log * P.factor : ph.unfin;
    if (Exact) pd.step = (m.kind & kPlainDiv) ? optical / m.mut : div_rn(optical, m.mut, m.inv_mut);
    else pd.step = optical * m.inv_mut;
    if (ambient) pd.step = 0.0f;
    ph.unfin = alive ? 0.0f : ph.unfin;
    // reach: the production arithmetic also takes a face that lies up to a few rounding
    // units beyond the step as the step's boundary.  A hit computed just past the step
    // although it lies just within it would otherwise let the photon end its step on the
    // far side of the face, outside the region it is labelled with.  The photon then stops
    // on the face (and is moved off it, see boundary_event) with no residual step.
    pd.reach = Exact ? pd.step : pd.step + P.boundary_push + 1e-6f * pd.step;
    // safe_here: lower bound of the distance from p to every triangle, the larger of the
    // carried one and that of a cell no triangle touches (safe_distance is 0 for the others).
    // A step shorter than it cannot reach a triangle, so its bounded query would return "no
    // hit" and is skipped; after the step the bound shrinks by the step (plus the rounding of
    // the move).
    pd.safe_here = NoGrid ? ph.safe : fmaxf(ph.safe, safe_distance(P, ph.word));
    const bool want = alive && (ambient || !(pd.reach < pd.safe_here));
    float thit;
    const int tri = query_step<STACK, NoGrid>(P, M, SM, Q, s_media, want, ph, cnt, pd, thit);
    const float step = ambient ? thit : pd.step;
    // a query returns no hit beyond the step's reach
    if (alive && (tri >= 0 || kNoHit <= step)) {
        cnt.boundary++;
        ph = boundary_event<Exact, Grad>(P, s_media, s_region, s_cnt, ph, Grad ? ga : nullptr, tri, thit, step, d.u1);
        if (!NoGrid) ph.word = cell_at(P, ph.px, ph.py, ph.pz);
    } else if (alive) {
        scatter_event<Exact, Grad, Agg, NoGrid>(P, m, s_cnt, ph, cnt, step, pd.safe_here, d, rz_copy);
    }
    ph.steps += alive ? 1u : 0u;
    if (alive && (ph.w < P.w_th || ph.steps >= P.step_cap)) {
        if (ph.w < P.w_th && ph.w > 0.0f) {
            cnt.roulette++;
            ph.w = d.u3 < P.chance ? ph.w / P.chance : 0.0f;
        }
        if (ph.steps >= P.step_cap && ph.w > 0.0f) {
            atomicAdd(s_cnt + 5, 1ull);
            ph.w = 0.0f;
        }
    }
    return ph.w > 0.0f;
}

struct SmemLayout {
    int off_media, off_region, off_cnt, off_na, off_nb, off_nc, off_nd, off_tri, bytes;
};

__host__ __device__ inline SmemLayout smem_layout(int nodes_smem, int tris_smem)
{
    SmemLayout L;
    int o = 0;
    L.off_media = o; o += kMaxMedia * (int)sizeof(Medium);
    L.off_region = o; o += kMaxMedia * 8;
    L.off_cnt = o; o += 16 * 8;
    L.off_na = o; o += nodes_smem * 16;
    L.off_nb = o; o += nodes_smem * 16;
    L.off_nc = o; o += nodes_smem * 16;
    L.off_nd = o; o += nodes_smem * 16;
    L.off_tri = o; o += tris_smem * 48;
    L.bytes = o;
    return L;
}

__device__ __forceinline__ MeshView stage_mesh(const KParams &P, unsigned char *smem, const SmemLayout &L)
{
    MeshView M;
    M.na = P.node_a; M.nb = P.node_b; M.nc = P.node_c; M.nd = P.node_d;
    M.tri = P.tri;
    float4 *sa = reinterpret_cast<float4 *>(smem + L.off_na);
    float4 *sb = reinterpret_cast<float4 *>(smem + L.off_nb);
    float4 *sc = reinterpret_cast<float4 *>(smem + L.off_nc);
    int4 *sd = reinterpret_cast<int4 *>(smem + L.off_nd);
    float4 *tri = reinterpret_cast<float4 *>(smem + L.off_tri);
    for (int i = threadIdx.x; i < P.nodes_smem; i += blockDim.x) {
        sa[i] = P.node_a[i]; sb[i] = P.node_b[i]; sc[i] = P.node_c[i]; sd[i] = P.node_d[i];
    }
    for (int i = threadIdx.x; i < 3 * P.tris_smem; i += blockDim.x) tri[i] = P.tri[i];
    M.s_na = sa; M.s_nb = sb; M.s_nc = sc; M.s_nd = sd;
    M.s_tri = tri;
    M.nodes_smem = P.nodes_smem;
    M.tris_smem = P.tris_smem;
    M.n_nodes = P.n_nodes;
    M.n_tri = P.n_tri;
    M.dbg = P.counters ? P.counters + kBoundsCounter : nullptr;
    M.tri_eps = P.tri_eps;
    return M;
}

// NoGrid: the mesh has no cell grid (mesh_query).
// MinBlocks: resident blocks per SM it is compiled for.
template <bool Exact, bool Grad, bool Agg = false, bool NoGrid = false, int MinBlocks = LP_TRANSPORT_MIN_BLOCKS>
__global__ void __launch_bounds__(kBlock, MinBlocks) transport_kernel(const __grid_constant__ KParams P)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ WarpQueue queues[kBlock / 32];
    __shared__ WarpDraws draws[kBlock / 32];
    const SmemLayout L = smem_layout(P.nodes_smem, P.tris_smem);
    Medium *s_media = reinterpret_cast<Medium *>(smem + L.off_media);
    unsigned long long *s_region = reinterpret_cast<unsigned long long *>(smem + L.off_region);
    unsigned long long *s_cnt = reinterpret_cast<unsigned long long *>(smem + L.off_cnt);
    for (int i = threadIdx.x; i < P.n_media; i += blockDim.x) {
        s_media[i] = P.media[i];
        s_region[i] = 0;
    }
    if (threadIdx.x < 16) s_cnt[threadIdx.x] = 0;
    const MeshView M = stage_mesh(P, smem, L);
    __shared__ MeshView shared_view;
    if (threadIdx.x == 0) shared_view = M;
    __syncthreads();

    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    const uint32_t rz_copy = rz_copy_of(P);
    Counters cnt = {};
    uint32_t photons = 0;
    Photon ph;
    GradAcc ga;
    uint32_t next = 0;
    bool alive = false;
    bool exhausted = false;
    ph.idx = ph.steps = 0;
    ph.curr = 0;
    for (;;) {
        unsigned live = __ballot_sync(0xffffffffu, alive);
        if (live != P.lane_mask && !exhausted) {
            const unsigned need = P.lane_mask & ~live;
            const int k = __popc(need);
            next = 0;   // the new photons' events are to be drawn
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(P.work, (unsigned long long)k);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base + (unsigned long long)k >= (unsigned long long)P.n) exhausted = true;
            if ((need >> lane) & 1u) {
                const unsigned long long idx = base + __popc(need & lt_mask);
                if (idx < (unsigned long long)P.n) {
                    start_photon(P, ph, (uint32_t)idx);
                    if (NoGrid) ph.word = kRestFirst << 8 | kRestFirst;
                    if (Grad) {
                        for (int r = 0; r < P.n_media; ++r) {
                            ga.L[r] = 0.0f;
                            ga.k[r] = 0;
                        }
                    }
                    alive = true;
                }
            }
            live = __ballot_sync(0xffffffffu, alive);
        }
        if (!live) break;
        const bool more = step_photon<Exact, Grad, kStackDepth, Agg, NoGrid>(P, M, shared_view, queues[threadIdx.x >> 5],
                                                                     s_media, s_region, s_cnt, live, alive, ph, cnt, &ga,
                                                                     draws[threadIdx.x >> 5], next, rz_copy);
        if (alive) {
            if (!more) {
                if (ph.region_acc) atomicAdd(s_region + ph.curr, ph.region_acc);
                if (Grad) {
                    ga.L[ph.curr] += ph.seg_len;
                    ga.k[ph.curr] += ph.seg_k;
                }
                finish_photon<Grad>(P, exit_state(ph), Grad ? &ga : nullptr);
                cnt.steps += ph.steps;
                photons++;
                alive = false;
            }
        }
    }
    // block-level reduction of counters and region sums
    const uint32_t cv[8] = {cnt.scatter(), cnt.boundary, cnt.query, cnt.roulette, 0u, 0u, cnt.rz_drop, cnt.vox_drop};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (i == 4 || i == 5) continue;
        unsigned long long x = cv[i];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0 && x) atomicAdd(s_cnt + i, x);
    }
    {
        unsigned long long x = photons;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0 && x) atomicAdd(s_cnt + 8, x);
        x = cnt.skip();
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0 && x) atomicAdd(s_cnt + 10, x);
        x = cnt.bvh;
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0 && x) atomicAdd(s_cnt + 11, x);
    }
    __syncthreads();
    if (threadIdx.x < 16 && s_cnt[threadIdx.x]) atomicAdd(P.counters + threadIdx.x, s_cnt[threadIdx.x]);
    for (int i = threadIdx.x; i < P.n_media; i += blockDim.x)
        if (s_region[i]) atomicAdd(P.region + i, s_region[i]);
}

// Lets `kernel` be launched with smem bytes of dynamic shared memory.  The limit belongs to the
// kernel (on the current device), so it is raised where it is too low and never lowered: another
// thread's launch, or one that is captured into a graph later, may need more than this one.
template <class Kernel>
cudaError_t allow_smem(Kernel *kernel, int smem)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess || a.maxDynamicSharedSizeBytes >= smem) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

template <bool Exact, bool Grad, bool Agg, bool NoGrid, int MinBlocks>
cudaError_t launch_instance(const KParams &P, int grid, int smem, cudaStream_t s)
{
    const cudaError_t e = allow_smem(transport_kernel<Exact, Grad, Agg, NoGrid, MinBlocks>, smem);
    if (e != cudaSuccess) return e;
    transport_kernel<Exact, Grad, Agg, NoGrid, MinBlocks><<<grid, kBlock, smem, s>>>(P);
    return cudaGetLastError();
}

// P.grad selects the differentiating instantiation.
// The warp-aggregated form exists for the production arithmetic without differentiation
// only (P.agg_tallies is ignored otherwise).
template <bool Exact>
cudaError_t launch_transport_t(const KParams &P, int grid, int smem, cudaStream_t s)
{
    if (!Exact && !P.grad && P.agg_tallies)
        return launch_instance<false, false, true, false, LP_TRANSPORT_MIN_BLOCKS>(P, grid, smem, s);
    if (P.few_blocks)
        return P.grad ? launch_instance<Exact, true, false, false, kFewBlocks>(P, grid, smem, s)
                      : launch_instance<Exact, false, false, false, kFewBlocks>(P, grid, smem, s);
    return P.grad ? launch_instance<Exact, true, false, false, LP_TRANSPORT_MIN_BLOCKS>(P, grid, smem, s)
                  : launch_instance<Exact, false, false, false, LP_TRANSPORT_MIN_BLOCKS>(P, grid, smem, s);
}

template <bool Exact, bool Grad>
cudaError_t transport_occupancy_t(int smem, int *blocks_per_sm)
{
    const cudaError_t e = allow_smem(transport_kernel<Exact, Grad>, smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, transport_kernel<Exact, Grad>, kBlock, smem);
}

}  // namespace lp
