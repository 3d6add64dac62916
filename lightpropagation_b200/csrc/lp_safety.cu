// lp_safety.cu -- cell grid over the mesh, built once per mesh on the GPU: per cell the list
// of the triangles touching it (widened by a margin), or, for a cell without any, a lower
// bound of the distance from ANY of its points to the nearest triangle.  A transport step
// shorter than that bound cannot reach a triangle, so the bounded nearest-hit query would
// return "no hit": the kernel skips it and the result is unchanged.
#include <algorithm>

#include "lp_kernel.cuh"

namespace lp {

// Triangle / cube overlap by the separating-axis theorem: the cube c +- r and the
// triangle (a, b, d) are disjoint iff their projections are disjoint on one of 13
// axes: the 3 cube axes, the triangle normal, and the 9 cross products of a cube axis
// with a triangle edge (Akenine-Moller, "Fast 3D triangle-box overlap testing", 2001).
// r includes a margin far above the rounding of the projections, so the test never
// reports "disjoint" for a triangle that touches the cube.
__device__ bool tri_cube_overlap(V3 c, float r, V3 a, V3 b, V3 d)
{
    const V3 v0 = sub3(a, c), v1 = sub3(b, c), v2 = sub3(d, c);
    if (fminf(v0.x, fminf(v1.x, v2.x)) > r || fmaxf(v0.x, fmaxf(v1.x, v2.x)) < -r) return false;
    if (fminf(v0.y, fminf(v1.y, v2.y)) > r || fmaxf(v0.y, fmaxf(v1.y, v2.y)) < -r) return false;
    if (fminf(v0.z, fminf(v1.z, v2.z)) > r || fmaxf(v0.z, fmaxf(v1.z, v2.z)) < -r) return false;
    const V3 e[3] = {sub3(v1, v0), sub3(v2, v1), sub3(v0, v2)};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const V3 f = e[i];
        // axis x cross f = (0, -f.z, f.y)
        float p0 = f.y * v0.z - f.z * v0.y, p1 = f.y * v1.z - f.z * v1.y, p2 = f.y * v2.z - f.z * v2.y;
        float rr = r * (fabsf(f.y) + fabsf(f.z));
        if (fminf(p0, fminf(p1, p2)) > rr || fmaxf(p0, fmaxf(p1, p2)) < -rr) return false;
        // axis y cross f = (f.z, 0, -f.x)
        p0 = f.z * v0.x - f.x * v0.z; p1 = f.z * v1.x - f.x * v1.z; p2 = f.z * v2.x - f.x * v2.z;
        rr = r * (fabsf(f.x) + fabsf(f.z));
        if (fminf(p0, fminf(p1, p2)) > rr || fmaxf(p0, fmaxf(p1, p2)) < -rr) return false;
        // axis z cross f = (-f.y, f.x, 0)
        p0 = f.x * v0.y - f.y * v0.x; p1 = f.x * v1.y - f.y * v1.x; p2 = f.x * v2.y - f.y * v2.x;
        rr = r * (fabsf(f.x) + fabsf(f.y));
        if (fminf(p0, fminf(p1, p2)) > rr || fmaxf(p0, fmaxf(p1, p2)) < -rr) return false;
    }
    // of a sliver the normal may be nothing but rounding: an axis like any other then, along
    // which the vertices do not coincide
    const V3 n = cross3(e[0], e[1]);
    const float p0 = dot3(n, v0), p1 = dot3(n, v1), p2 = dot3(n, v2);
    const float rr = r * (fabsf(n.x) + fabsf(n.y) + fabsf(n.z));
    return fminf(p0, fminf(p1, p2)) <= rr && fmaxf(p0, fmaxf(p1, p2)) >= -rr;
}

// One pass over the triangles (BVH order): every cell that a triangle touches (cells
// widened by eps) gets a count (refs == nullptr) or, in the second pass, the triangle's
// index at start[cell] + the next free slot (count re-zeroed before that pass).  One warp
// per triangle, its lanes striding over the cells of the triangle's box, and all warps of
// the launch shared out where there are fewer triangles than those: a slab face covers 10^5
// cells, and with one warp each the 32 triangles' passes took 23 ms of a first run of 27 (now
// 0.13 of 5).  The order of the entries within a cell is not defined, and no query depends on
// it.
__global__ void __launch_bounds__(256) cell_lists_kernel(const __grid_constant__ KParams P, int n_tri, float h,
                                                         float eps, uint32_t *count, const uint32_t *start,
                                                         int32_t *refs)
{
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    // warps per triangle: a mesh of few triangles has them large
    const int share = n_tri < n_warps ? n_warps / n_tri : 1;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t first = (int64_t)(warp % share) * 32 + (threadIdx.x & 31);
    for (int j = warp / share; j < n_tri; j += n_warps / share) {
        const TriRec T = load_tri(P.tri, j);
        const float4 ta = T.a, tb = T.b, tc = T.c;
        const V3 a = v3(ta.x, ta.y, ta.z);
        const V3 b = add3(a, v3(ta.w, tb.x, tb.y)), d = add3(a, v3(tb.z, tb.w, tc.x));
        const float lo[3] = {fminf(a.x, fminf(b.x, d.x)), fminf(a.y, fminf(b.y, d.y)), fminf(a.z, fminf(b.z, d.z))};
        const float hi[3] = {fmaxf(a.x, fmaxf(b.x, d.x)), fmaxf(a.y, fmaxf(b.y, d.y)), fmaxf(a.z, fmaxf(b.z, d.z))};
        const float o[3] = {P.g_ox, P.g_oy, P.g_oz};
        const int n[3] = {P.g_nx, P.g_ny, P.g_nz};
        int c0[3], c1[3];
        for (int k = 0; k < 3; ++k) {
            c0[k] = min(max((int)floorf((lo[k] - eps - o[k]) * P.g_inv_h), 0), n[k] - 1);
            c1[k] = min(max((int)floorf((hi[k] + eps - o[k]) * P.g_inv_h), 0), n[k] - 1);
        }
        const int ex = c1[0] - c0[0] + 1, ey = c1[1] - c0[1] + 1;
        const int64_t n_cells = (int64_t)ex * ey * (c1[2] - c0[2] + 1);
        for (int64_t q = first; q < n_cells; q += 32 * share) {
            const int x = c0[0] + (int)(q % ex);
            const int y = c0[1] + (int)((q / ex) % ey);
            const int z = c0[2] + (int)(q / ((int64_t)ex * ey));
            const V3 c = v3(o[0] + ((float)x + 0.5f) * h, o[1] + ((float)y + 0.5f) * h, o[2] + ((float)z + 0.5f) * h);
            if (!tri_cube_overlap(c, 0.5f * h + eps, a, b, d)) continue;
            const int64_t cell = ((int64_t)z * n[1] + y) * n[0] + x;
            const uint32_t k = atomicAdd(count + cell, 1u);
            if (refs) refs[start[cell] + k] = j;
        }
    }
}

// Distance bounds of the empty cells, from the lists alone.  Say a triangle's point x lies
// within the margin m (in cells) of the cells j0..j1 along an axis, and an empty cell i does
// not belong to them: then x is farther than (|i - j| - 1 + m) cells from every point of the
// cell along that axis, j the nearer of j0, j1; along the axes where i belongs to them it is
// at least 0 away.  The cell made of those j lists the triangle.  So with f(0) = 0 and
// f(d) = (|d| - 1 + m)^2, the smallest sum of f(dx) + f(dy) + f(dz) over the listed cells is
// a lower bound of the squared distance (in cells) to every triangle, within a cell of the
// true one along the axes.  A sum over axes has a separable minimum: one pass along x (rows
// of occupied bits), one along y, one along z, each looking outwards until f alone is larger
// than what it has.  Cells farther than kGapMax along an axis count as (kGapMax + m)^2.
// (A search of the tree from every cell, as before, took 12.5 ms for 25,600 triangles and 32
// ms for 202,500 at 2^24 cells; these passes take 1.3 ms for both.)
constexpr int kGapMax = 64;
constexpr int kGapNone = 255;

// gap[c] = distance in cells along x to the nearest cell with a triangle (kGapNone: farther
// than kGapMax).  One warp per row.
__global__ void __launch_bounds__(256) row_gap_kernel(int nx, int64_t rows, const uint32_t *count, uint8_t *gap)
{
    const int lane = threadIdx.x & 31;
    const unsigned le = 0xffffffffu >> (31 - lane), ge = 0xffffffffu << lane;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += n_warps) {
        const int64_t row = r * nx;
        int last = -1000;   // nearest occupied cell to the left of the chunk
        for (int x0 = 0; x0 < nx; x0 += 32) {
            const int x = x0 + lane;
            const unsigned m = __ballot_sync(0xffffffffu, x < nx && count[row + x] != 0);
            const int near = (m & le) ? x0 + 31 - __clz(m & le) : last;
            if (x < nx) gap[row + x] = (uint8_t)(x - near <= kGapMax ? x - near : kGapNone);
            if (m) last = x0 + 31 - __clz(m);
        }
        last = nx + 1000;   // to the right of it
        for (int x0 = (nx - 1) / 32 * 32; x0 >= 0; x0 -= 32) {
            const int x = x0 + lane;
            const unsigned m = __ballot_sync(0xffffffffu, x < nx && count[row + x] != 0);
            const int near = (m & ge) ? x0 + __ffs(m & ge) - 1 : last;
            if (x < nx && near - x <= kGapMax && near - x < (int)gap[row + x]) gap[row + x] = (uint8_t)(near - x);
            if (m) last = x0 + __ffs(m) - 1;
        }
    }
}

__device__ __forceinline__ float gap_square(int d, float m)
{
    const float g = (float)(d - 1) + m;
    return d > 0 ? g * g : 0.0f;
}

// The pass along y: the smallest f(dx) + f(dy) over the rows of the cell's z layer.
__global__ void __launch_bounds__(256) layer_gap_kernel(int nx, int ny, int64_t n, float m, const uint8_t *gap, float *d2)
{
    const float cap = gap_square(kGapMax + 1, m);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int y = (int)((i / nx) % ny);
        const int g0 = gap[i];
        float best = g0 == kGapNone ? cap : fminf(cap, gap_square(g0, m));
        for (int d = 1; d <= kGapMax; ++d) {
            const float f = gap_square(d, m);
            if (f >= best) break;
            if (y >= d) {
                const int g = gap[i - (int64_t)d * nx];
                if (g != kGapNone) best = fminf(best, f + gap_square(g, m));
            }
            if (y + d < ny) {
                const int g = gap[i + (int64_t)d * nx];
                if (g != kGapNone) best = fminf(best, f + gap_square(g, m));
            }
        }
        d2[i] = best;
    }
}

// The pass along z, and the cell words (see KParams::cell_word).  lists == false: every cell
// carries its distance bound only (0 where a triangle touches it).
__global__ void __launch_bounds__(256) cell_word_kernel(int64_t layer, int nz, float m, float h, float eps, float unit,
                                                        const float *d2, const uint32_t *count, const uint32_t *start,
                                                        bool lists, uint32_t *word)
{
    const int64_t n = layer * nz;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t k = count[i];
        uint32_t w;
        if (k == 0) {
            const int z = (int)(i / layer);
            float best = d2[i];
            for (int d = 1; d <= kGapMax; ++d) {
                const float f = gap_square(d, m);
                if (f >= best) break;
                if (z >= d) best = fminf(best, f + d2[i - d * layer]);
                if (z + d < nz) best = fminf(best, f + d2[i + d * layer]);
            }
            const float safe = sqrtf(best) * h * 0.9999f - eps;
            w = kCellEmpty | (uint32_t)fminf(safe > 0.0f ? floorf(safe / unit) : 0.0f, 65535.0f);
        } else if (!lists) {
            w = kCellEmpty;
        } else if (k >= kCellDense || start[i] + k > 0xffffffu) {
            w = kCellDense << 24;
        } else {
            w = start[i] | (k << 24);
        }
        word[i] = w;
    }
}

cudaError_t launch_cell_lists(const KParams &P, int n_tri, float h, float eps, uint32_t *count, const uint32_t *start,
                              int32_t *refs, cudaStream_t s)
{
    const int grid = 148 * 16;
    cell_lists_kernel<<<grid, 256, 0, s>>>(P, n_tri, h, eps, count, start, refs);
    return cudaGetLastError();
}

// gap: scratch of one byte per cell, d2: of one float per cell.  m: the lists' margin in
// cells; P.g_eps: the rounding they allow for on top.
cudaError_t launch_cell_words(const KParams &P, float m, const uint32_t *count, const uint32_t *start, bool lists,
                              uint8_t *gap, float *d2, uint32_t *word, cudaStream_t s)
{
    const int64_t n = (int64_t)P.g_nx * P.g_ny * P.g_nz, rows = (int64_t)P.g_ny * P.g_nz;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16));
    const int row_grid = (int)std::max<int64_t>(1, std::min<int64_t>((rows + 7) / 8, 148 * 16));
    row_gap_kernel<<<row_grid, 256, 0, s>>>(P.g_nx, rows, count, gap);
    layer_gap_kernel<<<grid, 256, 0, s>>>(P.g_nx, P.g_ny, n, m, gap, d2);
    cell_word_kernel<<<grid, 256, 0, s>>>((int64_t)P.g_nx * P.g_ny, P.g_nz, m, P.g_h, P.g_eps, P.g_unit, d2, count, start,
                                          lists, word);
    return cudaGetLastError();
}

}  // namespace lp
