// Direct sums of the near / small field with several right-hand sides (near_field_run, F3M_src/n_tree.cu:831-902).
//
// A pair costs its exponent (d multiply-adds in the expanded form, 2 d in the difference form), one exponential and R
// multiply-adds into the columns.  On the CUDA cores the last part dominates at R = 8, and every source row of d + R
// floats has to be broadcast out of shared memory to all 32 lanes for two targets each.  Here that part is the
// contraction it is, C(16 targets x 8 columns) += E(16 x 8 sources) B(8 x 8), on mma.m16n8k8.tf32: a lane of the A
// fragment owns the exponentials of two targets (g, g+8) and two sources (t, t+4), so no value is computed twice and a
// source row is loaded once per four lanes.  The tile is too narrow for tcgen05 (N = 8 columns, E made in registers), and
// mma.sync keeps up: the exponentials stay the limit.
//
// Precision: E and B are split into two TF32 numbers each (hi rounded to 11 bits, lo = the exact remainder), and hi hi + hi lo +
// lo hi is accumulated in FP32; what is dropped is below 2^-22 of a term.  The tensor core's own accumulator, which
// truncates, only ever sums one group of eight sources; groups and boxes are added with rounded FP32 additions.
#include <math.h>
#include <algorithm>
#include "common.cuh"

namespace f3m {

constexpr int CW = 4;        // warps per CTA, each with a tile of its own
constexpr int CT = 64;       // targets per tile: up to four groups of 16 (one m16n8k8 row block each)
constexpr int CR = 8;        // columns

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 c_pack(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void c_unpack(f32x2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 c_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 c_mul(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 c_add(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float c_ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// nearest number with 11 significant bits (ties away from zero)
__device__ __forceinline__ float tf32_head(float v) { return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u); }
__device__ __forceinline__ void mma_tf32(float (&c)[4], const float (&a)[4], float b0, float b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
          "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// Packed sources: groups of eight, [coordinate k][t][sources t, t+4], then B in fragment order [lane][rows t, t+4 of column g].
__host__ __device__ constexpr int col_group_floats(int D) { return 8 * D + 8 * CR; }
// first group of a box: boxes are padded to whole groups (ceil(len / 8) never exceeds the distance to the next box's start)
__host__ __device__ __forceinline__ int64_t col_group_start(int off, int box) { return ((int64_t)off + 7 * (int64_t)box + 7) >> 3; }

// one warp per source box and part
template <int D, bool DIFF>
__global__ void __launch_bounds__(256) pack_columns(const float *__restrict__ pts, int n, const float *__restrict__ bs, int R, int r0,
                                                   float scale, const int *__restrict__ off_y, int nby, const float *__restrict__ ctr_y,
                                                   const unsigned char *__restrict__ need, int nsplit, float *packed) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int by = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (by >= nby || (need && !need[by])) return;
    const int s0 = off_y[by], len = off_y[by + 1] - s0, ngr = (len + 7) >> 3;
    float c[D];
#pragma unroll
    for (int k = 0; k < D; k++) c[k] = ctr_y[by * D + k];
    for (int gr = blockIdx.y; gr < ngr; gr += nsplit) {
        float *dst = packed + (size_t)(col_group_start(s0, by) + gr) * col_group_floats(D);
        float b2[2], y2[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int j = gr * 8 + t + 4 * h;
            b2[h] = y2[h] = 0.f;   // the sources that fill the last group weigh nothing
            if (j < len) {
                float n2 = 0.f;
#pragma unroll
                for (int k = 0; k < D; k++) {
                    const float v = scale * (pts[(size_t)k * n + s0 + j] - c[k]);
                    n2 = fmaf(v, v, n2);
                    if (k == g) y2[h] = DIFF ? -v : 2.f * v;
                }
                if (r0 + g < R) b2[h] = bs[(size_t)(s0 + j) * R + r0 + g] * (DIFF ? 1.f : c_ex2(-n2));
            }
        }
        if (g < D) *reinterpret_cast<float2 *>(dst + g * 8 + t * 2) = make_float2(y2[0], y2[1]);
        *reinterpret_cast<float2 *>(dst + 8 * D + lane * 2) = make_float2(b2[0], b2[1]);
    }
}

// tiles[b] = tiles of the rows of target box b inside [row_begin, row_end)
__global__ void __launch_bounds__(256) col_tiles_per_box(int nbx, const int *__restrict__ off_x, const int *__restrict__ ptr, int row_begin,
                                                        int row_end, int *tiles) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nbx) return;
    int t = 0;
    if (b < nbx && ptr[b + 1] > ptr[b]) t = (max(0, min(off_x[b + 1], row_end) - max(off_x[b], row_begin)) + CT - 1) / CT;
    tiles[b] = t;
}

// xs: the tile's coordinates in shared memory, [row block m][k][g] = targets (16 m + g, 16 m + g + 8)
template <int D, bool DIFF, int MT>
__device__ __forceinline__ void column_tile(const float2 *xs, const int *__restrict__ idx, int e0, int e1, const int *__restrict__ off_y,
                                            const float *__restrict__ ctr_y, const float *__restrict__ packed, float scale, int R, int r0,
                                            float *out, int t0, int nt) {
    constexpr int GF = col_group_floats(D);
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const f32x2 minus1 = c_pack(-1.f, -1.f), scale2 = c_pack(scale, scale);
    f32x2 tot[MT][2];
#pragma unroll
    for (int m = 0; m < MT; m++) tot[m][0] = tot[m][1] = c_pack(0.f, 0.f);
    int by = idx[e0], s0 = off_y[by], ngr = (off_y[by + 1] - s0 + 7) >> 3;
    const float *p = packed + (size_t)col_group_start(s0, by) * GF;
    float2 ny[D], nb;   // the group after the current one, on its way from L2
    auto fetch = [&](const float *q) {
#pragma unroll
        for (int k = 0; k < D; k++) ny[k] = __ldg(reinterpret_cast<const float2 *>(q + k * 8 + t * 2));
        nb = __ldg(reinterpret_cast<const float2 *>(q + 8 * D + lane * 2));
    };
    fetch(p);
    for (int e = e0; e < e1; e++) {
        float c[D];
#pragma unroll
        for (int k = 0; k < D; k++) c[k] = __ldg(ctr_y + by * D + k);
        const int by_n = e + 1 < e1 ? idx[e + 1] : by;
        const int s0_n = off_y[by_n], ngr_n = (off_y[by_n + 1] - s0_n + 7) >> 3;
        const float *p_n = packed + (size_t)col_group_start(s0_n, by_n) * GF;
        f32x2 xr[MT][D], acc[MT][2];
        float fx[MT][2];
#pragma unroll
        for (int m = 0; m < MT; m++) {
            f32x2 n2 = c_pack(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < D; k++) {
                const float2 x = xs[(m * D + k) * 8 + g];
                xr[m][k] = c_mul(scale2, c_add(c_pack(x.x, x.y), c_pack(-c[k], -c[k])));
                if (!DIFF) n2 = c_fma(xr[m][k], xr[m][k], n2);
            }
            if (!DIFF) {
                float a, b;
                c_unpack(n2, a, b);
                fx[m][0] = c_ex2(-a);
                fx[m][1] = c_ex2(-b);
            } else
                fx[m][0] = fx[m][1] = 1.f;
            acc[m][0] = acc[m][1] = c_pack(0.f, 0.f);
        }
#pragma unroll 1
        for (int gr = 0; gr < ngr; gr++) {
            f32x2 y[2][D];
#pragma unroll
            for (int k = 0; k < D; k++) {
                y[0][k] = c_pack(ny[k].x, ny[k].x);
                y[1][k] = c_pack(ny[k].y, ny[k].y);
            }
            const float bh0 = tf32_head(nb.x), bh1 = tf32_head(nb.y), bl0 = tf32_head(nb.x - bh0), bl1 = tf32_head(nb.y - bh1);
            fetch(gr + 1 < ngr ? p + (size_t)(gr + 1) * GF : p_n);
#pragma unroll
            for (int m = 0; m < MT; m++) {
                float hi[4], lo[4];
#pragma unroll
                for (int h = 0; h < 2; h++) {   // sources t (h = 0) and t + 4, targets g and g + 8
                    f32x2 v;
                    if (DIFF) {
                        f32x2 df = c_add(xr[m][0], y[h][0]);
                        v = c_mul(df, df);
#pragma unroll
                        for (int k = 1; k < D; k++) {
                            df = c_add(xr[m][k], y[h][k]);
                            v = c_fma(df, df, v);
                        }
                    } else {
                        v = c_mul(xr[m][0], y[h][0]);
#pragma unroll
                        for (int k = 1; k < D; k++) v = c_fma(xr[m][k], y[h][k], v);
                    }
                    float v0, v1;
                    c_unpack(v, v0, v1);
                    const float ea = c_ex2(DIFF ? -v0 : v0), eb = c_ex2(DIFF ? -v1 : v1);
                    hi[2 * h] = tf32_head(ea);
                    hi[2 * h + 1] = tf32_head(eb);
                    c_unpack(c_fma(c_pack(hi[2 * h], hi[2 * h + 1]), minus1, c_pack(ea, eb)), lo[2 * h], lo[2 * h + 1]);
                }
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                mma_tf32(d, lo, bh0, bh1);
                mma_tf32(d, hi, bl0, bl1);
                mma_tf32(d, hi, bh0, bh1);
                acc[m][0] = c_add(acc[m][0], c_pack(d[0], d[1]));
                acc[m][1] = c_add(acc[m][1], c_pack(d[2], d[3]));
            }
        }
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) tot[m][h] = c_fma(c_pack(fx[m][h], fx[m][h]), acc[m][h], tot[m][h]);
        by = by_n;
        ngr = ngr_n;
        p = p_n;
    }
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = 16 * m + g + 8 * h, r = r0 + 2 * t;
            if (i >= nt) continue;
            float a, b;
            c_unpack(tot[m][h], a, b);
            float *o = out + (size_t)(t0 + i) * R + r;
            if (r < R) o[0] += a;
            if (r + 1 < R) o[1] += b;
        }
}

template <int D, bool DIFF>
__global__ void __launch_bounds__(32 * CW, 4) near_columns(const float *__restrict__ xpts, int n_x, const int *__restrict__ off_x, int nbx,
                                                          const int *__restrict__ tile_off, const int *__restrict__ ptr,
                                                          const int *__restrict__ idx, const int *__restrict__ off_y,
                                                          const float *__restrict__ ctr_y, const float *__restrict__ packed, float scale,
                                                          int R, int r0, float *out, int row_begin, int row_end) {
    __shared__ float2 xs_all[CW][4 * D * 8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * CW + warp;
    if (item >= tile_off[nbx]) return;      // the grid is sized by a bound on the tiles, no read-back
    const int box = box_of_row(tile_off, nbx, item);
    // the box's groups of 16 rows are dealt out evenly over its tiles
    const int a = max(off_x[box], row_begin), len = min(off_x[box + 1], row_end) - a;
    const int tile = item - tile_off[box], ntiles = tile_off[box + 1] - tile_off[box], units = (len + 15) >> 4;
    const int t0 = a + 16 * (int)(((long long)units * tile) / ntiles);
    const int nt = min(a + 16 * (int)(((long long)units * (tile + 1)) / ntiles), a + len) - t0;
    float2 *xs = xs_all[warp];
    const int mt = (nt + 15) >> 4;
    for (int q = lane; q < mt * 8 * D; q += 32) {
        const int gg = q & 7, k = (q >> 3) % D, m = (q >> 3) / D;
        const int i0 = 16 * m + gg, i1 = i0 + 8;
        xs[q] = make_float2(xpts[(size_t)k * n_x + t0 + min(i0, nt - 1)], xpts[(size_t)k * n_x + t0 + min(i1, nt - 1)]);
    }
    __syncwarp();
    const int e0 = ptr[box], e1 = ptr[box + 1];
    if (mt == 4) column_tile<D, DIFF, 4>(xs, idx, e0, e1, off_y, ctr_y, packed, scale, R, r0, out, t0, nt);
    else if (mt == 3) column_tile<D, DIFF, 3>(xs, idx, e0, e1, off_y, ctr_y, packed, scale, R, r0, out, t0, nt);
    else if (mt == 2) column_tile<D, DIFF, 2>(xs, idx, e0, e1, off_y, ctr_y, packed, scale, R, r0, out, t0, nt);
    else column_tile<D, DIFF, 1>(xs, idx, e0, e1, off_y, ctr_y, packed, scale, R, r0, out, t0, nt);
}

template <int D, bool DIFF>
static void columns_impl(f3m_plan *pl, int level, const PairCSR &csr, const float *bs, int R, int r0, float *out, int row_begin, int row_end,
                         cudaStream_t s) {
    Tree &tx = pl->tx, &ty = *pl->ty;
    Level &lx = tx.levels[level], &ly = ty.levels[level];
    const float scale = sqrtf(pl->lcs * 1.4426950408889634f);
    DevBuf<int> tiles;
    tiles.alloc((size_t)lx.nb + 1, s);
    col_tiles_per_box<<<(unsigned)((lx.nb + 1 + 255) / 256), 256, 0, s>>>(lx.nb, lx.off.p, csr.ptr.p, row_begin, row_end, tiles.p);
    F3M_LAUNCH_CHECK();
    exclusive_scan_i32(tiles.p, tiles.p, (int64_t)lx.nb + 1, s);
    // packed sources are kept for the "small" and the near list of one level
    f3m_plan::PackCache &pc = pl->pack_cache;
    if (!(pc.level == level && pc.r0 == r0 && pc.rb == CR && pc.expanded == !DIFF)) {
        pc.buf.alloc((size_t)(col_group_start((int)ty.n, ly.nb) + 1) * col_group_floats(D), s);
        pc.level = level; pc.r0 = r0; pc.rb = CR; pc.expanded = !DIFF;
        pl->last.begin(ST_PERMUTE, s);
        const unsigned char *need = level_source_flags(pl, level, s);
        const int nsplit = std::max(1, std::min(1024, (ly.max_count + 511) / 512));
        pack_columns<D, DIFF><<<dim3((unsigned)(((int64_t)ly.nb * 32 + 255) / 256), nsplit), 256, 0, s>>>(
            ty.pts.p, (int)ty.n, bs, R, r0, scale, ly.off.p, ly.nb, ly.ctr.p, need, nsplit, pc.buf.p);
        pl->last.end(s);
        F3M_LAUNCH_CHECK();
    }
    const int64_t max_items = (int64_t)(row_end - row_begin) / CT + lx.nb + 1;
    pl->last.begin(ST_DIRECT, s);
    near_columns<D, DIFF><<<(unsigned)((max_items + CW - 1) / CW), 32 * CW, 0, s>>>(
        tx.pts.p, (int)tx.n, lx.off.p, lx.nb, tiles.p, csr.ptr.p, csr.idx.p, ly.off.p, ly.ctr.p, pc.buf.p, scale, R, r0, out, row_begin, row_end);
    pl->last.end(s);
    pl->last.direct_launches++;
    pl->last.direct_variants[DIFF ? DV_DIRECT : DV_MUFU]++;
    F3M_LAUNCH_CHECK();
}

// up to eight columns starting at r0; expanded: the exponent bound of the list allows the expanded form
void column_sums(f3m_plan *pl, int level, const PairCSR &csr, bool expanded, const float *bs, int R, int r0, float *out, int row_begin, int row_end,
                 cudaStream_t s) {
    if (row_end <= row_begin) return;
#define F3M_COLS(D_)                                                                                  \
    case D_:                                                                                          \
        if (expanded) columns_impl<D_, false>(pl, level, csr, bs, R, r0, out, row_begin, row_end, s); \
        else columns_impl<D_, true>(pl, level, csr, bs, R, r0, out, row_begin, row_end, s);           \
        break;
    switch (pl->d) {
        F3M_COLS(1)
        F3M_COLS(2)
        F3M_COLS(3)
        F3M_COLS(4)
        F3M_COLS(5)
    }
#undef F3M_COLS
}

}  // namespace f3m
