// Direct sums of the near / small field with several right-hand sides (near_field_run, F3M_src/n_tree.cu:831-902).
//
// Boxes of a few to some forty points (near.cu has the rule).  A pair costs its exponent (d multiply-adds in the expanded form,
// 2 d in the difference form), one exponential and R multiply-adds into the columns.  The CUDA-core kernels lose their time there
// on every source box: its rows through shared memory, target coordinates and factors anew, tiles and row pairs half empty.  Here the
// sources of a tile are one stream, and the sum over columns is the contraction C(16 targets x 8 columns) += E(16 x 8
// sources) B(8 x 8) on mma.m16n8k8.tf32: a lane of the A fragment owns the exponentials of two targets (g, g+8) and two
// sources (t, t+4), so no value is computed twice and a source is loaded once per four lanes.  The tile is too narrow for
// tcgen05 (N = 8 columns, E made in registers).  What bounds it: the three mma.sync per 128 pairs, 0.9e12 pairs/s at any
// occupancy (1e6 points N(0,I), 8 columns: d = 4 35.5 -> 27.6 ms, d = 5 178 -> 166 ms; 3e5 points, d = 5: 33.6 -> 15.3 ms).
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

// Group of eight sources in shared memory: [row k][t][sources t, t+4] for the D coordinates and, in the expanded form, minus the
// squared length; then B in fragment order [lane][rows t, t+4 of column g].
template <int D, bool DIFF> struct ColGroup {
    static constexpr int ROWS = DIFF ? D : D + 1;
    static constexpr int FLOATS = 8 * ROWS + 8 * CR;
};
constexpr int CST = 64;      // sources staged per warp: two chunks of 32, so that a full chunk always fits behind a remainder

// tiles[b] = tiles of the rows of target box b inside [row_begin, row_end)
__global__ void __launch_bounds__(256) col_tiles_per_box(int nbx, const int *__restrict__ off_x, const int *__restrict__ ptr, int row_begin,
                                                        int row_end, int *tiles) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nbx) return;
    int t = 0;
    if (b < nbx && ptr[b + 1] > ptr[b]) t = (max(0, min(off_x[b + 1], row_end) - max(off_x[b], row_begin)) + CT - 1) / CT;
    tiles[b] = t;
}

// The sources of a tile's list arrive as ONE stream, box borders left out: 32 list entries at a time (lane = entry) are prefix-summed,
// and a lane finds the source of its stream position by bisection.  All coordinates are relative to the centre c of the TARGET box,
// which keeps them for the whole list: with X = s (x-c), Y = s (y-c) the exponent -|X-Y|^2 is, in the expanded form,
// (2 X.Y - |Y|^2) - |X|^2, whose last part leaves the sum; |X|^2 is at most d/4 there (boxes up to one scaled unit), so the
// terms of the bracket cancel by no more than that and no factor overflows.  Wide boxes take the differences.
// Against packed rows per source box this drops the groups' padding at every box border, the target coordinates per
// source box and the packing pass: boxes of a few points were two thirds overhead.
template <int D, bool DIFF, int MT>
__device__ __forceinline__ void column_tile(const float2 *xs, float *stage, int *entries, const int *__restrict__ idx, int e0, int e1,
                                            const int *__restrict__ off_y, const float *__restrict__ ypts, int n_y,
                                            const float *__restrict__ bs, const float (&c)[D], float scale, int R, int r0, bool vec,
                                            float *out, int t0, int nt) {
    using G = ColGroup<D, DIFF>;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const f32x2 minus1 = c_pack(-1.f, -1.f);
    f32x2 xr[MT][D], tot[MT][2], acc[MT][2];
#pragma unroll
    for (int m = 0; m < MT; m++) {
#pragma unroll
        for (int k = 0; k < D; k++) {
            const float2 x = xs[(m * D + k) * 8 + g];
            xr[m][k] = DIFF ? c_pack(x.x, x.y) : c_pack(2.f * x.x, 2.f * x.y);
        }
        tot[m][0] = tot[m][1] = acc[m][0] = acc[m][1] = c_pack(0.f, 0.f);
    }
    int e = e0, total = 0, pos = 0;   // entries not loaded yet, stream positions loaded and used
    int fill = 0, since = 0;          // staged sources, groups since the last flush of acc
    while (true) {
        // stage up to 32 more sources
        if (pos == total && e < e1) {
            int len = 0, s0 = 0;
            if (e + lane < e1) {
                const int by = idx[e + lane];
                s0 = off_y[by];
                len = off_y[by + 1] - s0;
            }
            int inc = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            total = __shfl_sync(0xffffffffu, inc, 31);
            __syncwarp();
            entries[lane] = inc - len;               // first stream position of the entry
            entries[32 + lane] = s0 - (inc - len);   // sorted row of stream position p: p + this
            __syncwarp();
            pos = 0;
            e = min(e + 32, e1);
        }
        const int take = min(32, total - pos);
        if (lane < take) {
            const int p = pos + lane;
            int lo = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (entries[lo + step] <= p) lo += step;
            const int j = p + entries[32 + lo];
            const int q = fill + lane;
            float *dst = stage + (q >> 3) * G::FLOATS + 2 * (q & 3) + ((q >> 2) & 1);
            float n2 = 0.f;
#pragma unroll
            for (int k = 0; k < D; k++) {
                const float v = scale * (ypts[(size_t)k * n_y + j] - c[k]);
                n2 = fmaf(-v, v, n2);
                dst[8 * k] = DIFF ? -v : v;
            }
            if (!DIFF) dst[8 * D] = n2;
            const float *b = bs + (size_t)j * R + r0;
            float v[CR];
            if (vec) {
                const float4 lo4 = __ldg(reinterpret_cast<const float4 *>(b)), hi4 = __ldg(reinterpret_cast<const float4 *>(b) + 1);
                v[0] = lo4.x; v[1] = lo4.y; v[2] = lo4.z; v[3] = lo4.w; v[4] = hi4.x; v[5] = hi4.y; v[6] = hi4.z; v[7] = hi4.w;
            } else {
#pragma unroll
                for (int r = 0; r < CR; r++) v[r] = r0 + r < R ? __ldg(b + r) : 0.f;
            }
#pragma unroll
            for (int r = 0; r < CR; r++) dst[8 * G::ROWS + 8 * r] = v[r];
        }
        pos += take;
        fill += take;
        const bool last = pos == total && e >= e1;
        if (fill < 32 && !last) continue;
        // the sources that fill the last group weigh nothing
        int ngr = fill >> 3;
        if (last && (fill & 7)) {
            const int q = fill + lane;
            if (q < 8 * (ngr + 1)) {
                float *dst = stage + (q >> 3) * G::FLOATS + 2 * (q & 3) + ((q >> 2) & 1);
#pragma unroll
                for (int k = 0; k < G::ROWS + CR; k++) dst[8 * k] = 0.f;
            }
            ngr++;
        }
        __syncwarp();
#pragma unroll 1
        for (int gr = 0; gr < ngr; gr++) {
            const float *p = stage + gr * G::FLOATS;
            f32x2 y[2][G::ROWS];
#pragma unroll
            for (int k = 0; k < G::ROWS; k++) {
                const float2 v = *reinterpret_cast<const float2 *>(p + 8 * k + 2 * t);
                y[0][k] = c_pack(v.x, v.x);
                y[1][k] = c_pack(v.y, v.y);
            }
            const float2 nb = *reinterpret_cast<const float2 *>(p + 8 * G::ROWS + 2 * lane);
            const float bh0 = tf32_head(nb.x), bh1 = tf32_head(nb.y), bl0 = tf32_head(nb.x - bh0), bl1 = tf32_head(nb.y - bh1);
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
                        v = c_fma(xr[m][0], y[h][0], y[h][G::ROWS - 1]);
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
        since += ngr;
        if (since >= 16 || last) {   // blocked accumulation: partial sums of some 128 to 160 sources
#pragma unroll
            for (int m = 0; m < MT; m++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    tot[m][h] = c_add(tot[m][h], acc[m][h]);
                    acc[m][h] = c_pack(0.f, 0.f);
                }
            since = 0;
        }
        if (last) break;
        __syncwarp();
        // the remainder of less than a group moves to the front
        const int rest = fill & 7;
        if (rest) {
            for (int q = lane; q < G::FLOATS; q += 32) stage[q] = stage[(fill >> 3) * G::FLOATS + q];
            __syncwarp();
        }
        fill = rest;
    }
#pragma unroll
    for (int m = 0; m < MT; m++) {
        float f[2] = {1.f, 1.f};
        if (!DIFF) {   // 2^(-|X|^2) of the thread's two targets; xr holds 2 X
            f32x2 n2 = c_pack(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < D; k++) n2 = c_fma(xr[m][k], xr[m][k], n2);
            c_unpack(n2, f[0], f[1]);
            f[0] = c_ex2(-0.25f * f[0]);
            f[1] = c_ex2(-0.25f * f[1]);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = 16 * m + g + 8 * h, r = r0 + 2 * t;
            if (i >= nt) continue;
            float a, b;
            c_unpack(tot[m][h], a, b);
            float *o = out + (size_t)(t0 + i) * R + r;
            if (r < R) o[0] += f[h] * a;
            if (r + 1 < R) o[1] += f[h] * b;
        }
    }
}

template <int D, bool DIFF>
__global__ void __launch_bounds__(32 * CW, 4) near_columns(const float *__restrict__ xpts, int n_x, const int *__restrict__ off_x, int nbx,
                                                          const float *__restrict__ ctr_x, const int *__restrict__ tile_off,
                                                          const int *__restrict__ ptr, const int *__restrict__ idx,
                                                          const int *__restrict__ off_y, const float *__restrict__ ypts, int n_y,
                                                          const float *__restrict__ bs, float scale, int R, int r0, bool vec, float *out,
                                                          int row_begin, int row_end) {
    __shared__ float2 xs_all[CW][4 * D * 8];
    __shared__ __align__(16) float stage_all[CW][CST / 8 * ColGroup<D, DIFF>::FLOATS];
    __shared__ int entries_all[CW][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * CW + warp;
    if (item >= tile_off[nbx]) return;      // the grid is sized by a bound on the tiles, no read-back
    const int box = box_of_row(tile_off, nbx, item);
    // the box's groups of 16 rows are dealt out evenly over its tiles
    const int a = max(off_x[box], row_begin), len = min(off_x[box + 1], row_end) - a;
    const int tile = item - tile_off[box], ntiles = tile_off[box + 1] - tile_off[box], units = (len + 15) >> 4;
    const int t0 = a + 16 * (int)(((long long)units * tile) / ntiles);
    const int nt = min(a + 16 * (int)(((long long)units * (tile + 1)) / ntiles), a + len) - t0;
    float c[D];
#pragma unroll
    for (int k = 0; k < D; k++) c[k] = ctr_x[box * D + k];
    // scaled coordinates of the tile's targets, [row block m][k][g] = targets (16 m + g, 16 m + g + 8)
    float2 *xs = xs_all[warp];
    const int mt = (nt + 15) >> 4;
    for (int q = lane; q < mt * 8 * D; q += 32) {
        const int gg = q & 7, k = (q >> 3) % D, m = (q >> 3) / D;
        const int i0 = min(16 * m + gg, nt - 1), i1 = min(16 * m + gg + 8, nt - 1);
        const float ck = ctr_x[box * D + k];
        xs[q] = make_float2(scale * (xpts[(size_t)k * n_x + t0 + i0] - ck), scale * (xpts[(size_t)k * n_x + t0 + i1] - ck));
    }
    __syncwarp();
    const int e0 = ptr[box], e1 = ptr[box + 1];
    float *st = stage_all[warp];
    int *en = entries_all[warp];
#define F3M_TILE(MT_) column_tile<D, DIFF, MT_>(xs, st, en, idx, e0, e1, off_y, ypts, n_y, bs, c, scale, R, r0, vec, out, t0, nt)
    if (mt == 4) F3M_TILE(4);
    else if (mt == 3) F3M_TILE(3);
    else if (mt == 2) F3M_TILE(2);
    else F3M_TILE(1);
#undef F3M_TILE
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
    const int64_t max_items = (int64_t)(row_end - row_begin) / CT + lx.nb + 1;
    const bool vec = R % 4 == 0 && r0 + CR <= R;   // rows of b as two 16-byte loads (bs starts on a 256-byte boundary)
    pl->last.begin(ST_DIRECT, s);
    near_columns<D, DIFF><<<(unsigned)((max_items + CW - 1) / CW), 32 * CW, 0, s>>>(
        tx.pts.p, (int)tx.n, lx.off.p, lx.nb, lx.ctr.p, tiles.p, csr.ptr.p, csr.idx.p, ly.off.p, ty.pts.p, (int)ty.n, bs, scale, R, r0, vec, out,
        row_begin, row_end);
    pl->last.end(s);
    pl->last.direct_launches++;
    pl->last.direct_variants[DIFF ? DV_DIRECT : DV_MUFU]++;
    F3M_LAUNCH_CHECK();
}

// up to eight columns starting at r0; expanded: boxes at most one scaled unit wide
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
