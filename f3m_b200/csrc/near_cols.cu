// Direct sums of the near / small field with several right-hand sides (near_field_run, F3M_src/n_tree.cu:831-902).
//
// Boxes of a few to some forty points (near.cu has the rule).  A pair costs its exponent (d multiply-adds in the expanded form,
// 2 d in the difference form), one exponential and 8 multiply-adds into the columns.  The kernels of near.cu lose their time
// there on every source box: its rows through shared memory, target coordinates and factors anew, tiles and row pairs half empty.
// Here the sources of a tile are ONE stream, box borders left out, and a warp takes 8 MT targets and 16 sources at a time: lane
// (g, t) owns the targets g, g + 8, .. and the sources 4t .. 4t + 3 of the 16.  Two columns share an instruction (f32x2).  All
// in FP32: the columns as split TF32 products on mma.sync lost what the split's parts cannot hold (the NaN of GPU arithmetic,
// values near either end of the exponent range) and were no faster.
//
// What bounds it: FMA lanes (57 % busy at boxes of 246 points, d = 4) and the shared-memory pipe (70 %), which carries a source
// to every tile that reads it; with short boxes the latter, as a source then serves few rows.  Direct sums of 8 columns, all lists on
// the kernels of near.cu / short boxes as split TF32 / short boxes here: 1e6 points N(0,I), d = 5 60.7 / 36.0 / 31.7 ms, d = 4 33.5 /
// 26.5 / 22.6 ms; 3e5 points U[0,1]^5 in boxes of nine 40.3 / 17.9 / 14.4 ms.  All lists here: 1e6 points in boxes of 246, d = 4 8.0 -> 9.1 ms.
#include <math.h>
#include <algorithm>
#include "common.cuh"
#include "packed.cuh"

namespace f3m {

constexpr int CM = 4;        // target rows per lane
constexpr int CT = 8 * CM;   // targets per tile
constexpr int CR = 8;        // columns

// asynchronous copies into shared memory
__device__ __forceinline__ void c_copy4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void c_copy16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void c_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr int CST = 128;     // sources staged before they are summed: their copies are in flight together
// Staged sources: a plane per coordinate (in the expanded form one more for minus the squared length), read four sources at a
// time, then the rows of b; every four rows are followed by four floats, so that the lanes' 16-byte accesses meet no bank twice.
template <int D, bool DIFF> struct ColStage {
    static constexpr int COORDS = DIFF ? D : D + 1;
    static constexpr int FLOATS = COORDS * CST + CST / 4 * (4 * CR + 4);
    static __device__ __forceinline__ int b_row(int q) { return COORDS * CST + q * CR + (q >> 2) * 4; }
};

// tiles[b] = tiles of the rows of target box b inside [row_begin, row_end)
__global__ void __launch_bounds__(256) col_tiles_per_box(int nbx, const int *__restrict__ off_x, const int *__restrict__ ptr, int row_begin,
                                                        int row_end, int *tiles) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nbx) return;
    int t = 0;
    if (b < nbx && ptr[b + 1] > ptr[b]) t = (max(0, min(off_x[b + 1], row_end) - max(off_x[b], row_begin)) + CT - 1) / CT;
    tiles[b] = t;
}

// how the rows of b are copied: eight columns in two 16-byte copies, or four in one
enum ColCopy { COPY_8, COPY_4 };

// Rows of eight columns, from r0 on, zeros where b has none: other row lengths than multiples of four would be copied float by
// float, which meets the same banks (direct sums of 2 columns, 1e6 normal points, d = 5: 37.6 ms, with padded rows 28.0).
__global__ void __launch_bounds__(256) pad_columns(const float *__restrict__ bs, int64_t n, int R, int r0, float *dst) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n * CR) return;
    const int r = r0 + (int)(i % CR);
    dst[i] = r < R ? bs[i / CR * R + r] : 0.f;
}

// stream positions pos .. pos + take of the loaded entries -> staged sources fill .. fill + take
template <int D, bool DIFF, int COPY>
__device__ __forceinline__ void col_gather(float *stage, const int *entries, int pos, int fill, int take, const float *__restrict__ ypts,
                                           int n_y, const float *__restrict__ bs, int bw) {
    using S = ColStage<D, DIFF>;
    const int lane = threadIdx.x;
#pragma unroll
    for (int u = 0; u < CST / 32; u++) {
        if (lane + 32 * u >= take) continue;
        const int p = pos + lane + 32 * u;
        int lo = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
            if (entries[lo + step] <= p) lo += step;
        const int j = p + entries[32 + lo];
        const int q = fill + lane + 32 * u;
#pragma unroll
        for (int k = 0; k < D; k++) c_copy4(stage + k * CST + q, ypts + (size_t)k * n_y + j);
        float *dst = stage + S::b_row(q);
        const float *b = bs + (size_t)j * bw;
        c_copy16(dst, b);
        if (COPY == COPY_8) c_copy16(dst + 4, b + 4);
    }
}

// The list arrives 32 entries at a time (lane = entry): they are prefix-summed, and a lane finds the source of its stream position
// by bisection.  All coordinates are relative to the centre c of the TARGET box, which keeps them for the whole list: with
// X = s (x-c), Y = s (y-c) the exponent -|X-Y|^2 is, in the expanded form, (2 X.Y - |Y|^2) - |X|^2, whose last part leaves the
// sum; |X|^2 is at most d/4 there (boxes up to one scaled unit), so the terms of the bracket cancel by no more than that and no
// factor overflows.  Wide boxes take the differences.
template <int D, bool DIFF, int MT>
__device__ __forceinline__ void column_tile(const float *__restrict__ xpts, int n_x, float *stage, int *entries,
                                            const int *__restrict__ idx, int e0, int e1, const int *__restrict__ off_y,
                                            const float *__restrict__ ypts, int n_y, const float *__restrict__ bs, const float (&c)[D],
                                            float scale, int bw, int copy, int R, int r0, float *out, int t0, int nt) {
    using S = ColStage<D, DIFF>;
    const int lane = threadIdx.x, g = lane >> 2, t = lane & 3;
    float xr[MT][D];
    f32x2 acc[MT][CR / 2], tot[MT][CR / 2];
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const int i = t0 + min(8 * m + g, nt - 1);
#pragma unroll
        for (int k = 0; k < D; k++) {
            const float x = scale * (xpts[(size_t)k * n_x + i] - c[k]);
            xr[m][k] = DIFF ? x : 2.f * x;
        }
#pragma unroll
        for (int r = 0; r < CR / 2; r++) acc[m][r] = tot[m][r] = pack2(0.f, 0.f);
    }
    if (copy == COPY_4)   // the other four columns are never copied
        for (int q = S::COORDS * CST + lane; q < S::FLOATS; q += 32) stage[q] = 0.f;
    int e = e0, total = 0, pos = 0;   // entries not loaded yet, stream positions loaded and used
    int fill = 0;                     // staged sources
    while (true) {
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
        const int take = min(CST - fill, total - pos);
        // one loop per kind of copy: the four gathers of a lane stay together only without branches inside
        if (copy == COPY_8) col_gather<D, DIFF, COPY_8>(stage, entries, pos, fill, take, ypts, n_y, bs, bw);
        else col_gather<D, DIFF, COPY_4>(stage, entries, pos, fill, take, ypts, n_y, bs, bw);
        pos += take;
        fill += take;
        const bool last = pos == total && e >= e1;
        if (fill < CST && !last) continue;
        c_copy_wait();
        __syncwarp();
        const int ngr = (fill + 15) >> 4;
        for (int q = lane; q < 16 * ngr; q += 32) {
            if (q < fill) {
                float n2 = 0.f;
#pragma unroll
                for (int k = 0; k < D; k++) {
                    const float v = scale * (stage[k * CST + q] - c[k]);
                    n2 = fmaf(-v, v, n2);
                    stage[k * CST + q] = v;
                }
                if (!DIFF) stage[D * CST + q] = n2;
            } else {   // the sources that fill the last group weigh nothing
#pragma unroll
                for (int k = 0; k < S::COORDS; k++) stage[k * CST + q] = 0.f;
#pragma unroll
                for (int r = 0; r < CR; r++) stage[S::b_row(q) + r] = 0.f;
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int gr = 0; gr < ngr; gr++) {
            const float *p = stage + 16 * gr + 4 * t;
            float y[S::COORDS][4];
#pragma unroll
            for (int k = 0; k < S::COORDS; k++) {
                const float4 v = *reinterpret_cast<const float4 *>(p + k * CST);
                y[k][0] = v.x; y[k][1] = v.y; y[k][2] = v.z; y[k][3] = v.w;
            }
            const ulonglong2 *pb = reinterpret_cast<const ulonglong2 *>(stage + S::b_row(16 * gr + 4 * t));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const ulonglong2 b01 = pb[2 * q], b23 = pb[2 * q + 1];
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    float v;
                    if (DIFF) {
                        float df = xr[m][0] - y[0][q];
                        v = -df * df;
#pragma unroll
                        for (int k = 1; k < D; k++) {
                            df = xr[m][k] - y[k][q];
                            v = fmaf(-df, df, v);
                        }
                    } else {
                        v = fmaf(xr[m][0], y[0][q], y[S::COORDS - 1][q]);
#pragma unroll
                        for (int k = 1; k < D; k++) v = fmaf(xr[m][k], y[k][q], v);
                    }
                    const float ev = ex2_approx(v);
                    const f32x2 e2 = pack2(ev, ev);
                    acc[m][0] = fma2(e2, b01.x, acc[m][0]);
                    acc[m][1] = fma2(e2, b01.y, acc[m][1]);
                    acc[m][2] = fma2(e2, b23.x, acc[m][2]);
                    acc[m][3] = fma2(e2, b23.y, acc[m][3]);
                }
            }
        }
        // blocked accumulation: a partial sum holds at most 32 sources
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int r = 0; r < CR / 2; r++) {
                tot[m][r] = add2(tot[m][r], acc[m][r]);
                acc[m][r] = pack2(0.f, 0.f);
            }
        if (last) break;
        fill = 0;
        __syncwarp();
    }
#pragma unroll
    for (int m = 0; m < MT; m++) {
        // the four lanes of a target add up their sources: columns 2t, 2t + 1 end in lane t
        float v[CR], half[CR / 2], sum[2];
#pragma unroll
        for (int r = 0; r < CR / 2; r++) unpack2(tot[m][r], v[2 * r], v[2 * r + 1]);
#pragma unroll
        for (int r = 0; r < CR / 2; r++)
            half[r] = ((t & 2) ? v[r + 4] : v[r]) + __shfl_xor_sync(0xffffffffu, (t & 2) ? v[r] : v[r + 4], 2);
#pragma unroll
        for (int r = 0; r < 2; r++)
            sum[r] = ((t & 1) ? half[r + 2] : half[r]) + __shfl_xor_sync(0xffffffffu, (t & 1) ? half[r] : half[r + 2], 1);
        float f = 1.f;
        if (!DIFF) {   // 2^(-|X|^2); xr holds 2 X
            float n2 = 0.f;
#pragma unroll
            for (int k = 0; k < D; k++) n2 = fmaf(xr[m][k], xr[m][k], n2);
            f = ex2_approx(-0.25f * n2);
        }
        const int i = 8 * m + g, r = r0 + 2 * t;
        if (i >= nt) continue;
        float *o = out + (size_t)(t0 + i) * R + r;
        if (r < R) o[0] += f * sum[0];
        if (r + 1 < R) o[1] += f * sum[1];
    }
}

template <int D, bool DIFF>
__global__ void __launch_bounds__(32, 16) near_columns(const float *__restrict__ xpts, int n_x, const int *__restrict__ off_x, int nbx,
                                                       const float *__restrict__ ctr_x, const int *__restrict__ tile_off,
                                                       const int *__restrict__ ptr, const int *__restrict__ idx,
                                                       const int *__restrict__ off_y, const float *__restrict__ ypts, int n_y,
                                                       const float *__restrict__ bs, float scale, int bw, int copy, int R, int r0, float *out,
                                                       int row_begin, int row_end) {
    __shared__ __align__(16) float stage[ColStage<D, DIFF>::FLOATS];
    __shared__ int entries[64];
    const int item = blockIdx.x;
    if (item >= tile_off[nbx]) return;      // the grid is sized by a bound on the tiles, no read-back
    const int box = box_of_row(tile_off, nbx, item);
    // the box's groups of 8 rows are dealt out evenly over its tiles
    const int a = max(off_x[box], row_begin), len = min(off_x[box + 1], row_end) - a;
    const int tile = item - tile_off[box], ntiles = tile_off[box + 1] - tile_off[box], units = (len + 7) >> 3;
    const int t0 = a + 8 * (int)(((long long)units * tile) / ntiles);
    const int nt = min(a + 8 * (int)(((long long)units * (tile + 1)) / ntiles), a + len) - t0;
    float c[D];
#pragma unroll
    for (int k = 0; k < D; k++) c[k] = ctr_x[box * D + k];
    const int mt = (nt + 7) >> 3;
    const int e0 = ptr[box], e1 = ptr[box + 1];
#define F3M_TILE(MT_) column_tile<D, DIFF, MT_>(xpts, n_x, stage, entries, idx, e0, e1, off_y, ypts, n_y, bs, c, scale, bw, copy, R, r0, out, t0, nt)
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
    // rows of b start on 16 bytes: bs starts on 256 bytes, and so does the padded copy that other row lengths get
    DevBuf<float> padded;
    if (R % 4) {
        padded.alloc((size_t)ty.n * CR, s);
        pl->last.begin(ST_PERMUTE, s);
        pad_columns<<<(unsigned)((ty.n * CR + 255) / 256), 256, 0, s>>>(bs, ty.n, R, r0, padded.p);
        pl->last.end(s);
        F3M_LAUNCH_CHECK();
    }
    const float *b = R % 4 ? padded.p : bs + r0;
    const int bw = R % 4 ? CR : R, copy = R % 4 || R - r0 >= CR ? COPY_8 : COPY_4;
    pl->last.begin(ST_DIRECT, s);
    near_columns<D, DIFF><<<(unsigned)max_items, 32, 0, s>>>(
        tx.pts.p, (int)tx.n, lx.off.p, lx.nb, lx.ctr.p, tiles.p, csr.ptr.p, csr.idx.p, ly.off.p, ty.pts.p, (int)ty.n, b, scale, bw, copy, R, r0, out,
        row_begin, row_end);
    pl->last.end(s);
    pl->last.direct_launches++;
    pl->last.direct_variants[DIFF ? DV_DIRECT : DV_MUFU]++;
    pl->last.column_launches++;
    if (r0 == 0) pl->last.pairs[DIFF ? DV_DIRECT : DV_MUFU] += csr.pairs;
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
        F3M_COLS(2)
        F3M_COLS(3)
        F3M_COLS(4)
        F3M_COLS(5)
    }
#undef F3M_COLS
}

}  // namespace f3m
