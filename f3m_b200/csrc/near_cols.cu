// Direct sums of the near / small field with several right-hand sides (near_field_run, F3M_src/n_tree.cu:831-902).
//
// A pair costs its exponent (d multiply-adds in the expanded form, 2 d in the difference form), one exponential and 8 (or 4)
// multiply-adds into the columns.  The kernels of near.cu lose their time on every source box: its rows through shared memory,
// target coordinates and factors anew, tiles and row pairs half empty.  Here the sources of a tile are ONE stream, box borders left out,
// and the targets of sibling boxes with equal lists are one box (near.cu has the rule when which kernel runs).  A warp takes up
// to 64 targets: a lane owns four of them and every second quadruple of sources (smaller tiles: every fourth), so that a source's row
// is read by half-warps at one address each.  Sources are rows of 64 bytes, copied 64 at a time with cp.async while the 64 before
// them are summed.  Two columns share an instruction (f32x2).  All in FP32: the columns as split TF32 products on mma.sync lost
// what the split's parts cannot hold (the NaN of GPU arithmetic, values near either end of the exponent range) and were no faster.
//
// What bounds it: FMA lanes and the issue slots of the pairs.  8 columns, d = 5: 16.7 cycles per 32 pairs and SM quarter with everything in
// registers, 23 here (FMA pipe 59 % busy, 12.9 instructions of the ideal 11; d = 4: 21 and 58 %).  Before, tiles of 32 targets each box by itself, sources
// gathered float by float and no overlap of copies and sums took 34 to 50.  Direct sums of 8 columns, then / now: 1e6 points N(0,I), d = 5 (boxes
// of 18 points on average, 139 weighted by pairs) 119.5 / 87.4 ms, d = 4 21.8 / 15.3 ms; 3e5 points, d = 5 22.1 / 10.9 ms.
#include <math.h>
#include <algorithm>
#include "common.cuh"
#include "packed.cuh"

namespace f3m {

constexpr int CT = 64;       // targets per tile

__device__ __forceinline__ void c_copy16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void c_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void c_copy_wait_but_last() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// A source is a row of 16 floats: its coordinates (in shared memory scaled and, in the expanded form, followed by minus their
// squared length), at CB the columns of b.  Staged rows are 20 floats apart: the lanes' 16-byte accesses to eight rows meet no bank twice.
constexpr int CROW = 16, CB = 8, CSTRIDE = 20;
constexpr int CST = 64;      // sources staged at a time; the next ones are copied while these are summed

// Siblings whose rows of the list are equal -- most of them, where all boxes around are small: the classes depend on the two boxes' sizes
// first -- are summed as one target box, around their parent's centre: tiles fill up, and a source is fetched once for all of
// them.  first[b] = 1 where a new group begins (always at a new parent); a warp per box.
__global__ void __launch_bounds__(256) col_groups(int nbx, const int *__restrict__ parent, const int *__restrict__ ptr, const int *__restrict__ idx,
                                                 int group, int *first) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b > nbx) return;
    bool same = group && b > 0 && b < nbx && parent[b] == parent[b - 1];
    if (same) {
        const int p0 = ptr[b - 1], p1 = ptr[b], len = p1 - p0;
        same = ptr[b + 1] - p1 == len;
        for (int e = lane; same && e - lane < len; e += 32) same = !__any_sync(0xffffffffu, e < len && idx[p0 + e] != idx[p1 + e]);
    }
    if (lane == 0) first[b] = !same;
}

// items[b] = tiles of the rows of the group that begins with target box b inside [row_begin, row_end), times the parts its list is cut
// into (chunk sources each, 0: not cut), slots[b] = as many where there is more than one part; a warp per box
struct ColGroup { int boxes, parts; };
__global__ void __launch_bounds__(256) col_items(int nbx, const int *__restrict__ off_x, const int *__restrict__ ptr, const int *__restrict__ idx,
                                                const int *__restrict__ off_y, const int *__restrict__ first, int chunk, int row_begin,
                                                int row_end, int *items, int *slots, ColGroup *groups) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b > nbx) return;
    int t = 0;
    ColGroup g{1, 1};
    if (b < nbx && first[b] && ptr[b + 1] > ptr[b]) {
        while (!first[b + g.boxes]) g.boxes++;      // first[nbx] = 1
        t = (max(0, min(off_x[b + g.boxes], row_end) - max(off_x[b], row_begin)) + CT - 1) / CT;
        if (chunk && t) {
            int64_t sum = 0;
            for (int e = ptr[b] + lane; e < ptr[b + 1]; e += 32) { const int by = idx[e]; sum += off_y[by + 1] - off_y[by]; }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            g.parts = (int)min((int64_t)(ptr[b + 1] - ptr[b]), max((int64_t)1, (sum + chunk - 1) / chunk));
        }
    }
    if (lane == 0) {
        items[b] = t * g.parts;
        slots[b] = g.parts > 1 ? t * g.parts : 0;
        if (b < nbx) groups[b] = g;
    }
}

template <int D>
__global__ void __launch_bounds__(256) pack_column_rows(const float *__restrict__ pts, int64_t n, const float *__restrict__ bs, int R, int r0,
                                                       float *rows) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x, j = i / CROW;
    if (j >= n) return;
    const int c = (int)(i % CROW), r = r0 + c - CB;
    rows[i] = c < D ? pts[(size_t)c * n + j] : (c >= CB && r < R) ? bs[j * R + r] : 0.f;
}

// The list arrives 32 entries at a time (lane = entry; the next 32 are read ahead) and is prefix-summed; 32 stream positions at a
// time, a lane counts the entries that start up to its own.  All coordinates are relative to the centre c of the TARGET box, which keeps them for the
// whole list: with X = s (x-c), Y = s (y-c) the exponent -|X-Y|^2 is, in the expanded form, (2 X.Y - |Y|^2) - |X|^2, whose last part
// leaves the sum; |X|^2 is at most d/4 there (boxes up to one scaled unit), so the terms of the bracket cancel by no more than that and
// no factor overflows.  Wide boxes take the differences.
// A lane owns MT target rows, TR = 32 / G of them apart, and every G-th quadruple of sources; NC = 8 or 4 columns.  slot: where in parts
// a part of a list leaves its sums, or -1: they are added to out.
template <int D, bool DIFF, int NC, int G, int MT>
__device__ __forceinline__ void column_tile(const float *__restrict__ xpts, int n_x, float *stages, const int *__restrict__ idx, int e0,
                                            int e1, const int *__restrict__ off_y, const float *__restrict__ rows, const float (&c)[D],
                                            float scale, int R, int r0, float *out, int t0, int nt, float *parts, int slot) {
    constexpr int TR = 32 / G, STEP = 4 * G;
    const int lane = threadIdx.x, g = lane % TR, h = lane / TR;
    float xr[MT][D];
    f32x2 acc[MT][NC / 2], tot[MT][NC / 2];
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const int i = t0 + min(TR * m + g, nt - 1);
#pragma unroll
        for (int k = 0; k < D; k++) {
            const float x = scale * (xpts[(size_t)k * n_x + i] - c[k]);
            xr[m][k] = DIFF ? x : 2.f * x;
        }
#pragma unroll
        for (int r = 0; r < NC / 2; r++) acc[m][r] = tot[m][r] = pack2(0.f, 0.f);
    }
    int e = e0, total = 0, pos = 0;    // entries not loaded yet, stream positions loaded and used
    int start = 0, shift = 0;          // the lane's entry: its first stream position (past all for none), sorted row of position p: p + shift
    int nlen = 0, nrow = 0;            // the lane's entry among the next 32
    auto read_ahead = [&]() {
        nlen = nrow = 0;
        if (e + lane < e1) {
            const int by = idx[e + lane];
            nrow = off_y[by];
            nlen = off_y[by + 1] - nrow;
        }
    };
    read_ahead();
    // copies the next sources of the stream into a stage, as many as fit; how many they are
    auto fetch = [&](float *stage) {
        int fill = 0;
        while (fill < CST) {
            if (pos == total) {
                if (e >= e1) break;
                const int len = nlen, s0 = nrow;
                e = min(e + 32, e1);
                read_ahead();
                int inc = len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += v;
                }
                total = __shfl_sync(0xffffffffu, inc, 31);
                start = len ? inc - len : 0x7fffffff;
                shift = s0 - (inc - len);
                pos = 0;
            }
            const int take = min(32, min(CST - fill, total - pos));
            const int before = __popc(__ballot_sync(0xffffffffu, start < pos)), rel = start - pos;
            const unsigned starts = __reduce_or_sync(0xffffffffu, (unsigned)rel < 32u ? 1u << rel : 0u);
            const int entry = before + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
            const int j = pos + lane + __shfl_sync(0xffffffffu, shift, entry & 31);
            if (lane < take) {
                const float *src = rows + (size_t)j * CROW;
                float *dst = stage + (fill + lane) * CSTRIDE;
#pragma unroll
                for (int q = 0; q < CROW; q += 4)
                    if (q < D || (q >= CB && q < CB + NC)) c_copy16(dst + q, src + q);
            }
            pos += take;
            fill += take;
        }
        return fill;
    };
    int fill = fetch(stages), cur = 0;
    c_copy_commit();
    while (fill > 0) {
        float *stage = stages + cur * (CST * CSTRIDE);
        const int next = fetch(stages + (cur ^ 1) * (CST * CSTRIDE));
        c_copy_commit();
        c_copy_wait_but_last();
        __syncwarp();
        const int ngr = (fill + STEP - 1) / STEP;
        for (int q = lane; q < STEP * ngr; q += 32) {
            float4 *row = reinterpret_cast<float4 *>(stage + q * CSTRIDE);
            if (q < fill) {
                float y[8];
#pragma unroll
                for (int k = 0; k < (D > 4 ? 8 : 4); k += 4) {
                    const float4 v = row[k / 4];
                    y[k] = v.x; y[k + 1] = v.y; y[k + 2] = v.z; y[k + 3] = v.w;
                }
                float n2 = 0.f;
#pragma unroll
                for (int k = 0; k < D; k++) {
                    y[k] = scale * (y[k] - c[k]);
                    n2 = fmaf(-y[k], y[k], n2);
                }
                if (!DIFF) y[D] = n2;
                row[0] = make_float4(y[0], y[1], y[2], y[3]);
                if (D + !DIFF > 4) *reinterpret_cast<float2 *>(row + 1) = make_float2(y[4], y[5]);
            } else {   // the sources that fill the last group weigh nothing
#pragma unroll
                for (int k = 0; k < CROW / 4; k++) row[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int gr = 0; gr < ngr; gr++) {
            const float *p = stage + (STEP * gr + 4 * h) * CSTRIDE;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float y[6];
                const float4 y0 = *reinterpret_cast<const float4 *>(p + q * CSTRIDE);
                y[0] = y0.x; y[1] = y0.y; y[2] = y0.z; y[3] = y0.w;
                if (D + !DIFF > 4) {
                    const float2 y4 = *reinterpret_cast<const float2 *>(p + q * CSTRIDE + 4);
                    y[4] = y4.x; y[5] = y4.y;
                }
                const ulonglong2 b01 = *reinterpret_cast<const ulonglong2 *>(p + q * CSTRIDE + CB);
                const ulonglong2 b23 = NC > 4 ? *reinterpret_cast<const ulonglong2 *>(p + q * CSTRIDE + CB + 4) : b01;
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    float v;
                    if (DIFF) {
                        float df = xr[m][0] - y[0];
                        v = -df * df;
#pragma unroll
                        for (int k = 1; k < D; k++) {
                            df = xr[m][k] - y[k];
                            v = fmaf(-df, df, v);
                        }
                    } else {
                        v = fmaf(xr[m][0], y[0], y[D]);
#pragma unroll
                        for (int k = 1; k < D; k++) v = fmaf(xr[m][k], y[k], v);
                    }
                    const float ev = ex2_approx(v);
                    const f32x2 e2 = pack2(ev, ev);
                    acc[m][0] = fma2(e2, b01.x, acc[m][0]);
                    acc[m][1] = fma2(e2, b01.y, acc[m][1]);
                    if (NC > 4) {
                        acc[m][NC / 2 - 2] = fma2(e2, b23.x, acc[m][NC / 2 - 2]);
                        acc[m][NC / 2 - 1] = fma2(e2, b23.y, acc[m][NC / 2 - 1]);
                    }
                }
            }
        }
        // blocked accumulation: a partial sum holds at most 32 sources
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int r = 0; r < NC / 2; r++) {
                tot[m][r] = add2(tot[m][r], acc[m][r]);
                acc[m][r] = pack2(0.f, 0.f);
            }
        __syncwarp();
        fill = next;
        cur ^= 1;
    }
#pragma unroll
    for (int m = 0; m < MT; m++) {
        // the G lanes of a target add up their sources: columns CPL h .. CPL h + CPL - 1 end in lane h
        constexpr int CPL = NC / G;
        float v[NC], half[NC / 2], sum[CPL];
#pragma unroll
        for (int r = 0; r < NC / 2; r++) unpack2(tot[m][r], v[2 * r], v[2 * r + 1]);
        const bool up = h >= G / 2, odd = h & 1;
#pragma unroll
        for (int r = 0; r < NC / 2; r++) half[r] = (up ? v[r + NC / 2] : v[r]) + __shfl_xor_sync(0xffffffffu, up ? v[r] : v[r + NC / 2], 16);
#pragma unroll
        for (int r = 0; r < CPL; r++) {
            const float other = half[(r + CPL) % (NC / 2)];
            sum[r] = G == 2 ? half[r] : (odd ? other : half[r]) + __shfl_xor_sync(0xffffffffu, odd ? half[r] : other, TR);
        }
        float f = 1.f;
        if (!DIFF) {   // 2^(-|X|^2); xr holds 2 X
            float n2 = 0.f;
#pragma unroll
            for (int k = 0; k < D; k++) n2 = fmaf(xr[m][k], xr[m][k], n2);
            f = ex2_approx(-0.25f * n2);
        }
        const int i = TR * m + g, r = r0 + CPL * h;
        if (i >= nt) continue;
        float *o = out + (size_t)(t0 + i) * R + r;
#pragma unroll
        for (int q = 0; q < CPL; q++) {
            if (slot >= 0) parts[(size_t)slot * (CT * NC) + i * NC + CPL * h + q] = f * sum[q];
            else if (r + q < R) o[q] += f * sum[q];
        }
    }
}

// A group's rows inside the slice, dealt out evenly over its tiles, 16 at a time
struct ColTile { int begin, rows; };
__device__ __forceinline__ ColTile col_tile(const int *__restrict__ off_x, int box, int boxes, int tile, int ntiles, int row_begin, int row_end) {
    const int a = max(off_x[box], row_begin), len = min(off_x[box + boxes], row_end) - a, units = (len + 15) >> 4;
    const int t0 = a + 16 * (int)(((long long)units * tile) / ntiles);
    return ColTile{t0, min(a + 16 * (int)(((long long)units * (tile + 1)) / ntiles), a + len) - t0};
}

// The sums of a list's parts, in the order of the list: a block per slot, those of a tile's first part work
template <int NC>
__global__ void __launch_bounds__(CT * NC / 4) col_parts_sum(const int *__restrict__ off_x, int nbx, const int *__restrict__ item_off,
                                                    const int *__restrict__ slot_off, const ColGroup *__restrict__ groups,
                                                    const float *__restrict__ parts, int R, int r0, float *out, int row_begin, int row_end) {
    const int box = box_of_row(slot_off, nbx, blockIdx.x);
    const ColGroup group = groups[box];
    const int q = blockIdx.x - slot_off[box], np = group.parts;
    if (q % np) return;
    const ColTile t = col_tile(off_x, box, group.boxes, q / np, (item_off[box + 1] - item_off[box]) / np, row_begin, row_end);
    const int e = threadIdx.x, i = e / (NC / 4), r = r0 + e % (NC / 4) * 4;   // four columns of a row
    if (i >= t.rows) return;
    const float4 *src = reinterpret_cast<const float4 *>(parts) + (size_t)blockIdx.x * (CT * NC / 4) + e;
    float4 v = src[0];
#pragma unroll 4
    for (int p = 1; p < np; p++) {
        const float4 w = src[(size_t)p * (CT * NC / 4)];
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
    }
    const float sum[4] = {v.x, v.y, v.z, v.w};
    float *o = out + (size_t)(t.begin + i) * R + r;
#pragma unroll
    for (int c = 0; c < 4; c++)
        if (r + c < R) o[c] += sum[c];
}

template <int D, bool DIFF, int NC>
__global__ void __launch_bounds__(32, 16) near_columns(const float *__restrict__ xpts, int n_x, const int *__restrict__ off_x, int nbx,
                                                       const float *__restrict__ ctr_x, const int *__restrict__ parent,
                                                       const float *__restrict__ parent_ctr, const int *__restrict__ item_off,
                                                       const int *__restrict__ slot_off, const ColGroup *__restrict__ groups,
                                                       const int *__restrict__ ptr, const int *__restrict__ idx, const int *__restrict__ off_y,
                                                       const float *__restrict__ rows, float scale, int R, int r0, float *out, float *parts,
                                                       int row_begin, int row_end) {
    __shared__ __align__(16) float stage[2 * CST * CSTRIDE];
    const int item = blockIdx.x;
    if (item >= item_off[nbx]) return;      // the grid may be sized by a bound
    const int box = box_of_row(item_off, nbx, item);
    const ColGroup group = groups[box];
    const int np = group.parts, q = item - item_off[box], part = q % np;
    const ColTile tile = col_tile(off_x, box, group.boxes, q / np, (item_off[box + 1] - item_off[box]) / np, row_begin, row_end);
    const int t0 = tile.begin, nt = tile.rows;
    const int slot = np > 1 ? slot_off[box] + q : -1;
    float c[D];
    const float *centre = group.boxes > 1 ? parent_ctr + parent[box] * D : ctr_x + box * D;
#pragma unroll
    for (int k = 0; k < D; k++) c[k] = centre[k];
    const int p0 = ptr[box], n_entries = ptr[box + 1] - p0;
    const int e0 = p0 + (int)(((long long)n_entries * part) / np), e1 = p0 + (int)(((long long)n_entries * (part + 1)) / np);
#define F3M_TILE(G_, MT_) \
    column_tile<D, DIFF, NC, G_, MT_>(xpts, n_x, stage, idx, e0, e1, off_y, rows, c, scale, R, r0, out, t0, nt, parts, slot)
    if (nt > 48) F3M_TILE(2, 4);
    else if (nt > 32) F3M_TILE(2, 3);
    else if (nt > 24) F3M_TILE(4, 4);
    else if (nt > 16) F3M_TILE(4, 3);
    else if (nt > 8) F3M_TILE(4, 2);
    else F3M_TILE(4, 1);
#undef F3M_TILE
}

template <int D, bool DIFF>
static void columns_impl(f3m_plan *pl, int level, const PairCSR &csr, const float *bs, int R, int r0, float *out, int row_begin, int row_end,
                         cudaStream_t s) {
    Tree &tx = pl->tx, &ty = *pl->ty;
    Level &lx = tx.levels[level], &ly = ty.levels[level];
    const float scale = sqrtf(pl->lcs * 1.4426950408889634f);
    // Boxes in the middle of a cloud have lists a hundred times as long as the average: such a list, summed by one warp, outlasts all others.
    // Lists of large calls are cut into parts (chunk sources or so each, some ten thousand items in all, and at most some 2^17: a part
    // keeps 64 rows of sums until they are added up in the order of the list), and the host reads how many items there are; small
    // calls launch a bound.
    int chunk = 0;
    if (csr.pairs >= 100000000) {
        const int64_t even = std::min<int64_t>(32768, std::max<int64_t>(1024, csr.pairs / 600000));
        chunk = (int)std::min<int64_t>(1 << 20, std::max<int64_t>(even, csr.pairs / (CT << 17)));
    }
    // Groups of the expanded form: |X|^2 stays below d/4 times 1.25^2 around a parent's centre; boxes that narrow have sources no further away
    // than ungrouped ones of one scaled unit.  Error against float64 of boxes 0.6 units wide, alone / grouped at 1.19, positive weights: d = 3
    // 0.91 / 0.88e-7, d = 4 1.00 / 0.98e-7, d = 5 1.09 / 1.09e-7; normal ones 1.60 / 1.58, 2.07 / 2.03 and 2.01 / 1.97e-7.
    const bool grouped = DIFF || scale * tx.levels[level - 1].edge <= 1.25f;
    // one set of rows serves every list of the product
    f3m_plan::ColumnRows &cr = pl->column_rows;
    if (cr.r0 != r0) {
        cr.buf.alloc((size_t)ty.n * CROW, s);
        cr.r0 = r0;
        pl->last.begin(ST_PERMUTE, s);
        pack_column_rows<D><<<(unsigned)((ty.n * CROW + 255) / 256), 256, 0, s>>>(ty.pts.p, ty.n, bs, R, r0, cr.buf.p);
        F3M_LAUNCH_CHECK();
        pl->last.end(s);
    }
    const int nc = R - r0 <= 4 ? 4 : 8;
    DevBuf<int> items, slots, first;
    DevBuf<ColGroup> groups;
    DevBuf<float> parts;
    items.alloc((size_t)lx.nb + 1, s);
    slots.alloc((size_t)lx.nb + 1, s);
    first.alloc((size_t)lx.nb + 1, s);
    groups.alloc((size_t)lx.nb, s);
    const unsigned box_warps = (unsigned)(((int64_t)(lx.nb + 1) * 32 + 255) / 256);
    col_groups<<<box_warps, 256, 0, s>>>(lx.nb, lx.parent.p, csr.ptr.p, csr.idx.p, grouped, first.p);
    F3M_LAUNCH_CHECK();
    int64_t max_items = (int64_t)(row_end - row_begin) / CT + lx.nb + 1, nslots = 0;
    while (true) {
        col_items<<<box_warps, 256, 0, s>>>(lx.nb, lx.off.p, csr.ptr.p, csr.idx.p, ly.off.p, first.p, chunk, row_begin, row_end, items.p, slots.p,
                                            groups.p);
        F3M_LAUNCH_CHECK();
        int *scanned[2] = {items.p, slots.p};
        exclusive_scan_multi(scanned, chunk ? 2 : 1, (int64_t)lx.nb + 1, nullptr, s);
        if (!chunk) break;
        F3M_CUDA(cudaMemcpyAsync(pl->h_pinned, items.p + lx.nb, sizeof(int), cudaMemcpyDeviceToHost, s));
        F3M_CUDA(cudaMemcpyAsync(pl->h_pinned + 1, slots.p + lx.nb, sizeof(int), cudaMemcpyDeviceToHost, s));
        F3M_CUDA(cudaStreamSynchronize(s));
        max_items = pl->h_pinned[0];
        nslots = pl->h_pinned[1];
        if (max_items <= 0) return;
        if (!nslots) break;
        try {
            parts.alloc((size_t)nslots * CT * nc, s);
            break;
        } catch (const Fail &) {   // no memory for the parts' sums: lists are not cut
            cudaGetLastError();
            chunk = 0;
            nslots = 0;
            max_items = (int64_t)(row_end - row_begin) / CT + lx.nb + 1;
        }
    }
    pl->last.begin(ST_DIRECT, s);
    auto launch = [&](auto kernel) {
        kernel<<<(unsigned)max_items, 32, 0, s>>>(tx.pts.p, (int)tx.n, lx.off.p, lx.nb, lx.ctr.p, lx.parent.p, tx.levels[level - 1].ctr.p, items.p,
                                                 slots.p, groups.p, csr.ptr.p, csr.idx.p, ly.off.p, cr.buf.p, scale, R, r0, out, parts.p, row_begin,
                                                 row_end);
    };
    auto sum = [&](auto kernel) {
        kernel<<<(unsigned)nslots, CT * nc / 4, 0, s>>>(tx.levels[level].off.p, lx.nb, items.p, slots.p, groups.p, parts.p, R, r0, out, row_begin, row_end);
    };
    if (nc == 4) launch(near_columns<D, DIFF, 4>);
    else launch(near_columns<D, DIFF, 8>);
    if (nslots) {
        F3M_LAUNCH_CHECK();
        if (nc == 4) sum(col_parts_sum<4>);
        else sum(col_parts_sum<8>);
    }
    F3M_LAUNCH_CHECK();
    pl->last.end(s);
    pl->last.direct_launches++;
    pl->last.direct_variants[DIFF ? DV_DIRECT : DV_MUFU]++;
    pl->last.column_launches++;
    if (r0 == 0) pl->last.pairs[DIFF ? DV_DIRECT : DV_MUFU] += csr.pairs;
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
