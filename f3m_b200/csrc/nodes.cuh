// Interpolation shared by the far field (far_fast.cu) and the direct lists that go through nodes (near_nodes.cu): nodes, the order of a
// target box's rows, points to moments and local expansions to points in three dimensions.
#pragma once
#include <math.h>
#include <algorithm>
#include "common.cuh"
#include "packed.cuh"

namespace f3m {

constexpr int NOFF2 = 16;     // tabulated box offsets per dimension
constexpr int PMAX_FAST = 8;  // nodes per dimension the far field's fast path handles
constexpr int PMAX_NODES = 13;   // and the direct lists that go through nodes

struct NodeTab2 {
    int p;
    float node[PMAX_NODES];
    float c[PMAX_NODES];   // 1 / prod_{l != i} (node_i - node_l)
};

struct Geom2 {
    int dqmin[MAXD];
    double shift[MAXD];
};

__host__ __device__ constexpr int mat_stride(int p) { return (p * p + 3) / 4 * 4; }

static NodeTab2 make_nodes2(int p) {
    NodeTab2 t{};
    t.p = p;
    float w[PMAX_NODES];   // barycentric weights: the reference's form, not used here
    cheb_nodes_weights(p, t.node, w);
    for (int i = 0; i < p; i++) {
        double v = 1.0;
        for (int l = 0; l < p; l++)
            if (l != i) v *= (double)t.node[i] - (double)t.node[l];
        t.c[i] = (float)(1.0 / v);
    }
    return t;
}

__host__ __device__ constexpr int cpow(int b, int e) { return e <= 0 ? 1 : b * cpow(b, e - 1); }

static __global__ void __launch_bounds__(256) decode_cells_kernel(int nb, int level, int d, const uint32_t *__restrict__ code, int *cell) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const uint32_t c = code[b];
    for (int k = 0; k < d; k++) {
        int q = 0;
        for (int jb = 0; jb < level; jb++) q |= (int)((c >> (d * jb + k)) & 1u) << jb;
        cell[b * d + k] = q;
    }
}

// One warp per target box: packed offsets of its far pairs (axis 0 most significant) and the row in
// ascending order of them.  The source boxes of one row have distinct cells, hence distinct keys below
// 16^3: the rank of a key is the number of set bits below it in a bitmap of the row.
// In four and five dimensions the rank key is the base-8 number of the offsets counted from the lowest one
// that can occur (tabulated offset 4): 8^4 and 8^5 keys.  An offset outside that window is clamped; if two
// pairs of a row then share a rank key the row keeps its list order (every order is correct, see above).
// The row may be spread over several CSR lists (the cut level takes far, small and kept pairs alike): its segments are
// ordered together and written where a list holding all of them has the row.
struct ListSet {
    const int *ptr[3], *idx[3];
    int n;
};
static __global__ void __launch_bounds__(256) add_list_ptrs(int count, ListSet ls, int *ptr) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    int v = 0;
    for (int l = 0; l < ls.n; l++) v += ls.ptr[l][b];
    ptr[b] = v;
}

template <int WPL>   // bitmap words per lane: 4 -> 4096 rank keys, 32 -> 32768
static __global__ void __launch_bounds__(128) far_order_kernel(int nbx, int d, ListSet ls, const int *__restrict__ cell_x, const int *__restrict__ cell_y,
                                                       Geom2 geo, uint32_t *okey, int *oidx, int *err,
                                                       const int *__restrict__ off_x, int row_begin, int row_end) {
    constexpr int ORD_WORDS = 32 * WPL;
    __shared__ uint32_t bits[4][ORD_WORDS];
    __shared__ int below[4][ORD_WORDS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bx = blockIdx.x * 4 + w;
    if (bx >= nbx) return;
    if (off_x[bx + 1] <= row_begin || off_x[bx] >= row_end) return;   // no row of this box in the slice being computed
    int e0 = 0, n = 0, seg[3], cnt[3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
        seg[l] = cnt[l] = 0;
        if (l >= ls.n) continue;
        seg[l] = ls.ptr[l][bx];
        cnt[l] = ls.ptr[l][bx + 1] - seg[l];
        e0 += seg[l];
        n += cnt[l];
    }
    if (n == 0) return;
    auto source = [&](int i) {   // i-th source box of the row
        if (i < cnt[0]) return ls.idx[0][seg[0] + i];
        i -= cnt[0];
        return i < cnt[1] ? ls.idx[1][seg[1] + i] : ls.idx[2][seg[2] + i - cnt[1]];
    };
    const bool compact = d > 3;
    // key: one nibble per axis, last axis lowest, axis 0 on top; rkey: what the row is ordered by
    auto key_of = [&](int by, uint32_t &rkey) {
        uint32_t key = 0;
        rkey = 0;
        for (int k = 0; k < d; k++) {
            int o = cell_y[by * d + k] - cell_x[bx * d + k] - geo.dqmin[k];
            if (o < 0 || o >= NOFF2) { atomicExch(err, 2); o = 0; }
            key |= (uint32_t)o << (4 * (d - 1 - k));
            rkey = rkey * 8u + (uint32_t)min(max(o - 4, 0), 7);
        }
        if (!compact) rkey = key;
        return key;
    };
    for (int q = lane; q < ORD_WORDS; q += 32) bits[w][q] = 0u;
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        uint32_t rkey;
        key_of(source(i), rkey);
        atomicOr(&bits[w][rkey >> 5], 1u << (rkey & 31u));
    }
    __syncwarp();
    // exclusive prefix of the word populations: WPL words per lane, then a warp scan
    int tot = 0;
#pragma unroll 4
    for (int q = 0; q < WPL; q++) tot += __popc(bits[w][lane * WPL + q]);
    int incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    int run = incl - tot;
#pragma unroll 4
    for (int q = 0; q < WPL; q++) { below[w][lane * WPL + q] = run; run += __popc(bits[w][lane * WPL + q]); }
    const int distinct = __shfl_sync(0xffffffffu, incl, 31);
    __syncwarp();
    if (distinct != n) {   // cannot happen for d <= 3 (boxes of one level have distinct cells); keep the list order
        if (lane == 0 && !compact) atomicExch(err, 2);
        for (int i = lane; i < n; i += 32) { int by = source(i); uint32_t rk; okey[e0 + i] = key_of(by, rk); oidx[e0 + i] = by; }
        return;
    }
    for (int i = lane; i < n; i += 32) {
        const int by = source(i);
        uint32_t rkey;
        const uint32_t key = key_of(by, rkey);
        const int rank = below[w][rkey >> 5] + __popc(bits[w][rkey >> 5] & ((1u << (rkey & 31u)) - 1u));
        okey[e0 + rank] = key;
        oidx[e0 + rank] = by;
    }
}

// Lagrange basis at t (lagrange_data_load + calculate_barycentric_lagrange, 1_d_conv.cu:217-238, 418-448), as products of the
// differences t - t_l before and after node i: some 5 p multiplications and additions and no division; a point on a node
// needs no case of its own.  The barycentric form cost a reciprocal, a comparison and a select per node: half of all instructions
// of the leaf kernels.
// The middle entry is what the others leave of one, added from either end.  The roundings of a product are those of its p - 1 factors;
// where all entries carry them, the sum of the row is off by as much and with it every interpolated value, however smooth; now
// an entry's rounding meets the difference between its node's value and the middle one's only.  Emulated per axis, rows of both sides and the
// matrix in float32, p = 6 / 8 / 9 at 0.2 / 0.36 / 1.09 lengthscales: products 1.4 / 1.7 / 1.6e-7, barycentric (normalised)
// 1.1 / 1.25 / 1.3e-7, so 0.9 / 1.0 / 1.06e-7; rows rounded once from float64 0.8 / 0.9 / 0.9e-7.
template <int PP>
__device__ __forceinline__ void lagrange_pp(float t, const NodeTab2 &nt, float *L) {
    constexpr int MID = PP / 2;
    float diff[PP], after[PP];
#pragma unroll
    for (int i = 0; i < PP; i++) diff[i] = t - nt.node[i];
    after[PP - 1] = 1.f;
#pragma unroll
    for (int i = PP - 2; i >= 0; i--) after[i] = (i == PP - 2) ? diff[PP - 1] : after[i + 1] * diff[i + 1];
    float before = 1.f;
#pragma unroll
    for (int i = 0; i < PP; i++) {
        const float cb = i == 0 ? nt.c[0] : nt.c[i] * before;
        L[i] = i == PP - 1 ? cb : cb * after[i];
        before = i == 0 ? diff[0] : before * diff[i];
    }
    float low = L[0], high = MID == PP - 1 ? 0.f : L[PP - 1];   // of the entries as they are stored: nothing contracted
#pragma unroll
    for (int i = 1; i < MID; i++) low = __fadd_rn(low, L[i]);
#pragma unroll
    for (int i = PP - 2; i > MID; i--) high = __fadd_rn(high, L[i]);
    L[MID] = __fsub_rn(__fsub_rn(1.f, low), high);
}
// the same for two points at once
template <int PP>
__device__ __forceinline__ void lagrange_pair(f32x2 t, const NodeTab2 &nt, f32x2 (&L)[PP]) {
    constexpr int MID = PP / 2;
    const f32x2 one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
    f32x2 diff[PP], after[PP];
#pragma unroll
    for (int i = 0; i < PP; i++) diff[i] = add2(t, pack2(-nt.node[i], -nt.node[i]));
#pragma unroll
    for (int i = PP - 2; i >= 0; i--) after[i] = (i == PP - 2) ? diff[PP - 1] : mul2(after[i + 1], diff[i + 1]);
    f32x2 before = diff[0];
#pragma unroll
    for (int i = 0; i < PP; i++) {
        if (i != MID) {
            f32x2 cb = pack2(nt.c[i], nt.c[i]);
            if (i > 0) cb = mul2(cb, before);
            L[i] = i == PP - 1 ? cb : mul2(cb, after[i]);
        }
        if (i > 0) before = mul2(before, diff[i]);
    }
    f32x2 low = L[0], high = MID == PP - 1 ? 0ull : L[PP - 1];
#pragma unroll
    for (int i = 1; i < MID; i++) low = add2(low, L[i]);
#pragma unroll
    for (int i = PP - 2; i > MID; i--) high = add2(high, L[i]);
    L[MID] = fma2(minus, high, fma2(minus, low, one));
}

// What a CTA of the P2M kernels sums: the first nlist take a box each (all its rows, unless the box is long), the others a slot of
// the long boxes' parts.  Boxes that start outside [src_begin, src_end) belong to another slice of the sorted sources.
struct LeafWork { int box, s0, s1; int64_t slot; };
__device__ __forceinline__ LeafWork leaf_work(const int *__restrict__ off, int nb, int n, const int *__restrict__ box_list, int nlist, int chunk,
                                              int src_begin, int src_end) {
    LeafWork w{0, 0, 0, -1};
    if ((int)blockIdx.x < nlist) {
        w.box = box_list ? box_list[blockIdx.x] : (int)blockIdx.x;
        w.s0 = off[w.box];
        w.s1 = off[w.box + 1];
        if (chunk && w.s1 - w.s0 > chunk) w.s1 = w.s0;
    } else {
        w.slot = blockIdx.x - nlist;
        const BoxPart p = part_of_slot(off, nb, n, chunk, w.slot);
        w.box = p.box; w.s0 = p.begin; w.s1 = p.end;
    }
    const int a = off[w.box];
    if (a < src_begin || a >= src_end) w.s1 = w.s0;
    return w;
}

// Moments of the long boxes: the sums of their parts, in the order of the rows, with the rounding of every addition carried along
// (Knuth's two-sum; the loads of the parts take the time).  A tree that ends at a level whose boxes hold hundreds of thousands of points has
// hundreds of parts per box, and a plain running sum was most of the product's error.  Error over sqrt(n), normal weights, l = 10, 300
// products each, plain / now: 3e6 points 3.65 / 2.46e-7, 1e7 3.77 / 2.77e-7, 3e7 4.53 / 2.74e-7; a kept plan, which interpolates its
// sources further down and adds them in a tree (far_fast.cu, SRC_LEAF), 2.71, 3.24 and 3.45e-7 with plain sums.
static __global__ void __launch_bounds__(128) p2m_combine(const int *__restrict__ off, int nb, int n, int chunk, int PR, int src_begin, int src_end,
                                                  const float *__restrict__ part, float *mom) {
    const LongBox l = long_box_of_chunk(off, nb, n, chunk, blockIdx.x);
    if (l.box < 0 || off[l.box] < src_begin || off[l.box] >= src_end) return;
    for (int q = threadIdx.x; q < PR; q += 128) {
        float v = part[l.first_slot * PR + q], lost = 0.f;
        for (int64_t t = (l.first_slot | 1) + 1; t <= l.last_slot; t += 2) {
            const float x = part[t * PR + q], sum = __fadd_rn(v, x), w = __fsub_rn(sum, v);
            lost += __fadd_rn(__fsub_rn(v, __fsub_rn(sum, w)), __fsub_rn(x, w));
            v = sum;
        }
        mom[(size_t)l.box * PR + q] = isfinite(v) ? v + lost : v;
    }
}

// ---------------------------------------------------------------------------------------------
// P2M / L2P for d = 3 and one column, register-tiled.  A lane is (stream, m2): it keeps the PP x PP block (m0, m1) of the
// box's moments (or local expansion) for its m2 in registers and takes two points at a time, one in either half of every
// packed instruction, so that nothing has to be duplicated: PP multiplications and PP^2 multiply-adds per two points against
// 16-byte loads of their Lagrange rows.  A warp works alone: its lanes first build the rows of two points each (coordinates
// of the next ones are on their way meanwhile), then 32 / PP streams share them; CTAs meet only to add up.  Bound: FP32 lanes, PP^2 + PP
// of them per point and m2 besides some 30 per axis for the rows.  1e8 points, 216 nodes, against one point at
// a time, barycentric rows and CTA-wide chunks: p2m_leaf3 2.11 -> 1.61 ms, l2p_leaf3 2.46 -> 1.56 ms (0.62 at the FMA rate).
// A row [L0 | L1 | L2] holds its two points alternating; rows are RS floats apart, an odd number of 16-byte groups, which puts
// the streams of a warp on different banks.
// ---------------------------------------------------------------------------------------------
template <int PP>
struct Leaf3 {
    static constexpr int SUB = 32 / PP;              // streams per warp
    static constexpr int ROWS = 32 / SUB * SUB;      // rows (pairs of points) per warp and chunk
    static constexpr int WP = 2 * ROWS;              // points per warp and chunk
    static constexpr int NSTREAM = 4 * SUB;          // per CTA
    static constexpr int AX = (2 * PP + 3) / 4 * 4;  // floats per axis
    static constexpr int RS = 3 * AX % 8 == 4 ? 3 * AX : 3 * AX + 4;
};

template <int PP>
__device__ __forceinline__ void leaf3_rows(const float *__restrict__ pts, int n, int i, const float (&c)[3], float factor,
                                           const NodeTab2 &nt, float scale2, float *row) {
    float L[PP];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        lagrange_pp<PP>(factor * (pts[(size_t)k * n + i] - c[k]), nt, L);
#pragma unroll
        for (int q = 0; q < PP; q++) row[8 * k + q] = (k == 2) ? scale2 * L[q] : L[q];
    }
}

// rows of two points at once, xa and xb; the third axis carries the factors f
// Centre of a box: a float per axis (the level's ctr), or FINE, two floats whose sum it is (fine_centres below).  Node-to-node tables know
// whole multiples of the edge: a centre rounded to a float is off by up to 1e-7 of its own size, which boxes about as wide as the
// lengthscale would see as 1e-6 of the kernel.
template <bool FINE> struct Centre3 {
    float hi[3], lo[3];
    __device__ __forceinline__ Centre3(const float *__restrict__ ctr, int box) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            hi[k] = ctr[(FINE ? 6 : 3) * box + k];
            lo[k] = FINE ? ctr[6 * box + 3 + k] : 0.f;
        }
    }
    __device__ __forceinline__ float from(float x, int k) const { return FINE ? (x - hi[k]) - lo[k] : x - hi[k]; }
};
struct Origin3 { float x[3]; };
static __global__ void __launch_bounds__(256) fine_centres(int nb, Origin3 o, double edge, const int *__restrict__ cell, float *ctr) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= 3 * nb) return;
    const int box = i / 3, k = i - 3 * box;
    const double c = (double)o.x[k] + ((double)cell[i] + 0.5) * edge;
    ctr[6 * box + k] = (float)c;
    ctr[6 * box + 3 + k] = (float)(c - (double)(float)c);
}

template <int PP, bool FINE>
__device__ __forceinline__ void leaf3_row_pair(const float (&xa)[3], const float (&xb)[3], const Centre3<FINE> &c, float factor,
                                               const NodeTab2 &nt, f32x2 f, float *row) {
    using G = Leaf3<PP>;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const f32x2 t = pack2(factor * c.from(xa[k], k), factor * c.from(xb[k], k));
        f32x2 L[PP];
        lagrange_pair<PP>(t, nt, L);
        if (k == 2)
#pragma unroll
            for (int i = 0; i < PP; i++) L[i] = mul2(L[i], f);
        ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(row + k * G::AX);
#pragma unroll
        for (int q = 0; q < G::AX / 4; q++) dst[q] = make_ulonglong2(L[2 * q], 2 * q + 1 < PP ? L[2 * q + 1] : 0ull);
    }
}
template <int PP>
__device__ __forceinline__ void leaf3_load_axis(const float *axis, f32x2 (&l)[PP]) {
#pragma unroll
    for (int q = 0; q < PP / 2; q++) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(axis)[q];
        l[2 * q] = v.x;
        l[2 * q + 1] = v.y;
    }
    if (PP & 1) l[PP - 1] = *reinterpret_cast<const f32x2 *>(axis + 2 * PP - 2);
}

template <int PP, bool FINE>
static __global__ void __launch_bounds__(128) p2m_leaf3(const float *__restrict__ pts, int n, const float *__restrict__ bs, int R, int r0,
                                                const int *__restrict__ off, const float *__restrict__ ctr, float factor,
                                                NodeTab2 nt, int nb, int chunk, int src_begin, int src_end, float *mom, float *part,
                                                const int *__restrict__ box_list, int nlist) {
    using G = Leaf3<PP>;
    constexpr int P = PP * PP * PP;
    // the warps' rows; at the end of a block of points the same memory holds one partial moment array per stream
    constexpr int NSCR = (4 * G::ROWS * G::RS > G::NSTREAM * P) ? 4 * G::ROWS * G::RS : G::NSTREAM * P;
    __shared__ __align__(16) float scr[NSCR];
    const LeafWork lw = leaf_work(off, nb, n, box_list, nlist, chunk, src_begin, src_end);
    const int box = lw.box, s0 = lw.s0, s1 = lw.s1;
    if (s0 >= s1) return;
    const Centre3<FINE> c(ctr, box);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / PP, m2 = lane - sub * PP;
    const bool active = sub < G::SUB;
    const int stream = warp * G::SUB + sub;
    float *rows = scr + warp * G::ROWS * G::RS;
    // Running sums grow inaccurate with the square root of their length: after some fifty terms in either half of a stream (BLOCK
    // points) they are added up over the streams and kept by the threads that write the moments.
    constexpr int BLOCK = 2048 / (4 * G::WP) * (4 * G::WP);
    float tot[(P + 127) / 128];
#pragma unroll
    for (int t = 0; t < (P + 127) / 128; t++) tot[t] = 0.f;
    // the next two points of the lane are fetched while the streams consume the current ones; points past the end weigh nothing
    float xa[3], xb[3], ba, bb;
    auto fetch = [&](int base) {
        const int ia = base + lane, ib = ia + G::ROWS;
        const bool ha = ia < s1, hb = ib < s1;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            xa[k] = ha ? pts[(size_t)k * n + ia] : c.hi[k];
            xb[k] = hb ? pts[(size_t)k * n + ib] : c.hi[k];
        }
        ba = ha ? bs[(size_t)ia * R + r0] : 0.f;
        bb = hb ? bs[(size_t)ib * R + r0] : 0.f;
    };
    fetch(s0 + warp * G::WP);
    for (int block = s0; block < s1; block += BLOCK) {
        f32x2 acc[PP][PP];
#pragma unroll
        for (int i = 0; i < PP; i++)
#pragma unroll
            for (int j = 0; j < PP; j++) acc[i][j] = 0ull;
        const int bend = min(block + BLOCK, s1);
        for (int base = block + warp * G::WP; base < bend; base += 4 * G::WP) {
            __syncwarp();
            if (lane < G::ROWS) leaf3_row_pair<PP, FINE>(xa, xb, c, factor, nt, pack2(ba, bb), rows + lane * G::RS);
            fetch(base + 4 * G::WP);
            __syncwarp();
            const int cnt = min(G::ROWS, s1 - base);
            if (active)
#pragma unroll 1
                for (int j = sub; j < cnt; j += G::SUB) {
                    const float *row = rows + j * G::RS;
                    f32x2 l0[PP], l1[PP];
                    leaf3_load_axis<PP>(row, l0);
                    leaf3_load_axis<PP>(row + G::AX, l1);
                    const f32x2 w2 = *reinterpret_cast<const f32x2 *>(row + 2 * G::AX + 2 * m2);
#pragma unroll
                    for (int i1 = 0; i1 < PP; i1++) {
                        const f32x2 u = mul2(w2, l1[i1]);
#pragma unroll
                        for (int i0 = 0; i0 < PP; i0++) acc[i1][i0] = fma2(u, l0[i0], acc[i1][i0]);
                    }
                }
        }
        __syncthreads();
        if (active) {
            float *mine = scr + stream * P + PP * PP * m2;
#pragma unroll
            for (int i1 = 0; i1 < PP; i1++)
#pragma unroll
                for (int i0 = 0; i0 < PP; i0++) {
                    float a, b;
                    unpack2(acc[i1][i0], a, b);
                    mine[i0 + PP * i1] = a + b;
                }
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < (P + 127) / 128; t++) {
            const int q = threadIdx.x + 128 * t;
            float v = 0.f;
            if (q < P) {
#pragma unroll
                for (int st = 0; st < G::NSTREAM; st++) v += scr[st * P + q];
            }
            tot[t] += v;
        }
        __syncthreads();
    }
    float *dst = lw.slot < 0 ? mom + (size_t)box * P : part + lw.slot * P;
#pragma unroll
    for (int t = 0; t < (P + 127) / 128; t++)
        if ((int)threadIdx.x + 128 * t < P) dst[threadIdx.x + 128 * t] = tot[t];
}

template <int PP, bool FINE>
static __global__ void __launch_bounds__(128) l2p_leaf3(const float *__restrict__ pts, int n, const int *__restrict__ off,
                                                const float *__restrict__ ctr, float factor, NodeTab2 nt, int nsplit,
                                                int row_begin, int row_end, const float *__restrict__ loc, int R, int r0,
                                                float *out, const int *__restrict__ box_list) {
    using G = Leaf3<PP>;
    constexpr int P = PP * PP * PP;
    __shared__ __align__(16) float scr[4 * G::ROWS * G::RS];
    const int box = box_list ? box_list[blockIdx.x] : (int)blockIdx.x;
    const int a = off[box], b = off[box + 1];
    if (a < row_begin || a >= row_end) return;    // finest-level boxes belong to the slice their first point is in
    const int len = b - a;
    const int s0 = a + (int)(((long long)len * blockIdx.y) / nsplit), s1 = a + (int)(((long long)len * (blockIdx.y + 1)) / nsplit);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (s0 + warp * G::WP >= s1) return;          // warps do not meet
    const Centre3<FINE> c(ctr, box);
    const int sub = lane / PP, m2 = lane - sub * PP;
    const bool active = sub < G::SUB;
    float *rows = scr + warp * G::ROWS * G::RS;
    f32x2 lc[PP][PP];   // loc[m0][m1][m2] of this lane's m2, twice
#pragma unroll
    for (int i1 = 0; i1 < PP; i1++)
#pragma unroll
        for (int i0 = 0; i0 < PP; i0++) {
            const float v = active ? __ldg(loc + (size_t)box * P + i0 + PP * i1 + PP * PP * m2) : 0.f;
            lc[i1][i0] = pack2(v, v);
        }
    float xa[3], xb[3], oa, ob;
    auto fetch = [&](int base) {
        const int ia = base + lane, ib = ia + G::ROWS;
        const bool mine = lane < G::ROWS, ha = mine && ia < s1, hb = mine && ib < s1;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            xa[k] = ha ? pts[(size_t)k * n + ia] : c.hi[k];
            xb[k] = hb ? pts[(size_t)k * n + ib] : c.hi[k];
        }
        oa = ha ? out[(size_t)ia * R + r0] : 0.f;
        ob = hb ? out[(size_t)ib * R + r0] : 0.f;
    };
    fetch(s0 + warp * G::WP);
    for (int base = s0 + warp * G::WP; base < s1; base += 4 * G::WP) {
        __syncwarp();
        if (lane < G::ROWS) leaf3_row_pair<PP, FINE>(xa, xb, c, factor, nt, pack2(1.f, 1.f), rows + lane * G::RS);
        const float pa = oa, pb = ob;
        fetch(base + 4 * G::WP);   // the next points and their sums so far, while the streams consume these
        __syncwarp();
        const int cnt = min(G::ROWS, s1 - base);
        if (active)
#pragma unroll 1
            for (int j = sub; j < cnt; j += G::SUB) {
                float *row = rows + j * G::RS;
                f32x2 l0[PP], l1[PP];
                leaf3_load_axis<PP>(row, l0);
                leaf3_load_axis<PP>(row + G::AX, l1);
                f32x2 *w2 = reinterpret_cast<f32x2 *>(row + 2 * G::AX + 2 * m2);
                f32x2 sum = 0ull;
#pragma unroll
                for (int i1 = 0; i1 < PP; i1++) {
                    f32x2 t = mul2(l0[0], lc[i1][0]);
#pragma unroll
                    for (int i0 = 1; i0 < PP; i0++) t = fma2(l0[i0], lc[i1][i0], t);
                    sum = fma2(l1[i1], t, sum);
                }
                *w2 = mul2(*w2, sum);   // only this lane reads the entry: the partial sums over m2 take its place
            }
        __syncwarp();
        if (lane < cnt) {
            f32x2 l2[PP];
            leaf3_load_axis<PP>(rows + lane * G::RS + 2 * G::AX, l2);
            f32x2 v = l2[0];
#pragma unroll
            for (int q = 1; q < PP; q++) v = add2(v, l2[q]);
            float va, vb;
            unpack2(v, va, vb);
            const int ia = base + lane, ib = ia + G::ROWS;
            out[(size_t)ia * R + r0] = pa + va;
            if (ib < s1) out[(size_t)ib * R + r0] = pb + vb;
        }
    }
}

// Parts the target boxes of a level are cut into (every box into the same number): at most 8192 points in the longest box, and short
// enough that the parts of all boxes fill the SMs four times over (a cut at level 1 or 2 leaves 8 or 64 boxes), but not below
// 512 points.  Levels of uneven occupancy would launch a part for each of a million short boxes because one is long: the number of CTAs
// is held to the boxes plus four times the parts that an even level would have, but parts never grow beyond what 64 parts of
// 8192 points give.  The parts are the second dimension of a grid: at most 65535.
static int target_parts(int max_count, int64_t n, int nb) {
    const int64_t part = std::max<int64_t>(512, std::min<int64_t>(8192, n / (4 * NUM_SMS_HINT)));
    const int64_t want = (max_count + part - 1) / part, even = 1 + 4 * n / (part * nb), at_least = std::min(64, (max_count + 8191) / 8192);
    return (int)std::min<int64_t>(65535, std::max<int64_t>(1, std::max<int64_t>(at_least, std::min<int64_t>(want, even))));
}
// Rows from which a source box is summed in parts; 0: no box of the level is that long.  A CTA works through its rows one chunk of
// 128 after the other, so a box that is much longer than the SMs' even share ends last.  Whole calls in us, parts per SM 4 / 8 / 12:
// two trees in 2-D, 60 007 sources, 3 columns (p2m_leaf) 856 / 817 / -; FALKON, 2e6 sources (p2m_leaf3) 454 / 443 / 441, 1024 rows 433.
static int source_chunk(int max_count, int64_t n, bool blocked) {
    const int64_t share = n / ((blocked ? 8 : 16) * NUM_SMS_HINT);
    const int chunk = (int)std::max<int64_t>(blocked ? 256 : 512, std::min<int64_t>(8192, share));
    return max_count > chunk ? chunk : 0;
}

}  // namespace f3m
