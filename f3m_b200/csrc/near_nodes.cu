// Direct lists through interpolation nodes (three dimensions, one column, one point set).
//
// The pairs of a near / small list (near_field_run, F3M_src/n_tree.cu:831-902) are pairs of boxes of one level.  Where the boxes
// are populated and no wider than about two lengthscales, p nodes per axis, p chosen here whatever the caller's node count,
// reproduce the kernel to rounding for every pair of points (bound below), and the list becomes: points to moments, a node-to-node step per
// pair of boxes, local expansions to points.  A pair of boxes then costs p^4 multiply-adds for the axis that changes from pair to
// pair, and the other axes once per group of pairs (the nested form of far_fast.cu), against n_x n_y exponentials and 4 n_x n_y
// multiply-adds: 6561 against some 15 000 pairs at 122 points per box and p = 9.  The far field's pairs are not touched: they keep the
// caller's nodes.
#include <math.h>
#include <algorithm>
#include "common.cuh"
#include "nodes.cuh"
#include "packed.cuh"

namespace f3m {

// ---------------------------------------------------------------------------------------------
// Nodes a list needs.  Per axis g(u) = exp(-u^2 / 2 l^2) is interpolated in x and in y over an edge e: with Cramer's inequality the
// error is at most (1 + Lambda_p) 2 * 1.0865 (e / 4 l)^p / sqrt(p!), Lambda_p <= 1 + (2 / pi) ln p (the derivation stands in
// far_fast.cu); the axes' errors add up.  The bound is taken against the kernel's largest value, 1: a row is off by at most NODE_EPS times the
// sum of |b| over its list, besides roundings of the same kind.  (The cut of far_fast.cu bounds every pair against its own value,
// which these wide boxes cannot meet at their far corners.)  At the bound the products of 64 bits differ by a fifth of it in the 2-norm:
// boxes 1.09 l wide, 9 nodes, bound 3.1e-7, measured 1e-8; 0.55 l, 7 nodes, bound 2.6e-7, measured 5e-8 -- below the roundings.
// Against float64, pairs of near.cu (whole products) / nodes, 2-norm, 1e-7: normal weights, 0.55 l 4.2 / 2.5, 1.09 l 3.3 / 2.6, 2.3 l 6.3 / 3.4;
// positive ones 1.5 / 1.2, 1.7 / 1.6, 2.1 / 1.9; targets by themselves beside boxes of 2e4 points, worst row relative to its sum of
// |K b|: 0.55 l 52 / 7, 1.09 l 134 / 85.  Few weights that are not zero make short sums, whose pairs are the more exact ones: one in
// a hundred 1.8 / 2.5, 1.9 / 2.4, 5.4 / 3.1, a single one 1.0 / 1.6, 1.1 / 1.8, 4.2 / 2.5, and entries far below 1 keep their digits.  From
// one in ten on they are even, so products of sparser weights sum the pairs.
// ---------------------------------------------------------------------------------------------
constexpr double NODE_EPS = 4e-7;
constexpr int SPARSE_WEIGHTS = 10;   // fewer than one weight in so many not zero: pairs
constexpr int PMIN_NODES = 5;

static int nodes_needed(double edge_over_l) {
    for (int p = PMIN_NODES; p <= PMAX_NODES; p++) {
        double fact = 1.0;
        for (int i = 2; i <= p; i++) fact *= i;
        const double E = 2.0 * 1.0865 * pow(edge_over_l / 4.0, p) / sqrt(fact);
        if (3.0 * E * (2.0 + 2.0 / 3.14159265358979323846 * log((double)p)) <= NODE_EPS) return p;
    }
    return 0;
}

// ---------------------------------------------------------------------------------------------
// P2M / L2P for more than eight nodes: as p2m_leaf3 / l2p_leaf3 (two points per packed instruction, rows in shared memory), but a
// unit of work is (m2, group of G1 values of m1), so that its block of G1 x PP entries fits the registers, and the CTA shares its rows.
// ---------------------------------------------------------------------------------------------
template <int PP>
struct Wide3 {
    static constexpr int G1 = PP == 9 ? 3 : PP == 10 ? 5 : PP == 11 ? 6 : PP == 12 ? 4 : 5;
    static constexpr int NG = (PP + G1 - 1) / G1;
    static constexpr int UNITS = PP * NG;
    static constexpr int S = 128 / UNITS;              // streams per CTA
    static constexpr int ROWS = 64;                    // pairs of points per chunk
    static constexpr int AX0 = (2 * PP + 3) / 4 * 4;   // floats of the first and last axis
    static constexpr int AX1 = (2 * NG * G1 + 3) / 4 * 4;
    static constexpr int LEN = 2 * AX0 + AX1;
    static constexpr int RS = LEN % 8 == 4 ? LEN : LEN + 4;
};

template <int PP>
__device__ __forceinline__ void wide_row_pair(const float (&xa)[3], const float (&xb)[3], const Centre3<true> &c, float factor,
                                              const NodeTab2 &nt, f32x2 f, float *row) {
    using G = Wide3<PP>;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const f32x2 t = pack2(factor * c.from(xa[k], k), factor * c.from(xb[k], k));
        f32x2 L[PP];
        lagrange_pair<PP>(t, nt, L);
        f32x2 *dst = reinterpret_cast<f32x2 *>(row + (k == 0 ? 0 : k == 1 ? G::AX0 : G::AX0 + G::AX1));
#pragma unroll
        for (int i = 0; i < PP; i++) dst[i] = k == 2 ? mul2(L[i], f) : L[i];
        if (k == 1)
#pragma unroll
            for (int i = PP; i < G::NG * G::G1; i++) dst[i] = 0ull;   // the last group's surplus
    }
}
template <int PP>
__device__ __forceinline__ void wide_load_l0(const float *row, f32x2 (&l)[PP]) {
#pragma unroll
    for (int q = 0; q < PP / 2; q++) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(row)[q];
        l[2 * q] = v.x;
        l[2 * q + 1] = v.y;
    }
    if (PP & 1) l[PP - 1] = *reinterpret_cast<const f32x2 *>(row + 2 * PP - 2);
}

template <int PP>
__global__ void __launch_bounds__(128) p2m_wide3(const float *__restrict__ pts, int n, const float *__restrict__ bs,
                                                const int *__restrict__ off, const float *__restrict__ ctr, float factor, NodeTab2 nt,
                                                int nb, int chunk, float *mom, float *part) {
    using G = Wide3<PP>;
    constexpr int P = PP * PP * PP;
    extern __shared__ __align__(16) float rows[];   // rows of a chunk, or at the end one partial array per stream
    const LeafWork lw = leaf_work(off, nb, n, nullptr, nb, chunk, 0, n);
    const int box = lw.box, s0 = lw.s0, s1 = lw.s1;
    if (s0 >= s1) return;
    const Centre3<true> c(ctr, box);
    const int tid = threadIdx.x, stream = tid / G::UNITS, unit = tid - stream * G::UNITS, m2 = unit / G::NG, g = unit - m2 * G::NG;
    const bool active = stream < G::S;
    constexpr int BLOCK = 1024;   // points between two sums over the streams (p2m_leaf3)
    float tot[(P + 127) / 128];
#pragma unroll
    for (int t = 0; t < (P + 127) / 128; t++) tot[t] = 0.f;
    for (int block = s0; block < s1; block += BLOCK) {
        f32x2 acc[G::G1][PP];
#pragma unroll
        for (int i = 0; i < G::G1; i++)
#pragma unroll
            for (int j = 0; j < PP; j++) acc[i][j] = 0ull;
        const int bend = min(block + BLOCK, s1);
        for (int base = block; base < bend; base += 2 * G::ROWS) {
            const int cnt = min(2 * G::ROWS, bend - base), nrow = min(G::ROWS, cnt);
            __syncthreads();
            if (tid < nrow) {   // the row of the points tid and tid + ROWS of the chunk; one past the end weighs nothing
                const int ia = base + tid, ib = ia + G::ROWS;
                const bool hb = ib < bend;
                float xa[3], xb[3];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    xa[k] = pts[(size_t)k * n + ia];
                    xb[k] = hb ? pts[(size_t)k * n + ib] : c.hi[k];
                }
                wide_row_pair<PP>(xa, xb, c, factor, nt, pack2(bs[ia], hb ? bs[ib] : 0.f), rows + tid * G::RS);
            }
            __syncthreads();
            if (active)
#pragma unroll 1
                for (int j = stream; j < nrow; j += G::S) {
                    const float *row = rows + j * G::RS;
                    f32x2 l0[PP];
                    wide_load_l0<PP>(row, l0);
                    const f32x2 *l1 = reinterpret_cast<const f32x2 *>(row + G::AX0) + g * G::G1;
                    const f32x2 w2 = reinterpret_cast<const f32x2 *>(row + G::AX0 + G::AX1)[m2];
#pragma unroll
                    for (int i1 = 0; i1 < G::G1; i1++) {
                        const f32x2 u = mul2(w2, l1[i1]);
#pragma unroll
                        for (int i0 = 0; i0 < PP; i0++) acc[i1][i0] = fma2(u, l0[i0], acc[i1][i0]);
                    }
                }
        }
        __syncthreads();
        if (active)
#pragma unroll
            for (int i1 = 0; i1 < G::G1; i1++)
                if (g * G::G1 + i1 < PP)
#pragma unroll
                    for (int i0 = 0; i0 < PP; i0++) {
                        float a, b;
                        unpack2(acc[i1][i0], a, b);
                        rows[stream * P + i0 + PP * (g * G::G1 + i1) + PP * PP * m2] = a + b;
                    }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < (P + 127) / 128; t++) {
            const int q = tid + 128 * t;
            float v = 0.f;
            if (q < P) {
#pragma unroll
                for (int st = 0; st < G::S; st++) v += rows[st * P + q];
            }
            tot[t] += v;
        }
    }
    float *dst = lw.slot < 0 ? mom + (size_t)box * P : part + lw.slot * P;
#pragma unroll
    for (int t = 0; t < (P + 127) / 128; t++)
        if (tid + 128 * t < P) dst[tid + 128 * t] = tot[t];
}

template <int PP>
__global__ void __launch_bounds__(128) l2p_wide3(const float *__restrict__ pts, int n, const int *__restrict__ off,
                                                const float *__restrict__ ctr, float factor, NodeTab2 nt, int nsplit,
                                                const int *__restrict__ ptr1, const int *__restrict__ ptr2, const float *__restrict__ loc,
                                                float *out) {
    using G = Wide3<PP>;
    constexpr int P = PP * PP * PP, PS = G::UNITS | 1;
    extern __shared__ __align__(16) float rows[];
    f32x2 *part = reinterpret_cast<f32x2 *>(rows + G::ROWS * G::RS);   // per row: the units' shares of its two points
    const int box = blockIdx.x;
    if (ptr1[box] == ptr1[box + 1] && (!ptr2 || ptr2[box] == ptr2[box + 1])) return;
    const int a = off[box], len = off[box + 1] - a;
    const int s0 = a + (int)(((long long)len * blockIdx.y) / nsplit), s1 = a + (int)(((long long)len * (blockIdx.y + 1)) / nsplit);
    if (s0 >= s1) return;
    const Centre3<true> c(ctr, box);
    const int tid = threadIdx.x, stream = tid / G::UNITS, unit = tid - stream * G::UNITS, m2 = unit / G::NG, g = unit - m2 * G::NG;
    const bool active = stream < G::S;
    f32x2 lc[G::G1][PP];
#pragma unroll
    for (int i1 = 0; i1 < G::G1; i1++)
#pragma unroll
        for (int i0 = 0; i0 < PP; i0++) {
            const int m1 = g * G::G1 + i1;
            const float v = active && m1 < PP ? __ldg(loc + (size_t)box * P + i0 + PP * m1 + PP * PP * m2) : 0.f;
            lc[i1][i0] = pack2(v, v);
        }
    for (int base = s0; base < s1; base += 2 * G::ROWS) {
        const int nrow = min(G::ROWS, s1 - base);
        const int ia = base + tid, ib = ia + G::ROWS;
        const bool ha = tid < nrow, hb = ha && ib < s1;
        float oa = 0.f, ob = 0.f;
        __syncthreads();
        if (ha) {
            float xa[3], xb[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                xa[k] = pts[(size_t)k * n + ia];
                xb[k] = hb ? pts[(size_t)k * n + ib] : c.hi[k];
            }
            oa = out[ia];
            if (hb) ob = out[ib];
            wide_row_pair<PP>(xa, xb, c, factor, nt, pack2(1.f, 1.f), rows + tid * G::RS);
        }
        __syncthreads();
        if (active)
#pragma unroll 1
            for (int j = stream; j < nrow; j += G::S) {
                const float *row = rows + j * G::RS;
                f32x2 l0[PP];
                wide_load_l0<PP>(row, l0);
                const f32x2 *l1 = reinterpret_cast<const f32x2 *>(row + G::AX0) + g * G::G1;
                f32x2 sum = 0ull;
#pragma unroll
                for (int i1 = 0; i1 < G::G1; i1++) {
                    f32x2 t = mul2(l0[0], lc[i1][0]);
#pragma unroll
                    for (int i0 = 1; i0 < PP; i0++) t = fma2(l0[i0], lc[i1][i0], t);
                    sum = fma2(l1[i1], t, sum);
                }
                part[j * PS + unit] = mul2(reinterpret_cast<const f32x2 *>(row + G::AX0 + G::AX1)[m2], sum);
            }
        __syncthreads();
        if (ha) {
            f32x2 v = part[tid * PS];
#pragma unroll 4
            for (int q = 1; q < G::UNITS; q++) v = add2(v, part[tid * PS + q]);
            float va, vb;
            unpack2(v, va, vb);
            out[ia] = oa + va;
            if (hb) out[ib] = ob + vb;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Node-to-node step: one CTA per target box, its groups of WPG warps share the row, which is ordered by (o0, o1, o2).  A thread
// owns FPT fibres (positions m0, m1) of the sums V over the pairs of one (o0, o1): per pair it reads their PP moments along the last
// axis and applies that axis' matrix, whose columns come from shared memory as broadcasts -- FPT * PP multiply-adds per PP / 4 of
// them, two outputs per instruction (p = 9: 2.67 -> 2.28 ms; one by one the issue slots were 65 % busy, the FMA pipe 47 %).  When (o0, o1) changes V is laid out anew for the axis before, as in m2l_nested.  Bound: FP32 lanes (NF of FPT * 32 * WPG
// busy), then the groups' ends.
// ---------------------------------------------------------------------------------------------
template <int PP>
struct ColCfg {
    static constexpr int NF = PP * PP, P = PP * PP * PP;
    static constexpr int WPG = PP <= 11 ? 1 : 2;
    static constexpr int NT = 32 * WPG, NGRP = 4 / WPG;
    static constexpr int FPT = (NF + NT - 1) / NT;
    static constexpr int MSR = (PP + 3) / 4 * 4;      // floats per matrix column
    static constexpr int MS = PP * MSR;
    static constexpr size_t smem = (size_t)(3 * NOFF2 * MS + 2 * NGRP * P) * sizeof(float);
};

// T[k][o][j * MSR + i] = exp(-lcs (g_i - g_j - delta)^2), delta = (o + dqmin) edge (the tables of setup_levels in far_fast.cu, columns first)
static __global__ void column_table(NodeTab2 nt, double edge, double lcs, int dqmin, float *T) {
    const int p = nt.p, MSR = (p + 3) / 4 * 4, MS = p * MSR, tot = 3 * NOFF2 * MS;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += gridDim.x * blockDim.x) {
        const int q = e % MS, o = (e / MS) % NOFF2, j = q / MSR, i = q - j * MSR;
        float v = 0.f;
        if (i < p) {
            const double diff = ((double)nt.node[i] - (double)nt.node[j]) * edge * 0.5 - (double)(o + dqmin) * edge;
            v = (float)exp(-lcs * diff * diff);
        }
        T[e] = v;
    }
}

template <int WPG>
__device__ __forceinline__ void group_sync(int group) {
    if (WPG == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(32 * WPG) : "memory");
}

// A thread's sums: PP values of each of its fibres, two to a register pair (the last one of an odd number by itself)
template <int PP>
struct ColAcc {
    static constexpr int FPT = ColCfg<PP>::FPT, NP = PP / 2, ODD = PP & 1;
    f32x2 p[FPT][NP];
    float last[FPT];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int r = 0; r < FPT; r++) {
#pragma unroll
            for (int i = 0; i < NP; i++) p[r][i] = 0ull;
            last[r] = 0.f;
        }
    }
    // stores entry i of fibre r at dst[i * stride]
    __device__ __forceinline__ void store(int r, float *dst, int stride) const {
#pragma unroll
        for (int i = 0; i < NP; i++) {
            float lo, hi;
            unpack2(p[r][i], lo, hi);
            dst[2 * i * stride] = lo;
            dst[(2 * i + 1) * stride] = hi;
        }
        if (ODD) dst[(PP - 1) * stride] = last[r];
    }
};
// acc[r][i] += sum_j M[j][i] v[r][j]: two outputs per instruction, the column's entries come in pairs from shared memory
template <int PP>
__device__ __forceinline__ void column_apply(const float (&v)[ColCfg<PP>::FPT][PP], const float *M, ColAcc<PP> &acc) {
    using C = ColCfg<PP>;
    using A = ColAcc<PP>;
#pragma unroll
    for (int j = 0; j < PP; j++) {
        f32x2 m[C::MSR / 2];
        const ulonglong2 *M4 = reinterpret_cast<const ulonglong2 *>(M + j * C::MSR);
#pragma unroll
        for (int q = 0; q < C::MSR / 4; q++) {
            const ulonglong2 w = M4[q];
            m[2 * q] = w.x;
            m[2 * q + 1] = w.y;
        }
        float m_last, unused;
        unpack2(m[A::NP < C::MSR / 2 ? A::NP : 0], m_last, unused);
#pragma unroll
        for (int r = 0; r < C::FPT; r++) {
            const f32x2 vv = pack2(v[r][j], v[r][j]);
#pragma unroll
            for (int i = 0; i < A::NP; i++) acc.p[r][i] = fma2(m[i], vv, acc.p[r][i]);
            if (A::ODD) acc.last[r] = fmaf(m_last, v[r][j], acc.last[r]);
        }
    }
}

template <int PP>
__global__ void __launch_bounds__(128) m2l_columns(const int *__restrict__ fptr, const uint32_t *__restrict__ okey, const int *__restrict__ oidx,
                                                  const float *__restrict__ T, const float *__restrict__ mom, float *loc) {
    using C = ColCfg<PP>;
    constexpr int NF = C::NF, P = C::P, FPT = C::FPT, NT = C::NT;
    extern __shared__ __align__(16) float sm[];
    const int bx = blockIdx.x, e0 = fptr[bx], e1 = fptr[bx + 1];
    if (e0 == e1) return;
    float *Tsm = sm;
    for (int q = threadIdx.x; q < 3 * NOFF2 * C::MS; q += 128) Tsm[q] = T[q];
    const int group = threadIdx.x / NT, t = threadIdx.x - group * NT, lane = threadIdx.x & 31;
    float *buf = sm + 3 * NOFF2 * C::MS + (size_t)group * P, *sum = buf + (size_t)C::NGRP * P;   // the group's transposes, its sums
    for (int q = t; q < P; q += NT) sum[q] = 0.f;
    ColAcc<PP> V, U;
    V.clear();
    U.clear();
    __syncthreads();
    // fibre f of the middle axis: m0 = f % PP, m2 = f / PP; of the first axis: m1 = f % PP, m2 = f / PP
    auto mid = [&](int f) { return f / PP * NF + f % PP; };
    auto close_columns = [&](uint32_t key, bool all) {
#pragma unroll
        for (int r = 0; r < FPT; r++) {
            const int f = t + r * NT;
            if (f < NF) V.store(r, buf + f, NF);
        }
        V.clear();
        group_sync<C::WPG>(group);
        float v[FPT][PP];
#pragma unroll
        for (int r = 0; r < FPT; r++) {
            const int f = min(t + r * NT, NF - 1);
#pragma unroll
            for (int j = 0; j < PP; j++) v[r][j] = buf[mid(f) + PP * j];
        }
        column_apply<PP>(v, Tsm + (NOFF2 + ((key >> 4) & 15u)) * C::MS, U);
        group_sync<C::WPG>(group);
        if (!all) return;
#pragma unroll
        for (int r = 0; r < FPT; r++) {
            const int f = t + r * NT;
            if (f < NF) U.store(r, buf + mid(f), PP);
        }
        U.clear();
        group_sync<C::WPG>(group);
#pragma unroll
        for (int r = 0; r < FPT; r++) {
            const int f = min(t + r * NT, NF - 1);
#pragma unroll
            for (int j = 0; j < PP; j++) v[r][j] = buf[PP * f + j];
        }
        column_apply<PP>(v, Tsm + ((key >> 8) & 15u) * C::MS, U);
        group_sync<C::WPG>(group);
#pragma unroll
        for (int r = 0; r < FPT; r++) {
            const int f = t + r * NT;
            if (f < NF) {   // the fibre's own entries of buf were read by this thread only
                U.store(r, buf + PP * f, 1);
#pragma unroll
                for (int i = 0; i < PP; i++) sum[PP * f + i] += buf[PP * f + i];
            }
        }
        U.clear();
        group_sync<C::WPG>(group);
    };
    const int len = e1 - e0;
    const int cb = e0 + (int)(((long long)len * group) / C::NGRP), ce = e0 + (int)(((long long)len * (group + 1)) / C::NGRP);
    uint32_t prev = 0xffffffffu;
    for (int c = cb; c < ce; c += 32) {
        const int cn = min(32, ce - c);
        uint32_t mykey = 0;
        int myidx = 0;
        if (lane < cn) { mykey = okey[c + lane]; myidx = oidx[c + lane]; }
        for (int q = 0; q < cn; q++) {
            const uint32_t key = __shfl_sync(0xffffffffu, mykey, q);
            const float *src = mom + (size_t)__shfl_sync(0xffffffffu, myidx, q) * P;
            float v[FPT][PP];
#pragma unroll
            for (int r = 0; r < FPT; r++) {
                const int f = min(t + r * NT, NF - 1);
#pragma unroll
                for (int j = 0; j < PP; j++) v[r][j] = __ldg(src + f + NF * j);
            }
            if (prev != 0xffffffffu && (key >> 4) != (prev >> 4)) close_columns(prev, (key >> 8) != (prev >> 8));
            column_apply<PP>(v, Tsm + (2 * NOFF2 + (key & 15u)) * C::MS, V);
            prev = key;
        }
    }
    if (prev != 0xffffffffu) close_columns(prev, true);
    __syncthreads();
    const float *sums = sm + 3 * NOFF2 * C::MS + (size_t)C::NGRP * P;
    for (int q = threadIdx.x; q < P; q += 128) {
        float v = 0.f;
#pragma unroll
        for (int g = 0; g < C::NGRP; g++) v += sums[(size_t)g * P + q];
        loc[(size_t)bx * P + q] = v;
    }
}

// true into words[0] when a weight is not finite or so large that moments could overflow where the pairs' sums do not; words[1]: the
// weights that are not zero
static __global__ void __launch_bounds__(256) weights_check(const float *__restrict__ b, int64_t n, int *words) {
    bool any = false;
    int nonzero = 0;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        any |= !(fabsf(b[i]) <= 1e30f);
        nonzero += b[i] != 0.f;
    }
    any = __any_sync(0xffffffffu, any);
    nonzero = __reduce_add_sync(0xffffffffu, nonzero);
    __shared__ int sums[8];
    if ((threadIdx.x & 31) == 0) {
        sums[threadIdx.x >> 5] = nonzero;
        if (any) atomicOr(words, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) nonzero += sums[w];
        if (nonzero) atomicAdd(words + 1, nonzero);
    }
}

// ---------------------------------------------------------------------------------------------
// Rule.  Estimated seconds of the lists of one level through nodes: the points' two passes, the pairs of boxes, and what the form pays
// once (launches, the order of the rows, the check of the weights with its read-back).  Measured: 1.8e-13 s per point and node for
// both passes up to eight nodes, 2.4e-13 beyond; 0.9e-13 to 1.2e-13 per pair of boxes and p^4 (p = 9, 4.15e6 pairs in rows of 127:
// 2.28 ms; p = 7, 3.7e6 in rows of 63: 1.08 ms).  Whole calls, lists summed directly / here: 4e6 uniform points, boxes of 122, 1.09
// lengthscales wide 18.2 / 5.4 ms; 2.9e7 points, l = 0.19 of sqrt12, 179 / 9.2 ms; 6e6 normal points 10.7 / 7.2 ms; 3.6e5 points 3.0 /
// 0.87 ms; a mixture of 1e7 points that ends at its last level 22.8 / 16.8 ms (7.7 where it ends above, far_cut); 6e4 points, 1.5e8 to 7e8
// pairs: even, so NODE_FIXED.
// ---------------------------------------------------------------------------------------------
constexpr double NODE_FIXED = 1e-4;
static double node_seconds(const f3m_plan *pl, int p, int64_t box_pairs) {
    const double P = (double)p * p * p;
    return NODE_FIXED + (double)pl->tx.n * P * (p <= 8 ? 1.8e-13 : 2.4e-13) + (double)box_pairs * P * p * 1.1e-13;
}

NodeChoice node_end(const f3m_plan *pl, int level) {
    NodeChoice c;
    const LevelLists &ll = pl->lists[level];
    if (pl->d != 3 || !pl->same || level < 1 || (pl->prm.flags & (F3M_FLAG_NEAR_MOMENTS | F3M_FLAG_NEAR_TENSOR_CORES))) return c;
    c.p = nodes_needed((double)pl->tx.levels[level].edge * sqrt(2.0 * (double)pl->lcs));
    if (!c.p) return c;
    c.small = ll.small.count > 0;
    c.keep = ll.keep.count > 0;
    c.seconds = node_seconds(pl, c.p, ll.small.count + ll.keep.count);
    return c;
}

NodeChoice node_choice(const f3m_plan *pl, int level, int R) {
    NodeChoice c;
    const LevelLists &ll = pl->lists[level];
    const int64_t ns = ll.small.count, nk = level == pl->levels ? ll.keep.count : 0;
    const double ds = ns ? direct_list_seconds(pl, level, ll.small, R) : 0.0, dk = nk ? direct_list_seconds(pl, level, ll.keep, R) : 0.0;
    c.seconds = ds + dk;
    if (pl->d != 3 || R != 1 || !pl->same || level < 1 || c.seconds <= NODE_FIXED ||
        (pl->prm.flags & (F3M_FLAG_NEAR_MOMENTS | F3M_FLAG_NEAR_TENSOR_CORES)))
        return c;
    const int p = nodes_needed((double)pl->tx.levels[level].edge * sqrt(2.0 * (double)pl->lcs));
    if (!p) return c;
    auto offer = [&](double t, bool s, bool k) {
        if (t < c.seconds) { c.seconds = t; c.small = s; c.keep = k; c.p = p; }
    };
    if (ns) offer(node_seconds(pl, p, ns) + dk, true, false);
    if (nk) offer(ds + node_seconds(pl, p, nk), false, true);
    if (ns && nk) offer(node_seconds(pl, p, ns + nk), true, true);
    return c;
}

template <int PP>
static void run_nodes(f3m_plan *pl, int level, const PairCSR *l1, const PairCSR *l2, const int *fptr, const uint32_t *okey, const int *oidx,
                      const float *T, const float *ctr, float *mom, float *loc, float *part, int chunk, const float *bs, float *out, cudaStream_t s) {
    Tree &t = pl->tx;
    Level &lv = t.levels[level];
    const int n = (int)t.n;
    const NodeTab2 nt = make_nodes2(PP);
    const float factor = 2.f / lv.edge;
    const int64_t slots = chunk ? part_slots(n, chunk) : 0;
    const int nsplit = target_parts(lv.max_count, n, lv.nb);
    if constexpr (PP <= PMAX_FAST)
        p2m_leaf3<PP, true><<<(unsigned)(lv.nb + slots), 128, 0, s>>>(t.pts.p, n, bs, 1, 0, lv.off.p, ctr, factor, nt, lv.nb, chunk, 0, n, mom, part,
                                                               nullptr, lv.nb);
    else {
        using G = Wide3<PP>;
        const size_t smem = sizeof(float) * std::max(G::ROWS * G::RS, G::S * PP * PP * PP);
        F3M_CUDA(cudaFuncSetAttribute(p2m_wide3<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        p2m_wide3<PP><<<(unsigned)(lv.nb + slots), 128, smem, s>>>(t.pts.p, n, bs, lv.off.p, ctr, factor, nt, lv.nb, chunk, mom, part);
    }
    F3M_LAUNCH_CHECK();
    if (chunk) {
        p2m_combine<<<(unsigned)(slots / 2), 128, 0, s>>>(lv.off.p, lv.nb, n, chunk, PP * PP * PP, 0, n, part, mom);
        F3M_LAUNCH_CHECK();
    }
    using C = ColCfg<PP>;
    F3M_CUDA(cudaFuncSetAttribute(m2l_columns<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem));
    m2l_columns<PP><<<lv.nb, 128, C::smem, s>>>(fptr, okey, oidx, T, mom, loc);
    F3M_LAUNCH_CHECK();
    if constexpr (PP <= PMAX_FAST)
        l2p_leaf3<PP, true><<<dim3(lv.nb, nsplit), 128, 0, s>>>(t.pts.p, n, lv.off.p, ctr, factor, nt, nsplit, 0, n, loc, 1, 0, out, nullptr);
    else {
        using G = Wide3<PP>;
        const size_t smem = sizeof(float) * (G::ROWS * G::RS + 2 * G::ROWS * (G::UNITS | 1));
        F3M_CUDA(cudaFuncSetAttribute(l2p_wide3<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        l2p_wide3<PP><<<dim3(lv.nb, nsplit), 128, smem, s>>>(t.pts.p, n, lv.off.p, ctr, factor, nt, nsplit, l1->ptr.p, l2 ? l2->ptr.p : nullptr,
                                                           loc, out);
    }
    F3M_LAUNCH_CHECK();
}

// The level's lists that the choice names, added to out (sorted order).  false: nothing was added and the lists have to be summed directly
// -- the memory for the moments is not to be had, a weight is not finite (its box's moments would carry it with either sign), or few
// weights are other than zero (above).
bool node_sums(f3m_plan *pl, int level, const NodeChoice &choice, const float *bs, float *out, cudaStream_t s) {
    Tree &t = pl->tx;
    Level &lv = t.levels[level];
    LevelLists &ll = pl->lists[level];
    const int p = choice.p, P = p * p * p, n = (int)t.n, nb = lv.nb;
    const PairCSR *l1 = choice.small ? &ll.small : &ll.keep, *l2 = choice.small && choice.keep ? &ll.keep : nullptr;
    const int64_t count = l1->count + (l2 ? l2->count : 0);
    if (count > 0x7fffffffLL) return false;
    if (pl->weights_ok < 0) {   // once per product
        int *words = pl->d_flags + FL_WEIGHTS;
        F3M_CUDA(cudaMemsetAsync(words, 0, 2 * sizeof(int), s));
        weights_check<<<(unsigned)std::min<int64_t>((t.n + 1023) / 1024, 8 * NUM_SMS_HINT), 256, 0, s>>>(bs, t.n, words);
        F3M_LAUNCH_CHECK();
        F3M_CUDA(cudaMemcpyAsync(pl->h_pinned + FL_WEIGHTS, words, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
        F3M_CUDA(cudaStreamSynchronize(s));
        pl->weights_ok = pl->h_pinned[FL_WEIGHTS] == 0 && (int64_t)pl->h_pinned[FL_WEIGHTS + 1] * SPARSE_WEIGHTS >= t.n;
    }
    if (!pl->weights_ok) return false;
    const int MS = p * ((p + 3) / 4 * 4), chunk = source_chunk(lv.max_count, t.n, false);
    if ((int)pl->node_rows.size() <= level) pl->node_rows.resize(level + 1);
    f3m_plan::NodeRows &rows = pl->node_rows[level];
    DevBuf<float> mom, loc, part, T, ctr;
    DevBuf<int> cell;
    const bool order = !rows.ready || rows.small != choice.small || rows.keep != choice.keep;
    try {
        if (order) {
            rows.ready = false;
            rows.ptr.alloc((size_t)nb + 1, s);
            rows.okey.alloc((size_t)count, s);
            rows.oidx.alloc((size_t)count, s);
        }
        cell.alloc((size_t)nb * 3, s);
        ctr.alloc((size_t)nb * 6, s);
        mom.alloc((size_t)nb * P, s);
        loc.alloc((size_t)nb * P, s);
        if (chunk) part.alloc((size_t)part_slots(n, chunk) * P, s);
        T.alloc((size_t)3 * NOFF2 * MS, s);
    } catch (const Fail &) {
        cudaGetLastError();
        rows = f3m_plan::NodeRows{};
        return false;
    }
    Geom2 geo{};
    for (int k = 0; k < 3; k++) geo.dqmin[k] = 1 - NOFF2 / 2;
    pl->last.begin(ST_DIRECT, s);
    decode_cells_kernel<<<(nb + 255) / 256, 256, 0, s>>>(nb, level, 3, lv.code.p, cell.p);
    F3M_LAUNCH_CHECK();
    fine_centres<<<(3 * nb + 255) / 256, 256, 0, s>>>(nb, Origin3{{t.origin[0], t.origin[1], t.origin[2]}}, (double)lv.edge, cell.p, ctr.p);
    F3M_LAUNCH_CHECK();
    if (order) {
        const ListSet ls{{l1->ptr.p, l2 ? l2->ptr.p : nullptr, nullptr}, {l1->idx.p, l2 ? l2->idx.p : nullptr, nullptr}, l2 ? 2 : 1};
        add_list_ptrs<<<(nb + 1 + 255) / 256, 256, 0, s>>>(nb + 1, ls, rows.ptr.p);
        F3M_LAUNCH_CHECK();
        far_order_kernel<4><<<(nb + 3) / 4, 128, 0, s>>>(nb, 3, ls, cell.p, cell.p, geo, rows.okey.p, rows.oidx.p, pl->d_flags, lv.off.p, 0, n);
        F3M_LAUNCH_CHECK();
        rows.ready = true;
        rows.small = choice.small;
        rows.keep = choice.keep;
    }
    column_table<<<16, 256, 0, s>>>(make_nodes2(p), (double)lv.edge, (double)pl->lcs, geo.dqmin[0], T.p);
    F3M_LAUNCH_CHECK();
    if (p <= PMAX_FAST) loc.zero();   // l2p_leaf3 visits boxes without pairs too
#define F3M_NODES(PP_) \
    case PP_: run_nodes<PP_>(pl, level, l1, l2, rows.ptr.p, rows.okey.p, rows.oidx.p, T.p, ctr.p, mom.p, loc.p, part.p, chunk, bs, out, s); break
    switch (p) {
        F3M_NODES(5);
        F3M_NODES(6);
        F3M_NODES(7);
        F3M_NODES(8);
        F3M_NODES(9);
        F3M_NODES(10);
        F3M_NODES(11);
        F3M_NODES(12);
        F3M_NODES(13);
    }
#undef F3M_NODES
    pl->last.end(s);
    pl->last.direct_launches++;
    pl->last.direct_variants[DV_NODES]++;
    pl->last.box_pairs += count;
    return true;
}

}  // namespace f3m
