// Far field, fast path: one pass over the points, box-to-box translations in between.
//
// The reference interpolates every level directly from and to the points: P2M and L2P touch all N
// points at every level, and the node-to-node step evaluates P^2 exponentials per box pair
// (far_field_compute_v2, F3M_src/n_tree.cu:489-593; kernels F3M_src/1_d_conv.cu:451-659, 741-817).
// Here, with p nodes per dimension and P = p^d:
//
//   P2M   only at the finest level (one CTA per box, no atomics);
//   M2M   moments of a box = sum over its children of (A_s0 x A_s1 x ..) child moments, where
//         A_s[i][j] = L_i(s/2 + t_j/2) is the parent's 1-D Lagrange basis at the child's nodes.  A
//         parent basis function restricted to a child is a polynomial of degree p-1 per dimension, so
//         interpolating it on the child's p nodes is exact: these are the moments the reference
//         computes from the points, up to rounding;
//   M2L   per far pair the P x P Gaussian block is the Kronecker product of d tabulated p x p
//         matrices that depend only on the integer box offset per dimension: d*p*P multiply-adds and
//         no exponential per pair;
//   L2L   the transpose of M2M, pushing local expansions down to the finest level;
//   L2P   only at the finest level.
//
// All three translations are "apply d small matrices along the d axes of a p^d array"; a warp does
// that for one box (pair) at a time with the array in its own shared-memory buffers.  Every kernel
// here is bound by shared-memory / L2 bandwidth and FP32 issue, not HBM: the moment arrays of the
// finest level (boxes * P floats) are read a few times from L2/HBM, the points once.
#include <math.h>
#include <algorithm>
#include <vector>
#include "common.cuh"
#include "nodes.cuh"
#include "packed.cuh"

namespace f3m {

// ---------------------------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------------------------
// T[k][o][i*p+j] = exp(-lcs (g_i - g_j - delta)^2), delta = (o + dqmin_k) edge + shift_k, g = node*edge/2
// (setup_skip_conv n_tree.cu:433-486 adds the centres to the scaled nodes; the +edge/2 of n_tree.cu:510 cancels)
// What the node-to-node steps of a product need of their levels: the tables, and the cells of the boxes of rows that have no order yet.
// One launch for all levels (blockIdx.y), which also lays out the matrices between a box and its children.
struct SetupLevel {
    float *T;              // null: kept from an earlier product
    double edge;
    Geom2 geo;
    const uint32_t *code[2];
    int *cell[2];          // null: not needed
    int nb[2], level;
};
struct ShiftTables { float a[2 * mat_stride(PMAX_FAST)], at[2 * mat_stride(PMAX_FAST)]; };
struct SetupArgs {
    SetupLevel lv[F3M_MAX_LEVELS];
    ShiftTables shift;
    float *shift_a, *shift_at;   // null: kept from an earlier product
};
__global__ void __launch_bounds__(256) setup_levels(NodeTab2 nt, int d, double lcs, const __grid_constant__ SetupArgs a) {
    const SetupLevel &lv = a.lv[blockIdx.y];
    const int p = nt.p, MS = mat_stride(p), first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    if (lv.T)
        for (int e = first; e < d * NOFF2 * MS; e += step) {
            const int q = e % MS, o = (e / MS) % NOFF2, k = e / (MS * NOFF2);
            float v = 0.f;
            if (q < p * p) {
                const int in = q / p, jn = q % p;
                const double delta = (double)(o + lv.geo.dqmin[k]) * lv.edge + lv.geo.shift[k];
                const double diff = ((double)nt.node[in] - (double)nt.node[jn]) * lv.edge * 0.5 - delta;
                v = (float)exp(-lcs * diff * diff);
            }
            lv.T[e] = v;
        }
#pragma unroll
    for (int t = 0; t < 2; t++)
        if (lv.cell[t])
            for (int b = first; b < lv.nb[t]; b += step) {
                const uint32_t c = lv.code[t][b];
                for (int k = 0; k < d; k++) {
                    int q = 0;
                    for (int jb = 0; jb < lv.level; jb++) q |= (int)((c >> (d * jb + k)) & 1u) << jb;
                    lv.cell[t][b * d + k] = q;
                }
            }
    if (a.shift_a && blockIdx.y == 0)
        for (int i = first; i < 2 * MS; i += step) {
            a.shift_a[i] = a.shift.a[i];
            a.shift_at[i] = a.shift.at[i];
        }
}

// A[s][i*p+j] = L_i(xi), xi = (s ? +0.5 : -0.5) + 0.5 t_j ; AT is its transpose.  Exact Lagrange products in double.
static void make_shift_tables(const NodeTab2 &nt, std::vector<float> &A, std::vector<float> &AT) {
    const int p = nt.p, MS = mat_stride(p);
    A.assign(2 * MS, 0.f);
    AT.assign(2 * MS, 0.f);
    for (int s = 0; s < 2; s++)
        for (int j = 0; j < p; j++) {
            double xi = (s ? 0.5 : -0.5) + 0.5 * (double)nt.node[j];
            for (int i = 0; i < p; i++) {
                double L = 1.0;
                for (int l = 0; l < p; l++)
                    if (l != i) L *= (xi - (double)nt.node[l]) / ((double)nt.node[i] - (double)nt.node[l]);
                A[s * MS + i * p + j] = (float)L;
                AT[s * MS + j * p + i] = (float)L;
            }
        }
}

// ---------------------------------------------------------------------------------------------
// warp-level "apply d matrices along the d axes"
// Array layout: index = m*RB + r, m = sum_k m_k p^k (dimension 0 fastest), r the column.
// Stage k transforms axis k: out[.., i, ..] = sum_j M_k[i][j] in[.., j, ..].  The last stage adds into acc.
// ---------------------------------------------------------------------------------------------
struct KronCfg {
    int d, RB, P, nf;        // nf = (P/p)*RB fibres per stage
    int st[MAXD];            // element stride of axis k: RB * p^k
    float inv_st[MAXD];
};

static KronCfg make_kron_cfg(int d, int p, int RB) {
    KronCfg c{};
    c.d = d; c.RB = RB;
    c.P = 1;
    for (int k = 0; k < d; k++) c.P *= p;
    c.nf = (c.P / p) * RB;
    int st = RB;
    for (int k = 0; k < MAXD; k++) {
        c.st[k] = st;
        c.inv_st[k] = 1.0f / (float)st;
        if (k < d) st *= p;
    }
    return c;
}

// A lane owns whole fibres (p consecutive entries along the axis being transformed): it loads the p x p
// matrix of the stage into registers once, then p inputs -> p outputs per fibre.  With ACC_REG the
// outputs of the last stage are accumulated in registers (possible when a stage has at most 64 fibres,
// i.e. two rounds per lane); otherwise in the warp's shared-memory accumulator.
// DD > 0: dimension known at compile time and one column (RB = 1): every stride is a constant, so the
// index arithmetic folds into immediate offsets.  DD = 0: dimension and column block taken from cfg.
template <int PP, bool ACC_REG, int DD>
__device__ __forceinline__ void warp_kron(const float *src0, float *bufA, float *bufB, float *acc_sm,
                                          float (&acc_reg)[2][PP], float &acc_left, const float *const (&mats)[MAXD],
                                          const KronCfg &cfg, int lane) {
    constexpr int MS = mat_stride(PP);
    const float *src = src0;
    float *dst = bufA;
    const int nf = DD ? cpow(PP, DD - 1) : cfg.nf;
    const int dd = DD ? DD : cfg.d;
#pragma unroll
    for (int k = 0; k < MAXD; k++) {
        if (k < dd) {
            const bool last = (k == dd - 1);
            const int st = DD ? cpow(PP, k) : cfg.st[k];
            const float inv = DD ? 1.0f / (float)cpow(PP, k) : cfg.inv_st[k];
            float M[MS];
            const float4 *M4 = reinterpret_cast<const float4 *>(mats[k]);
#pragma unroll
            for (int q = 0; q < MS / 4; q++) {
                float4 v = M4[q];
                M[4 * q] = v.x; M[4 * q + 1] = v.y; M[4 * q + 2] = v.z; M[4 * q + 3] = v.w;
            }
            auto fibre = [&](int f, float *areg) {
                const int hi = last ? 0 : (DD ? f / st : __float2int_rz(((float)f + 0.5f) * inv));
                const int base = hi * st * PP + (f - hi * st);
                float v[PP];
#pragma unroll
                for (int j = 0; j < PP; j++) v[j] = src[base + j * st];
#pragma unroll
                for (int i = 0; i < PP; i++) {
                    float o = 0.f;
#pragma unroll
                    for (int j = 0; j < PP; j++) o = fmaf(M[i * PP + j], v[j], o);
                    if (!last) dst[base + i * st] = o;
                    else if (ACC_REG) areg[i] += o;
                    else acc_sm[base + i * st] += o;
                }
            };
            if (ACC_REG) {   // at most two rounds, register accumulators indexed statically
                if (lane < nf) fibre(lane, acc_reg[0]);
                const int left = nf - 32;
                if (left > 0 && left * PP <= 32) {
                    // a short second round (e.g. 36 fibres): one OUTPUT per lane instead of one fibre per lane
                    if (lane < left * PP) {
                        const int lf = lane / PP, i = lane - lf * PP, f = 32 + lf;
                        const int hi = last ? 0 : (DD ? f / st : __float2int_rz(((float)f + 0.5f) * inv));
                        const int base = hi * st * PP + (f - hi * st);
                        const float *mrow = mats[k] + i * PP;
                        float o = 0.f;
#pragma unroll
                        for (int j = 0; j < PP; j++) o = fmaf(mrow[j], src[base + j * st], o);
                        if (!last) dst[base + i * st] = o;
                        else acc_left += o;
                    }
                } else if (lane + 32 < nf) fibre(lane + 32, acc_reg[1]);
            } else {
                for (int f = lane; f < nf; f += 32) fibre(f, acc_reg[0]);
            }
            __syncwarp();
            src = dst;
            dst = (dst == bufA) ? bufB : bufA;
        }
    }
}

// after the last pair: registers -> the warp's shared-memory accumulator (layout of the last stage: base = fibre)
template <int PP>
__device__ __forceinline__ void flush_acc(float (&acc_reg)[2][PP], float acc_left, float *acc_sm, const KronCfg &cfg,
                                          int lane) {
    const int st = cfg.st[cfg.d - 1];   // for one column this equals the number of fibres
    const int left = cfg.nf - 32;
    const bool short_round = left > 0 && left * PP <= 32;
#pragma unroll
    for (int rnd = 0; rnd < 2; rnd++) {
        const int f = lane + rnd * 32;
        if (f < cfg.nf && !(rnd == 1 && short_round))
#pragma unroll
            for (int i = 0; i < PP; i++) acc_sm[f + i * st] = acc_reg[rnd][i];
    }
    if (short_round && lane < left * PP) {
        const int lf = lane / PP, i = lane - lf * PP;
        acc_sm[32 + lf + i * st] = acc_left;
    }
}

// ---------------------------------------------------------------------------------------------
// M2L: one CTA per target box, its warps share the far row
// ---------------------------------------------------------------------------------------------
template <int PP, bool ACC_REG, int DD>
__global__ void __launch_bounds__(128, 5) m2l_fast(int nbx, int d, const int *__restrict__ fptr, const int *__restrict__ fidx,
                                               const int *__restrict__ cell_x, const int *__restrict__ cell_y,
                                               const int *__restrict__ off_x, int row_begin, int row_end,
                                               const float *__restrict__ T, Geom2 geo, KronCfg cfg,
                                               const float *__restrict__ mom, float *loc, int *err) {
    extern __shared__ __align__(16) float sm[];
    constexpr int MS = mat_stride(PP);
    const int bx = blockIdx.x;
    const int e0 = fptr[bx], e1 = fptr[bx + 1];
    if (off_x[bx + 1] <= row_begin || off_x[bx] >= row_end) return;   // box has no point in this rank's slice
    if (e0 == e1) {
        for (int q = threadIdx.x; q < cfg.P * cfg.RB; q += blockDim.x) loc[(size_t)bx * cfg.P * cfg.RB + q] = 0.f;
        return;
    }
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int PR = cfg.P * cfg.RB, ntab = d * NOFF2 * MS;
    float *Tsm = sm;
    float *wbuf = sm + ntab + (size_t)w * 3 * PR;
    float *bufA = wbuf, *bufB = wbuf + PR, *acc = wbuf + 2 * PR;
    for (int q = threadIdx.x; q < ntab; q += blockDim.x) Tsm[q] = T[q];
    for (int q = lane; q < PR; q += 32) acc[q] = 0.f;
    float acc_reg[2][PP], acc_left = 0.f;
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int i = 0; i < PP; i++) acc_reg[a][i] = 0.f;
    __syncthreads();
    int qx[MAXD];
#pragma unroll
    for (int k = 0; k < MAXD; k++) qx[k] = k < d ? cell_x[bx * d + k] : 0;
    for (int e = e0 + w; e < e1; e += nw) {
        const int by = fidx[e];
        const float *mats[MAXD];
        bool ok = true;
#pragma unroll
        for (int k = 0; k < MAXD; k++) {
            int o = 0;
            if (k < d) {
                o = cell_y[by * d + k] - qx[k] - geo.dqmin[k];
                if (o < 0 || o >= NOFF2) { ok = false; o = 0; }
            }
            mats[k] = Tsm + (k * NOFF2 + o) * MS;
        }
        if (!ok) { if (lane == 0) atomicExch(err, 2); continue; }
        warp_kron<PP, ACC_REG, DD>(mom + (size_t)by * PR, bufA, bufB, acc, acc_reg, acc_left, mats, cfg, lane);
    }
    if (ACC_REG) flush_acc<PP>(acc_reg, acc_left, acc, cfg, lane);
    __syncthreads();
    for (int q = threadIdx.x; q < PR; q += blockDim.x) {
        float s = 0.f;
        for (int ww = 0; ww < nw; ww++) s += sm[ntab + (size_t)ww * 3 * PR + 2 * PR + q];
        loc[(size_t)bx * PR + q] = s;
    }
}

// ---------------------------------------------------------------------------------------------
// M2L, nested form (d = 2, 3, one column).  T(pair) = T_{d-1}(o_{d-1}) x .. x T_0(o_0) and the sum over the
// far pairs of a target box can be taken axis by axis:
//     loc = sum_{o0} T0(o0) [ sum_{o1} T1(o1) [ sum_{o2} T2(o2) mom(o0,o1,o2) ] ]
// With the row ordered by (o0, o1, o2) only the last-axis transform is applied per pair; the axis-1 transform
// once per (o0,o1) group and the axis-0 transform once per o0 group: ~240 instead of 567 stage applications
// for the 189 far pairs of an interior box.  Any order is correct (a group is flushed whenever the higher
// offsets change), ordering only increases the sharing.
// ---------------------------------------------------------------------------------------------
// Accumulators of one lane for one buffer of the nested transform: the fibres lane and lane+32 of the
// axis that produced it, or (when only a few fibres are left after the first 32) one output of a fibre
// beyond 32 per lane.
template <int PP>
struct FibreAcc {
    float r0[PP], r1[PP], left;
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < PP; i++) r0[i] = r1[i] = 0.f;
        left = 0.f;
    }
};

template <int PP, int DD>
struct NestGeom {
    static constexpr int MS = mat_stride(PP);
    static constexpr int P = cpow(PP, DD);
    static constexpr int nf = cpow(PP, DD - 1);
    static constexpr int left = nf - 32;
    static constexpr bool short_round = left > 0 && left * PP <= 32;
    static constexpr bool second_round = left > 0 && !short_round;
    template <int K>
    static __device__ __forceinline__ int base(int f) {
        constexpr int st = cpow(PP, K);
        const int hi = f / st;
        return hi * st * PP + (f - hi * st);
    }
};

// inputs of one lane for one application along axis K
template <int PP>
struct FibreIn {
    float v0[PP], v1[PP];
};

template <int PP, int K, int DD, bool GLOBAL>
__device__ __forceinline__ void nest_load(const float *src, FibreIn<PP> &in, int lane) {
    using G = NestGeom<PP, DD>;
    constexpr int st = cpow(PP, K);
    if (lane < G::nf) {
        const int base = G::template base<K>(lane);
#pragma unroll
        for (int j = 0; j < PP; j++) in.v0[j] = GLOBAL ? __ldg(src + base + j * st) : src[base + j * st];
    }
    if (G::short_round) {
        if (lane < G::left * PP) {
            const int base = G::template base<K>(32 + lane / PP);
#pragma unroll
            for (int j = 0; j < PP; j++) in.v1[j] = GLOBAL ? __ldg(src + base + j * st) : src[base + j * st];
        }
    } else if (G::second_round) {
        if (lane + 32 < G::nf) {
            const int base = G::template base<K>(lane + 32);
#pragma unroll
            for (int j = 0; j < PP; j++) in.v1[j] = GLOBAL ? __ldg(src + base + j * st) : src[base + j * st];
        }
    }
}

// out += M_k applied along the axis to the loaded fibres
template <int PP, int DD>
__device__ __forceinline__ void nest_apply(const FibreIn<PP> &in, const float *Mk, FibreAcc<PP> &out, int lane) {
    using G = NestGeom<PP, DD>;
    float M[G::MS];
    const float4 *M4 = reinterpret_cast<const float4 *>(Mk);
#pragma unroll
    for (int q = 0; q < G::MS / 4; q++) {
        float4 v = M4[q];
        M[4 * q] = v.x; M[4 * q + 1] = v.y; M[4 * q + 2] = v.z; M[4 * q + 3] = v.w;
    }
    if (lane < G::nf) {
#pragma unroll
        for (int i = 0; i < PP; i++) {
            float o = 0.f;
#pragma unroll
            for (int j = 0; j < PP; j++) o = fmaf(M[i * PP + j], in.v0[j], o);
            out.r0[i] += o;
        }
    }
    if (G::short_round) {
        if (lane < G::left * PP) {
            const float *mrow = Mk + (lane % PP) * PP;
            float o = 0.f;
#pragma unroll
            for (int j = 0; j < PP; j++) o = fmaf(mrow[j], in.v1[j], o);
            out.left += o;
        }
    } else if (G::second_round) {
        if (lane + 32 < G::nf) {
#pragma unroll
            for (int i = 0; i < PP; i++) {
                float o = 0.f;
#pragma unroll
                for (int j = 0; j < PP; j++) o = fmaf(M[i * PP + j], in.v1[j], o);
                out.r1[i] += o;
            }
        }
    }
}

// registers -> shared memory in the layout of axis K (the axis that produced them), then clear
template <int PP, int K, int DD>
__device__ __forceinline__ void nest_spill(FibreAcc<PP> &a, float *dst, int lane) {
    using G = NestGeom<PP, DD>;
    constexpr int st = cpow(PP, K);
    if (lane < G::nf) {
        const int base = G::template base<K>(lane);
#pragma unroll
        for (int i = 0; i < PP; i++) dst[base + i * st] = a.r0[i];
    }
    if (G::short_round) {
        if (lane < G::left * PP) dst[G::template base<K>(32 + lane / PP) + (lane % PP) * st] = a.left;
    } else if (G::second_round) {
        if (lane + 32 < G::nf) {
            const int base = G::template base<K>(lane + 32);
#pragma unroll
            for (int i = 0; i < PP; i++) dst[base + i * st] = a.r1[i];
        }
    }
    a.clear();
}

// The per-pair transform runs along the LAST axis (its fibres are strided by the number of fibres, so a
// warp reads 32 consecutive floats per load); the packed key of a pair holds the offset of that axis in
// its lowest 4 bits, the next axis above it, axis 0 on top.
template <int PP, int DD>
__global__ void __launch_bounds__(128, PP <= 6 ? 4 : 2) m2l_nested(int nbx, const int *__restrict__ fptr,
                                                                   const uint32_t *__restrict__ okey, const int *__restrict__ oidx,
                                                                   const int *__restrict__ off_x, int row_begin, int row_end,
                                                                   const float *__restrict__ T, const float *__restrict__ mom,
                                                                   float *loc) {
    extern __shared__ __align__(16) float sm[];
    using G = NestGeom<PP, DD>;
    constexpr int MS = G::MS, P = G::P;
    constexpr int KA = DD - 1;               // axis applied per pair
    const int bx = blockIdx.x;
    const int e0 = fptr[bx], e1 = fptr[bx + 1];
    if (off_x[bx + 1] <= row_begin || off_x[bx] >= row_end) return;
    if (e0 == e1) {
        for (int q = threadIdx.x; q < P; q += blockDim.x) loc[(size_t)bx * P + q] = 0.f;
        return;
    }
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int ntab = DD * NOFF2 * MS;
    float *Tsm = sm;
    float *buf = sm + ntab + (size_t)w * P;  // one transpose buffer per warp
    for (int q = threadIdx.x; q < ntab; q += blockDim.x) Tsm[q] = T[q];
    FibreAcc<PP> V, U, A;
    V.clear(); U.clear(); A.clear();
    __syncthreads();
    const int len = e1 - e0;
    const int cb = e0 + (int)(((long long)len * w) / nw), ce = e0 + (int)(((long long)len * (w + 1)) / nw);
    // matrix of axis k for the offset stored in nibble (DD-1-k) of the key
    auto mat = [&](int k, uint32_t key) { return Tsm + (k * NOFF2 + ((key >> (4 * (DD - 1 - k))) & 15u)) * MS; };
    auto close_groups = [&](uint32_t key, bool all) {
        FibreIn<PP> in;
        nest_spill<PP, KA, DD>(V, buf, lane);
        __syncwarp();
        if (DD == 3) {
            nest_load<PP, 1, DD, false>(buf, in, lane);
            nest_apply<PP, DD>(in, mat(1, key), U, lane);
            __syncwarp();
            if (all) {
                nest_spill<PP, 1, DD>(U, buf, lane);
                __syncwarp();
                nest_load<PP, 0, DD, false>(buf, in, lane);
                nest_apply<PP, DD>(in, mat(0, key), A, lane);
                __syncwarp();
            }
        } else {
            nest_load<PP, 0, DD, false>(buf, in, lane);
            nest_apply<PP, DD>(in, mat(0, key), A, lane);
            __syncwarp();
        }
    };
    uint32_t prev = 0xffffffffu;
    for (int c = cb; c < ce; c += 32) {
        const int cn = min(32, ce - c);
        uint32_t mykey = 0;
        int myidx = 0;
        if (lane < cn) { mykey = okey[c + lane]; myidx = oidx[c + lane]; }
        FibreIn<PP> cur;
        nest_load<PP, KA, DD, true>(mom + (size_t)__shfl_sync(0xffffffffu, myidx, 0) * P, cur, lane);
        for (int t = 0; t < cn; t++) {
            const uint32_t key = __shfl_sync(0xffffffffu, mykey, t);
            FibreIn<PP> nxt;
            const int tn = min(t + 1, cn - 1);   // the last one re-reads itself: no branch around the loads
            nest_load<PP, KA, DD, true>(mom + (size_t)__shfl_sync(0xffffffffu, myidx, tn) * P, nxt, lane);
            if (prev != 0xffffffffu && (key >> 4) != (prev >> 4)) close_groups(prev, DD == 3 ? (key >> 8) != (prev >> 8) : true);
            nest_apply<PP, DD>(cur, mat(KA, key), V, lane);
            prev = key;
            cur = nxt;
        }
    }
    if (prev != 0xffffffffu) close_groups(prev, true);
    // layout of axis 0: the lane's fibre is PP consecutive entries
    float *accw = sm + ntab + (size_t)w * P;
    nest_spill<PP, 0, DD>(A, accw, lane);
    __syncthreads();
    for (int q = threadIdx.x; q < P; q += blockDim.x) {
        float s = 0.f;
        for (int ww = 0; ww < nw; ww++) s += sm[ntab + (size_t)ww * P + q];
        loc[(size_t)bx * P + q] = s;
    }
}

// ---------------------------------------------------------------------------------------------
// M2L, nested form for several columns and for d = 4, 5: one CTA per target box, every thread owns FPT
// fibres of each axis and keeps the partial sums of ALL nesting levels in registers.  A far pair costs one
// coalesced read of the source box's moments and the last-axis transform, with no shared-memory traffic;
// shared memory is only used to re-lay the sums out for the next axis when a group of offsets closes.
// ---------------------------------------------------------------------------------------------
template <int PP, int DD, int RBB>
struct RowCfg {
    static constexpr int MS = mat_stride(PP);
    static constexpr int P = cpow(PP, DD), PR = P * RBB, NF = PR / PP;
    static constexpr int MAX_ACC = 64;   // accumulator registers of a thread over all levels
    static constexpr int pick_threads() {
        int best = 0;
        long best_u = -1;
        for (int nt = 32; nt <= 256; nt += 32) {
            const int fpt = (NF + nt - 1) / nt;
            if (DD * fpt * PP > MAX_ACC) continue;
            const long u = (long)NF * 1000000 / ((long)fpt * nt);   // share of fibre slots that hold a fibre
            if (u >= best_u) { best_u = u; best = nt; }
        }
        return best;
    }
    static constexpr int NT = pick_threads();
    static constexpr int FPT = NT ? (NF + NT - 1) / NT : 1;
    static constexpr int DEPTH = FPT * PP * 4 <= 40 ? 4 : 2;   // source boxes in flight per CTA (divides 32)
    static constexpr size_t smem = ((size_t)DD * NOFF2 * MS + (size_t)PR) * sizeof(float);
    static constexpr bool ok = NT > 0 && smem <= 160 * 1024;
    template <int K>
    static __device__ __forceinline__ int base(int f) {
        constexpr int st = RBB * cpow(PP, K);
        const int hi = f / st;
        return hi * st * PP + (f - hi * st);
    }
};

template <int PP>
__device__ __forceinline__ void load_matrix(const float *Mk, float (&M)[mat_stride(PP)]) {
    const float4 *M4 = reinterpret_cast<const float4 *>(Mk);
#pragma unroll
    for (int q = 0; q < mat_stride(PP) / 4; q++) {
        float4 v = M4[q];
        M[4 * q] = v.x; M[4 * q + 1] = v.y; M[4 * q + 2] = v.z; M[4 * q + 3] = v.w;
    }
}

// Closes nesting level K: the sums over the last offsets (axes K..DD-1 already applied) go through shared memory
// into the layout of axis K-1, that axis' matrix for the group's offset is applied, and the result is added to
// level K-1; level K-1 closes too when the offsets above it change.
template <int PP, int DD, int RBB, int K>
__device__ __forceinline__ void rows_close(float (&acc)[DD][RowCfg<PP, DD, RBB>::FPT][PP], float *buf, const float *Tsm,
                                           uint32_t prev, uint32_t key, bool final, int tid) {
    using C = RowCfg<PP, DD, RBB>;
    if constexpr (K >= 1) {
        constexpr int stK = RBB * cpow(PP, K), stL = RBB * cpow(PP, K - 1);
#pragma unroll
        for (int r = 0; r < C::FPT; r++) {
            const int f = tid + r * C::NT;
            if (f < C::NF) {
                const int base = C::template base<K>(f);
#pragma unroll
                for (int i = 0; i < PP; i++) { buf[base + i * stK] = acc[K][r][i]; acc[K][r][i] = 0.f; }
            }
        }
        __syncthreads();
        float M[C::MS];
        load_matrix<PP>(Tsm + ((K - 1) * NOFF2 + ((prev >> (4 * (DD - K))) & 15u)) * C::MS, M);
#pragma unroll
        for (int r = 0; r < C::FPT; r++) {
            const int f = tid + r * C::NT;
            if (f < C::NF) {
                const int base = C::template base<K - 1>(f);
                float v[PP];
#pragma unroll
                for (int j = 0; j < PP; j++) v[j] = buf[base + j * stL];
#pragma unroll
                for (int i = 0; i < PP; i++) {
                    float o = 0.f;
#pragma unroll
                    for (int j = 0; j < PP; j++) o = fmaf(M[i * PP + j], v[j], o);
                    acc[K - 1][r][i] += o;
                }
            }
        }
        __syncthreads();
        if constexpr (K >= 2) {
            constexpr int sh = 4 * (DD - K + 1);   // nibbles of the axes K-1..DD-1
            if (final || (key >> sh) != (prev >> sh)) rows_close<PP, DD, RBB, K - 1>(acc, buf, Tsm, prev, key, final, tid);
        }
    }
}

template <int PP, int DD, int RBB>
__global__ void __launch_bounds__(RowCfg<PP, DD, RBB>::NT ? RowCfg<PP, DD, RBB>::NT : 32)
m2l_rows(int nbx, const int *__restrict__ fptr, const uint32_t *__restrict__ okey, const int *__restrict__ oidx,
         const int *__restrict__ off_x, int row_begin, int row_end, const float *__restrict__ T,
         const float *__restrict__ mom, float *loc) {
    using C = RowCfg<PP, DD, RBB>;
    constexpr int MS = C::MS, PR = C::PR, NF = C::NF, NT = C::NT ? C::NT : 32, FPT = C::FPT;
    constexpr int KA = DD - 1;   // axis applied per pair: its fibres are strided by NF, fibre f starts at element f
    extern __shared__ __align__(16) float sm[];
    const int bx = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int e0 = fptr[bx], e1 = fptr[bx + 1];
    if (off_x[bx + 1] <= row_begin || off_x[bx] >= row_end) return;
    if (e0 == e1) {
        for (int q = tid; q < PR; q += NT) loc[(size_t)bx * PR + q] = 0.f;
        return;
    }
    constexpr int ntab = DD * NOFF2 * MS;
    float *Tsm = sm, *buf = sm + ntab;
    for (int q = tid; q < ntab; q += NT) Tsm[q] = T[q];
    float acc[DD][FPT][PP];
#pragma unroll
    for (int k = 0; k < DD; k++)
#pragma unroll
        for (int r = 0; r < FPT; r++)
#pragma unroll
            for (int i = 0; i < PP; i++) acc[k][r][i] = 0.f;
    __syncthreads();
    auto fetch = [&](int by, float (&v)[FPT][PP]) {
        const float *src = mom + (size_t)by * PR;
#pragma unroll
        for (int r = 0; r < FPT; r++) {
            const int f = tid + r * NT;
#pragma unroll
            for (int j = 0; j < PP; j++) v[r][j] = f < NF ? __ldg(src + f + j * NF) : 0.f;
        }
    };
    // DEPTH source boxes are on their way while one is consumed; the row's keys and boxes are read 32 at a time, one
    // per lane, the next 32 a chunk ahead (entries past the end of the row repeat its last pair and are never consumed)
    constexpr int DEPTH = C::DEPTH;
    float pre[DEPTH][FPT][PP];
    uint32_t prev = 0xffffffffu;
    int nxtidx = oidx[min(e0 + lane, e1 - 1)];
    uint32_t nxtkey = okey[min(e0 + lane, e1 - 1)];
#pragma unroll
    for (int u = 0; u < DEPTH; u++) fetch(__shfl_sync(0xffffffffu, nxtidx, u), pre[u]);
    for (int c = e0; c < e1; c += 32) {
        const int cn = min(32, e1 - c);
        const uint32_t mykey = nxtkey;
        const int myidx = nxtidx;
        nxtidx = oidx[min(c + 32 + lane, e1 - 1)];
        nxtkey = okey[min(c + 32 + lane, e1 - 1)];
        for (int t0 = 0; t0 < cn; t0 += DEPTH) {
#pragma unroll
            for (int u = 0; u < DEPTH; u++) {
                const int t = t0 + u;
                if (t < cn) {
                    const uint32_t key = __shfl_sync(0xffffffffu, mykey, t);
                    if (prev != 0xffffffffu && (key >> 4) != (prev >> 4))
                        rows_close<PP, DD, RBB, KA>(acc, buf, Tsm, prev, key, false, tid);
                    float M[MS];
                    load_matrix<PP>(Tsm + (KA * NOFF2 + (key & 15u)) * MS, M);
#pragma unroll
                    for (int r = 0; r < FPT; r++)
#pragma unroll
                        for (int i = 0; i < PP; i++) {
                            float o = 0.f;
#pragma unroll
                            for (int j = 0; j < PP; j++) o = fmaf(M[i * PP + j], pre[u][r][j], o);
                            acc[KA][r][i] += o;
                        }
                    prev = key;
                    const int ahead = t + DEPTH;
                    const int a0 = __shfl_sync(0xffffffffu, myidx, ahead & 31), a1 = __shfl_sync(0xffffffffu, nxtidx, ahead & 31);
                    fetch(ahead < 32 ? a0 : a1, pre[u]);
                }
            }
        }
    }
    rows_close<PP, DD, RBB, KA>(acc, buf, Tsm, prev, prev, true, tid);
    // level 0 holds the box's local expansion in the layout of axis 0
    float *dst = loc + (size_t)bx * PR;
#pragma unroll
    for (int r = 0; r < FPT; r++) {
        const int f = tid + r * NT;
        if (f < NF) {
            const int base = C::template base<0>(f);
#pragma unroll
            for (int i = 0; i < PP; i++) dst[base + i * RBB] = acc[0][r][i];
        }
    }
}

// Host side of m2l_rows: the kernel exists for the (nodes, dimension, columns) whose accumulators fit the registers.
template <int PP, int DD, int RBB>
static bool m2l_rows_launch_one(bool probe, int nbx, const int *fptr, const uint32_t *okey, const int *oidx, const int *offx, int rb,
                                int re, const float *T, const float *mom, float *loc, cudaStream_t s) {
    using C = RowCfg<PP, DD, RBB>;
    if constexpr (C::ok) {
        if (probe) return true;
        F3M_CUDA(cudaFuncSetAttribute(m2l_rows<PP, DD, RBB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem));
        m2l_rows<PP, DD, RBB><<<nbx, C::NT, C::smem, s>>>(nbx, fptr, okey, oidx, offx, rb, re, T, mom, loc);
        return true;
    } else
        return false;
}

template <int PP, int RBB>
static bool m2l_rows_dispatch(bool probe, int d, int nbx, const int *fptr, const uint32_t *okey, const int *oidx, const int *offx,
                              int rb, int re, const float *T, const float *mom, float *loc, cudaStream_t s) {
    switch (d) {
    case 2: return m2l_rows_launch_one<PP, 2, RBB>(probe, nbx, fptr, okey, oidx, offx, rb, re, T, mom, loc, s);
    case 3: return m2l_rows_launch_one<PP, 3, RBB>(probe, nbx, fptr, okey, oidx, offx, rb, re, T, mom, loc, s);
    case 4: return m2l_rows_launch_one<PP, 4, RBB>(probe, nbx, fptr, okey, oidx, offx, rb, re, T, mom, loc, s);
    case 5: return m2l_rows_launch_one<PP, 5, RBB>(probe, nbx, fptr, okey, oidx, offx, rb, re, T, mom, loc, s);
    default: return false;
    }
}

template <int PP, int RBB>
static bool rows_form_available(int d) {
    return m2l_rows_dispatch<PP, RBB>(true, d, 0, nullptr, nullptr, nullptr, nullptr, 0, 0, nullptr, nullptr, nullptr, nullptr);
}

template <int PP, int RBB>
static void launch_m2l_rows(int d, int nbx, const int *fptr, const uint32_t *okey, const int *oidx, const int *offx, int rb, int re,
                            const float *T, const float *mom, float *loc, cudaStream_t s) {
    m2l_rows_dispatch<PP, RBB>(false, d, nbx, fptr, okey, oidx, offx, rb, re, T, mom, loc, s);
}

// is there a row form for p nodes per dimension and 8 columns?
static bool rows_form_for(int p, int d) {
    switch (p) {
        case 2: return rows_form_available<2, 8>(d);
        case 3: return rows_form_available<3, 8>(d);
        case 4: return rows_form_available<4, 8>(d);
        case 5: return rows_form_available<5, 8>(d);
        case 6: return rows_form_available<6, 8>(d);
        case 7: return rows_form_available<7, 8>(d);
        default: return rows_form_available<8, 8>(d);
    }
}

// M2M: one CTA per parent box, warps share the children
template <int PP>
__global__ void __launch_bounds__(128) m2m_fast(int nbp, int d, const int *__restrict__ child_start,
                                               const uint32_t *__restrict__ code_child, const float *__restrict__ A,
                                               KronCfg cfg, const float *__restrict__ mom_child, float *mom_parent) {
    extern __shared__ __align__(16) float sm[];
    constexpr int MS = mat_stride(PP);
    const int pb = blockIdx.x;
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int PR = cfg.P * cfg.RB, ntab = 2 * MS;
    float *Asm = sm;
    float *wbuf = sm + ntab + (size_t)w * 3 * PR;
    float *bufA = wbuf, *bufB = wbuf + PR, *acc = wbuf + 2 * PR;
    for (int q = threadIdx.x; q < ntab; q += blockDim.x) Asm[q] = A[q];
    for (int q = lane; q < PR; q += 32) acc[q] = 0.f;
    float acc_reg[2][PP], acc_left = 0.f;
    __syncthreads();
    const int c0 = child_start[pb], c1 = child_start[pb + 1];
    for (int c = c0 + w; c < c1; c += nw) {
        const uint32_t code = code_child[c];
        const float *mats[MAXD];
#pragma unroll
        for (int k = 0; k < MAXD; k++) mats[k] = Asm + ((code >> k) & 1u) * MS;
        warp_kron<PP, false, 0>(mom_child + (size_t)c * PR, bufA, bufB, acc, acc_reg, acc_left, mats, cfg, lane);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < PR; q += blockDim.x) {
        float s = 0.f;
        for (int ww = 0; ww < nw; ww++) s += sm[ntab + (size_t)ww * 3 * PR + 2 * PR + q];
        mom_parent[(size_t)pb * PR + q] = s;
    }
}

// L2L: one warp per child box
template <int PP>
__global__ void __launch_bounds__(128) l2l_fast(int nbc, int d, const int *__restrict__ parent,
                                               const uint32_t *__restrict__ code_child, const int *__restrict__ off_c,
                                               int row_begin, int row_end, const float *__restrict__ AT, KronCfg cfg,
                                               const float *__restrict__ loc_parent, float *loc_child) {
    extern __shared__ __align__(16) float sm[];
    constexpr int MS = mat_stride(PP);
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int PR = cfg.P * cfg.RB, ntab = 2 * MS;
    float *Asm = sm;
    float *wbuf = sm + ntab + (size_t)w * 3 * PR;
    float *bufA = wbuf, *bufB = wbuf + PR, *acc = wbuf + 2 * PR;
    for (int q = threadIdx.x; q < ntab; q += blockDim.x) Asm[q] = AT[q];
    __syncthreads();
    const int c = blockIdx.x * nw + w;
    if (c >= nbc) return;
    if (off_c[c + 1] <= row_begin || off_c[c] >= row_end) return;
    for (int q = lane; q < PR; q += 32) acc[q] = 0.f;
    __syncwarp();
    const uint32_t code = code_child[c];
    const float *mats[MAXD];
#pragma unroll
    for (int k = 0; k < MAXD; k++) mats[k] = Asm + ((code >> k) & 1u) * MS;
    float acc_reg[2][PP], acc_left = 0.f;
    warp_kron<PP, false, 0>(loc_parent + (size_t)parent[c] * PR, bufA, bufB, acc, acc_reg, acc_left, mats, cfg, lane);
    for (int q = lane; q < PR; q += 32) loc_child[(size_t)c * PR + q] += acc[q];
}

// ---------------------------------------------------------------------------------------------
// P2M / L2P at the finest level: one CTA per (box, split)
// ---------------------------------------------------------------------------------------------
// P2M.  A thread owns one combination (m_1 .. m_{d-1}) of the slower node indices and all p values of
// the fastest one: per point it forms w = b * prod_{k>=1} L_k[m_k] once and adds w * L_0[i] to p
// accumulators, so a (point, node) pair costs about one shared-memory read and one multiply-add.
// Threads beyond the number of combinations form further groups that take every G-th point.
template <int PP, int RB>
__global__ void __launch_bounds__(256) p2m_leaf(const float *__restrict__ pts, int n, int d, const float *__restrict__ bs, int R,
                                               int r0, const int *__restrict__ off, const float *__restrict__ ctr,
                                               float factor, NodeTab2 nt, int P, int nb, int chunk, int src_begin, int src_end,
                                               float *mom, float *part) {
    extern __shared__ __align__(16) float sm[];
    constexpr int TP = 128, NTH = 256, LS = TP + 1;
    float *Ls = sm;                                   // [d*PP][TP+1]
    float *bsm = Ls + (size_t)d * PP * LS;            // [TP][RB]
    float *accsm = bsm + (size_t)TP * RB;             // [P][RB]
    const LeafWork lw = leaf_work(off, nb, n, nullptr, nb, chunk, src_begin, src_end);
    const int box = lw.box, s0 = lw.s0, s1 = lw.s1;
    if (s0 >= s1) return;
    const int PR = P * RB, C = P / PP;
    // the PP x RB block of one combination starts an odd number of floats after the previous one: the lanes of a
    // warp (consecutive combinations) then add to different banks
    constexpr int CS = (PP * RB) | 1;
    for (int q = threadIdx.x; q < C * CS; q += NTH) accsm[q] = 0.f;
    float c[MAXD];
    for (int k = 0; k < d; k++) c[k] = ctr[box * d + k];
    const int G = C >= NTH ? 1 : NTH / C;             // point groups
    const int g = C >= NTH ? 0 : threadIdx.x / C;
    float acc[PP][RB];
#pragma unroll
    for (int i = 0; i < PP; i++)
#pragma unroll
        for (int r = 0; r < RB; r++) acc[i][r] = 0.f;
    int chunks = 0;
    for (int base = s0; base < s1; base += TP) {
        const int cnt = min(TP, s1 - base);
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            const int i = base + threadIdx.x;
            for (int k = 0; k < d; k++) {
                float L[PP];
                lagrange_pp<PP>(factor * (pts[(size_t)k * n + i] - c[k]), nt, L);
#pragma unroll
                for (int q = 0; q < PP; q++) Ls[(k * PP + q) * LS + threadIdx.x] = L[q];
            }
#pragma unroll
            for (int r = 0; r < RB; r++) bsm[threadIdx.x * RB + r] = (r0 + r < R) ? bs[(size_t)i * R + r0 + r] : 0.f;
        }
        __syncthreads();
        // A thread of a single combination keeps its sums over G chunks (128 terms), then adds them to the shared ones: added after every
        // chunk, three terms at a time, the atomics of 2-D boxes took most of the kernel (6e4 sources, 36 nodes, three columns: 48.9 -> 29.5 us).
        const bool flush = C > NTH || ++chunks == G || base + TP >= s1;
        if (g < G) {
            for (int cc = (C >= NTH ? (int)threadIdx.x : (int)threadIdx.x - g * C); cc < C; cc += NTH) {
                const float *lp[MAXD];
                int rem = cc;
#pragma unroll
                for (int k = 1; k < MAXD; k++) {
                    lp[k] = Ls;
                    if (k < d) { lp[k] = Ls + (size_t)(k * PP + rem % PP) * LS; rem /= PP; }
                }
                for (int j = g; j < cnt; j += G) {
                    float w = 1.f;
#pragma unroll
                    for (int k = 1; k < MAXD; k++)
                        if (k < d) w *= lp[k][j];
                    float wb[RB];
#pragma unroll
                    for (int r = 0; r < RB; r++) wb[r] = w * bsm[j * RB + r];
#pragma unroll
                    for (int i = 0; i < PP; i++) {
                        const float l0 = Ls[i * LS + j];
#pragma unroll
                        for (int r = 0; r < RB; r++) acc[i][r] = fmaf(l0, wb[r], acc[i][r]);
                    }
                }
                if (!flush) continue;
#pragma unroll
                for (int i = 0; i < PP; i++)
#pragma unroll
                    for (int r = 0; r < RB; r++) {
                        atomicAdd(&accsm[cc * CS + i * RB + r], acc[i][r]);
                        acc[i][r] = 0.f;
                    }
            }
        }
        if (flush) chunks = 0;
    }
    __syncthreads();
    float *dst = lw.slot < 0 ? mom + (size_t)box * PR : part + lw.slot * PR;
    constexpr int BLK = PP * RB;
    for (int q = threadIdx.x; q < PR; q += NTH) dst[q] = accsm[q + (q / BLK) * (CS - BLK)];
}

template <int PP, int RB>
__global__ void __launch_bounds__(128) l2p_leaf(const float *__restrict__ pts, int n, int d, const int *__restrict__ off,
                                               const float *__restrict__ ctr, float factor, NodeTab2 nt, int P, int nsplit,
                                               int row_begin, int row_end, const float *__restrict__ loc, int R, int r0,
                                               float *out) {
    extern __shared__ __align__(16) float sm[];
    constexpr int TP = 128;
    const int PR = P * RB;
    float *locsm = sm;                 // [P][RB]
    float *Ls = sm + PR;               // [(d-1)*PP][TP]
    const int box = blockIdx.x;
    const int a = off[box], b = off[box + 1];
    if (a < row_begin || a >= row_end) return;    // finest-level boxes belong to the slice their first point is in
    const int len = b - a;
    const int s0 = a + (int)(((long long)len * blockIdx.y) / nsplit), s1 = a + (int)(((long long)len * (blockIdx.y + 1)) / nsplit);
    if (s0 >= s1) return;
    for (int q = threadIdx.x; q < PR; q += TP) locsm[q] = loc[(size_t)box * PR + q];
    __syncthreads();
    float c[MAXD];
    for (int k = 0; k < d; k++) c[k] = ctr[box * d + k];
    const int outer = P / PP;
    for (int i = s0 + threadIdx.x; i < s1; i += TP) {
        float l0[PP];
        lagrange_pp<PP>(factor * (pts[i] - c[0]), nt, l0);
        for (int k = 1; k < d; k++) {
            float L[PP];
            lagrange_pp<PP>(factor * (pts[(size_t)k * n + i] - c[k]), nt, L);
#pragma unroll
            for (int q = 0; q < PP; q++) Ls[((k - 1) * PP + q) * TP + threadIdx.x] = L[q];
        }
        float acc[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) acc[r] = 0.f;
        for (int o = 0; o < outer; o++) {
            float wgt = 1.f;
            int rem = o;
            for (int k = 1; k < d; k++) {
                wgt *= Ls[((k - 1) * PP + rem % PP) * TP + threadIdx.x];
                rem /= PP;
            }
            float sacc[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) sacc[r] = 0.f;
            const float *lp = locsm + (size_t)o * PP * RB;
#pragma unroll
            for (int i0 = 0; i0 < PP; i0++)
#pragma unroll
                for (int r = 0; r < RB; r++) sacc[r] = fmaf(l0[i0], lp[i0 * RB + r], sacc[r]);
#pragma unroll
            for (int r = 0; r < RB; r++) acc[r] = fmaf(wgt, sacc[r], acc[r]);
        }
#pragma unroll
        for (int r = 0; r < RB; r++)
            if (r0 + r < R) out[(size_t)i * R + r0 + r] += acc[r];
    }
}

// Small finest-level boxes (clustered data leaves millions of boxes with a handful of points): one warp per box, so
// that a box costs a few hundred instructions instead of a CTA's launch, barriers and reductions.
constexpr int LEAF_SMALL = 32;
constexpr int SMALL_RS = 28;   // floats between their rows [L0 (8) | L1 (8) | L2 (8) | pad (4)]

__global__ void __launch_bounds__(256) split_leaf_boxes(int nb, const int *__restrict__ off, int *small_list, int *big_list, int *counts) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int len = off[b + 1] - off[b];
    if (len <= LEAF_SMALL) small_list[atomicAdd(counts, 1)] = b;
    else big_list[atomicAdd(counts + 1, 1)] = b;
}

// P2M: lanes = nodes (ceil(P / 32) per lane), points in turn; the points' Lagrange rows go through shared memory
template <int PP>
__global__ void __launch_bounds__(128) p2m_small3(const float *__restrict__ pts, int n, const float *__restrict__ bs, int R, int r0,
                                                 const int *__restrict__ off, const float *__restrict__ ctr, float factor,
                                                 NodeTab2 nt, int src_begin, int src_end, float *mom,
                                                 const int *__restrict__ box_list, int nlist) {
    constexpr int P = PP * PP * PP, NPL = (P + 31) / 32;
    __shared__ __align__(16) float rows_s[4][LEAF_SMALL * SMALL_RS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int li = blockIdx.x * 4 + warp;
    if (li >= nlist) return;
    const int box = box_list[li];
    const int a = off[box], len = off[box + 1] - a;
    if (a < src_begin || a >= src_end) return;
    const float c[3] = {ctr[box * 3], ctr[box * 3 + 1], ctr[box * 3 + 2]};
    float *rows = rows_s[warp];
    if (lane < len) leaf3_rows<PP>(pts, n, a + lane, c, factor, nt, bs[(size_t)(a + lane) * R + r0], rows + lane * SMALL_RS);
    __syncwarp();
    float acc[NPL];
    int o0[NPL], o1[NPL], o2[NPL];
#pragma unroll
    for (int q = 0; q < NPL; q++) {
        const int m = min(lane + 32 * q, P - 1);
        acc[q] = 0.f;
        o0[q] = m % PP; o1[q] = 8 + (m / PP) % PP; o2[q] = 16 + m / (PP * PP);
    }
    for (int j = 0; j < len; j++) {
        const float *row = rows + j * SMALL_RS;
#pragma unroll
        for (int q = 0; q < NPL; q++) acc[q] = fmaf(row[o2[q]] * row[o1[q]], row[o0[q]], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < NPL; q++)
        if (lane + 32 * q < P) mom[(size_t)box * P + lane + 32 * q] = acc[q];
}

// L2P: lanes = points; the box's local expansion is staged in shared memory and read by every lane
template <int PP>
__global__ void __launch_bounds__(128) l2p_small3(const float *__restrict__ pts, int n, const int *__restrict__ off,
                                                 const float *__restrict__ ctr, float factor, NodeTab2 nt, int row_begin,
                                                 int row_end, const float *__restrict__ loc, int R, int r0, float *out,
                                                 const int *__restrict__ box_list, int nlist) {
    constexpr int P = PP * PP * PP;
    __shared__ float loc_s[4][P];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int li = blockIdx.x * 4 + warp;
    if (li >= nlist) return;
    const int box = box_list[li];
    const int a = off[box], len = off[box + 1] - a;
    if (a < row_begin || a >= row_end) return;
    for (int q = lane; q < P; q += 32) loc_s[warp][q] = __ldg(loc + (size_t)box * P + q);
    __syncwarp();
    if (lane >= len) return;
    const float c[3] = {ctr[box * 3], ctr[box * 3 + 1], ctr[box * 3 + 2]};
    float row[24];
    leaf3_rows<PP>(pts, n, a + lane, c, factor, nt, 1.f, row);
    float v = 0.f;
#pragma unroll
    for (int i2 = 0; i2 < PP; i2++) {
        float s2 = 0.f;
#pragma unroll
        for (int i1 = 0; i1 < PP; i1++) {
            float s1 = 0.f;
#pragma unroll
            for (int i0 = 0; i0 < PP; i0++) s1 = fmaf(row[i0], loc_s[warp][i0 + PP * i1 + PP * PP * i2], s1);
            s2 = fmaf(row[8 + i1], s1, s2);
        }
        v = fmaf(row[16 + i2], s2, v);
    }
    out[(size_t)(a + lane) * R + r0] += v;
}

// lists of the small and the large boxes of the far field's last level, of one tree (0: targets, 1: sources); kept in the plan
// (A few thousand boxes take a CTA each whatever they hold: the split and its read-back would cost more than it saves.)
constexpr int LEAF_SPLIT = 4096;
static void ensure_leaf_split(f3m_plan *pl, int which, int level, cudaStream_t s) {
    if (pl->leaf_level[which] == level) return;
    Level &lv = (which == 0 ? pl->tx : *pl->ty).levels[level];
    if (lv.nb <= LEAF_SPLIT) {
        pl->leaf_big[which].release();   // no list: all boxes
        pl->n_leaf_big[which] = lv.nb;
        pl->n_leaf_small[which] = 0;
        pl->leaf_level[which] = level;
        return;
    }
    pl->leaf_small[which].alloc((size_t)lv.nb, s);
    pl->leaf_big[which].alloc((size_t)lv.nb, s);
    int *counts = pl->d_flags + FL_LEAF;
    F3M_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(int), s));
    split_leaf_boxes<<<(lv.nb + 255) / 256, 256, 0, s>>>(lv.nb, lv.off.p, pl->leaf_small[which].p, pl->leaf_big[which].p, counts);
    F3M_LAUNCH_CHECK();
    F3M_CUDA(cudaMemcpyAsync(pl->h_pinned, counts, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    F3M_CUDA(cudaStreamSynchronize(s));
    pl->n_leaf_small[which] = pl->h_pinned[0];
    pl->n_leaf_big[which] = pl->h_pinned[1];
    pl->leaf_level[which] = level;
}

// ---------------------------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------------------------
// P2M of one level: boxes of the list (or all), the parts of the long ones, and their sums
template <int PP, int RB>
static void p2m_level(f3m_plan *pl, Level &ly, int which, const float *bs, int R, int r0, const NodeTab2 &nt, int P, int chunk, int src_begin,
                      int src_end, float *mom, cudaStream_t s) {
    Tree &ty = *pl->ty;
    const int d = pl->d, n = (int)ty.n, PR = P * RB;
    const float factor = 2.f / ly.edge;          // 1_d_conv.cu:473
    const int64_t slots = chunk ? part_slots(n, chunk) : 0;
    DevBuf<float> part;
    if (chunk) part.alloc((size_t)slots * PR, s);
    if (RB == 1 && d == 3) {
        const int64_t big = pl->n_leaf_big[which];
        if (big + slots)
            p2m_leaf3<PP, false><<<(unsigned)(big + slots), 128, 0, s>>>(ty.pts.p, n, bs, R, r0, ly.off.p, ly.ctr.p, factor, nt, ly.nb, chunk, src_begin,
                                                                 src_end, mom, part.p, pl->leaf_big[which].p, (int)big);
        if (pl->n_leaf_small[which])
            p2m_small3<PP><<<(pl->n_leaf_small[which] + 3) / 4, 128, 0, s>>>(ty.pts.p, n, bs, R, r0, ly.off.p, ly.ctr.p, factor, nt, src_begin,
                                                                            src_end, mom, pl->leaf_small[which].p, pl->n_leaf_small[which]);
    } else {
        const size_t smem = ((size_t)d * PP * 129 + (size_t)128 * RB + (size_t)PR + (size_t)(P / PP)) * sizeof(float);
        F3M_CUDA(cudaFuncSetAttribute(p2m_leaf<PP, RB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        p2m_leaf<PP, RB><<<(unsigned)(ly.nb + slots), 256, smem, s>>>(ty.pts.p, n, d, bs, R, r0, ly.off.p, ly.ctr.p, factor, nt, P, ly.nb, chunk,
                                                                     src_begin, src_end, mom, part.p);
    }
    F3M_LAUNCH_CHECK();
    if (chunk) {
        p2m_combine<<<(unsigned)(slots / 2), 128, 0, s>>>(ly.off.p, ly.nb, n, chunk, PR, src_begin, src_end, part.p, mom);
        F3M_LAUNCH_CHECK();
    }
}

// Sources are interpolated at the first level from L on whose boxes hold at most this many points on average, and moved up by
// M2M, which adds in a tree: with 375 000 sources per box summed at the cut, 3e6 points and l = 10 were 8.4e-7 from float64,
// the finest level's 5.6e-7.  A tree that was built no deeper than the cut has no such level; what makes its sums as good are those of the
// parts of long boxes, which keep their roundings (p2m_combine).
constexpr int64_t SRC_LEAF = 8192;

template <int PP, int RB>
static void far_fast_block(f3m_plan *pl, const float *bs, int R, int r0, float *out, int rb, int re, int lmin, int L, int Ls, int cut,
                           cudaStream_t s) {
    // L: the last level with pairs, whose local expansions go to the targets; Ls >= L: the level the sources are interpolated
    // to; cut == L: that level takes far, small and kept pairs
    Tree &tx = pl->tx, &ty = *pl->ty;
    const int d = pl->d;
    int P = 1;
    for (int k = 0; k < d; k++) P *= PP;
    const int PR = P * RB;
    constexpr int MS = mat_stride(PP);
    NodeTab2 nt = make_nodes2(PP);
    const KronCfg cfg = make_kron_cfg(d, PP, RB);
    const int n_x = (int)tx.n;
    if (RB == 1 && d == 3) {
        ensure_leaf_split(pl, 0, L, s);
        if (!pl->same || Ls != L) ensure_leaf_split(pl, 1, Ls, s);
    }

    if (pl->moments_out) {
        // sharded P2M: finest-level moments of the source boxes that start in [mom_begin, mom_end), zero elsewhere
        Level &ly = ty.levels[L];
        if (pl->mom_box_end >= 0)   // the caller's array holds the boxes [mom_box_begin, mom_box_end) only
            F3M_CUDA(cudaMemsetAsync(pl->moments_out + pl->mom_box_begin * PR, 0,
                                     (size_t)(pl->mom_box_end - pl->mom_box_begin) * PR * sizeof(float), s));
        else
            F3M_CUDA(cudaMemsetAsync(pl->moments_out, 0, (size_t)ly.nb * PR * sizeof(float), s));
        pl->last.begin(ST_P2M, s);
        p2m_level<PP, RB>(pl, ly, pl->same ? 0 : 1, bs, R, r0, nt, P, ly.max_count > 8192 ? 8192 : 0, (int)pl->mom_begin, (int)pl->mom_end,
                          pl->moments_out, s);
        pl->last.end(s);
        return;
    }
    std::vector<DevBuf<float>> mom(Ls + 1), loc(L + 1);
    std::vector<const float *> momp(Ls + 1, nullptr);
    for (int l = lmin; l <= Ls; l++) {
        if (!(l == Ls && pl->ext_mom)) mom[l].alloc((size_t)ty.levels[l].nb * PR, s);
        momp[l] = (l == Ls && pl->ext_mom) ? pl->ext_mom : mom[l].p;
    }
    for (int l = lmin; l <= L; l++) {
        loc[l].alloc((size_t)tx.levels[l].nb * PR, s);
        // the node-to-node kernels write every box of the levels they run on
        if ((l == cut ? pl->cut_lists : pl->lists[l]).far.count == 0) loc[l].zero();
    }
    // tables and cells (setup_levels)
    const bool nested = RB == 1 && (d == 2 || d == 3) && cfg.nf <= 64;
    const bool rows = !nested && rows_form_available<PP, RB>(d);
    std::vector<DevBuf<int>> cellx(L + 1), celly(L + 1);
    auto level_rows = [&](int l) -> LevelLists & { return l == cut ? pl->cut_lists : pl->lists[l]; };
    auto level_geometry = [&](int l) {
        Geom2 geo{};
        for (int k = 0; k < d; k++) {
            double sh = pl->same ? 0.0 : (double)ty.origin[k] - (double)tx.origin[k];
            geo.shift[k] = sh;
            // pairs of level >= 2 descend from parent pairs closer than two parent edges, so their offset lies
            // within a few boxes of -shift/edge; level-1 pairs are children of the root pair: offsets -1, 0, 1
            geo.dqmin[k] = (l == 1 ? 0 : (int)floor(-sh / (double)tx.levels[l].edge)) - NOFF2 / 2 + 1;
        }
        return geo;
    };
    {
        SetupArgs sa{};
        int nlev = 0, most = d * NOFF2 * MS;
        for (int l = lmin; l <= L; l++) {
            LevelLists &ll = level_rows(l);
            const bool cells = !(nested || rows) || !ll.far_ordered;   // the ordered rows hold the offsets
            if (ll.far.count == 0 || (ll.T_ready && !cells)) continue;
            SetupLevel &q = sa.lv[nlev++];
            Level *lv[2] = {&tx.levels[l], &ty.levels[l]};
            if (!ll.T_ready) {   // a constant of the plan: every product uses as many nodes on the level
                ll.T.alloc((size_t)d * NOFF2 * MS, s);
                q.T = ll.T.p;
            }
            q.edge = (double)lv[0]->edge;
            q.geo = level_geometry(l);
            q.level = l;
            for (int t = 0; t < (pl->same ? 1 : 2) && cells; t++) {
                DevBuf<int> &c = t ? celly[l] : cellx[l];
                c.alloc((size_t)lv[t]->nb * d, s);
                q.code[t] = lv[t]->code.p;
                q.cell[t] = c.p;
                q.nb[t] = lv[t]->nb;
                most = std::max(most, lv[t]->nb);
            }
        }
        if (pl->shift_p != PP) {
            std::vector<float> hA, hAT;
            make_shift_tables(nt, hA, hAT);
            pl->shift_p = 0;
            pl->shift_a.alloc(hA.size(), s);
            pl->shift_at.alloc(hAT.size(), s);
            std::copy(hA.begin(), hA.end(), sa.shift.a);
            std::copy(hAT.begin(), hAT.end(), sa.shift.at);
            sa.shift_a = pl->shift_a.p;
            sa.shift_at = pl->shift_at.p;
        }
        if (nlev || sa.shift_a) {
            setup_levels<<<dim3((unsigned)std::min((most + 255) / 256, 4 * NUM_SMS_HINT), std::max(nlev, 1)), 256, 0, s>>>(nt, d, (double)pl->lcs, sa);
            F3M_LAUNCH_CHECK();
            pl->shift_p = PP;
            for (int l = lmin; l <= L; l++) level_rows(l).T_ready = level_rows(l).T.p != nullptr;
        }
    }
    const float *A = pl->shift_a.p, *AT = pl->shift_at.p;

    // warps per CTA of the translation kernels, limited by shared memory
    const size_t per_warp = (size_t)3 * PR * sizeof(float);
    auto warps_for = [&](size_t table_bytes) {
        size_t avail = 200 * 1024 - table_bytes;
        int nw = (int)std::min<size_t>(4, avail / per_warp);
        return nw;
    };

    // ---- P2M at level Ls, M2M upwards ------------------------------------------------------------
    pl->last.begin(ST_P2M, s);
    {
        if (!pl->ext_mom) {
            Level &ly = ty.levels[Ls];
            p2m_level<PP, RB>(pl, ly, pl->same && Ls == L ? 0 : 1, bs, R, r0, nt, P, source_chunk(ly.max_count, ty.n, !(RB == 1 && d == 3)), 0,
                              (int)ty.n, mom[Ls].p, s);
        }
        const int nw = warps_for(2 * MS * sizeof(float));
        size_t sm2 = (size_t)2 * MS * sizeof(float) + nw * per_warp;
        F3M_CUDA(cudaFuncSetAttribute(m2m_fast<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2));
        for (int l = Ls - 1; l >= lmin; l--) {
            Level &lp = ty.levels[l], &lc = ty.levels[l + 1];
            m2m_fast<PP><<<lp.nb, 32 * nw, sm2, s>>>(lp.nb, d, lp.child_start.p, lc.code.p, A, cfg, momp[l + 1], mom[l].p);
            F3M_LAUNCH_CHECK();
        }
    }
    pl->last.end(s);
    // ---- M2L at every level that has far pairs -------------------------------------------------
    pl->last.begin(ST_M2L, s);
    {
        const size_t tab = (size_t)d * NOFF2 * MS * sizeof(float);
        const int nw = warps_for(tab);
        size_t smem = tab + nw * per_warp;
        const bool acc_reg = cfg.nf <= 64;
        // launcher: static strides for d = 2, 3 with one column, runtime strides otherwise
        auto launch_m2l = [&](int nbx, const int *fptr, const int *fidx, const int *cx, const int *cy, const int *offx,
                              const float *T, const Geom2 &geo, const float *momL, float *locL) {
#define F3M_M2L_CALL(ACC_, DD_)                                                                                          \
    {                                                                                                                    \
        F3M_CUDA(cudaFuncSetAttribute(m2l_fast<PP, ACC_, DD_>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
        m2l_fast<PP, ACC_, DD_><<<nbx, 32 * nw, smem, s>>>(nbx, d, fptr, fidx, cx, cy, offx, rb, re, T, geo, cfg, momL,  \
                                                          locL, pl->d_flags);                                            \
    }
            if (RB == 1 && d == 3) { if (acc_reg) F3M_M2L_CALL(true, 3) else F3M_M2L_CALL(false, 3) }
            else if (RB == 1 && d == 2) { if (acc_reg) F3M_M2L_CALL(true, 2) else F3M_M2L_CALL(false, 2) }
            else { if (acc_reg) F3M_M2L_CALL(true, 0) else F3M_M2L_CALL(false, 0) }
#undef F3M_M2L_CALL
        };
        for (int l = lmin; l <= L; l++) {
            const bool at_cut = l == cut;
            LevelLists &level_lists = pl->lists[l];
            LevelLists &ll = level_rows(l);
            if (ll.far.count == 0) continue;
            if (r0 == 0) pl->last.box_pairs += ll.far.count;
            Level &lx = tx.levels[l];
            const ListSet ls{{level_lists.far.ptr.p, level_lists.small.ptr.p, level_lists.keep.ptr.p},
                             {level_lists.far.idx.p, level_lists.small.idx.p, level_lists.keep.idx.p}, at_cut ? 3 : 1};
            if (at_cut && !ll.far_ordered) {
                ll.far.ptr.alloc((size_t)lx.nb + 1, s);
                add_list_ptrs<<<(lx.nb + 1 + 255) / 256, 256, 0, s>>>(lx.nb + 1, ls, ll.far.ptr.p);
                F3M_LAUNCH_CHECK();
            }
            const Geom2 geo = level_geometry(l);
            const float *T = ll.T.p;
            const int *cx = cellx[l].p, *cy = pl->same ? cx : celly[l].p;
            if (nested || rows) {
                if (!ll.far_ordered) {
                    ll.far_okey.alloc((size_t)ll.far.count, s);
                    ll.far_oidx.alloc((size_t)ll.far.count, s);
                    if (d <= 4)
                        far_order_kernel<4><<<(lx.nb + 3) / 4, 128, 0, s>>>(lx.nb, d, ls, cx, cy, geo,
                                                                           ll.far_okey.p, ll.far_oidx.p, pl->d_flags, lx.off.p, rb, re);
                    else
                        far_order_kernel<32><<<(lx.nb + 3) / 4, 128, 0, s>>>(lx.nb, d, ls, cx, cy, geo,
                                                                            ll.far_okey.p, ll.far_oidx.p, pl->d_flags, lx.off.p, rb, re);
                    F3M_LAUNCH_CHECK();
                    // kept for later products of this plan only when every box was ordered
                    ll.far_ordered = rb <= 0 && re >= n_x;
                }
            }
            if (rows) {
                launch_m2l_rows<PP, RB>(d, lx.nb, ll.far.ptr.p, ll.far_okey.p, ll.far_oidx.p, lx.off.p, rb, re, T, momp[l], loc[l].p, s);
            } else if (nested) {
                const size_t smem_n = tab + (size_t)4 * P * sizeof(float);   // tables + one buffer per warp
                if (d == 3) {
                    F3M_CUDA(cudaFuncSetAttribute(m2l_nested<PP, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_n));
                    m2l_nested<PP, 3><<<lx.nb, 128, smem_n, s>>>(lx.nb, ll.far.ptr.p, ll.far_okey.p, ll.far_oidx.p, lx.off.p, rb, re,
                                                                  T, momp[l], loc[l].p);
                } else {
                    F3M_CUDA(cudaFuncSetAttribute(m2l_nested<PP, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_n));
                    m2l_nested<PP, 2><<<lx.nb, 128, smem_n, s>>>(lx.nb, ll.far.ptr.p, ll.far_okey.p, ll.far_oidx.p, lx.off.p, rb, re,
                                                                  T, momp[l], loc[l].p);
                }
            } else
                launch_m2l(lx.nb, ll.far.ptr.p, ll.far.idx.p, cx, cy, lx.off.p, T, geo, momp[l], loc[l].p);
            F3M_LAUNCH_CHECK();
        }
    }
    pl->last.end(s);
    // ---- L2L downwards, L2P at the finest level -------------------------------------------------
    pl->last.begin(ST_L2P, s);
    {
        const int nw = warps_for(2 * MS * sizeof(float));
        size_t sm2 = (size_t)2 * MS * sizeof(float) + nw * per_warp;
        F3M_CUDA(cudaFuncSetAttribute(l2l_fast<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2));
        for (int l = lmin; l < L; l++) {
            Level &lc = tx.levels[l + 1];
            l2l_fast<PP><<<(lc.nb + nw - 1) / nw, 32 * nw, sm2, s>>>(lc.nb, d, lc.parent.p, lc.code.p, lc.off.p, rb, re, AT, cfg,
                                                                    loc[l].p, loc[l + 1].p);
            F3M_LAUNCH_CHECK();
        }
        Level &lx = tx.levels[L];
        const float factor = 2.f / lx.edge;
        const int nsplit = target_parts(lx.max_count, tx.n, lx.nb);
        size_t smem = ((size_t)PR + (size_t)std::max(1, d - 1) * PP * 128) * sizeof(float);
        F3M_CUDA(cudaFuncSetAttribute(l2p_leaf<PP, RB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (RB == 1 && d == 3) {
            if (pl->n_leaf_big[0])
                l2p_leaf3<PP, false><<<dim3(pl->n_leaf_big[0], nsplit), 128, 0, s>>>(tx.pts.p, n_x, lx.off.p, lx.ctr.p, factor, nt, nsplit, rb, re,
                                                                            loc[L].p, R, r0, out, pl->leaf_big[0].p);
            if (pl->n_leaf_small[0])
                l2p_small3<PP><<<(pl->n_leaf_small[0] + 3) / 4, 128, 0, s>>>(tx.pts.p, n_x, lx.off.p, lx.ctr.p, factor, nt, rb, re, loc[L].p,
                                                                           R, r0, out, pl->leaf_small[0].p, pl->n_leaf_small[0]);
        } else
        l2p_leaf<PP, RB><<<dim3(lx.nb, nsplit), 128, smem, s>>>(tx.pts.p, n_x, d, lx.off.p, lx.ctr.p, factor, nt, P, nsplit, rb, re,
                                                               loc[L].p, R, r0, out);
        F3M_LAUNCH_CHECK();
    }
    pl->last.end(s);
}

template <int PP>
static void far_fast_p(f3m_plan *pl, const float *bs, int R, float *out, int rb, int re, int lmin, int L, int Ls, int cut, cudaStream_t s) {
    int P = 1;
    for (int k = 0; k < pl->d; k++) P *= PP;
    // 8 columns at a time when the three per-warp buffers of the translation kernels fit, else one
    const bool wide = R > 1 && (size_t)3 * P * 8 * sizeof(float) + (size_t)pl->d * NOFF2 * mat_stride(PP) * sizeof(float) <= 200 * 1024;
    for (int r0 = 0; r0 < R;) {
        if (wide) { far_fast_block<PP, 8>(pl, bs, R, r0, out, rb, re, lmin, L, Ls, cut, s); r0 += 8; }
        else { far_fast_block<PP, 1>(pl, bs, R, r0, out, rb, re, lmin, L, Ls, cut, s); r0 += 1; }
    }
}

// Number of floats of the finest-level moment array when the far field of (plan, R) runs as one column block on
// the single-pass path, else 0 (then moments cannot be exchanged between ranks and every rank computes its own).
int64_t far_moments_size(const f3m_plan *pl, int R) {
    const int L = pl->levels;
    int lmin = 0, p = 0;
    bool uniform = true;
    for (int l = 1; l <= L; l++) {
        if (pl->lists[l].far.count == 0) continue;
        if (!lmin) { lmin = l; p = pl->lists[l].p; }
        else if (pl->lists[l].p != p) uniform = false;
    }
    if (!lmin || !uniform || p > PMAX_FAST || p < 2) return 0;
    int P = 1;
    for (int k = 0; k < pl->d; k++) P *= p;
    const size_t tab = (size_t)pl->d * NOFF2 * mat_stride(p) * sizeof(float);
    if ((size_t)3 * P * sizeof(float) + tab > 200 * 1024) return 0;
    int RB = 1;
    if (R > 1) {
        if (R > 8 || (size_t)3 * P * 8 * sizeof(float) + tab > 200 * 1024) return 0;
        RB = 8;
    }
    return (int64_t)pl->ty->levels[L].nb * P * RB;
}

// ---------------------------------------------------------------------------------------------
// Where the tree can stop.  The P-node interpolation converges like (edge / 4 l)^p / sqrt(p!), so some levels below the
// first it reproduces the kernel to rounding for EVERY pair of boxes, neighbours and the box itself included: there the
// split into far, small and kept pairs no longer matters, and all child pairs of the kept parents are taken through M2L at
// once.  That level (the cut) ends the product: no direct sums, no deeper lists, no translations below it.
// Measured with box moments / with the cut too: 1e8 points in [0, sqrt12]^3, l = 1, 216 nodes 44.3 -> 18.5 ms (cut at level 4 of 6, M2L
// 13.5 -> 0.24 ms), 1e7 points from host tensors 8.8 -> 5.5 ms, a mixture of 1e7 points, l = 0.5 50.8 -> 22.8 ms (level 7 of 8).  Error
// against float64 unchanged or smaller (1e6 points, l = 4, positive weights 1.5e-7 -> 1.3e-7).
//
// Bound.  The kernel is a product over the axes, so the relative error of a pair is the sum over the axes of that of one axis.
// There g(u) = exp(-u^2 / 2 l^2) is interpolated in x and in y over an edge e: error <= (1 + Lambda_p) E, with E =
// max |g^(p)| / p! (e/2)^p / 2^(p-1) and max |g^(p)| <= 1.0865 sqrt(p!) / l^p (Cramer's inequality), Lambda_p <= 1 + (2/pi) ln p;
// and g is at least exp(-(r e)^2 / 2 l^2), r - 1 the offset of the boxes along the axis.  Offsets (near_moments.cu): on one tree the
// children of kept parents are (3,3,3,..) or (5,1,..) boxes apart, on two trees below 5 along every axis.  The sum must stay below
// CUT_EPS = 1.2e-7, half the error of ex2.approx.
// ---------------------------------------------------------------------------------------------
constexpr double CUT_EPS = 1.2e-7;

// edge: of the level; offset: between the two trees' origins, null for one tree
static bool cut_is_exact(int d, double edge, double lcs, const double *offset, int level, int p) {
    const bool same = offset == nullptr;
    const double e = edge * sqrt(2.0 * lcs);   // edge / l
    auto inv_g = [&](double r) { return exp(0.5 * r * r * e * e); };
    double sum;
    if (level == 1) {   // children of the root pair, which is kept without a distance test
        sum = 0.0;
        for (int k = 0; k < d; k++)
            sum += inv_g(2.0 + (same ? 0.0 : fabs(offset[k]) / edge));
    } else
        sum = same ? std::max(d * inv_g(4.0), inv_g(6.0) + (d - 1) * inv_g(2.0)) : d * inv_g(6.0);
    double fact = 1.0;
    for (int i = 2; i <= p; i++) fact *= i;
    const double E = 2.0 * 1.0865 * pow(e / 4.0, p) / sqrt(fact);
    return E * (2.0 + 2.0 / 3.14159265358979323846 * log((double)p)) * sum <= CUT_EPS;
}

// Level at which the product ends (0: no cut, all lists are used).  Among the levels that qualify the one with the smallest
// estimated time wins.  Measured rates behind the estimate: M2L 1.25e-12 s per pair, node and column (0.25 ns per pair at 216
// nodes, 2.5 ns at 243 nodes and 8 columns), translations 8e-12 s per box, node and column, direct lists see
// node_choice; a cut orders a list of its own and sets up the level (20 us), which small trees do not win back.
static bool cut_kernels_fit(const f3m_plan *pl, int R, int p, bool &wide) {
    const int d = pl->d;
    if ((pl->prm.flags & F3M_FLAG_NEAR_TENSOR_CORES) || pl->prm.var_compression || p < 2 || p > PMAX_FAST || d < 2) return false;
    int P = 1;
    for (int k = 0; k < d; k++) P *= p;
    const size_t tab = (size_t)d * NOFF2 * mat_stride(p) * sizeof(float);
    if ((size_t)3 * P * sizeof(float) + tab > 200 * 1024) return false;
    wide = R > 1 && (size_t)3 * P * 8 * sizeof(float) + tab <= 200 * 1024;
    // the combined list exists in ordered form only, which these kernels read
    return wide ? rows_form_for(p, d) : (d <= 3 && P / p <= 64);
}

// The level at which a plan for one product can end, known before its points are sorted; 0: unknown.  It is the first level whose
// interpolation is exact for all pairs, where its boxes hold STOP_POINTS points on average however they are spread: neither the pairs
// nor the moments of so full boxes take less time than one node-to-node step, and the levels below have a multiple of its pairs.
constexpr int64_t STOP_POINTS = 256;
int far_stop_level(const f3m_plan *pl, int R, float edge0, const float *xmin, const float *ymin, int64_t n) {
    const int d = pl->d, p = nodes_per_dim(d, pl->prm.nr_interpolation);
    bool wide;
    if (!cut_kernels_fit(pl, R, p, wide)) return 0;
    double off[MAXD];
    for (int k = 0; k < d && ymin; k++) off[k] = (double)xmin[k] - (double)ymin[k];
    for (int l = 1; (n >> (d * l)) >= STOP_POINTS; l++)
        if (cut_is_exact(d, ldexp((double)edge0, -l), (double)pl->lcs, ymin ? off : nullptr, l, p)) return l;
    return 0;
}

// A second way to end: at a level whose own nodes do not reproduce its near pairs, but whose children's do.  The far pairs of the levels
// below are then as good as exact, so that the small and kept pairs of this level can take all that stands in for them: through
// more nodes, the number near_nodes.cu needs (one column, three dimensions).  Mixture of 1e7 points, l = 0.5, 216 nodes: level 6
// with 7 nodes for 4.0e6 pairs in place of level 7 and its 1.96e7, whole call 16.8 -> 7.9 ms (M2L 5.4 -> 0.9, levels 7 and 8 neither built nor sorted for).
static bool ends_exactly_below(const f3m_plan *pl, double edge, int level) {
    const int p = nodes_per_dim(pl->d, pl->prm.nr_interpolation);
    bool wide;
    return cut_kernels_fit(pl, 1, p, wide) && pl->same && cut_is_exact(pl->d, 0.5 * edge, (double)pl->lcs, nullptr, level + 1, p);
}

CutChoice far_cut(const f3m_plan *pl, int R, bool nodes_allowed) {
    CutChoice best;
    const int L = pl->levels, d = pl->d;
    if (L < 1) return best;
    const int p = pl->lists[1].p;
    bool wide;
    if (!cut_kernels_fit(pl, R, p, wide)) return best;
    int P = 1;
    for (int k = 0; k < d; k++) P *= p;
    double off[MAXD];
    for (int k = 0; k < d; k++) off[k] = (double)pl->tx.origin[k] - (double)pl->ty->origin[k];
    const double cols = wide ? 8.0 * ((R + 7) / 8) : R;
    auto m2l = [&](const PairCSR &c) { return (double)c.count * P * cols * 1.25e-12; };
    auto shifts = [&](int l) { return ((double)pl->tx.levels[l].nb + pl->ty->levels[l].nb) * P * cols * 8e-12; };
    std::vector<double> direct(L + 1);
    double full = 0.0;
    for (int l = 1; l <= L; l++) {
        direct[l] = node_choice(pl, l, R).seconds;
        full += direct[l] + m2l(pl->lists[l].far) + shifts(l);
    }
    double best_t = full, head = 20e-6;
    for (int l = 1; l <= L; l++) {
        const LevelLists &ll = pl->lists[l];
        const double t = head + m2l(ll.far) + m2l(ll.small) + m2l(ll.keep) + shifts(l);
        if (t < best_t && ll.far.count + ll.small.count + ll.keep.count <= 0x7fffffffLL &&
            cut_is_exact(d, (double)pl->ty->levels[l].edge, (double)pl->lcs, pl->same ? nullptr : off, l, p)) {
            best = CutChoice{};
            best.level = l;
            best_t = t;
        }
        if (nodes_allowed && R == 1 && l < L && ends_exactly_below(pl, (double)pl->ty->levels[l].edge, l)) {
            const NodeChoice n = node_end(pl, l);
            const double tn = head + m2l(ll.far) + shifts(l) + n.seconds;
            if (n.p && tn < best_t) {
                best.level = l;
                best.nodes = n;
                best_t = tn;
            }
        }
        head += direct[l] + m2l(ll.far) + shifts(l);
    }
    return best;
}

// The first level at which a product could end that way, from the cube's edge; 0: none within the key's depth
int far_node_end_level(const f3m_plan *pl, float edge0, int lmax) {
    for (int l = 1; l < lmax; l++)
        if (ends_exactly_below(pl, ldexp((double)edge0, -l), l)) return pl->d == 3 ? l : 0;
    return 0;
}

// While the tree of a plan for one product is built: may it end at this level, whose lists are there?  If it can (above) and going on
// would cost more: one node-to-node step for every child pair of the kept pairs, of which there are 2^d or more per pair where its boxes
// are populated, besides the lists and the deeper sort.
// A product that refuses the nodes (node_sums) sums this level's lists pair by pair, in boxes wider than the full tree's.  Whole calls with one
// infinite weight / finite, and of the full tree as it was: mixture of 1e7 points 24.4 / 13.5, 33 ms; 2e7 normal points, l = 0.3, 42.6 / 22.6,
// 60 ms; twenty narrow clouds, 2e6 to 1e8 points, 1.0 to 2.2 times the finite call: where boxes are that full, small lists, box
// moments and the far field's exact level (far_cut) are left.
bool far_ends_with_nodes(const f3m_plan *pl, int level) {
    const int p = nodes_per_dim(pl->d, pl->prm.nr_interpolation);
    if (!ends_exactly_below(pl, (double)pl->ty->levels[level].edge, level)) return false;
    const NodeChoice n = node_end(pl, level);
    if (!n.p) return false;
    const LevelLists &ll = pl->lists[level];
    const double P = pow((double)p, pl->d), small = ll.small.count ? direct_list_seconds(pl, level, ll.small, 1) : 0.0;
    const double below = (double)ll.keep.count * (1 << pl->d) * P * 1.25e-12 + 2.0 * pl->tx.levels[level].nb * (1 << pl->d) / 2 * P * 8e-12;
    return n.seconds <= small + below;
}

// Far field of the whole product.  Fast path when every level with far pairs uses the same p <= 8;
// otherwise (var_compression switching node counts between levels, or more nodes per dimension) the
// per-level path of far.cu.  cut > 0 (far_cut): the product ends at that level, all of whose pairs are taken here.
void far_field(f3m_plan *pl, const float *b_sorted, int R, float *out_sorted, int64_t row_begin, int64_t row_end, int cut, int end,
               cudaStream_t s) {
    int lmin = 0, llast = 0, p = 0;
    bool uniform = true;
    if (cut && pl->cut_level != cut) {   // the number of columns can move the cut
        LevelLists &ll = pl->lists[cut], &all = pl->cut_lists;
        all.far_ordered = false;
        all.T_ready = false;
        all.far.count = ll.far.count + ll.small.count + ll.keep.count;
        all.p = ll.p;
        pl->cut_level = cut;
    }
    for (int l = 1; l <= end; l++) {
        if ((l == cut ? pl->cut_lists.far.count : pl->lists[l].far.count) == 0) continue;
        llast = l;
        if (!lmin) { lmin = l; p = pl->lists[l].p; }
        else if (pl->lists[l].p != p) uniform = false;
    }
    if (!lmin) return;
    int P = 1;
    for (int k = 0; k < pl->d; k++) P *= p;
    const bool fits = (size_t)3 * P * sizeof(float) + (size_t)pl->d * NOFF2 * mat_stride(p) * sizeof(float) <= 200 * 1024;
    if (!uniform || p > PMAX_FAST || p < 2 || !fits) {
        for (int l = lmin; l <= end; l++) far_field_level(pl, l, b_sorted, R, out_sorted, row_begin, row_end, s);
        return;
    }
    const int rb = (int)row_begin, re = (int)row_end;
    // Points are interpolated to the deepest level that has far pairs: below it there is nothing to translate (a mixture of
    // 1e7 points has 1.55 M boxes of six points and no far pair on its last level).  Slices of the rows and exchanged
    // moments are cut at boxes of the last level, so they stay there.
    const bool whole = rb <= 0 && re >= (int)pl->tx.n && !pl->moments_out && !pl->ext_mom && !pl->shard.active;
    const int last = whole ? llast : pl->levels;
    int src = last;
    while (whole && src < pl->levels && pl->ty->n / pl->ty->levels[src].nb > SRC_LEAF) src++;
    switch (p) {
        case 2: far_fast_p<2>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
        case 3: far_fast_p<3>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
        case 4: far_fast_p<4>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
        case 5: far_fast_p<5>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
        case 6: far_fast_p<6>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
        case 7: far_fast_p<7>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
        default: far_fast_p<8>(pl, b_sorted, R, out_sorted, rb, re, lmin, last, src, cut, s); break;
    }
}

}  // namespace f3m
