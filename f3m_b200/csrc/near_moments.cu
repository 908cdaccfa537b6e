// Near sums through box moments.
//
// The pairs of a near / small list (near_field_run, F3M_src/n_tree.cu:831-902) are summed here without visiting the
// pairs, wherever the boxes are small against the lengthscale.  With c the centre of the source box,
//     exp(-|x-y|^2 / (2 l^2)) = exp(-|x-c|^2 / (2 l^2)) * exp(-|y-c|^2 / (2 l^2)) * exp(t),   t = (x-c).(y-c) / l^2.
// The first factor belongs to the target, the second to the source's weight.  |t| is bounded over the whole list by its
// geometry, and exp(t) is replaced by the polynomial of degree K through the Chebyshev points of [-h, h]: its relative
// error stays below MOM_EPS = 1.2e-7 (half the error of ex2.approx, which the pair form uses).  A polynomial of
// the inner product is a sum of products of target and source monomials, so a source box enters only through
//     M_q = c_|q| * multiplicity_q * sum_j b_j exp(-|y_j-c|^2 / (2 l^2)) (y_j-c)^q / l^(2|q|),   |q| <= K,
// and a target costs one exponential and C(K+d, d) multiply-adds per source BOX: 20 at d = 3, K = 3, against one
// multiply-add chain and one exponential per source POINT.
//
// Measured (near sums of one product, pair form -> this form): 1e8 points in [0, sqrt12]^3, l = 1, K = 3, 381 points per
// box 223.7 -> 10.0 ms; 1e7 points 19.9 -> 1.6 ms (K = 4); 1e5 points in the unit cube (K = 3) 0.187 -> 0.029 ms; 2e4 points
// (K = 6) 0.176 -> 0.025 ms; the two lists of a mixture of 1e7 points whose boxes are narrow enough 56.4 -> 35.4 ms of all
// lists.  near_moments_eval is bound by issue slots (about 37 per target and box at K = 3), near_moments_build by HBM.
#include <math.h>
#include <algorithm>
#include "common.cuh"
#include "packed.cuh"

namespace f3m {

constexpr double MOM_EPS = 1.2e-7;        // relative truncation error of the default form
constexpr double MOM_EPS_FLAG = 1e-6;     // on request (F3M_FLAG_NEAR_MOMENTS)
constexpr int MOM_KMAX = 6;

__host__ __device__ constexpr int mom_binom(int n, int k) {
    int r = 1;
    for (int i = 1; i <= k; i++) r = r * (n - k + i) / i;
    return r;
}
__host__ __device__ constexpr int mom_count(int D, int K) { return mom_binom(D + K, D); }
// highest degree instantiated: C(K+d, d) stays near 80, above that a box would need hundreds of points to pay
__host__ __device__ constexpr int mom_kmax(int D) { return D <= 3 ? 6 : 3; }
// a box's record: its centre, then RB columns of moments, moment by moment (four columns start on a 16-byte boundary)
__host__ __device__ constexpr int mom_first(int D, int RB) { return RB == 1 ? D : 4 * ((D + 3) / 4); }
__host__ __device__ constexpr int mom_record(int D, int K, int RB) { return (mom_first(D, RB) + RB * mom_count(D, K) + 3) / 4 * 4; }

struct MomFactors { float f[84]; };

// Monomials x_a x_b x_c .. with a <= b <= c .., depth first: node (DEPTH, AMIN, Q) is monomial number Q of degree DEPTH,
// its children multiply by x_A for A >= AMIN.
template <int D, int K, int DEPTH, int AMIN, int Q>
struct MomTree {
    __host__ __device__ static constexpr int sub(int A) { return mom_binom(K - DEPTH - 1 + D - A, D - A); }
    template <int A, int QQ>
    static __device__ __forceinline__ void build_from(float w, const float (&y)[D], float *acc) {
        if constexpr (A < D) {
            if constexpr (DEPTH + 1 == K) acc[QQ] = fmaf(w, y[A], acc[QQ]);
            else MomTree<D, K, DEPTH + 1, A, QQ>::build(w * y[A], y, acc);
            build_from<A + 1, QQ + sub(A)>(w, y, acc);
        }
    }
    static __device__ __forceinline__ void build(float w, const float (&y)[D], float *acc) {
        acc[Q] += w;
        build_from<AMIN, Q + 1>(w, y, acc);
    }
    template <int A, int QQ, typename V>
    static __device__ __forceinline__ V eval_from(V v, const typename V::X (&x)[D], const float *m) {
        if constexpr (A < D) {
            V c;
            if constexpr (DEPTH + 1 == K) c = V::load(m, QQ);
            else c = MomTree<D, K, DEPTH + 1, A, QQ>::template eval<V>(x, m);
            return eval_from<A + 1, QQ + sub(A), V>(V::fma(x[A], c, v), x, m);
        } else
            return v;
    }
    template <typename V>
    static __device__ __forceinline__ V eval(const typename V::X (&x)[D], const float *m) {
        return eval_from<AMIN, Q + 1, V>(V::load(m, Q), x, m);
    }
    // coefficient and multinomial factor of every monomial: mult = DEPTH! / prod n_a!, run = how often the last letter
    // occurs already (one more when the child repeats it)
    static void factors(const double *cf, double mult, int run, float *f) {
        f[Q] = (float)(cf[DEPTH] * mult);
        factors_from<AMIN, Q + 1>(cf, mult, run, f);
    }
    template <int A, int QQ>
    static void factors_from(const double *cf, double mult, int run, float *f) {
        if constexpr (A < D) {
            const int r = (A == AMIN && DEPTH > 0) ? run + 1 : 1;
            const double m = mult * (DEPTH + 1) / r;
            if constexpr (DEPTH + 1 == K) f[QQ] = (float)(cf[K] * m);
            else MomTree<D, K, DEPTH + 1, A, QQ>::factors(cf, m, r, f);
            factors_from<A + 1, QQ + sub(A)>(cf, mult, run, f);
        }
    }
};

struct Val1 {   // one column; the record already lies in registers
    typedef float X;
    float v;
    static __device__ __forceinline__ Val1 load(const float *m, int q) { return Val1{m[q]}; }
    static __device__ __forceinline__ Val1 fma(float x, Val1 a, Val1 c) { return Val1{fmaf(x, a.v, c.v)}; }
};
struct Val4 {   // four columns of one moment: one 16-byte load, two packed multiply-adds
    typedef f32x2 X;
    f32x2 lo, hi;
    static __device__ __forceinline__ Val4 load(const float *m, int q) {
        const ulonglong2 w = __ldg(reinterpret_cast<const ulonglong2 *>(m + 4 * q));
        return Val4{w.x, w.y};
    }
    static __device__ __forceinline__ Val4 fma(X x, Val4 a, Val4 c) { return Val4{fma2(x, a.lo, c.lo), fma2(x, a.hi, c.hi)}; }
};

// A group of T threads (one warp, or a CTA of 256 when the boxes are long) per (source box, column).  Boxes of more than `chunk`
// rows (0: there are none) are summed in parts by the groups behind, a group per (slot, column); near_moments_combine adds
// them up.
template <int D, int K, int RB, int T>
__global__ void __launch_bounds__(256) near_moments_build(const float *__restrict__ pts, int n, const float *__restrict__ bs, int R,
                                                         int r0, float unit, float s2, const int *__restrict__ off_y, int nby,
                                                         const float *__restrict__ ctr_y, const unsigned char *__restrict__ need,
                                                         MomFactors fac, int chunk, float *rec, float *parts) {
    constexpr int NM = mom_count(D, K), REC = mom_record(D, K, RB);
    __shared__ float part[T == 32 ? 1 : 8][NM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t g = ((int64_t)blockIdx.x * 256 + threadIdx.x) / T, boxes = (int64_t)nby * RB;
    const bool in_part = g >= boxes;
    if (in_part && (T == 32 || !chunk)) return;      // whole groups leave: T = 256 is the whole CTA
    const int64_t item = (in_part ? g - boxes : g) / RB;
    const int r = (int)((in_part ? g - boxes : g) - item * RB);
    BoxPart bp{(int)item, 0, 0};
    if (T == 256 && in_part) bp = part_of_slot(off_y, nby, n, chunk, item);
    else { bp.begin = off_y[item]; bp.end = off_y[item + 1]; }
    const int by = bp.box, a = bp.begin, b = bp.end;
    if (in_part ? a == b : (chunk && b - a > chunk)) return;
    if (need && !need[by]) return;           // a slice of the targets names only some source boxes
    float c[D];
#pragma unroll
    for (int k = 0; k < D; k++) c[k] = ctr_y[by * D + k];
    float acc[NM];
#pragma unroll
    for (int q = 0; q < NM; q++) acc[q] = 0.f;
    if (r0 + r < R)
        for (int j = a + (int)(threadIdx.x % T); j < b; j += T) {
            float y[D], n2 = 0.f;
#pragma unroll
            for (int k = 0; k < D; k++) {
                const float v = unit * (pts[(size_t)k * n + j] - c[k]);
                n2 = fmaf(v, v, n2);
                y[k] = 2.f * s2 * v;
            }
            MomTree<D, K, 0, 0, 0>::build(bs[(size_t)j * R + r0 + r] * ex2_approx(-s2 * n2), y, acc);
        }
#pragma unroll
    for (int q = 0; q < NM; q++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    float *dst = rec + (size_t)by * REC;
    auto put = [&](int q, float v) {
        dst[mom_first(D, RB) + q * RB + r] = v * fac.f[q];
    };
    // Where the sum of the weights is not finite, it alone stays: the pairs' terms are positive, so their sum is that value too, while
    // the other moments would carry it with either sign.
    if (T == 32) {
        const bool bad = !isfinite(acc[0]);
#pragma unroll
        for (int q = 0; q < NM; q++)
            if (lane == (q & 31)) put(q, q && bad ? 0.f : acc[q]);
    } else {
#pragma unroll
        for (int q = 0; q < NM; q++)
            if (lane == (q & 31)) part[T == 32 ? 0 : warp][q] = acc[q];
        __syncthreads();
        for (int q = threadIdx.x; q < NM; q += T) {
            float v = 0.f, v0 = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w++) {
                v += part[T == 32 ? 0 : w][q];
                v0 += part[T == 32 ? 0 : w][0];
            }
            if (in_part) parts[((size_t)item * RB + r) * NM + q] = v;
            else put(q, q && !isfinite(v0) ? 0.f : v);
        }
    }
    if (r == 0 && !in_part && (int)(threadIdx.x % T) < D) dst[threadIdx.x % T] = unit * ctr_y[by * D + threadIdx.x % T];
}

// records of the long boxes: their parts added in the order of the rows, a CTA per chunk of rows
template <int D, int K, int RB>
__global__ void __launch_bounds__(128) near_moments_combine(float unit, const int *__restrict__ off_y, int nby, int n,
                                                           const float *__restrict__ ctr_y, const unsigned char *__restrict__ need,
                                                           MomFactors fac, int chunk, const float *__restrict__ parts, float *rec) {
    constexpr int NM = mom_count(D, K);
    const LongBox l = long_box_of_chunk(off_y, nby, n, chunk, blockIdx.x);
    if (l.box < 0 || (need && !need[l.box])) return;
    float *dst = rec + (size_t)l.box * mom_record(D, K, RB);
    auto sum = [&](int q, int r) {
        float v = parts[((size_t)l.first_slot * RB + r) * NM + q];
        for (int64_t t = (l.first_slot | 1) + 1; t <= l.last_slot; t += 2) v += parts[((size_t)t * RB + r) * NM + q];
        return v;
    };
    for (int i = threadIdx.x; i < NM * RB; i += 128) {
        const int q = i / RB, r = i - q * RB;
        const float v = sum(q, r);
        dst[mom_first(D, RB) + q * RB + r] = (q && !isfinite(sum(0, r)) ? 0.f : v) * fac.f[q];
    }
    if (threadIdx.x < D) dst[threadIdx.x] = unit * ctr_y[l.box * D + threadIdx.x];
}

// One thread per target row.  Rows are in box order, so the lanes of a warp read the same record (a broadcast) except
// where it straddles two boxes; no tiles, no scan and no host read-back are needed.  Two lists of the level (small and
// near) are walked one after the other and written once.  G lanes share a row (every G-th box of its lists each): calls
// whose rows do not fill the SMs would wait out the boxes one after the other (2e4 rows, K = 6: 29.2 -> 14.1 us; 1e5 rows, K = 3, the lanes' shorter
// runs and wider gathers cost more than they hide: 16.1 -> 20.4 us).
template <int D, int K, int RB, int G>
__global__ void __launch_bounds__(128) near_moments_eval(const float *__restrict__ xpts, int n_x, const int *__restrict__ off_x, int nbx,
                                                        int row_begin, int row_end, const int *__restrict__ ptr1,
                                                        const int *__restrict__ idx1, const int *__restrict__ ptr2,
                                                        const int *__restrict__ idx2, const float *__restrict__ rec, float unit, float s2,
                                                        int R, int r0, float *out) {
    constexpr int REC = mom_record(D, K, RB);
    const int lane = threadIdx.x & 31, sub = lane % G;
    const int i0 = row_begin + (int)((blockIdx.x * 128 + (threadIdx.x & ~31)) / G);
    if (i0 >= row_end) return;
    // boxes of the warp's first and last row by two lanes, then each lane searches between them
    int box = box_of_row(off_x, nbx, lane == 31 ? min(i0 + 32 / G - 1, row_end - 1) : i0);
    const int b_lo = __shfl_sync(0xffffffffu, box, 0), b_hi = __shfl_sync(0xffffffffu, box, 31);
    const bool mine = i0 + lane / G < row_end;
    const int i = mine ? i0 + lane / G : row_end - 1;
    box = b_lo + (b_hi > b_lo ? box_of_row(off_x + b_lo, b_hi - b_lo + 1, i) : 0);
    float x[D], tot[RB];
#pragma unroll
    for (int k = 0; k < D; k++) x[k] = unit * xpts[(size_t)k * n_x + i];
#pragma unroll
    for (int r = 0; r < RB; r++) tot[r] = 0.f;
    bool any = false;
#pragma unroll 1
    for (int l = 0; l < 2; l++) {
        const int *ptr = l ? ptr2 : ptr1, *idx = l ? idx2 : idx1;
        if (!ptr) continue;
        const int e0 = ptr[box], e1 = ptr[box + 1];
        any = any || e1 > e0;
        int by = e0 + sub < e1 ? idx[e0 + sub] : 0;
        for (int e = e0 + sub; e < e1; e += G) {
            const float *m = rec + (size_t)by * REC;
            if (e + G < e1) by = idx[e + G];
            if constexpr (RB == 1) {
                float mr[REC];
#pragma unroll
                for (int q = 0; q < REC / 4; q++) {
                    const float4 v = __ldg(reinterpret_cast<const float4 *>(m) + q);
                    mr[4 * q] = v.x; mr[4 * q + 1] = v.y; mr[4 * q + 2] = v.z; mr[4 * q + 3] = v.w;
                }
                float xr[D], n2 = 0.f;
#pragma unroll
                for (int k = 0; k < D; k++) {
                    xr[k] = x[k] - mr[k];
                    n2 = fmaf(xr[k], xr[k], n2);
                }
                tot[0] = fmaf(ex2_approx(-s2 * n2), MomTree<D, K, 0, 0, 0>::template eval<Val1>(xr, mr + mom_first(D, RB)).v, tot[0]);
            } else {
                f32x2 xr[D];
                float n2 = 0.f;
#pragma unroll
                for (int k = 0; k < D; k++) {
                    const float v = x[k] - __ldg(m + k);
                    n2 = fmaf(v, v, n2);
                    xr[k] = pack2(v, v);
                }
                const Val4 p = MomTree<D, K, 0, 0, 0>::template eval<Val4>(xr, m + mom_first(D, RB));
                const float fx = ex2_approx(-s2 * n2);
                float pv[4];
                unpack2(p.lo, pv[0], pv[1]);
                unpack2(p.hi, pv[2], pv[3]);
#pragma unroll
                for (int r = 0; r < RB; r++) tot[r] = fmaf(fx, pv[r], tot[r]);
            }
        }
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1)
#pragma unroll
        for (int r = 0; r < RB; r++) tot[r] += __shfl_xor_sync(0xffffffffu, tot[r], o);
    if (!any || !mine || sub) return;
#pragma unroll
    for (int r = 0; r < RB; r++)
        if (r0 + r < R) out[(size_t)i * R + r0 + r] += tot[r];
}

// Polynomial of degree K through the Chebyshev points of [-h, h] for exp, as monomial coefficients.
static void exp_poly_fit(double h, int K, double (&cf)[MOM_KMAX + 1]) {
    double tn[MOM_KMAX + 1], dd[MOM_KMAX + 1];
    const int m = K + 1;
    h = std::max(h, 1e-3);   // keeps the divided differences well conditioned; the error there is far below the bound
    for (int i = 0; i < m; i++) {
        tn[i] = h * cos((2 * i + 1) * 3.14159265358979323846 / (2.0 * m));
        dd[i] = exp(tn[i]);
    }
    for (int j = 1; j < m; j++)
        for (int i = m - 1; i >= j; i--) dd[i] = (dd[i] - dd[i - 1]) / (tn[i] - tn[i - j]);
    for (double &c : cf) c = 0.0;
    for (int i = m - 1; i >= 0; i--) {
        for (int q = m - 1; q >= 1; q--) cf[q] = cf[q - 1] - tn[i] * cf[q];
        cf[0] = -tn[i] * cf[0] + dd[i];
    }
}

// Bound h of |(x-c).(y-c)| / l^2 over the pairs of a list, x a target, y a point of a source box with centre c.  In box
// edges: |y-c| <= sqrt(d)/2 and |x-c| <= centre distance + sqrt(d)/2, and per axis |y_k-c_k| <= 1/2, so the lesser of
// (dist + sqrt(d)/2) sqrt(d)/2 and (sum_k |centre offset_k| + d/2) / 2 holds.  On one tree offsets are whole boxes.  Kept pairs
// are at most two boxes apart in the 2-norm (two exactly when the far test rounds down): (1,1,1,..) or (2,0,..).  "Small"
// pairs are children of kept parents: (3,3,3,..) or (5,1,..).  Two trees have fractional offsets: 2, and 4 plus sqrt(d)/2 from either
// child's centre to its parent's.  Level-1 pairs descend from the root pair, which is kept without a test: one box apart per
// axis on one tree, plus the two cubes' offset otherwise.
static double list_exponent_bound(const f3m_plan *pl, int level, bool keep) {
    const int d = pl->d;
    const double sd = sqrt((double)d), e = (double)pl->ty->levels[level].edge;
    double dist, sum;   // 2-norm and 1-norm of the centre offset
    if (level == 1 && !keep) {
        dist = sum = 0.0;
        for (int k = 0; k < d; k++) {
            const double o = 1.0 + (pl->same ? 0.0 : fabs((double)pl->tx.origin[k] - (double)pl->ty->origin[k]) / e);
            dist += o * o;
            sum += o;
        }
        dist = sqrt(dist);
    } else if (keep) {
        dist = 2.0;
        sum = pl->same ? std::max(2.0, std::min((double)d, 4.0)) : 2.0 * sd;
    } else {
        dist = pl->same ? sqrt(std::max(9.0 * d, 24.0 + d)) : 4.0 + sd;
        sum = pl->same ? std::max(3.0 * d, 4.0 + d) : sd * dist;
    }
    const double bound = std::min((dist + 0.5 * sd) * 0.5 * sd, (sum + 0.5 * d) * 0.5);
    return 1.01 * bound * e * e * 2.0 * (double)pl->lcs;   // 1 / l^2 = 2 lcs; 1 % for the rounding of centres and far test
}

// Estimated device time of a list's moments: evaluations, and what every block of columns pays once.  Measured: one column 3.2e-12 s per
// (target, box) of 20 terms + 17 other issue slots, so 8.6e-14 s per slot; a block of four columns, whose records come through
// L1, 1.2e-11 s at 10 terms, 2.1e-11 at 35, 3.2e-11 at 84.  A block builds the records of all boxes and looks up every row.
struct MomentSeconds { double eval, fixed; };
static MomentSeconds moment_seconds(const f3m_plan *pl, const PairCSR &csr, int K, int R) {
    const double nm = mom_count(pl->d, K), build = (double)pl->ty->n * (nm + 20.0) * 8.6e-14, rows = (double)pl->tx.n * 1e-11;
    const int fours = R % 4 == 1 ? R / 4 : (R + 3) / 4, ones = R % 4 == 1;
    return {(double)csr.row_boxes * (fours * (8e-12 + 3.5e-13 * nm) + ones * (nm + 17.0) * 8.6e-14),
            fours * (4.0 * build + rows) + ones * (build + rows)};
}

// Degree for one list, 0 when its pairs are summed one by one.  The Chebyshev interpolation error is at most
// e^h h^(K+1) / (2^K (K+1)!), and exp(t) >= e^-h.
static int list_moment_degree(const f3m_plan *pl, int level, bool keep, int R) {
    const PairCSR &csr = keep ? pl->lists[level].keep : pl->lists[level].small;
    const bool flag = pl->prm.flags & F3M_FLAG_NEAR_MOMENTS;
    if (level < 1 || csr.count == 0) return 0;
    if ((pl->prm.flags & F3M_FLAG_NEAR_TENSOR_CORES) && !flag) return 0;
    const double h = list_exponent_bound(pl, level, keep), eps = flag ? MOM_EPS_FLAG : MOM_EPS;
    double term = h;   // h^K / K!
    for (int K = 2; K <= mom_kmax(pl->d); K++) {
        term *= h / K;
        if (exp(2.0 * h) * term * h / (K + 1) * ldexp(1.0, -K) <= eps) {
            if (flag) return K;
            // Moments where they take less time than the pairs.  Either form also launches a few kernels per block of columns, 10 us
            // for tiles, scan, packing and sums.  One column: an evaluation of 20 terms at 3.2e11 /s against pairs at 5.2e12 /s (3.5e12
            // without polynomial pairs) is about one term per 0.5 to 0.8 pairs;
            // the pair form's own preparation (flags, packing, read-backs) costs lists of a few pairs no less than the records do (mixture of
            // 1.4e7 points, l = 5.5: 24.8 ms with moments, 25.4 with pairs).  Two columns and more, eight columns measured,
            // moments / pairs: d = 1, 1e6 normal points, lists of a few pairs on eight levels 0.72 / 0.56 ms; d = 3, l = 0.3, 1e6 normal
            // points, boxes of twelve 10.1 / 4.3 ms; d = 2, 1e6 uniform points 0.25 / 0.59 ms.
            if (R == 1) return (double)csr.pairs >= 0.5 * mom_count(pl->d, K) * (double)csr.row_boxes ? K : 0;
            const MomentSeconds t = moment_seconds(pl, csr, K, R);
            const double pairs = pair_list_seconds(pl, level, csr, R) + 1e-5 * ((R + 7) / 8);
            // Ties go to moments.  Measured there, moments / pairs: d = 4, 4.8e5 uniform points, 2 columns 3442 / 3455 us, 4 columns 4374 / 4411;
            // but d = 5, 3e4 points, 2 to 4 columns 1164 to 1180 / 624 us: calls that small leave SMs idle, which this estimate does not know.
            return t.eval + t.fixed <= 1.05 * pairs ? K : 0;
        }
    }
    return 0;
}

// Estimated device time of a direct list.
double direct_list_seconds(const f3m_plan *pl, int level, const PairCSR &csr, int R) {
    if (csr.count == 0) return 0.0;
    const int K = list_moment_degree(pl, level, &csr == &pl->lists[level].keep, R);
    if (!K) return pair_list_seconds(pl, level, csr, R);
    const MomentSeconds t = moment_seconds(pl, csr, K, R);
    return t.eval + t.fixed;
}

template <int D, int K, int RB>
static void moment_impl(f3m_plan *pl, int level, const PairCSR *l1, const PairCSR *l2, double h, const float *bs, int R, int r0, float *out,
                        int rb, int re, cudaStream_t s) {
    Tree &tx = pl->tx, &ty = *pl->ty;
    Level &lx = tx.levels[level], &ly = ty.levels[level];
    // exp(-lcs v) = 2^(-s2 v).  Lengths are taken in a power of two near 1 / sqrt(s2), which rounds nothing, so that powers of
    // them up to the sixth neither overflow nor vanish whatever the caller's unit.
    const double s2_input = (double)pl->lcs * 1.4426950408889634;
    int ex;
    frexp(sqrt(s2_input), &ex);
    const float unit = (float)ldexp(1.0, ex), s2 = (float)ldexp(s2_input, -2 * ex);
    double cf[MOM_KMAX + 1];
    exp_poly_fit(h, K, cf);
    const double ln2 = 0.6931471805599453;
    double pw = 1.0;
    for (int k = 0; k <= K; k++) { cf[k] *= pw; pw *= ln2; }          // the records hold y 2 s2 = y / (l^2 ln 2) (l, y in that unit)
    MomFactors fac{};
    MomTree<D, K, 0, 0, 0>::factors(cf, 1.0, 0, fac.f);
    constexpr int CHUNK = 16384;
    const int chunk = ly.max_count > CHUNK ? CHUNK : 0;
    const int64_t groups = (int64_t)ly.nb * RB, slots = chunk ? part_slots(ty.n, chunk) : 0;
    DevBuf<float> rec, parts;
    rec.alloc((size_t)ly.nb * mom_record(D, K, RB), s);
    if (chunk) parts.alloc((size_t)slots * RB * mom_count(D, K), s);
    pl->last.begin(ST_DIRECT, s);
    const unsigned char *need = pl->shard.active && !pl->shard.all_sources ? pl->shard.need[level].p : nullptr;
    // a warp per box, unless the boxes are long or too few to fill the SMs (64 boxes of 312 points, K = 6: 13.5 -> 5.2 us with
    // a CTA per box; 512 boxes of 195 points, K = 3: 5.5 -> 6.8 us)
    if (ly.max_count <= 1024 && (groups >= 2 * NUM_SMS_HINT || ly.max_count <= 64))
        near_moments_build<D, K, RB, 32><<<(unsigned)((groups + 7) / 8), 256, 0, s>>>(ty.pts.p, (int)ty.n, bs, R, r0, unit, s2, ly.off.p, ly.nb,
                                                                                      ly.ctr.p, need, fac, 0, rec.p, nullptr);
    else
        near_moments_build<D, K, RB, 256><<<(unsigned)(groups + slots * RB), 256, 0, s>>>(ty.pts.p, (int)ty.n, bs, R, r0, unit, s2, ly.off.p, ly.nb,
                                                                                         ly.ctr.p, need, fac, chunk, rec.p, parts.p);
    F3M_LAUNCH_CHECK();
    if (chunk) {
        near_moments_combine<D, K, RB><<<(unsigned)(slots / 2), 128, 0, s>>>(unit, ly.off.p, ly.nb, (int)ty.n, ly.ctr.p, need, fac, chunk, parts.p,
                                                                            rec.p);
        F3M_LAUNCH_CHECK();
    }
    auto eval = [&](auto kernel, int G) {
        kernel<<<(unsigned)(((int64_t)(re - rb) * G + 127) / 128), 128, 0, s>>>(tx.pts.p, (int)tx.n, lx.off.p, lx.nb, rb, re, l1->ptr.p, l1->idx.p,
                                                                               l2 ? l2->ptr.p : nullptr, l2 ? l2->idx.p : nullptr, rec.p, unit, s2, R,
                                                                               r0, out);
    };
    if ((int64_t)(re - rb) >= 256 * NUM_SMS_HINT) eval(near_moments_eval<D, K, RB, 1>, 1);
    else eval(near_moments_eval<D, K, RB, 4>, 4);
    F3M_LAUNCH_CHECK();
    pl->last.end(s);
    pl->last.direct_launches++;
    pl->last.direct_variants[DV_MOMENTS]++;
    if (K == 2) pl->last.direct_variants[DV_POLY2]++;
    if (K == 3) pl->last.direct_variants[DV_POLY3]++;
}

template <int D, int K>
static void moment_columns(f3m_plan *pl, int level, const PairCSR *l1, const PairCSR *l2, double h, const float *bs, int R, float *out, int rb,
                           int re, cudaStream_t s) {
    for (int r0 = 0; r0 < R;) {
        if (R - r0 >= 2) { moment_impl<D, K, 4>(pl, level, l1, l2, h, bs, R, r0, out, rb, re, s); r0 += 4; }
        else { moment_impl<D, K, 1>(pl, level, l1, l2, h, bs, R, r0, out, rb, re, s); r0 += 1; }
    }
}

template <int D>
static void moment_degree(f3m_plan *pl, int level, int K, const PairCSR *l1, const PairCSR *l2, double h, const float *bs, int R, float *out,
                          int rb, int re, cudaStream_t s) {
    if (K == 2) return moment_columns<D, 2>(pl, level, l1, l2, h, bs, R, out, rb, re, s);
    if (K == 3) return moment_columns<D, 3>(pl, level, l1, l2, h, bs, R, out, rb, re, s);
    if constexpr (mom_kmax(D) >= 6) {
        if (K == 4) return moment_columns<D, 4>(pl, level, l1, l2, h, bs, R, out, rb, re, s);
        if (K == 5) return moment_columns<D, 5>(pl, level, l1, l2, h, bs, R, out, rb, re, s);
        return moment_columns<D, 6>(pl, level, l1, l2, h, bs, R, out, rb, re, s);
    }
}

// Sums the list through moments when its geometry allows; false: the caller sums the pairs.  On the last level the small
// list waits for the near list when both take this form: one set of records and one pass over the rows then serve both.
// alone: the level's other list is summed elsewhere (near_nodes.cu), neither waited for nor taken along.
bool moment_sums(f3m_plan *pl, int level, const PairCSR &csr, bool alone, const float *bs, int R, float *out, int rb, int re, cudaStream_t s) {
    if (level < 1) return false;
    LevelLists &ll = pl->lists[level];
    const bool keep = &csr == &ll.keep;
    int K = list_moment_degree(pl, level, keep, R);
    if (K == 0) return false;
    double h = list_exponent_bound(pl, level, keep);
    const PairCSR *other = nullptr;
    if (level == pl->levels && !alone) {
        const int Ko = list_moment_degree(pl, level, !keep, R);
        if (Ko) {
            if (!keep) return true;   // summed with the near list
            other = &ll.small;
            K = std::max(K, Ko);
            h = std::max(h, list_exponent_bound(pl, level, false));
        }
    }
    if (re <= rb) return true;
    switch (pl->d) {
        case 1: moment_degree<1>(pl, level, K, &csr, other, h, bs, R, out, rb, re, s); break;
        case 2: moment_degree<2>(pl, level, K, &csr, other, h, bs, R, out, rb, re, s); break;
        case 3: moment_degree<3>(pl, level, K, &csr, other, h, bs, R, out, rb, re, s); break;
        case 4: moment_degree<4>(pl, level, K, &csr, other, h, bs, R, out, rb, re, s); break;
        default: moment_degree<5>(pl, level, K, &csr, other, h, bs, R, out, rb, re, s); break;
    }
    return true;
}

}  // namespace f3m
