// Exact dense Gaussian products.
//
// Replaces rbf_call / rbf_call_grad (F3M_src/n_tree.cu:185-241) with rbf_1d_reduce_shared_torch(_grad)
// (F3M_src/1_d_conv.cu:126-214).
#include <math.h>
#include <algorithm>
#include "common.cuh"
#include "packed.cuh"

namespace f3m {

// A pair costs d differences, d multiply-adds, one exponential and RB multiply-adds (one more multiply for the gradient):
// FP32 lanes (128 per clock and SM) and the exponential unit (16) are the limit, not memory.  The coordinates are
// subtracted before they are squared: the product has no box centres to expand about, and the expanded form would lose
// the digits that two distant points share.
//   * Two SOURCES share every instruction (f32x2); a source pair is laid out column by column in shared memory, so one
//     16-byte broadcast load yields two packed operands, and each thread holds DT = 2 targets to halve the loads.
//   * A CTA takes DTILE = 256 targets and one SLICE of the sources, straight from the caller's rows.  With one CTA per
//     target tile a call of 2e4 points ran 157 four-warp CTAs on 148 SMs: most of the chip idle, then a second, nearly empty wave.
//     The slices' partial sums are added in a fixed order by dense_combine, so results do not depend on scheduling.
// Measured, product + gradient of 2e4 points, d = 3, 3 columns: 1280 -> 358 us on the device (171 + 181, floor 87 + 98 at nine and ten
// FP32 lanes a pair); error against float64 5.4e-7 -> 3.1e-7.  With four source pairs in flight per thread and registers for them (six CTAs
// per SM) instead of two (eight): 169 + 181 -> 160 + 168 us, the two calls 397 -> 373; one column of 2e4 points 120 -> 114, five dimensions
// and 3 columns 212 -> 201; eight columns in three dimensions gain nothing and stay at two.
constexpr int DNT = 128, DT = 2, DTILE = DNT * DT;
constexpr int DST = 256;   // sources per shared-memory tile; also the length of the blocked partial sums

// columns of a source pair in shared memory: minus the scaled coordinates, then the RB values; even, for 16-byte loads
__host__ __device__ constexpr int dense_width(int D, int RB) { return (D + RB + 1) / 2 * 2; }

// dst: the product itself (stride R, column r0) when there is one slice, else partial sums (slices, N, RB)
template <int D, int RB, bool GRAD>
__global__ void __launch_bounds__(DNT, RB <= 4 ? 6 : 4) dense_kernel(const float *__restrict__ X, int64_t n, const float *__restrict__ Y,
                                                                     const float *__restrict__ b, int64_t m, int64_t slice, float scale,
                                                                     float post, int R, int r0, float *dst) {
    constexpr int W = dense_width(D, RB), UNROLL = RB <= 4 || D >= 4 ? 4 : 2;
    __shared__ __align__(16) float smem[DST * W];
    const int64_t i0 = (int64_t)blockIdx.x * DTILE + threadIdx.x;
    const int64_t m0 = (int64_t)blockIdx.y * slice, m1 = min(m, m0 + slice);
    f32x2 x[DT][D];
    float tot[DT][RB];
#pragma unroll
    for (int u = 0; u < DT; u++) {
        const int64_t i = i0 + u * DNT, ii = i < n ? i : n - 1;
#pragma unroll
        for (int k = 0; k < D; k++) {
            const float v = scale * X[ii * D + k];
            x[u][k] = pack2(v, v);
        }
#pragma unroll
        for (int r = 0; r < RB; r++) tot[u][r] = 0.f;
    }
    for (int64_t base = m0; base < m1; base += DST) {
        const int cnt = (int)min((int64_t)DST, m1 - base), np = (cnt + 1) >> 1;
        __syncthreads();
        // row j of the tile -> half (j & 1) of pair j / 2; an odd tile's partner has weight 0 and the last source's place, so that
        // its distances are no larger than the sources' own
        for (int q = threadIdx.x; q < 2 * np * D; q += DNT) {
            const int j = q / D, k = q - j * D;
            smem[(j >> 1) * 2 * W + 2 * k + (j & 1)] = -scale * Y[base * D + (j < cnt ? q : q - D)];
        }
        for (int q = threadIdx.x; q < 2 * np * (W - D); q += DNT) {
            const int j = q / (W - D), r = q - j * (W - D);
            smem[(j >> 1) * 2 * W + 2 * (D + r) + (j & 1)] = (j < cnt && r < RB && r0 + r < R) ? b[(base + j) * R + r0 + r] : 0.f;
        }
        __syncthreads();
        f32x2 acc[DT][RB];
#pragma unroll
        for (int u = 0; u < DT; u++)
#pragma unroll
            for (int r = 0; r < RB; r++) acc[u][r] = pack2(0.f, 0.f);
#pragma unroll UNROLL
        for (int p = 0; p < np; p++) {
            f32x2 col[W];
            const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(smem + p * 2 * W);
#pragma unroll
            for (int q = 0; q < W / 2; q++) {
                const ulonglong2 v = src[q];
                col[2 * q] = v.x;
                col[2 * q + 1] = v.y;
            }
#pragma unroll
            for (int u = 0; u < DT; u++) {
                f32x2 df = add2(x[u][0], col[0]);
                f32x2 r2 = mul2(df, df);
#pragma unroll
                for (int k = 1; k < D; k++) {
                    df = add2(x[u][k], col[k]);
                    r2 = fma2(df, df, r2);
                }
                float ra, rb;
                unpack2(r2, ra, rb);
                f32x2 e = pack2(ex2_approx(-ra), ex2_approx(-rb));
                if (GRAD) e = mul2(e, r2);
#pragma unroll
                for (int r = 0; r < RB; r++) acc[u][r] = fma2(e, col[D + r], acc[u][r]);
            }
        }
#pragma unroll
        for (int u = 0; u < DT; u++)
#pragma unroll
            for (int r = 0; r < RB; r++) {   // blocked accumulation: one partial sum per tile
                float lo, hi;
                unpack2(acc[u][r], lo, hi);
                tot[u][r] += lo + hi;
            }
    }
#pragma unroll
    for (int u = 0; u < DT; u++) {
        const int64_t i = i0 + u * DNT;
        if (i >= n) continue;
#pragma unroll
        for (int r = 0; r < RB; r++) {
            if (gridDim.y > 1) dst[((int64_t)blockIdx.y * n + i) * RB + r] = tot[u][r];
            else if (r0 + r < R) dst[i * R + r0 + r] = tot[u][r] * post;
        }
    }
}

__global__ void __launch_bounds__(256) dense_combine(const float *__restrict__ part, int64_t n, int RB, int nslice, float post, int R, int r0,
                                                    float *out) {
    const int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (q >= n * RB) return;
    const int64_t i = q / RB;
    const int r = (int)(q - i * RB);
    if (r0 + r >= R) return;
    float v = 0.f;
#pragma unroll 4
    for (int s = 0; s < nslice; s++) v += part[(int64_t)s * n * RB + q];
    out[i * R + r0 + r] = v * post;
}

// Slices of the sources.  An SM works through ceil(CTAs / SMs) CTAs of slice + DENSE_FIXED source rows each (DENSE_FIXED: what
// a CTA spends outside the pair loop, in rows); below four resident CTAs it waits for latencies, so fewer count as four.  The
// smallest product wins, and the fewest slices among equals -- among partial sums of at most DENSE_FREE_FLOATS; larger ones have to
// gain DENSE_GAIN: a product of many targets gains nothing from slices that take memory (1.8e6 targets, 8 columns: 510 MB for
// 0.5 %).  max_floats bounds the partial sums.
constexpr int64_t DENSE_FIXED = 48, DENSE_MAX_SLICES = 64;
constexpr int64_t DENSE_FREE_FLOATS = (int64_t)1 << 22;   // 16 MB
constexpr double DENSE_GAIN = 1.02;
static int dense_slices(int64_t n, int64_t m, int RB, int64_t max_floats) {
    const int64_t tiles = (n + DTILE - 1) / DTILE;
    int best = 1;
    double best_cost = 0.0;
    for (int64_t s = 1; s <= DENSE_MAX_SLICES; s++) {
        if (s > 1 && (m / s < 32 || s * n * RB > max_floats)) break;
        const int64_t len = (((m + s - 1) / s) + 1) & ~(int64_t)1;
        const double cost = (double)std::max<int64_t>((tiles * s + NUM_SMS_HINT - 1) / NUM_SMS_HINT, 4) * (double)(len + DENSE_FIXED);
        const double gain = s * n * RB <= DENSE_FREE_FLOATS ? 1.0 : DENSE_GAIN;
        if (s == 1 || cost * gain < best_cost) { best = (int)s; best_cost = cost; }
    }
    return best;
}

template <int D, int RB, bool GRAD>
static void dense_block(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, int r0, float scale, float post, float *out,
                        float *scratch, int64_t max_floats, cudaStream_t s) {
    const int want = dense_slices(N, M, RB, max_floats);
    int64_t slice = (((M + want - 1) / want) + 1) & ~(int64_t)1;
    int ns = (int)((M + slice - 1) / slice);
    DevBuf<float> part;
    if (ns > 1 && !scratch) {
        try {
            part.alloc((size_t)ns * N * RB, s);
            scratch = part.p;
        } catch (const Fail &) {   // no memory left for partial sums: the product does without
            (void)cudaGetLastError();
            slice = (M + 1) & ~(int64_t)1;
            ns = 1;
        }
    }
    const dim3 grid((unsigned)((N + DTILE - 1) / DTILE), (unsigned)ns);
    dense_kernel<D, RB, GRAD><<<grid, DNT, 0, s>>>(X, N, Y, b, M, slice, scale, post, R, r0, ns > 1 ? scratch : out);
    F3M_LAUNCH_CHECK();
    if (ns > 1) {
        dense_combine<<<(unsigned)((N * RB + 255) / 256), 256, 0, s>>>(scratch, N, RB, ns, post, R, r0, out);
        F3M_LAUNCH_CHECK();
    }
}

template <int D, bool GRAD>
static void dense_d(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, float ls, float *out, float *scratch,
                    int64_t max_floats, cudaStream_t s) {
    const float lcs = 1.f / (2.f * ls * ls);
    const float scale = sqrtf(lcs * 1.4426950408889634f);
    // GRAD: sum r^2 exp(..) b / ls^3 with r^2 = (scaled r^2) / scale^2   (n_tree.cu:222-239)
    const float post = GRAD ? 1.f / (scale * scale) / (ls * ls * ls) : 1.f;
    for (int r0 = 0; r0 < R;) {
        const int left = R - r0;   // 5 to 7 columns: one block of 8 repeats no exponential
        if (left >= 5) { dense_block<D, 8, GRAD>(X, N, Y, M, b, R, r0, scale, post, out, scratch, max_floats, s); r0 += 8; }
        else if (left == 4) { dense_block<D, 4, GRAD>(X, N, Y, M, b, R, r0, scale, post, out, scratch, max_floats, s); r0 += 4; }
        else if (left == 3) { dense_block<D, 3, GRAD>(X, N, Y, M, b, R, r0, scale, post, out, scratch, max_floats, s); r0 += 3; }
        else if (left == 2) { dense_block<D, 2, GRAD>(X, N, Y, M, b, R, r0, scale, post, out, scratch, max_floats, s); r0 += 2; }
        else { dense_block<D, 1, GRAD>(X, N, Y, M, b, R, r0, scale, post, out, scratch, max_floats, s); r0 += 1; }
    }
}

template <bool GRAD>
static void dense_any(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, int d, float ls, float *out, float *scratch,
                      int64_t max_floats, cudaStream_t s) {
    switch (d) {
        case 1: dense_d<1, GRAD>(X, N, Y, M, b, R, ls, out, scratch, max_floats, s); break;
        case 2: dense_d<2, GRAD>(X, N, Y, M, b, R, ls, out, scratch, max_floats, s); break;
        case 3: dense_d<3, GRAD>(X, N, Y, M, b, R, ls, out, scratch, max_floats, s); break;
        case 4: dense_d<4, GRAD>(X, N, Y, M, b, R, ls, out, scratch, max_floats, s); break;
        default: dense_d<5, GRAD>(X, N, Y, M, b, R, ls, out, scratch, max_floats, s); break;
    }
}

// the partial sums of a call stay below 512 MB
constexpr int64_t DENSE_PART_FLOATS = (int64_t)1 << 27;

template <bool GRAD>
void dense_f32(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, int d, float ls, float *out,
               cudaStream_t s) {
    dense_any<GRAD>(X, N, Y, M, b, R, d, ls, out, nullptr, DENSE_PART_FLOATS, s);
}
template void dense_f32<false>(const float *, int64_t, const float *, int64_t, const float *, int, int, float, float *, cudaStream_t);
template void dense_f32<true>(const float *, int64_t, const float *, int64_t, const float *, int, int, float, float *, cudaStream_t);

// float64 dense product with a double-precision exponential (accuracy reference on the device).
// grid.y slices the sources so that a few thousand target rows still fill the GPU; slices are combined
// with double atomics into a zeroed output.
__global__ void __launch_bounds__(128) dense_f64_kernel(const double *__restrict__ X, int64_t n, const double *__restrict__ Y,
                                                       int64_t m, const double *__restrict__ b, int R, int d, double lcs,
                                                       double *out) {
    __shared__ double sy[128 * F3M_MAX_DIM];
    const int64_t i = (int64_t)blockIdx.x * 128 + threadIdx.x;
    const int64_t per = (m + gridDim.y - 1) / gridDim.y;
    const int64_t m0 = (int64_t)blockIdx.y * per, m1 = min(m, m0 + per);
    double xi[F3M_MAX_DIM];
    for (int k = 0; k < d; k++) xi[k] = X[(i < n ? i : n - 1) * d + k];
    for (int r = 0; r < R; r++) {
        double acc = 0.;
        for (int64_t base = m0; base < m1; base += 128) {
            int cnt = (int)min((int64_t)128, m1 - base);
            __syncthreads();
            for (int q = threadIdx.x; q < cnt * d; q += 128) sy[q] = Y[base * d + q];
            __syncthreads();
            for (int j = 0; j < cnt; j++) {
                double r2 = 0.;
                for (int k = 0; k < d; k++) { double dk = xi[k] - sy[j * d + k]; r2 += dk * dk; }
                acc += exp(-r2 * lcs) * b[(base + j) * R + r];
            }
        }
        if (i < n) atomicAdd(&out[i * R + r], acc);
    }
}

void dense_f64(const double *X, int64_t N, const double *Y, int64_t M, const double *b, int R, int d, double ls, double *out,
               cudaStream_t s) {
    F3M_CUDA(cudaMemsetAsync(out, 0, (size_t)N * R * sizeof(double), s));
    const unsigned gx = (unsigned)((N + 127) / 128);
    int64_t want = (int64_t)NUM_SMS_HINT * 16 / gx;
    unsigned gy = (unsigned)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, (M + 4095) / 4096), 4096));
    dense_f64_kernel<<<dim3(gx, gy), 128, 0, s>>>(X, N, Y, M, b, R, d, 1.0 / (2.0 * ls * ls), out);
    F3M_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------------------------
// Exact dense product without any allocation.
//
// Some hosts may not touch the CUDA allocator once they are running: a service that handed all device
// memory to its own pool at start-up, or a control loop with a "no allocation after initialisation"
// rule, because an allocation can stall the whole device.  For them f3m_rbf_dense_f32_static computes
// the same product as f3m_rbf_dense_f32 with its only scratch buffer -- the partial sums of the source slices -- in a
// fixed array that is part of the library image.  Every GPU that loads libf3m.so holds this array
// (F3M_STATIC_SCRATCH_FLOATS floats = 16 MiB) until the process exits.
//
// In host code the array's name is only a stand-in, not a device address; the address a kernel can use
// is obtained once per device, with that device current, through cudaGetSymbolAddress.  The first call
// on a device performs this look-up, so make that first call before any stream capture starts.
// All calls share the one array: it keeps whatever the previous call left (every value a call reads is
// written by that call first, so nothing has to be cleared), and two calls that overlap on the GPU
// -- different streams, or different host threads -- race on it.
// ---------------------------------------------------------------------------------------------
static __device__ __align__(256) float g_static_scratch[F3M_STATIC_SCRATCH_FLOATS];

static float *static_scratch_for_current_device() {
    static std::atomic<float *> ptr_of_device[64];   // zero-initialised; two threads may both look the address up, both get the same
    int dev = 0;
    F3M_CUDA(cudaGetDevice(&dev));
    F3M_REQUIRE(dev >= 0 && dev < 64, F3M_ERR_UNSUPPORTED, "device ordinal %d not supported by the static entry point", dev);
    float *p = ptr_of_device[dev].load(std::memory_order_acquire);
    if (!p) {
        F3M_CUDA(cudaGetSymbolAddress((void **)&p, g_static_scratch));
        ptr_of_device[dev].store(p, std::memory_order_release);
    }
    return p;
}

// The capacity of this entry point is stated in floats of source rows of (d + columns) padded to four, as its callers know it.
void dense_f32_static(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, int d, float ls, float *out,
                      cudaStream_t s) {
    const int64_t width = (d + (R >= 2 ? 4 : 1) + 3) / 4 * 4;
    F3M_REQUIRE(M * width <= (int64_t)F3M_STATIC_SCRATCH_FLOATS, F3M_ERR_TOO_LARGE,
                "f3m_rbf_dense_f32_static holds %lld packed floats; M=%lld sources of %lld floats each need %lld "
                "(use f3m_rbf_dense_f32, which allocates)",
                (long long)F3M_STATIC_SCRATCH_FLOATS, (long long)M, (long long)width, (long long)(M * width));
    dense_any<false>(X, N, Y, M, b, R, d, ls, out, static_scratch_for_current_device(), F3M_STATIC_SCRATCH_FLOATS, s);
}

}  // namespace f3m
