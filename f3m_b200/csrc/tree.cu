// Box division, second half (per-level boxes read off the sorted keys) and interaction lists.
//
// Replaces n_tree_cuda::divide (F3M_src/n_tree.cu:105-179), get_new_interactions (n_tree.cu:594-641),
// filter_out_interactions (n_tree.cu:788-811) and separate_interactions (n_tree.cu:701-787) with
// their kernels (F3M_src/1_d_conv.cu:903-1125).  The reference materialises all 4^d child pairs of
// every surviving pair, masks them three times and rebuilds CSR rows with sorts and hash tables; here
// one warp per target box walks its parent's row, classifies the child pairs in registers and writes
// the three lists directly as CSR rows (count pass, scan, write pass).  Box ids are dense ranks, so
// no hash table is needed anywhere.
#include <algorithm>
#include "common.cuh"

namespace f3m {

// ---------------------------------------------------------------------------------------------
// Boxes of a level = runs of equal key prefix in the sorted key array.  A point starts a box at level l and at
// every deeper level when its key differs from its predecessor's in a bit of level l or above, so ONE pass over
// the keys finds the box starts of a whole batch of levels: count per tile and level, scan per level over the
// tiles, write offsets and prefixes.
// ---------------------------------------------------------------------------------------------
constexpr int HT = 256, HI = 8, HTILE = HT * HI;
constexpr int HB = HEADS_BATCH;   // levels per batch

// coarsest level at which point i starts a box (lmax + 1: at none of the levels the key holds)
__device__ __forceinline__ int first_head_level(uint32_t key, uint32_t prev, bool first, int d, int lmax) {
    if (first) return 1;
    const uint32_t x = key ^ prev;
    if (!x) return lmax + 1;
    // bit h belongs to the d-bit group of level lmax - h / d; h < 32 and d <= 5, so h / d = (h * ceil(2^16 / d)) >> 16
    const int h = 31 - __clz(x);
    return lmax - ((h * ((65536 + d - 1) / d)) >> 16);
}

// the HI consecutive keys of a thread and the one before them
__device__ __forceinline__ void load_head_levels(const uint32_t *__restrict__ keys, int64_t n, int64_t base, int d, int lmax,
                                                 int (&l0)[8]) {
    uint32_t k[9];
    k[0] = (base > 0 && base - 1 < n) ? keys[base - 1] : 0u;
#pragma unroll
    for (int q = 0; q < 8; q++) k[q + 1] = (base + q < n) ? keys[base + q] : 0u;
#pragma unroll
    for (int q = 0; q < 8; q++) l0[q] = (base + q < n) ? first_head_level(k[q + 1], k[q], base + q == 0, d, lmax) : lmax + 1;
}

// part[v * nt + tile] = boxes of level l_first + v that start inside the tile
__global__ void __launch_bounds__(HT) heads_count(const uint32_t *__restrict__ keys, int64_t n, int d, int lmax, int l_first,
                                                 int nlev, int nt, int *part) {
    __shared__ int tot[HB];
    if (threadIdx.x < HB) tot[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * HTILE + (int64_t)threadIdx.x * HI;
    int l0[HI], c[HB];
    load_head_levels(keys, n, base, d, lmax, l0);
    int deepest = lmax + 1;
#pragma unroll
    for (int k = 0; k < HI; k++) deepest = min(deepest, l0[k]);
    // most warps hold no box start at any level of the batch (a box has hundreds of points)
    if (!__any_sync(0xffffffffu, deepest <= l_first + nlev - 1)) deepest = lmax + 1;
#pragma unroll
    for (int v = 0; v < HB; v++) c[v] = 0;
    if (deepest <= l_first + nlev - 1) {
#pragma unroll
        for (int k = 0; k < HI; k++)
#pragma unroll
            for (int v = 0; v < HB; v++) c[v] += (l0[k] <= l_first + v);
    }
#pragma unroll
    for (int v = 0; v < HB; v++) {
        if (v < nlev && __any_sync(0xffffffffu, c[v] > 0)) {
            int x = c[v];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if ((threadIdx.x & 31) == 0 && x) atomicAdd(&tot[v], x);
        }
    }
    __syncthreads();
    if (threadIdx.x < nlev) part[(size_t)threadIdx.x * nt + blockIdx.x] = tot[threadIdx.x];
}

// one block per level of the batch: exclusive scan of the level's tile counts, total -> totals[level]
__global__ void __launch_bounds__(1024) heads_scan(int *part, int nt, int *totals) {
    __shared__ int sm[33];
    int *row = part + (size_t)blockIdx.x * nt;
    int carry = 0;
    for (int base = 0; base < nt; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < nt ? row[i] : 0;
        int total;
        const int ex = block_exclusive_scan(v, &total, sm);
        if (i < nt) row[i] = ex + carry;
        carry += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

struct HeadsOut {
    int *off[HB];
    uint32_t *code[HB];
    int nb[HB];
};

__global__ void __launch_bounds__(HT) heads_write(const uint32_t *__restrict__ keys, int64_t n, int d, int lmax, int l_first,
                                                 int nlev, int nt, const int *__restrict__ part, HeadsOut out) {
    __shared__ int wtot[HB][HT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * HTILE + (int64_t)threadIdx.x * HI;
    int l0[HI], c[HB];
    load_head_levels(keys, n, base, d, lmax, l0);
#pragma unroll
    for (int v = 0; v < HB; v++) c[v] = 0;
#pragma unroll
    for (int k = 0; k < HI; k++)
#pragma unroll
        for (int v = 0; v < HB; v++) c[v] += (l0[k] <= l_first + v);
    int ex[HB];   // boxes of the level that start before this thread's keys, inside the warp
#pragma unroll
    for (int v = 0; v < HB; v++) {
        int inc = c[v];
        if (v < nlev && __any_sync(0xffffffffu, inc > 0)) {   // warp-uniform: most warps hold no box start
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
        }
        ex[v] = inc - c[v];
        if (lane == 31) wtot[v][w] = inc;
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < HB; v++) {
        if (v >= nlev || c[v] == 0) continue;
        int r = part[(size_t)v * nt + blockIdx.x] + ex[v];
        for (int ww = 0; ww < w; ww++) r += wtot[v][ww];
        const int shift = d * (lmax - (l_first + v));
#pragma unroll
        for (int k = 0; k < HI; k++)
            if (l0[k] <= l_first + v) {
                out.off[v][r] = (int)(base + k);
                out.code[v][r] = keys[base + k] >> shift;
                r++;
            }
        if (blockIdx.x == 0 && threadIdx.x == 0) out.off[v][out.nb[v]] = (int)n;
    }
}

// Parents, centres, first children and the largest box of all levels of a batch.  Entry v + 1 of the arrays is level l_first + v, entry 0
// the level above the batch.
struct LinkArgs {
    const int *off[HB + 1];
    const uint32_t *code[HB + 1];
    int *parent[HB + 1], *child_start[HB + 1];
    float *ctr[HB + 1];
    int nb[HB + 1];
    int l_first;
    float root[MAXD], edge0;
};
__device__ __forceinline__ int first_at_least(const int *__restrict__ v, int n, int target) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (v[mid] < target) lo = mid + 1; else hi = mid;
    }
    return lo;
}
template <int D>
__global__ void __launch_bounds__(256) level_links(LinkArgs a, int *maxcount, int *err) {
    const int v = blockIdx.y + 1, level = a.l_first + blockIdx.y, b = blockIdx.x * blockDim.x + threadIdx.x;
    const int nb = a.nb[v], nbp = a.nb[v - 1];
    if (blockIdx.x * blockDim.x > max(nb, nbp)) return;
    int cnt = 0;
    if (b < nb) {
        const uint32_t c = a.code[v][b], pc = c >> D;
        const uint32_t *pcode = a.code[v - 1];
        int lo = 0, hi = nbp;   // lower_bound of pc in pcode
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (pcode[mid] < pc) lo = mid + 1; else hi = mid;
        }
        if (lo >= nbp || pcode[lo] != pc) { atomicExch(err, 1); lo = 0; }
        a.parent[v][b] = lo;
        // natural_center_divide (n_tree.cu:98-104): centre = parent centre + (0.25*parent edge)*(+-1),
        // one float32 addition per coordinate and level, from the root down
#pragma unroll
        for (int k = 0; k < D; k++) {
            float x = a.root[k], edge = a.edge0;
            for (int j = 1; j <= level; j++) {
                const float quarter = 0.25f * edge;
                x = __fadd_rn(x, ((c >> (D * (level - j) + k)) & 1u) ? quarter : -quarter);
                edge *= 0.5f;
            }
            a.ctr[v][b * D + k] = x;
        }
        cnt = a.off[v][b + 1] - a.off[v][b];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, o));
    if ((threadIdx.x & 31) == 0 && cnt > 0) atomicMax(maxcount + blockIdx.y, cnt);
    // first child of parent b: the child whose point range starts where the parent's does
    if (b < nbp) a.child_start[v - 1][b] = first_at_least(a.off[v], nb, a.off[v - 1][b]);
    if (b == nbp) a.child_start[v - 1][b] = nb;
}

// The root's arrays come from kernel parameters: copies from host arrays would need a wait before those go out of scope.
struct RootValues {
    int n, d;
    float c[MAXD];
    int *off;
    uint32_t *code;
    int *parent;
    float *ctr;
};
__global__ void roots_kernel(RootValues x, RootValues y, int two, int *ptr, int *idx) {
    for (int t = 0; t <= two; t++) {
        const RootValues &v = t ? y : x;
        v.off[0] = 0;
        v.off[1] = v.n;
        v.code[0] = 0;
        v.parent[0] = 0;
        for (int k = 0; k < v.d; k++) v.ctr[k] = v.c[k];
    }
    ptr[0] = 0;
    ptr[1] = 1;
    idx[0] = 0;
}
static void root_centre(const Tree &t, float *c) {
    const float half = 0.5f * t.edge0;                       // exact
    for (int k = 0; k < t.d; k++) c[k] = t.origin[k] + half;   // n_tree.cu:93, float32 add
}
static RootValues make_root(Tree &t, cudaStream_t s) {
    t.levels.clear();
    t.levels.emplace_back();
    Level &L = t.levels.back();
    L.nb = 1;
    L.edge = t.edge0;
    L.max_count = (int)t.n;
    L.off.alloc(2, s); L.code.alloc(1, s); L.parent.alloc(1, s); L.ctr.alloc(t.d, s);
    RootValues v{(int)t.n, t.d, {0}, L.off.p, L.code.p, L.parent.p, L.ctr.p};
    root_centre(t, v.c);
    return v;
}
void build_roots(f3m_plan *pl, cudaStream_t s) {
    const RootValues x = make_root(pl->tx, s), y = pl->same ? x : make_root(*pl->ty, s);
    pl->lists.clear();
    pl->lists.emplace_back();
    PairCSR &k = pl->lists[0].keep;
    k.ptr.alloc(2, s); k.idx.alloc(1, s);
    roots_kernel<<<1, 1, 0, s>>>(x, y, !pl->same, k.ptr.p, k.idx.p);
    F3M_LAUNCH_CHECK();
    k.count = 1;
}

__global__ void __launch_bounds__(256) remap_offsets_kernel(int count, int *off, const int *__restrict__ fine_off) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) off[i] = fine_off[off[i]];
}

// A tree that waits for its sorted runs: one pseudo key per occupied finest cell stands for the cell's points, and the box starts found
// among them are translated into offsets of the merged order.
static const uint32_t *head_keys(const Tree &t) { return t.runs.pending ? t.runs.pkeys.p : t.keys.p; }
static int64_t head_count(const Tree &t) { return t.runs.pending ? t.runs.nocc : t.n; }

void heads_begin(Tree &t, HeadsBatch &hb, int l_first, int l_last, int *d_tot, cudaStream_t s) {
    F3M_REQUIRE(l_last <= t.sorted_depth, F3M_ERR_INTERNAL, "level %d requested, keys are sorted to level %d", l_last, t.sorted_depth);
    const int64_t n = head_count(t);
    hb.l_first = l_first;
    hb.nlev = std::min(HB, l_last - l_first + 1);
    hb.nt = (int)((n + HTILE - 1) / HTILE);
    hb.part.alloc((size_t)hb.nlev * hb.nt, s);
    heads_count<<<hb.nt, HT, 0, s>>>(head_keys(t), n, t.d, t.lmax, l_first, hb.nlev, hb.nt, hb.part.p);
    F3M_LAUNCH_CHECK();
    heads_scan<<<hb.nlev, 1024, 0, s>>>(hb.part.p, hb.nt, d_tot);
    F3M_LAUNCH_CHECK();
}

// h_tot: the boxes of the batch's levels, on the host; the levels' largest boxes are left at d_max (zero before)
void heads_finish(Tree &t, HeadsBatch &hb, const int *h_tot, int *d_max, int *d_err, cudaStream_t s) {
    HeadsOut ho{};
    LinkArgs la{};
    int most = 0;
    for (int v = -1; v < hb.nlev; v++) {
        if (v >= 0) {
            t.levels.emplace_back();
            Level &L = t.levels.back();
            L.nb = h_tot[v];
            L.edge = t.levels[hb.l_first + v - 1].edge * 0.5f;
            L.off.alloc((size_t)L.nb + 1, s); L.code.alloc(L.nb, s); L.parent.alloc(L.nb, s); L.ctr.alloc((size_t)L.nb * t.d, s);
            ho.off[v] = L.off.p; ho.code[v] = L.code.p; ho.nb[v] = L.nb;
        }
        Level &L = t.levels[hb.l_first + v];
        if (v < hb.nlev - 1) L.child_start.alloc((size_t)L.nb + 1, s);
        la.off[v + 1] = L.off.p; la.code[v + 1] = L.code.p; la.parent[v + 1] = L.parent.p; la.ctr[v + 1] = L.ctr.p;
        la.child_start[v + 1] = L.child_start.p;
        la.nb[v + 1] = L.nb;
        most = std::max(most, L.nb);
    }
    const int64_t n = head_count(t);
    heads_write<<<hb.nt, HT, 0, s>>>(head_keys(t), n, t.d, t.lmax, hb.l_first, hb.nlev, hb.nt, hb.part.p, ho);
    F3M_LAUNCH_CHECK();
    if (t.runs.pending)
        for (int v = 0; v < hb.nlev; v++) {
            remap_offsets_kernel<<<(unsigned)((ho.nb[v] + 1 + 255) / 256), 256, 0, s>>>(ho.nb[v] + 1, ho.off[v], t.runs.fine_off.p);
            F3M_LAUNCH_CHECK();
        }
    la.l_first = hb.l_first;
    la.edge0 = t.edge0;
    root_centre(t, la.root);
    const dim3 g((unsigned)(most / 256 + 1), hb.nlev);
    switch (t.d) {
        case 1: level_links<1><<<g, 256, 0, s>>>(la, d_max, d_err); break;
        case 2: level_links<2><<<g, 256, 0, s>>>(la, d_max, d_err); break;
        case 3: level_links<3><<<g, 256, 0, s>>>(la, d_max, d_err); break;
        case 4: level_links<4><<<g, 256, 0, s>>>(la, d_max, d_err); break;
        default: level_links<5><<<g, 256, 0, s>>>(la, d_max, d_err); break;
    }
    F3M_LAUNCH_CHECK();
    hb.part.release();
}

// Appends the levels after the last one built, up to l_last, in batches: two host synchronisations per batch (box counts before the
// arrays are sized, largest boxes after the links).
void build_levels(Tree &t, int l_last, f3m_plan *pl, cudaStream_t s) {
    int *d_err = pl->d_flags + FL_ERR, *d_tot = pl->d_flags + FL_LVTOT, *d_max = pl->d_flags + FL_LVMAX;
    while ((int)t.levels.size() <= l_last) {
        HeadsBatch hb;
        heads_begin(t, hb, (int)t.levels.size(), l_last, d_tot, s);
        F3M_CUDA(cudaMemcpyAsync(pl->h_pinned + FL_LVTOT, d_tot, hb.nlev * sizeof(int), cudaMemcpyDeviceToHost, s));
        F3M_CUDA(cudaMemsetAsync(d_max, 0, hb.nlev * sizeof(int), s));
        F3M_CUDA(cudaStreamSynchronize(s));
        heads_finish(t, hb, pl->h_pinned + FL_LVTOT, d_max, d_err, s);
        F3M_CUDA(cudaMemcpyAsync(pl->h_pinned + FL_LVMAX, d_max, hb.nlev * sizeof(int), cudaMemcpyDeviceToHost, s));
        F3M_CUDA(cudaMemcpyAsync(pl->h_pinned + FL_ERR, d_err, sizeof(int), cudaMemcpyDeviceToHost, s));
        F3M_CUDA(cudaStreamSynchronize(s));
        F3M_REQUIRE(pl->h_pinned[FL_ERR] == 0, F3M_ERR_INTERNAL, "a box of levels %d..%d has no parent one level up", hb.l_first,
                    hb.l_first + hb.nlev - 1);
        for (int v = 0; v < hb.nlev; v++) t.levels[hb.l_first + v].max_count = pl->h_pinned[FL_LVMAX + v];
    }
}

// ---------------------------------------------------------------------------------------------
// interaction lists
// ---------------------------------------------------------------------------------------------
struct ClassifyParams {
    int two_p;          // 2 * interpolation nodes
    int two_small;      // 2 * small_field_points
    float edge2;        // 2 * box edge
    int do_init;        // n_tree.cu:729-734
    int var_comp;
    int enable_pair, enable_all;   // n_tree.cu:738-739
    float crit, lcs;               // n_tree.cu:740
    int ieee;
};
enum { CLS_KEEP = 0, CLS_FAR = 1, CLS_SMALL = 2, CLS_DROP = 3 };

// boolean_separate_interactions_small / _var_comp (1_d_conv.cu:903-1029), same order of tests
template <int D>
__device__ __forceinline__ int classify(int size, const float *cx, const float *cy, const ClassifyParams &cp) {
    if (cp.do_init && size < cp.two_p) return CLS_SMALL;
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < D; k++) {
        float dk = __fsub_rn(cy[k], cx[k]);
        acc = cp.ieee ? __fadd_rn(acc, __fmul_rn(dk, dk)) : __fmaf_rn(dk, dk, acc);
    }
    float nrm;
    if (cp.ieee) nrm = __fsqrt_rn(acc);
    else asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(nrm) : "f"(acc));
    if (nrm >= cp.edge2) return cp.do_init ? CLS_FAR : CLS_DROP;
    if (cp.var_comp) {
        if (cp.enable_pair && (double)__fmul_rn(__fmul_rn(nrm, nrm), cp.lcs) <= 1e-2) return CLS_FAR;
        if (cp.enable_all && nrm <= cp.crit) return CLS_FAR;
    }
    if (size < cp.two_small) return CLS_SMALL;
    return CLS_KEEP;
}

// What the lists' sums cost, pairs of points and (target point, source box) pairs of the small and of the kept list: summed by the warps
// that write the lists, one set of atomics per block.
struct ListRoom { int far, small, keep; };
// One warp per target box of the new level, boxes in turn.  pass 0: count per class; pass 1: write source ids.
template <int D>
__global__ void __launch_bounds__(256) lists_kernel(int pass, int nbx, const int *__restrict__ parent_x,
                                                   const int *__restrict__ kptr, const int *__restrict__ kidx,
                                                   const int *__restrict__ cs_y, const int *__restrict__ off_x,
                                                   const int *__restrict__ off_y, const float *__restrict__ ctr_x,
                                                   const float *__restrict__ ctr_y, ClassifyParams cp, int *far_ptr,
                                                   int *small_ptr, int *keep_ptr, int *far_idx, int *small_idx,
                                                   int *keep_idx, ListRoom room, unsigned long long *work, int *over) {
    constexpr int NCH = 1 << D;
    constexpr int EPW = 32 / NCH;
    const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    const unsigned lt = (1u << lane) - 1;
    const int sub = lane / NCH, ch = lane % NCH;
    long long sums[4] = {0, 0, 0, 0};
    const bool cut_short = *over != 0;   // the kept list of the level above is incomplete: this level's lists stay empty
    if (cut_short && pass == 1) return;
    for (int box = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; box < nbx; box += warps) {
        const int px = parent_x[box];
        const int e0 = kptr[px], e1 = cut_short ? e0 : kptr[px + 1];
        const int nx = off_x[box + 1] - off_x[box];
        float cx[D];
#pragma unroll
        for (int k = 0; k < D; k++) cx[k] = ctr_x[box * D + k];
        int nf = 0, ns = 0, nk = 0;
        if (pass == 1) { nf = far_ptr[box]; ns = small_ptr[box]; nk = keep_ptr[box]; }
        const int ns0 = ns, nk0 = nk;
        int y_small = 0, y_keep = 0;   // points of the listed source boxes, this lane's share
        for (int it = e0; it < e1; it += EPW) {
            int e = it + sub;
            int cls = -1, by = 0, ny = 0;
            if (e < e1) {
                int py = kidx[e];
                int c0 = cs_y[py], c1 = cs_y[py + 1];
                by = c0 + ch;
                if (by < c1) {
                    float cy[D];
#pragma unroll
                    for (int k = 0; k < D; k++) cy[k] = ctr_y[by * D + k];
                    ny = off_y[by + 1] - off_y[by];
                    cls = classify<D>(nx + ny, cx, cy, cp);
                }
            }
            unsigned mf = __ballot_sync(0xffffffffu, cls == CLS_FAR);
            unsigned ms = __ballot_sync(0xffffffffu, cls == CLS_SMALL);
            unsigned mk = __ballot_sync(0xffffffffu, cls == CLS_KEEP);
            if (pass == 1) {
                if (cls == CLS_FAR && nf + __popc(mf & lt) < room.far) far_idx[nf + __popc(mf & lt)] = by;
                if (cls == CLS_SMALL && ns + __popc(ms & lt) < room.small) small_idx[ns + __popc(ms & lt)] = by;
                if (cls == CLS_KEEP && nk + __popc(mk & lt) < room.keep) keep_idx[nk + __popc(mk & lt)] = by;
                if (cls == CLS_SMALL) y_small += ny;
                if (cls == CLS_KEEP) y_keep += ny;
            }
            nf += __popc(mf); ns += __popc(ms); nk += __popc(mk);
        }
        if (pass == 0) {
            if (lane == 0) {
                far_ptr[box] = nf; small_ptr[box] = ns; keep_ptr[box] = nk;
                if (box == nbx - 1) far_ptr[nbx] = small_ptr[nbx] = keep_ptr[nbx] = 0;   // the scan makes totals of them
            }
        } else {
            sums[0] += (long long)y_small * nx;
            sums[2] += (long long)y_keep * nx;
            if (lane == 0) {
                sums[1] += (long long)(ns - ns0) * nx;
                sums[3] += (long long)(nk - nk0) * nx;
                if (nf > room.far || ns > room.small || nk > room.keep) atomicExch(over, 1);
            }
        }
    }
    if (pass == 0) return;
    __shared__ long long block_sums[8][4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sums[q] += __shfl_xor_sync(0xffffffffu, sums[q], o);
        if (lane == 0) block_sums[threadIdx.x >> 5][q] = sums[q];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        long long v = 0;
        for (int w = 0; w < 8; w++) v += block_sums[w][threadIdx.x];
        if (v) atomicAdd(work + threadIdx.x, (unsigned long long)v);
    }
}

static ClassifyParams classify_params(const f3m_plan *pl, int level) {
    const Level &lx = pl->tx.levels[level];
    const f3m_params &prm = pl->prm;
    const int d = pl->d;
    ClassifyParams cp{};
    cp.two_p = 2 * prm.nr_interpolation;
    cp.two_small = 2 * prm.small_field_points;
    cp.edge2 = lx.edge * 2.f;
    cp.ieee = prm.math_mode == F3M_MATH_IEEE;
    cp.var_comp = prm.var_compression != 0;
    cp.lcs = pl->lcs;
    float square_edge = lx.edge * lx.edge * pl->lcs;          // n_tree.cu:728
    cp.do_init = cp.var_comp ? (square_edge <= 5) : 1;
    if (cp.var_comp) {
        cp.enable_pair = (d * square_edge / 4) <= prm.eff_var_limit;
        cp.enable_all = (d * square_edge / 4) <= (prm.eff_var_limit / 2);
        cp.crit = sqrtf(prm.eff_var_limit * 2 / (d * pl->lcs));
    }
    return cp;
}

static void run_lists(f3m_plan *pl, int level, int pass, const ListRoom &room, cudaStream_t s) {
    Tree &tx = pl->tx, &ty = *pl->ty;
    Level &lx = tx.levels[level], &ly = ty.levels[level], &py = ty.levels[level - 1];
    LevelLists &prev = pl->lists[level - 1], &cur = pl->lists[level];
    const ClassifyParams cp = classify_params(pl, level);
    const int64_t blocks = ((int64_t)lx.nb * 32 + 255) / 256;
    // the sums of pass 1 end in four atomics per block: few blocks, many boxes each
    const unsigned grid = (unsigned)(pass ? std::min<int64_t>(blocks, NUM_SMS_HINT * 16) : blocks);
    unsigned long long *work = reinterpret_cast<unsigned long long *>(pl->d_flags + FL_PAIRWORK) + 4 * level;
    auto run = [&](auto kernel) {
        kernel<<<grid, 256, 0, s>>>(pass, lx.nb, lx.parent.p, prev.keep.ptr.p, prev.keep.idx.p, py.child_start.p, lx.off.p, ly.off.p, lx.ctr.p,
                                    ly.ctr.p, cp, cur.far.ptr.p, cur.small.ptr.p, cur.keep.ptr.p, cur.far.idx.p, cur.small.idx.p,
                                    cur.keep.idx.p, room, work, pl->d_flags + FL_LISTOVER);
    };
    switch (pl->d) {
        case 1: run(lists_kernel<1>); break;
        case 2: run(lists_kernel<2>); break;
        case 3: run(lists_kernel<3>); break;
        case 4: run(lists_kernel<4>); break;
        default: run(lists_kernel<5>); break;
    }
    F3M_LAUNCH_CHECK();
}

void lists_count(f3m_plan *pl, int level, cudaStream_t s) {
    LevelLists &cur = pl->lists[level];
    const int nbx = pl->tx.levels[level].nb;
    cur.far.ptr.alloc((size_t)nbx + 1, s); cur.small.ptr.alloc((size_t)nbx + 1, s); cur.keep.ptr.alloc((size_t)nbx + 1, s);
    run_lists(pl, level, 0, ListRoom{0, 0, 0}, s);
    int *ptrs[3] = {cur.far.ptr.p, cur.small.ptr.p, cur.keep.ptr.p};
    exclusive_scan_multi(ptrs, 3, (int64_t)nbx + 1, reinterpret_cast<long long *>(pl->d_flags + FL_LISTS) + 3 * level, s);
}

void lists_write(f3m_plan *pl, int level, const int64_t cap[3], cudaStream_t s) {
    LevelLists &cur = pl->lists[level];
    cur.far.idx.alloc((size_t)cap[0], s); cur.small.idx.alloc((size_t)cap[1], s); cur.keep.idx.alloc((size_t)cap[2], s);
    run_lists(pl, level, 1, ListRoom{(int)cap[0], (int)cap[1], (int)cap[2]}, s);
}

}  // namespace f3m
