// Internal declarations shared by the translation units of libf3m.so.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <atomic>
#include <vector>
#include "f3m.h"

namespace f3m {

constexpr int MAXD = F3M_MAX_DIM;
constexpr int MAXP = 64;   // interpolation nodes per dimension the kernels hold
constexpr int NUM_SMS_HINT = 148;

// ---- error handling: every CUDA call is checked, the message is kept per thread --------------
void set_error(const char *fmt, ...);
struct Fail {
    int code;
};
#define F3M_CUDA(call)                                                                           \
    do {                                                                                         \
        cudaError_t e__ = (call);                                                                \
        if (e__ != cudaSuccess) {                                                                \
            f3m::set_error("%s failed at %s:%d: %s", #call, __FILE__, __LINE__,                  \
                           cudaGetErrorString(e__));                                             \
            throw f3m::Fail{F3M_ERR_CUDA};                                                       \
        }                                                                                        \
    } while (0)
extern std::atomic<long long> g_launches;   // kernels launched by this library (all threads; informational)
#define F3M_LAUNCH_CHECK()                                                                       \
    do {                                                                                         \
        f3m::g_launches.fetch_add(1, std::memory_order_relaxed);                                                                   \
        F3M_CUDA(cudaGetLastError());                                                            \
    } while (0)
#define F3M_REQUIRE(cond, code, ...)                                                             \
    do {                                                                                         \
        if (!(cond)) {                                                                           \
            f3m::set_error(__VA_ARGS__);                                                         \
            throw f3m::Fail{code};                                                               \
        }                                                                                        \
    } while (0)

// ---- device buffers --------------------------------------------------------------------------
// Device memory comes from a small caching allocator inside the library (api.cu): blocks are obtained
// with cudaMalloc once, kept on a free list when released and handed out again to requests of a similar
// size, so that a repeated product makes no driver call at all.  (The driver's stream-ordered pool
// was tried first; with multi-GB buffers freed and re-requested every call it re-mapped memory at
// unpredictable times, 200 ms at a time.)  A released block may be reused immediately by work that is
// enqueued later on the same stream; every entry point synchronises its stream before it returns, so
// blocks never cross streams while in use.  f3m_release_cached_memory() returns the free list to the driver.
bool dev_in_workspace();   // this thread's buffers come out of a caller's workspace
void *dev_alloc(size_t bytes, size_t *granted, int *device);
void dev_free(void *p, size_t granted, int device);

template <typename T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    size_t granted = 0;
    int device = 0;
    cudaStream_t s = nullptr;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept : p(o.p), n(o.n), granted(o.granted), device(o.device), s(o.s) { o.p = nullptr; o.n = 0; }
    DevBuf &operator=(DevBuf &&o) noexcept {
        if (this != &o) {
            release();
            p = o.p; n = o.n; granted = o.granted; device = o.device; s = o.s;
            o.p = nullptr; o.n = 0;
        }
        return *this;
    }
    void alloc(size_t count, cudaStream_t stream) {
        release();
        s = stream;
        n = count;
        if (count == 0) count = 1;
        p = static_cast<T *>(dev_alloc(count * sizeof(T), &granted, &device));
    }
    void zero() { F3M_CUDA(cudaMemsetAsync(p, 0, (n ? n : 1) * sizeof(T), s)); }
    void release() {
        if (p) dev_free(p, granted, device);
        p = nullptr;
        n = 0;
    }
    ~DevBuf() { release(); }
};

// ---- block-wide exclusive scan (all threads of the block call it; blockDim.x a multiple of 32, at most 1024) ----
__device__ __forceinline__ int block_exclusive_scan(int v, int *total_out, int *smem /* >= 33 ints */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) smem[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int w = lane < nw ? smem[lane] : 0;
        int winc = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += t;
        }
        smem[lane] = winc - w;
        if (lane == 31) smem[32] = winc;
    }
    __syncthreads();
    int res = smem[wid] + inc - v;
    if (total_out) *total_out = smem[32];
    __syncthreads();
    return res;
}

// largest b with off[b] <= i: the box of sorted row i (off = box offsets of a level, nb boxes)
__device__ __forceinline__ int box_of_row(const int *__restrict__ off, int nb, int i) {
    int lo = 0, hi = nb;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// The same by a whole warp, every lane of it with the same i: 32 probes a round
__device__ __forceinline__ int box_of_row_warp(const int *__restrict__ off, int nb, int i) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = nb;   // the box lies in [lo, hi)
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) >> 5, probe = lo + (lane + 1) * step;
        const int below = __popc(__ballot_sync(0xffffffffu, probe < hi && off[probe] <= i));
        lo += below * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// Sums over long boxes (more than `chunk` rows) are cut where a multiple of chunk rows falls, and the parts' sums are added in
// the order of the rows: results do not depend on which part ends first.  Chunk k has two slots: (k, 0) belongs to a long box
// that holds the chunk's first row, (k, 1) to one that starts behind it and goes on in the next chunk.  Every part of every long box
// has a slot of its own, and 2 * chunks of them are enough whatever the boxes hold.
__host__ __device__ inline int64_t part_slots(int64_t n, int chunk) { return 2 * ((n + chunk - 1) / chunk); }
struct BoxPart { int box, begin, end; };
// rows of a slot, begin == end when it has no part (all lanes of the warp call it with the same slot)
__device__ __forceinline__ BoxPart part_of_slot(const int *__restrict__ off, int nb, int n, int chunk, int64_t slot) {
    const int64_t first = (slot >> 1) * chunk, probe = first + (slot & 1) * chunk;
    BoxPart p{0, 0, 0};
    if (probe >= n) return p;
    p.box = box_of_row_warp(off, nb, (int)probe);
    const int a = off[p.box], e = off[p.box + 1];
    if (e - a <= chunk || ((slot & 1) && a <= first)) return p;
    p.begin = (int)(a > first ? a : first);
    p.end = (int)(e < first + chunk ? e : first + chunk);
    return p;
}
// the long box that starts in chunk k and its slots [s0, then 2 (k + 1), 2 (k + 2), .. last]; box < 0: none
struct LongBox { int box; int64_t first_slot, last_slot; };
__device__ __forceinline__ LongBox long_box_of_chunk(const int *__restrict__ off, int nb, int n, int chunk, int64_t k) {
    LongBox l{-1, 0, 0};
    const int64_t next = (k + 1) * chunk;
    if (next > n) return l;                       // it would have to go on in the next chunk
    const int box = box_of_row_warp(off, nb, (int)(next - 1));
    const int a = off[box], e = off[box + 1];
    if (a < k * chunk || e - a <= chunk) return l;
    l.box = box;
    l.first_slot = 2 * k + (a > k * chunk);
    l.last_slot = 2 * ((int64_t)(e - 1) / chunk);
    return l;
}

// chebyshev_nodes_1D / get_w_j_first_kind (F3M_src/n_tree.cu:265-285): first-kind Chebyshev nodes and barycentric
// weights with the reference's float32 expression (PI as a float, arguments rounded to float before cos / sin).
inline void cheb_nodes_weights(int p, float *node, float *w) {
    const float PI = (float)(atan(1.) * 4.);
    for (int i = 0; i < p; i++) {
        const float arg = ((float)i * 2.f + 1.f) * PI / (float)(2 * (p - 1) + 2);
        node[i] = (float)cos((double)arg);
        w[i] = (float)(pow(-1.0, i) * sin(((2. * (float)i + 1.) * PI) / (2. * (float)(p - 1.0) + 2.)));
    }
}

// ---- small per-plan device words (f3m_plan::d_flags) and their pinned host mirror ------------------
constexpr int FLAG_WORDS = 640;
enum FlagSlot {
    FL_ERR = 0,          // device-side consistency check failed
    FL_LISTOVER = 1,     // a list is longer than the memory it was given on a bound
    FL_LISTTOT = 8,      // 4 words: 64-bit totals of a merged tree
    FL_BBOX = 16,        // 2 * MAXD words
    FL_MMA_COUNTER = 32, // tile cursor of the tensor-core near kernel
    FL_LEAF = 40,        // 2 words: small / big finest-level boxes
    FL_NSMALL = 42,      // target tiles of at most 32 points
    FL_WEIGHTS = 43,     // a weight is not finite, or near the largest float; the next word: weights that are not zero
    FL_BBOX_Y = 48,      // 2 * MAXD words, the second point set
    FL_LVTOT = 64,       // boxes per level of the batch being built (F3M_MAX_LEVELS words)
    FL_LVMAX = 96,       // largest box per level (F3M_MAX_LEVELS words)
    FL_LVTOT_Y = 128, FL_LVMAX_Y = 160,   // the same of the second tree
    FL_LISTS = 192,      // 6 words per level: 64-bit far / small / keep pair counts
    FL_PAIRWORK = 352    // 8 words per level: 64-bit sums of n_x * n_y and of n_x over the box pairs of the small list and of the kept one
};
static_assert(FL_LISTS + 6 * (F3M_MAX_LEVELS + 1) <= FL_PAIRWORK && FL_PAIRWORK + 8 * (F3M_MAX_LEVELS + 1) <= FLAG_WORDS, "flag words");

// ---- tree ------------------------------------------------------------------------------------
struct Level {
    int nb = 0;             // occupied boxes
    float edge = 0.f;       // box edge at this level
    int max_count = 0;
    DevBuf<int> off;        // (nb+1) offsets into the sorted point order
    DevBuf<uint32_t> code;  // (nb) Morton prefix
    DevBuf<int> parent;     // (nb) compact id of the parent box one level up
    DevBuf<int> child_start;// (nb+1) first child (compact id one level down); filled when that level exists
    DevBuf<float> ctr;      // (nb,d) centres
};

struct Tree {
    int64_t n = 0;
    int d = 0;
    const float *data = nullptr;   // caller's rows
    float origin[MAXD] = {0};      // per-dimension minimum
    float edge0 = 0.f;             // cube edge
    int lmax = 0;                  // depth of the Morton key
    int sorted_depth = 0;          // the keys are sorted by their first sorted_depth levels (d bits each)
    DevBuf<uint32_t> keys;         // (n) Morton keys at depth lmax, sorted by their first sorted_depth levels
    DevBuf<int> perm;              // (n) sorted position -> input row
    DevBuf<float> pts;             // (d,n) sorted coordinates, one plane per dimension
    std::vector<Level> levels;     // levels[0] is the root
    // A tree whose points arrive as sorted runs (one per rank): the levels are built from one pseudo key per occupied
    // finest sorted cell (pkeys) and offsets into the merged order (fine_off) before the points are attached.
    struct Runs {
        bool pending = false;      // levels may be built, points not merged in yet
        int nruns = 0, ncells = 0, nocc = 0;
        DevBuf<int> counts;        // (nruns, ncells) points per cell and run
        DevBuf<int> seg_start;     // (nruns, ncells + 1) position of the cell inside its run
        DevBuf<int> cell_off;      // (ncells + 1) merged offset of the cell
        DevBuf<uint32_t> pkeys;    // (nocc) pseudo key of every occupied cell
        DevBuf<int> fine_off;      // (nocc + 1) merged offset of every occupied cell
    } runs;
};

struct PairCSR {
    DevBuf<int> ptr;  // (boxes_x+1)
    DevBuf<int> idx;  // source box per pair
    int64_t count = 0;
    // direct lists: pairs of points, and (target point, source box) pairs
    int64_t pairs = 0, row_boxes = 0;
};

struct LevelLists {
    PairCSR far, small, keep;
    int p = 0;        // nodes per dimension used for the far field of this level
    // far rows re-ordered by box offset (last axis most significant) with the packed offsets, built on first use
    DevBuf<uint32_t> far_okey;
    DevBuf<int> far_oidx;
    bool far_ordered = false;
    DevBuf<float> T;   // axis matrices of the level (far_fast.cu), built on first use
    bool T_ready = false;
};

// Device time per stage, from CUDA events recorded on the product's stream and read after its
// final synchronisation (no extra synchronisation inside the product).
enum Stage { ST_PERMUTE = 0, ST_DIRECT = 1, ST_P2M = 2, ST_M2L = 3, ST_L2P = 4, ST_UNPERMUTE = 5, ST_TOTAL = 6, ST_BUILD = 7 };
// forms of the direct-sum kernels (counted per launch; the first six by f3m_plan_last_direct_variants)
enum DirectVariant { DV_MUFU = 0, DV_POLY2 = 1, DV_POLY3 = 2, DV_DIRECT = 3, DV_MOMENTS = 4, DV_TENSOR = 5, DV_NODES = 6, DV_COUNT = 7 };
struct Timings {
    float ms[8] = {0};
    int direct_launches = 0;
    int direct_variants[DV_COUNT] = {0};
    int column_launches = 0;           // of those, launches of the several-column kernel (near_cols.cu)
    int64_t pairs[DV_COUNT] = {0};     // pairs of points in the lists summed pair by pair, by the form of the sum
    int64_t box_pairs = 0;             // box pairs of the far field
    int cut = 0;                       // level the product ended at before the last one, 0: none
    void clear_counts() {
        direct_launches = column_launches = cut = 0;
        box_pairs = 0;
        for (int &v : direct_variants) v = 0;
        for (int64_t &v : pairs) v = 0;
    }
    // Events are created once and recycled with the plan's scratch slot (api.cu).  They are read when somebody asks (resolve), not by
    // every product: a query costs as much as a launch.  A span that begins where the one before ended shares its event.
    struct Span { int stage, a, b; };      // event numbers; b < 0: not closed
    std::vector<Span> spans;
    std::vector<cudaEvent_t> *events = nullptr;
    int used = 0, last_end = -1;
    long long launches_at_end = 0;
    float build_ms = 0.f;
    int record(cudaStream_t s) {
        if (used == (int)events->size()) {
            cudaEvent_t e;
            F3M_CUDA(cudaEventCreate(&e));
            events->push_back(e);
        }
        F3M_CUDA(cudaEventRecord((*events)[used], s));
        return used++;
    }
    void begin(int stage, cudaStream_t s) {
        const bool adjoins = last_end >= 0 && launches_at_end == g_launches.load(std::memory_order_relaxed);
        spans.push_back(Span{stage, adjoins ? last_end : record(s), -1});
        last_end = -1;
    }
    void end(cudaStream_t s) { close(spans.size() - 1, s); }
    void close(size_t span, cudaStream_t s) {
        spans[span].b = last_end = record(s);
        launches_at_end = g_launches.load(std::memory_order_relaxed);
    }
    // a product begins: the spans of the one before are forgotten, the plan's own (the build, if nobody has read it yet) is kept
    void start_product() {
        const bool build = !spans.empty() && spans[0].stage == ST_BUILD && spans[0].b >= 0;
        spans.resize(build ? 1 : 0);
        used = build ? spans[0].b + 1 : 0;
        last_end = -1;
        for (float &m : ms) m = 0.f;
    }
    // Call after the stream has been synchronised (an event that has not passed all the same is waited for: a span once dropped is never
    // read).  A span that was never closed (the product failed in between) is dropped; a failed query must not stay behind as the
    // runtime's last error, or the next launch check of an unrelated call would report it.
    void resolve() {
        for (auto &sp : spans) {
            float t = 0.f;
            if (sp.b < 0) continue;
            if (cudaEventSynchronize((*events)[sp.b]) != cudaSuccess || cudaEventElapsedTime(&t, (*events)[sp.a], (*events)[sp.b]) != cudaSuccess)
                (void)cudaGetLastError();
            else if (sp.stage == ST_BUILD) build_ms = t;
            else ms[sp.stage] += t;
        }
        spans.clear();
        used = 0;
        last_end = -1;
        ms[ST_BUILD] = build_ms;
    }
};

}  // namespace f3m

struct f3m_plan {
    int device = 0;
    int d = 0;
    bool same = false;
    f3m_params prm{};
    float lcs = 0.f;
    f3m::Tree tx, ty_store;
    f3m::Tree *ty = nullptr;
    std::vector<f3m::LevelLists> lists;   // lists[l] for level l (index 0 unused)
    f3m::LevelLists cut_lists;            // all pairs of the level a product is cut at (count, row pointers and the ordered rows)
    int cut_level = 0;
    f3m::DevBuf<float> shift_a, shift_at; // matrices between a box and its children, for shift_p nodes; built on first use
    int shift_p = 0;
    int levels = 0;
    f3m_plan_stats stats{};
    f3m::Timings last;
    // sharded moments (multi-GPU): either write the finest-level moments of a slice of the source boxes
    // into moments_out and stop, or take the complete finest-level moments from ext_mom instead of computing them
    // finest-level boxes split by size for P2M / L2P (index 0: target tree, 1: source tree): boxes of at most
    // LEAF_SMALL points are handled one per warp, the others one per CTA; built on first use
    f3m::DevBuf<int> leaf_small[2], leaf_big[2];
    int n_leaf_small[2] = {0, 0}, n_leaf_big[2] = {0, 0};
    int leaf_level[2] = {-1, -1};         // level the two lists were built for
    float *moments_out = nullptr;
    int64_t mom_begin = 0, mom_end = 0;
    int64_t mom_box_begin = -1, mom_box_end = -1;   // >= 0: moments_out covers these source boxes only
    const float *ext_mom = nullptr;
    // source boxes named by the direct lists of a level over ALL targets (a constant of the plan, built on first use)
    std::vector<f3m::DevBuf<unsigned char>> src_need;
    // packed sources of the last direct list (valid inside one product)
    struct PackCache {
        int level = -1, r0 = 0, rb = 0;
        bool expanded = false;
        f3m::DevBuf<float> buf;
        void reset() { level = -1; buf.release(); }
    } pack_cache;
    // direct lists taken through nodes (near_nodes.cu): a level's rows in the order of the box offsets, built on first use
    struct NodeRows {
        bool ready = false, small = false, keep = false;   // which lists the rows hold
        f3m::DevBuf<int> ptr, oidx;
        f3m::DevBuf<uint32_t> okey;
    };
    std::vector<NodeRows> node_rows;
    int weights_ok = -1;                  // of the product under way: finite, and not mostly zeros (-1: not looked at yet)
    // source rows of the several-column kernel (near_cols.cu; valid inside one product)
    struct ColumnRows {
        int r0 = -1;
        f3m::DevBuf<float> buf;
        void reset() { r0 = -1; buf.release(); }
    } column_rows;
    // a product shared by several GPUs, in phases (f3m_plan_shard_begin / _near / _far): state kept between the calls
    struct Shard {
        bool active = false;
        bool all_sources = false;                          // no halo bookkeeping: bs holds every row
        int R = 0;
        int64_t row_begin = 0, row_end = 0;
        f3m::DevBuf<float> bs;                             // b in sorted order, filled for the boxes this rank reads
        std::vector<f3m::DevBuf<unsigned char>> need;      // per level: source boxes named by the rank's direct lists
    } shard;
    // a plan for one product (f3m_kmvm_f32): it may end at the level where that product will (far_stop_level), and b may have been sorted
    // with its points
    bool one_product = false;
    int stop_level = 0;
    const float *carry_b = nullptr;
    f3m::DevBuf<float> carried_b;
    long long launches_at_wait = -1;      // g_launches when the build last waited for its stream
    int *h_pinned = nullptr;              // pinned host words for count read-back (FLAG_WORDS ints)
    int *d_flags = nullptr;               // device status / counters (FLAG_WORDS ints, see FlagSlot)
    std::vector<cudaEvent_t> *events = nullptr;   // of the scratch slot, see Timings
    ~f3m_plan();
};

namespace f3m {

// ---- sort.cu ---------------------------------------------------------------------------------
void bounding_box(const float *X, int64_t n, int d, unsigned *words, cudaStream_t s);   // 2 * MAXD device words, zero before
void bounding_box_values(const unsigned *words, int d, float *h_min, float *h_max);     // the words on the host, decoded
// The cube on the host, or still on the device: the words of bounding_box, of the set itself and of the one it shares the edge with
struct Cube {
    const float *origin = nullptr;
    float edge0 = 0.f;
    const unsigned *own = nullptr, *other = nullptr;
};
int sort_passes_for(int bits);
bool sort_carries(int d, int depth);   // a sort to this depth takes a value per point along at less cost than a gather
// b (or null): a value per point that travels along, in sorted order at b_out
void build_sorted_tree(Tree &t, const float *X, int64_t n, int d, const Cube &cube, int math_mode, int depth, cudaStream_t s,
                       const float *b = nullptr, DevBuf<float> *b_out = nullptr);
int record_words(int d);   // 32-bit words of the record [input row, coordinates] that travels with a key in the sort
void sort_shard(const float *X, int64_t n, int64_t row0, int d, const float *origin, float edge0, int math_mode, int depth,
                uint32_t *recs_out, int *cell_counts_out, cudaStream_t s);
void tree_from_cell_counts(Tree &t, const int *counts, int nruns, int d, const float *origin, float edge0, int depth, f3m_plan *pl,
                           cudaStream_t s);
void tree_attach_runs(Tree &t, const uint32_t *recs, int64_t stride, cudaStream_t s);
void exclusive_scan_i32(const int *in, int *out, int64_t n, cudaStream_t s);  // n values; out may alias in
// up to four arrays of n values scanned in place by one set of launches; their sums as 64-bit numbers -> totals64 (device)
void exclusive_scan_multi(int *const *arrays, int narr, int64_t n, long long *totals64, cudaStream_t s);
void gather_rows(const float *src, const int *perm, float *dst, int64_t n, int cols, cudaStream_t s, float *zeroed = nullptr, int64_t nz = 0);
void scatter_rows(const float *src, const int *perm, float *dst, int64_t n, int cols, cudaStream_t s);
void scatter_rows_nonzero(const float *src, const int *perm, float *dst, int64_t n, int cols, cudaStream_t s);

// ---- tree.cu ---------------------------------------------------------------------------------
void build_roots(f3m_plan *pl, cudaStream_t s);   // of both trees, and the list of their one pair (n_tree.cu:1071)
// box starts of the levels after the last one built, up to l_last (at most HEADS_BATCH of them): counted, then written
constexpr int HEADS_BATCH = 8;
struct HeadsBatch {
    DevBuf<int> part;
    int l_first = 0, nlev = 0, nt = 0;
};
void heads_begin(Tree &t, HeadsBatch &hb, int l_first, int l_last, int *d_tot, cudaStream_t s);
void heads_finish(Tree &t, HeadsBatch &hb, const int *h_tot, int *d_max, int *d_err, cudaStream_t s);
void build_levels(Tree &t, int l_last, f3m_plan *pl, cudaStream_t s);   // appends levels up to l_last (<= sorted_depth)
// interaction lists of a level from lists[level-1].keep: counted (FL_LISTS), then written; cap: entries each list has room for
void lists_count(f3m_plan *pl, int level, cudaStream_t s);
void lists_write(f3m_plan *pl, int level, const int64_t cap[3], cudaStream_t s);

// near_nodes.cu: the direct lists of a level through interpolation nodes (whole products of one column)
struct NodeChoice {
    int p = 0;                          // nodes per axis, 0: no list of the level takes this form
    bool small = false, keep = false;   // the lists that do (near list: last level only)
    double seconds = 0.0;               // estimated time of the level's direct lists with this choice
};
// ---- far.cu ----------------------------------------------------------------------------------
int nodes_per_dim(int d, int nr_interpolation);   // get_node_list for perfect powers, floor otherwise
void far_field_level(f3m_plan *pl, int level, const float *b_sorted, int R, float *out_sorted,
                     int64_t row_begin, int64_t row_end, cudaStream_t s);   // per-level path (far.cu)
// end: the last level whose far pairs are taken; cut == end: that level's small and kept pairs too
void far_field(f3m_plan *pl, const float *b_sorted, int R, float *out_sorted, int64_t row_begin, int64_t row_end, int cut, int end,
               cudaStream_t s);                                               // whole product (far_fast.cu)
int64_t far_moments_size(const f3m_plan *pl, int R);
// Where a product over all rows may end before the last level of its tree.  nodes: the level's small and kept pairs go through that many
// nodes of their own (near_nodes.cu); 0: all its pairs go through the far field's.
struct CutChoice {
    int level = 0;      // 0: the product visits all levels
    NodeChoice nodes;
};
CutChoice far_cut(const f3m_plan *pl, int R, bool nodes_allowed = true);
bool far_ends_with_nodes(const f3m_plan *pl, int level);   // a plan for one product: nothing below this level will be visited
int far_node_end_level(const f3m_plan *pl, float edge0, int lmax);
int far_stop_level(const f3m_plan *pl, int R, float edge0, const float *xmin, const float *ymin, int64_t n);   // before the tree is built

// ---- shard.cu --------------------------------------------------------------------------------
const unsigned char *level_source_flags(f3m_plan *pl, int level, cudaStream_t s);   // per source box of the level: named by a direct list?
void shard_partition(f3m_plan *pl, int R, int nparts, int64_t *h_bounds, cudaStream_t s);
void shard_mark_and_gather(f3m_plan *pl, const float *b, int R, int row_begin, int row_end, int box_begin, int box_end,
                           bool everything, cudaStream_t s);
void shard_count_rows_by_owner(const f3m_plan *pl, int64_t row_begin, int64_t row_end, const int64_t *h_bounds, int nranks,
                               int64_t *h_counts, cudaStream_t s);
void shard_pack_rows_by_owner(const f3m_plan *pl, const float *acc_sorted, int R, int64_t row_begin, int64_t row_end,
                              const int64_t *h_bounds, int nranks, const int64_t *h_counts, float *send, cudaStream_t s);
void shard_gathered_rows_to_input_order(const f3m_plan *pl, const float *gathered, int R, const int64_t *h_slice_bounds, int nslices,
                                        int64_t stride, int64_t in_lo, int64_t in_hi, float *out, cudaStream_t s);
void shard_place_rows(const float *recs, int64_t n, int R, int64_t in_lo, int64_t in_hi, float *out, int *d_err, cudaStream_t s);
void shard_rows_to_input_order(const f3m_plan *pl, const float *acc_sorted, int R, int64_t in_lo, int64_t in_hi, float *out,
                               cudaStream_t s);

// ---- near.cu ---------------------------------------------------------------------------------
void direct_sums(f3m_plan *pl, int level, const PairCSR &csr, const float *b_sorted, int R, float *out_sorted,
                 int64_t row_begin, int64_t row_end, cudaStream_t s);
double pair_list_seconds(const f3m_plan *pl, int level, const PairCSR &csr, int R);   // estimate
// near_cols.cu: up to eight columns of a direct list, starting at r0 (two dimensions and more)
void column_sums(f3m_plan *pl, int level, const PairCSR &csr, bool expanded, const float *b_sorted, int R, int r0, float *out_sorted,
                 int row_begin, int row_end, cudaStream_t s);
// near_moments.cu: sums a direct list through box moments when its geometry allows; false: sum the pairs
bool moment_sums(f3m_plan *pl, int level, const PairCSR &csr, bool alone, const float *b_sorted, int R, float *out_sorted, int row_begin,
                 int row_end, cudaStream_t s);
double direct_list_seconds(const f3m_plan *pl, int level, const PairCSR &csr, int R);   // estimate, pairs or moments
NodeChoice node_choice(const f3m_plan *pl, int level, int R);
// the same for a level at which the product ends: its small and kept pairs together, seconds their time (p = 0: not possible)
NodeChoice node_end(const f3m_plan *pl, int level);
bool node_sums(f3m_plan *pl, int level, const NodeChoice &choice, const float *b_sorted, float *out_sorted, cudaStream_t s);
template <bool GRAD>
void dense_f32(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, int d, float ls, float *out,
               cudaStream_t s);
void dense_f64(const double *X, int64_t N, const double *Y, int64_t M, const double *b, int R, int d, double ls, double *out,
               cudaStream_t s);
void measure_peaks(double *gexp, double *gfma, cudaStream_t s);
void dense_f32_static(const float *X, int64_t N, const float *Y, int64_t M, const float *b, int R, int d, float ls, float *out,
                      cudaStream_t s);

}  // namespace f3m
