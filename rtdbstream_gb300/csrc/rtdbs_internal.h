// rtdbs_internal.h -- device-side state layout shared by the kernels and the
// host engine of the streaming DBSCAN path.
//
// HBM layout of one stream (W slots, chunk C <= kChunkMax points):
//   ring   float4[W]      point of each ring slot (x, y, z, slot bits); the
//                         reference's params.window (src/dbscan/dbscan.h:23)
//   kslot  u64[W]         cell key of each slot (reference: point_cell_id)
//   skey   u64[2][W]      window sorted by (cell key, slot): keys
//   spt    float4[2][W]   ... points in that order (.w = slot as int bits)
//   scnt   i32[2][W]      ... exact neighbour count in that order
//                         (double-buffered; the reference's pos_arr/
//                         tmp_pos_arr, src/dbscan/grid.cpp:181-199)
//   table  {u64,u64}[2][P] open-addressed cell table: tagged key -> [start,end)
//                         (replaces the OptiX BVH, src/dbscan/optix.cpp:438-483)
//   parent i32[W]         union-find forest by slot (reference: cluster_id)
//   sroot  i32[W]         per sorted position: root hint during the union, then
//                         the root (-1: not core)
//   label, cid i32[W]     outputs by slot
//   nlist  i32[W][stride] neighbour list of every non-core point by slot
//                         (cap = MinPts - 2 entries, rows padded to a multiple
//                         of 4 for 16-byte loads; -1 = empty entry)
//   rslot  i32[W]         per slot after the flatten: root (core) or -1
//   damaged i32[W]        per previous root: the component lost a core this slide
//   ntrack i32[W]         1: the slot's list is exact; 0: not kept (core, or
//                         rebuilt at the end of the slide)
//   sprev  i32[2][W]      per sorted position: the point's root at the last
//                         clustering (-1: not core), carried by the merges
//   chunk scratch: sort words, expired points.
#pragma once

#include <cstdint>
#include <math.h>
#include <cuda_runtime.h>

namespace rtdbs {

constexpr int kChunkMax = 16384;   // points per grid-update chunk
constexpr int kOffBits = 14;       // in-chunk offset bits of a sort word
constexpr int kKeyBitsMax = 50;    // cell-key bits (key << 14 | offset fits in 64 bits)
constexpr unsigned long long kKeyMask = (1ull << kKeyBitsMax) - 1ull;
constexpr unsigned kGenMod = 16383;  // table generations 1..16383 (tag = gen << 50 | key)
constexpr int kMergeTile = 1024;   // old entries per merge block
constexpr int kMergeThreads = 256;
constexpr int kSortRun = 1024;     // words per radix-sort CTA (one per thread)
constexpr int kSortBits = 9;       // most digit bits of a chunk sort pass
constexpr int kBuildThreads = 512;
constexpr int kClusterThreads = 256;
constexpr int kLinkThreads = 256;
constexpr int kQueryLanes = 16;    // lanes per query point in the count passes where the queries
                                   // fill the GPU (one cell per Eps: two points per warp
                                   // overlap their loads)
constexpr int kMaxIter = 1 << 20;  // bound on every device-side retry loop
constexpr int kListCap = 30;       // longest neighbour list kept (MinPts <= 32)

// Bits of Ctl::err.
constexpr int kErrHashFull = 1;
constexpr int kErrUnionIter = 2;
constexpr int kErrChunk = 8;
constexpr int kErrList = 16;

// Device-resident control block of one stream.  Every field that changes
// from slide to slide lives here (not in kernel arguments), so one captured
// CUDA graph replays every slide.
struct Ctl {
    long long b;               // grid builds so far (merge + table build)
    long long slide;           // slides completed
    int unit;                  // slide % units: the stride of ring slots that comes next
    int nocc[2];               // entries in sorted buffer 0 / 1
    int nitems;                // cell runs (within 32 sorted positions) of the current grid
    int ncells;                // cells of the current grid
    int err;                   // kErr* bits
    int prev_ok;               // label/cid hold the clustering of the window before
                               // this slide's changes (the forest can be reused)
    int union_next;            // next block of positions handed out by k_union
    unsigned long long band_rechecks;
    // counters of the reference's debug build (src/dbscan/dbscan.cpp:145-212):
    // [0] count passes (core identification), [1] clustering scans; spread over 8
    unsigned long long ptests[2][8];   // distance tests
    unsigned long long phits[2][8];    // ... that found a neighbour
    int qmax[8];                       // most distance tests of one count query
    int reused;                // cores that joined a reused component this slide
    int reuse_skip;            // slides left without forest reuse (it paid off too little)
    long long last_reused;     // `reused` of the last clustering
    long long kept_from;       // first slide since when every slide kept its chunks' orders
    const float* input;        // new points of this slide
    int* out_label;            // caller's outputs of this slide or clustering, written beside
    int* out_cid;              // label and cid (null: none)
    long long b_done;          // builds whose table is in place (b, while no build is under way)
};

// What a slide or a clustering exchanges with its caller: the kernels read the
// new points and write the results there, so no copies run around them.  All
// pointers are accessible to the kernels (device memory, or pinned host
// memory); label / cid may be null.
struct SlideIO {
    const float* input;
    int* label;
    int* cid;
};

// Everything a kernel needs for one stream, passed by value.
struct View {
    // geometry: cell (i, j, k) = clamp(floor((x - origin) * inv_cell), 0, ext - 1),
    // key = i << shift[0] | j << shift[1] | k (bit fields, shift[2] = 0)
    double origin[3];
    double inv_cell;
    float origin32[3], inv_cell32;  // the same in single precision, with the
    float key_err[3];               // largest error of its quotient, in cells (> 1/2: not used)
    long long ext[3];
    int shift[3];
    int dim;
    int cell_mult;              // K: cells per Eps along each axis (1 or 2)
    int grab;                   // cell runs a union warp takes from the queue at a time (whole
                                // blocks of positions: one per 16 runs, at least one)
    int qlanes;                 // lanes per query point in the count passes (16 or 32)
    // parameters
    int W, S, min_pts, units;   // units = W / S
    int chunk;                  // C
    int pbits;                  // log2 of table capacity
    unsigned pmask;
    float r2f;                  // FP32 mode: (float)eps * (float)eps
    float lo, hi;               // FP64 mode: FP32 filter band (NaN: every test in FP64)
    double E;                   // FP64 mode: eps * eps
    int key_bits;
    int sort_passes, sort_bits;  // radix passes over a chunk's keys, bits per pass
    int block_pts;              // sorted positions a union warp takes as one block (8, 16 or 32;
                                // pool launches take 32)
    int precision;              // RTDBS_PREC_* (batched launches dispatch on it)
    int list_cap;               // entries per neighbour list; -1: no lists (the
                                // label pass then scans the grid)
    int list_stride;            // ints per list row (list_cap rounded up to 4)
    // buffers
    float4* ring;
    unsigned long long* kslot;
    unsigned long long* skey[2];
    float4* spt[2];
    int* scnt[2];
    ulonglong2* table[2];
    int* parent;
    int* sroot;                  // per sorted position: root hint during the union
                                 // (-1: not core), then the root (-1: not core)
    int* label;
    int* cid;
    int* nlist;                  // [W][list_stride] neighbours of non-core points
    int* rslot;                  // per slot: root of a core, -1 otherwise
    int* damaged;                // per old root slot: its component lost a core this
                                 // slide (0 outside the union phase)
    int* ntrack;                 // per slot: 1 list exact, 0 not kept
    int* sprev[2];               // per sorted position (with the sorted buffers): the
                                 // point's root at the last clustering, -1 if it was not
                                 // core (or not there); carried by the merges for forest
                                 // reuse; null without neighbour lists
    unsigned long long* nsort;   // chunk sort words in (key << 14 | offset)
    unsigned long long* xsort;
    unsigned long long* xkey;    // cell keys of the chunk's expired points by offset
    unsigned long long* nword;   // sorted
    unsigned long long* xword;
    float4* xpt;                 // expired points of the chunk by offset
    int* sorder;                 // per slot el + r: offset (slot - el) of the chunk's r-th
                                 // point in (key, slot) order, kept from the slide that
                                 // brought the chunk in; null: not kept
    const float* staging;        // new points [S][dim]
    Ctl* ctl;
};

// Cell coordinate along axis a: clamp(floor((x - origin) * inv_cell), 0, ext - 1)
// in double, NaN in cell 0.  The single-precision quotient differs from the
// double one by at most key_err cells (see set_geometry), so its floor is the
// double's wherever no cell edge lies within that; the others, and quotients
// outside [0, 2^22), are redone in double.  (FP64 runs at 1/64 of the FP32
// rate here: a first window of 1M points took 50 us longer all in double, and
// the decrement, which recomputed its queries' keys, 7 us per slide.)
__host__ __device__ __forceinline__ long long cell_coord(const View& v, int a, float x) {
#ifdef __CUDA_ARCH__  // (separate roundings; on the host by -ffp-contract=off)
    const float t32 = __fmul_rn(__fsub_rn(x, v.origin32[a]), v.inv_cell32);
    const float f = floorf(t32), in = __fsub_rn(t32, f);
#else
    const float t32 = (x - v.origin32[a]) * v.inv_cell32;
    const float f = floorf(t32), in = t32 - f;
#endif
    long long c;
    if (t32 >= 0.0f && t32 < 4194304.0f && in >= v.key_err[a] && in <= 1.0f - v.key_err[a]) {
        c = (long long)(int)f;
        const long long top = v.ext[a] - 1;
        return c > top ? top : c;
    }
    double t = floor(((double)x - v.origin[a]) * v.inv_cell);
    if (!(t >= 0.0)) t = 0.0;  // also maps NaN to cell 0
    const double top = (double)(v.ext[a] - 1);
    if (t > top) t = top;
    return (long long)t;
}

// Combined template code of a stream's work kernels: dim + 4 (cells per Eps - 1).
__host__ __device__ inline int dk_of(const View& v) { return v.dim + 4 * (v.cell_mult - 1); }

// Kernel phases of a slide, in launch order.
enum Phase : int {
    kPhaseIngest = 0,
    kPhaseSort,
    kPhaseDecrement,
    kPhaseMerge,
    kPhaseBuild,
    kPhaseIncrement,
    kPhaseUnion,
    kPhaseFlatten,
    kPhaseLabel,
    kNumPhases
};
constexpr int kChunkPhases = 6;  // ingest .. increment, once per chunk

// Launchers (rtdbs_kernels.cu).  j = chunk index within the slide (or the
// load), c = points in the chunk, init = 1 while loading the first window,
// advance = 1 when the label phase ends a slide.
// io: for the ingest (input null: the one that the slide's first ingest left in
// the control block).
cudaError_t launch_phase(int phase, const View& v, int precision, int j, int c, int init,
                         int staging_offset, int advance, cudaStream_t s, bool pdl = false,
                         const SlideIO& io = SlideIO{});
// With a side stream and two events, the decrement pass (which needs only
// the ingest) runs on `side` beside the sort, joined before the merge.  pdl:
// programmatic dependence on the kernel launched before on the same stream.
// ingested: the chunk's ingest has been launched already (outside a captured
// graph, as its arguments change from slide to slide).
cudaError_t launch_chunk_step(const View& v, int precision, int j, int c, int init,
                              int staging_offset, cudaStream_t s, const SlideIO& io, bool ingested = false,
                              cudaStream_t side = nullptr, cudaEvent_t fork = nullptr,
                              cudaEvent_t join = nullptr);
// The grid of all W slots built at once (see the kernels): slots
// [0, count) while loading (init), else the slide's slots, take the new points
// (count = S in a slide).
cudaError_t launch_window_build(const View& v, int precision, const SlideIO& io, int count, int init,
                                cudaStream_t s, bool ingested = false);
cudaError_t launch_window_phase(int phase, const View& v, int precision, const SlideIO& io, int count, int init,
                                cudaStream_t s, bool pdl = false);
int window_build_launches(const View& v);
// Bounding box of n points per axis as order-keeping unsigned keys: minima
// in box[0..2] (~0: no finite coordinate), maxima in box[3..5] (device).
cudaError_t launch_bbox(const float* pts, long long n, int dim, unsigned* box, cudaStream_t s);
inline int slot_bits(int W) {
    int b = 0;
    while ((1ll << b) < (long long)W) ++b;
    return b;
}
// Whether key and slot fit one sort word there.
inline bool window_build_fits(const View& v) {
    return v.W <= kChunkMax || v.key_bits + slot_bits(v.W) <= 64;
}
// Whether a slide of two chunks or more, and at least a twentieth of the window,
// is cheaper built from all slots than by chunk steps, by what the first window's
// build counted: its cell runs and distance tests.  In units of a window position
// that a chunk step rewrites: the steps rewrite W positions per chunk and, for
// every new and expired point (both in one figure), look up its stencil (5/4 a
// cell) and test its candidates (1/25 a test); the build orders W positions (3/4), looks up the stencil of
// every cell run (3/10 a cell) and tests every point against its candidates (1/80
// a test; 1/30 in 1-D, where steps keep most of the forest besides).  Fitted to
// 990 pairs of times (W 40k to 2M, S W/100 to W, MinPts 3 to 30, streams from
// near-empty cells to 13,000 tests a point, one and two cells per Eps): 0.7% over
// the better of both in the geometric mean, 1.6 times at worst.  By S >= W/20 alone
// it was 11% and 4.8 times (1-D prices with 13,000 tests a point, S = W/20, 1M points:
// 17.5 ms stepped, 73.5 built; the offset stream with two cells per Eps 0.73 and
// 2.31; 2-D mixture with 30 neighbours, S = W/2, 3.1 and 0.55).
inline bool window_build_pays(int W, int S, int dim, int cells_per_eps, long long runs, double tests) {
    double cells = 1.0;  // of the stencil
    for (int a = 0; a < dim; ++a) cells *= 2 * cells_per_eps + 1;
    const int chunks = (S + kChunkMax - 1) / kChunkMax;
    const double steps = (double)chunks * W + 1.25 * cells * S + 0.04 * tests * S / W;
    const double build = 0.75 * W + 0.3 * cells * (double)runs + tests / (dim == 1 ? 30.0 : 80.0);
    return chunks > 1 && 20ll * S >= W && steps > build;
}
// fresh_hints: start the union from fresh hints and forest (no reuse), for a
// clustering of the window as it stands rather than after a slide, with its
// outputs in io (a slide's io goes to its ingest).
// outputs_free: an event the label pass (which rewrites label/cid) waits for
// first, with wait_flags (cudaEventWaitExternal inside a stream capture).
cudaError_t launch_cluster(const View& v, int precision, int advance, cudaStream_t s, bool fresh_hints = false,
                           cudaEvent_t outputs_free = nullptr, unsigned wait_flags = 0,
                           const SlideIO& io = SlideIO{});
cudaError_t launch_counts_by_slot(const View& v, int* nn_by_slot, cudaStream_t s);
cudaError_t configure_kernels();
// Warps of the count passes that the configured device holds at once.
int count_pass_warps();

// Host helpers shared by the engine and the allocation-free entry point
// (rtdbs_engine.cpp).
// Records the text rtdbs_last_error returns on this thread; returns status.
int set_error(int status, const char* fmt, ...);
// FP32 filter band of the FP64 predicate and the FP32 radius (View::lo, hi,
// E, r2f) for this Eps.
void set_band(View& v, double eps);
// Grid geometry of View v (origin, extents, key fields, inv_cell, key_bits,
// sort_passes) for cells of side Eps (1 + 2^-12) / cells_per_eps over the
// box [bmin, bmax] of `dim` axes, widened by 25% (and at least 4 cells) when
// `widen`; the cell side doubles until the key fits kKeyBitsMax bits.
// Returns RTDBS_OK or RTDBS_ERR_INVALID (empty or non-finite box); the side
// used goes to *cell_side.
int set_geometry(View& v, int dim, double eps, int cells_per_eps, const float* bmin, const float* bmax,
                 bool widen, double* cell_side);

// ------------------------------------------------------------ batched launches
// One launch of a phase covers many streams: block b belongs to the item i
// with prefix[i] <= b < prefix[i+1] and runs that stream's kernel body with
// block index b - prefix[i] of prefix[i+1] - prefix[i].

enum BatchPhase : int {
    kBatchIngest = 0,
    kBatchSort,
    kBatchRunmerge,
    kBatchDecrement,
    kBatchMerge,
    kBatchBuild,
    kBatchIncrement,
    kBatchLink,
    kBatchUnion,
    kBatchFlatten,
    kBatchLabel,
    kNumBatchPhases
};
constexpr int kBatchChunkPhases = 7;  // ingest .. increment

struct BatchItem {
    int view;            // index into the View array
    int j;               // chunk index within the slide
    int c;               // points in the chunk
    int stg_off;         // offset of the chunk within the stream's new points
    const float* input;  // the stream's new points of this slide (device)
};

struct BatchLaunch {
    const View* views;
    const BatchItem* items;
    const int* prefix;   // n + 1 entries
    int n;
};

// Blocks one item needs in a phase (same shapes as the single-stream launches).
int batch_blocks(int phase, const View& v, int c);
int batch_threads(int phase);
// Phases launched once per (precision, dim) group of streams (the others
// take every stream in one launch; prec and dim are then ignored).
// `dim` here is the stream group's dk_of code (dimension and cells per Eps).
bool batch_phase_split(int phase);
cudaError_t launch_batch(int phase, int prec, int dim, const BatchLaunch& L, int total_blocks, int max_c,
                         cudaStream_t s);
// Packs n device arrays (count[i] floats from src[i]) into dst at dst_off[i];
// the three tables are device memory.
cudaError_t launch_gather(const float* const* src, const long long* dst_off, const int* count, float* dst,
                          int n, int max_count, cudaStream_t s);

}  // namespace rtdbs
