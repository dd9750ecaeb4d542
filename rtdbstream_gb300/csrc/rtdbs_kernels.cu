// rtdbs_kernels.cu -- sm_103a kernels of the per-slide streaming DBSCAN path.
//
// One slide = ceil(S / C) grid-update chunk steps followed by one clustering
// step (reference level-9 loop, src/dbscan/dbscan.cpp:2276-2362):
//
//   chunk step (C <= 16384 new points replacing the points of the same slots)
//     k_ingest  new points -> ring slots + cell keys; expired points saved
//               (reference: H2D 2289 + compute_cell_id, src/dbscan/aabb.cu:589-610)
//     k_sort    LSD radix sort of the new and of the expired (cell key, slot)
//               words in runs of 1024, one CTA per run, then k_runmerge
//               ranks the runs into one list (reference: sortByCellIdAndOrder,
//               src/dbscan/thrust_helper.cu:21-29); expired words whose order
//               was kept from their arrival are gathered instead of sorted
//     k_decr    exact -1 on the neighbour counts of every survivor within Eps
//               of an expired point, on the old grid, beside the sort
//     k_merge   old sorted window minus expired plus new, one pass, merge-path
//               tiles (reference: merge_by_cell_id_and_idx,
//               src/dbscan/thrust_helper.cu:31-51)
//     k_build   cell table (tagged open addressing; replaces
//               compute_offsets_of_cells / set_hybrid_spheres_info /
//               optixAccelBuild, src/dbscan/aabb.cu:377-544,
//               src/dbscan/optix.cpp:438-483)
//     k_incr    full count of every new point and exact +1 on its neighbours
//               on the new grid (reference: __raygen__grid/__intersection__grid,
//               src/dbscan/dbscan.cu:155-194,250-270, which recounts all W)
//   or, for first windows and large slides, one build from all W slots:
//     k_ingest_all, k_rad_* (or k_sort), k_fill, k_build, k_count
//   clustering step
//     k_link    cores joined within 32 sorted positions
//     k_union   union-find over core-core pairs by blocks of positions
//               (reference: __raygen__cluster/__intersection__hybrid_radius_sphere,
//               src/dbscan/dbscan.cu:279-321,354-394; find_repres/unite 9-43)
//     k_flatten, k_border (neighbour lists) or k_flatten, k_label (grid scan)
//               labels and ids by slot; border = minimum id of the
//               adjacent clusters (reference: set_label_kernel + post_cluster_t,
//               src/dbscan/aabb.cu:173-196,575-587)
//
// Neighbour predicate: a warp holds 32 candidates in lanes (coalesced float4
// loads of the cell-sorted window) and tests them against home points
// kept in shared memory.  Squared distances use explicitly rounded IEEE
// operations (no FMA contraction; the count passes evaluate two candidates'
// differences and squares with paired FP32 instructions, each half rounded
// the same way), so FP32 mode is bit-identical to the reference's CPU checker
// (src/dbscan/util.cpp:308-316).
#include "rtdbs_internal.h"

#include <atomic>
#include <climits>
#include <cstdint>
#include <type_traits>

namespace rtdbs {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPrecFp64 = 0;
constexpr int kPrecFp32 = 1;

// Programmatic dependent launch: a kernel so launched starts while its
// predecessor runs and waits here, before anything else, for the
// predecessor's end and memory; its own successor may then start likewise.
// (No effect on other launches.)
__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ int slot_of(const float4& p) { return __float_as_int(p.w); }


__device__ __forceinline__ unsigned lanemask_lt(int lane) { return (1u << lane) - 1u; }

// ------------------------------------------------------------------ geometry

__device__ __forceinline__ unsigned long long cell_key(const View& v, float x, float y, float z) {
    unsigned long long key = (unsigned long long)cell_coord(v, 0, x) << v.shift[0];
    if (v.dim > 1) key |= (unsigned long long)cell_coord(v, 1, y) << v.shift[1];
    if (v.dim > 2) key |= (unsigned long long)cell_coord(v, 2, z);
    return key;
}

__device__ __forceinline__ unsigned gen_of_build(long long b) {
    return (unsigned)((b >> 1) % (long long)kGenMod) + 1u;
}

__device__ __forceinline__ int chunk_base_slot(const View& v, int j, int init) {
    const int base = init ? 0 : v.ctl->unit * v.S;
    return base + j * v.chunk;
}

__device__ __forceinline__ void end_slide(const View& v) {
    v.ctl->slide += 1;
    v.ctl->unit = v.ctl->unit + 1 < v.units ? v.ctl->unit + 1 : 0;
}

// The expiring chunk's (key, slot) order is known from the slide that
// brought it in (sorder), so its words need no sort: true once every slot of
// the window arrived by a slide that kept its order (a whole-window build
// keeps none).  Keys do not change while a point is in the window.
__device__ __forceinline__ bool expired_presorted(const View& v, int init) {
    return !init && v.sorder != nullptr && v.ctl->slide >= v.ctl->kept_from + (long long)v.units;
}

// ----------------------------------------------------------------- predicate

template <int DIM>
__device__ __forceinline__ float sqdist32(const float4& a, const float4& b) {
    const float dx = __fsub_rn(a.x, b.x);
    float d = __fmul_rn(dx, dx);
    if (DIM > 1) {
        const float dy = __fsub_rn(a.y, b.y);
        d = __fadd_rn(d, __fmul_rn(dy, dy));
    }
    if (DIM > 2) {
        const float dz = __fsub_rn(a.z, b.z);
        d = __fadd_rn(d, __fmul_rn(dz, dz));
    }
    return d;
}

template <int DIM>
__device__ __forceinline__ double sqdist64(const float4& a, const float4& b) {
    const double dx = __dsub_rn((double)a.x, (double)b.x);
    double d = __dmul_rn(dx, dx);
    if (DIM > 1) {
        const double dy = __dsub_rn((double)a.y, (double)b.y);
        d = __dadd_rn(d, __dmul_rn(dy, dy));
    }
    if (DIM > 2) {
        const double dz = __dsub_rn((double)a.z, (double)b.z);
        d = __dadd_rn(d, __dmul_rn(dz, dz));
    }
    return d;
}

// Neighbour test of two distinct points.  FP32 mode: the reference predicate
// d32 < r2f.  FP64 mode: d32 < lo and d32 >= hi are decided by the float
// value (the band [lo, hi) around Eps^2 bounds the float evaluation's
// rounding error, see oracle_band); everything else in double.
// Per-thread counters: distance tests, those re-decided in FP64, and those
// that found a neighbour.
struct Tally {
    unsigned tests = 0;
    unsigned rechecks = 0;
    unsigned hits = 0;
};

// The decision on d = sqdist32(a, b).
template <int MODE, int DIM>
__device__ __forceinline__ bool nbr_decide(const View& v, float d, const float4& a, const float4& b, Tally& t) {
    ++t.tests;
    bool nb;
    if (MODE == kPrecFp32) {
        nb = d < v.r2f;
    } else if (d < v.lo) {  // (lo and hi are NaN where the filter is off: all in double)
        nb = true;
    } else if (d >= v.hi) {
        nb = false;
    } else {
        ++t.rechecks;
        nb = sqdist64<DIM>(a, b) < v.E;
    }
    t.hits += nb ? 1u : 0u;
    return nb;
}

template <int MODE, int DIM>
__device__ __forceinline__ bool is_nbr(const View& v, const float4& a, const float4& b, Tally& t) {
    return nbr_decide<MODE, DIM>(v, sqdist32<DIM>(a, b), a, b, t);
}

// sqdist32(a, b0) and sqdist32(a, b1) at once: the differences and squares
// with paired FP32 instructions (Blackwell f32x2, each half an IEEE single
// operation rounded to nearest), the sums in scalar, in the same order as
// sqdist32, so both results are bit-identical to it.  (Paired sums are not
// used: the paired multiply-then-add did not round like the two separate
// scalar operations.)
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ void sq_diff2(float a, float b0, float b1, float& s0, float& s1) {
    unsigned long long t, m;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(pack2(a, a)), "l"(pack2(b0, b1)));
    asm("mul.rn.f32x2 %0, %1, %1;" : "=l"(m) : "l"(t));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(m));
}

template <int DIM>
__device__ __forceinline__ void sqdist32x2(const float4& a, const float4& b0, const float4& b1, float& d0,
                                           float& d1) {
    sq_diff2(a.x, b0.x, b1.x, d0, d1);
    if (DIM > 1) {
        float y0, y1;
        sq_diff2(a.y, b0.y, b1.y, y0, y1);
        d0 = __fadd_rn(d0, y0);
        d1 = __fadd_rn(d1, y1);
    }
    if (DIM > 2) {
        float z0, z1;
        sq_diff2(a.z, b0.z, b1.z, z0, z1);
        d0 = __fadd_rn(d0, z0);
        d1 = __fadd_rn(d1, z1);
    }
}

// ---------------------------------------------------------------- cell table

// Home slot of a cell key: the key folded to 32 bits, then Fibonacci
// hashing (pbits <= 31); keys below 2^32 fold to themselves, so the stencil
// lookups of small grids hash in 32-bit arithmetic (table_home32).  The fold
// spreads the upper half first (by an odd constant, MurmurHash3's): folded as it is,
// the first coordinate of a grid with 16 bits an axis fell onto the last one's
// bits, and all cells of a cluster with equal x ^ z on one slot (3-D, keys of 48
// bits, 400k points, a slide in us: MinPts 40, 4 neighbours 489 -> 204; two cells per
// Eps, 40 neighbours, MinPts 3 1126 -> 453).
__device__ __forceinline__ unsigned table_home32(unsigned key, int pbits) {
    return (key * 0x9E3779B1u) >> (32 - pbits);
}

__device__ __forceinline__ unsigned table_home(unsigned long long key, int pbits) {
    return table_home32((unsigned)key ^ (unsigned)(key >> 32) * 0x85EBCA6Bu, pbits);
}

__device__ __forceinline__ unsigned long long tag_of(unsigned long long key, unsigned gen) {
    return ((unsigned long long)gen << kKeyBitsMax) | key;
}

// [start, end) of a cell, (0, 0) if the cell is empty in this generation;
// `home` is the key's home slot.
__device__ __forceinline__ int2 table_find_at(const ulonglong2* T, unsigned pmask, unsigned home,
                                              unsigned long long tag) {
    unsigned s = home;
    const unsigned long long gen = tag >> kKeyBitsMax;
    for (unsigned i = 0; i <= pmask; ++i) {
        const ulonglong2 e = T[s];
        if (e.x == tag) return make_int2((int)(unsigned)e.y, (int)(unsigned)(e.y >> 32));
        if ((e.x >> kKeyBitsMax) != gen) break;  // empty or stale slot ends the probe
        s = (s + 1) & pmask;
    }
    return make_int2(0, 0);
}

// A table entry as four words: tag (low, high), start, end.  The 32-bit key
// path compares words: the tag of a key below 2^32 is the key and gen << 18.
__device__ __forceinline__ uint4 table_entry(const ulonglong2* T, unsigned s) {
    return reinterpret_cast<const uint4*>(T)[s];
}

// table_find_at for a 32-bit key, from slot s on.
__device__ __forceinline__ int2 table_find_from32(const ulonglong2* T, unsigned pmask, unsigned s, unsigned key,
                                                  unsigned ghi) {
    for (unsigned i = 0; i <= pmask; ++i) {
        const uint4 e = table_entry(T, s);
        if (e.x == key && e.y == ghi) return make_int2((int)e.z, (int)e.w);
        if ((e.y ^ ghi) >> (kKeyBitsMax - 32)) break;  // empty or stale slot ends the probe
        s = (s + 1) & pmask;
    }
    return make_int2(0, 0);
}

__device__ __forceinline__ int2 table_find(const ulonglong2* T, unsigned pmask, int pbits,
                                           unsigned long long tag) {
    return table_find_at(T, pmask, table_home(tag & kKeyMask, pbits), tag);
}

// Claims (or finds) the slot of `tag` and stores one half of its range:
// which = 0 -> start, 1 -> end, 2 -> both (value = start, value2 = end).
// Entries of older generations count as free.
__device__ bool table_set(ulonglong2* T, unsigned pmask, int pbits, unsigned long long tag,
                          int which, int value, int value2 = 0) {
    unsigned s = table_home(tag & kKeyMask, pbits);
    const unsigned long long gen = tag >> kKeyBitsMax;
    for (unsigned i = 0; i <= pmask; ++i) {
        unsigned long long* kp = reinterpret_cast<unsigned long long*>(&T[s].x);
        unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(kp);
        for (int t = 0; t < 8; ++t) {
            bool mine = cur == tag;
            if (!mine) {
                if ((cur >> kKeyBitsMax) == gen) break;  // another cell of this generation
                const unsigned long long prev = atomicCAS(kp, cur, tag);
                mine = prev == cur;
                cur = prev;
            }
            if (mine) {
                if (which == 2)
                    T[s].y = (unsigned long long)(unsigned)value | ((unsigned long long)(unsigned)value2 << 32);
                else
                    reinterpret_cast<int*>(&T[s].y)[which] = value;
                return true;
            }
        }
        s = (s + 1) & pmask;
    }
    return false;
}

// Rows of the stencil.  With K cells per Eps along each axis (cell side
// Eps (1 + 2^-12) / K) a point's neighbours lie within K cells per axis, in
// the (2K+1)^DIM cells around its own.  The 2K+1 cells of one row (last axis
// -K..K) have consecutive keys, so a row is one contiguous range of the
// cell-sorted window; the full stencil has (2K+1)^(DIM-1) rows.  The upper
// half (HALF) keeps only the rows whose keys are not below the home cell's --
// the centre row (without its negative cells) and the rows after it in key
// order -- since every position below the home cell is clipped away by a
// pair-once union anyway.
//
// The work kernels take a combined template parameter DK = DIM + 4 (K - 1):
// DK 1..3 for one cell per Eps, 5..7 for two.
template <int DIM, bool HALF, int K = 1>
struct Stencil {
    static constexpr int kW = 2 * K + 1;  // cells per row
    static constexpr int kAllRows = DIM == 1 ? 1 : (DIM == 2 ? kW : kW * kW);
    static constexpr int kFirst = HALF ? (kAllRows - 1) / 2 : 0;  // first row kept
    static constexpr int kRows = kAllRows - kFirst;
};
constexpr int kMaxRows = 25;  // (2K+1)^2 rows for K = 2 in 3-D

// Row ranges of the stencil around `key`, computed by a group of G lanes
// (the whole warp, or each 16-lane half for its own key; `lane` counts within
// the group; a lane looks up one to four cells).  On return group lane
// r < kRows holds row r as [rs, re) (empty rows: rs == re).
template <int DIM, int K = 1, int G = 32>
__device__ __forceinline__ void row_ranges(const View& v, const ulonglong2* T, unsigned gen,
                                           unsigned long long key, int lane, int& rs, int& re) {
    using St = Stencil<DIM, false, K>;
    constexpr int kW = St::kW;
    constexpr int kSlots = kW * St::kRows;           // cell slots, row by row
    constexpr int kPer = (kSlots + G - 1) / G;       // cells per lane
    static_assert(kPer <= 4 && St::kRows <= G, "stencil too large for the lane group");
    int2 rg[kPer];
    if (v.key_bits <= 31) {
        // keys, cell coordinates and extents fit 32 bits: the lookups in
        // 32-bit arithmetic (coordinates wrap below zero, so one unsigned
        // comparison bounds each axis)
        const unsigned k32 = (unsigned)key;
        const int s0 = v.shift[0], s1 = v.shift[1];
        const unsigned c2 = k32 & ((1u << s1) - 1u);
        const unsigned c1 = (k32 >> s1) & ((1u << (s0 - s1)) - 1u);
        const unsigned c0 = k32 >> s0;
        const unsigned e0 = (unsigned)v.ext[0], e1 = (unsigned)v.ext[1], e2 = (unsigned)v.ext[2];
        const unsigned ghi = gen << (kKeyBitsMax - 32);
        uint4 e[kPer];  // first probes, issued together
        unsigned nks[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            rg[k] = make_int2(0, 0);
            e[k] = make_uint4(0, 0, 0, 0);  // no generation
            nks[k] = 0;
            const int cs = lane + k * G;
            const int row = cs / kW, d_last = cs % kW - K;
            if (cs < kSlots) {
                unsigned q0 = c0, q1 = c1, q2 = c2;
                if (DIM == 1) {
                    q0 += (unsigned)d_last;
                } else if (DIM == 2) {
                    q0 += (unsigned)(row - K);
                    q1 += (unsigned)d_last;
                } else {
                    q0 += (unsigned)(row / kW - K);
                    q1 += (unsigned)(row % kW - K);
                    q2 += (unsigned)d_last;
                }
                if (q0 < e0 && q1 < e1 && q2 < e2) {
                    nks[k] = (q0 << s0) | (q1 << s1) | q2;
                    e[k] = table_entry(T, table_home32(nks[k], v.pbits));
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if ((e[k].y ^ ghi) >> (kKeyBitsMax - 32)) continue;
            rg[k] = e[k].x == nks[k]
                        ? make_int2((int)e[k].z, (int)e[k].w)
                        : table_find_from32(T, v.pmask, (table_home32(nks[k], v.pbits) + 1) & v.pmask, nks[k], ghi);
        }
    } else {
    const long long c2 = (long long)(key & ((1ull << v.shift[1]) - 1ull));
    const long long c1 = (long long)((key >> v.shift[1]) & ((1ull << (v.shift[0] - v.shift[1])) - 1ull));
    const long long c0 = (long long)(key >> v.shift[0]);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        rg[k] = make_int2(0, 0);
        const int cs = lane + k * G;                                  // = kW * row + cell
        const int row = cs / kW, d_last = cs % kW - K;
        if (cs < kSlots) {
            long long q0 = c0, q1 = c1, q2 = c2;
            if (DIM == 1) {
                q0 += d_last;
            } else if (DIM == 2) {
                q0 += row - K;
                q1 += d_last;
            } else {
                q0 += row / kW - K;
                q1 += row % kW - K;
                q2 += d_last;
            }
            const bool ok = q0 >= 0 && q0 < v.ext[0] && q1 >= 0 && q1 < v.ext[1] && q2 >= 0 && q2 < v.ext[2];
            if (ok) {
                const unsigned long long nk = ((unsigned long long)q0 << v.shift[0]) |
                                              ((unsigned long long)q1 << v.shift[1]) | (unsigned long long)q2;
                rg[k] = table_find(T, v.pmask, v.pbits, tag_of(nk, gen));
            }
        }
    }
    }
    int s = INT_MAX, e = INT_MIN;
#pragma unroll
    for (int k = 0; k < kW; ++k) {
        const int cs = min(kW * lane + k, kSlots - 1);   // slot of row `lane`'s cell k
        const int src = cs % G, which = cs / G;
        int a = 0, b = 0;
#pragma unroll
        for (int w = 0; w < kPer; ++w) {
            const int aw = __shfl_sync(kFull, rg[w].x, src, G);
            const int bw = __shfl_sync(kFull, rg[w].y, src, G);
            if (w == which) {
                a = aw;
                b = bw;
            }
        }
        if (b > a) {
            s = min(s, a);
            e = max(e, b);
        }
    }
    if (e == INT_MIN) s = e = 0;
    rs = s;
    re = e;
}

// One row of the stencil around a cell, looked up by one lane: kept row
// `row` of Stencil<DIM, HALF, K> as a range of sorted positions (empty: 0, 0).
// The first probes of the row's cells are issued together.
template <int DIM, bool HALF, int K>
__device__ __forceinline__ int2 row_range_lane32(const View& v, const ulonglong2* T, unsigned gen, unsigned key,
                                                 int row) {
    using St = Stencil<DIM, HALF, K>;
    constexpr int kW = St::kW;
    const int arow = St::kFirst + row;
    const bool centre = HALF && row == 0;  // its cells below the home cell are not kept
    const int s0 = v.shift[0], s1 = v.shift[1];
    // coordinates wrap below zero, so one unsigned comparison bounds each axis
    unsigned ql, el, rowkey;  // along the row: coordinate and extent; the rest of the key
    int sl;
    bool in = true;
    if (DIM == 1) {
        ql = key >> s0;
        el = (unsigned)v.ext[0];
        rowkey = 0;
        sl = s0;
    } else if (DIM == 2) {
        const unsigned q0 = (key >> s0) + (unsigned)(arow - K);
        in = q0 < (unsigned)v.ext[0];
        ql = (key >> s1) & ((1u << (s0 - s1)) - 1u);
        el = (unsigned)v.ext[1];
        rowkey = q0 << s0;
        sl = s1;
    } else {
        const unsigned q0 = (key >> s0) + (unsigned)(arow / kW - K);
        const unsigned q1 = ((key >> s1) & ((1u << (s0 - s1)) - 1u)) + (unsigned)(arow % kW - K);
        in = q0 < (unsigned)v.ext[0] && q1 < (unsigned)v.ext[1];
        ql = key & ((1u << s1) - 1u);
        el = (unsigned)v.ext[2];
        rowkey = (q0 << s0) | (q1 << s1);
        sl = 0;
    }
    if (!in) return make_int2(0, 0);
    const unsigned ghi = gen << (kKeyBitsMax - 32);
    uint4 e[kW];
#pragma unroll
    for (int k = 0; k < kW; ++k) {
        const unsigned q = ql + (unsigned)(k - K);
        e[k] = make_uint4(0, 0, 0, 0);  // no generation
        if (q < el && !(centre && k < K)) e[k] = table_entry(T, table_home32(rowkey | (q << sl), v.pbits));
    }
    int rs = INT_MAX, re = 0;
    if constexpr (DIM == 3 && K == 2) {
        // the probes past the first slots side by side as well.  One cell's
        // after the other, in a table half full, held up the label pass and
        // the union (130k points, MinPts 40: label 286 -> 184 us with blocks of
        // 16; pools of such streams 643 -> 478 and 2845 -> 1682 us a round).  In 1-D
        // and 2-D, with fewer rows and fuller cells, nothing is gained
        unsigned open = 0;  // cells whose first slot holds another cell
#pragma unroll
        for (int k = 0; k < kW; ++k)
            if (!((e[k].y ^ ghi) >> (kKeyBitsMax - 32)) && e[k].x != (rowkey | ((ql + (unsigned)(k - K)) << sl)))
                open |= 1u << k;
        for (unsigned step = 1; open && step <= v.pmask; ++step) {
#pragma unroll
            for (int k = 0; k < kW; ++k)
                if ((open >> k) & 1u)
                    e[k] = table_entry(T, (table_home32(rowkey | ((ql + (unsigned)(k - K)) << sl), v.pbits) + step) &
                                              v.pmask);
#pragma unroll
            for (int k = 0; k < kW; ++k)
                if (((e[k].y ^ ghi) >> (kKeyBitsMax - 32)) || e[k].x == (rowkey | ((ql + (unsigned)(k - K)) << sl)))
                    open &= ~(1u << k);
        }
#pragma unroll
        for (int k = 0; k < kW; ++k) {
            if (((open >> k) & 1u) || ((e[k].y ^ ghi) >> (kKeyBitsMax - 32)) || (int)e[k].w <= (int)e[k].z) continue;
            rs = min(rs, (int)e[k].z);
            re = max(re, (int)e[k].w);
        }
    } else {
#pragma unroll
        for (int k = 0; k < kW; ++k) {
            if ((e[k].y ^ ghi) >> (kKeyBitsMax - 32)) continue;  // out of the grid, or an empty or stale slot
            const unsigned nk = rowkey | ((ql + (unsigned)(k - K)) << sl);
            int2 c = make_int2((int)e[k].z, (int)e[k].w);
            if (e[k].x != nk)
                c = table_find_from32(T, v.pmask, (table_home32(nk, v.pbits) + 1) & v.pmask, nk, ghi);
            if (c.y > c.x) {
                rs = min(rs, c.x);
                re = max(re, c.y);
            }
        }
    }
    return re > 0 ? make_int2(rs, re) : make_int2(0, 0);
}

template <int DIM, bool HALF, int K>
__device__ __noinline__ int2 row_range_lane64(const View& v, const ulonglong2* T, unsigned gen,
                                              unsigned long long key, int row) {
    using St = Stencil<DIM, HALF, K>;
    constexpr int kW = St::kW;
    const int arow = St::kFirst + row;
    const int s0 = v.shift[0], s1 = v.shift[1];
    long long q[3] = {(long long)(key >> s0), (long long)((key >> s1) & ((1ull << (s0 - s1)) - 1ull)),
                      (long long)(key & ((1ull << s1) - 1ull))};
    if (DIM == 2) q[0] += arow - K;
    if (DIM == 3) {
        q[0] += arow / kW - K;
        q[1] += arow % kW - K;
    }
    const long long mid = q[DIM - 1];
    int rs = INT_MAX, re = 0;
    for (int k = HALF && row == 0 ? K : 0; k < kW; ++k) {
        q[DIM - 1] = mid + (k - K);
        bool in = true;
        for (int a = 0; a < DIM; ++a) in = in && q[a] >= 0 && q[a] < v.ext[a];
        if (!in) continue;
        const unsigned long long nk = ((unsigned long long)q[0] << s0) | ((unsigned long long)q[1] << s1) |
                                      (unsigned long long)q[2];
        const int2 c = table_find(T, v.pmask, v.pbits, tag_of(nk, gen));
        if (c.y > c.x) {
            rs = min(rs, c.x);
            re = max(re, c.y);
        }
    }
    return re > 0 ? make_int2(rs, re) : make_int2(0, 0);
}

template <int DIM, bool HALF, int K>
__device__ __forceinline__ int2 row_range_lane(const View& v, const ulonglong2* T, unsigned gen,
                                               unsigned long long key, int row) {
    if (v.key_bits <= 31) return row_range_lane32<DIM, HALF, K>(v, T, gen, (unsigned)key, row);
    return row_range_lane64<DIM, HALF, K>(v, T, gen, key, row);
}

// The group's row ranges (group lanes 0..ROWS-1) laid end to end: candidate
// idx in [0, total) lives at sorted position start[r] + idx - pre[r] for the row
// r with pre[r] <= idx < pre[r+1].
// Concatenating the rows keeps the candidate chunks full.  Called by the
// whole warp; G-lane groups work independently.
template <int ROWS, int G = 32>
__device__ __forceinline__ int candidate_stream(int rs, int re, int lane, int* sstart, int* spre) {
    const int len = lane < ROWS ? re - rs : 0;
    int incl = len;
#pragma unroll
    for (int o = 1; o < (ROWS > 16 ? 32 : 16); o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o, G);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(kFull, incl, ROWS - 1, G);
    __syncwarp();
    if (lane < ROWS) {
        sstart[lane] = rs;
        spre[lane] = incl - len;
    }
    if (lane == 0) spre[ROWS] = total;
    __syncwarp();
    return total;
}

// Sorted position of candidate idx; r is the lane's row cursor (rows only
// advance as idx grows).
__device__ __forceinline__ int stream_pos(int idx, int& r, const int* sstart, const int* spre) {
    while (idx >= spre[r + 1]) ++r;
    return sstart[r] + idx - spre[r];
}

// ---------------------------------------------------------------- union-find

// Root of v with intermediate pointer jumping (each visited node is pointed
// at its grandparent).  Parents only ever decrease, so the walk terminates.
__device__ __forceinline__ int uf_find(int* parent, int v) {
    volatile int* P = parent;
    int curr = P[v];
    if (curr != v) {
        int next, prev = v;
        while (curr > (next = P[curr])) {
            P[prev] = next;
            prev = curr;
            curr = next;
        }
    }
    return curr;
}

// Lock-free union of the sets of a and b, each an ancestor of one of the two
// points (a cached or freshly found root; it need not still be a root).  The
// larger of the two is hooked under the smaller with one atomicCAS, which only
// succeeds on a root; on failure the walk resumes from the root that the CAS
// revealed.  max(a, b) falls every round, so the loop ends, and parents only
// ever point to smaller slots, so every root is the minimum slot of its set.
// Returns an ancestor of both points afterwards.
__device__ __forceinline__ int uf_hook(int* parent, int a, int b, int& err) {
    for (int it = 0; it < kMaxIter; ++it) {
        if (a == b) return a;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(&parent[a], a, b);
        if (old == a) return b;
        a = uf_find(parent, old);
    }
    err |= kErrUnionIter;
    return a < b ? a : b;
}

// Warp totals of the counters into the control block; pass 0 = count passes
// (core identification), 1 = clustering scans.
__device__ __forceinline__ void flush_stats(const View& v, const Tally& t, int err, int lane, int pass) {
    const unsigned r = __reduce_add_sync(kFull, t.rechecks);
    const unsigned n = __reduce_add_sync(kFull, t.tests);
    const unsigned h = __reduce_add_sync(kFull, t.hits);
    const int e = __reduce_or_sync(kFull, (unsigned)err);
    if (lane == 0) {
        const int k = (threadIdx.x >> 5) & 7;
        if (r) atomicAdd(&v.ctl->band_rechecks, (unsigned long long)r);
        if (n) atomicAdd(&v.ctl->ptests[pass][k], (unsigned long long)n);
        if (h) atomicAdd(&v.ctl->phits[pass][k], (unsigned long long)h);
        if (e) atomicOr(&v.ctl->err, e);
    }
}

// Most distance tests of one query over the warp's lane groups of G lanes
// (each lane's `tests` counts its own query only) into Ctl::qmax.
template <int G>
__device__ __forceinline__ void flush_query_max(const View& v, unsigned tests, int lane) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) tests += __shfl_xor_sync(kFull, tests, o);
#pragma unroll
    for (int o = G; o < 32; o <<= 1) tests = max(tests, __shfl_xor_sync(kFull, tests, o));
    if (lane == 0 && tests) atomicMax(&v.ctl->qmax[(threadIdx.x >> 5) & 7], (int)tests);
}

// ------------------------------------------------------- neighbour lists
// Every non-core point keeps the slots of its neighbours (at most MinPts - 2
// besides itself) in a fixed list by slot, maintained from the same distance
// tests that keep the counts exact: an expired neighbour is removed in the
// decrement pass, a new one appended in the increment pass.  A point that
// becomes core stops keeping its list (ntrack 0); one that is below MinPts
// without a list once the slide's counts are final (it lost core status) gets
// its list rebuilt by one scan.  The label pass then reads lists instead of
// scanning the grid.

// First index of `x` among the four entries of e (base: index of e.x), or -1.
__device__ __forceinline__ int find4(const int4& e, int x, int base) {
    return e.x == x ? base : e.y == x ? base + 1 : e.z == x ? base + 2 : e.w == x ? base + 3 : -1;
}

// Appends slot p to q's list (q tracked); a full list means q has reached
// MinPts, so it stops being kept.  A list row is read 16 bytes at a time
// from L2 (other SMs may have just written it).  The append claims the first
// free entry by CAS and looks again if another point took it first; a row
// still contended after a few looks also stops being kept (the flatten pass
// rebuilds it).  Padding entries past the cap stay -1 and are never claimed.
__device__ __forceinline__ void list_append(const View& v, int q, int p) {
    int* L = v.nlist + (size_t)q * v.list_stride;
    const int4* L4 = reinterpret_cast<const int4*>(L);
    const int n4 = v.list_stride >> 2;
    for (int look = 0; look < 4; ++look) {
        int k = -1;
        for (int b = 0; b < n4 && k < 0; ++b) k = find4(__ldcg(L4 + b), -1, 4 * b);
        if (k < 0 || k >= v.list_cap) break;
        if (atomicCAS(&L[k], -1, p) == -1) return;
    }
    v.ntrack[q] = 0;
}

// Removes slot p from q's list (q tracked; only this thread removes p).
__device__ __forceinline__ void list_remove(const View& v, int q, int p) {
    int* L = v.nlist + (size_t)q * v.list_stride;
    const int4* L4 = reinterpret_cast<const int4*>(L);
    const int n4 = v.list_stride >> 2;
    for (int b = 0; b < n4; ++b) {
        const int k = find4(__ldcg(L4 + b), p, 4 * b);
        if (k >= 0) {
            L[k] = -1;
            return;
        }
    }
    atomicOr(&v.ctl->err, kErrList);
}

// Called by the whole warp; each group of G lanes (gl = lane within the
// group) adds its lanes' neighbour slots (nb) to its own buffer in lane
// order; returns the group's new number found (entries past cap are
// dropped, the list is then not kept anyway).
template <int G = 32>
__device__ __forceinline__ int list_collect(bool nb, int qs, int nfound, int cap, int* buf, int lane) {
    const unsigned all = __ballot_sync(kFull, nb);
    const int gl = lane & (G - 1);
    const unsigned m = G == 32 ? all : (all >> (lane - gl)) & ((1u << G) - 1u);
    const int at = nfound + __popc(m & lanemask_lt(gl));
    if (nb && at < cap) buf[at] = qs;
    return nfound + __popc(m);
}

// Called by the whole warp; a group with a point (`has`) writes slot a's
// list from its buffer (kept iff a is not core); the row's padding past
// list_cap stays -1.
template <int G = 32>
__device__ __forceinline__ void list_store(const View& v, int a, int nfound, const int* buf, int lane,
                                           bool has = true) {
    __syncwarp();
    const int gl = lane & (G - 1);
    if (has) {
        const bool keep = nfound + 1 < v.min_pts;
        int* L = v.nlist + (size_t)a * v.list_stride;
        if (keep)
            for (int k = gl; k < v.list_stride; k += G) L[k] = k < nfound ? buf[k] : -1;
        if (gl == 0) v.ntrack[a] = keep ? 1 : 0;
    }
    __syncwarp();
}

// ------------------------------------------------------------------- kernels

// ------------------------------------------------------ forest reuse
// A component of the previous clustering that lost no core this slide (no
// core expired, no core fell below MinPts) is still connected: all its
// cores and the edges between them remain.  Its cores start the union as
// one set under the old root (still its minimum slot), with that root as
// their hint, so pairs inside it are skipped by hint equality; every other
// core starts as a singleton.  The union still visits every core pair, so
// merges through new cores and splits of damaged components come out exactly
// as in a union from scratch.  Used with neighbour lists, where k_border
// leaves the previous labels and ids by slot and resets the forest.
//
// No pass of its own: the old root of every core lost this slide is marked
// damaged as the loss happens -- an expired core in the ingest, a core whose
// count falls below MinPts in the decrement (a count that falls below and
// rises again within the slide only marks a component that did not need it;
// it is then re-united from scratch, still exactly) -- and the merge, which
// rewrites every position, starts each core under its old root or alone
// (start_hint); the increment then sets the hints of new points and of points
// it lifts to MinPts.  label/cid hold the previous clustering until the
// border pass ends the slide.

// Reuse is skipped for 15 slides after a slide where fewer than 1 in 16 of
// the window's points joined a reused component (streams whose expiries
// touch every cluster), then tried again.
constexpr int kReuseRetry = 15;

__device__ __forceinline__ bool damage_on(const View& v) {
    return v.list_cap >= 0 && v.ctl->prev_ok && v.ctl->reuse_skip <= 0;
}

// Root hint a position starts the union with: -1 for a non-core point; the
// old root `prev` of a core of an intact component (the root the point had
// at the last clustering, carried with it by the merges; -1 for a point that
// was not core then); else its own slot.  Counts 1 in `reused` for a
// reused core.  The parents need no change: the union and the flatten only
// ever start from a point's hint, and the border pass leaves every parent at
// its own slot.
__device__ __forceinline__ int start_hint(const View& v, int s, int cnt, int prev, bool reuse,
                                          unsigned& reused) {
    if (cnt < v.min_pts) return -1;
    if (reuse && prev >= 0 && !__ldg(&v.damaged[prev])) {
        ++reused;
        return prev;
    }
    return s;
}

__device__ __forceinline__ void mark_damage(const View& v, int slot) {
    if (v.label[slot] == 0) v.damaged[v.cid[slot]] = 1;
}

// New points of chunk j -> ring slots [el, el+c): float4 + cell key; the
// points they replace are kept for the decrement pass.
// The slide's first ingest (an input given) leaves the slide's pointers in the
// control block for the later ones and the label pass.
__device__ __forceinline__ void ingest_body(const View& v, int j, int c, int init, int stg_off, const SlideIO& io,
                                            int bx) {
    const float* input = io.input ? io.input : v.ctl->input;
    if (bx == 0 && threadIdx.x == 0) {
        v.ctl->b += 1;  // no reader in this kernel
        if (io.input) {
            v.ctl->input = io.input;  // (its readers here have the argument)
            v.ctl->out_label = io.label;
            v.ctl->out_cid = io.cid;
        }
    }
    const int k = bx * blockDim.x + threadIdx.x;
    if (k >= c) return;
    const int slot = chunk_base_slot(v, j, init) + k;
    if (!init) {
        v.xpt[k] = v.ring[slot];
        const unsigned long long old = v.kslot[slot];
        v.xkey[k] = old;
        v.xsort[k] = (old << kOffBits) | (unsigned long long)k;
        if (damage_on(v)) mark_damage(v, slot);  // an expired core
    }
    const float* p = input + (size_t)(stg_off + k) * v.dim;
    const float x = p[0];
    const float y = v.dim > 1 ? p[1] : 0.0f;
    const float z = v.dim > 2 ? p[2] : 0.0f;
    v.ring[slot] = make_float4(x, y, z, __int_as_float(slot));
    const unsigned long long key = cell_key(v, x, y, z);
    v.kslot[slot] = key;
    v.nsort[k] = (key << kOffBits) | (unsigned long long)k;
}

__global__ void k_ingest(View v, int j, int c, int init, int stg_off, SlideIO io) {
    pdl_wait();
    ingest_body(v, j, c, init, stg_off, io, blockIdx.x);
}

// Exclusive scan of one value per thread over a 1024-thread block.
__device__ __forceinline__ unsigned block_excl_scan_1024(unsigned val, unsigned* wsum) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned incl = val;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
        const unsigned x = wsum[lane];
        unsigned xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(kFull, xi, o);
            if (lane >= o) xi += t;
        }
        wsum[lane] = xi - x;
    }
    __syncthreads();
    const unsigned r = wsum[w] + incl - val;
    __syncthreads();
    return r;
}

// Stable LSD radix sort (digits of up to 9 bits over the key bits of the sort word) of
// the chunk's words in independent runs of kSortRun: block (r, 0) sorts run r
// of the new words, block (r, 1) run r of the expired ones, one word per
// thread.  Warp-level multisplit: lanes with equal digits are ranked from
// a ballot per digit bit; per-(digit, warp) counters are scanned in digit-major order
// so the order of equal digits is the item order.  Bound by latency (barriers
// and shared memory); with 8-bit digits and the run merge searching one run
// after the other, 10 runs took 29.6 us instead of 23.6 (25-bit keys), one run
// 12.3 instead of 10.2 (18-bit keys).
struct SortSmem {
    unsigned long long buf[kSortRun];
    uint4 whist[(1 << kSortBits) * 32 * 2 / 16];  // 16-bit counters [digit][warp]
    unsigned wsum[32];
};

// single: the chunk is one run (c <= kSortRun), so the sorted run is the
// final list: it goes straight to nword / xword (and presorted expired words
// are gathered here), and no run merge follows.
__device__ __forceinline__ void sort_body(const View& v, int j, int c, int init, int bx, int by, SortSmem& sm,
                                          bool single) {
    unsigned long long* buf = sm.buf;
    unsigned short* whist = reinterpret_cast<unsigned short*>(sm.whist);
    unsigned* wsum = sm.wsum;
    const int which = by;
    if (which == 1 && init) return;
    if (which == 1 && expired_presorted(v, init)) {
        if (single) {  // the run merge's gather of the kept order
            const int i = threadIdx.x;
            if (i >= c) return;
            const int k = v.sorder[chunk_base_slot(v, j, 0) + i];
            if (k < 0 || k >= c) {
                atomicOr(&v.ctl->err, kErrChunk);
                v.xword[i] = ~0ull;
                return;
            }
            v.xword[i] = v.xsort[k];
        }
        return;
    }
    const int r0 = bx * kSortRun;
    const int len = min(kSortRun, c - r0);
    if (len <= 0) return;
    unsigned long long* run = (which ? v.xsort : v.nsort) + r0;  // sorted in place
    unsigned long long* dst = single ? (which ? v.xword : v.nword) : run;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const unsigned lt = lanemask_lt(lane);
    unsigned long long it = tid < len ? run[tid] : ~0ull;
    for (int pass = 0; pass < v.sort_passes; ++pass) {
        const int shift = kOffBits + v.sort_bits * pass;
#pragma unroll
        for (int k = 0; k < (int)(sizeof(sm.whist) / sizeof(uint4)) / kSortRun; ++k)
            sm.whist[tid + k * kSortRun] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        const unsigned d = (unsigned)(it >> shift) & ((1u << v.sort_bits) - 1u);
        unsigned peers = kFull;
        for (int bit = 0; bit < v.sort_bits; ++bit) {
            const unsigned bm = __ballot_sync(kFull, (d >> bit) & 1u);
            peers &= ((d >> bit) & 1u) ? bm : ~bm;
        }
        const unsigned rank = __popc(peers & lt);
        if (rank == 0) whist[d * 32 + w] = (unsigned short)__popc(peers);
        __syncthreads();
        // each thread's 16 consecutive counters, scanned in place
        uint4 q[2] = {sm.whist[2 * tid], sm.whist[2 * tid + 1]};
        unsigned* c = &q[0].x;
        unsigned sum = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += (c[k] & 0xffffu) + (c[k] >> 16);
        unsigned pre = block_excl_scan_1024(sum, wsum);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const unsigned lo = c[k] & 0xffffu, hi = c[k] >> 16;
            c[k] = pre | ((pre + lo) << 16);
            pre += lo + hi;
        }
        sm.whist[2 * tid] = q[0];
        sm.whist[2 * tid + 1] = q[1];
        __syncthreads();
        buf[whist[d * 32 + w] + rank] = it;
        __syncthreads();
        it = buf[tid];
    }
    if (tid < len) dst[tid] = it;
}

__global__ void __launch_bounds__(kSortRun) k_sort(View v, int j, int c, int init, int single) {
    pdl_wait();
    __shared__ SortSmem sm;
    sort_body(v, j, c, init, blockIdx.x, blockIdx.y, sm, single != 0);
}

// Merges the sorted runs of kSortRun words into one sorted list: a word's
// rank is its index in its run plus the words below it in every other run
// (words are distinct, so ranks are too).  Block (r, y) ranks run r of the
// new (y = 0) or expired (y = 1) words; all c words are staged in shared
// memory first, so the binary searches stay on chip.  Presorted expired
// words are gathered in their kept order instead.
__device__ __forceinline__ void runmerge_body(const View& v, int j, int c, int init, int bx, int by,
                                              unsigned long long* words) {
    const int which = by;
    if (which == 1 && init) return;
    if (which == 1 && expired_presorted(v, init)) {
        const int i = bx * kSortRun + threadIdx.x;
        if (i >= c) return;
        const int k = v.sorder[chunk_base_slot(v, j, 0) + i];
        if (k < 0 || k >= c) {
            atomicOr(&v.ctl->err, kErrChunk);
            v.xword[i] = ~0ull;
            return;
        }
        v.xword[i] = v.xsort[k];
        return;
    }
    const unsigned long long* runs = which ? v.xsort : v.nsort;
    unsigned long long* out = which ? v.xword : v.nword;
    const int nruns = (c + kSortRun - 1) / kSortRun;
    for (int i = threadIdx.x; i < nruns * kSortRun; i += blockDim.x) words[i] = i < c ? runs[i] : ~0ull;
    __syncthreads();
    const int own = bx;
    const int i = own * kSortRun + threadIdx.x;
    if (i >= c) return;
    const unsigned long long w = words[i];
    int rank = threadIdx.x;
    // four runs at a time, their searches side by side (the last run is filled
    // up with words above all)
    for (int r0 = 0; r0 < nruns; r0 += 4) {
        const unsigned long long* run[4];
        int at[4] = {0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < 4; ++u) run[u] = words + min(r0 + u, nruns - 1) * kSortRun;
#pragma unroll
        for (int step = kSortRun / 2; step > 0; step >>= 1)
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (run[u][at[u] + step - 1] < w) at[u] += step;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (r0 + u >= nruns || r0 + u == own) continue;
            rank += at[u] + (run[u][at[u]] < w ? 1 : 0);
        }
    }
    out[rank] = w;
}

__global__ void __launch_bounds__(kSortRun) k_runmerge(View v, int j, int c, int init) {
    pdl_wait();
    extern __shared__ unsigned long long words[];
    runmerge_body(v, j, c, init, blockIdx.x, blockIdx.y, words);
}

// Count passes of a stream slid alone: blocks of 128 threads, 9 per SM (56
// registers), so that the 5,000 warps of 10,000 queries are resident at once.
// They are one wave of dependent loads, bound by latency.  With 256-thread
// blocks, 5 per SM, a candidate pair's loads only when it was worked on and the
// table probes of a lane one after the other, decrement and increment took 31 +
// 39 us on 200k trajectories (now 26 + 35), 30 + 35 on 100k prices (26 + 29),
// 24 + 23 on 1M walkers (21 + 25); 8 and 10 blocks per SM: walkers 27 + 27 and 22
// + 25, trajectories 26 + 33 and 32 + 41.
constexpr int kQueryThreads = 128;
constexpr int kQueryBlocks = 9;

// -1 on the count of every surviving neighbour of each expired point (old grid).
// G lanes scan one query point's neighbourhood (View::qlanes): 16 (two points
// per warp, so two queries' dependent loads overlap) or 32; the 25 rows of the
// two-cells-per-Eps stencil need the whole warp.

constexpr int kFlattenQueue = 128;  // list rebuilds a flatten block queues for its warps to share

struct StreamSmem {
    int rstart[8][kMaxRows], rpre[8][kMaxRows + 1];
    int grstart[8][2][kMaxRows], grpre[8][2][kMaxRows + 1];  // per lane group (count passes)
    int nbuf[8][kListCap];
    int gnbuf[8][2][kListCap];
    int queue[kFlattenQueue];  // k_flatten: positions of the block whose lists are rebuilt
    int nq;
};

template <int MODE, int DK, int G, bool AHEAD>
__device__ __forceinline__ void decr_g(const View& v, int j, int c, int bx, StreamSmem& sm) {
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;  // dimension, cells per Eps
    constexpr int kPerWarp = 32 / G;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int grp = lane / G, gl = lane % G;
    const int gw = (bx * blockDim.x + threadIdx.x) >> 5;
    if (gw * kPerWarp >= c) return;
    const int qi = gw * kPerWarp + grp;
    bool has = qi < c;
    int* rstart = sm.grstart[wib][grp];
    int* rpre = sm.grpre[wib][grp];
    const long long b = v.ctl->b;
    const int old = (int)((b - 1) & 1);
    const unsigned gen = gen_of_build(b - 1);
    const int el = chunk_base_slot(v, j, 0);
    // Expired points with their kept keys (the sort words are being sorted):
    // the pass does not wait for the chunk's sort, and runs beside it.  Taken
    // in their kept (key, slot) order where there is one, so neighbouring warps
    // read the same cells.
    int k = qi;
    if (has && expired_presorted(v, 0)) {
        k = v.sorder[el + qi];
        if (k < 0 || k >= c) {
            atomicOr(&v.ctl->err, kErrChunk);
            has = false;
        }
    }
    const float4 xp = has ? v.xpt[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned long long key = has ? v.xkey[k] : 0ull;
    int rs, re;
    row_ranges<DIM, K, G>(v, v.table[old], gen, key, gl, rs, re);
    int total = candidate_stream<Stencil<DIM, false, K>::kRows, G>(rs, re, gl, rstart, rpre);
    if (!has) total = 0;
    const float4* spt = v.spt[old];
    int* scnt = v.scnt[old];
    const bool lists = v.list_cap >= 0;
    const bool damage = damage_on(v);
    const int xs = slot_of(xp);
    Tally tally;
    int r = 0;
    // Two candidates per lane and trip (idx and idx + G): their loads are in
    // flight together and one paired distance evaluation serves both.  AHEAD
    // (streams slid alone, whose passes are one wave of dependent loads): the
    // next trip's loads are issued before this one is worked on.
    int npos0 = 0, npos1 = 0, ncnt0 = 0, ncnt1 = 0;
    float4 nq0 = make_float4(0.f, 0.f, 0.f, 0.f), nq1 = nq0;
    auto fetch = [&](int at) {
        npos0 = stream_pos(at, r, rstart, rpre);
        npos1 = at + G < total ? stream_pos(at + G, r, rstart, rpre) : npos0;
        nq0 = spt[npos0];
        nq1 = spt[npos1];
        // counts only fall here: >= MinPts means no list kept
        ncnt0 = scnt[npos0];
        ncnt1 = scnt[npos1];
    };
    if (AHEAD && gl < total) fetch(gl);
    for (int idx = gl; idx < total; idx += 2 * G) {
        const bool two = idx + G < total;
        if (!AHEAD) fetch(idx);
        const int pos0 = npos0, pos1 = npos1, cnt0 = ncnt0, cnt1 = ncnt1;
        const float4 q0 = nq0, q1 = nq1;
        if (AHEAD && idx + 2 * G < total) fetch(idx + 2 * G);
        const int qs0 = slot_of(q0), qs1 = slot_of(q1);
        float d0, d1;
        sqdist32x2<DIM>(xp, q0, q1, d0, d1);
        // counts only fall here: one read below MinPts cannot cross it, so
        // only the others need the count the decrement leaves
        if ((qs0 < el || qs0 >= el + c) && nbr_decide<MODE, DIM>(v, d0, xp, q0, tally)) {
            if (!damage || cnt0 < v.min_pts)
                atomicSub(&scnt[pos0], 1);
            else if (atomicSub(&scnt[pos0], 1) == v.min_pts)
                mark_damage(v, qs0);  // a core falls below MinPts
            if (lists && cnt0 < v.min_pts && v.ntrack[qs0] == 1) list_remove(v, qs0, xs);
        }
        if (two && (qs1 < el || qs1 >= el + c) && nbr_decide<MODE, DIM>(v, d1, xp, q1, tally)) {
            if (!damage || cnt1 < v.min_pts)
                atomicSub(&scnt[pos1], 1);
            else if (atomicSub(&scnt[pos1], 1) == v.min_pts)
                mark_damage(v, qs1);
            if (lists && cnt1 < v.min_pts && v.ntrack[qs1] == 1) list_remove(v, qs1, xs);
        }
    }
    flush_query_max<G>(v, tally.tests, lane);
    flush_stats(v, tally, 0, lane, 0);
}

// The count passes' lane group, chosen per stream at run time (uniform per
// launch): 16 or 32 lanes with one cell per Eps, 32 with two.
template <int MODE, int DK, bool AHEAD>
__device__ __forceinline__ void decr_body(const View& v, int j, int c, int bx, StreamSmem& sm) {
    if constexpr ((DK >> 2) == 0) {
        if (v.qlanes == 16) {
            decr_g<MODE, DK, 16, AHEAD>(v, j, c, bx, sm);
            return;
        }
    }
    decr_g<MODE, DK, 32, AHEAD>(v, j, c, bx, sm);
}

template <int MODE, int DK>
__global__ void __launch_bounds__(kQueryThreads, kQueryBlocks) k_decr(View v, int j, int c) {
    pdl_wait();
    __shared__ StreamSmem sm;
    decr_body<MODE, DK, true>(v, j, c, blockIdx.x, sm);
}

__device__ __forceinline__ bool tuple_less(unsigned long long ka, int sa, unsigned long long kb,
                                           int sb) {
    return ka < kb || (ka == kb && sa < sb);
}

// Number of sorted chunk words (key, el + offset) strictly below (key, slot).
__device__ __forceinline__ int count_words_less(const unsigned long long* words, int n, int el,
                                                unsigned long long key, int slot) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const unsigned long long w = words[mid];
        if (tuple_less(w >> kOffBits, el + (int)(w & ((1u << kOffBits) - 1)), key, slot))
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// Warp-wide count of sorted words below (key, slot): a 32-way search, one
// dependent load per factor-32 narrowing (3 rounds for a 16384-word chunk).
__device__ __forceinline__ int warp_count_words_less(const unsigned long long* words, int n, int el,
                                                     unsigned long long key, int slot, int lane) {
    int lo = 0, hi = n;  // words below lo are less, words from hi on are not
    while (hi - lo > 32) {
        const int step = (hi - lo + 31) >> 5;
        const int piv = lo + lane * step;
        bool less = false;
        if (piv < hi) {
            const unsigned long long w = words[piv];
            less = tuple_less(w >> kOffBits, el + (int)(w & ((1u << kOffBits) - 1)), key, slot);
        }
        const int c = __popc(__ballot_sync(kFull, less));
        if (c == 0) {
            hi = lo;
            break;
        }
        const int nlo = lo + (c - 1) * step + 1;
        hi = min(hi, lo + c * step);
        lo = nlo;
    }
    bool less = false;
    if (lo + lane < hi) {
        const unsigned long long w = words[lo + lane];
        less = tuple_less(w >> kOffBits, el + (int)(w & ((1u << kOffBits) - 1)), key, slot);
    }
    return lo + __popc(__ballot_sync(kFull, less));
}

// Old sorted window minus the expired slots [el, el+c), merged with the c
// new entries; tile t of the old window goes to output offset
// ts - (#expired before ts) + (#new before old[ts]).
constexpr int kMergeStage = 1024;  // new words of a tile staged in shared memory
template <int TILE>
struct MergeSmem {
    unsigned long long tkey[TILE];
    unsigned long long nw[kMergeStage];
    int tslot[TILE];
    int spre[TILE + 1];
    unsigned wsum[32];
    int bnd[3];
};

template <int TILE>
__device__ __forceinline__ void merge_body(const View& v, int j, int c, int init, int bx, int nbx,
                                           MergeSmem<TILE>& sm) {
    constexpr int kPer = TILE / kMergeThreads;  // old entries per thread
    unsigned long long* tkey = sm.tkey;
    int* tslot = sm.tslot;
    int* spre = sm.spre;
    unsigned* wsum = sm.wsum;
    const long long b = v.ctl->b;
    const int src = (int)((b - 1) & 1), dst = (int)(b & 1);
    const int n_old = v.ctl->nocc[src];
    const int n_new = n_old - (init ? 0 : c) + c;
    const int el = chunk_base_slot(v, j, init);
    const int tid = threadIdx.x;
    // a fresh union-find forest: with neighbour lists k_border resets it by
    // slot at the end of every clustering, so only the first window needs it
    const bool reset_parent = init || v.list_cap < 0;
    // forest reuse: the hints of the slide's last chunk step stand (every
    // loss of the slide is marked by then), so only that step counts reuses
    const bool reuse = !init && damage_on(v);
    const bool last_step = j * v.chunk + c >= v.S;
    unsigned reused = 0;
    if (bx == 0 && tid == 0) {
        v.ctl->nocc[dst] = n_new;
        v.ctl->nitems = 0;
        v.ctl->ncells = 0;
        v.ctl->union_next = 0;
    }
    // Table generations wrap every kGenMod builds of a table: clear it then.
    if (b >= 2 && ((b >> 1) % (long long)kGenMod) == 0) {
        ulonglong2* T = v.table[dst];
        for (unsigned i = bx * blockDim.x + tid; i <= v.pmask; i += nbx * blockDim.x)
            T[i] = make_ulonglong2(0ull, 0ull);
    }
    const int ntiles = n_old > 0 ? (n_old + TILE - 1) / TILE : 1;
    const int t = bx;
    if (t >= ntiles) return;
    const int ts = t * TILE;
    const int te = min(ts + TILE, n_old);
    const int tlen = te - ts;
    const unsigned long long* okey = v.skey[src];
    const float4* opt = v.spt[src];
    const int* ocnt = v.scnt[src];
    unsigned long long* dkey = v.skey[dst];
    float4* dpt = v.spt[dst];
    int* dcnt = v.scnt[dst];
    // previous roots are only read by this slide's reuse (a slide without
    // reuse leaves them to the flatten, which writes them afresh)
    const int* oprev = reuse ? v.sprev[src] : nullptr;
    int* dprev = reuse ? v.sprev[dst] : nullptr;

    // tile bounds among the new / expired words: warps 0, 1, 2 search at once
    {
        const int lane = tid & 31, w = tid >> 5;
        if (w < 3) {
            const bool need = tlen > 0 && (w == 0 ? t > 0 : (w == 1 ? !init : t < ntiles - 1));
            int r = w == 2 ? c : 0;
            if (need) {
                const int at = w == 2 ? te : ts;
                r = warp_count_words_less(w == 1 ? v.xword : v.nword, c, el, okey[at], slot_of(opt[at]),
                                          lane);
            }
            if (lane == 0) sm.bnd[w] = r;
        }
    }
    // tile -> shared memory; survivor prefix in item order
    for (int i = tid; i < tlen; i += kMergeThreads) {
        tkey[i] = okey[ts + i];
        tslot[i] = slot_of(opt[ts + i]);
    }
    __syncthreads();
    const int jt0 = sm.bnd[0], e0 = sm.bnd[1], jt1 = sm.bnd[2];
    const int base = ts - e0 + jt0;
    const int m = jt1 - jt0;
    const bool staged = m <= kMergeStage;
    const unsigned long long* nw = staged ? sm.nw : v.nword + jt0;  // the tile's new words
    if (staged)
        for (int i = tid; i < m; i += kMergeThreads) sm.nw[i] = v.nword[jt0 + i];
    unsigned flags[kPer];
    unsigned cnt = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int i = tid * kPer + k;
        const bool surv = i < tlen && (init || tslot[i] < el || tslot[i] >= el + c);
        flags[k] = surv ? 1u : 0u;
        cnt += flags[k];
    }
    {
        const int lane = tid & 31, w = tid >> 5;
        unsigned incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned x = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += x;
        }
        if (lane == 31) wsum[w] = incl;
        __syncthreads();
        if (w == 0) {
            const unsigned x = lane < kMergeThreads / 32 ? wsum[lane] : 0u;
            unsigned xi = x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(kFull, xi, o);
                if (lane >= o) xi += y;
            }
            if (lane < kMergeThreads / 32) wsum[lane] = xi - x;
        }
        __syncthreads();
        unsigned pre = wsum[w] + incl - cnt;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            spre[tid * kPer + k] = (int)pre;
            pre += flags[k];
        }
        if (tid == kMergeThreads - 1) spre[TILE] = (int)pre;
    }
    __syncthreads();

    // survivors (coalesced, item order i = tid + 256 k; unrolled, with loads
    // that may pass the stores: 1M points 24.6 -> 22.5 us)
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int i = tid + u * kMergeThreads;
        if (i >= tlen) continue;
        const int s = tslot[i];
        if (!(init || s < el || s >= el + c)) continue;
        const int lessnew = m > 0 ? count_words_less(nw, m, el, tkey[i], s) : 0;
        const int o = base + spre[i] + lessnew;
        if (o < 0 || o >= n_new) {
            atomicOr(&v.ctl->err, kErrChunk);
            continue;
        }
        dkey[o] = tkey[i];
        dpt[o] = __ldg(&opt[ts + i]);
        const int cnt = __ldg(&ocnt[ts + i]);
        dcnt[o] = cnt;
        const int prev = oprev ? __ldg(&oprev[ts + i]) : -1;
        if (dprev) dprev[o] = prev;
        v.sroot[o] = start_hint(v, s, cnt, prev, reuse, reused);
        if (reset_parent) v.parent[s] = s;
    }
    if (last_step) {
        reused = __reduce_add_sync(kFull, reused);
        if ((tid & 31) == 0 && reused) atomicAdd(&v.ctl->reused, (int)reused);
    }
    // new entries of this tile
    for (int q = jt0 + tid; q < jt1; q += kMergeThreads) {
        const unsigned long long wd = nw[q - jt0];
        const unsigned long long key = wd >> kOffBits;
        const int slot = el + (int)(wd & ((1u << kOffBits) - 1));
        int lo = 0, hi = tlen;  // old tile entries below (key, slot)
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (tuple_less(tkey[mid], tslot[mid], key, slot))
                lo = mid + 1;
            else
                hi = mid;
        }
        const int o = base + (q - jt0) + spre[lo];
        if (o < 0 || o >= n_new || slot < 0 || slot >= v.W) {
            atomicOr(&v.ctl->err, kErrChunk);
            continue;
        }
        dkey[o] = key;
        dpt[o] = v.ring[slot];
        dcnt[o] = 0;
        if (dprev) dprev[o] = -1;
        v.sroot[o] = -1;  // the increment sets the count and the hint
        if (reset_parent) v.parent[slot] = slot;
        // the chunk's order, for the slide that expires it (every reader of
        // the expired order of these slots ran before this pass)
        if (!init && v.sorder) v.sorder[el + q] = slot - el;
    }
}

template <int TILE>
__global__ void __launch_bounds__(kMergeThreads) k_merge(View v, int j, int c, int init) {
    pdl_wait();
    __shared__ MergeSmem<TILE> sm;
    merge_body(v, j, c, init, blockIdx.x, gridDim.x, sm);
}

// Cell table of the new sorted window.  A cell that starts and ends in one
// warp's positions is entered once, by its first point; otherwise its first
// point enters the start, its last the end.  Cells and cell runs (within 32
// positions) are counted once per block, behind two barriers, for the statistics
// and the choice between whole builds and chunk steps.  Bound by the latency of
// the inserts (a read, a CAS and a store to a random slot; 25 of 36 cycles per
// issue, the barriers 8): 1M walkers, 275k cells, 25 us (29 with a work list of
// cell runs for the union and the label pass, which now take blocks of positions).
struct BuildSmem {
    int cells, runs;
};

__device__ __forceinline__ void build_body(const View& v, int bx, BuildSmem& sm) {
    if (threadIdx.x == 0) sm.cells = sm.runs = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int gw = (bx * blockDim.x + threadIdx.x) >> 5;
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    const unsigned gen = gen_of_build(b);
    const int n = v.ctl->nocc[cur];
    const int i = gw * 32 + lane;
    const unsigned long long* skey = v.skey[cur];
    const bool valid = i < n;
    const unsigned long long k = valid ? skey[i] : ~0ull;
    unsigned long long kp = __shfl_up_sync(kFull, k, 1);
    unsigned long long kn = __shfl_down_sync(kFull, k, 1);
    if (lane == 0) kp = (valid && i > 0) ? skey[i - 1] : ~0ull;
    if (lane == 31) kn = (i + 1 < n) ? skey[i + 1] : ~0ull;
    const bool first = valid && (i == 0 || kp != k);
    const bool last = valid && (i == n - 1 || kn != k);
    const unsigned firsts = __ballot_sync(kFull, first);
    const unsigned lasts = __ballot_sync(kFull, last);
    if (lane == 0) {
        const int runs = __popc(firsts | (valid ? 1u : 0u));
        if (firsts) atomicAdd(&sm.cells, __popc(firsts));
        if (runs) atomicAdd(&sm.runs, runs);
    }
    int err = 0;
    ulonglong2* T = v.table[cur];
    const unsigned long long tag = tag_of(k & kKeyMask, gen);
    if (first) {
        const unsigned ends = lasts & ~((1u << lane) - 1u);  // my cell's last is the lowest
        const bool ok = ends ? table_set(T, v.pmask, v.pbits, tag, 2, i, gw * 32 + __ffs(ends))
                             : table_set(T, v.pmask, v.pbits, tag, 0, i);
        if (!ok) err |= kErrHashFull;
    }
    if (last && !(firsts & ((2u << lane) - 1u)) && !table_set(T, v.pmask, v.pbits, tag, 1, i + 1))
        err |= kErrHashFull;
    if (err) atomicOr(&v.ctl->err, err);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sm.cells) atomicAdd(&v.ctl->ncells, sm.cells);
        if (sm.runs) atomicAdd(&v.ctl->nitems, sm.runs);
        if (bx == 0) v.ctl->b_done = b;  // not read here
    }
}

__global__ void __launch_bounds__(kBuildThreads) k_build(View v) {
    pdl_wait();
    __shared__ BuildSmem sm;
    build_body(v, blockIdx.x, sm);
}

// Full count of each new point and +1 on every older neighbour (new grid).
template <int MODE, int DK, int G, bool AHEAD>
__device__ __forceinline__ void incr_g(const View& v, int j, int c, int init, int bx, StreamSmem& sm) {
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;  // dimension, cells per Eps
    constexpr int kPerWarp = 32 / G;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int grp = lane / G, gl = lane % G;
    const int gw = (bx * blockDim.x + threadIdx.x) >> 5;
    if (gw * kPerWarp >= c) return;
    const int qi = gw * kPerWarp + grp;
    const bool has = qi < c;
    int* rstart = sm.grstart[wib][grp];
    int* rpre = sm.grpre[wib][grp];
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    const unsigned gen = gen_of_build(b);
    const int el = chunk_base_slot(v, j, init);
    const unsigned long long word = has ? v.nword[qi] : 0ull;
    const unsigned long long key = word >> kOffBits;
    const int aslot = el + (int)(word & ((1u << kOffBits) - 1));
    const float4 ap = has ? v.ring[aslot] : make_float4(0.f, 0.f, 0.f, 0.f);
    int rs, re;
    row_ranges<DIM, K, G>(v, v.table[cur], gen, key, gl, rs, re);
    int total = candidate_stream<Stencil<DIM, false, K>::kRows, G>(rs, re, gl, rstart, rpre);
    if (!has) total = 0;
    int tmax = total;
#pragma unroll
    for (int o = G; o < 32; o <<= 1) tmax = max(tmax, __shfl_xor_sync(kFull, tmax, o));
    const float4* spt = v.spt[cur];
    int* scnt = v.scnt[cur];
    const bool lists = v.list_cap >= 0;
    int* nbuf = sm.gnbuf[wib][grp];
    Tally tally;
    int count = 0, mypos = -1, r = 0, nfound = 0;
    // Two candidates per lane and trip (idx and idx + G), as in the decrement.
    int npos[2] = {0, 0}, ncnt[2] = {0, 0};
    float4 nq[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    auto fetch = [&](int at, int* p, int* n, float4* c4) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (at + u * G >= total) continue;
            p[u] = stream_pos(at + u * G, r, rstart, rpre);
            c4[u] = spt[p[u]];
            n[u] = scnt[p[u]];  // counts only rise here: >= MinPts means no list kept
        }
    };
    if (AHEAD) fetch(gl, npos, ncnt, nq);
    for (int base = 0; base < tmax; base += 2 * G) {
        const int idx = base + gl;
        const bool h0 = idx < total, h1 = idx + G < total;
        int pos[2] = {0, 0}, cnt[2] = {0, 0}, qs[2] = {-1, -1};
        float4 q[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        if (AHEAD) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                pos[u] = npos[u];
                cnt[u] = ncnt[u];
                q[u] = nq[u];
            }
            fetch(idx + 2 * G, npos, ncnt, nq);
        } else {
            fetch(idx, pos, cnt, q);
        }
        float d[2];
        sqdist32x2<DIM>(ap, q[0], q[1], d[0], d[1]);
        bool nb[2] = {false, false};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (!(u == 0 ? h0 : h1)) continue;
            qs[u] = slot_of(q[u]);
            if (qs[u] == aslot) {
                ++count;
                mypos = pos[u];
            } else if (nbr_decide<MODE, DIM>(v, d[u], ap, q[u], tally)) {
                ++count;
                nb[u] = true;
                if (qs[u] < el || qs[u] >= el + c) {
                    // counts only rise here: one read below MinPts may be the
                    // increment that makes the point core, which sets its hint
                    if (cnt[u] >= v.min_pts)
                        atomicAdd(&scnt[pos[u]], 1);
                    else if (atomicAdd(&scnt[pos[u]], 1) == v.min_pts - 1)
                        v.sroot[pos[u]] = qs[u];  // now core
                    if (lists && cnt[u] < v.min_pts && v.ntrack[qs[u]] == 1) list_append(v, qs[u], aslot);
                }
            }
        }
        if (lists) {
            nfound = list_collect<G>(nb[0], qs[0], nfound, v.list_cap, nbuf, lane);
            nfound = list_collect<G>(nb[1], qs[1], nfound, v.list_cap, nbuf, lane);
        }
    }
    if (lists) list_store<G>(v, aslot, nfound, nbuf, lane, has);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        count += __shfl_xor_sync(kFull, count, o);
        mypos = max(mypos, __shfl_xor_sync(kFull, mypos, o));
    }
    int err = 0;
    if (gl == 0 && has) {
        if (mypos >= 0) {
            scnt[mypos] = count;
            v.sroot[mypos] = count >= v.min_pts ? aslot : -1;
        } else {
            err = kErrChunk;
        }
    }
    flush_query_max<G>(v, tally.tests, lane);
    flush_stats(v, tally, err, lane, 0);
}

template <int MODE, int DK, bool AHEAD>
__device__ __forceinline__ void incr_body(const View& v, int j, int c, int init, int bx, StreamSmem& sm) {
    if constexpr ((DK >> 2) == 0) {
        if (v.qlanes == 16) {
            incr_g<MODE, DK, 16, AHEAD>(v, j, c, init, bx, sm);
            return;
        }
    }
    incr_g<MODE, DK, 32, AHEAD>(v, j, c, init, bx, sm);
}

template <int MODE, int DK>
__global__ void __launch_bounds__(kQueryThreads, kQueryBlocks) k_incr(View v, int j, int c, int init) {
    pdl_wait();
    __shared__ StreamSmem sm;
    incr_body<MODE, DK, true>(v, j, c, init, blockIdx.x, sm);
}

// ------------------------------------------------------ whole-window build
// The first window, and a slide that replaces a large share of the window,
// build the grid from all W slots at once: one pass writes every slot's sort
// word, a radix sort orders them, one pass lays the window out in that order,
// the cell table is built once and every point's neighbours are counted once
// (k_count), instead of W / 16384 chunk steps that each rewrite the window.
// A 1M-point walker window: load 9.9 -> 0.40 ms (sort 52 us, count 240 us; the
// box of the points is taken on the device, not in a host loop over a copy);
// 48k points replaced per slide: 327 -> 137 us for the grid.
// Words are key << ob | slot (ob bits for the slots; the host takes the chunk
// steps where key and slot do not fit 64 bits).  The sort alternates between
// the two key buffers and ends in the one that the window's layout does not
// take; the counters of its tiles lie in that side's counts.

constexpr int kRadThreads = 512;
constexpr int kRadItems = 8;                           // words per thread
constexpr int kRadTile = kRadThreads * kRadItems;      // words per block
constexpr int kRadWarps = kRadThreads / 32;
// Digits of up to 10 bits, as equal as the key's bits allow: a key of 18 or 20
// bits takes two passes, one of 25 three, where 8-bit digits took three and
// four (48k points 44 -> 25 us, 1M 97 -> 52).
constexpr int kRadBits = 10;
inline int rad_passes(const View& v) { return (v.key_bits + kRadBits - 1) / kRadBits; }
inline int rad_bits(const View& v) {  // (at least 5: the scan takes 32 digits a block)
    const int p = rad_passes(v);
    return p ? max(5, (v.key_bits + p - 1) / p) : 5;
}
// Up to this many tiles every scatter block sums the tiles' counters itself;
// above, a scan kernel does it once.
constexpr int kRadInline = 32;

// Input buffer of radix pass `pass` of `passes` (pass == passes: the sorted words).
__device__ __forceinline__ unsigned long long* rad_buffer(const View& v, int pass, int passes) {
    const int cur = (int)(v.ctl->b & 1);
    return v.skey[((passes - pass) & 1) ? cur : cur ^ 1];
}

// Slots [base, base + count) take the new points (base by the slide's place
// in the ring, 0 while loading); every slot's sort word goes to the first
// pass's input (chunk < 0), or the new points' chunk words to nsort.
__global__ void k_ingest_all(View v, SlideIO io, int count, int init, int ob, int passes) {
    pdl_wait();
    const long long b = v.ctl->b_done + 1;  // this build (k_build keeps b_done)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        v.ctl->b = b;
        v.ctl->out_label = io.label;
        v.ctl->out_cid = io.cid;
        if (!init) {
            v.ctl->prev_ok = 0;     // no forest reuse in this clustering,
            v.ctl->reuse_skip = 2;  // no roots kept for the next,
            v.ctl->kept_from = v.ctl->slide + 1;  // nor this slide's order
        }
    }
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= v.W) return;
    const int base = chunk_base_slot(v, 0, init);
    unsigned long long key;
    if (s >= base && s < base + count) {
        const float* p = io.input + (size_t)(s - base) * v.dim;
        const float x = p[0];
        const float y = v.dim > 1 ? p[1] : 0.0f;
        const float z = v.dim > 2 ? p[2] : 0.0f;
        v.ring[s] = make_float4(x, y, z, __int_as_float(s));
        key = cell_key(v, x, y, z);
        v.kslot[s] = key;
    } else {
        key = v.kslot[s];
    }
    const unsigned long long word = (key << ob) | (unsigned long long)s;
    if (passes < 0) {
        v.nsort[s] = word;
    } else {
        const int cur = (int)(b & 1);
        v.skey[(passes & 1) ? cur : cur ^ 1][s] = word;
    }
}

__global__ void __launch_bounds__(kRadThreads) k_rad_hist(View v, int pass, int passes, int shift, int bits) {
    pdl_wait();
    __shared__ int hist[1 << kRadBits];
    const int bins = 1 << bits;
    const unsigned long long* in = rad_buffer(v, pass, passes);
    int* counts = v.scnt[(v.ctl->b & 1) ^ 1];
    for (int d = threadIdx.x; d < bins; d += kRadThreads) hist[d] = 0;
    __syncthreads();
    unsigned long long w[kRadItems];
#pragma unroll
    for (int k = 0; k < kRadItems; ++k) {
        const int i = blockIdx.x * kRadTile + k * kRadThreads + threadIdx.x;
        w[k] = i < v.W ? in[i] : 0ull;
    }
#pragma unroll
    for (int k = 0; k < kRadItems; ++k) {
        const int i = blockIdx.x * kRadTile + k * kRadThreads + threadIdx.x;
        if (i < v.W) atomicAdd(&hist[(unsigned)(w[k] >> shift) & (bins - 1)], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < bins; d += kRadThreads) counts[blockIdx.x * bins + d] = hist[d];
}

// Exclusive scan over the tiles of 32 digits per block (a warp's lanes side by
// side), 32 warps on a part of the tiles each; the digits' totals follow the
// tiles' counters.  Only where there are many tiles (kRadInline).
__global__ void __launch_bounds__(1024) k_rad_scan(View v, int ntiles, int bins) {
    pdl_wait();
    __shared__ int part[32][32];
    int* counts = v.scnt[(v.ctl->b & 1) ^ 1];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = blockIdx.x * 32 + lane;
    const int per = (ntiles + 31) / 32, t0 = min(w * per, ntiles), t1 = min(t0 + per, ntiles);
    int sum = 0;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) sum += counts[t * bins + d];
    part[w][lane] = sum;
    __syncthreads();
    int at = 0;
    for (int k = 0; k < w; ++k) at += part[k][lane];
#pragma unroll 8
    for (int t = t0; t < t1; ++t) {
        const int x = counts[t * bins + d];
        counts[t * bins + d] = at;
        at += x;
    }
    if (w == 31) counts[ntiles * bins + d] = at;
}

// Stable scatter of one tile by its digit: each warp ranks its 256
// consecutive words in order (lanes with equal digits from a ballot per
// digit bit), warp counters are scanned per digit, and every word goes to its
// place.
__global__ void __launch_bounds__(kRadThreads) k_rad_scatter(View v, int pass, int passes, int shift, int bits,
                                                             int scanned) {
    pdl_wait();
    __shared__ unsigned short cnt[kRadWarps][1 << kRadBits];  // of a warp, then before it in the tile
    __shared__ int base[1 << kRadBits];                      // the tile's first place of a digit
    __shared__ int wsum[kRadWarps];
    const int bins = 1 << bits;
    const unsigned long long* in = rad_buffer(v, pass, passes);
    unsigned long long* out = rad_buffer(v, pass + 1, passes);
    const int* counts = v.scnt[(v.ctl->b & 1) ^ 1];
    const int ntiles = gridDim.x, tile = blockIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kRadWarps * (1 << kRadBits) / 2; k += kRadThreads)
        reinterpret_cast<unsigned*>(&cnt[0][0])[k] = 0;
    unsigned long long it[kRadItems];
    int rank[kRadItems];
    const int i0 = tile * kRadTile + w * (32 * kRadItems) + lane;
#pragma unroll
    for (int k = 0; k < kRadItems; ++k) it[k] = i0 + 32 * k < v.W ? in[i0 + 32 * k] : ~0ull;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRadItems; ++k) {
        const bool has = i0 + 32 * k < v.W;
        const unsigned d = (unsigned)(it[k] >> shift) & (bins - 1);
        unsigned peers = __ballot_sync(kFull, has);
        for (int bit = 0; bit < bits; ++bit) {
            const unsigned bm = __ballot_sync(kFull, (d >> bit) & 1u);
            peers &= ((d >> bit) & 1u) ? bm : ~bm;
        }
        const int before = cnt[w][d];
        __syncwarp();
        rank[k] = before + __popc(peers & lanemask_lt(lane));
        if (has && !(peers & lanemask_lt(lane))) cnt[w][d] = (unsigned short)(before + __popc(peers));
        __syncwarp();
    }
    // digit totals -> digit bases: each thread two neighbouring digits
    int total[2] = {0, 0}, mine[2] = {0, 0};  // words of the digit: all, before this tile
    const int d0 = 2 * threadIdx.x;
    if (d0 < bins) {
        if (scanned) {
            for (int u = 0; u < 2; ++u) {
                total[u] = counts[ntiles * bins + d0 + u];
                mine[u] = counts[tile * bins + d0 + u];
            }
        } else {
#pragma unroll 8
            for (int t = 0; t < ntiles; ++t) {
                const int2 x = *reinterpret_cast<const int2*>(&counts[t * bins + d0]);
                total[0] += x.x;
                total[1] += x.y;
                mine[0] += t < tile ? x.x : 0;
                mine[1] += t < tile ? x.y : 0;
            }
        }
    }
    int incl = total[0] + total[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();  // (every warp's counts are in, too)
    if (d0 < bins) {
        int at = incl - total[0] - total[1];
        for (int k = 0; k < w; ++k) at += wsum[k];
        base[d0] = at + mine[0];
        base[d0 + 1] = at + total[0] + mine[1];
        for (int u = 0; u < 2; ++u) {
            int before = 0;
            for (int k = 0; k < kRadWarps; ++k) {
                const int x = cnt[k][d0 + u];
                cnt[k][d0 + u] = (unsigned short)before;
                before += x;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRadItems; ++k) {
        if (i0 + 32 * k >= v.W) continue;
        const unsigned d = (unsigned)(it[k] >> shift) & (bins - 1);
        const int o = base[d] + cnt[w][d] + rank[k];
        if (o >= 0 && o < v.W)
            out[o] = it[k];
        else
            atomicOr(&v.ctl->err, kErrChunk);
    }
}

// The window laid out in the order of its sorted words (counts and hints
// follow in k_count), a fresh forest, and the build's counters reset.
__global__ void k_fill(View v, int ob, int passes) {
    pdl_wait();
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        v.ctl->nocc[cur] = v.W;
        v.ctl->nitems = 0;
        v.ctl->ncells = 0;
        v.ctl->union_next = 0;
    }
    // table generations wrap every kGenMod builds of a table, as in the merge
    if (b >= 2 && ((b >> 1) % (long long)kGenMod) == 0) {
        ulonglong2* T = v.table[cur];
        for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i <= v.pmask; i += gridDim.x * blockDim.x)
            T[i] = make_ulonglong2(0ull, 0ull);
    }
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= v.W) return;
    const unsigned long long word = passes < 0 ? v.nword[o] : v.skey[cur ^ 1][o];
    const int slot = (int)(word & ((1ull << ob) - 1ull));
    if (slot >= v.W) {
        atomicOr(&v.ctl->err, kErrChunk);
        return;
    }
    v.skey[cur][o] = word >> ob;
    v.spt[cur][o] = v.ring[slot];
    v.parent[slot] = slot;
}

// Neighbour counts, start hints and neighbour lists of every point, from one
// scan of the grid.  As in the union, a warp takes a block of consecutive
// sorted positions, looks up the stencil rows of all its cells (the whole
// stencil here) lane by lane and walks them as one candidate stream; every
// lane tests its candidate against the points of its own cell run, the runs'
// points in step, two at a time, so one vote counts a whole chunk for each of
// them.  The lists of the few non-core points with neighbours are collected
// from their candidates afterwards (kept while counting, they took a
// rank and a store per test: 1M walkers 349 us against 276, 200k dense
// trajectories 263 against 136).  Bound by instruction issue; against one
// whole-stencil query per point with atomics on its neighbours, as the chunk
// steps count, 1M walkers take 0.24 ms instead of 1.8.
// Blocks per SM 8 / 10 / 12: 1M walkers 268 / 245 / 240 us, though at 12 up to 16
// bytes a thread are spilled; two cells per Eps lose more above 8 (48k points
// replaced per slide 115 / 125 / 122).
constexpr int kCountThreads = 128;

template <int DIM, int K>
struct CountShape {
    static constexpr int kRows = Stencil<DIM, false, K>::kRows;
    static constexpr int kBlock = kRows > 9 ? 16 : 32;  // positions per warp (shared memory)
    static constexpr int kTasks = kBlock * kRows;
};

template <int DIM, int K>
struct CountSmem {
    using C = CountShape<DIM, K>;
    static constexpr int kWarps = kCountThreads / 32;
    float4 pt[kWarps][C::kBlock];  // home points
    unsigned long long skey[kWarps][C::kBlock];
    int first[kWarps][C::kBlock + 1];  // first home point of a run
    int sbeg[kWarps][C::kBlock + 1];   // first candidate of a run
    int tbeg[kWarps][C::kBlock];       // first stored row of a run
    int tstart[kWarps][C::kTasks];
    int tpre[kWarps][C::kTasks + 1];
    unsigned char tseg[kWarps][C::kTasks];
};

__device__ __forceinline__ unsigned lane_range(int lo, int hi) {  // lanes [lo, hi), clamped
    const unsigned up = hi >= 32 ? kFull : (hi <= 0 ? 0u : lanemask_lt(hi));
    return up & ~(lo >= 32 ? kFull : (lo <= 0 ? 0u : lanemask_lt(lo)));
}

template <int MODE, int DK>
__global__ void __launch_bounds__(kCountThreads, (DK >> 2) == 0 ? 12 : 8) k_count(View v, int P) {
    pdl_wait();
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;
    using C = CountShape<DIM, K>;
    constexpr int R = C::kRows;
    __shared__ CountSmem<DIM, K> sm;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    const unsigned gen = gen_of_build(b);
    const int n = v.ctl->nocc[cur];
    const int start = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * P;
    if (start >= n) return;
    const int m = min(P, n - start);
    const bool hv = lane < m;
    float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned long long key = 0;
    if (hv) {
        h = v.spt[cur][start + lane];
        key = v.skey[cur][start + lane];
    }
    // runs of one cell
    const unsigned long long kprev = __shfl_up_sync(kFull, key, 1);
    const unsigned leaders = __ballot_sync(kFull, hv && (lane == 0 || kprev != key));
    const int ns = __popc(leaders);
    const int run = __popc(leaders & (lanemask_lt(lane) | (1u << lane))) - 1;
    if (hv) {
        sm.pt[wib][lane] = h;
        if ((leaders >> lane) & 1u) {
            sm.skey[wib][run] = key;
            sm.first[wib][run] = lane;
        }
    }
    if (lane == 0) sm.first[wib][ns] = m;
    __syncwarp();
    int* tstart = sm.tstart[wib];
    int* tpre = sm.tpre[wib];
    unsigned char* tseg = sm.tseg[wib];
    int nt = 0, total = 0;
    for (int t0 = 0; t0 < ns * R; t0 += 32) {
        const int t = t0 + lane, seg = t / R;
        int a = 0, len = 0;
        if (t < ns * R) {
            const int2 rr = row_range_lane<DIM, false, K>(v, v.table[cur], gen, sm.skey[wib][seg], t - seg * R);
            a = rr.x;
            len = rr.y - rr.x;
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += x;
        }
        const unsigned some = __ballot_sync(kFull, len > 0);
        if (t < ns * R && t == seg * R) {
            sm.sbeg[wib][seg] = total + incl - len;
            sm.tbeg[wib][seg] = nt + __popc(some & lanemask_lt(lane));
        }
        if (len > 0) {
            const int at = nt + __popc(some & lanemask_lt(lane));
            tstart[at] = a;
            tpre[at] = total + incl - len;
            tseg[at] = (unsigned char)seg;
        }
        nt += __popc(some);
        total += __shfl_sync(kFull, incl, 31);
    }
    if (lane == 0) {
        tpre[nt] = total;
        sm.sbeg[wib][ns] = total;
    }
    __syncwarp();
    const int ord = hv ? lane - sm.first[wib][run] : -1;
    const int hb = hv ? sm.sbeg[wib][run] : 0, he = hv ? sm.sbeg[wib][run + 1] : 0;
    const float4* spt = v.spt[cur];
    Tally tally;
    int r = 0, count = 0;
    for (int base = 0; base < total; base += 32) {
        const int idx = base + lane;
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        int f = 0, len = 0;
        if (idx < total) {
            while (idx >= tpre[r + 1]) ++r;
            q = spt[tstart[r] + idx - tpre[r]];
            const int s = tseg[r];
            f = sm.first[wib][s];
            len = sm.first[wib][s + 1] - f;
        }
        const unsigned home = lane_range(hb - base, he - base);  // the chunk's candidates of the home point
        const int steps = (int)__reduce_max_sync(kFull, (unsigned)len);
        for (int t = 0; t < steps; t += 2) {  // two home points a step
            bool n0 = false, n1 = false;
            if (t < len) {
                const float4 h0 = sm.pt[wib][f + t], h1 = sm.pt[wib][f + min(t + 1, len - 1)];
                float d0, d1;
                sqdist32x2<DIM>(q, h0, h1, d0, d1);
                n0 = slot_of(h0) != slot_of(q) && nbr_decide<MODE, DIM>(v, d0, h0, q, tally);
                n1 = t + 1 < len && slot_of(h1) != slot_of(q) && nbr_decide<MODE, DIM>(v, d1, h1, q, tally);
            }
            const unsigned b0 = __ballot_sync(kFull, n0), b1 = __ballot_sync(kFull, n1);
            if ((ord >> 1) == (t >> 1)) count += __popc(((ord & 1) ? b1 : b0) & home);
        }
    }
    const int slot = slot_of(h), all = count + 1;  // the point itself included
    const bool core = all >= v.min_pts;
    if (hv) {
        v.scnt[cur][start + lane] = all;
        v.sroot[start + lane] = core ? slot : -1;
    }
    if (v.list_cap >= 0) {
        if (hv) v.ntrack[slot] = core ? 0 : 1;
        if (hv && !core) {
            int4* L = reinterpret_cast<int4*>(v.nlist + (size_t)slot * v.list_stride);
            for (int k = 0; k < v.list_stride >> 2; ++k) L[k] = make_int4(-1, -1, -1, -1);
        }
        __syncwarp();
        // lists of the non-core points with neighbours: the point's candidates
        // once more (few points, in the sparser cells)
        unsigned todo = __ballot_sync(kFull, hv && !core && count > 0);
        while (todo) {
            const int l = __ffs(todo) - 1;
            todo &= todo - 1;
            const int s = __shfl_sync(kFull, run, l), aslot = __shfl_sync(kFull, slot, l);
            const int from = sm.sbeg[wib][s], to = sm.sbeg[wib][s + 1];
            const float4 hp = sm.pt[wib][l];
            int* L = v.nlist + (size_t)aslot * v.list_stride;
            int found = 0;
            r = sm.tbeg[wib][s];
            for (int base = from; base < to; base += 32) {
                const int idx = base + lane;
                bool nb = false;
                int qs = -1;
                if (idx < to) {
                    while (idx >= tpre[r + 1]) ++r;
                    const float4 q = spt[tstart[r] + idx - tpre[r]];
                    qs = slot_of(q);
                    nb = qs != aslot && is_nbr<MODE, DIM>(v, hp, q, tally);
                }
                const unsigned hits = __ballot_sync(kFull, nb);
                const int k = found + __popc(hits & lanemask_lt(lane));
                if (nb && k < v.list_cap) L[k] = qs;
                found += __popc(hits);
            }
        }
    }
    const unsigned most = __reduce_max_sync(kFull, (unsigned)max(he - hb - 1, 0));
    if (lane == 0 && most) atomicMax(&v.ctl->qmax[wib & 7], (int)most);
    flush_stats(v, tally, 0, lane, 0);
}

// Fresh start hints without reuse (-1 for a non-core position, its own
// slot for a core) and a fresh forest, for a clustering of the window as it
// stands (rtdbs_cluster), whose hints may hold the last union's roots.
__global__ void k_hints(View v, SlideIO io) {
    pdl_wait();
    const int cur = (int)(v.ctl->b & 1);
    const int n = v.ctl->nocc[cur];
    const int* scnt = v.scnt[cur];
    const int* sw = reinterpret_cast<const int*>(v.spt[cur]) + 3;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        v.ctl->prev_ok = 0;  // no reuse to judge (read by k_border)
        v.ctl->out_label = io.label;
        v.ctl->out_cid = io.cid;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = sw[4 * (size_t)i];
        v.sroot[i] = scnt[i] >= v.min_pts ? s : -1;
        v.parent[s] = s;
    }
}

// Cores linked within their own warp's 32 sorted positions, before the union:
// the points of one cell, and of the cells that follow it in its stencil row,
// are neighbours in the sorted window, so most sets can be joined there from
// coalesced loads and warp votes alone -- no table lookups, no walks and no
// atomics (a point's parent is written only by the warp that holds it; a
// component kept from the last slide is joined by smaller roots in the union
// only).  The union then starts from these sets' roots as hints.  Each lane
// looks at the kLinkReach positions after its own.
// Bound by instruction issue (22 M warp instructions for a 1M-point walker
// window with a reach of 8).  Link and union together, us, by reach 0 / 4 / 8:
// 1M walkers 207 / 168 / 170, 200k trajectories 107 / 80 / 82, 100k prices
// 131 / 61 / 64, a pool of 32 mixed streams 505 / 338 / 342.
constexpr int kLinkReach = 4;

struct LinkSmem {
    float4 pt[kLinkThreads / 32][32];  // .w = root hint
    unsigned long long key[kLinkThreads / 32][32];
};

template <int MODE, int DK>
__device__ __forceinline__ void link_body(const View& v, int bx, LinkSmem& sm) {
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;  // dimension, cells per Eps
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int cur = (int)(v.ctl->b & 1);
    const int n = v.ctl->nocc[cur];
    const int i = bx * blockDim.x + threadIdx.x;
    if ((i & ~31) >= n) return;
    const bool valid = i < n;
    const int hint = valid ? v.sroot[i] : -1;
    const bool core = hint >= 0;
    const unsigned cores = __ballot_sync(kFull, core);
    if (!cores) return;
    const int h0 = __shfl_sync(kFull, hint, __ffs(cores) - 1);
    if (__all_sync(kFull, !core || hint == h0)) return;  // one set already (or one core)
    float4 p = valid ? v.spt[cur][i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned long long key = valid ? v.skey[cur][i] : ~0ull;
    const int slot = slot_of(p);
    p.w = __int_as_float(hint);
    sm.pt[wib][lane] = p;
    sm.key[wib][lane] = key;
    __syncwarp();
    Tally tally;
    unsigned adj = 1u << lane;  // lanes in this lane's set
    for (int d = 1; d <= kLinkReach; ++d) {
        const int o = lane + d;
        const bool near = o < 32 && valid && sm.key[wib][o & 31] - key <= (unsigned long long)K;
        if (!__any_sync(kFull, near)) break;
        bool nb = false;
        if (near && core) {
            const float4 q = sm.pt[wib][o];
            const int qh = __float_as_int(q.w);
            nb = qh >= 0 && qh != hint && is_nbr<MODE, DIM>(v, p, q, tally);
        }
        const unsigned b = __ballot_sync(kFull, nb);
        if (nb) adj |= 1u << o;
        if (lane >= d && ((b >> (lane - d)) & 1u)) adj |= 1u << (lane - d);
    }
    // transitive closure: each lane takes in the sets of its set's lanes
    unsigned todo = adj & ~(1u << lane);
    while (__any_sync(kFull, todo != 0)) {
        const int src = todo ? __ffs(todo) - 1 : lane;
        const unsigned m = __shfl_sync(kFull, adj, src);
        todo &= ~(1u << src);
        todo |= m & ~adj;
        adj |= m;
    }
    if (core && (adj & (adj - 1u))) {
        const int root = (int)__reduce_min_sync(adj, (unsigned)hint);
        // a core under the old root of a kept component stays under it
        if (hint == slot && root < slot) {
            v.parent[slot] = root;
            v.sroot[i] = root;
        }
    }
    flush_stats(v, tally, 0, lane, 1);
}

template <int MODE, int DK>
__global__ void __launch_bounds__(kLinkThreads) k_link(View v) {
    pdl_wait();
    __shared__ LinkSmem sm;
    link_body<MODE, DK>(v, blockIdx.x, sm);
}

// Blocks of positions a union warp takes at a time: one, as a block holds
// about 8 cell runs (2 blocks: walkers 168 -> 178 us, trajectories 79 -> 109);
// the stream's setting counts cell runs.
__device__ __forceinline__ int union_grab(const View& v) { return max(1, v.grab >> 4); }

// Union of every core-core neighbour pair.  A warp takes a block of P
// consecutive sorted positions (View::block_pts), whose cores fall into runs
// of one cell (segments).  The upper-half stencil rows of all segments are
// looked up by lanes side by side, the non-empty ones are laid end to end as
// one candidate stream (positions above a segment's first core), and every
// lane tests its candidate against the cores of its own segment until one
// under another root is near.  Hints may be behind the forest, so before any
// test the open candidates and the home points look up their current roots:
// a load or two in place of a test against every home point, as most of the
// pairs whose hints differ have been joined meanwhile.  The near pairs of a
// chunk are then joined at once: the smallest root per home root by a warp
// minimum, every other root hooked under it by a lane of its own, so lanes of
// a warp rarely meet on one parent.  Roots known for home points are kept in
// shared memory, for candidates in their hints.
//
// Bound by instruction issue and L2 latency (DRAM throughput 5%).  Against one
// cell per warp, candidates looked up 14 cells at a time with shuffles, a find
// and a hook per near pair: link and union 225 -> 168 us on the 1M-point
// walker window (10.8 -> 4.4 M distance tests), 74 -> 41 us on the 500k
// precision stream, 297 -> 79 us on 200k trajectories, 520 -> 62 us on 100k
// prices, 606 -> 286 us per round of a 32-stream pool.
// Without the root lookups before the tests: 204, 41, 129, 142, 430.
// Row lookups in 32-bit words, and no filter flag beside the band, took most of its
// register spills away (100-230 bytes a thread): walkers 168 -> 162, pool 288 -> 278.
// Thread blocks per SM 4 / 5 / 6: walkers 172 / 162 / 156 us, pool round 298 / 278 /
// 287 (registers against warps in flight).  Stores of spilled registers that are
// left, in bytes a thread: one cell per Eps in 2-D and 3-D 48 and 52 (FP64), in
// pools 28; two cells per Eps 88 and 96, in pools 60 and 92.
constexpr int kUnionBlocks = 6;      // of a window slid alone
constexpr int kPoolUnionBlocks = 5;

// Most positions of a block (View::block_pts, a pool's blocks).  In a stream slid
// alone the 13 rows of two cells per Eps in 3-D take 37 KB of shared memory a thread block for 32
// positions, which leaves next to no L1 for the lookups, most of whose lines the
// neighbouring cells share; 16 take half.  us per slide with room for 16 / 32, the
// blocks 16 positions either way (3-D mixture, MinPts 3, 4 neighbours): 50k points
// 162 / 172 (one cell per warp 165), 500k 508 / 587 (533), 2M 1847 / 2520 (2016);
// walkers 500k 390 / 475 (512), 2M 1499 / 2217 (1884).  Pools of such streams lose by
// blocks of 16 (walkers 4 x 300k points 628 -> 658 us a round, mixtures 988 -> 1005).
constexpr __host__ __device__ int union_room(int dk, bool pooled) { return dk == 7 && !pooled ? 16 : 32; }

template <int DIM, int K, int ROOM>
struct UnionSmem {
    static constexpr int kTasks = ROOM * Stencil<DIM, true, K>::kRows;  // stencil rows of a block's segments, at most
    float4 pt[kClusterThreads / 32][32];  // home points, .w = root known
    unsigned long long skey[kClusterThreads / 32][32];
    unsigned segm[kClusterThreads / 32][32];  // home cores of a segment
    int tstart[kClusterThreads / 32][kTasks];
    int tpre[kClusterThreads / 32][kTasks + 1];
    unsigned char tseg[kClusterThreads / 32][kTasks];
};

template <int MODE, int DK, class Smem>
__device__ __forceinline__ void union_body(const View& v, Smem& sm, int P, int grab) {
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;  // dimension, cells per Eps
    constexpr int R = Stencil<DIM, true, K>::kRows;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float4* hpt = sm.pt[wib];
    int* tstart = sm.tstart[wib];
    int* tpre = sm.tpre[wib];
    unsigned char* tseg = sm.tseg[wib];
    unsigned* segm = sm.segm[wib];
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    const unsigned gen = gen_of_build(b);
    const int n = v.ctl->nocc[cur];
    const int nblk = (n + P - 1) / P;
    const float4* spt = v.spt[cur];
    const ulonglong2* T = v.table[cur];
    int* parent = v.parent;
    // Root hints by sorted position (an ancestor of the point: its own slot,
    // its set's root from the link pass or the old root of its intact
    // component; -1 for a non-core point, so the hint alone tells a core):
    // coalesced with the candidate loads, and refreshed as roots are found,
    // so find walks stay short.
    volatile int* hint = v.sroot;
    Tally tally;
    int err = 0;
    int bk1 = 0;
    for (int bk = nblk;;) {
        if (bk >= bk1) {
            int got = 0;
            if (lane == 0) got = atomicAdd(&v.ctl->union_next, grab);
            bk = __shfl_sync(kFull, got, 0);
            if (bk >= nblk) break;
            bk1 = min(bk + grab, nblk);
        }
        const int start = bk++ * P;
        const int i = start + lane;
        const bool hv = lane < P && i < n;
        const int hh = hv ? hint[i] : -1;
        const bool hcore = hh >= 0;
        const unsigned hmask = __ballot_sync(kFull, hcore);
        if (!hmask) continue;
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
        unsigned long long key = 0;
        if (hcore) {
            h = spt[i];
            key = v.skey[cur][i];
        }
        int hr = hh;  // the root known for the lane's home point
        h.w = __int_as_float(hh);
        // segments: the cores of one cell
        const unsigned below = hmask & lanemask_lt(lane);
        const unsigned long long kprev = __shfl_sync(kFull, key, below ? 31 - __clz(below) : lane);
        const unsigned leaders = __ballot_sync(kFull, hcore && (!below || kprev != key));
        const int ns = __popc(leaders);
        const unsigned upto = leaders & (lanemask_lt(lane) | (1u << lane));
        const int first = upto ? 31 - __clz(upto) : 0;  // first core of the lane's segment
        __syncwarp();
        hpt[lane] = h;
        if ((leaders >> lane) & 1u) {
            const unsigned later = leaders & ~((2u << lane) - 1u);
            const int at = __popc(upto) - 1;
            segm[at] = hmask & ~lanemask_lt(lane) & (later ? lanemask_lt(__ffs(later) - 1) : kFull);
            sm.skey[wib][at] = key;
        }
        __syncwarp();
        // rows of all segments, the non-empty ones end to end
        int nt = 0, total = 0;
        for (int t0 = 0; t0 < ns * R; t0 += 32) {
            const int t = t0 + lane, seg = t / R;
            int a = 0, len = 0;
            if (t < ns * R) {
                const int2 rr = row_range_lane<DIM, true, K>(v, T, gen, sm.skey[wib][seg], t - seg * R);
                a = max(rr.x, start + __ffs(segm[seg]));
                len = max(rr.y - a, 0);
            }
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += x;
            }
            const unsigned some = __ballot_sync(kFull, len > 0);
            if (len > 0) {
                const int at = nt + __popc(some & lanemask_lt(lane));
                tstart[at] = a;
                tpre[at] = total + incl - len;
                tseg[at] = (unsigned char)seg;
            }
            nt += __popc(some);
            total += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0) tpre[nt] = total;
        int fr = __shfl_sync(kFull, hr, first);
        unsigned mixed = __ballot_sync(kFull, hcore && hr != fr);  // cores not under their segment's first root
        __syncwarp();
        int r = 0;
        for (int base = 0; base < total; base += 32) {
            const int idx = base + lane;
            int pos = 0, qh = -1;
            unsigned mm = 0;
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (idx < total) {
                while (idx >= tpre[r + 1]) ++r;
                pos = tstart[r] + idx - tpre[r];
                q = spt[pos];
                qh = hint[pos];
                mm = segm[tseg[r]];
                // a segment under one root and a candidate under it: one set
                if (qh < 0 || (!(mixed & mm) && __float_as_int(hpt[__ffs(mm) - 1].w) == qh)) mm = 0;
            }
            if (!__any_sync(kFull, mm != 0)) continue;
            {
                // hints may be behind the forest: the current roots of the open
                // candidates and of the home points
                volatile int* up = parent;
                const int uq = mm ? up[qh] : qh, uh = hcore ? up[hr] : hr;
                if (uq != qh) {
                    qh = uf_find(parent, uq);
                    hint[pos] = qh;
                }
                if (uh != hr) hr = uf_find(parent, uh);
                __syncwarp();
                if (__any_sync(kFull, uh != hr || uh != __float_as_int(h.w))) {
                    h.w = __int_as_float(hr);
                    if (hcore) hpt[lane].w = h.w;
                    fr = __shfl_sync(kFull, hr, first);
                    mixed = __ballot_sync(kFull, hcore && hr != fr);
                    __syncwarp();
                }
                if (mm && !(mixed & mm) && __float_as_int(hpt[__ffs(mm) - 1].w) == qh) mm = 0;
            }
            while (__any_sync(kFull, mm != 0)) {
                int ga = 0;
                bool nb = false;
                while (__any_sync(kFull, mm != 0 && !nb)) {
                    if (mm != 0 && !nb) {
                        const float4 hp = hpt[__ffs(mm) - 1];
                        mm &= mm - 1;
                        ga = __float_as_int(hp.w);
                        nb = ga != qh && is_nbr<MODE, DIM>(v, hp, q, tally);
                    }
                }
                const unsigned near = __ballot_sync(kFull, nb);
                if (!near) break;
                int top = 0;
                bool lead = false;
                if (nb) {
                    const unsigned pq = __match_any_sync(near, qh), pa = __match_any_sync(near, ga);
                    top = min(ga, (int)__reduce_min_sync(pa, (unsigned)qh));
                    int res = top;
                    if (!(pq & pa & lanemask_lt(lane)) && qh != top) res = uf_hook(parent, qh, top, err);
                    lead = !(pa & lanemask_lt(lane));
                    if (lead && ga != top) res = min(res, uf_hook(parent, ga, top, err));
                    __syncwarp(near);
                    top = (int)__reduce_min_sync(pa, (unsigned)res);
                    if (qh != top) {
                        hint[pos] = top;
                        qh = top;
                    }
                }
                // the home points' roots
                unsigned todo = __ballot_sync(kFull, lead);
                while (todo) {
                    const int l = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const int from = __shfl_sync(kFull, ga, l), to = __shfl_sync(kFull, top, l);
                    if (hr == from) hr = to;
                }
                __syncwarp();
                h.w = __int_as_float(hr);
                if (hcore) hpt[lane].w = h.w;
                fr = __shfl_sync(kFull, hr, first);
                mixed = __ballot_sync(kFull, hcore && hr != fr);
                __syncwarp();
            }
        }
        if (hcore && hr != hh) hint[i] = hr;
        __syncwarp();
    }
    flush_stats(v, tally, err, lane, 1);
}

template <int MODE, int DK>
__global__ void __launch_bounds__(kClusterThreads, kUnionBlocks) k_union(View v) {
    pdl_wait();
    __shared__ UnionSmem<(DK & 3), (DK >> 2) + 1, union_room(DK, false)> sm;
    union_body<MODE, DK>(v, sm, v.block_pts, union_grab(v));
}

// The neighbour list of the non-core point at sorted position `at`, from one
// scan of the current grid (called by the whole warp).
template <int MODE, int DIM, int K>
__device__ __forceinline__ void rebuild_list(const View& v, int at, int cur, unsigned gen, int lane, int* rstart,
                                             int* rpre, int* nbuf, Tally& tally) {
    const float4* spt = v.spt[cur];
    const float4 ap = spt[at];
    const int a = slot_of(ap);
    int rs, re;
    row_ranges<DIM, K>(v, v.table[cur], gen, v.skey[cur][at], lane, rs, re);
    const int total = candidate_stream<Stencil<DIM, false, K>::kRows>(rs, re, lane, rstart, rpre);
    int r = 0, nfound = 0;
    for (int base = 0; base < total; base += 32) {
        const int idx = base + lane;
        bool nb = false;
        int qs = -1;
        if (idx < total) {
            const float4 q = spt[stream_pos(idx, r, rstart, rpre)];
            qs = slot_of(q);
            nb = qs != a && is_nbr<MODE, DIM>(v, ap, q, tally);
        }
        nfound = list_collect(nb, qs, nfound, v.list_cap, nbuf, lane);
    }
    list_store(v, a, nfound, nbuf, lane);
}

// Root of every core point, walked from the position's root hint.  Without
// neighbour lists: by sorted position (-1 for non-core points), for the grid
// scan of k_label.  With lists: by slot (rslot), which k_border turns into
// the outputs; and a point below MinPts without a list (it lost core status
// this slide) gets its list rebuilt here from one scan of the final grid, by
// the warp whose 32 positions hold it.
template <int MODE, int DK>
__device__ __forceinline__ void flatten_body(const View& v, int bx, int nbx, StreamSmem& sm) {
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;  // dimension, cells per Eps
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    const int n = v.ctl->nocc[cur];
    const int* scnt = v.scnt[cur];
    if (v.list_cap < 0) {
        for (int i = bx * blockDim.x + threadIdx.x; i < n; i += nbx * blockDim.x)
            v.sroot[i] = scnt[i] >= v.min_pts ? uf_find(v.parent, v.sroot[i]) : -1;
        return;
    }
    int(&rstart)[8][kMaxRows] = sm.rstart;
    int(&rpre)[8][kMaxRows + 1] = sm.rpre;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const unsigned gen = gen_of_build(b);
    const int* sw = reinterpret_cast<const int*>(v.spt[cur]) + 3;  // .w = slot
    int* nbuf = sm.nbuf[wib];
    // the roots by position for the next slide's reuse: not while reuse
    // stays off for it (k_border counts reuse_skip down after this pass)
    const bool keep_roots = v.ctl->reuse_skip <= 1;
    Tally tally;
    // Roots first (no barrier); the positions whose lists are rebuilt go to
    // the block's queue, which its warps share once the block has been
    // through its positions (one barrier), so rebuilds of neighbouring points
    // do not fall on one warp.  A full queue is rebuilt by the warp itself.
    if (threadIdx.x == 0) sm.nq = 0;
    __syncthreads();
    for (int i0 = (bx * blockDim.x + threadIdx.x) & ~31; i0 < n; i0 += nbx * blockDim.x) {  // warp-uniform
        const int i = i0 + lane;
        bool need = false;
        if (i < n) {
            const int slot = sw[4 * (size_t)i];
            const int at = v.sroot[i];
            if (at >= 0) {
                const int root = uf_find(v.parent, at);
                v.rslot[slot] = root;
                if (keep_roots) v.sprev[cur][i] = root;  // the next slide's reuse reads it by position
            } else {
                v.rslot[slot] = -1;
                if (keep_roots) v.sprev[cur][i] = -1;
                need = v.ntrack[slot] != 1;
            }
        }
        bool inline_rebuild = false;
        if (need) {
            const int at = atomicAdd(&sm.nq, 1);
            if (at < kFlattenQueue)
                sm.queue[at] = i;
            else
                inline_rebuild = true;
        }
        unsigned todo = __ballot_sync(kFull, inline_rebuild);
        while (todo) {
            rebuild_list<MODE, DIM, K>(v, i0 + __ffs(todo) - 1, cur, gen, lane, rstart[wib], rpre[wib], nbuf, tally);
            todo &= todo - 1;
        }
    }
    __syncthreads();
    const int nq = min(sm.nq, kFlattenQueue);
    for (int e = wib; e < nq; e += wpb)
        rebuild_list<MODE, DIM, K>(v, sm.queue[e], cur, gen, lane, rstart[wib], rpre[wib], nbuf, tally);
    flush_stats(v, tally, 0, lane, 1);
}

template <int MODE, int DK>
__global__ void __launch_bounds__(256, 6) k_flatten(View v) {
    pdl_wait();
    __shared__ StreamSmem sm;
    flatten_body<MODE, DK>(v, blockIdx.x, gridDim.x, sm);
}

// Labels and ids by slot: core -> 0 and its root; non-core -> 1 and the
// minimum root over adjacent cores, or 2 and its own slot.  As in the count, a
// warp takes a block of consecutive sorted positions, whose non-core points
// with neighbours are its home points, and walks the whole stencil of their
// cells as one candidate stream; a core candidate is tested against those
// home points of its segment whose minimum it would lower.  Bound by load
// latency.
template <int DIM, int K, int THREADS, int BLOCK>
struct LabelSmem {
    static constexpr int kWarps = THREADS / 32;
    static constexpr int kTasks = BLOCK * CountShape<DIM, K>::kRows;
    float4 pt[kWarps][BLOCK];
    unsigned long long skey[kWarps][BLOCK];
    unsigned segm[kWarps][BLOCK];  // home points of a segment
    int best[kWarps][BLOCK];       // minimum root near a home point
    int tstart[kWarps][kTasks];
    int tpre[kWarps][kTasks + 1];
    unsigned char tseg[kWarps][kTasks];
};

__device__ __forceinline__ void put_result(const View& v, int* ol, int* oc, int slot, int lab, int id) {
    v.label[slot] = lab;
    v.cid[slot] = id;
    if (ol) ol[slot] = lab;
    if (oc) oc[slot] = id;
}

template <int MODE, int DK, class Smem>
__device__ __forceinline__ void label_body(const View& v, int advance, int bx, int nbx, Smem& sm, int P) {
    constexpr int DIM = DK & 3, K = (DK >> 2) + 1;  // dimension, cells per Eps
    constexpr int R = CountShape<DIM, K>::kRows;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    float4* hpt = sm.pt[wib];
    unsigned* segm = sm.segm[wib];
    int* best = sm.best[wib];
    int* tstart = sm.tstart[wib];
    int* tpre = sm.tpre[wib];
    unsigned char* tseg = sm.tseg[wib];
    const long long b = v.ctl->b;
    const int cur = (int)(b & 1);
    const unsigned gen = gen_of_build(b);
    const int n = v.ctl->nocc[cur];
    const int nblk = (n + P - 1) / P, step = nbx * Smem::kWarps;
    const float4* spt = v.spt[cur];
    const int* sroot = v.sroot;
    int* ol = v.ctl->out_label;
    int* oc = v.ctl->out_cid;
    Tally tally;
    for (int bk = bx * Smem::kWarps + wib; bk < nblk; bk += step) {
        const int i = bk * P + lane;
        const bool hv = lane < P && i < n;
        float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
        bool home = false;
        unsigned long long key = 0;
        int hslot = -1;
        if (hv) {
            h = spt[i];
            hslot = slot_of(h);
            const int hr = sroot[i];
            // (a point with no neighbour but itself is noise without a scan)
            home = hr < 0 && v.scnt[cur][i] > 1;
            if (!home) {
                put_result(v, ol, oc, hslot, hr >= 0 ? 0 : 2, hr >= 0 ? hr : hslot);
            } else {
                key = v.skey[cur][i];
            }
        }
        const unsigned hmask = __ballot_sync(kFull, home);
        if (!hmask) continue;
        // segments: the home points of one cell
        const unsigned below = hmask & lanemask_lt(lane);
        const unsigned long long kprev = __shfl_sync(kFull, key, below ? 31 - __clz(below) : lane);
        const unsigned leaders = __ballot_sync(kFull, home && (!below || kprev != key));
        const int ns = __popc(leaders);
        if (home) {
            hpt[lane] = h;
            best[lane] = INT_MAX;
        }
        if ((leaders >> lane) & 1u) {
            const unsigned later = leaders & ~((2u << lane) - 1u);
            const int at = __popc(leaders & lanemask_lt(lane));
            segm[at] = hmask & ~lanemask_lt(lane) & (later ? lanemask_lt(__ffs(later) - 1) : kFull);
            sm.skey[wib][at] = key;
        }
        __syncwarp();
        int nt = 0, total = 0;
        for (int t0 = 0; t0 < ns * R; t0 += 32) {
            const int t = t0 + lane, seg = t / R;
            int a = 0, len = 0;
            if (t < ns * R) {
                const int2 rr = row_range_lane<DIM, false, K>(v, v.table[cur], gen, sm.skey[wib][seg], t - seg * R);
                a = rr.x;
                len = rr.y - rr.x;
            }
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += x;
            }
            const unsigned some = __ballot_sync(kFull, len > 0);
            if (len > 0) {
                const int at = nt + __popc(some & lanemask_lt(lane));
                tstart[at] = a;
                tpre[at] = total + incl - len;
                tseg[at] = (unsigned char)seg;
            }
            nt += __popc(some);
            total += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0) tpre[nt] = total;
        __syncwarp();
        int r = 0;
        for (int base = 0; base < total; base += 32) {
            const int idx = base + lane;
            unsigned mm = 0;
            int qr = -1;
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (idx < total) {
                while (idx >= tpre[r + 1]) ++r;
                const int pos = tstart[r] + idx - tpre[r];
                qr = sroot[pos];
                q = spt[pos];
                if (qr >= 0) mm = segm[tseg[r]];
            }
            while (mm) {
                const int hi = __ffs(mm) - 1;
                mm &= mm - 1;
                if (qr < *(volatile int*)&best[hi] && is_nbr<MODE, DIM>(v, hpt[hi], q, tally))
                    atomicMin(&best[hi], qr);
            }
        }
        __syncwarp();
        if (home) {
            const int to = best[lane];
            put_result(v, ol, oc, hslot, to != INT_MAX ? 1 : 2, to != INT_MAX ? to : hslot);
        }
        __syncwarp();
    }
    flush_stats(v, tally, 0, lane, 1);
    if (bx == 0 && threadIdx.x == 0) {
        v.ctl->union_next = 0;                // the next clustering's queue; not read here
        if (advance) end_slide(v);            // no reader here
    }
}

// Positions a label warp takes as one block: short chains while the blocks are
// few (48k points, 4 / 8 / 16 / 32: 16 / 14 / 21 / 25 us, a queue of single cells 18;
// slides with MinPts 40 and 8 / 16 / 32: 3-D mixture with 5 neighbours 100k points
// 91 / 93 / 103, 400k 198 / 189 / 193, 1M 503 / 472 / 462; the same with keys of 48 bits
// 100k 179 / 196 / 233, 400k 470 / 479 / 534, queue 202 and 473; walkers 100k 105 / 104 /
// 109, 400k 204 / 191 / 191, 1M 494 / 452 / 439).  At any size 8 for the 25 rows of two
// cells per Eps in 3-D (8 / 16, mixture and walkers: 80k points 78 / 88, 72 / 78,
// 130k 167 / 184, 127 / 131, 200k 180 / 186, 158 / 158; single cells 98, 94,
// 201, 159, 227, 205; pool rounds of mixtures, MinPts 40, 32 x 2k points 709 / 829,
// 16 x 20k 1292 / 1363, 4 x 600k 4351 / 4404, single cells 4288).
constexpr __host__ __device__ __forceinline__ int label_block(int W, int dk, bool pooled) {
    if (dk == 7) return 8;
    return pooled || W >= 524288 ? 32 : (W >= 131072 ? 16 : 8);
}

// Thread blocks of the label pass of a stream slid alone: two warps.  The warps'
// work is so uneven that blocks of 8 warps, 4 per SM, kept 31% of an SM's warps
// active (two cells per Eps in 3-D, 300k points: 357 us, where single cells from a
// queue had taken 250).  Slide in us with blocks of 8 and 2 warps at the same
// registers, MinPts 40: two cells per Eps, 3-D mixture with 25 neighbours, 130k
// points 277 / 261, 300k 581 / 513, 1M 2201 / 1908; one cell, 60 neighbours, 400k 340 /
// 315, 1M 635 / 586, walkers 1M 455 / 439.  20 blocks per SM (48 registers) instead of
// 16 for two cells per Eps in 3-D: 300k 480, 1M 1750; 24: 514, 1827.
constexpr int kLabelThreads = 64;

template <int MODE, int DK>
__global__ void __launch_bounds__(kLabelThreads, DK == 7 ? 20 : 16) k_label(View v, int advance) {
    pdl_wait();
    __shared__ LabelSmem<(DK & 3), (DK >> 2) + 1, kLabelThreads, label_block(INT_MAX, DK, false)> sm;
    label_body<MODE, DK>(v, advance, blockIdx.x, gridDim.x, sm, label_block(v.W, DK, false));
}

// Outputs by slot from the roots and the lists: core -> 0 and its root; a
// non-core point with a core neighbour -> 1 and the minimum root over its
// core neighbours; else noise -> 2 and its own slot.  Resets the union-find
// forest for the next clustering (coalesced, by slot) and ends the slide
// like k_label.
__device__ __forceinline__ void border_body(const View& v, int advance, int bx, int nbx) {
    int* ol = v.ctl->out_label;
    int* oc = v.ctl->out_cid;
    for (int s = bx * blockDim.x + threadIdx.x; s < v.W; s += nbx * blockDim.x) {
        const int root = v.rslot[s];
        int lab = 0, id = root;
        if (root < 0) {
            if (v.ntrack[s] != 1) atomicOr(&v.ctl->err, kErrList);
            const int4* L = reinterpret_cast<const int4*>(v.nlist + (size_t)s * v.list_stride);
            int best = INT_MAX;
            for (int k = 0; k < (v.list_stride >> 2); ++k) {
                const int4 e = L[k];
                const int r0 = e.x >= 0 ? v.rslot[e.x] : -1;
                const int r1 = e.y >= 0 ? v.rslot[e.y] : -1;
                const int r2 = e.z >= 0 ? v.rslot[e.z] : -1;
                const int r3 = e.w >= 0 ? v.rslot[e.w] : -1;
                if (r0 >= 0) best = min(best, r0);
                if (r1 >= 0) best = min(best, r1);
                if (r2 >= 0) best = min(best, r2);
                if (r3 >= 0) best = min(best, r3);
            }
            lab = best != INT_MAX ? 1 : 2;
            id = best != INT_MAX ? best : s;
        }
        v.label[s] = lab;
        v.cid[s] = id;
        if (ol) ol[s] = lab;
        if (oc) oc[s] = id;
        v.parent[s] = s;
        v.damaged[s] = 0;
    }
    if (bx == 0 && threadIdx.x == 0) {
        v.ctl->union_next = 0;                // the next clustering's queue; not read here
        // the reuse of this clustering is counted: judge it
        // (not after a fresh window, which had no previous forest)
        if (v.ctl->reuse_skip > 0)
            v.ctl->reuse_skip -= 1;
        else if (v.ctl->prev_ok && v.ctl->reused < v.W / 16)
            v.ctl->reuse_skip = kReuseRetry;
        v.ctl->last_reused = v.ctl->reused;
        v.ctl->reused = 0;
        v.ctl->prev_ok = 1;                   // the forest of this clustering can be reused
        if (advance) end_slide(v);            // no reader here
    }
}

__global__ void k_border(View v, int advance) { pdl_wait(); border_body(v, advance, blockIdx.x, gridDim.x); }

__global__ void k_counts_by_slot(View v, int* nn) {
    const int cur = (int)(v.ctl->b & 1);
    const int n = v.ctl->nocc[cur];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        nn[slot_of(v.spt[cur][i])] = v.scnt[cur][i];
}

int g_num_sms = 0;
// ------------------------------------------------------------- batched kernel

template <int PHASE>
struct PhaseShape;
template <> struct PhaseShape<kBatchIngest> { static constexpr int threads = 256, min_blocks = 1; };
template <> struct PhaseShape<kBatchSort> { static constexpr int threads = kSortRun, min_blocks = 1; };
template <> struct PhaseShape<kBatchRunmerge> { static constexpr int threads = kSortRun, min_blocks = 1; };
template <> struct PhaseShape<kBatchDecrement> { static constexpr int threads = 256, min_blocks = 6; };
template <> struct PhaseShape<kBatchMerge> { static constexpr int threads = kMergeThreads, min_blocks = 1; };
template <> struct PhaseShape<kBatchBuild> { static constexpr int threads = kBuildThreads, min_blocks = 1; };
template <> struct PhaseShape<kBatchIncrement> { static constexpr int threads = 256, min_blocks = 6; };
template <> struct PhaseShape<kBatchLink> { static constexpr int threads = kLinkThreads, min_blocks = 1; };
template <> struct PhaseShape<kBatchUnion> { static constexpr int threads = kClusterThreads, min_blocks = kPoolUnionBlocks; };
template <> struct PhaseShape<kBatchFlatten> { static constexpr int threads = 256, min_blocks = 6; };
template <> struct PhaseShape<kBatchLabel> { static constexpr int threads = kClusterThreads, min_blocks = 5; };

// One phase over many streams.  The block finds its item, copies that
// stream's View into shared memory and runs the stream's kernel body.
// Phases whose bodies depend on the precision mode and dimension are
// instantiated per (MODE, DIM) and launched once per group of streams that
// share them, so each instantiation holds one body (registers as in the
// single-stream kernels); the other phases use MODE = DIM = 0.
template <int PHASE, int MODE, int DK>
__global__ void __launch_bounds__(PhaseShape<PHASE>::threads, PhaseShape<PHASE>::min_blocks)
    k_batch(BatchLaunch L) {
    __shared__ View sv;
    __shared__ int s_item, s_bx, s_nbx;
    if (threadIdx.x == 0) {
        int lo = 0, hi = L.n;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (L.prefix[mid] <= (int)blockIdx.x)
                lo = mid;
            else
                hi = mid;
        }
        s_item = lo;
        s_bx = (int)blockIdx.x - L.prefix[lo];
        s_nbx = L.prefix[lo + 1] - L.prefix[lo];
    }
    __syncthreads();
    const BatchItem it = L.items[s_item];
    {
        const int* src = reinterpret_cast<const int*>(L.views + it.view);
        int* dst = reinterpret_cast<int*>(&sv);
        for (int i = threadIdx.x; i < (int)(sizeof(View) / sizeof(int)); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    const int bx = s_bx, nbx = s_nbx;
    if constexpr (PHASE == kBatchIngest) {
        ingest_body(sv, it.j, it.c, 0, it.stg_off, SlideIO{it.input, nullptr, nullptr}, bx);
    } else if constexpr (PHASE == kBatchSort) {
        __shared__ SortSmem sm;
        const int nruns = (it.c + kSortRun - 1) / kSortRun;
        sort_body(sv, it.j, it.c, 0, bx % nruns, bx / nruns, sm, false);
    } else if constexpr (PHASE == kBatchRunmerge) {
        extern __shared__ unsigned long long words[];
        const int nruns = (it.c + kSortRun - 1) / kSortRun;
        runmerge_body(sv, it.j, it.c, 0, bx % nruns, bx / nruns, words);
    } else if constexpr (PHASE == kBatchDecrement) {
        __shared__ StreamSmem sm;
        decr_body<MODE, DK, false>(sv, it.j, it.c, bx, sm);
    } else if constexpr (PHASE == kBatchMerge) {
        __shared__ MergeSmem<kMergeTile> sm;
        merge_body(sv, it.j, it.c, 0, bx, nbx, sm);
    } else if constexpr (PHASE == kBatchBuild) {
        __shared__ BuildSmem sm;
        build_body(sv, bx, sm);
    } else if constexpr (PHASE == kBatchIncrement) {
        __shared__ StreamSmem sm;
        incr_body<MODE, DK, false>(sv, it.j, it.c, 0, bx, sm);
    } else if constexpr (PHASE == kBatchLink) {
        __shared__ LinkSmem sm;
        link_body<MODE, DK>(sv, bx, sm);
    } else if constexpr (PHASE == kBatchUnion) {
        __shared__ UnionSmem<(DK & 3), (DK >> 2) + 1, union_room(DK, true)> sm;
        union_body<MODE, DK>(sv, sm, union_room(DK, true), union_grab(sv));
    } else if constexpr (PHASE == kBatchFlatten) {
        __shared__ StreamSmem sm;
        flatten_body<MODE, DK>(sv, bx, nbx, sm);
    } else {
        __shared__ LabelSmem<(DK & 3), (DK >> 2) + 1, kClusterThreads, label_block(0, DK, true)> sm;
        if (sv.list_cap >= 0)
            border_body(sv, 1, bx, nbx);
        else
            label_body<MODE, DK>(sv, 1, bx, nbx, sm, label_block(sv.W, DK, true));
    }
}

std::atomic<unsigned long long> g_runmerge_ready{0};  // one bit per device

// k_runmerge stages up to kChunkMax words (128 KB) in dynamic shared memory;
// allow that once per device (a host-side attribute, not a stream operation).
size_t runmerge_smem(int c) { return sizeof(unsigned long long) * ((c + kSortRun - 1) / kSortRun * kSortRun); }

void ensure_runmerge_smem() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    const unsigned long long bit = 1ull << dev;
    if (g_runmerge_ready.load() & bit) return;
    const int bytes = (int)(sizeof(unsigned long long) * kChunkMax);
    if (cudaFuncSetAttribute(k_runmerge, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
        cudaFuncSetAttribute(k_batch<kBatchRunmerge, 0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
            cudaSuccess)
        g_runmerge_ready.fetch_or(bit);
}

}  // namespace

// Kernel launch, with programmatic dependence on the launch before it on this
// stream where `pdl` (that launch must be a kernel that calls pdl_wait).
template <class... P, class... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl, A... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// Launch of a work kernel instantiated for (precision, DK); dk = dim + 4 (K - 1).
#define RTDBS_DISPATCH(prec, dk_expr, KERNEL, GRID, BLOCK, STREAM, PDL, ...)          \
    do {                                                                         \
        const int dk = (dk_expr);                                                \
        if ((prec) == kPrecFp32) {                                               \
            switch (dk) {                                                        \
                case 1: launch(KERNEL<kPrecFp32, 1>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 2: launch(KERNEL<kPrecFp32, 2>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 3: launch(KERNEL<kPrecFp32, 3>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 5: launch(KERNEL<kPrecFp32, 5>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 6: launch(KERNEL<kPrecFp32, 6>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                default: launch(KERNEL<kPrecFp32, 7>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
            }                                                                    \
        } else {                                                                 \
            switch (dk) {                                                        \
                case 1: launch(KERNEL<kPrecFp64, 1>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 2: launch(KERNEL<kPrecFp64, 2>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 3: launch(KERNEL<kPrecFp64, 3>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 5: launch(KERNEL<kPrecFp64, 5>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                case 6: launch(KERNEL<kPrecFp64, 6>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
                default: launch(KERNEL<kPrecFp64, 7>, GRID, BLOCK, 0, STREAM, PDL, __VA_ARGS__); break; \
            }                                                                    \
        }                                                                        \
    } while (0)

cudaError_t configure_kernels() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    return cudaSuccess;
}

int count_pass_warps() { return (g_num_sms > 0 ? g_num_sms : 152) * kQueryBlocks * (kQueryThreads / 32); }

// Slides of windows up to this size launch their kernels with programmatic
// dependence: they are short enough for the launch and the first instructions
// to show (slides of 2.5k / 10k / 100k points 112 -> 106, 98 -> 95, 312 -> 291
// us); on larger ones the waiting blocks take SM slots from the running kernel
// (500k points 168 -> 186 us, 1M 324 -> 342).
// With two cells per Eps in 3-D the clustering kernels are several times as long
// and want the slots earlier.  us with it / without (3-D mixture): Eps 0.3,
// MinPts 2, 10k points 88 / 90, 32k 168 / 160, 80k 189 / 176, MinPts 40, 130k 432
// / 393; Eps 0.6, MinPts 8, 50k 164 / 170, 80k 181 / 168; mean gain of a mixture
// and walkers at 32k to 130k points 2.5%.
constexpr int kPdlWindow = 131072;
constexpr int kPdlWindowRows = 16384;  // two cells per Eps in 3-D
bool pdl_on(const View& v) { return v.W <= (v.dim == 3 && v.cell_mult == 2 ? kPdlWindowRows : kPdlWindow); }

cudaError_t launch_phase(int phase, const View& v, int precision, int j, int c, int init,
                         int stg_off, int advance, cudaStream_t s, bool pdl, const SlideIO& io) {
    const int warp_blocks = (c * v.qlanes + kQueryThreads - 1) / kQueryThreads;  // count passes
    switch (phase) {
        case kPhaseIngest:
            launch(k_ingest, (c + 255) / 256, 256, 0, s, pdl, v, j, c, init, stg_off, io);
            break;
        case kPhaseSort: {
            const int single = c <= kSortRun;  // one run: sorted straight into place, no run merge
            launch(k_sort, dim3((c + kSortRun - 1) / kSortRun, init ? 1 : 2), kSortRun, 0, s, pdl, v, j, c, init, single);
            if (single) break;
            ensure_runmerge_smem();
            launch(k_runmerge, dim3((c + kSortRun - 1) / kSortRun, init ? 1 : 2), kSortRun, runmerge_smem(c),
                   s, pdl, v, j, c, init);
            break;
        }
        case kPhaseDecrement:
            if (!init) RTDBS_DISPATCH(precision, dk_of(v), k_decr, warp_blocks, kQueryThreads, s, pdl, v, j, c);
            break;
        case kPhaseMerge:
            // short tiles where the blocks are few (10k points 14 -> 10 us, 200k
            // 14 -> 10), fewer searches above (500k 25 -> 16, 1M 37 -> 25)
            if (v.W < 262144)
                launch(k_merge<256>, (v.W + 255) / 256, kMergeThreads, 0, s, pdl, v, j, c, init);
            else
                launch(k_merge<kMergeTile>, (v.W + kMergeTile - 1) / kMergeTile, kMergeThreads, 0, s, pdl, v, j, c, init);
            break;
        case kPhaseBuild:
            launch(k_build, (v.W + kBuildThreads - 1) / kBuildThreads, kBuildThreads, 0, s, pdl, v);
            break;
        case kPhaseIncrement:
            RTDBS_DISPATCH(precision, dk_of(v), k_incr, warp_blocks, kQueryThreads, s, pdl, v, j, c, init);
            break;
        case kPhaseLabel:
            if (v.list_cap >= 0) {
                const int sms = g_num_sms > 0 ? g_num_sms : 152;
                launch(k_border, max(1, min(sms * 8, (v.W + 255) / 256)), 256, 0, s, pdl, v, advance);
                break;
            }
            {
                const int per = label_block(v.W, dk_of(v), false) * (kLabelThreads / 32);  // positions per thread block
                RTDBS_DISPATCH(precision, dk_of(v), k_label, (v.W + per - 1) / per, kLabelThreads, s, pdl, v, advance);
            }
            break;
        case kPhaseUnion: {
            // queue-fed blocks, as many as the window has or the SMs hold
            const int sms = g_num_sms > 0 ? g_num_sms : 152;
            const int per = v.block_pts * (kClusterThreads / 32);
            const int blocks = max(1, min(sms * kUnionBlocks, (v.W + per - 1) / per));
            RTDBS_DISPATCH(precision, dk_of(v), k_link, (v.W + kLinkThreads - 1) / kLinkThreads, kLinkThreads, s, pdl, v);
            RTDBS_DISPATCH(precision, dk_of(v), k_union, blocks, kClusterThreads, s, pdl, v);
            break;
        }
        case kPhaseFlatten: {
            const int sms = g_num_sms > 0 ? g_num_sms : 152;
            RTDBS_DISPATCH(precision, dk_of(v), k_flatten, max(1, min(sms * 16, (v.W + 255) / 256)), 256, s, pdl, v);
            break;
        }
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_chunk_step(const View& v, int precision, int j, int c, int init, int stg_off, cudaStream_t s,
                              const SlideIO& io, bool ingested, cudaStream_t side, cudaEvent_t fork,
                              cudaEvent_t join) {
    if (c <= 0 || c > kChunkMax) return cudaErrorInvalidValue;
    const bool beside = side && fork && join && !init;  // the decrement beside the sort
    for (int ph = 0; ph < kChunkPhases; ++ph) {
        cudaError_t e = cudaSuccess;
        if (beside && ph == kPhaseDecrement) continue;  // launched on the side stream
        if (beside && ph == kPhaseMerge && (e = cudaStreamWaitEvent(s, join, 0)) != cudaSuccess) return e;
        // (the ingest follows a copy or another chunk's work, the merge two streams)
        // (a launch behind an ingest outside the graph is the graph's first node)
        const bool pdl = pdl_on(v) && ph != kPhaseIngest && ph != kPhaseDecrement && ph != kPhaseMerge &&
                         !(ingested && ph == kPhaseSort);
        if (!(ingested && ph == kPhaseIngest)) {
            e = launch_phase(ph, v, precision, j, c, init, stg_off, 0, s, pdl, io);
            if (e != cudaSuccess) return e;
        }
        // (after the ingest, but launched behind the sort, whose few large blocks
        // should not wait for the decrement's to leave: 500k points 174 -> 166 us
        // per slide, 1M 325 -> 318)
        if (beside && ph == kPhaseIngest && (e = cudaEventRecord(fork, s)) != cudaSuccess) return e;
        if (beside && ph == kPhaseSort) {
            if ((e = cudaStreamWaitEvent(side, fork, 0)) != cudaSuccess) return e;
            if ((e = launch_phase(kPhaseDecrement, v, precision, j, c, init, stg_off, 0, side)) != cudaSuccess)
                return e;
            if ((e = cudaEventRecord(join, side)) != cudaSuccess) return e;
        }
    }
    return cudaSuccess;
}

cudaError_t launch_window_phase(int phase, const View& v, int precision, const SlideIO& io, int count, int init,
                                cudaStream_t s, bool pdl) {
    const int grid = (v.W + 255) / 256;
    const bool chunk = v.W <= kChunkMax;  // one chunk: its runs are sorted and ranked on chip
    const int ob = chunk ? kOffBits : slot_bits(v.W);
    const int passes = chunk ? -1 : rad_passes(v), bits = rad_bits(v);
    switch (phase) {
        case kPhaseIngest:
            launch(k_ingest_all, grid, 256, 0, s, pdl, v, io, count, init, ob, passes);
            break;
        case kPhaseSort:
            if (chunk) {
                const int runs = (v.W + kSortRun - 1) / kSortRun;
                launch(k_sort, dim3(runs, 1), kSortRun, 0, s, pdl, v, 0, v.W, 1, runs == 1);
                if (runs == 1) break;
                ensure_runmerge_smem();
                launch(k_runmerge, dim3(runs, 1), kSortRun, runmerge_smem(v.W), s, pdl, v, 0, v.W, 1);
                break;
            }
            for (int p = 0; p < passes; ++p) {
                const int tiles = (v.W + kRadTile - 1) / kRadTile, shift = ob + bits * p;
                launch(k_rad_hist, tiles, kRadThreads, 0, s, pdl, v, p, passes, shift, bits);
                const int scanned = tiles > kRadInline;
                if (scanned) launch(k_rad_scan, (1 << bits) / 32, 1024, 0, s, true, v, tiles, 1 << bits);
                launch(k_rad_scatter, tiles, kRadThreads, 0, s, true, v, p, passes, shift, bits, scanned);
                pdl = true;
            }
            break;
        case kPhaseDecrement: break;  // counted afresh
        case kPhaseMerge:
            launch(k_fill, grid, 256, 0, s, pdl, v, ob, passes);
            break;
        case kPhaseBuild:
            launch(k_build, (v.W + kBuildThreads - 1) / kBuildThreads, kBuildThreads, 0, s, pdl, v);
            break;
        case kPhaseIncrement: {
            // positions per warp (at most CountShape's): short chains while the
            // blocks are few, fuller lookups above.  us with 8 / 16 / 32: 20k
            // points 14 / 20 / 28, 48k 39 / 43 / 66, 200k trajectories 141 / 136
            // / 152, 1M walkers 358 / 300 / 276 (at 8 blocks per SM)
            const int block = v.W < 65536 ? 8 : (v.W < 524288 || (v.dim == 3 && v.cell_mult == 2) ? 16 : 32);
            const int per = block * (kCountThreads / 32);
            RTDBS_DISPATCH(precision, dk_of(v), k_count, (v.W + per - 1) / per, kCountThreads, s, pdl, v, block);
            break;
        }
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_window_build(const View& v, int precision, const SlideIO& io, int count, int init,
                                cudaStream_t s, bool ingested) {
    if (!window_build_fits(v)) return cudaErrorInvalidValue;
    cudaError_t e = cudaSuccess;
    for (int ph = ingested ? kPhaseSort : kPhaseIngest; ph < kChunkPhases && e == cudaSuccess; ++ph)
        // (kernels that follow each other closely at any size: a first window of
        // 1M points 864 -> 820 us, of 20k 205 -> 179)
        e = launch_window_phase(ph, v, precision, io, count, init, s,
                                ph != kPhaseIngest && !(ingested && ph == kPhaseSort));
    return e;
}

int window_build_launches(const View& v) {
    const int per = (v.W + kRadTile - 1) / kRadTile > kRadInline ? 3 : 2;
    const int sorts = v.W > kChunkMax ? per * rad_passes(v) : (v.W > kSortRun ? 2 : 1);
    return 4 + sorts;
}

// Finite bounding box of n points per axis, as order-keeping unsigned keys
// (box[0..2] minima from ~0, box[3..5] maxima from 0).
__global__ void __launch_bounds__(256) k_bbox(const float* pts, long long n, int dim, unsigned* box) {
    __shared__ unsigned sbox[6];  // (one global atomic per block and bound)
    if (threadIdx.x < 6) sbox[threadIdx.x] = threadIdx.x < 3 ? ~0u : 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    unsigned lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0u, 0u, 0u};
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (a >= dim) break;
            const float x = pts[i * dim + a];
            if (!isfinite(x)) continue;
            const unsigned u = __float_as_uint(x);
            const unsigned k = (u >> 31) ? ~u : u | 0x80000000u;
            lo[a] = min(lo[a], k);
            hi[a] = max(hi[a], k);
        }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const unsigned l = __reduce_min_sync(kFull, lo[a]), h = __reduce_max_sync(kFull, hi[a]);
        if (lane == 0 && l <= h) {
            atomicMin(&sbox[a], l);
            atomicMax(&sbox[3 + a], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3 && sbox[threadIdx.x] <= sbox[3 + threadIdx.x]) {
        atomicMin(&box[threadIdx.x], sbox[threadIdx.x]);
        atomicMax(&box[3 + threadIdx.x], sbox[3 + threadIdx.x]);
    }
}

cudaError_t launch_bbox(const float* pts, long long n, int dim, unsigned* box, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(box, 0xff, 3 * sizeof(unsigned), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(box + 3, 0, 3 * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
    const int sms = g_num_sms > 0 ? g_num_sms : 152;
    k_bbox<<<(int)max(1ll, min((long long)sms * 4, (n + 255) / 256)), 256, 0, s>>>(pts, n, dim, box);
    return cudaGetLastError();
}

cudaError_t launch_cluster(const View& v, int precision, int advance, cudaStream_t s, bool fresh_hints,
                           cudaEvent_t outputs_free, unsigned wait_flags, const SlideIO& io) {
    cudaError_t e = cudaSuccess;
    if (fresh_hints) {
        const int sms = g_num_sms > 0 ? g_num_sms : 152;
        k_hints<<<max(1, min(sms * 8, (v.W + 255) / 256)), 256, 0, s>>>(v, io);
        e = cudaGetLastError();
    }
    for (int ph = kPhaseUnion; ph <= kPhaseLabel && e == cudaSuccess; ++ph) {
        if (ph == kPhaseLabel && outputs_free) e = cudaStreamWaitEvent(s, outputs_free, wait_flags);
        const bool pdl = pdl_on(v) && !(ph == kPhaseLabel && outputs_free);
        if (e == cudaSuccess) e = launch_phase(ph, v, precision, 0, 0, 0, 0, advance, s, pdl);
    }
    return e;
}

int batch_threads(int phase) {
    switch (phase) {
        case kBatchSort:
        case kBatchRunmerge: return kSortRun;
        case kBatchMerge: return kMergeThreads;
        case kBatchBuild: return kBuildThreads;
        case kBatchUnion:
        case kBatchLabel: return kClusterThreads;
        default: return 256;
    }
}

int batch_blocks(int phase, const View& v, int c) {
    const int runs = (c + kSortRun - 1) / kSortRun;
    switch (phase) {
        case kBatchIngest: return (c + 255) / 256;
        case kBatchSort:
        case kBatchRunmerge: return 2 * runs;
        case kBatchDecrement:
        case kBatchIncrement: return (c * v.qlanes + 255) / 256;
        case kBatchMerge: return (v.W + kMergeTile - 1) / kMergeTile;
        case kBatchBuild: return (v.W + kBuildThreads - 1) / kBuildThreads;
        case kBatchLink: return (v.W + kLinkThreads - 1) / kLinkThreads;
        case kBatchUnion: return max(1, min(1024, (v.W + 1023) / 1024));  // persistent, queue-fed
        case kBatchLabel:
            if (v.list_cap >= 0) return max(1, min(1024, (v.W + 1023) / 1024));  // k_border
            return max(1, min(1024, (v.W + 4095) / 4096));  // grid-strided
        case kBatchFlatten: return max(1, min(1024, (v.W + 1023) / 1024));  // (2,048 points a block: 74 us a round against 55)
        default: return 0;
    }
}

bool batch_phase_split(int phase) {
    return phase == kBatchDecrement || phase == kBatchIncrement || phase == kBatchLink || phase == kBatchUnion ||
           phase == kBatchFlatten || phase == kBatchLabel;
}

#define RTDBS_BATCH_MD(PH, GRID, BLOCK, STREAM)                                      \
    do {                                                                           \
        const int dk = dim;                                                        \
        if (prec == kPrecFp32) {                                                   \
            switch (dk) {                                                          \
                case 1: k_batch<PH, kPrecFp32, 1><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 2: k_batch<PH, kPrecFp32, 2><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 3: k_batch<PH, kPrecFp32, 3><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 5: k_batch<PH, kPrecFp32, 5><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 6: k_batch<PH, kPrecFp32, 6><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                default: k_batch<PH, kPrecFp32, 7><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
            }                                                                      \
        } else {                                                                   \
            switch (dk) {                                                          \
                case 1: k_batch<PH, kPrecFp64, 1><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 2: k_batch<PH, kPrecFp64, 2><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 3: k_batch<PH, kPrecFp64, 3><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 5: k_batch<PH, kPrecFp64, 5><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                case 6: k_batch<PH, kPrecFp64, 6><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
                default: k_batch<PH, kPrecFp64, 7><<<GRID, BLOCK, 0, STREAM>>>(L); break; \
            }                                                                      \
        }                                                                          \
    } while (0)

cudaError_t launch_batch(int phase, int prec, int dim, const BatchLaunch& L, int total_blocks, int max_c,
                         cudaStream_t s) {
    if (total_blocks <= 0 || L.n <= 0) return cudaSuccess;
    const int t = batch_threads(phase);
    switch (phase) {
        case kBatchIngest: k_batch<kBatchIngest, 0, 0><<<total_blocks, t, 0, s>>>(L); break;
        case kBatchSort: k_batch<kBatchSort, 0, 0><<<total_blocks, t, 0, s>>>(L); break;
        case kBatchRunmerge:
            ensure_runmerge_smem();
            k_batch<kBatchRunmerge, 0, 0><<<total_blocks, t, runmerge_smem(max_c), s>>>(L);
            break;
        case kBatchMerge: k_batch<kBatchMerge, 0, 0><<<total_blocks, t, 0, s>>>(L); break;
        case kBatchBuild: k_batch<kBatchBuild, 0, 0><<<total_blocks, t, 0, s>>>(L); break;
        case kBatchDecrement: RTDBS_BATCH_MD(kBatchDecrement, total_blocks, t, s); break;
        case kBatchIncrement: RTDBS_BATCH_MD(kBatchIncrement, total_blocks, t, s); break;
        case kBatchLink: RTDBS_BATCH_MD(kBatchLink, total_blocks, t, s); break;
        case kBatchUnion: RTDBS_BATCH_MD(kBatchUnion, total_blocks, t, s); break;
        case kBatchFlatten: RTDBS_BATCH_MD(kBatchFlatten, total_blocks, t, s); break;
        case kBatchLabel: RTDBS_BATCH_MD(kBatchLabel, total_blocks, t, s); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Copies n separate point arrays into one packed buffer: block (x, y) moves
// part of array y.
__global__ void k_gather(const float* const* src, const long long* dst_off, const int* count, float* dst) {
    const int y = blockIdx.y;
    const float* a = src[y];
    float* d = dst + dst_off[y];
    const int n = count[y];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) d[i] = a[i];
}

cudaError_t launch_gather(const float* const* src, const long long* dst_off, const int* count, float* dst,
                          int n, int max_count, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int bx = max(1, min(64, (max_count + 1023) / 1024));
    k_gather<<<dim3(bx, n), 1024, 0, s>>>(src, dst_off, count, dst);
    return cudaGetLastError();
}

cudaError_t launch_counts_by_slot(const View& v, int* nn, cudaStream_t s) {
    const int sms = g_num_sms > 0 ? g_num_sms : 152;
    k_counts_by_slot<<<sms * 4, 256, 0, s>>>(v, nn);
    return cudaGetLastError();
}

}  // namespace rtdbs
