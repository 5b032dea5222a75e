// Neighbour search + smoothing-length solve, the plain seed, and the per-row
// FP64 distance accessor.
//
// Replaces cKDTree.query(pos[mask], des_ngb) (src/meshoid/Meshoid.py:157)
// followed by HsmlIter (src/meshoid/kernel_density.py:15-56).
//
// Search, first pass (k_knn_group, k <= 32): one thread per query over the
// particles streamed once for its warp of 32 consecutive queries; it accepts a
// query only when an error bound proves its set exact, and queues the rest.
//
// Search, warp path (k_knn_hsml; for k > 32 every query, in k_knn_pass):
// the query's radius R comes from a seed or the queue.  The level L with cell
// side s_L >= R (or R / 2) is chosen, the level-L cells that meet the sphere
// of radius R are looked up (dense table for L <= grid_level, refinement
// tables or a binary search of the Morton keys below), a list of too many
// particles is narrowed by splitting its cells (narrow_list), and every
// particle of those cells with FP32 d^2 <= R^2 is appended to a per-warp
// shared-memory buffer.  Fewer than k hits, or more than the buffer holds, and
// the warp searches again with a corrected radius.  The k smallest are
// picked by a 32-bucket histogram in (d/R)^dim; entries within 1e-5
// (relative, in d^2) of the k-th distance are re-decided with exact FP64
// distances and the particle index, so the set equals the k smallest by
// (FP64 d^2, index).
//
// h: norm * sum_j W(d_j/h) = k (norm = 32/3, 40/7, 8/3 in 3/2/1-D), solved by
// bracketed Newton (bisection fallback), one thread per query, on the k FP32
// distances of its row.  The function is C^2 and increasing in h, so the root
// is unique; the reference bisects to |n - k| <= 1e-13 and outputs the
// midpoint, i.e. the same root.
#include <algorithm>
#include <atomic>
#include <cfloat>

#include "mg_common.cuh"
#include "mg_f32x2.cuh"
#include "mg_grad2.cuh"
#include "mg_hsml.cuh"
#include "mg_refine.cuh"

namespace mg {

constexpr int kKnnWarps = 8;     // warps per block
constexpr float kBandEps = 1e-5f;
// The search loop's dynamic-trip-count loops are kept rolled: the kernel is
// bound by instruction issue and fetch (32 warps per SM at different points of
// a long loop body), and unrolled copies of these loops made it 14% slower
// (2^22 Plummer, first pass).
#define KNN_LOOP_HINT _Pragma("unroll 1")
#ifdef MG_KNN_SELECT_NOINLINE
#define KNN_SELECT_INLINE __noinline__
#else
#define KNN_SELECT_INLINE __forceinline__
#endif
#ifndef MG_KNN_MINBLOCKS
#define MG_KNN_MINBLOCKS 4
#endif
constexpr int kKnnMinBlocks = MG_KNN_MINBLOCKS;  // resident blocks per SM the register budget is cut for
constexpr int kList = 128;       // scan-list capacity per warp
constexpr int kScanLimit = 1 << 20;  // scan-list particles above which a first radius is cut unscanned
// Scan-list particles above which the list is narrowed (narrow_list) before it
// is scanned: about three times what a sphere with a buffer-full of
// neighbours lists.
#ifndef MG_KNN_NARROW
#define MG_KNN_NARROW 640
#endif
constexpr int kNarrow = MG_KNN_NARROW;
constexpr int kNarrowCell = 48;  // cells of up to this many particles are not split
// Queries taken from the common counter at a time: one from the queue, whose
// cost is uneven (2^22 clump mixture, searching: 18.4 ms one at a time, 19.2
// in runs of four), a run of consecutive queries when the warp path serves
// them all, so that a warp reuses its cell box.
constexpr unsigned kRun = 8;

// Passes over the queue (k_knn_pass, k_knn_heavy)
constexpr int kChunk = 32;     // consecutive queries per warp on the first pass
constexpr int kSplit = 192;    // cells holding more particles than this are split when they straddle the sphere
constexpr int kHeavy = 2048;   // scan-list particles above which a query goes to the block-wide path
constexpr int kHeavyItem = 2 * kList + 4;  // int32 words per queued heavy query: qi, nlist, pa[], off[]
constexpr int kHeavyThreads = 256;
constexpr int kHeavyBins = 1024;
constexpr int kHeavyCap = 1 << 16;   // heavy queries queued per pass (beyond: scanned by their warp)

struct KnnArgs {
    CellIndex ci;
    int64_t n;
    int dim, Lg;
    bool periodic;
    float box_hi, box_lo;
    double box64;  // the box side (periodic), FP64
    const double *frame;
    const uint64_t *keys;
    const uint32_t *cell_start;
    const int32_t *order;
    const float4 *hi;
    const float4 *lo;
    const double *pos64;
    const int32_t *queries;
    int64_t nq;
    int k;
    const float *seed_h;
    float radius_factor;
    float *radius;
    int32_t *ngb;
    float *hsml;
    int32_t *qstatus;
    const int32_t *qin;          // queries of the warp path (nullptr: all of them)
    const int32_t *qin_count;
    unsigned *next;              // next query of the warp path to take
    int32_t *qout;               // queries that the first pass leaves to the warp path
    int32_t *qout_count;
    int64_t *stats;
    int max_tries;   // radii searched per query
    int level_bias;  // search cells of side s with s >= R / 2^level_bias
};

struct KnnPassArgs : KnnArgs {
    float *rlo;  // largest radius seen with fewer than k particles (0: none)
    float *rhi;  // smallest radius seen with too many particles to scan (0: none)
    int last_pass;
    int32_t *heavy;        // heavy-query items of this pass (kHeavyItem words each)
    int32_t *heavy_count;  // items queued this pass (may exceed heavy_cap: the excess was not queued)
    int32_t *heavy_next;   // next item to take (block-wide path)
    int heavy_cap;
};

// Slot range [a, b) of the level-L cell with coordinates (cx, cy, cz).
#ifdef MG_KNN_LOOKUP_NOINLINE
#define KNN_LOOKUP_INLINE __noinline__
#else
#define KNN_LOOKUP_INLINE __forceinline__
#endif
__device__ KNN_LOOKUP_INLINE void cell_range(const CellIndex &ci, int L, uint32_t cx, uint32_t cy, uint32_t cz,
                                             uint32_t &a, uint32_t &b) {
    cell_lookup(ci, L, morton3(cx, cy, cz), a, b);
}

__device__ __forceinline__ float bucket_of(float t, int dim) {
    // t = d^2 / R^2 in [0, 1]; buckets uniform in enclosed volume (d/R)^dim
    float v = dim == 3 ? t * sqrtf(t) : (dim == 2 ? t : sqrtf(t));
    return fminf(31.0f, floorf(32.0f * v));
}

// FP64 squared distance, evaluated as ((dx*dx + dy*dy) + dz*dz) without
// contraction, nearest image when periodic; this is the parity rule's metric.
__device__ __forceinline__ double d2_exact(const double *__restrict__ p64, int32_t a, int32_t b,
                                           bool periodic, double box) {
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double d = __dsub_rn(p64[(int64_t)b * 3 + c], p64[(int64_t)a * 3 + c]);
        if (periodic && fabs(d) > 0.5 * box) d = -copysign(__dsub_rn(box, fabs(d)), d);
        s = __dadd_rn(s, __dmul_rn(d, d));
    }
    return s;
}

// Bitonic sort of one (key, tie) pair per lane, ascending.
template <class K>
__device__ __forceinline__ void warp_sort_pairs(K &key, int32_t &tie) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            K ok = __shfl_xor_sync(0xffffffffu, key, stride);
            int32_t ot = __shfl_xor_sync(0xffffffffu, tie, stride);
            const bool up = ((lane & size) == 0);
            const bool lower = ((lane & stride) == 0);
            const bool other_less = (ok < key) || (ok == key && ot < tie);
            // lower lane keeps the smaller when ascending
            const bool take = (lower == up) ? other_less : !other_less && !(ok == key && ot == tie);
            if (take) {
                key = ok;
                tie = ot;
            }
        }
    }
}

// Box index c (< 128) -> (ix, iy, iz) without integer division: the float
// quotients are exact enough for these small operands.
__device__ __forceinline__ void box_index(int c, float inv_nx, float inv_nxy, const int cnum[3], int &ix, int &iy,
                                          int &iz) {
    iz = (int)(((float)c + 0.5f) * inv_nxy);
    const int r = c - iz * cnum[0] * cnum[1];
    iy = (int)(((float)r + 0.5f) * inv_nx);
    ix = r - iy * cnum[0];
}

// Per-warp shared memory (KPL = neighbours per lane: k <= 32 KPL).
template <int KPL>
struct KnnSmem {
    static constexpr int kCap = KPL == 1 ? 224 : (KPL == 2 ? 320 : 448);  // candidate buffer
    float d[kCap];                  // candidate d^2
    int32_t i[kCap];                // candidate slot
    int32_t hist[32];
    float sel[32 * KPL];            // d^2 of the selected neighbours
    uint32_t ca[kList], cb[kList];  // cached box: cell ranges by box index
    uint32_t pa[kList], pb[kList];  // scan list of the current query
    uint64_t pc[kList];             // scan-list cell: level | x << 5 | y << 24 | z << 43 (periodic: x + 2^level, ..)
    uint32_t off[kList + 1];        // scan-list prefix offsets
};

struct WarpStats {
    int64_t cand = 0, retry = 0, band = 0, unres = 0, newton = 0, heavy = 0;
    int tries = 0;
    int64_t reason[3] = {0, 0, 0};
    int64_t phase[6] = {0, 0, 0, 0, 0, 0};
};

// Optional per-phase cycle counters (build with -DMG_KNN_PROFILE): stats[10..13]
// accumulate clock64() cycles of box lookup, list building, scan and selection,
// summed over warps; stats[14] the cycles of the slowest warp, stats[15] the
// number of scans over more than 8192 particles done by one warp.
#ifdef MG_KNN_PROFILE
#define KNN_TICK(var) const long long var = clock64()
#define KNN_PHASE(i, t0, t1) st.phase[i] += (t1) - (t0)
#else
#define KNN_TICK(var)
#define KNN_PHASE(i, t0, t1)
#endif

// Rare path: more than 32 candidates share the histogram bucket of the k-th
// neighbour (heavy exact or near ties).  Takes the r smallest one at a time.
// Returns the k-th squared distance.
template <class SM>
__device__ __noinline__ float select_boundary_slow(SM &S, int cnt, float invR2, int dim, int b_star, int c_lo,
                                                   int r, int32_t *row) {
    const int lane = threadIdx.x & 31;
    float T = 0.0f;
    for (int rep = 0; rep < r; ++rep) {
        float best = FLT_MAX;
        int32_t bslot = INT_MAX;
        int bidx = -1;
        for (int e = lane; e < cnt; e += 32) {
            if ((int)bucket_of(S.d[e] * invR2, dim) != b_star || S.i[e] < 0) continue;
            if (S.d[e] < best || (S.d[e] == best && S.i[e] < bslot)) {
                best = S.d[e];
                bslot = S.i[e];
                bidx = e;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int32_t os = __shfl_xor_sync(0xffffffffu, bslot, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
            if (ob < best || (ob == best && os < bslot)) {
                best = ob;
                bslot = os;
                bidx = oi;
            }
        }
        if (lane == 0) {
            row[c_lo + rep] = bslot;
            S.sel[c_lo + rep] = best;
            S.i[bidx] = -1 - bslot;  // mark taken
        }
        __syncwarp();
        T = best;
    }
    for (int e = lane; e < cnt; e += 32)
        if (S.i[e] < 0) S.i[e] = -1 - S.i[e];
    __syncwarp();
    return T;
}

// Absolute half-width added to the FP64 re-decision band around the k-th
// squared distance T.  FP32 d^2 from the hi/lo positions differs from the
// FP64 d^2 by up to ~2^-23 of itself, which the relative band (kBandEps)
// covers, plus 2 sqrt(T) dd, with dd ~3e-14 |x| the separation's share of the
// positions' hi/lo representation and of the low parts' rounding (2^-46 |x|
// per axis, over three axes).  That term decides for pairs closer than ~1e-9
// of their coordinates (a tight clump far from the frame centre).  xmag: the
// query's largest coordinate magnitude (or the box side, if larger).
__device__ __forceinline__ float band_abs(float T, float xmag) {
    const float dd = 3e-14f * xmag;
    return 2.0f * sqrtf(T) * dd + dd * dd;
}
__device__ __forceinline__ float query_mag(const float4 *__restrict__ hi, int32_t p, bool periodic, float box_hi) {
    const float4 h = hi[p];
    const float m = fmaxf(fabsf(h.x), fmaxf(fabsf(h.y), fabsf(h.z)));
    return periodic ? fmaxf(m, box_hi) : m;
}

// Rare path: several candidates lie within 1e-5 (relative, in d^2, widened by
// band_abs) of the k-th distance T.  Those are re-ranked by exact FP64 d^2 and then particle index;
// everything below the band is kept.  Rewrites the whole row.  Returns false
// if the band holds more than 32 candidates (flagged unresolved).
template <class SM>
__device__ __noinline__ bool resolve_band_fp64(SM &S, int cnt, float T, float wabs, int k, int32_t p, int32_t *row,
                                               const double *__restrict__ pos64, const int32_t *__restrict__ order,
                                               bool periodic, double box) {
    const int lane = threadIdx.x & 31;
    const float lo_band = T * (1.0f - kBandEps) - wabs, hi_band = T * (1.0f + kBandEps) + wabs;
    int nb = 0, nsure = 0;
    for (int e0 = 0; e0 < cnt; e0 += 32) {
        const int e = e0 + lane;
        const bool inb = e < cnt && S.d[e] >= lo_band && S.d[e] <= hi_band;
        const bool sure = e < cnt && S.d[e] < lo_band;
        const unsigned mb = __ballot_sync(0xffffffffu, inb);
        const unsigned ms = __ballot_sync(0xffffffffu, sure);
        if (inb) {
            const int pos = nb + __popc(mb & ((1u << lane) - 1u));
            if (pos < 32) S.pb[pos] = (uint32_t)S.i[e];
        }
        if (sure) {
            const int pos = nsure + __popc(ms & ((1u << lane) - 1u));
            row[pos] = S.i[e];
            S.sel[pos] = S.d[e];
        }
        nb += __popc(mb);
        nsure += __popc(ms);
    }
    __syncwarp();
    const int need = k - nsure;
    double key = DBL_MAX;
    int32_t tie = INT_MAX, carry = p;
    if (lane < min(nb, 32)) {
        carry = (int32_t)S.pb[lane];
        key = d2_exact(pos64, p, carry, periodic, box);
        tie = order[carry];
    }
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const double okey = __shfl_xor_sync(0xffffffffu, key, stride);
            const int32_t otie = __shfl_xor_sync(0xffffffffu, tie, stride);
            const int32_t ocar = __shfl_xor_sync(0xffffffffu, carry, stride);
            const bool up = ((lane & size) == 0);
            const bool lower = ((lane & stride) == 0);
            const bool other_less = (okey < key) || (okey == key && otie < tie);
            const bool same = (okey == key && otie == tie);
            if ((lower == up) ? other_less : (!other_less && !same)) {
                key = okey;
                tie = otie;
                carry = ocar;
            }
        }
    }
    if (lane < need) {
        row[nsure + lane] = carry;
        S.sel[nsure + lane] = (float)key;
    }
    __syncwarp();
    return !(nb > 32 || need > 32 || need > nb);
}

// FP32 squared distance from the query (h0, l0) to slot t; one expression for
// every path so that all of them see the same value.
__device__ __forceinline__ float cand_d2p(const float4 *__restrict__ hi, const float4 *__restrict__ lo, bool periodic,
                                         float box_hi, float box_lo, const float4 &h0, const float4 &l0, uint32_t t) {
    const float4 hb = hi[t], lb = lo[t];
    const float3 sv = periodic ? sep_hilo_periodic(h0, l0, hb, lb, box_hi, box_lo) : sep_hilo(h0, l0, hb, lb);
    return __fmaf_rn(sv.z, sv.z, __fmaf_rn(sv.y, sv.y, __fmul_rn(sv.x, sv.x)));
}
__device__ __forceinline__ float cand_d2(const KnnArgs &a, const float4 &h0, const float4 &l0, uint32_t t) {
    return cand_d2p(a.hi, a.lo, a.periodic, a.box_hi, a.box_lo, h0, l0, t);
}

// Scan-list candidate g -> slot, for a 32-wide chunk starting at g0: the
// boundaries of entries that start inside the chunk are OR-reduced into a bit
// mask and each lane counts those at or below it.  j0: entry holding g0 (updated
// to the entry holding g0 + 32).
template <class SM>
__device__ __forceinline__ uint32_t chunk_slot(const SM &S, int nlist, int total, int g0, int &j0, int lane) {
    const int bidx = j0 + 1 + lane;
    const uint32_t bnd = bidx <= nlist ? S.off[bidx] : 0xffffffffu;
    const uint32_t rel = bnd - (uint32_t)g0;
    const uint32_t bit = (bnd != 0xffffffffu && rel < 32u) ? (1u << rel) : 0u;
    const uint32_t mask = __reduce_or_sync(0xffffffffu, bit);
    const int j = j0 + __popc(mask & ((2u << lane) - 1u));
    const uint32_t t = g0 + lane < total ? S.pa[j] + (uint32_t)(g0 + lane - (int)S.off[j]) : 0u;
    j0 = __shfl_sync(0xffffffffu, j, 31);
    if (j0 + 1 <= nlist && (int)S.off[j0 + 1] == g0 + 32) ++j0;
    return t;
}

// Rare path (out of line, so that it stays out of the scan loop's instruction
// stream): the buffer overflowed during the scan, whose in-radius candidates
// beyond the buffer were binned into S.hist (32 buckets of (d/R)^dim).  Narrows
// the bucket of the k-th neighbour with up to two re-scans of 32 sub-buckets
// each.  Returns the upper edge v_hi (in (d/R)^dim) of the narrowest bucket
// found whose cumulative count reaches k.
template <int DIM, class SM>
__device__ __noinline__ float overflow_window(SM &S, const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                                              bool periodic, float box_hi, float box_lo, float4 h0, float4 l0,
                                              int nlist, int total, float R2, int k, int cap) {
    const int lane = threadIdx.x & 31;
    const float invR2 = 1.0f / R2;
    float v_lo = 0.0f, v_w = 1.0f / 32.0f, v_hi = 1.0f;
    int c_below = 0;
    for (int level = 0; level < 3; ++level) {
        if (level > 0) {  // re-scan, binning the current window into 32 sub-buckets
            int j0 = 0;
            for (int g0 = 0; g0 < total; g0 += 32) {
                const uint32_t t = chunk_slot(S, nlist, total, g0, j0, lane);
                if (g0 + lane < total) {
                    const float dd = cand_d2p(hi, lo, periodic, box_hi, box_lo, h0, l0, t);
                    if (dd <= R2) {
                        const float tt = dd * invR2;
                        const float v = DIM == 3 ? tt * sqrtf(tt) : (DIM == 2 ? tt : sqrtf(tt));
                        if (v >= v_lo && v < v_hi) atomicAdd(&S.hist[min(31, (int)((v - v_lo) / v_w))], 1);
                    }
                }
            }
            __syncwarp();
        }
        // locate the sub-bucket holding the k-th and narrow the window
        const int hc = S.hist[lane];
        const int cum = warp_incl_scan(hc) + c_below;
        const int bk = __ffs(__ballot_sync(0xffffffffu, cum >= k)) - 1;
        const int cum_bk = __shfl_sync(0xffffffffu, cum, max(bk, 0));
        const int hc_bk = __shfl_sync(0xffffffffu, hc, max(bk, 0));
        if (bk < 0) break;  // numerical edge: keep the window
        v_hi = v_lo + (float)(bk + 1) * v_w;
        if (cum_bk <= cap) break;
        c_below = cum_bk - hc_bk;
        v_lo = v_lo + (float)bk * v_w;
        v_w = v_w / 32.0f;
        __syncwarp();
        S.hist[lane] = 0;
        __syncwarp();
    }
    return v_hi;
}

// Rare path: the buffer has just overflowed; bin the buffered candidates
// (kept out of the scan loop's instruction stream unless MG_KNN_LAZY_INLINE).
#ifdef MG_KNN_LAZY_INLINE
#define KNN_LAZY_INLINE __forceinline__
#else
#define KNN_LAZY_INLINE __noinline__
#endif
template <int DIM, class SM>
__device__ KNN_LAZY_INLINE void lazy_hist_init(SM &S, float invR2) {
    const int lane = threadIdx.x & 31;
    S.hist[lane] = 0;
    __syncwarp();
    for (int e = lane; e < SM::kCap; e += 32) atomicAdd(&S.hist[(int)bucket_of(S.d[e] * invR2, DIM)], 1);
    __syncwarp();
}

// Rare path (out of line): a scan list of too many particles (a sparse query
// beside a dense clump, a first radius far too large) is narrowed before it is
// scanned.  Each round (1) bounds the k-th distance from above: the far
// corners of the listed cells, binned in 32 shells between the nearest of them
// and the radius (a clump seen from afar fills few shells of the whole radius),
// and the first shell by which cells of at least k particles lie inside it
// entirely; (2) drops the cells beyond that radius; (3) splits the larger
// cells into their non-empty children, four cells at a time, one child per lane
// (table lookups down to the refinement tables' leaves), the nearest first: a
// tighter bound drops most of the others unsplit, whereas splitting them in
// list order filled the list with cells of the clump's whole near face (one
// query of 2^24 clumped particles then took 28 ms).  The list stays complete
// for the radius it returns, which holds at least k particles.
// Handing such a query with its whole list to a block of 256 threads, which
// read every listed particle at least twice, took 4.9 of the 9.5 ms of 10^6
// Plummer particles with learned first radii, and 19.5 ms of 2^24 clumped
// ones.  Lengths in sides of the level-L cells; m0: rounding margin.
template <int DIM, class SM>
__device__ __noinline__ int narrow_list(SM &S, const KnnArgs &a, int32_t p, int nlist, int target, int L, float ux,
                                        float uy, float uz, int full, float scale, float m0, float &Rl) {
    const bool periodic = a.periodic;
    const int k = a.k;
    const int lane = threadIdx.x & 31;
    const float half_box = 0.5f * (float)(1u << L);
    auto corners = [&](uint64_t pc, float &near2, float &far2) {
        const int lv = (int)(pc & 31u);
        const float f = exp2f((float)(L - lv));
        const int off = periodic ? 1 << lv : 0;
        const float u[3] = {ux, uy, uz};
        near2 = far2 = 0.0f;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const float x0 = (float)((int)((pc >> (5 + 19 * d)) & 0x7ffffu) - off) * f, x1 = x0 + f;
            float nr = fmaxf(0.0f, fmaxf(x0 - u[d], u[d] - x1));
            float fa = fmaxf(fabsf(u[d] - x0), fabsf(u[d] - x1));
            if (full >> d & 1) {  // every cell of the axis is listed once, unwrapped
                nr = 0.0f;
                fa = fminf(fa, half_box);
            }
            near2 += nr * nr;
            far2 += fa * fa;
        }
    };
    for (int round = 0; round < 32; ++round) {
        S.hist[lane] = 0;
        float least = Rl;
        for (int i = lane; i < nlist; i += 32) {
            float near2, far2;
            corners(S.pc[i], near2, far2);
            if (S.pb[i] > S.pa[i]) least = fminf(least, sqrtf(far2) * 1.000001f + m0);
        }
        least = warp_min(least);
        const float width = (Rl - least) * (1.0f / 32.0f), bscale = 1.0f / fmaxf(width, 1e-30f);
        for (int i = lane; i < nlist; i += 32) {
            const int c = (int)(S.pb[i] - S.pa[i]);
            float near2, far2;
            corners(S.pc[i], near2, far2);
            const float t = (sqrtf(far2) * 1.000001f + m0 - least) * bscale;
            if (c > 0 && t < 32.0f) atomicAdd(&S.hist[max(0, (int)t)], c);
        }
        __syncwarp();
        const int cum = warp_incl_scan(S.hist[lane]);
        const unsigned reach = __ballot_sync(0xffffffffu, cum >= k);
        if (reach) Rl = fminf(Rl, (least + width * (float)__ffs(reach)) * 1.000001f);
        // keep what meets the sphere, find what to split
        const float rc = Rl * (1.0f + 1e-5f) + m0;
        int w = 0, total = 0;
        for (int i0 = 0; i0 < nlist; i0 += 32) {
            const int i = i0 + lane;
            const uint32_t ca = i < nlist ? S.pa[i] : 0u, cb = i < nlist ? S.pb[i] : 0u;
            const uint64_t pc = i < nlist ? S.pc[i] : 0ull;
            float near2 = 0.0f, far2;
            if (cb > ca) corners(pc, near2, far2);
            const bool keep = cb > ca && near2 <= rc * rc;
            const unsigned m = __ballot_sync(0xffffffffu, keep);  // (also: the chunk is read before it is rewritten)
            if (keep) {
                const int pos = w + __popc(m & ((1u << lane) - 1u));
                S.pa[pos] = ca;
                S.pb[pos] = cb;
                S.pc[pos] = pc;
            }
            w += __popc(m);
            total += __reduce_add_sync(0xffffffffu, keep ? (int)(cb - ca) : 0);
            __syncwarp();
        }
        nlist = w;
        if (total <= target) break;
        // entries lane, lane + 32, .. that may be split, by distance
        unsigned key[kList / 32];
#pragma unroll
        for (int c = 0; c < kList / 32; ++c) {
            const int i = lane + 32 * c;
            key[c] = 0xffffffffu;
            if (i < nlist && (int)(S.pb[i] - S.pa[i]) > kNarrowCell) {
                float near2, far2;
                corners(S.pc[i], near2, far2);
                if ((int)(S.pc[i] & 31u) < (periodic ? kMaxLevel - 1 : kMaxLevel))
                    key[c] = (__float_as_uint(near2) & ~(unsigned)(kList - 1)) | (unsigned)i;
            }
        }
        bool any = false;
        for (int step = 0; step < 4; ++step) {
            // the four nearest, eight lanes each
            int mine = -1, n = 0;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                unsigned best = key[0];
#pragma unroll
                for (int c = 1; c < kList / 32; ++c) best = min(best, key[c]);
                best = __reduce_min_sync(0xffffffffu, best);
                if (best == 0xffffffffu) continue;
                ++n;
                if (lane >> 3 == g) mine = (int)(best & (unsigned)(kList - 1));
#pragma unroll
                for (int c = 0; c < kList / 32; ++c)
                    if (key[c] == best) key[c] = 0xffffffffu;
            }
            if (n == 0) break;
            uint32_t ca = 0, cb = 0;
            uint64_t child = 0;
            if (mine >= 0) {
                const uint64_t pc = S.pc[mine];
                const int lv = (int)(pc & 31u) + 1;
                const uint64_t x = 2 * ((pc >> 5) & 0x7ffffu) + (lane & 1),
                               y = 2 * ((pc >> 24) & 0x7ffffu) + ((lane >> 1) & 1),
                               z = 2 * ((pc >> 43) & 0x7ffffu) + ((lane >> 2) & 1);
                const uint32_t wrap = (1u << lv) - 1u;
                child = (uint64_t)lv | (x << 5) | (y << 24) | (z << 43);
                cell_lookup(a.ci, lv, morton3((uint32_t)x & wrap, (uint32_t)y & wrap, (uint32_t)z & wrap), ca, cb);
            }
            float near2 = 0.0f, far2;
            if (cb > ca) corners(child, near2, far2);
            const bool keep = cb > ca && near2 <= rc * rc;
            const unsigned km = __ballot_sync(0xffffffffu, keep);
            // a cell's first child takes its place, the others are appended; a cell
            // whose children do not fit stays as it is
            int add = 0, first = -1;  // this group's first appended entry
            unsigned done = 0u;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int more = max(0, __popc(km >> (8 * g) & 0xffu) - 1);
                if (g < n && nlist + add + more <= kList) {
                    if (lane >> 3 == g) first = nlist + add;
                    done |= 0xffu << (8 * g);
                    add += more;
                }
            }
            if (!done) break;
            any = true;
            if (first >= 0) {
                const unsigned mk = km >> (lane & 24) & 0xffu;
                const int r = __popc(mk & ((1u << (lane & 7)) - 1u));
                const int pos = r == 0 ? mine : first + r - 1;
                if (keep) {
                    S.pa[pos] = ca;
                    S.pb[pos] = cb;
                    S.pc[pos] = child;
                } else if (mk == 0u && (lane & 7) == 0) {
                    S.pb[mine] = S.pa[mine];
                }
            }
            nlist += add;
            __syncwarp();
        }
        if (!any) {
            // no cell fits (or none is left to split): the bound from the particles
            // of the small cells themselves
            const float4 h0 = a.hi[p], l0 = a.lo[p];
            float least = Rl;
            S.hist[lane] = 0;
            for (int i = lane; i < nlist; i += 32) {
                float near2, far2;
                corners(S.pc[i], near2, far2);
                if (S.pb[i] - S.pa[i] <= (uint32_t)kNarrowCell) least = fminf(least, sqrtf(near2));
            }
            least = warp_min(least);
            const float width = (Rl - least) * (1.0f / 32.0f), bscale = 1.0f / fmaxf(width, 1e-30f);
            __syncwarp();
            for (int i = 0; i < nlist; ++i) {
                const uint32_t ca = S.pa[i], cb = S.pb[i];
                if (cb - ca > (uint32_t)kNarrowCell) continue;
                for (uint32_t t = ca + lane; t < cb; t += 32) {
                    const float d = sqrtf(cand_d2(a, h0, l0, t)) * scale * 1.00001f;
                    const float x = (d - least) * bscale;
                    if (x < 32.0f) atomicAdd(&S.hist[max(0, (int)x)], 1);
                }
            }
            __syncwarp();
            const unsigned found = __ballot_sync(0xffffffffu, warp_incl_scan(S.hist[lane]) >= k);
            const float Rn = found ? (least + width * (float)__ffs(found)) * 1.00001f : Rl;
            __syncwarp();
            if (!(Rn < 0.9995f * Rl)) break;
            Rl = Rn;
        }
    }
    return nlist;
}

// The k smallest of the cnt buffered candidates (all with d^2 <= R^2) by a
// 32-bucket histogram in (d/R)^dim: buckets below the k-th one are taken
// whole, the k-th bucket is sorted.  Writes the row and S.sel; returns the
// k-th squared distance T.
template <int DIM, class SM>
__device__ KNN_SELECT_INLINE float select_k(SM &S, int cnt, float invR2, int k, int32_t *row) {
    const int lane = threadIdx.x & 31;
    float T;
    S.hist[lane] = 0;
    __syncwarp();
    KNN_LOOP_HINT
    for (int e = lane; e < cnt; e += 32) atomicAdd(&S.hist[(int)bucket_of(S.d[e] * invR2, DIM)], 1);
    __syncwarp();
    const int hcount = S.hist[lane];
    const int cum = warp_incl_scan(hcount);
    const int b_star = __ffs(__ballot_sync(0xffffffffu, cum >= k)) - 1;
    const int cum_b = __shfl_sync(0xffffffffu, cum, b_star);
    const int m_b = __shfl_sync(0xffffffffu, hcount, b_star);
    const int c_lo = cum_b - m_b;
    const int r = k - c_lo;
    int out = 0, nb = 0;
    KNN_LOOP_HINT
    for (int e0 = 0; e0 < cnt; e0 += 32) {
        const int e = e0 + lane;
        const float v = e < cnt ? S.d[e] : FLT_MAX;
        const int bk = e < cnt ? (int)bucket_of(v * invR2, DIM) : 99;
        const bool sure = bk < b_star;
        const unsigned ms = __ballot_sync(0xffffffffu, sure);
        if (sure) {
            const int pos = out + __popc(ms & ((1u << lane) - 1u));
            row[pos] = S.i[e];
            S.sel[pos] = v;
        }
        out += __popc(ms);
        const bool bnd = bk == b_star;
        const unsigned mb = __ballot_sync(0xffffffffu, bnd);
        if (bnd && m_b <= 32) {
            const int pos = nb + __popc(mb & ((1u << lane) - 1u));
            S.pa[pos] = __float_as_uint(v);
            S.pb[pos] = (uint32_t)S.i[e];
        }
        nb += __popc(mb);
    }
    __syncwarp();
    if (m_b <= 32) {
        float key = lane < m_b ? __uint_as_float(S.pa[lane]) : FLT_MAX;
        int32_t tie = lane < m_b ? (int32_t)S.pb[lane] : INT_MAX;
        warp_sort_pairs(key, tie);
        if (lane < r) {
            row[c_lo + lane] = tie;
            S.sel[c_lo + lane] = key;
        }
        T = __shfl_sync(0xffffffffu, key, r - 1);
    } else {
        T = select_boundary_slow(S, cnt, invR2, DIM, b_star, c_lo, r, row);
    }
    __syncwarp();
    return T;
}

// After select_k (band inside the radius): candidates within 1e-5 of T are
// re-decided in FP64, then the selected d^2 are stored for the h solve.  A band
// of more than 32 flags the query unresolved.
template <class SM>
__device__ KNN_SELECT_INLINE void finish_row(SM &S, int cnt, float T, int k, int32_t p, int32_t qi, const KnnArgs &a,
                                             double side, WarpStats &st) {
    const int lane = threadIdx.x & 31;
    int32_t *row = a.ngb + (int64_t)qi * k;
    const float wabs = band_abs(T, query_mag(a.hi, p, a.periodic, a.box_hi));
    const float lo_band = T * (1.0f - kBandEps) - wabs, hi_band = T * (1.0f + kBandEps) + wabs;
    int nband = 0;
    KNN_LOOP_HINT
    for (int e0 = 0; e0 < cnt; e0 += 32) {
        const int e = e0 + lane;
        const bool inb = e < cnt && S.d[e] >= lo_band && S.d[e] <= hi_band;
        nband += __popc(__ballot_sync(0xffffffffu, inb));
    }
    if (nband > 1) {
        st.band += 1;
        const bool ok = resolve_band_fp64(S, cnt, T, wabs, k, p, row, a.pos64, a.order, a.periodic, side);
        if (!ok) {
            if (lane == 0) {
                atomicOr(a.qstatus + qi, MG_Q_UNRESOLVED);
                a.hsml[qi] = -(float)(4000000);
            }
            st.unres += 1;
            return;
        }
        if (lane == 0) atomicOr(a.qstatus + qi, MG_Q_BAND_FP64);
    }
}

// ---- k > 32 and query lists: passes over a queue ----------------------------------
// For k > 32 h is solved in FP32 from the row's distances in the row's order,
// so that the order of a row, which follows from how its query was searched,
// shows in h and the density at ~3e-8; and the FP64 values that Slice and
// Reconstruct build on the derivatives of a query list show it at ~1e-8.  These
// rows keep the search that produced them so far, and with it every bit of
// their results: a pass of warps over the queue (k_knn_pass), then a block per
// crowded query (k_knn_heavy), undecided queries queued for the next pass.  For
// k <= 32 h is solved in float-float, where the order does not show above
// 1e-13, and over a full set k_knn_hsml decides every query in place.
// Rare path (out of line): entries of the scan-list chunk starting at i0 that
// hold more than kSplit particles and straddle the sphere are replaced by their
// non-empty children that meet it (open 3-D boxes; children of a level-l cell
// are consecutive Morton codes, so 7 binary searches inside the parent's range
// give all 8 ranges).  Returns the new list length.
template <class SM>
__device__ __noinline__ int split_chunk(SM &S, int i0, int nlist, float ux0, float uy0, float uz0, float Rs, float rc,
                                        int L, const uint64_t *__restrict__ keys) {
    const int lane = threadIdx.x & 31;
    const int i = i0 + lane;
    bool split = false;
    if (i < nlist && S.pb[i] - S.pa[i] > (uint32_t)kSplit) {
        const uint64_t pc = S.pc[i];
        const int lv = (int)(pc & 31u);
        if (lv < kMaxLevel) {
            const float f = exp2f((float)(lv - L));
            const float x0 = (float)((pc >> 5) & 0x7ffffu), y0 = (float)((pc >> 24) & 0x7ffffu),
                        z0 = (float)((pc >> 43) & 0x7ffffu);
            const float ux = ux0 * f, uy = uy0 * f, uz = uz0 * f;
            const float fx = fmaxf(fabsf(ux - x0), fabsf(ux - x0 - 1.0f));
            const float fy = fmaxf(fabsf(uy - y0), fabsf(uy - y0 - 1.0f));
            const float fz = fmaxf(fabsf(uz - z0), fabsf(uz - z0 - 1.0f));
            const float rin = Rs * f * (1.0f - 1e-5f);
            split = fx * fx + fy * fy + fz * fz > rin * rin;  // not entirely inside
        }
    }
    unsigned sm = __ballot_sync(0xffffffffu, split);
    while (sm) {
        const int j = __ffs(sm) - 1;
        sm &= sm - 1;
        const int idx = i0 + j;
        const uint32_t A = S.pa[idx], B = S.pb[idx];
        const uint64_t pc = S.pc[idx];
        const int lv = (int)(pc & 31u) + 1;
        const uint32_t x0 = (uint32_t)((pc >> 5) & 0x7ffffu) * 2u, y0 = (uint32_t)((pc >> 24) & 0x7ffffu) * 2u,
                       z0 = (uint32_t)((pc >> 43) & 0x7ffffu) * 2u;
        const int ch = lane & 7;
        const uint32_t cx = x0 + (ch & 1), cy = y0 + ((ch >> 1) & 1), cz = z0 + (ch >> 2);
        const uint64_t code = morton3(cx, cy, cz);
        uint32_t lo = A;
        if (lane >= 1 && lane < 8) lo = lower_bound_prefix(keys, A, B, code, 3 * (kKeyBits - lv));
        uint32_t hi = __shfl_down_sync(0xffffffffu, lo, 1);
        if (ch == 7) hi = B;
        bool keep = false;
        if (lane < 8 && hi > lo) {
            const float f = exp2f((float)(lv - L));
            const float ux = ux0 * f, uy = uy0 * f, uz = uz0 * f, rr = rc * f;
            const float dx = fmaxf(0.0f, fmaxf((float)cx - ux, ux - (float)(cx + 1)));
            const float dy = fmaxf(0.0f, fmaxf((float)cy - uy, uy - (float)(cy + 1)));
            const float dz = fmaxf(0.0f, fmaxf((float)cz - uz, uz - (float)(cz + 1)));
            keep = dx * dx + dy * dy + dz * dz <= rr * rr;
        }
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (nlist + __popc(km) <= kList) {
            const int pos = nlist + __popc(km & ((1u << lane) - 1u));
            if (keep) {
                S.pa[pos] = lo;
                S.pb[pos] = hi;
                S.pc[pos] = (uint64_t)lv | ((uint64_t)cx << 5) | ((uint64_t)cy << 24) | ((uint64_t)cz << 43);
            }
            nlist += __popc(km);
            if (lane == 0) S.pb[idx] = S.pa[idx];  // parent replaced by its children
        }
        __syncwarp();
    }
    return nlist;
}

template <int DIM, int KPL>
__global__ __launch_bounds__(kKnnWarps * 32, kKnnMinBlocks) void k_knn_pass(const __grid_constant__ KnnPassArgs a) {
    using SM = KnnSmem<KPL>;
    constexpr int kKnnCap = SM::kCap;
    extern __shared__ __align__(16) unsigned char knn_smem[];
    SM &S = reinterpret_cast<SM *>(knn_smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t gwarp = (int64_t)blockIdx.x * kKnnWarps + wib;
    const int64_t nwarps = (int64_t)gridDim.x * kKnnWarps;
    const int64_t count = a.qin ? (int64_t)*a.qin_count : a.nq;
    const Frame fr = load_frame(a.frame);
    const float side = (float)fr.side;
    const float half_side = 0.5f * side;
    const int k = a.k;

    WarpStats st;
    int32_t my_retry = -1;  // lane i holds the i-th pending retry of this warp
    int n_retry = 0;

    // Queries are dealt to the warps in turn (the queue's cost is uneven); a
    // warp reuses the cell-box ranges of its previous query when the next one
    // needs the same box.
    int cL = -1, cmin_c[3] = {0, 0, 0}, cnum_c[3] = {0, 0, 0};  // cached box
    for (int64_t item = gwarp; item < count; item += nwarps) {
        const int32_t qi = a.qin ? a.qin[item] : (int32_t)item;
        const int32_t p = a.queries ? a.queries[qi] : qi;
        float R = a.qin ? a.radius[qi] : a.seed_h[qi] * a.radius_factor;
        // a negative queued radius was set by the block-wide path from a histogram
        // of the distances: it holds at least k and at most a buffer, so it is
        // scanned by this warp whatever the size of its scan list
        const bool cert = a.qin && R < 0.0f;
        R = fabsf(R);
        if (!(R > 0.0f) || !isfinite(R)) R = side * 1e-3f;
        float rlo = a.qin ? a.rlo[qi] : 0.0f, rhi = a.qin ? a.rhi[qi] : 0.0f;
        const float4 h0 = a.hi[p], l0 = a.lo[p];

        // ---- level and cell box ------------------------------------------
        // level_bias 1 allows R up to two cell sides, so with the rounding
        // margin of rc a box can reach 6 cells per axis; a box over kList
        // cells (the per-warp cache) is redone one level coarser (<= 4 per axis)
        int L = (int)floorf(log2f(side / R)) + a.level_bias;
        L = max(0, min(kMaxLevel, L));
        float cells_per_side, scale, u[3], rc;
        int cmin[3], cnum[3], ncell;
        bool full[3];  // periodic axis covered entirely: no distance test
        for (;;) {
            cells_per_side = (float)(1u << L);
            scale = cells_per_side / side;
            u[0] = ((h0.x + half_side) + l0.x) * scale;
            u[1] = ((h0.y + half_side) + l0.y) * scale;
            u[2] = ((h0.z + half_side) + l0.z) * scale;
            rc = R * scale * (1.0f + 1e-5f) + 1e-3f + cells_per_side * 2.4e-7f;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                full[d] = false;
                if (d >= DIM) {
                    cmin[d] = 0;
                    cnum[d] = 1;
                    continue;
                }
                int lo_c = (int)floorf(u[d] - rc), hi_c = (int)floorf(u[d] + rc);
                if (a.periodic) {
                    if (hi_c - lo_c + 1 >= (int)cells_per_side) {
                        lo_c = 0;
                        hi_c = (int)cells_per_side - 1;
                        full[d] = true;
                    }
                } else {
                    lo_c = max(lo_c, 0);
                    hi_c = min(hi_c, (int)cells_per_side - 1);
                }
                cmin[d] = lo_c;
                cnum[d] = max(0, hi_c - lo_c + 1);
            }
            ncell = cnum[0] * cnum[1] * cnum[2];
            if (ncell <= kList || L == 0) break;
            --L;
        }
        const float R2 = R * R;
        const float inv_nx = 1.0f / (float)max(cnum[0], 1), inv_nxy = 1.0f / (float)max(cnum[0] * cnum[1], 1);

        // ---- cell ranges: look up the box unless it is the cached one --------
        const bool same_box = (L == cL) && cmin[0] == cmin_c[0] && cmin[1] == cmin_c[1] && cmin[2] == cmin_c[2] &&
                              cnum[0] == cnum_c[0] && cnum[1] == cnum_c[1] && cnum[2] == cnum_c[2];
        if (!same_box) {
            // Cells that the previous box (same level) also held are copied from
            // the cache instead of looked up again (consecutive queries' boxes
            // are mostly shifted copies of each other); the new ranges are staged
            // in the scan-list arrays, free at this point, then moved.
            const bool shift_ok = L == cL;
            KNN_LOOP_HINT
            for (int cb = 0; cb < ncell; cb += 32) {
                const int c = cb + lane;
                if (c < ncell) {
                    int ix, iy, iz;
                    box_index(c, inv_nx, inv_nxy, cnum, ix, iy, iz);
                    int gx = cmin[0] + ix, gy = cmin[1] + iy, gz = cmin[2] + iz;
                    const int ox = gx - cmin_c[0], oy = gy - cmin_c[1], oz = gz - cmin_c[2];
                    uint32_t ca, cbnd;
                    if (shift_ok && ox >= 0 && ox < cnum_c[0] && oy >= 0 && oy < cnum_c[1] && oz >= 0 &&
                        oz < cnum_c[2]) {
                        const int oc = ox + cnum_c[0] * (oy + cnum_c[1] * oz);
                        ca = S.ca[oc];
                        cbnd = S.cb[oc];
                    } else {
                        const int M = (int)cells_per_side;
                        if (a.periodic) {
                            gx = ((gx % M) + M) % M;
                            gy = ((gy % M) + M) % M;
                            gz = ((gz % M) + M) % M;
                        }
                        if (DIM < 3) gz = 0;
                        if (DIM < 2) gy = 0;
                        cell_range(a.ci, L, (uint32_t)gx, (uint32_t)gy, (uint32_t)gz, ca, cbnd);
                    }
                    S.pa[c] = ca;
                    S.pb[c] = cbnd;
                }
            }
            __syncwarp();
            KNN_LOOP_HINT
            for (int c = lane; c < ncell; c += 32) {
                S.ca[c] = S.pa[c];
                S.cb[c] = S.pb[c];
            }
            cL = L;
            for (int d = 0; d < 3; ++d) {
                cmin_c[d] = cmin[d];
                cnum_c[d] = cnum[d];
            }
            __syncwarp();
        }
        // prune to the non-empty cells that meet this query's sphere
        int nlist = 0;
        KNN_LOOP_HINT
        for (int cb = 0; cb < ncell; cb += 32) {
            const int c = cb + lane;
            bool use = false;
            uint32_t ca = 0, cbnd = 0;
            int gx = 0, gy = 0, gz = 0;
            if (c < ncell) {
                ca = S.ca[c];
                cbnd = S.cb[c];
                int ix, iy, iz;
                box_index(c, inv_nx, inv_nxy, cnum, ix, iy, iz);
                gx = cmin[0] + ix;
                gy = cmin[1] + iy;
                gz = cmin[2] + iz;
                float dx = full[0] ? 0.0f : fmaxf(0.0f, fmaxf((float)gx - u[0], u[0] - (float)(gx + 1)));
                float dy = full[1] ? 0.0f : fmaxf(0.0f, fmaxf((float)gy - u[1], u[1] - (float)(gy + 1)));
                float dz = full[2] ? 0.0f : fmaxf(0.0f, fmaxf((float)gz - u[2], u[2] - (float)(gz + 1)));
                if (DIM < 3) dz = 0.0f;
                if (DIM < 2) dy = 0.0f;
                use = cbnd > ca && dx * dx + dy * dy + dz * dz <= rc * rc;
            }
            const unsigned m = __ballot_sync(0xffffffffu, use);
            const int pos = nlist + __popc(m & ((1u << lane) - 1u));
            if (use) {
                S.pa[pos] = ca;
                S.pb[pos] = cbnd;
                S.pc[pos] = (uint64_t)L | ((uint64_t)(uint32_t)gx << 5) | ((uint64_t)(uint32_t)gy << 24) |
                            ((uint64_t)(uint32_t)gz << 43);
            }
            nlist += __popc(m);
        }
        __syncwarp();
        // Split big cells that straddle the sphere into their 8 children: near a
        // dense clump or core the coarse cells of a sparse query would otherwise
        // put far more particles into the scan than the sphere holds.
        if (DIM == 3 && !a.periodic) {
            KNN_LOOP_HINT
            for (int i0 = 0; i0 < nlist; i0 += 32) {
                const int i = i0 + lane;
                const bool big = i < nlist && S.pb[i] - S.pa[i] > (uint32_t)kSplit;
                if (__any_sync(0xffffffffu, big)) nlist = split_chunk(S, i0, nlist, u[0], u[1], u[2], R * scale, rc, L, a.keys);
            }
        }
        // drop emptied entries and form prefix offsets (entries strictly non-empty)
        {
            int w = 0, total = 0;
            KNN_LOOP_HINT
            for (int i0 = 0; i0 < nlist; i0 += 32) {
                const int i = i0 + lane;
                const uint32_t ra = i < nlist ? S.pa[i] : 0u, rb = i < nlist ? S.pb[i] : 0u;
                const int n_i = (int)(rb - ra);
                __syncwarp();
                const unsigned m = __ballot_sync(0xffffffffu, n_i > 0);
                const int inc = warp_incl_scan(n_i);
                if (n_i > 0) {
                    const int pos = w + __popc(m & ((1u << lane) - 1u));
                    S.pa[pos] = ra;
                    S.pb[pos] = rb;
                    S.off[pos] = (uint32_t)(total + inc - n_i);
                }
                w += __popc(m);
                total += __shfl_sync(0xffffffffu, inc, 31);
            }
            nlist = w;
            if (lane == 0) S.off[nlist] = (uint32_t)total;
            __syncwarp();
            st.cand += total;
            // ---- gather candidates with d^2 <= R^2 -------------------------
            // mode 0 fills the buffer; modes 1..3 (only after an overflow) scan
            // again and histogram the in-radius candidates so the next radius
            // can be cut to the bucket that holds the k-th neighbour.  More than
            // kScanLimit particles in the scan list: no scan, the radius shrinks
            // by the volume ratio (bracketed).
            int cnt = 0;
            const float invR2 = 1.0f / R2;
            // (only before any radius of this query has held fewer than k:
            // after that the box is always scanned, so the search converges)
            const bool too_big = total > kScanLimit && rlo == 0.0f && !cert;
            // a long scan list goes to the block-wide path (k_knn_heavy) with
            // its list, so that one warp does not scan it several times while
            // the rest of the grid waits for it
            if (!too_big && !cert && total > kHeavy && a.heavy_cap > 0) {
                int slot = 0;
                if (lane == 0) slot = atomicAdd(a.heavy_count, 1);
                slot = __shfl_sync(0xffffffffu, slot, 0);
                if (slot < a.heavy_cap) {
                    int32_t *item = a.heavy + (int64_t)slot * kHeavyItem;
                    if (lane == 0) {
                        item[0] = qi;
                        item[1] = nlist;
                        a.radius[qi] = R;
                        a.rlo[qi] = rlo;
                        a.rhi[qi] = rhi;
                    }
                    for (int e = lane; e < nlist; e += 32) item[2 + e] = (int32_t)S.pa[e];
                    for (int e = lane; e <= nlist; e += 32) item[2 + kList + e] = (int32_t)S.off[e];
                    st.heavy += 1;
                    __syncwarp();
                    continue;
                }
            }
            float v_hi = 1.0f;
            if (!too_big) {
                int j0 = 0;
                KNN_LOOP_HINT
                for (int g0 = 0; g0 < total; g0 += 32) {
                    const uint32_t t = chunk_slot(S, nlist, total, g0, j0, lane);
                    const float dd = g0 + lane < total ? cand_d2(a, h0, l0, t) : FLT_MAX;
                    const bool in = dd <= R2;
                    const unsigned m = __ballot_sync(0xffffffffu, in);
                    const int pos = cnt + __popc(m & ((1u << lane) - 1u));
                    if (in && pos < kKnnCap) {
                        S.d[pos] = dd;
                        S.i[pos] = (int32_t)t;
                    }
                    const int before = cnt;
                    cnt += __popc(m);
                    // Lazy histogram: the first time the buffer overflows, the
                    // buffered candidates are binned; from then on every new
                    // in-radius candidate is binned directly, so an overflow
                    // usually needs no second scan.
                    if (before <= kKnnCap && cnt > kKnnCap) lazy_hist_init<DIM>(S, invR2);
                    if (cnt > kKnnCap && in && pos >= kKnnCap) atomicAdd(&S.hist[(int)bucket_of(dd * invR2, DIM)], 1);
                }
                __syncwarp();
                if (cnt > kKnnCap)
                    v_hi = overflow_window<DIM>(S, a.hi, a.lo, a.periodic, a.box_hi, a.box_lo, h0, l0, nlist, total, R2,
                                                k, kKnnCap);
            }

            // ---- radius updates (bracketed) ------------------------------------
            // rlo: largest radius seen holding fewer than k; rhi: smallest radius
            // seen holding more than the buffer (so at least k).  Growth is a
            // geometric guess capped by rhi (geometric mean once both are known);
            // an overflow cuts the radius to the histogram bucket holding the k-th
            // neighbour, which holds at least k by construction.
            float Rnew = -1.0f;
            int reason = 0;
            if (too_big) {
                Rnew = R * fmaxf(0.25f, powf(0.5f * kKnnCap / (float)total, 1.0f / DIM));
                reason = 2;
            } else if (cnt < k) {
                rlo = fmaxf(rlo, R);
                const float g = 1.25f * powf((float)k / (float)max(cnt, 1), 1.0f / DIM);
                Rnew = R * fminf(fmaxf(g, 1.25f), 4.0f);
                if (rhi > 0.0f && Rnew >= rhi) Rnew = sqrtf(rlo * rhi);
                reason = 1;
            } else if (cnt > kKnnCap) {
                rhi = (rhi > 0.0f) ? fminf(rhi, R) : R;
                Rnew = R * (DIM == 3 ? cbrtf(v_hi) : (DIM == 2 ? sqrtf(v_hi) : v_hi)) * 1.00001f;
                if (Rnew >= R) Rnew = R * 0.999f;
                reason = 2;
            }

            // ---- select the k smallest: bucket histogram ------------------------
            float T = 0.0f;
            int32_t *row = a.ngb + (int64_t)qi * k;
            if (Rnew < 0.0f) {
                T = select_k<DIM>(S, cnt, invR2, k, row);
                // the band around T must lie inside the searched radius
                const float wabs = band_abs(T, query_mag(a.hi, p, a.periodic, a.box_hi));
                if (T * (1.0f + kBandEps) + 2.0f * wabs > R2) {
                    Rnew = sqrtf(T * (1.0f + 2.0f * kBandEps) + 4.0f * wabs) * 1.0001f;
                    reason = 3;
                }
            }

            if (Rnew > 0.0f) {
                st.reason[reason - 1] += 1;
                if (a.last_pass) {
                    if (lane == 0) {
                        atomicOr(a.qstatus + qi, MG_Q_UNRESOLVED);
                        // diagnostics for the caller: last radius and candidate count
                        a.radius[qi] = R;
                        a.hsml[qi] = -(float)((too_big ? total : cnt) + 1000000 * reason);
                    }
                    st.unres += 1;
                } else {
                    if (lane == 0) {
                        a.radius[qi] = Rnew;
                        a.rlo[qi] = rlo;
                        a.rhi[qi] = rhi;
                    }
                    if (lane == n_retry) my_retry = qi;
                    ++n_retry;
                    st.retry += 1;
                    if (n_retry == 32) {
                        int base = 0;
                        if (lane == 0) base = atomicAdd(a.qout_count, 32);
                        base = __shfl_sync(0xffffffffu, base, 0);
                        a.qout[base + lane] = my_retry;
                        n_retry = 0;
                    }
                }
                continue;
            }

            finish_row(S, cnt, T, k, p, qi, a, fr.side, st);
        }
    }

    // flush pending retries
    if (n_retry > 0) {
        int base = 0;
        if (lane == 0) base = atomicAdd(a.qout_count, n_retry);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < n_retry) a.qout[base + lane] = my_retry;
    }
    // statistics: one atomic per warp
    if (lane == 0 && a.stats) {
        if (st.cand) atomicAdd((unsigned long long *)&a.stats[1], (unsigned long long)st.cand);
        if (st.retry) atomicAdd((unsigned long long *)&a.stats[2], (unsigned long long)st.retry);
        if (st.band) atomicAdd((unsigned long long *)&a.stats[3], (unsigned long long)st.band);
        if (st.unres) atomicAdd((unsigned long long *)&a.stats[4], (unsigned long long)st.unres);
        if (st.newton) atomicAdd((unsigned long long *)&a.stats[5], (unsigned long long)st.newton);
        for (int r = 0; r < 3; ++r)
            if (st.reason[r]) atomicAdd((unsigned long long *)&a.stats[6 + r], (unsigned long long)st.reason[r]);
        if (st.heavy) atomicAdd((unsigned long long *)&a.stats[9], (unsigned long long)st.heavy);
    }
}

// ---- heavy queries: one block per query ------------------------------------------
// A query whose scan list holds more than kHeavy particles (a dense clump inside
// the sphere of a sparse query) is handed over with its list.  A block
// histograms the in-radius candidates in kHeavyBins bins of (d/R)^dim, narrows
// the bin holding the k-th neighbour until it and everything below it fit the
// buffer, gathers those (d^2 <= Rc^2) and warp 0 selects as the warp path does.
template <int DIM>
__device__ __forceinline__ float vol_of(float t) {  // t = d^2 / R^2
    return DIM == 3 ? t * sqrtf(t) : (DIM == 2 ? t : sqrtf(t));
}
template <int DIM>
__device__ __forceinline__ float radius_of_vol(float v) {
    return DIM == 3 ? cbrtf(v) : (DIM == 2 ? sqrtf(v) : v);
}

template <int KPL>
struct HeavySmem {
    KnnSmem<KPL> S;  // warp 0's selection buffer
    uint32_t pa[kList];
    uint32_t off[kList + 1];
    int hist[kHeavyBins];
    int wsum[kHeavyThreads / 32];
    int item, bstar, cum_prev, cum_b, cnt, total_in;
};

template <int DIM, int KPL>
__global__ __launch_bounds__(kHeavyThreads) void k_knn_heavy(const __grid_constant__ KnnPassArgs a) {
    __shared__ HeavySmem<KPL> H;
    constexpr int kCap = KnnSmem<KPL>::kCap;
    static_assert(kHeavyBins == 4 * kHeavyThreads, "four bins per thread");
    static_assert(2 * kCap <= kHeavyBins, "sort scratch lives in the histogram");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int navail = min(*a.heavy_count, a.heavy_cap);
    const Frame fr = load_frame(a.frame);
    const int k = a.k;
    WarpStats st;
    for (;;) {
        if (tid == 0) H.item = atomicAdd(a.heavy_next, 1);
        __syncthreads();
        const int h = H.item;
        if (h >= navail) break;
        const int32_t *item = a.heavy + (int64_t)h * kHeavyItem;
        const int32_t qi = item[0];
        const int nlist = item[1];
        for (int e = tid; e < nlist; e += kHeavyThreads) H.pa[e] = (uint32_t)item[2 + e];
        for (int e = tid; e <= nlist; e += kHeavyThreads) H.off[e] = (uint32_t)item[2 + kList + e];
        __syncthreads();
        const int total = (int)H.off[nlist];
        const int32_t p = a.queries ? a.queries[qi] : qi;
        const float4 h0 = a.hi[p], l0 = a.lo[p];
        const float R = a.radius[qi];
        float rlo = a.rlo[qi], rhi = a.rhi[qi];
        const float R2 = R * R, invR2 = 1.0f / R2;
        // candidate g of the flattened list -> slot (largest entry with off <= g)
        auto slot_of = [&](int g) -> uint32_t {
            int lo = 0, hi = nlist - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((int)H.off[mid] <= g)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            return H.pa[lo] + (uint32_t)(g - (int)H.off[lo]);
        };

        // ---- narrow the bin of the k-th neighbour ----------------------------
        float v_lo = 0.0f, v_w = 1.0f / kHeavyBins, Rc = -1.0f;
        int c_below = 0, in_radius = -1;
        for (int lev = 0; lev < 3; ++lev) {
            for (int b = tid; b < kHeavyBins; b += kHeavyThreads) H.hist[b] = 0;
            if (tid == 0) H.bstar = -1;
            __syncthreads();
            for (int g0 = tid; g0 < total; g0 += 4 * kHeavyThreads) {
                float dd[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int g = g0 + u * kHeavyThreads;
                    dd[u] = g < total ? cand_d2(a, h0, l0, slot_of(g)) : FLT_MAX;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (dd[u] <= R2) {
                        const float v = vol_of<DIM>(dd[u] * invR2);
                        if (v >= v_lo) {
                            const float x = (v - v_lo) / v_w;  // lev 0: v <= 1, the last bin takes v == 1
                            if (x < (float)kHeavyBins)
                                atomicAdd(&H.hist[(int)x], 1);
                            else if (lev == 0)
                                atomicAdd(&H.hist[kHeavyBins - 1], 1);
                        }
                    }
                }
            }
            __syncthreads();
            {
                int c[4], sum = 0;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    c[u] = H.hist[4 * tid + u];
                    sum += c[u];
                }
                const int incl = warp_incl_scan(sum);
                if (lane == 31) H.wsum[warp] = incl;
                __syncthreads();
                int woff = 0;
                for (int w = 0; w < warp; ++w) woff += H.wsum[w];
                int run = c_below + woff + incl - sum;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int before = run;
                    run += c[u];
                    if (before < k && run >= k) {
                        H.bstar = 4 * tid + u;
                        H.cum_prev = before;
                        H.cum_b = run;
                    }
                }
                if (tid == kHeavyThreads - 1) H.total_in = run;
            }
            __syncthreads();
            const int bstar = H.bstar;
            if (lev == 0) in_radius = H.total_in;
            if (bstar < 0) break;  // fewer than k inside R (level 0), else a numerical edge
            const float v_hi = v_lo + (float)(bstar + 1) * v_w;
            if (H.cum_b <= kCap || lev == 2) {
                Rc = R * radius_of_vol<DIM>(fminf(v_hi, 1.0f)) * 1.00001f;
                break;
            }
            c_below = H.cum_prev;
            v_lo = v_lo + (float)bstar * v_w;
            v_w = v_w / (float)kHeavyBins;
            __syncthreads();
        }

        // ---- outcome: gather + select, or a new radius ------------------------
        float Rnew = -1.0f;
        bool certify = false;
        int reason = 0;
        if (in_radius >= 0 && in_radius < k) {  // too few inside R: grow (bracketed)
            rlo = fmaxf(rlo, R);
            const float g = 1.25f * powf((float)k / (float)max(in_radius, 1), 1.0f / DIM);
            Rnew = R * fminf(fmaxf(g, 1.25f), 4.0f);
            if (rhi > 0.0f && Rnew >= rhi) Rnew = sqrtf(rlo * rhi);
            reason = 1;
        } else {
            if (in_radius > kCap) rhi = (rhi > 0.0f) ? fminf(rhi, R) : R;
            if (Rc < 0.0f) Rc = R;
            const float Rc2 = Rc * Rc;
            if (tid == 0) H.cnt = 0;
            __syncthreads();
            for (int g0 = tid; g0 < total; g0 += 4 * kHeavyThreads) {
                float dd[4];
                uint32_t t[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int g = g0 + u * kHeavyThreads;
                    t[u] = g < total ? slot_of(g) : 0u;
                    dd[u] = g < total ? cand_d2(a, h0, l0, t[u]) : FLT_MAX;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (dd[u] <= Rc2) {
                        const int pos = atomicAdd(&H.cnt, 1);
                        if (pos < kCap) {
                            H.S.d[pos] = dd[u];
                            H.S.i[pos] = (int32_t)t[u];
                        }
                    }
                }
            }
            __syncthreads();
            const int cnt = H.cnt;
            if (cnt < k || cnt > kCap) {
                // rounding at the bin edge or ties finer than the bins: the warp
                // path scans this radius and handles the overflow itself
                Rnew = Rc;
                certify = true;
                reason = 2;
            } else {
                // deterministic buffer order (by slot) before selecting
                int *tmp_i = H.hist;
                float *tmp_d = reinterpret_cast<float *>(H.hist + kCap);
                for (int e = tid; e < cnt; e += kHeavyThreads) {
                    const int32_t me = H.S.i[e];
                    int r = 0;
                    for (int j = 0; j < cnt; ++j) r += H.S.i[j] < me || (H.S.i[j] == me && j < e);
                    tmp_i[r] = me;
                    tmp_d[r] = H.S.d[e];
                }
                __syncthreads();
                for (int e = tid; e < cnt; e += kHeavyThreads) {
                    H.S.i[e] = tmp_i[e];
                    H.S.d[e] = tmp_d[e];
                }
                __syncthreads();
                if (warp == 0) {
                    int32_t *row = a.ngb + (int64_t)qi * k;
                    const float T = select_k<DIM>(H.S, cnt, 1.0f / Rc2, k, row);
                    const float wabs = band_abs(T, query_mag(a.hi, p, a.periodic, a.box_hi));
                    if (T * (1.0f + kBandEps) + 2.0f * wabs > Rc2) {
                        Rnew = sqrtf(T * (1.0f + 2.0f * kBandEps) + 4.0f * wabs) * 1.0001f;
                        certify = true;
                        reason = 3;
                    } else {
                        finish_row(H.S, cnt, T, k, p, qi, a, fr.side, st);
                    }
                }
            }
        }
        if (tid == 0 && Rnew > 0.0f) {
            st.reason[reason - 1] += 1;
            if (a.last_pass) {
                atomicOr(a.qstatus + qi, MG_Q_UNRESOLVED);
                a.radius[qi] = R;
                a.hsml[qi] = -(float)(in_radius + 1000000 * reason);
                st.unres += 1;
            } else {
                a.radius[qi] = certify ? -Rnew : Rnew;
                a.rlo[qi] = rlo;
                a.rhi[qi] = rhi;
                a.qout[atomicAdd(a.qout_count, 1)] = qi;
                st.retry += 1;
            }
        }
        __syncthreads();
    }
    if (tid == 0 && a.stats) {
        if (st.retry) atomicAdd((unsigned long long *)&a.stats[2], (unsigned long long)st.retry);
        if (st.band) atomicAdd((unsigned long long *)&a.stats[3], (unsigned long long)st.band);
        if (st.unres) atomicAdd((unsigned long long *)&a.stats[4], (unsigned long long)st.unres);
        for (int r = 0; r < 3; ++r)
            if (st.reason[r]) atomicAdd((unsigned long long *)&a.stats[6 + r], (unsigned long long)st.reason[r]);
    }
}

// Warp-per-query path: persistent warps take queries from a common counter and
// search each until it is decided, growing or cutting its radius in place; a
// query is not queued again for another pass.  Passing the undecided queries
// through a queue took a launch pair and an empty-queue check per possible
// pass (45 launches, most on an empty queue: ~0.1 ms of the 1.3 ms of a small
// set).
template <int DIM>
__global__ __launch_bounds__(kKnnWarps * 32, kKnnMinBlocks) void k_knn_hsml(const __grid_constant__ KnnArgs a) {
    using SM = KnnSmem<1>;
    constexpr int kKnnCap = SM::kCap;
    extern __shared__ __align__(16) unsigned char knn_smem[];
    SM &S = reinterpret_cast<SM *>(knn_smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned count = a.qin ? (unsigned)*a.qin_count : (unsigned)a.nq;
    const unsigned run = a.qin ? 1u : kRun;
    const Frame fr = load_frame(a.frame);
    const float side = (float)fr.side;
    const float half_side = 0.5f * side;
    const int k = a.k;

    WarpStats st;
#ifdef MG_KNN_PROFILE
    const long long t_warp0 = clock64();
#endif
    // the cell-box ranges of the warp's previous search, reused when the next
    // one needs the same box (consecutive queries are neighbours in Morton order)
    int cL = -1, cmin_c[3] = {0, 0, 0}, cnum_c[3] = {0, 0, 0};  // cached box
    for (;;) {
    unsigned c0 = 0;
    if (lane == 0) c0 = atomicAdd(a.next, run);
    c0 = __shfl_sync(0xffffffffu, c0, 0);
    if (c0 >= count) break;
    const unsigned c1 = min(count, c0 + run);
    for (unsigned item = c0; item < c1; ++item) {
        const int32_t qi = a.qin ? a.qin[item] : (int32_t)item;
        const int32_t p = a.queries ? a.queries[qi] : qi;
        float R = a.qin ? a.radius[qi] : a.seed_h[qi] * a.radius_factor;
        if (!(R > 0.0f) || !isfinite(R)) R = side * 1e-3f;
        // rlo: largest radius seen holding fewer than k; rhi: smallest radius
        // seen holding more than the buffer (so at least k); 0: none
        float rlo = 0.0f, rhi = 0.0f;
        const float4 h0 = a.hi[p], l0 = a.lo[p];
        bool listed = false;  // the scan list is complete for this radius
        int nlist = 0, total = 0;
        for (int tries = 1;; ++tries) {
        KNN_TICK(t_a);
        if (!listed) {
        // ---- level and cell box ------------------------------------------
        // level_bias 1 allows R up to two cell sides, so with the rounding
        // margin of rc a box can reach 6 cells per axis; a box over kList
        // cells (the per-warp cache) is redone one level coarser (<= 4 per axis)
        int L = (int)floorf(log2f(side / R)) + a.level_bias;
        L = max(0, min(kMaxLevel, L));
        float cells_per_side, scale, u[3], rc;
        int cmin[3], cnum[3], ncell;
        bool full[3];  // periodic axis covered entirely: no distance test
        for (;;) {
            cells_per_side = (float)(1u << L);
            scale = cells_per_side / side;
            u[0] = ((h0.x + half_side) + l0.x) * scale;
            u[1] = ((h0.y + half_side) + l0.y) * scale;
            u[2] = ((h0.z + half_side) + l0.z) * scale;
            rc = R * scale * (1.0f + 1e-5f) + 1e-3f + cells_per_side * 2.4e-7f;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                full[d] = false;
                if (d >= DIM) {
                    cmin[d] = 0;
                    cnum[d] = 1;
                    continue;
                }
                int lo_c = (int)floorf(u[d] - rc), hi_c = (int)floorf(u[d] + rc);
                if (a.periodic) {
                    if (hi_c - lo_c + 1 >= (int)cells_per_side) {
                        lo_c = 0;
                        hi_c = (int)cells_per_side - 1;
                        full[d] = true;
                    }
                } else {
                    lo_c = max(lo_c, 0);
                    hi_c = min(hi_c, (int)cells_per_side - 1);
                }
                cmin[d] = lo_c;
                cnum[d] = max(0, hi_c - lo_c + 1);
            }
            ncell = cnum[0] * cnum[1] * cnum[2];
            if (ncell <= kList || L == 0) break;
            --L;
        }
        const float inv_nx = 1.0f / (float)max(cnum[0], 1), inv_nxy = 1.0f / (float)max(cnum[0] * cnum[1], 1);

        // ---- cell ranges: look up the box unless it is the cached one --------
        const bool same_box = (L == cL) && cmin[0] == cmin_c[0] && cmin[1] == cmin_c[1] && cmin[2] == cmin_c[2] &&
                              cnum[0] == cnum_c[0] && cnum[1] == cnum_c[1] && cnum[2] == cnum_c[2];
        if (!same_box) {
            // Cells that the previous box (same level) also held are copied from
            // the cache instead of looked up again (consecutive queries' boxes
            // are mostly shifted copies of each other); the new ranges are staged
            // in the scan-list arrays, free at this point, then moved.
            const bool shift_ok = L == cL;
            KNN_LOOP_HINT
            for (int cb = 0; cb < ncell; cb += 32) {
                const int c = cb + lane;
                if (c < ncell) {
                    int ix, iy, iz;
                    box_index(c, inv_nx, inv_nxy, cnum, ix, iy, iz);
                    int gx = cmin[0] + ix, gy = cmin[1] + iy, gz = cmin[2] + iz;
                    const int ox = gx - cmin_c[0], oy = gy - cmin_c[1], oz = gz - cmin_c[2];
                    uint32_t ca, cbnd;
                    if (shift_ok && ox >= 0 && ox < cnum_c[0] && oy >= 0 && oy < cnum_c[1] && oz >= 0 &&
                        oz < cnum_c[2]) {
                        const int oc = ox + cnum_c[0] * (oy + cnum_c[1] * oz);
                        ca = S.ca[oc];
                        cbnd = S.cb[oc];
                    } else {
                        const int M = (int)cells_per_side;
                        if (a.periodic) {
                            gx = ((gx % M) + M) % M;
                            gy = ((gy % M) + M) % M;
                            gz = ((gz % M) + M) % M;
                        }
                        if (DIM < 3) gz = 0;
                        if (DIM < 2) gy = 0;
                        cell_range(a.ci, L, (uint32_t)gx, (uint32_t)gy, (uint32_t)gz, ca, cbnd);
                    }
                    S.pa[c] = ca;
                    S.pb[c] = cbnd;
                }
            }
            __syncwarp();
            KNN_LOOP_HINT
            for (int c = lane; c < ncell; c += 32) {
                S.ca[c] = S.pa[c];
                S.cb[c] = S.pb[c];
            }
            cL = L;
            for (int d = 0; d < 3; ++d) {
                cmin_c[d] = cmin[d];
                cnum_c[d] = cnum[d];
            }
            __syncwarp();
        }
        KNN_TICK(t_b);
        KNN_PHASE(0, t_a, t_b);
        // prune to the non-empty cells that meet this query's sphere
        nlist = 0;
        int listed_total = 0;
        const uint32_t gofs = a.periodic ? (uint32_t)cells_per_side : 0u;
        KNN_LOOP_HINT
        for (int cb = 0; cb < ncell; cb += 32) {
            const int c = cb + lane;
            bool use = false;
            uint32_t ca = 0, cbnd = 0;
            int gx = 0, gy = 0, gz = 0;
            if (c < ncell) {
                ca = S.ca[c];
                cbnd = S.cb[c];
                int ix, iy, iz;
                box_index(c, inv_nx, inv_nxy, cnum, ix, iy, iz);
                gx = cmin[0] + ix;
                gy = cmin[1] + iy;
                gz = cmin[2] + iz;
                float dx = full[0] ? 0.0f : fmaxf(0.0f, fmaxf((float)gx - u[0], u[0] - (float)(gx + 1)));
                float dy = full[1] ? 0.0f : fmaxf(0.0f, fmaxf((float)gy - u[1], u[1] - (float)(gy + 1)));
                float dz = full[2] ? 0.0f : fmaxf(0.0f, fmaxf((float)gz - u[2], u[2] - (float)(gz + 1)));
                if (DIM < 3) dz = 0.0f;
                if (DIM < 2) dy = 0.0f;
                use = cbnd > ca && dx * dx + dy * dy + dz * dz <= rc * rc;
            }
            const unsigned m = __ballot_sync(0xffffffffu, use);
            const int pos = nlist + __popc(m & ((1u << lane) - 1u));
            if (use) {
                S.pa[pos] = ca;
                S.pb[pos] = cbnd;
                S.pc[pos] = (uint64_t)L | ((uint64_t)((uint32_t)gx + gofs) << 5) |
                            ((uint64_t)((uint32_t)gy + gofs) << 24) | ((uint64_t)((uint32_t)gz + gofs) << 43);
            }
            nlist += __popc(m);
            listed_total += __reduce_add_sync(0xffffffffu, use ? (int)(cbnd - ca) : 0);
        }
        __syncwarp();
        // (a coordinate of the list holds 19 bits: three boxes of level 17)
        if (listed_total > kNarrow && (!a.periodic || L < kMaxLevel)) {
            float Rl = R * scale;
            const float R0 = Rl;
            const int fm = (full[0] ? 1 : 0) | (full[1] ? 2 : 0) | (full[2] ? 4 : 0);
            nlist = narrow_list<DIM>(S, a, p, nlist, kNarrow / 2, L, u[0], u[1], u[2], fm, scale,
                                     1e-3f + cells_per_side * 2.4e-7f, Rl);
            if (Rl < R0) R = Rl / scale;
            st.heavy += 1;
        }
        // drop emptied entries and form prefix offsets (entries strictly non-empty)
        {
            int w = 0;
            total = 0;
            KNN_LOOP_HINT
            for (int i0 = 0; i0 < nlist; i0 += 32) {
                const int i = i0 + lane;
                const uint32_t ra = i < nlist ? S.pa[i] : 0u, rb = i < nlist ? S.pb[i] : 0u;
                const int n_i = (int)(rb - ra);
                __syncwarp();
                const unsigned m = __ballot_sync(0xffffffffu, n_i > 0);
                const int inc = warp_incl_scan(n_i);
                if (n_i > 0) {
                    const int pos = w + __popc(m & ((1u << lane) - 1u));
                    S.pa[pos] = ra;
                    S.pb[pos] = rb;
                    S.off[pos] = (uint32_t)(total + inc - n_i);
                }
                w += __popc(m);
                total += __shfl_sync(0xffffffffu, inc, 31);
            }
            nlist = w;
            if (lane == 0) S.off[nlist] = (uint32_t)total;
            __syncwarp();
        }
        st.cand += total;
        listed = true;
        }
        KNN_TICK(t_c);
        KNN_PHASE(1, t_a, t_c);
        // ---- gather candidates with d^2 <= R^2 -------------------------
        // More than the buffer holds: the rest is binned, and the radius is cut
        // to the bucket that holds the k-th neighbour.  More than kScanLimit
        // particles in the list (before any radius of this query has held
        // fewer than k): no scan, the radius shrinks by the volume ratio.
        int cnt = 0;
        const float R2 = R * R, invR2 = 1.0f / R2;
        const bool too_big = total > kScanLimit && rlo == 0.0f;
        float v_hi = 1.0f;
        if (!too_big) {
            int j0 = 0;
            KNN_LOOP_HINT
            for (int g0 = 0; g0 < total; g0 += 32) {
                const uint32_t t = chunk_slot(S, nlist, total, g0, j0, lane);
                const float dd = g0 + lane < total ? cand_d2(a, h0, l0, t) : FLT_MAX;
                const bool in = dd <= R2;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                const int pos = cnt + __popc(m & ((1u << lane) - 1u));
                if (in && pos < kKnnCap) {
                    S.d[pos] = dd;
                    S.i[pos] = (int32_t)t;
                }
                const int before = cnt;
                cnt += __popc(m);
                // Lazy histogram: the first time the buffer overflows, the
                // buffered candidates are binned; from then on every new
                // in-radius candidate is binned directly, so an overflow
                // usually needs no second scan.
                if (before <= kKnnCap && cnt > kKnnCap) lazy_hist_init<DIM>(S, invR2);
                if (cnt > kKnnCap && in && pos >= kKnnCap) atomicAdd(&S.hist[(int)bucket_of(dd * invR2, DIM)], 1);
            }
            __syncwarp();
            if (cnt > kKnnCap)
                v_hi = overflow_window<DIM>(S, a.hi, a.lo, a.periodic, a.box_hi, a.box_lo, h0, l0, nlist, total, R2,
                                            k, kKnnCap);
        }
        KNN_TICK(t_d);
        KNN_PHASE(2, t_c, t_d);
        // ---- radius updates (bracketed) ------------------------------------
        // Growth is a geometric guess capped by rhi (geometric mean once both
        // are known); an overflow cuts the radius to the histogram bucket
        // holding the k-th neighbour, which holds at least k by construction,
        // and scans the same list again.
        float Rnew = -1.0f;
        int reason = 0;
        if (too_big) {
            Rnew = R * fmaxf(0.25f, powf(0.5f * kKnnCap / (float)total, 1.0f / DIM));
            reason = 2;
            listed = false;
        } else if (cnt < k) {
            rlo = fmaxf(rlo, R);
            const float g = 1.25f * powf((float)k / (float)max(cnt, 1), 1.0f / DIM);
            Rnew = R * fminf(fmaxf(g, 1.25f), 4.0f);
            if (rhi > 0.0f && Rnew >= rhi) Rnew = sqrtf(rlo * rhi);
            reason = 1;
            listed = false;
        } else if (cnt > kKnnCap) {
            rhi = (rhi > 0.0f) ? fminf(rhi, R) : R;
            Rnew = R * (DIM == 3 ? cbrtf(v_hi) : (DIM == 2 ? sqrtf(v_hi) : v_hi)) * 1.00001f;
            if (Rnew >= R) Rnew = R * 0.999f;
            reason = 2;
        }
        // ---- select the k smallest: bucket histogram ------------------------
        float T = 0.0f;
        if (Rnew < 0.0f) {
            T = select_k<DIM>(S, cnt, invR2, k, a.ngb + (int64_t)qi * k);
            // the band around T must lie inside the searched radius
            const float wabs = band_abs(T, query_mag(a.hi, p, a.periodic, a.box_hi));
            if (T * (1.0f + kBandEps) + 2.0f * wabs > R2) {
                Rnew = sqrtf(T * (1.0f + 2.0f * kBandEps) + 4.0f * wabs) * 1.0001f;
                reason = 3;
                listed = false;  // (the selection used the list's memory)
            }
        }
        KNN_TICK(t_e);
        KNN_PHASE(3, t_d, t_e);
        if (!(Rnew > 0.0f)) {
            finish_row(S, cnt, T, k, p, qi, a, fr.side, st);
            st.tries = max(st.tries, tries - 1);
            break;
        }
        st.reason[reason - 1] += 1;
        if (tries >= a.max_tries) {
            if (lane == 0) {
                atomicOr(a.qstatus + qi, MG_Q_UNRESOLVED);
                // diagnostics for the caller: last radius and candidate count
                a.radius[qi] = R;
                a.hsml[qi] = -(float)((too_big ? total : cnt) + 1000000 * reason);
            }
            st.unres += 1;
            break;
        }
        st.retry += 1;
        R = Rnew;
        __syncwarp();
        }
    }
    }

    // statistics: one atomic per warp
    if (lane == 0 && a.stats) {
        if (st.tries) atomicMax((unsigned long long *)&a.stats[0], (unsigned long long)st.tries);
        if (st.cand) atomicAdd((unsigned long long *)&a.stats[1], (unsigned long long)st.cand);
        if (st.retry) atomicAdd((unsigned long long *)&a.stats[2], (unsigned long long)st.retry);
        if (st.band) atomicAdd((unsigned long long *)&a.stats[3], (unsigned long long)st.band);
        if (st.unres) atomicAdd((unsigned long long *)&a.stats[4], (unsigned long long)st.unres);
        if (st.newton) atomicAdd((unsigned long long *)&a.stats[5], (unsigned long long)st.newton);
        for (int r = 0; r < 3; ++r)
            if (st.reason[r]) atomicAdd((unsigned long long *)&a.stats[6 + r], (unsigned long long)st.reason[r]);
        if (st.heavy) atomicAdd((unsigned long long *)&a.stats[9], (unsigned long long)st.heavy);
#ifdef MG_KNN_PROFILE
        for (int r = 0; r < 6; ++r)
            if (r != 4 && st.phase[r]) atomicAdd((unsigned long long *)&a.stats[10 + r], (unsigned long long)st.phase[r]);
        atomicMax((unsigned long long *)&a.stats[14], (unsigned long long)(clock64() - t_warp0));  // slowest warp
#endif
    }
}

// ---- first pass, one thread per query over a warp's candidates -----------------
// The 32 queries of a warp are consecutive (neighbours in Morton order).  The
// warp takes the boxes of each eight queries' first-radius spheres (queries whose
// radius is over kGroupOutlier times the warp's smallest are left to the warp
// path), looks up the cells over them as runs of consecutive slots, and streams
// those particles: 128 are loaded at a time, the ones inside the common box are
// staged in shared memory as offsets from its centre (FP32), and every lane
// tests them against its
// own query and lists those with d~ <= R as one word: d~^2 / R^2 in 20 bits and
// the particle's place in the stream in 12.  Each lane then selects from its
// list: two passes count it in 8 and 8 x 8 buckets of d~^2 and a third takes
// those below the k-th neighbour's bucket and sets its bucket aside, whose
// smallest are taken one by one.
//
// d~ differs from the distance by at most e (a bound from the box size, and half
// a unit of the 20 bits), so the set is the exact k nearest when the k-th d~
// plus e stays inside R (every particle that is not listed is farther than R)
// and the next d~ is more than 2e beyond the k-th.  Every other query (too few
// in radius, a near tie, a crowded bucket, a full list, a box over too many
// particles) goes to the work queue, and the warp path finishes it.  Only the
// rows' slots are written, in stream order; h is solved from them by
// k_hsml_solve_rows with the warp path's FP32 hi/lo distances (cand_d2p).
//
// Nothing is shared between warps: no block barrier, and no buffer whose overflow
// sends a block's queries away.  Staging once for 128 queries, with barriers
// between its rounds, held 12 warps per SM at 40% issue and left 7% of the
// queries to the warp path; here 14 warps issue on ~60% of the cycles.  2^22
// Plummer particles, first pass 7.33 -> 3.3 ms, warp path 1.74 -> 1.0 ms; 2^24
// clump mixture 29.0 -> 14 and 11.6 -> 7 ms.  Bound: instruction issue: testing
// the ~700 particles in the box against each query (a third), streaming ~1700 to
// find them (a quarter), the selection (a fifth).
constexpr int kGroupWarps = 2;      // warps per block (independent of each other)
constexpr int kGroupRuns = 128;     // runs of slots per warp
constexpr int kGroupStream = 4096;  // particles a warp streams at most (12 bits; 13: no faster)
// Listed candidates per query: 16.5 KB per warp, 14 warps per SM.  88 and 104
// entries: 3% and 4% slower on 2^22 Plummer particles (more queries left to the
// warp path; fewer warps); lists cut back to their k nearest when full instead:
// 80 to 88 entries, 7% slower (the check in the inner loop).
constexpr int kGroupList = 96;
constexpr int kGroupBoundary = 8;   // entries of the k-th neighbour's bucket
constexpr int kGroupUnroll = 4;     // chunks of 32 particles loaded together
constexpr int kGroupBoxes = 4;      // boxes per warp, of eight queries each
#ifndef MG_KNN_GROUP_OUTLIER
#define MG_KNN_GROUP_OUTLIER 2.0f
#endif
constexpr float kGroupOutlier = MG_KNN_GROUP_OUTLIER;  // radius above this multiple of the warp's smallest: warp path

struct GroupSmem {  // per warp
    static constexpr int kStage = 32 * kGroupUnroll + 4;
    float sx[kStage], sy[kStage], sz[kStage];  // staged: offsets from the box centre
    uint32_t sg[kStage];                       // and place in the stream
    // entry e of lane t at 32 e + t: one bank per lane, whatever the entries.  The
    // k-th neighbours' buckets take the staging arrays once the stream is done.
    uint32_t list[32 * kGroupList];
    uint32_t pa[kGroupRuns];      // first slot of each run
    uint32_t off[kGroupRuns + 4]; // prefix offsets of the runs in the stream
    int cells[kGroupBoxes][6];    // cells over each box: first x y z, last x y z
};

// First slots of the eight children (level L) of the level L - 1 cell `code`
// where a table holds them: child i starts at p[i << sh], i up to 8.  Without a
// table (a cell of few particles, or no refinement tables): false, and [A, B)
// is the range of the smallest tabled cell around it.
__device__ __forceinline__ bool child_table(const CellIndex &ci, int L, uint64_t code, const uint32_t *&p, int &sh,
                                            uint32_t &A, uint32_t &B) {
    if (L <= ci.Lg) {
        sh = 3 * (ci.Lg - L);
        p = ci.cs + ((code << 3) << sh);
        return true;
    }
    const uint64_t c = code >> (3 * (L - 1 - ci.Lg));
    A = __ldg(ci.cs + c);
    B = __ldg(ci.cs + c + 1);
    int br = ci.brick_of ? __ldg(ci.brick_of + c) : -1;
    int base = ci.Lg;
    while (br >= 0) {
        const uint32_t *st = ci.bricks + (size_t)br * kBrickWords;
        if (L <= base + 3) {
            sh = 3 * (base + 3 - L);
            p = st + ((uint32_t)((code & ((1ull << (3 * (L - 1 - base))) - 1ull)) << 3) << sh);
            return true;
        }
        const uint32_t sub = (uint32_t)((code >> (3 * (L - 1 - base - 3))) & 511ull);
        A = __ldg(st + sub);
        B = __ldg(st + sub + 1);
        br = (int)__ldg(st + kBrickChild + sub);
        base += 3;
    }
    return false;
}

// Offset of a position (hi, lo) from the box centre: its nearest image when
// periodic, the wrap carried error-free (wrap1's form).
template <bool PERIODIC>
__device__ __forceinline__ float group_offset(float h, float l, float c, float box_hi, float box_lo) {
    if (!PERIODIC) return __fadd_rn(__fsub_rn(h, c), l);
    float s, e;
    two_sum(h, -c, s, e);
    if (fabsf(s) > 0.5f * box_hi) {
        const float sg = s > 0.0f ? 1.0f : -1.0f;
        float s2, e2;
        two_sum(s, -sg * box_hi, s2, e2);
        return s2 + ((e2 + e + l) - sg * box_lo);
    }
    return s + (e + l);
}

// The byte (0 to 7) of the packed counts at which their running sum from `below`
// reaches k; below: the sum before it, in: its count.
__device__ __forceinline__ int group_bucket(unsigned long long counts, int k, int &below, int &in) {
    int b = 7;
    bool found = false;
    int run = below, at = below, n = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int c = (int)(counts >> (8 * i)) & 255;
        const bool here = !found && run + c >= k;
        b = here ? i : b;
        at = here ? run : at;
        n = here ? c : n;
        found = found || here;
        run += c;
    }
    below = at;
    in = n;
    return b;
}

template <int DIM, bool PERIODIC>
__global__ __launch_bounds__(32 * kGroupWarps, 7) void k_knn_group(const __grid_constant__ KnnArgs a) {
    extern __shared__ __align__(16) unsigned char group_smem[];
    GroupSmem &S = reinterpret_cast<GroupSmem *>(group_smem)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int64_t qi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool valid = qi < a.nq;
    const Frame fr = load_frame(a.frame);
    const float side = (float)fr.side;
    const float half_side = 0.5f * side;
    const int k = a.k;

    float4 h0 = make_float4(0.f, 0.f, 0.f, 0.f), l0 = h0;
    float R = 0.0f;
    if (valid) {
        const int32_t p = a.queries ? a.queries[qi] : (int32_t)qi;
        h0 = a.hi[p];
        l0 = a.lo[p];
        R = a.seed_h[qi] * a.radius_factor;
        if (!(R > 0.0f) || !isfinite(R)) R = side * 1e-3f;
    }
    // ---- members and their box (hi parts) ----------------------------------------
    const float rmin = warp_min(valid ? R : FLT_MAX);
    const bool mine = valid && R <= kGroupOutlier * rmin;
    float blo[3] = {0.0f, 0.0f, 0.0f}, bhi[3] = {0.0f, 0.0f, 0.0f};
    {
        const float h[3] = {h0.x, h0.y, h0.z};
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            blo[d] = warp_min(mine ? h[d] - R : FLT_MAX);
            bhi[d] = -warp_min(mine ? -(h[d] + R) : FLT_MAX);
        }
    }
    const float rmax = -warp_min(mine ? -R : FLT_MAX);
    // the hi parts differ from the positions by up to 2^-24 |x|
    float xm = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) xm = fmaxf(xm, fmaxf(fabsf(blo[d]), fabsf(bhi[d])));
    if (PERIODIC) xm = fmaxf(xm, a.box_hi);
    const float mg = 1e-5f * rmax + 4e-7f * xm + 1e-30f;
    float ctr[3] = {0.0f, 0.0f, 0.0f}, ext = 0.0f, ehalf = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        blo[d] -= mg;
        bhi[d] += mg;
        ctr[d] = 0.5f * (blo[d] + bhi[d]);
        ext = fmaxf(ext, bhi[d] - blo[d]);
        ehalf = fmaxf(ehalf, fmaxf(fabsf(blo[d] - ctr[d]), fabsf(bhi[d] - ctr[d])));
    }
    // offsets from the centre carry at most ~2^-23 ehalf of rounding per axis,
    // and the hi/lo split of each position ~2^-48 |x| of representation error
    // (2^-46 |x| per axis for a difference, with the low parts' rounding):
    // bound on |d~ - d| for d <= R (twice the analysis)
    const float eg = 1e-6f * ehalf + 3e-7f * rmax + 3e-14f * xm;
    float qx = 0.0f, qy = 0.0f, qz = 0.0f;
    qx = __fadd_rn(__fsub_rn(h0.x, ctr[0]), l0.x);
    if (DIM > 1) qy = __fadd_rn(__fsub_rn(h0.y, ctr[1]), l0.y);
    if (DIM > 2) qz = __fadd_rn(__fsub_rn(h0.z, ctr[2]), l0.z);
    // box of the member spheres, and those of each eight queries (lanes 8 b ..
    // 8 b + 7), in offsets
    float qlo[3], qhi[3];  // of all
    float elo[3], ehi[3];  // of this lane's eight
    {
        const float rr = R * (1.0f + 1e-6f) + eg;
        const float qv[3] = {qx, qy, qz};
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            elo[d] = mine ? qv[d] - rr : FLT_MAX;
            ehi[d] = mine ? qv[d] + rr : -FLT_MAX;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                elo[d] = fminf(elo[d], __shfl_xor_sync(0xffffffffu, elo[d], o));
                ehi[d] = fmaxf(ehi[d], __shfl_xor_sync(0xffffffffu, ehi[d], o));
            }
            qlo[d] = elo[d];
            qhi[d] = ehi[d];
#pragma unroll
            for (int o = 8; o < 32; o <<= 1) {
                qlo[d] = fminf(qlo[d], __shfl_xor_sync(0xffffffffu, qlo[d], o));
                qhi[d] = fmaxf(qhi[d], __shfl_xor_sync(0xffffffffu, qhi[d], o));
            }
        }
    }
    // ---- cells over the box: finest level with at most 8 per axis -----------------
    int L = (int)floorf(log2f(side / ext)) + 3;
    L = max(1, min(kMaxLevel, L));
    int cmin[3] = {0, 0, 0}, cmax[3] = {0, 0, 0};
    bool ok = rmin < FLT_MAX;
    for (;;) {
        const float cps = (float)(1u << L), scale = cps / side;
        const float em = 1e-3f + cps * 2.4e-7f;
        bool fits = true;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            cmin[d] = (int)floorf((blo[d] + half_side) * scale - em);
            cmax[d] = (int)floorf((bhi[d] + half_side) * scale + em);
            if (!PERIODIC) {
                cmin[d] = max(0, cmin[d]);
                cmax[d] = min((int)cps - 1, cmax[d]);
            }
            fits = fits && cmax[d] - cmin[d] < 8;
        }
        if (fits) break;
        if (L == 1) {
            ok = false;
            break;
        }
        --L;
    }
    if ((lane & 7) == 0) {  // (an empty box: no cell)
        const float cps = (float)(1u << L), scale = cps / side;
        const float em = 1e-3f + cps * 2.4e-7f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const bool some = d < DIM && elo[d < DIM ? d : 0] <= ehi[d < DIM ? d : 0];
            const float c0 = d < DIM ? (elo[d] + ctr[d] - mg + half_side) * scale - em : 0.0f;
            const float c1 = d < DIM ? (ehi[d] + ctr[d] + mg + half_side) * scale + em : 0.0f;
            S.cells[lane >> 3][d] = some ? max(cmin[d], (int)floorf(c0)) : (d < DIM ? INT_MAX : 0);
            S.cells[lane >> 3][3 + d] = some ? min(cmax[d], (int)floorf(c1)) : (d < DIM ? INT_MIN : 0);
        }
    }
    __syncwarp();
    // a box of nearly the period's size: images would be ambiguous, cells repeat
    if (PERIODIC) ok = ok && ext < 0.4f * a.box_hi && L >= 4;
    // ---- runs of consecutive slots under those cells --------------------------------
    int nrun = 0, tot = 0;
    if (ok) {
        int pmin[3], pn[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            pmin[d] = cmin[d] >> 1;
            pn[d] = (cmax[d] >> 1) - pmin[d] + 1;  // <= 5
        }
        const int npar = pn[0] * pn[1] * pn[2];
        const float inv_nx = 1.0f / (float)pn[0], inv_nxy = 1.0f / (float)(pn[0] * pn[1]);
        const int wrap = (1 << (L - 1)) - 1;
        KNN_LOOP_HINT
        for (int c0 = 0; c0 < npar; c0 += 32) {
            const int c = c0 + lane;
            const uint32_t *tp = nullptr;
            int sh = 0;
            unsigned m = 0;
            uint32_t A = 0, B = 0;
            if (c < npar) {
                int ix, iy, iz;
                box_index(c, inv_nx, inv_nxy, pn, ix, iy, iz);
                const int X = pmin[0] + ix, Y = pmin[1] + iy, Z = pmin[2] + iz;
                // children inside some box's cells
#pragma unroll
                for (int b = 0; b < kGroupBoxes; ++b) {
                    const int *c = S.cells[b];
                    const int x = 2 * X, y = 2 * Y, z = 2 * Z;
                    unsigned mb = (x >= c[0] && x <= c[3] ? 0x55u : 0u) | (x + 1 >= c[0] && x < c[3] ? 0xaau : 0u);
                    mb &= (y >= c[1] && y <= c[4] ? 0x33u : 0u) | (y + 1 >= c[1] && y < c[4] ? 0xccu : 0u);
                    mb &= (z >= c[2] && z <= c[5] ? 0x0fu : 0u) | (z + 1 >= c[2] && z < c[5] ? 0xf0u : 0u);
                    m |= mb;
                }
                const uint64_t code = morton3((uint32_t)(X & wrap), (uint32_t)(Y & wrap), (uint32_t)(Z & wrap));
                if (m && !child_table(a.ci, L, code, tp, sh, A, B)) {
                    const int ks = 3 * (kKeyBits - L + 1);
                    A = lower_bound_prefix(a.keys, A, B, code, ks);
                    B = lower_bound_prefix(a.keys, A, B, code + 1, ks);
                    tp = nullptr;
                    m = 1u;
                }
            }
            while (__any_sync(0xffffffffu, m != 0u)) {
                uint32_t ra = 0, rb = 0;
                if (m) {
                    const int i = __ffs(m) - 1, n = __ffs(~(m >> i)) - 1;  // children i .. i + n - 1
                    ra = tp ? __ldg(tp + ((size_t)i << sh)) : A;
                    rb = tp ? __ldg(tp + ((size_t)(i + n) << sh)) : B;
                    m &= ~(((1u << n) - 1u) << i);
                }
                const int len = (int)(rb - ra);
                const unsigned some = __ballot_sync(0xffffffffu, len > 0);
                const int pos = nrun + __popc(some & ((1u << lane) - 1u));
                const int inc = warp_incl_scan(len);
                if (len > 0 && pos < kGroupRuns) {
                    S.pa[pos] = ra;
                    S.off[pos] = (uint32_t)(tot + inc - len);
                }
                nrun += __popc(some);
                tot += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        ok = nrun <= kGroupRuns && tot <= kGroupStream && tot >= 0;
        if (ok && lane == 0) S.off[nrun] = (uint32_t)tot;
        __syncwarp();
    }

    // ---- stream: load, stage what lies in the box, list ------------------------------
    // reason: 0 accepted, 1 too few in radius, 3 k-th too close to R, 4 other
    const bool act = ok && mine;
    const float R2 = R * R;
    int cnt = 0;
    bool full = false;
    if (ok) {
        // key of d~^2: its 20-bit fraction of R^2, read off the low mantissa bits
        // of d~^2 s + 2^23
        const float ks = 1048575.0f / R2;
        float R2a = act ? R2 : -1.0f;
        uint32_t *lp = S.list + lane;  // end of this lane's list
        const uint32_t *const lp_full = lp + 32 * (kGroupList - 4);
        const unsigned long long QX = f2_pack(qx), QY = f2_pack(qy), QZ = f2_pack(qz), KS = f2_pack(ks),
                                 MAGIC = f2_pack(8388608.0f);
        float4 hb[kGroupUnroll], lb[kGroupUnroll];
        int j0 = 0;
        auto fetch = [&](int g0) {
            uint32_t slot[kGroupUnroll];
#pragma unroll
            for (int u = 0; u < kGroupUnroll; ++u) {
                const int g = g0 + 32 * u;
                slot[u] = g < tot ? chunk_slot(S, nrun, tot, g, j0, lane) : 0u;
            }
#pragma unroll
            for (int u = 0; u < kGroupUnroll; ++u) {
                if (g0 + 32 * u + lane < tot) {
                    hb[u] = __ldg(a.hi + slot[u]);
                    lb[u] = __ldg(a.lo + slot[u]);
                }
            }
        };
        fetch(0);
        KNN_LOOP_HINT
        for (int g0 = 0; g0 < tot; g0 += 32 * kGroupUnroll) {
            int n = 0;
#pragma unroll
            for (int u = 0; u < kGroupUnroll; ++u) {
                const int g = g0 + 32 * u + lane;
                const float ox = group_offset<PERIODIC>(hb[u].x, lb[u].x, ctr[0], a.box_hi, a.box_lo);
                const float oy = DIM > 1 ? group_offset<PERIODIC>(hb[u].y, lb[u].y, ctr[1], a.box_hi, a.box_lo) : 0.0f;
                const float oz = DIM > 2 ? group_offset<PERIODIC>(hb[u].z, lb[u].z, ctr[2], a.box_hi, a.box_lo) : 0.0f;
                bool in = ox >= qlo[0] && ox <= qhi[0];
                if (DIM > 1) in = in && oy >= qlo[1] && oy <= qhi[1];
                if (DIM > 2) in = in && oz >= qlo[2] && oz <= qhi[2];
                in = in && g < tot;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                if (in) {
                    const int pos = n + __popc(m & ((1u << lane) - 1u));
                    S.sx[pos] = ox;
                    if (DIM > 1) S.sy[pos] = oy;
                    if (DIM > 2) S.sz[pos] = oz;
                    S.sg[pos] = (uint32_t)g;
                }
                n += __popc(m);
            }
            if (lane < 4) S.sx[n + lane] = 1e18f;  // pads the last four
            if (g0 + 32 * kGroupUnroll < tot) fetch(g0 + 32 * kGroupUnroll);
            __syncwarp();
            KNN_LOOP_HINT
            for (int w = 0; w < n; w += 4) {
                const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(S.sx + w);
                ulonglong2 Y, Z;
                if (DIM > 1) Y = *reinterpret_cast<const ulonglong2 *>(S.sy + w);
                if (DIM > 2) Z = *reinterpret_cast<const ulonglong2 *>(S.sz + w);
                const uint4 G = *reinterpret_cast<const uint4 *>(S.sg + w);
                R2a = lp > lp_full ? -1.0f : R2a;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned long long dx = f2_sub(h ? X.y : X.x, QX);
                    unsigned long long d2 = f2_mul(dx, dx);
                    if (DIM > 1) {
                        const unsigned long long dy = f2_sub(h ? Y.y : Y.x, QY);
                        d2 = f2_fma(dy, dy, d2);
                    }
                    if (DIM > 2) {
                        const unsigned long long dz = f2_sub(h ? Z.y : Z.x, QZ);
                        d2 = f2_fma(dz, dz, d2);
                    }
                    const unsigned long long t = f2_fma(d2, KS, MAGIC);
                    const uint32_t k0 = (uint32_t)t * 4096u + (h ? G.z : G.x);
                    const uint32_t k1 = (uint32_t)(t >> 32) * 4096u + (h ? G.w : G.y);
                    if (f2_low(d2) <= R2a) {
                        *lp = k0;
                        lp += 32;
                    }
                    if (f2_high(d2) <= R2a) {
                        *lp = k1;
                        lp += 32;
                    }
                }
            }
            __syncwarp();
        }
        cnt = (int)(lp - (S.list + lane)) >> 5;
        full = lp > lp_full;
    }
    // ---- per-lane selection ------------------------------------------------------------
    int reason = 4;
    float T = 0.0f;
    if (act && !full) {
        if (cnt < k) {
            reason = 1;
        } else {
            unsigned long long c8 = 0ull;
#pragma unroll 4
            for (int e = 0; e < cnt; ++e) c8 += 1ull << ((S.list[32 * e + lane] >> 29) << 3);
            int below = 0, in = 0;
            const uint32_t b1 = (uint32_t)group_bucket(c8, k, below, in);
            c8 = 0ull;
#pragma unroll 4
            for (int e = 0; e < cnt; ++e) {
                const uint32_t v = S.list[32 * e + lane];
                c8 += (v >> 29) == b1 ? 1ull << ((v >> 23) & 56u) : 0ull;
            }
            const uint32_t bstar = 8u * b1 + (uint32_t)group_bucket(c8, k, below, in);  // of 64
            if (in <= kGroupBoundary) {
                static_assert(32 * kGroupBoundary <= 2 * GroupSmem::kStage, "fits sx and sy");
                uint32_t *bnd = reinterpret_cast<uint32_t *>(S.sx);
                const int r = k - below;
                int ns = 0, nb = 0;
                uint32_t next = 0xffffffffu;  // smallest beyond the bucket
#pragma unroll 4
                for (int e = 0; e < cnt; ++e) {
                    const uint32_t v = S.list[32 * e + lane], b = v >> 26;
                    if (b < bstar) {
                        S.list[32 * ns + lane] = v;  // ns <= e
                        ++ns;
                    } else if (b == bstar) {
                        bnd[32 * nb + lane] = v;
                        ++nb;
                    } else {
                        next = min(next, v);
                    }
                }
                // the r smallest of the bucket (the words differ: each has its place
                // in the stream), then the one after them
                uint32_t last = 0u;
                bool any = false;
                KNN_LOOP_HINT
                for (int i = 0; i <= r; ++i) {
                    uint32_t best = i == r ? next : 0xffffffffu;
                    KNN_LOOP_HINT
                    for (int e = 0; e < nb; ++e) {
                        const uint32_t v = bnd[32 * e + lane];
                        if (!any || v > last) best = min(best, v);
                    }
                    if (i < r) {
                        S.list[32 * (below + i) + lane] = best;
                        last = best;
                        any = true;
                    } else {
                        next = best;
                    }
                }
                // exact set: the k-th stays inside R by more than the error bound,
                // and the next candidate is more than twice the bound beyond it
                const float unit = R2 * (1.0f / 1048575.0f);
                T = ((float)(last >> 12) + 0.5f) * unit;
                const float N = next == 0xffffffffu ? R2 : ((float)(next >> 12) - 0.5f) * unit;
                const float e2 = 1.01f * eg + 2e-7f * R;
                const float dT = sqrtf(T) * 1.000001f, dN = sqrtf(fmaxf(N, 0.0f)) * 0.999999f;
                if (dT + 2.0f * e2 > R)
                    reason = 3;
                else if (dN - dT > 2.0f * e2)
                    reason = 0;
            }
        }
    }
    // ---- rows of the accepted queries: places in the stream to slots ---------------------
    if (act && reason == 0) {
        int32_t *row = a.ngb + qi * k;
        auto slot_at = [&](int e) -> int32_t {
            const uint32_t g = S.list[32 * e + lane] & 4095u;
            int j = 0;
#pragma unroll
            for (int st = kGroupRuns / 2; st > 0; st >>= 1)
                if (j + st < nrun && S.off[j + st] <= g) j += st;
            return (int32_t)(S.pa[j] + (g - S.off[j]));
        };
        if ((k & 3) == 0 && ((uintptr_t)a.ngb & 15) == 0) {
            KNN_LOOP_HINT
            for (int e = 0; e < k; e += 4)
                *reinterpret_cast<int4 *>(row + e) = make_int4(slot_at(e), slot_at(e + 1), slot_at(e + 2), slot_at(e + 3));
        } else {
            KNN_LOOP_HINT
            for (int e = 0; e < k; ++e) row[e] = slot_at(e);
        }
    }
    // ---- everything else goes to the warp path -----------------------------------
    const bool push = valid && !(act && reason == 0);
    if (push) {
        float Rnew = R;
        if (reason == 1) {
            const float g = 1.25f * powf((float)k / (float)max(cnt, 1), 1.0f / DIM);
            Rnew = R * fminf(fmaxf(g, 1.25f), 4.0f);
        } else if (reason == 3) {
            Rnew = fmaxf(R, sqrtf(T) + 4.0f * (1.01f * eg + 2e-7f * R)) * 1.0001f;
        }
        a.radius[qi] = Rnew;
    }
    const unsigned pm = __ballot_sync(0xffffffffu, push);
    if (pm) {
        int base = 0;
        if (lane == 0) base = atomicAdd(a.qout_count, __popc(pm));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (push) a.qout[base + __popc(pm & ((1u << lane) - 1u))] = (int32_t)qi;
    }
    // statistics: streamed candidates per member query, retries and their reasons
    if (a.stats) {
        const int na = __popc(__ballot_sync(0xffffffffu, act));
        const int n1 = __popc(__ballot_sync(0xffffffffu, reason == 1));
        const int n3 = __popc(__ballot_sync(0xffffffffu, reason == 3));
#ifdef MG_KNN_GROUP_DEBUG
        // [10] warps not streamed, [11] runs, [12] streamed, [13] outliers, [14]
        // listed, [15] full lists
        const int ol = __popc(__ballot_sync(0xffffffffu, valid && !mine));
        const int fl = __popc(__ballot_sync(0xffffffffu, full));
        const int lc = warp_sum(cnt);
        if (lane == 0) {
            unsigned long long *st = (unsigned long long *)a.stats;
            atomicAdd(st + 10, ok ? 0ull : 1ull);
            atomicAdd(st + 11, (unsigned long long)nrun);
            atomicAdd(st + 12, (unsigned long long)tot);
            atomicAdd(st + 13, (unsigned long long)ol);
            atomicAdd(st + 14, (unsigned long long)lc);
            atomicAdd(st + 15, (unsigned long long)fl);
        }
#endif
        if (lane == 0) {
            if (na) atomicAdd((unsigned long long *)&a.stats[1], (unsigned long long)na * (unsigned long long)tot);
            if (pm) atomicAdd((unsigned long long *)&a.stats[2], (unsigned long long)__popc(pm));
            if (n1) atomicAdd((unsigned long long *)&a.stats[6], (unsigned long long)n1);
            if (n3) atomicAdd((unsigned long long *)&a.stats[8], (unsigned long long)n3);
        }
    }
}

// ---- first pass over a query list, one thread per query over a block's candidates ---
// Slice and Reconstruct return FP64 values built on the FP32 derivatives of a
// query list, in which the order of a row shows at ~1e-8; query lists keep the
// search that has produced their rows so far (see the passes above), and with
// it every bit of those results.
// The G queries of a block are consecutive (neighbours in Morton order).  The
// block looks up the cells over the bounding box of its queries' first-radius
// spheres and stages, once, every particle inside the box of some warp's
// spheres into shared memory as its offset from the block centre (FP32, with
// the slot).  Each thread then serves its own query from the staged set:
//   A: offsets compared against R (staged words outside the warp's box are
//      skipped) -> per-thread list of the candidates with d~ <= R;
//   B: 32-bucket histogram of the list in (d~/R)^dim;
//   C: buckets below the k-th neighbour's are taken whole, its bucket is
//      ordered by (d~^2, slot).
// d~ differs from the distance by at most e (a bound from the box size), so the
// set is the exact k nearest when the k-th d~ plus e stays inside R (every
// particle outside the staged boxes is farther than R) and the next d~ is more
// than 2e beyond the k-th (no other particle can change places with it).
// Every other query (too few in radius, a near tie, a crowded boundary
// bucket, a block whose staging overflows, a radius far above the block's
// smallest) goes to the work queue, and the passes finish it.  Only the
// rows' slots are written (the order inside a row is the staging order); h is
// solved from them by k_hsml_solve_rows with the warp path's FP32 hi/lo
// distances (cand_d2p).
constexpr int kBlockBins = 32;
constexpr int kBlockBoundary = 8;  // entries of the k-th neighbour's bucket kept per query
constexpr int kBlockUnroll = 4;    // particles per thread per staging round
constexpr int kBlockThreads = 128; // queries per block
constexpr int kBlockStage = 2048;  // staged candidates per block

template <int G, int C>
struct BlockSmem {
    static constexpr int kWarps = G / 32;
    static constexpr int kWords = C / 32;
    static constexpr int kCells = 512;  // local Morton space of an 8 x 8 x 8 cell box
    float sx[C], sy[C], sz[C];          // staged: offsets from the block centre
    uint32_t ss[C];                     // and slots
    float wbox[kWords][6];              // per staged word of 32: min x y z, max x y z
    float qbox[kWarps][6];              // per warp: box of its member queries' spheres
    uint16_t list[kGroupList * G];      // entry e of thread t at list_at(e, t); the
                                        // selected neighbours end up in the first k
    uint16_t bnd[kBlockBoundary * G];   // boundary-bucket staged indices
    float bnd_d[kBlockBoundary * G];    // and their d~^2
    uint8_t hist[kBlockBins * G];       // per-thread bucket counts
    uint32_t cell_a[kCells];            // first slot of each box cell
    uint32_t cell_off[kCells + 1];      // prefix offsets of the cells' particles
    float red[8][kWarps];               // block reductions
    int wtot[2][kWarps];
};

// Entry e of thread t in the per-thread lists (u16): a row of G entries per e,
// the two halves of each 32-bit word held by lanes of different warps, so
// that the 32 lanes of a warp always hit 32 different banks.
__device__ __forceinline__ int list_at(int e, int t) {
    return e * (int)blockDim.x + ((t >> 6) << 6) + ((t & 31) << 1) + ((t >> 5) & 1);
}

// Byte of thread t's counter of bucket b in the per-thread histograms of a
// block of G threads: the four counters b = 4 i .. 4 i + 3 of a thread share
// one 32-bit word, and word i of thread t sits at i * G + t, so that the 32
// lanes of a warp always address 32 different banks whatever their buckets.
template <int G>
__device__ __forceinline__ int hist_at(int b, int t) { return (((b >> 2) * G + t) << 2) + (b & 3); }

// d~^2 between offsets (one expression for every pass; the packed form below
// rounds each half the same way)
template <int DIM>
__device__ __forceinline__ float group_d2(float cx, float cy, float cz, float qx, float qy, float qz) {
    const float dx = __fsub_rn(cx, qx);
    float d2 = __fmul_rn(dx, dx);
    if (DIM > 1) {
        const float dy = __fsub_rn(cy, qy);
        d2 = __fmaf_rn(dy, dy, d2);
    }
    if (DIM > 2) {
        const float dz = __fsub_rn(cz, qz);
        d2 = __fmaf_rn(dz, dz, d2);
    }
    return d2;
}

template <int DIM, int G, int C>
__global__ __launch_bounds__(G) void k_knn_group_block(const __grid_constant__ KnnPassArgs a) {
    extern __shared__ __align__(16) unsigned char group_smem[];
    using SM = BlockSmem<G, C>;
    static_assert(G % 64 == 0 && SM::kCells % G == 0, "list_at and the cell split need G = 64 m, G | 512");
    constexpr int NW = SM::kWarps;
    SM &S = *reinterpret_cast<SM *>(group_smem);
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const int64_t qi = (int64_t)blockIdx.x * G + tid;
    const bool valid = qi < a.nq;
    const Frame fr = load_frame(a.frame);
    const float side = (float)fr.side;
    const float half_side = 0.5f * side;
    const int k = a.k;

    int32_t p = 0;
    float4 h0 = make_float4(0.f, 0.f, 0.f, 0.f), l0 = h0;
    float R = 0.0f;
    if (valid) {
        p = a.queries ? a.queries[qi] : (int32_t)qi;
        h0 = a.hi[p];
        l0 = a.lo[p];
        R = a.seed_h[qi] * a.radius_factor;
        if (!(R > 0.0f) || !isfinite(R)) R = side * 1e-3f;
    }
    // ---- members and the block's box (hi parts) --------------------------------
    float v = warp_min(valid ? R : FLT_MAX);
    if (lane == 0) S.red[0][wib] = v;
    __syncthreads();
    float rmin = S.red[0][0];
#pragma unroll
    for (int w = 1; w < NW; ++w) rmin = fminf(rmin, S.red[0][w]);
    const bool mine = valid && R <= kGroupOutlier * rmin;
    float bb[7];
    bb[0] = mine ? h0.x - R : FLT_MAX;
    bb[1] = mine ? h0.y - R : FLT_MAX;
    bb[2] = mine ? h0.z - R : FLT_MAX;
    bb[3] = mine ? -(h0.x + R) : FLT_MAX;
    bb[4] = mine ? -(h0.y + R) : FLT_MAX;
    bb[5] = mine ? -(h0.z + R) : FLT_MAX;
    bb[6] = mine ? -R : FLT_MAX;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        bb[i] = warp_min(bb[i]);
        if (lane == 0) S.red[1 + i][wib] = bb[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        float r = S.red[1 + i][0];
#pragma unroll
        for (int w = 1; w < NW; ++w) r = fminf(r, S.red[1 + i][w]);
        bb[i] = r;
    }
    const float rmax = -bb[6];
    // the hi parts differ from the positions by up to 2^-24 |x|
    float blo[3] = {bb[0], bb[1], bb[2]}, bhi[3] = {-bb[3], -bb[4], -bb[5]};
    float xm = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) xm = fmaxf(xm, fmaxf(fabsf(blo[d]), fabsf(bhi[d])));
    const float mg = 1e-5f * rmax + 4e-7f * xm + 1e-30f;
    float ctr[3] = {0.0f, 0.0f, 0.0f}, ext = 0.0f, ehalf = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        blo[d] -= mg;
        bhi[d] += mg;
        ctr[d] = 0.5f * (blo[d] + bhi[d]);
        ext = fmaxf(ext, bhi[d] - blo[d]);
        ehalf = fmaxf(ehalf, fmaxf(fabsf(blo[d] - ctr[d]), fabsf(bhi[d] - ctr[d])));
    }
    // offsets from the centre carry at most ~2^-23 ehalf of rounding per axis,
    // and the hi/lo split of each position ~2^-48 |x| of representation error
    // (2^-46 |x| per axis for a difference, with the low parts' rounding):
    // bound on |d~ - d| for d <= R (twice the analysis)
    const float eg = 1e-6f * ehalf + 3e-7f * rmax + 3e-14f * xm;
    float qx = 0.0f, qy = 0.0f, qz = 0.0f;
    if (DIM > 0) qx = __fadd_rn(__fsub_rn(h0.x, ctr[0]), l0.x);
    if (DIM > 1) qy = __fadd_rn(__fsub_rn(h0.y, ctr[1]), l0.y);
    if (DIM > 2) qz = __fadd_rn(__fsub_rn(h0.z, ctr[2]), l0.z);
    // per-warp box of the member spheres, in offsets
    {
        const float rr = R * (1.0f + 1e-6f) + eg;
        float wb[6];
        wb[0] = mine ? qx - rr : FLT_MAX;
        wb[1] = mine ? qy - rr : FLT_MAX;
        wb[2] = mine ? qz - rr : FLT_MAX;
        wb[3] = mine ? -(qx + rr) : FLT_MAX;
        wb[4] = mine ? -(qy + rr) : FLT_MAX;
        wb[5] = mine ? -(qz + rr) : FLT_MAX;
#pragma unroll
        for (int i = 0; i < 6; ++i) wb[i] = warp_min(wb[i]);
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < 6; ++i) S.qbox[wib][i] = i < 3 ? wb[i] : -wb[i];
        }
    }

    // ---- box cells: finest level with at most 8 cells per axis over the box ------
    // enumerated in local Morton order, so that consecutive staged particles
    // (a word of 32) are spatially compact and whole words can be skipped
    int L = (int)floorf(log2f(side / ext)) + 3;
    L = max(0, min(kMaxLevel, L));
    int cmin[3], cnum[3];
    for (;;) {
        const float cps = (float)(1u << L), scale = cps / side;
        const float em = 1e-3f + cps * 2.4e-7f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (d >= DIM) {
                cmin[d] = 0;
                cnum[d] = 1;
                continue;
            }
            const int c0 = max(0, (int)floorf((blo[d] + half_side) * scale - em));
            const int c1 = min((int)cps - 1, (int)floorf((bhi[d] + half_side) * scale + em));
            cmin[d] = c0;
            cnum[d] = max(0, c1 - c0 + 1);
        }
        if ((cnum[0] <= 8 && cnum[1] <= 8 && cnum[2] <= 8) || L == 0) break;
        --L;
    }
    constexpr int ncell = SM::kCells;
    constexpr int CPT = ncell / G;  // cells per thread
    const bool geom_ok = rmin < FLT_MAX && cnum[0] <= 8 && cnum[1] <= 8 && cnum[2] <= 8;
    const float cside = side / (float)(1u << L);
    // cell boxes are compared with the warps' boxes with this slack (FP32 cell
    // corners, key quantisation, offset rounding)
    const float cmarg = 2e-6f * side + 1e-3f * cside;
    __syncthreads();  // the warps' boxes
    // reason: 0 accepted, 1 too few in radius, 3 k-th too close to R, 4 other
    int reason = 4;
    int cnt = 0;
    float T = 0.0f;
    bool served = false;
    int my_nst = 0;
    const float R2 = R * R;
    // Warps still to serve, served gsz at a time from the lowest: a block
    // whose staging overflows is staged again as two halves (re-staging smaller
    // groups costs more than the warp passes take for their queries).
    unsigned todo = (1u << NW) - 1u;
    int gsz = NW;
    while (todo) {
    const unsigned wsel = (((1u << gsz) - 1u) << (__ffs(todo) - 1)) & todo;
    // ---- cells of the box that meet a selected warp's box: ranges, offsets ------
    bool block_ok = geom_ok;
    int tot = 0;
    if (block_ok) {
        uint32_t cnt4[CPT];
        int mine4 = 0;
#pragma unroll
        for (int e = 0; e < CPT; ++e) {
            const int c = CPT * tid + e;
            // local Morton index -> (ix, iy, iz), 3 bits each
            const int ix = (c & 1) | ((c >> 2) & 2) | ((c >> 4) & 4);
            const int iy = ((c >> 1) & 1) | ((c >> 3) & 2) | ((c >> 5) & 4);
            const int iz = ((c >> 2) & 1) | ((c >> 4) & 2) | ((c >> 6) & 4);
            cnt4[e] = 0u;
            S.cell_a[c] = 0u;
            bool use = ix < cnum[0] && iy < cnum[1] && iz < cnum[2];
            if (use) {
                const int ii[3] = {ix, iy, iz};
                float clo[3], chi[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    clo[d] = (float)(cmin[d] + ii[d]) * cside - half_side - ctr[d] - cmarg;
                    chi[d] = clo[d] + cside + 2.0f * cmarg;
                }
                bool any = false;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    if (!(wsel >> w & 1u)) continue;
                    bool ov = clo[0] <= S.qbox[w][3] && chi[0] >= S.qbox[w][0];
                    if (DIM > 1) ov = ov && clo[1] <= S.qbox[w][4] && chi[1] >= S.qbox[w][1];
                    if (DIM > 2) ov = ov && clo[2] <= S.qbox[w][5] && chi[2] >= S.qbox[w][2];
                    any = any || ov;
                }
                use = any;
            }
            if (use) {
                uint32_t ca, cb;
                cell_range(a.ci, L, (uint32_t)(cmin[0] + ix), (uint32_t)(cmin[1] + iy), (uint32_t)(cmin[2] + iz), ca,
                           cb);
                S.cell_a[c] = ca;
                cnt4[e] = cb - ca;
            }
            mine4 += (int)cnt4[e];
        }
        const int inc = warp_incl_scan(mine4);
        if (lane == 31) S.wtot[0][wib] = inc;
        __syncthreads();
        int woff = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const int t = S.wtot[0][w];
            if (w < wib) woff += t;
            tot += t;
        }
        int ex = woff + inc - mine4;
#pragma unroll
        for (int e = 0; e < CPT; ++e) {
            S.cell_off[CPT * tid + e] = (uint32_t)ex;
            ex += (int)cnt4[e];
        }
        if (tid == 0) S.cell_off[ncell] = (uint32_t)tot;
        __syncthreads();
        block_ok = tot <= 32 * C;
    }
    // far more particles than the buffer holds: straight to the halves
    if (geom_ok && 2 * gsz > NW && NW > 1 && tot > 3 * C) {
        gsz >>= 1;
        continue;
    }
    // ---- stage the particles inside some warp's box (deterministic order) -------
    int nst = 0;
    if (block_ok) {
        float qb[NW][6];
#pragma unroll
        for (int w = 0; w < NW; ++w)
#pragma unroll
            for (int i = 0; i < 6; ++i) qb[w][i] = (wsel >> w & 1u) ? S.qbox[w][i] : (i < 3 ? FLT_MAX : -FLT_MAX);
        // rounds of G * kBlockUnroll particles; the slots and loads of the next
        // round are issued before this round's compaction and barrier
        auto fetch = [&](int base, uint32_t(&sl)[kBlockUnroll], float4(&hv)[kBlockUnroll],
                         float4(&lv)[kBlockUnroll]) {
            const int g0 = base + tid * kBlockUnroll;
            int c = 0;
            if (g0 < tot) {
                int hi_c = ncell;
                while (hi_c - c > 1) {
                    const int mid = (c + hi_c) >> 1;
                    if ((int)S.cell_off[mid] <= g0)
                        c = mid;
                    else
                        hi_c = mid;
                }
            }
#pragma unroll
            for (int u = 0; u < kBlockUnroll; ++u) {
                const int g = g0 + u;
                sl[u] = 0xffffffffu;
                if (g < tot) {
                    while ((int)S.cell_off[c + 1] <= g) ++c;
                    sl[u] = S.cell_a[c] + (uint32_t)(g - (int)S.cell_off[c]);
                }
            }
#pragma unroll
            for (int u = 0; u < kBlockUnroll; ++u) {
                if (sl[u] != 0xffffffffu) {
                    hv[u] = a.hi[sl[u]];
                    lv[u] = a.lo[sl[u]];
                } else {
                    hv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    lv[u] = hv[u];
                }
            }
        };
        uint32_t slot[kBlockUnroll];
        float4 hb[kBlockUnroll], lb[kBlockUnroll];
        if (tot > 0) fetch(0, slot, hb, lb);
        int round = 0;
        for (int base = 0; base < tot; base += G * kBlockUnroll, ++round) {
            uint32_t slot_n[kBlockUnroll];
            float4 hb_n[kBlockUnroll], lb_n[kBlockUnroll];
            if (base + G * kBlockUnroll < tot) fetch(base + G * kBlockUnroll, slot_n, hb_n, lb_n);
            float ox_[kBlockUnroll], oy_[kBlockUnroll], oz_[kBlockUnroll];
            int nkeep = 0;
            unsigned keepm = 0;
#pragma unroll
            for (int u = 0; u < kBlockUnroll; ++u) {
                float ox = 0.0f, oy = 0.0f, oz = 0.0f;
                if (DIM > 0) ox = __fadd_rn(__fsub_rn(hb[u].x, ctr[0]), lb[u].x);
                if (DIM > 1) oy = __fadd_rn(__fsub_rn(hb[u].y, ctr[1]), lb[u].y);
                if (DIM > 2) oz = __fadd_rn(__fsub_rn(hb[u].z, ctr[2]), lb[u].z);
                ox_[u] = ox;
                oy_[u] = oy;
                oz_[u] = oz;
                bool keep = false;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    bool in = ox >= qb[w][0] && ox <= qb[w][3];
                    if (DIM > 1) in = in && oy >= qb[w][1] && oy <= qb[w][4];
                    if (DIM > 2) in = in && oz >= qb[w][2] && oz <= qb[w][5];
                    keep = keep || in;
                }
                keep = keep && slot[u] != 0xffffffffu;
                keepm |= keep ? 1u << u : 0u;
                nkeep += keep ? 1 : 0;
            }
            const int inc = warp_incl_scan(nkeep);
            if (lane == 31) S.wtot[round & 1][wib] = inc;
            __syncthreads();
            int woff = 0, btot = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const int t = S.wtot[round & 1][w];
                if (w < wib) woff += t;
                btot += t;
            }
            int pos = nst + woff + inc - nkeep;
#pragma unroll
            for (int u = 0; u < kBlockUnroll; ++u) {
                if (keepm >> u & 1u) {
                    if (pos < C) {
                        S.sx[pos] = ox_[u];
                        S.sy[pos] = oy_[u];
                        S.sz[pos] = oz_[u];
                        S.ss[pos] = slot[u];
                    }
                    ++pos;
                }
            }
            nst += btot;
#pragma unroll
            for (int u = 0; u < kBlockUnroll; ++u) {
                slot[u] = slot_n[u];
                hb[u] = hb_n[u];
                lb[u] = lb_n[u];
            }
        }
    }
    const bool stage_ok = block_ok && nst <= C;
    if (!stage_ok && block_ok && 2 * gsz > NW && NW > 1) {
        gsz >>= 1;
        __syncthreads();
        continue;
    }
    const int nw = (nst + 31) >> 5;
    if (stage_ok) {
        // pad the last word with far-away entries; boxes of the staged words
        for (int j = nst + tid; j < nw * 32; j += G) {
            S.sx[j] = 1e30f;
            S.sy[j] = 1e30f;
            S.sz[j] = 1e30f;
            S.ss[j] = 0u;
        }
        for (int w = tid; w < nw; w += G) {
            float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
            const int j1 = min(nst, w * 32 + 32);
            for (int j = w * 32; j < j1; ++j) {
                const float cx = S.sx[j], cy = S.sy[j], cz = S.sz[j];
                mn[0] = fminf(mn[0], cx); mx[0] = fmaxf(mx[0], cx);
                mn[1] = fminf(mn[1], cy); mx[1] = fmaxf(mx[1], cy);
                mn[2] = fminf(mn[2], cz); mx[2] = fmaxf(mx[2], cz);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                S.wbox[w][i] = mn[i];
                S.wbox[w][3 + i] = mx[i];
            }
        }
    }
    __syncthreads();

    // ---- per-thread selection ----------------------------------------------------
    const bool act = stage_ok && mine && (wsel >> wib & 1u);
    if (act) {
        served = true;
        my_nst = nst;
    }
    if (stage_ok && (wsel >> wib & 1u)) {
        // A: list the staged candidates with d~ <= R (words outside the warp's box skipped)
        float qb[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) qb[i] = S.qbox[wib][i];
        const float R2a = act ? R2 : -1.0f;
        const unsigned long long QX = f2_pack(qx), QY = f2_pack(qy), QZ = f2_pack(qz), R2A = f2_pack(R2a);
        // a word is scanned when some lane's sphere meets its box (distance
        // from the query to the box against R, with slack for rounding)
        const float R2w = act ? R2 * 1.0001f + 1e-30f : -1.0f;
        KNN_LOOP_HINT
        for (int w = 0; w < nw; ++w) {
            bool ov = S.wbox[w][0] <= qb[3] && S.wbox[w][3] >= qb[0];
            if (DIM > 1) ov = ov && S.wbox[w][1] <= qb[4] && S.wbox[w][4] >= qb[1];
            if (DIM > 2) ov = ov && S.wbox[w][2] <= qb[5] && S.wbox[w][5] >= qb[2];
            if (!ov) continue;
            {
                const float ex = fmaxf(0.0f, fmaxf(S.wbox[w][0] - qx, qx - S.wbox[w][3]));
                float bd2 = ex * ex;
                if (DIM > 1) {
                    const float ey = fmaxf(0.0f, fmaxf(S.wbox[w][1] - qy, qy - S.wbox[w][4]));
                    bd2 = fmaf(ey, ey, bd2);
                }
                if (DIM > 2) {
                    const float ez = fmaxf(0.0f, fmaxf(S.wbox[w][2] - qz, qz - S.wbox[w][5]));
                    bd2 = fmaf(ez, ez, bd2);
                }
                if (!__any_sync(0xffffffffu, bd2 <= R2w)) continue;
            }
            // the word's 32 distances first (independent loads, two per packed
            // instruction), then the list; bit b set when R^2 - d~^2 >= 0
            uint32_t mp[4] = {0u, 0u, 0u, 0u};
            const ulonglong2 *X = reinterpret_cast<const ulonglong2 *>(S.sx + w * 32);
            const ulonglong2 *Y = reinterpret_cast<const ulonglong2 *>(S.sy + w * 32);
            const ulonglong2 *Z = reinterpret_cast<const ulonglong2 *>(S.sz + w * 32);
#pragma unroll
            for (int b4 = 0; b4 < 8; ++b4) {
                const ulonglong2 xv = X[b4];
                ulonglong2 yv, zv;
                if (DIM > 1) yv = Y[b4];
                if (DIM > 2) zv = Z[b4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned long long dx = f2_sub(h ? xv.y : xv.x, QX);
                    unsigned long long d2 = f2_mul(dx, dx);
                    if (DIM > 1) {
                        const unsigned long long dy = f2_sub(h ? yv.y : yv.x, QY);
                        d2 = f2_fma(dy, dy, d2);
                    }
                    if (DIM > 2) {
                        const unsigned long long dz = f2_sub(h ? zv.y : zv.x, QZ);
                        d2 = f2_fma(dz, dz, d2);
                    }
                    const unsigned long long df = f2_sub(R2A, d2);
                    const int b = 4 * b4 + 2 * h;
                    mp[(2 * h) & 3] |= ((~(uint32_t)df) >> 31) << b;
                    mp[(2 * h + 1) & 3] |= ((~(uint32_t)(df >> 32)) >> 31) << (b + 1);
                }
            }
            uint32_t m = (mp[0] | mp[1]) | (mp[2] | mp[3]);
            while (m) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                if (cnt < kGroupList) S.list[list_at(cnt, tid)] = (uint16_t)(w * 32 + b);
                ++cnt;
            }
        }
    }
    if (act) {
        if (cnt < k) {
            reason = 1;
        } else if (cnt < kGroupList) {
            // B: histogram of the list in 32 buckets of d~^2 / R^2
            const float bscale = 32.0f / R2;
#pragma unroll
            for (int b = 0; b < kBlockBins; ++b) S.hist[hist_at<G>(b, tid)] = 0;
            KNN_LOOP_HINT
            for (int e0 = 0; e0 < cnt; e0 += 4) {
                int bk[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int e = min(e0 + u, cnt - 1);
                    const int j = S.list[list_at(e, tid)];
                    const float d2 = group_d2<DIM>(S.sx[j], S.sy[j], S.sz[j], qx, qy, qz);
                    bk[u] = e0 + u < cnt ? min(kBlockBins - 1, (int)(d2 * bscale)) : -1;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (bk[u] >= 0) ++S.hist[hist_at<G>(bk[u], tid)];
            }
            int cum = 0, bstar = kBlockBins - 1, c_lo = 0, m_b = 0;
            KNN_LOOP_HINT
            for (int b = 0; b < kBlockBins; ++b) {
                const int h = S.hist[hist_at<G>(b, tid)];
                if (cum + h >= k) {
                    bstar = b;
                    c_lo = cum;
                    m_b = h;
                    break;
                }
                cum += h;
            }
            if (m_b <= kBlockBoundary) {
                // C: buckets below taken whole, the boundary bucket kept aside
                int nsure = 0, nb = 0;
                float nextmin = R2;  // anything not listed lies beyond R
                KNN_LOOP_HINT
                for (int e0 = 0; e0 < cnt; e0 += 4) {
                    int jj[4], bk[4];
                    float dd[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int e = min(e0 + u, cnt - 1);
                        jj[u] = S.list[list_at(e, tid)];
                        dd[u] = group_d2<DIM>(S.sx[jj[u]], S.sy[jj[u]], S.sz[jj[u]], qx, qy, qz);
                        bk[u] = e0 + u < cnt ? min(kBlockBins - 1, (int)(dd[u] * bscale)) : kBlockBins;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (bk[u] < bstar) {
                            if (nsure < c_lo) S.list[list_at(nsure, tid)] = (uint16_t)jj[u];
                            ++nsure;
                        } else if (bk[u] == bstar) {
                            if (nb < m_b) {
                                S.bnd[nb * G + tid] = (uint16_t)jj[u];
                                S.bnd_d[nb * G + tid] = dd[u];
                            }
                            ++nb;
                        } else if (bk[u] < kBlockBins) {
                            nextmin = fminf(nextmin, dd[u]);
                        }
                    }
                }
                // the r smallest of the boundary bucket by (d~^2, slot), then the
                // next one; the counts of this pass must repeat the histogram's
                const int r = nsure == c_lo && nb == m_b ? k - c_lo : 0;
                uint32_t taken = 0;
                float nxt = nextmin;
                if (r > 0) {
                    KNN_LOOP_HINT
                    for (int i = 0; i <= r && i < nb; ++i) {
                        float best = FLT_MAX;
                        uint32_t bslot = 0xffffffffu;
                        int bi = 0;
                        KNN_LOOP_HINT
                        for (int e = 0; e < nb; ++e) {
                            if (taken >> e & 1u) continue;
                            const float dv = S.bnd_d[e * G + tid];
                            const uint32_t sl = S.ss[S.bnd[e * G + tid]];
                            if (dv < best || (dv == best && sl < bslot)) {
                                best = dv;
                                bslot = sl;
                                bi = e;
                            }
                        }
                        if (i < r) {
                            taken |= 1u << bi;
                            S.list[list_at(c_lo + i, tid)] = S.bnd[bi * G + tid];
                            T = best;
                        } else {
                            nxt = fminf(nxt, best);
                        }
                    }
                    // exact set: the k-th stays inside R by more than the error
                    // bound, and the next candidate is more than twice the bound
                    // beyond the k-th
                    const float e2 = 1.01f * eg + 2e-7f * R;
                    const float dT = sqrtf(T), dN = sqrtf(nxt);
                    if (dT + 2.0f * e2 > R)
                        reason = 3;
                    else if (dN - dT > 2.0f * e2)
                        reason = 0;
                }
            }
        }
    }

    // ---- rows of the accepted queries (coalesced, one row per warp step) ---------
    const unsigned acc = __ballot_sync(0xffffffffu, act && reason == 0);
    if (acc) {
        // the rows' slots only: h is solved from them afterwards
#pragma unroll 4
        for (int rr = 0; rr < 32; ++rr) {
            if (!(acc >> rr & 1u)) continue;
            const int64_t q = (int64_t)blockIdx.x * G + wib * 32 + rr;
            if (lane < k) {
                const int j = S.list[list_at(lane, wib * 32 + rr)];
                const uint32_t t = S.ss[j];
                a.ngb[q * k + lane] = (int32_t)t;
            }
        }
    }
    todo &= ~wsel;
    __syncthreads();  // the next group restages the shared buffers
    }
    // ---- everything else goes to the warp passes -----------------------------------
    const bool push = valid && !(served && reason == 0);
    if (push) {
        float Rnew = R;
        if (served && reason == 1) {
            const float g = 1.25f * powf((float)k / (float)max(cnt, 1), 1.0f / DIM);
            Rnew = R * fminf(fmaxf(g, 1.25f), 4.0f);
        } else if (served && reason == 3) {
            Rnew = fmaxf(R, sqrtf(T) + 4.0f * (1.01f * eg + 2e-7f * R)) * 1.0001f;
        }
        a.radius[qi] = Rnew;
        a.rlo[qi] = 0.0f;
        a.rhi[qi] = 0.0f;
    }
    const unsigned pm = __ballot_sync(0xffffffffu, push);
    if (pm) {
        int base = 0;
        if (lane == 0) base = atomicAdd(a.qout_count, __popc(pm));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (push) a.qout[base + __popc(pm & ((1u << lane) - 1u))] = (int32_t)qi;
    }
    // statistics: staged candidates per member query, retries and their reasons
    if (a.stats) {
        const int64_t cand = warp_sum<int64_t>(served ? (int64_t)my_nst : 0);
        const int n1 = __popc(__ballot_sync(0xffffffffu, push && served && reason == 1));
        const int n3 = __popc(__ballot_sync(0xffffffffu, push && served && reason == 3));
        if (lane == 0) {
            if (cand) atomicAdd((unsigned long long *)&a.stats[1], (unsigned long long)cand);
            if (pm) atomicAdd((unsigned long long *)&a.stats[2], (unsigned long long)__popc(pm));
            if (n1) atomicAdd((unsigned long long *)&a.stats[6], (unsigned long long)n1);
            if (n3) atomicAdd((unsigned long long *)&a.stats[8], (unsigned long long)n3);
        }
    }
}

// ---- smoothing length: one thread per query ------------------------------------
// hsml_newton (mg_hsml.cuh) solves each query's row.

// Newton iterations, summed per warp into stats[5]
__device__ __forceinline__ void add_newton_steps(int it, int64_t *stats) {
    int wsum = it;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if ((threadIdx.x & 31) == 0 && wsum && stats) atomicAdd((unsigned long long *)&stats[5], (unsigned long long)wsum);
}

// From given squared distances (nq rows of k).  KR > 0: the k <= KR distances
// are loaded once (16-byte loads when k is a multiple of 4) and kept in
// registers for all Newton steps; KR == 0: any k, read again on each step.
template <int DIM, int KR>
__global__ __launch_bounds__(128) void k_hsml_solve(const float *__restrict__ dsel, const int32_t *__restrict__ qstatus,
                                                    int64_t nq, int k, float *__restrict__ hsml,
                                                    float *__restrict__ hsml_lo, int64_t *__restrict__ stats) {
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int it = 0;
    if (q < nq && !(qstatus && (qstatus[q] & MG_Q_UNRESOLVED))) {
        const float *row = dsel + q * k;
        constexpr int KN = KR > 0 ? KR : 1;
        float dr[KN];
        if (KR > 0) {
            if ((k & 3) == 0) {
#pragma unroll
                for (int j = 0; j < KN; j += 4) {
                    if (j < k) {
                        const float4 v = __ldg(reinterpret_cast<const float4 *>(row + j));
                        dr[j] = sqrtf(v.x);
                        dr[j + 1] = sqrtf(v.y);
                        dr[j + 2] = sqrtf(v.z);
                        dr[j + 3] = sqrtf(v.w);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < KN; ++j)
                    if (j < k) dr[j] = sqrtf(__ldg(row + j));
            }
        }
        float hl = 0.0f;
        hsml[q] = hsml_newton<DIM, KR>([&](int j) -> float { return KR > 0 ? dr[j] : sqrtf(row[j]); }, k, it, &hl);
        if (hsml_lo) hsml_lo[q] = hl;
        it += 1;
    }
    add_newton_steps(it, stats);
}

// Float-float distance between a query and a neighbour from their hi/lo
// positions (hb, lb already loaded): separations by TwoSum (sep1_ff /
// wrap1_ff), squared and summed in float-float, one Newton correction of the
// square root.
template <int DIM>
__device__ __forceinline__ ff dist_ff(const float4 &h0, const float4 &l0, const float4 &hb, const float4 &lb,
                                      bool periodic, float box_hi, float box_lo) {
    const float bh[3] = {hb.x, hb.y, hb.z}, bl[3] = {lb.x, lb.y, lb.z};
    const float ah[3] = {h0.x, h0.y, h0.z}, al[3] = {l0.x, l0.y, l0.z};
    ff r2;
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
        float l;
        const float d = periodic ? wrap1_ff(bh[c], ah[c], bl[c], al[c], box_hi, box_lo, l)
                                 : sep1_ff(bh[c], ah[c], bl[c], al[c], l);
        const ff s = ff_sqr(ff{d, l});
        r2 = c == 0 ? s : ff_add(r2, s);
    }
    return ff_sqrt(r2);
}

// h from the neighbour rows (k <= 32), the search writing only the rows: the
// row's distances in FP32 (cand_d2p, the search's own expression) kept in
// registers, the Newton solve unrolled over them.
template <int DIM>
__global__ __launch_bounds__(128) void k_hsml_solve_rows(const int32_t *__restrict__ ngb,
                                                         const int32_t *__restrict__ queries,
                                                         const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                                                         bool periodic, float box_hi, float box_lo,
                                                         const int32_t *__restrict__ qstatus, int64_t nq, int k,
                                                         float *__restrict__ hsml, int64_t *__restrict__ stats) {
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int it = 0;
    if (q < nq && !(qstatus && (qstatus[q] & MG_Q_UNRESOLVED))) {
        const int32_t p = queries ? queries[q] : (int32_t)q;
        const float4 h0 = hi[p], l0 = lo[p];
        const int32_t *row = ngb + q * k;
        int32_t t[32];
        if ((k & 3) == 0) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                if (j < k) {
                    const int4 v = __ldg(reinterpret_cast<const int4 *>(row + j));
                    t[j] = v.x;
                    t[j + 1] = v.y;
                    t[j + 2] = v.z;
                    t[j + 3] = v.w;
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (j < k) t[j] = __ldg(row + j);
        }
        float dr[32];
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < k) dr[j] = sqrtf(cand_d2p(hi, lo, periodic, box_hi, box_lo, h0, l0, (uint32_t)t[j]));
        hsml[q] = hsml_newton<DIM, 32>([&](int j) -> float { return dr[j]; }, k, it);
        it += 1;
    }
    add_newton_steps(it, stats);
}

// Float-float h: the row's distances are computed in float-float as they are
// gathered (one gather), the FP32 Newton solve runs on their high parts, and
// one Newton step with the neighbour count in float-float (hsml_polish_ff)
// gives h = hsml + hsml_lo to ~1e-12.  An FP32-only h (~1e-7: FP32 distances
// and kernel values limit it on rows where a few neighbours dominate the
// slope) moved some order-1 derivatives by 1.6e-5.  The distances wait in
// shared memory (this thread's column) and every loop over them stays
// rolled: unrolled over 32 register-resident float-float distances, the
// kernel outgrew the instruction cache and stalled on instruction fetch.
// The hi/lo positions carry ~2^-48 |x| of representation error, ~1.2e-14 |x|
// of a distance: a row whose largest distance is below ~1e-4 of |x| (|x| the
// query's frame-relative coordinates, or the box side) would lose h beyond
// 1e-10 to it, so its distances are recomputed from the FP64 positions
// (d2_exact, the parity metric) before the solve.
template <int DIM>
__global__ __launch_bounds__(128) void k_hsml_solve_rows_ff(const int32_t *__restrict__ ngb,
                                                            const int32_t *__restrict__ queries,
                                                            const float4 *__restrict__ hi,
                                                            const float4 *__restrict__ lo, bool periodic, float box_hi,
                                                            float box_lo, const double *__restrict__ pos64,
                                                            double box64, const int32_t *__restrict__ qstatus,
                                                            int64_t nq, int k, float *__restrict__ hsml,
                                                            float *__restrict__ hsml_lo, int64_t *__restrict__ stats) {
    __shared__ float sdh[32 * 128], sdl[32 * 128];  // [neighbour][thread]
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int it = 0;
    if (q < nq && !(qstatus && (qstatus[q] & MG_Q_UNRESOLVED))) {
        const int32_t p = queries ? queries[q] : (int32_t)q;
        const float4 h0 = hi[p], l0 = lo[p];
        const int32_t *row = ngb + q * k;
        const int tx = threadIdx.x;
        float dmax = 0.0f;
        if ((k & 3) == 0) {
#pragma unroll 2
            for (int j = 0; j < k; j += 4) {
                const int4 v = __ldg(reinterpret_cast<const int4 *>(row + j));
                const int32_t tv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const ff d = dist_ff<DIM>(h0, l0, hi[tv[u]], lo[tv[u]], periodic, box_hi, box_lo);
                    sdh[(j + u) * 128 + tx] = d.hi;
                    sdl[(j + u) * 128 + tx] = d.lo;
                    dmax = fmaxf(dmax, d.hi);
                }
            }
        } else {
#pragma unroll 4
            for (int j = 0; j < k; ++j) {
                const int32_t s = __ldg(row + j);
                const ff d = dist_ff<DIM>(h0, l0, hi[s], lo[s], periodic, box_hi, box_lo);
                sdh[j * 128 + tx] = d.hi;
                sdl[j * 128 + tx] = d.lo;
                dmax = fmaxf(dmax, d.hi);
            }
        }
        float xq = fmaxf(fabsf(h0.x), fmaxf(fabsf(h0.y), fabsf(h0.z)));
        if (periodic) xq = fmaxf(xq, box_hi);
        if (1.2e-14f * xq > 1e-10f * dmax) {
#pragma unroll 1
            for (int j = 0; j < k; ++j) {
                const double d2 = d2_exact(pos64, p, __ldg(row + j), periodic, box64);
                const float d2h = (float)d2;
                const ff d = ff_sqrt(ff{d2h, (float)(d2 - (double)d2h)});
                sdh[j * 128 + tx] = d.hi;
                sdl[j * 128 + tx] = d.lo;
            }
        }
        const float h32 = hsml_newton<DIM, 0, true>([&](int j) -> float { return sdh[j * 128 + tx]; }, k, it);
        it += 1;
        const ff h = hsml_polish_ff<DIM, 1, 0>([&](int j) { return ff{sdh[j * 128 + tx], sdl[j * 128 + tx]}; }, k,
                                               h32);
        hsml[q] = h.hi;
        hsml_lo[q] = h.lo;
    }
    add_newton_steps(it, stats);
}

// Squared distances of the neighbour rows (k > 32, for k_hsml_solve<DIM, 0>).
__global__ __launch_bounds__(256) void k_row_d2(const int32_t *__restrict__ ngb, const int32_t *__restrict__ queries,
                                                const float4 *__restrict__ hi, const float4 *__restrict__ lo,
                                                bool periodic, float box_hi, float box_lo, int64_t nq, int k,
                                                float *__restrict__ d2) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= nq * (int64_t)k) return;
    const int64_t q = e / k;
    const int32_t p = queries ? queries[q] : (int32_t)q;
    d2[e] = cand_d2p(hi, lo, periodic, box_hi, box_lo, hi[p], lo[p], (uint32_t)ngb[e]);
}

template <int DIM>
static void launch_hsml_solve(unsigned hb, cudaStream_t st, const float *dsel, const int32_t *qstatus, int64_t nq,
                              int k, float *hsml, int64_t *stats) {
    if (k <= 32)
        k_hsml_solve<DIM, 32><<<hb, 128, 0, st>>>(dsel, qstatus, nq, k, hsml, nullptr, stats);
    else
        k_hsml_solve<DIM, 0><<<hb, 128, 0, st>>>(dsel, qstatus, nq, k, hsml, nullptr, stats);
}

// h of every resolved query from its neighbour row; dsel: nq * k scratch for k > 32
// hsml_lo (may be NULL): the low part of each h (float-float: k <= 32 from
// float-float distances; k > 32 the Newton solve's last step kept as an
// unevaluated sum, ~1e-8)
template <int DIM>
static int launch_hsml_rows(cudaStream_t st, const KnnArgs &a, const int32_t *qstatus, int64_t nq, int k,
                            float *dsel, float *hsml, float *hsml_lo, int64_t *stats) {
    const unsigned hb = (unsigned)((nq + 127) / 128);
    if (k <= 32) {
        if (hsml_lo)
            k_hsml_solve_rows_ff<DIM><<<hb, 128, 0, st>>>(a.ngb, a.queries, a.hi, a.lo, a.periodic, a.box_hi,
                                                          a.box_lo, a.pos64, a.box64, qstatus, nq, k, hsml, hsml_lo,
                                                          stats);
        else
            k_hsml_solve_rows<DIM><<<hb, 128, 0, st>>>(a.ngb, a.queries, a.hi, a.lo, a.periodic, a.box_hi, a.box_lo,
                                                       qstatus, nq, k, hsml, stats);
        MG_CHECK_LAUNCH();
        return MG_OK;
    }
    const int64_t ne = nq * (int64_t)k;
    k_row_d2<<<(unsigned)((ne + 255) / 256), 256, 0, st>>>(a.ngb, a.queries, a.hi, a.lo, a.periodic, a.box_hi,
                                                            a.box_lo, nq, k, dsel);
    MG_CHECK_LAUNCH();
    k_hsml_solve<DIM, 0><<<hb, 128, 0, st>>>(dsel, qstatus, nq, k, hsml, hsml_lo, stats);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

__global__ void k_count_pass(const int32_t *qcount, int64_t *stats) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && *qcount > 0) atomicAdd((unsigned long long *)&stats[0], 1ull);
}

// ---- plain seed --------------------------------------------------------------
// h from the particle count of the query's adaptive cell: the finest level whose
// cell around the query still holds at least max(2, k/4) particles.
__device__ __forceinline__ void own_cell_range(const CellIndex &ci, uint64_t key, int L, uint32_t &a, uint32_t &b) {
    cell_lookup(ci, L, key >> (3 * (kKeyBits - L)), a, b);
}

// Finest level at which the Morton keys a and b share a cell (kMaxLevel at most).
__device__ __forceinline__ int common_level(uint64_t a, uint64_t b) {
    const uint64_t x = a ^ b;
    if (x == 0) return kMaxLevel;
    const int hb = 63 - __clzll((long long)x);  // highest differing bit; level l uses bits >= 3 (21 - l)
    return min(kMaxLevel, (62 - hb) / 3);
}

// Adaptive level of slot p without cell lookups: the own cell at level l holds
// >= cmin particles exactly when some run of cmin consecutive slots containing
// p shares its level-l prefix, i.e. when the first and last keys of that run do
// (the keys are sorted).  Window w (0 <= w < cmin) is the run starting at
// p - w; the level is the largest common level over the windows.
__device__ __forceinline__ int window_level(const uint64_t *__restrict__ keys, int64_t n, int64_t p, int cmin, int w) {
    const int64_t s = p - w;
    if (w >= cmin || s < 0 || s + cmin - 1 >= n) return 0;
    return common_level(keys[s], keys[s + cmin - 1]);
}

__global__ void k_seed_plain(const CellIndex ci, int64_t n, const double *__restrict__ framep, const int32_t *queries,
                             int64_t nq, int k, int dim, float *__restrict__ seed_h) {
    int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= nq) return;
    const int32_t p = queries ? queries[q] : (int32_t)q;
    const int cmin = max(2, k / 4);
    int L = 0;
    for (int w = 0; w < cmin; ++w) L = max(L, window_level(ci.keys, n, p, cmin, w));
    uint32_t a0, b0;
    own_cell_range(ci, ci.keys[p], L, a0, b0);
    const uint32_t cnt = b0 - a0;
    // side / 2^L: the power-of-two scaling is exact, so scaling the FP32
    // rounding of side equals rounding the FP64 quotient (no FP64 division,
    // whose rate on this GPU made it the seed passes' bottleneck)
    const float s = ldexpf((float)framep[3], -L);
    const float c = (float)max(cnt, 1u);
    float h;
    if (dim == 3)
        h = s * cbrtf(3.0f * k / (4.0f * 3.14159265f * c));
    else if (dim == 2)
        h = s * sqrtf(k / (3.14159265f * c));
    else
        h = s * k / (2.0f * c);
    seed_h[q] = h;
}

// ---- seed-network features -----------------------------------------------------
// One warp per run of consecutive queries.  The adaptive level (finest level
// whose cell around the query holds >= max(2, k/4) particles) comes from the
// keys of the neighbouring slots (window_level), one window per lane.  Features: log2(1 + count) of
// the 27 cells around the query at levels L+1 and L (finer first); a query in
// the same level-(L+1) cell as the previous one reuses its values.
__global__ __launch_bounds__(256) void k_seed_features(const CellIndex ci, int64_t n,
                                                       const double *__restrict__ framep,
                                                       const int32_t *queries, int64_t nq, int k,
                                                       int dim, int periodic,
                                                       uint16_t *__restrict__ feat,
                                                       float *__restrict__ cell_side) {
    const int lane = threadIdx.x & 31;
    const int64_t gwarp = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t per = (nq + nwarps - 1) / nwarps;
    const int64_t q0 = gwarp * per, q1 = min(nq, q0 + per);
    const int cmin = max(2, k / 4);
    const float side = (float)framep[3];
    int cachedL = -1;
    uint64_t cachedCell = ~0ull;
    uint32_t w0 = 0, w1 = 0;  // packed bf16 pairs of this lane's two output columns
    for (int64_t q = q0; q < q1; ++q) {
        const int32_t p = queries ? queries[q] : (int32_t)q;
        const uint64_t key = ci.keys[p];
        // adaptive level from runs of cmin consecutive keys (lane w: the run
        // starting at p - w)
        int L = 0;
        for (int w = lane; w < cmin; w += 32) L = max(L, window_level(ci.keys, n, p, cmin, w));
        L = (int)__reduce_max_sync(0xffffffffu, (unsigned)L);
        const int Lf = min(L + 1, kMaxLevel);
        const uint64_t cellF = key >> (3 * (kKeyBits - Lf));
        if (L != cachedL || cellF != cachedCell) {
            cachedL = L;
            cachedCell = cellF;
            uint32_t c21[3] = {0, 0, 0};
            for (int b = 0; b < kKeyBits; ++b) {
                c21[0] |= (uint32_t)((key >> (3 * b)) & 1ull) << b;
                c21[1] |= (uint32_t)((key >> (3 * b + 1)) & 1ull) << b;
                c21[2] |= (uint32_t)((key >> (3 * b + 2)) & 1ull) << b;
            }
            float vals[2] = {0.0f, 0.0f};
            for (int lev = 0; lev < 2; ++lev) {
                const int LL = lev == 0 ? Lf : L;
                const int M = 1 << LL;
                if (lane < 27) {
                    const int off[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
                    int g[3];
                    bool inside = true;
                    for (int d = 0; d < 3; ++d) {
                        g[d] = (int)(c21[d] >> (kKeyBits - LL)) + (d < dim ? off[d] : 0);
                        if (d >= dim && off[d] != 0) inside = false;  // collapsed axis
                        if (periodic)
                            g[d] = ((g[d] % M) + M) % M;
                        else if (g[d] < 0 || g[d] >= M)
                            inside = false;
                    }
                    if (inside) {
                        uint32_t ca, cb;
                        cell_range(ci, LL, (uint32_t)g[0], (uint32_t)g[1], (uint32_t)g[2], ca, cb);
                        // the fast intrinsic: the feature is rounded to BF16
                        // (8 bits) for the network, far coarser than its error
                        vals[lev] = __log2f(1.0f + (float)(cb - ca));
                    }
                }
            }
            // columns: [0, 27) level L+1, [27, 54) level L, [54, 64) zero
            float c0 = 0.0f, c1 = 0.0f;
            {
                const int idx0 = lane, idx1 = lane + 32;
                const float x0 = __shfl_sync(0xffffffffu, vals[0], idx0 < 27 ? idx0 : 0);
                const float y0 = __shfl_sync(0xffffffffu, vals[1], (idx0 >= 27 && idx0 < 54) ? idx0 - 27 : 0);
                const float y1 = __shfl_sync(0xffffffffu, vals[1], (idx1 < 54) ? idx1 - 27 : 0);
                c0 = idx0 < 27 ? x0 : y0;
                c1 = idx1 < 54 ? y1 : 0.0f;
            }
            auto bf = [](float v) -> uint32_t {
                uint32_t bits = __float_as_uint(v);
                bits += 0x7fffu + ((bits >> 16) & 1u);
                return bits >> 16;
            };
            w0 = bf(c0);
            w1 = bf(c1);
        }
        uint16_t *row = feat + q * MG_MLP_IN_PAD;
        row[lane] = (uint16_t)w0;
        row[lane + 32] = (uint16_t)w1;
        if (lane == 0) cell_side[q] = ldexpf(side, -L);  // = (float)(side / 2^L), exact scaling
    }
}

// ---- smoothing lengths, densities and volumes in row order ----------------------
// src/meshoid/Meshoid.py:169-170: density = des_ngb m / (volnorm h^dim),
// vol = m / density, volnorm = 2, pi, 4 pi / 3 in 1/2/3-D.
__global__ void k_density(const int32_t *__restrict__ out_rows, const float *__restrict__ hsml,
                          const float *__restrict__ hsml_lo, int64_t nq,
                          const double *__restrict__ m_rows, double des_ngb, double inv_ngb, int dim,
                          double volnorm, double *__restrict__ h_out, double *__restrict__ density,
                          double *__restrict__ vol, bool gather) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nq) return;
    // scatter: query i to row out_rows[i]; gather: row i from query out_rows[i] (the
    // 4-byte h are read at random instead of 24 bytes of results written so)
    const int64_t j = out_rows ? (int64_t)out_rows[i] : i;
    const int64_t q = gather ? j : i, r = gather ? i : j;
    const double h = (double)hsml[q] + (hsml_lo ? (double)hsml_lo[q] : 0.0);
    const double hd = dim == 3 ? h * h * h : (dim == 2 ? h * h : h);
    const double m = m_rows ? m_rows[r] : 1.0;
    const double v = volnorm * hd;  // vol = m / density = volnorm h^dim / des_ngb
    h_out[r] = h;
    // one FP64 division per particle (they run at a small fraction of the
    // FP32 rate on this GPU); the volume takes 1 / des_ngb (from the host) as
    // a product
    if (density) density[r] = des_ngb * m / v;
    if (vol) vol[r] = v * inv_ngb;
}

// ---- per-row FP64 distances, sorted ---------------------------------------------
// A warp sorts one row: element 32 j + lane of the row sits in key[j], and a
// bitonic network over the 32 KPL elements orders them by (FP64 d^2, particle
// index); strides of 32 and more are exchanges between the lane's own
// elements, smaller ones shuffles.  d^2 >= 0 is compared by its bits as an
// integer, which order the same way: FP64 comparisons run at 1/64 of the FP32
// rate here (262,147 rows of 64 with them: 3.5 ms).  k is a run-time value and KPL = 1, 2 or 4
// covers it, so that a row of 32 pays for 32 elements and not for 128.  Bound:
// shuffles (three 32-bit words per exchange: 15 / 42 / 112 exchanges per lane
// at KPL 1 / 2 / 4) and the FP64 pipe (d^2 and the square root, ~25 operations
// a neighbour); the 16 B per neighbour of output are written coalesced and
// straight to the user's rows.  262,147 rows of 64: 0.89 ms; taking the
// minimum k times by a warp reduction, and permuting both outputs into the
// user's order afterwards, took 27.8 + 0.19 ms.
template <int KPL>
__global__ __launch_bounds__(256) void k_neighbor_dist(const double *__restrict__ pos64,
                                                       const int32_t *__restrict__ order,
                                                       const int32_t *queries, int64_t nq,
                                                       const int32_t *__restrict__ ngb, int k,
                                                       bool periodic, double box,
                                                       const int32_t *__restrict__ out_rows,
                                                       int64_t *__restrict__ out_idx,
                                                       double *__restrict__ out_d) {
    const int lane = threadIdx.x & 31;
    const int64_t q = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= nq) return;
    const int32_t p = queries ? queries[q] : (int32_t)q;
    const int32_t *row = ngb + q * k;
    const long long inf = 0x7ff0000000000000ll;
    long long key[KPL];
    int32_t tie[KPL];
#pragma unroll
    for (int j = 0; j < KPL; ++j) {
        const int e = lane + 32 * j;
        key[j] = inf;
        tie[j] = INT_MAX;
        if (e < k) {
            const int32_t s = row[e];
            key[j] = __double_as_longlong(d2_exact(pos64, p, s, periodic, box));
            tie[j] = order[s];
        }
    }
#pragma unroll
    for (int size = 2; size <= 32 * KPL; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
                const int js = stride >> 5;
#pragma unroll
                for (int j = 0; j < KPL; ++j) {
                    if (j & js) continue;
                    const bool up = ((32 * j) & size) == 0;
                    const bool gt = key[j] > key[j ^ js] || (key[j] == key[j ^ js] && tie[j] > tie[j ^ js]);
                    if (gt == up) {
                        const long long tk = key[j];
                        const int32_t tt = tie[j];
                        key[j] = key[j ^ js];
                        tie[j] = tie[j ^ js];
                        key[j ^ js] = tk;
                        tie[j ^ js] = tt;
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < KPL; ++j) {
                    const long long ok = __shfl_xor_sync(0xffffffffu, key[j], stride);
                    const int32_t ot = __shfl_xor_sync(0xffffffffu, tie[j], stride);
                    const bool up = (((32 * j) | lane) & size) == 0;
                    const bool lower = (lane & stride) == 0;
                    const bool gt = key[j] > ok || (key[j] == ok && tie[j] > ot);
                    const bool lt = key[j] < ok || (key[j] == ok && tie[j] < ot);
                    // the lower element of an ascending pair keeps the smaller of the two
                    if (lower == up ? gt : lt) {
                        key[j] = ok;
                        tie[j] = ot;
                    }
                }
            }
        }
    }
    const int64_t r = out_rows ? (int64_t)out_rows[q] : q;
#pragma unroll
    for (int j = 0; j < KPL; ++j) {
        const int e = lane + 32 * j;
        if (e < k) {
            out_idx[r * k + e] = tie[j];
            out_d[r * k + e] = sqrt(__longlong_as_double(key[j]));
        }
    }
}

}  // namespace mg

using namespace mg;

template <int DIM>
static int launch_knn_d(unsigned blocks, cudaStream_t st, const KnnArgs &a) {
    const size_t smem = sizeof(KnnSmem<1>) * kKnnWarps;
    MG_CUDA(cudaFuncSetAttribute(k_knn_hsml<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_knn_hsml<DIM><<<blocks, kKnnWarps * 32, smem, st>>>(a);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

template <int DIM, int KPL>
static int launch_pass_t(unsigned blocks, unsigned heavy_blocks, cudaStream_t st, const KnnPassArgs &a) {
    const size_t smem = sizeof(KnnSmem<KPL>) * kKnnWarps;
    MG_CUDA(cudaFuncSetAttribute(k_knn_pass<DIM, KPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_knn_pass<DIM, KPL><<<blocks, kKnnWarps * 32, smem, st>>>(a);
    MG_CHECK_LAUNCH();
    k_knn_heavy<DIM, KPL><<<heavy_blocks, kHeavyThreads, 0, st>>>(a);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

template <int DIM>
static int launch_pass_d(int k, unsigned blocks, unsigned heavy_blocks, cudaStream_t st, const KnnPassArgs &a) {
    if (k <= 32) return launch_pass_t<DIM, 1>(blocks, heavy_blocks, st, a);
    return k <= 64 ? launch_pass_t<DIM, 2>(blocks, heavy_blocks, st, a)
                   : launch_pass_t<DIM, 4>(blocks, heavy_blocks, st, a);
}

template <int DIM>
static int launch_group_d(cudaStream_t st, const KnnArgs &a) {
    auto fn = a.periodic ? k_knn_group<DIM, true> : k_knn_group<DIM, false>;
    const size_t smem = sizeof(GroupSmem) * kGroupWarps;
    MG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fn<<<(unsigned)((a.nq + 32 * kGroupWarps - 1) / (32 * kGroupWarps)), 32 * kGroupWarps, smem, st>>>(a);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

static int launch_group(int dim, cudaStream_t st, const KnnArgs &a) {
    if (dim == 1) return launch_group_d<1>(st, a);
    if (dim == 2) return launch_group_d<2>(st, a);
    return launch_group_d<3>(st, a);
}

template <int DIM>
static int launch_group_block_d(cudaStream_t st, const KnnPassArgs &a) {
    auto fn = k_knn_group_block<DIM, kBlockThreads, kBlockStage>;
    const size_t smem = sizeof(BlockSmem<kBlockThreads, kBlockStage>);
    MG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fn<<<(unsigned)((a.nq + kBlockThreads - 1) / kBlockThreads), kBlockThreads, smem, st>>>(a);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

static int launch_group_block(int dim, cudaStream_t st, const KnnPassArgs &a) {
    if (dim == 1) return launch_group_block_d<1>(st, a);
    if (dim == 2) return launch_group_block_d<2>(st, a);
    return launch_group_block_d<3>(st, a);
}

// process-wide switch of the first (group) pass; atomic so that a call on
// one host thread may flip it while another thread launches searches
static std::atomic<int> g_group_pass{1};

extern "C" int mg_knn_set_group_pass(int32_t enabled) {
    return g_group_pass.exchange(enabled ? 1 : 0);
}

// The warp path is launched the same way whatever this is set to.  It keeps its setting for its callers.
static std::atomic<int> g_persistent_passes{0};

extern "C" int mg_knn_set_persistent_passes(int32_t enabled) {
    return g_persistent_passes.exchange(enabled ? 1 : 0);
}

static int launch_knn(int dim, unsigned blocks, cudaStream_t st, const KnnArgs &a) {
    if (dim == 1) return launch_knn_d<1>(blocks, st, a);
    if (dim == 2) return launch_knn_d<2>(blocks, st, a);
    return launch_knn_d<3>(blocks, st, a);
}

static int launch_pass(int dim, unsigned blocks, unsigned heavy_blocks, cudaStream_t st, const KnnPassArgs &a) {
    if (dim == 1) return launch_pass_d<1>(a.k, blocks, heavy_blocks, st, a);
    if (dim == 2) return launch_pass_d<2>(a.k, blocks, heavy_blocks, st, a);
    return launch_pass_d<3>(a.k, blocks, heavy_blocks, st, a);
}

static inline CellIndex make_index(const mg_cells *c) {
    CellIndex ci;
    ci.Lg = c->grid_level;
    ci.keys = c->keys;
    ci.cs = c->cell_start;
    const bool use_bricks = c->brick_of && c->bricks && c->brick_capacity > 0;
    ci.brick_of = use_bricks ? c->brick_of : nullptr;
    ci.bricks = use_bricks ? c->bricks : nullptr;
    return ci;
}

static inline void fill_args(KnnArgs &a, const mg_cells *c) {
    a.ci = make_index(c);
    a.n = c->n;
    a.dim = c->dim;
    a.Lg = c->grid_level;
    a.periodic = c->boxsize > 0;
    a.box_hi = (float)c->boxsize;
    a.box64 = c->boxsize;
    a.box_lo = (float)(c->boxsize - (double)a.box_hi);
    a.frame = c->frame;
    a.keys = c->keys;
    a.cell_start = c->cell_start;
    a.order = c->order;
    a.hi = reinterpret_cast<const float4 *>(c->pos_hi);
    a.lo = reinterpret_cast<const float4 *>(c->pos_lo);
    a.pos64 = c->pos64;
}

static inline int64_t heavy_capacity(int64_t nq) { return nq < kHeavyCap ? nq : kHeavyCap; }

extern "C" size_t mg_knn_hsml_workspace_bytes(int64_t nq, int32_t k) {
    if (nq <= 0 || k < 1) return 0;
    // the selected-distance rows are scratch of the h solve only for k > 32
    const size_t dsel_entries = k > 32 ? (size_t)nq * (size_t)k : 0;
    return 3 * align_up(sizeof(float) * nq) + 2 * align_up(sizeof(int32_t) * nq) +
           align_up(sizeof(float) * dsel_entries) +
           align_up(sizeof(int32_t) * (size_t)heavy_capacity(nq) * kHeavyItem) + 3 * align_up(sizeof(int32_t) * 64) +
           1024;
}

// The search of k > 32 and of query lists: max_passes passes over the queue, the
// first one thread per query where it may be (block_first).
static int knn_passes(const mg_cells *c, const KnnArgs &a0, bool block_first, int max_passes, int nsm,
                      int32_t *counts, Carve &w, cudaStream_t st) {
    KnnPassArgs a;
    static_cast<KnnArgs &>(a) = a0;
    const int64_t nq = a.nq, hcap = heavy_capacity(nq);
    int32_t *qa = a.qout;
    a.rlo = w.take<float>(nq);
    a.rhi = w.take<float>(nq);
    int32_t *qb = w.take<int32_t>(nq);
    a.heavy = w.take<int32_t>((size_t)hcap * kHeavyItem);
    a.heavy_cap = (int)hcap;
    int32_t *hcounts = w.take<int32_t>(64), *hnext = w.take<int32_t>(64);
    if (!w.ok()) return MG_ERR_ARG;
    MG_CUDA(cudaMemsetAsync(hcounts, 0, sizeof(int32_t) * 64, st));
    MG_CUDA(cudaMemsetAsync(hnext, 0, sizeof(int32_t) * 64, st));
    const int npass = std::min(max_passes, 63);
    for (int pass = 0; pass < npass; ++pass) {
        a.qin = pass == 0 ? nullptr : (pass % 2 ? qa : qb);
        a.qin_count = pass == 0 ? nullptr : counts + (pass - 1);
        a.qout = pass % 2 ? qb : qa;
        a.qout_count = counts + pass;
        a.last_pass = pass == max_passes - 1;
        a.heavy_count = hcounts + pass;
        a.heavy_next = hnext + pass;
        // the first pass over all queries, the others persistent over the queue
        const int64_t blocks = pass == 0 ? (nq + kKnnWarps * kChunk - 1) / (kKnnWarps * kChunk) : (int64_t)nsm * 8;
        if (pass > 0) {
            k_count_pass<<<1, 32, 0, st>>>(counts + (pass - 1), a.stats);
            MG_CHECK_LAUNCH();
        }
        if (pass == 0 && block_first) {
            const int rc = launch_group_block(c->dim, st, a);
            if (rc) return rc;
            continue;
        }
        const int rc = launch_pass(c->dim, (unsigned)std::min<int64_t>(blocks, 2147483647), (unsigned)nsm * 4, st, a);
        if (rc) return rc;
    }
    return MG_OK;
}

extern "C" int mg_knn_hsml(const mg_cells *c, const int32_t *queries, int64_t nq, int32_t k,
                           const float *seed_h, float radius_factor, int32_t level_bias,
                           int32_t max_passes, int32_t *ngb,
                           float *hsml, float *hsml_lo, int32_t *qstatus, int64_t *stats, void *workspace,
                           size_t workspace_bytes, void *stream_) {
    if (!c || nq <= 0 || !seed_h || !ngb || !hsml || !qstatus || !stats) return MG_ERR_ARG;
    if (k < 1 || k > MG_MAX_K) return MG_ERR_UNSUPPORTED;
    if (k > c->n) return MG_ERR_ARG;
    if (max_passes < 1) max_passes = 1;
    if (workspace_bytes < mg_knn_hsml_workspace_bytes(nq, k)) return MG_ERR_ARG;
    cudaStream_t st = as_stream(stream_);
    Carve w(workspace, workspace_bytes);
    float *radius = w.take<float>(nq);  // first: the caller's diagnostics read it
    int32_t *queue = w.take<int32_t>(nq);
    int32_t *counts = w.take<int32_t>(64);  // queued queries (of each pass), next query to take
    float *dsel = w.take<float>(k > 32 ? (size_t)nq * (size_t)k : 0);
    if (!w.ok()) return MG_ERR_ARG;
    MG_CUDA(cudaMemsetAsync(counts, 0, sizeof(int32_t) * 64, st));
    MG_CUDA(cudaMemsetAsync(qstatus, 0, sizeof(int32_t) * nq, st));
    KnnArgs a;
    fill_args(a, c);
    a.queries = queries;
    a.nq = nq;
    a.k = k;
    a.seed_h = seed_h;
    a.radius_factor = radius_factor;
    a.level_bias = level_bias < 0 ? 0 : (level_bias > 1 ? 1 : level_bias);  // <= 5 cells per axis
    a.radius = radius;
    a.ngb = ngb;
    a.hsml = hsml;
    a.qstatus = qstatus;
    a.stats = stats;
    a.qin = nullptr;
    a.qin_count = nullptr;
    a.next = reinterpret_cast<unsigned *>(counts + 1);
    a.qout = queue;
    a.qout_count = counts;
    // a pass searched every undecided query once; a few more radii are tried in
    // place (a list is scanned again without being rebuilt), one when the
    // caller asks for one pass
    a.max_tries = max_passes == 1 ? 1 : 4 * std::min(max_passes, 64);
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const bool group = g_group_pass.load() && k <= 32 && max_passes >= 2;
    if (k > 32 || queries) {
        const int rc = knn_passes(c, a, group && !a.periodic, max_passes, nsm, counts, w, st);
        if (rc) return rc;
    } else {
        // first pass one thread per query over its warp's candidates; its leftovers
        // go to the warp path
        if (group) {
            const int rc = launch_group(c->dim, st, a);
            if (rc) return rc;
            a.qin = queue;
            a.qin_count = counts;
        }
        // persistent warps, as many blocks as the SMs hold at once
        const int64_t blocks = std::min((int64_t)nsm * kKnnMinBlocks, (nq + kKnnWarps - 1) / kKnnWarps);
        const int rc = launch_knn(c->dim, (unsigned)blocks, st, a);
        if (rc) return rc;
    }
    if (c->dim == 1) return launch_hsml_rows<1>(st, a, qstatus, nq, k, dsel, hsml, hsml_lo, stats);
    if (c->dim == 2) return launch_hsml_rows<2>(st, a, qstatus, nq, k, dsel, hsml, hsml_lo, stats);
    return launch_hsml_rows<3>(st, a, qstatus, nq, k, dsel, hsml, hsml_lo, stats);
}

extern "C" int mg_hsml_solve(const float *d2, int64_t nq, int32_t k, int32_t dim, float *hsml, int64_t *stats,
                             void *stream_) {
    if (!d2 || !hsml || nq <= 0 || k < 2 || dim < 1 || dim > 3) return MG_ERR_ARG;
    if (k > MG_MAX_K) return MG_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream_);
    const unsigned hb = (unsigned)((nq + 127) / 128);
    if (dim == 1)
        launch_hsml_solve<1>(hb, st, d2, nullptr, nq, k, hsml, stats);
    else if (dim == 2)
        launch_hsml_solve<2>(hb, st, d2, nullptr, nq, k, hsml, stats);
    else
        launch_hsml_solve<3>(hb, st, d2, nullptr, nq, k, hsml, stats);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

extern "C" int mg_seed_plain(const mg_cells *c, const int32_t *queries, int64_t nq, int32_t k,
                             float *seed_h, void *stream_) {
    if (!c || nq <= 0 || !seed_h || k < 1) return MG_ERR_ARG;
    cudaStream_t st = as_stream(stream_);
    k_seed_plain<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(make_index(c), c->n, c->frame, queries, nq, k,
                                                                  c->dim, seed_h);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

extern "C" int mg_seed_features(const mg_cells *c, const int32_t *queries, int64_t nq, int32_t k,
                                uint16_t *features, float *cell_side, void *stream_) {
    if (!c || nq <= 0 || !features || !cell_side || k < 1) return MG_ERR_ARG;
    cudaStream_t st = as_stream(stream_);
    int64_t blocks = (nq + 8 * 32 - 1) / (8 * 32);  // ~32 consecutive queries per warp
    k_seed_features<<<(unsigned)blocks, 256, 0, st>>>(make_index(c), c->n, c->frame, queries, nq, k, c->dim,
                                                                c->boxsize > 0 ? 1 : 0, features,
                                                                cell_side);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

static int density_rows(const int32_t *rows, bool gather, const float *hsml, const float *hsml_lo, int64_t nq,
                        const double *m_rows, int32_t des_ngb, int32_t dim, double *h_out, double *density,
                        double *vol, void *stream_) {
    if (nq <= 0 || !hsml || !h_out || dim < 1 || dim > 3 || des_ngb < 1) return MG_ERR_ARG;
    const double pi = 3.14159265358979323846;
    const double volnorm = dim == 1 ? 2.0 : (dim == 2 ? pi : 4.0 * pi / 3.0);
    k_density<<<(unsigned)((nq + 255) / 256), 256, 0, as_stream(stream_)>>>(rows, hsml, hsml_lo, nq, m_rows,
                                                                           (double)des_ngb, 1.0 / (double)des_ngb,
                                                                           dim, volnorm, h_out,
                                                                           density, vol, gather);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

extern "C" int mg_density(const int32_t *out_rows, const float *hsml, const float *hsml_lo, int64_t nq,
                          const double *m_rows, int32_t des_ngb, int32_t dim, double *h_out, double *density,
                          double *vol, void *stream_) {
    return density_rows(out_rows, false, hsml, hsml_lo, nq, m_rows, des_ngb, dim, h_out, density, vol, stream_);
}

extern "C" int mg_density_rows(const int32_t *queries_of_rows, const float *hsml, const float *hsml_lo, int64_t nq,
                               const double *m_rows, int32_t des_ngb, int32_t dim, double *h_out, double *density,
                               double *vol, void *stream_) {
    return density_rows(queries_of_rows, true, hsml, hsml_lo, nq, m_rows, des_ngb, dim, h_out, density, vol, stream_);
}

extern "C" int mg_neighbor_lists(const mg_cells *c, const int32_t *queries, int64_t nq,
                                 const int32_t *ngb, int32_t k, const int32_t *out_rows, int64_t *ngb_particles,
                                 double *dist, void *stream_) {
    if (!c || nq <= 0 || !ngb || !ngb_particles || !dist) return MG_ERR_ARG;
    if (k < 1 || k > MG_MAX_K) return MG_ERR_UNSUPPORTED;
    cudaStream_t st = as_stream(stream_);
    const unsigned blocks = (unsigned)((nq + 7) / 8);
    auto fn = k <= 32 ? k_neighbor_dist<1> : (k <= 64 ? k_neighbor_dist<2> : k_neighbor_dist<4>);
    fn<<<blocks, 256, 0, st>>>(c->pos64, c->order, queries, nq, ngb, k, c->boxsize > 0, c->boxsize, out_rows,
                               ngb_particles, dist);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

extern "C" int mg_neighbor_dist(const mg_cells *c, const int32_t *queries, int64_t nq,
                                const int32_t *ngb, int32_t k, int64_t *ngb_particles, double *dist,
                                void *stream_) {
    return mg_neighbor_lists(c, queries, nq, ngb, k, nullptr, ngb_particles, dist, stream_);
}
