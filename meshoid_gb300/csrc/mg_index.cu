// Spatial index: bounding frame, 63-bit Morton keys, LSD radix sort of
// (key, particle) pairs, slot-order FP32 hi/lo positions and the dense cell
// table.  This replaces cKDTree construction (src/meshoid/Meshoid.py:142-145);
// the neighbour query itself lives in mg_knn.cu.
#include <algorithm>
#include <cstdio>

#include "mg_common.cuh"
#include "mg_scan.cuh"

namespace mg {

constexpr int kRsThreads = 256;
constexpr int kRsRounds = 8;
constexpr int kRsTile = kRsThreads * kRsRounds;  // 2048 pairs per block
constexpr int kRsPasses = (64 - kSortLowBit + 7) / 8;  // 7 passes of 8 bits

// ---- bounding frame ---------------------------------------------------------

__global__ void k_bbox_partial(const double *__restrict__ pos, int64_t n, int dim,
                               double *__restrict__ partial) {
    // compared by their bits as integers (FP64 comparisons run at 1/64 of the FP32
    // rate): with a negative value's lower bits flipped they order alike; NaN skipped
    auto ordered = [](long long b) -> long long { return b ^ (b >> 63 & 0x7fffffffffffffffll); };
    long long lob[3], hib[3];
    for (int a = 0; a < 3; ++a) {
        lob[a] = ordered(__double_as_longlong(1e300));
        hib[a] = ordered(__double_as_longlong(-1e300));
    }
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (a >= dim) break;
            const long long b = __double_as_longlong(pos[i * dim + a]);
            if ((b & 0x7fffffffffffffffll) > 0x7ff0000000000000ll) continue;
            const long long k = ordered(b);
            lob[a] = min(lob[a], k);
            hib[a] = max(hib[a], k);
        }
    }
    double lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = __longlong_as_double(ordered(lob[a]));
        hi[a] = __longlong_as_double(ordered(hib[a]));
    }
    __shared__ double s[6][256];
    for (int a = 0; a < 3; ++a) {
        s[a][threadIdx.x] = lo[a];
        s[3 + a][threadIdx.x] = hi[a];
    }
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            for (int a = 0; a < 3; ++a) {
                s[a][threadIdx.x] = fmin(s[a][threadIdx.x], s[a][threadIdx.x + o]);
                s[3 + a][threadIdx.x] = fmax(s[3 + a][threadIdx.x], s[3 + a][threadIdx.x + o]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 6) partial[blockIdx.x * 6 + threadIdx.x] = s[threadIdx.x][0];
}

__global__ __launch_bounds__(256) void k_frame(const double *__restrict__ partial, int nparts, int dim,
                                               double boxsize, double *__restrict__ frame) {
    __shared__ double s[6][256];
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int b = threadIdx.x; b < nparts; b += blockDim.x)
        for (int a = 0; a < 3; ++a) {
            lo[a] = fmin(lo[a], partial[b * 6 + a]);
            hi[a] = fmax(hi[a], partial[b * 6 + 3 + a]);
        }
    for (int a = 0; a < 3; ++a) {
        s[a][threadIdx.x] = lo[a];
        s[3 + a][threadIdx.x] = hi[a];
    }
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o)
            for (int a = 0; a < 3; ++a) {
                s[a][threadIdx.x] = fmin(s[a][threadIdx.x], s[a][threadIdx.x + o]);
                s[3 + a][threadIdx.x] = fmax(s[3 + a][threadIdx.x], s[3 + a][threadIdx.x + o]);
            }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    for (int a = 0; a < 3; ++a) {
        lo[a] = a < dim ? s[a][0] : 0.0;
        hi[a] = a < dim ? s[3 + a][0] : 0.0;
    }
    double side;
    if (boxsize > 0) {
        lo[0] = lo[1] = lo[2] = 0.0;
        side = boxsize;
    } else {
        side = 0.0;
        for (int a = 0; a < dim; ++a) side = fmax(side, hi[a] - lo[a]);
        double mag = 0.0;
        for (int a = 0; a < dim; ++a) mag = fmax(mag, fmax(fabs(lo[a]), fabs(hi[a])));
        // pad so the maximum coordinate maps strictly inside the cube
        side = side * (1.0 + 1.0 / 1048576.0) + mag * 1e-12 + 1e-300;
        if (!(side > 0.0)) side = 1.0;
    }
    frame[0] = lo[0];
    frame[1] = lo[1];
    frame[2] = lo[2];
    frame[3] = side;
    frame[4] = 1.0 / side;
    for (int a = 0; a < 3; ++a) frame[5 + a] = (a < dim) ? lo[a] + 0.5 * side : 0.0;
}

// ---- keys ------------------------------------------------------------------

__global__ void k_keys(const double *__restrict__ pos, int64_t n, int dim,
                       const double *__restrict__ framep, uint64_t *__restrict__ keys,
                       int32_t *__restrict__ vals) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    Frame f = load_frame(framep);
    const double o[3] = {f.ox, f.oy, f.oz};
    const double scale = f.inv_side * (double)(1u << kKeyBits);
    uint32_t c[3] = {0, 0, 0};
    for (int a = 0; a < dim; ++a) {
        // the conversion saturates (below 0 and NaN to 0): the clamp needs no FP64
        c[a] = min(__double2uint_rz((pos[i * dim + a] - o[a]) * scale), (1u << kKeyBits) - 1u);
    }
    keys[i] = morton3(c[0], c[1], c[2]);
    vals[i] = (int32_t)i;
}

// ---- LSD radix sort (stable), 8-bit digits ------------------------------------

// Lanes whose digit equals this one's, for a valid lane: eight votes.  With
// __match_any_sync k_radix_scatter takes 36 us instead of 31 for 2^22 pairs, and the
// count of the digits 25 us instead of 7.5 with a shared add per key.
__device__ __forceinline__ unsigned digit_peers(uint32_t d, bool valid) {
    unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = d >> b & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

__global__ __launch_bounds__(kRsThreads) void k_radix_hist(const uint64_t *__restrict__ kin,
                                                           int64_t n, int shift,
                                                           uint32_t *__restrict__ counts, int nb) {
    __shared__ uint32_t h[256];
    const int tid = threadIdx.x;
    h[tid] = 0;
    __syncthreads();
    const int64_t t0 = (int64_t)blockIdx.x * kRsTile;
    uint64_t key[kRsRounds];
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
        const int64_t i = t0 + r * kRsThreads + tid;
        key[r] = i < n ? kin[i] : 0ull;
    }
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
        const int64_t i = t0 + r * kRsThreads + tid;
        if (i < n) atomicAdd(&h[(uint32_t)((key[r] >> shift) & 255u)], 1u);
    }
    __syncthreads();
    counts[(int64_t)tid * nb + blockIdx.x] = h[tid];
}

// A block's tile is ordered by digit in shared memory first and written out from
// there, so that neighbouring threads write neighbouring places: each warp ranks
// its 256 pairs by itself, one round of 32 after another, and the warps' counts are
// then scanned digit by digit.  2^22 pairs: 47 -> 31 us, of the 15 us their bytes
// take; a round of 256 at a time, written straight to its place, took four barriers
// a round and a sector a pair.
__global__ __launch_bounds__(kRsThreads) void k_radix_scatter(
    const uint64_t *__restrict__ kin, const int32_t *__restrict__ vin, uint64_t *__restrict__ kout,
    int32_t *__restrict__ vout, int64_t n, int shift, const uint32_t *__restrict__ offsets, int nb) {
    constexpr int kWarps = kRsThreads / 32;
    __shared__ uint64_t skey[kRsTile];
    __shared__ int32_t sval[kRsTile];
    __shared__ uint32_t wcnt[kWarps][256];  // per warp and digit: count, then first place in the tile
    __shared__ uint32_t to[256];            // place in the output less the place in the tile
    __shared__ uint32_t wsum[kWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) wcnt[w][tid] = 0;
    const int64_t t0 = (int64_t)blockIdx.x * kRsTile;
    const int64_t i0 = t0 + warp * (32 * kRsRounds) + lane;
    uint64_t key[kRsRounds];
    uint32_t rank[kRsRounds];
    int32_t val[kRsRounds];
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
        const int64_t i = i0 + 32 * r;
        key[r] = i < n ? kin[i] : 0ull;
        val[r] = i < n ? vin[i] : 0;
    }
    const uint32_t first = offsets[(int64_t)tid * nb + blockIdx.x];  // of digit tid
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
        const bool valid = i0 + 32 * r < n;
        const uint32_t d = (uint32_t)((key[r] >> shift) & 255u);
        const unsigned peers = digit_peers(d, valid);
        const uint32_t before = valid ? wcnt[warp][d] : 0u;
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = before + (uint32_t)__popc(peers);
        rank[r] = before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        __syncwarp();
    }
    __syncthreads();
    // digit tid: its pairs in the tile, and in the warps before each
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = wcnt[w][tid];
        wcnt[w][tid] = run;
        run += c;
    }
    const uint32_t inc = (uint32_t)warp_incl_scan((int)run);
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    uint32_t start = inc - run;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) start += w < warp ? wsum[w] : 0u;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) wcnt[w][tid] += start;
    to[tid] = first - start;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
        if (i0 + 32 * r < n) {
            const uint32_t at = wcnt[warp][(uint32_t)((key[r] >> shift) & 255u)] + rank[r];
            skey[at] = key[r];
            sval[at] = val[r];
        }
    }
    __syncthreads();
    const int m = (int)min((int64_t)kRsTile, n - t0);
    for (int i = tid; i < m; i += kRsThreads) {
        const uint64_t k = skey[i];
        const uint32_t p = to[(uint32_t)((k >> shift) & 255u)] + (uint32_t)i;
        kout[p] = k;
        vout[p] = sval[i];
    }
}

// Small sets in one block: keys and values stay in shared memory for all passes
// (two copies, 24 bytes a pair).  Warp w owns the w-th stretch of the pairs; per
// pass it counts its digits, the counts are scanned digit by digit over the warps,
// and it deals its pairs out in order, so that the sort is stable.  Seven passes
// of three to five launches each took 165 us of a set of 1,536, nearly all of it
// the launches.
constexpr int kRsOne = 8192;  // pairs at most: 192 KB, and 32 KB of counts

struct RsOneSmem {
    uint64_t key[2][kRsOne];
    int32_t val[2][kRsOne];
    uint16_t cnt[32][256];  // per warp and digit: count, then first place
    uint32_t dsum[256];
};

__global__ __launch_bounds__(1024) void k_radix_one(const uint64_t *__restrict__ kin, const int32_t *__restrict__ vin,
                                                    uint64_t *__restrict__ kout, int32_t *__restrict__ vout, int n,
                                                    int bit0, int passes) {
    extern __shared__ __align__(16) unsigned char rs_smem[];
    RsOneSmem &S = *reinterpret_cast<RsOneSmem *>(rs_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < n; i += 1024) {
        S.key[0][i] = kin[i];
        S.val[0][i] = vin[i];
    }
    const int per = ((n + 31) / 32 + 31) & ~31;  // a warp's stretch, whole chunks of 32
    const int i0 = min(n, warp * per), i1 = min(n, i0 + per);
    for (int p = 0; p < passes; ++p) {
        const int from = p & 1, shift = bit0 + 8 * p;
        for (int d = lane; d < 256; d += 32) S.cnt[warp][d] = 0;
        __syncthreads();  // the pass before has written its pairs
        for (int c = i0; c < i1; c += 32) {
            const int i = c + lane;
            const bool valid = i < i1;
            const uint32_t d = valid ? (uint32_t)((S.key[from][i] >> shift) & 255u) : 0u;
            const unsigned peers = digit_peers(d, valid);
            if (valid && lane == __ffs(peers) - 1) S.cnt[warp][d] += (uint16_t)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (tid < 256) {  // counts of one digit over the warps
            uint32_t run = 0;
#pragma unroll 8
            for (int w = 0; w < 32; ++w) {
                const uint32_t c = S.cnt[w][tid];
                S.cnt[w][tid] = (uint16_t)run;
                run += c;
            }
            S.dsum[tid] = run;
        }
        __syncthreads();
        if (warp == 0) {  // first place of each digit
            uint32_t carry = 0;
            for (int b = 0; b < 256; b += 32) {
                const uint32_t v = S.dsum[b + lane];
                const uint32_t inc = (uint32_t)warp_incl_scan((int)v);
                S.dsum[b + lane] = carry + inc - v;
                carry += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        __syncthreads();
        for (int c = i0; c < i1; c += 32) {
            const int i = c + lane;
            const bool valid = i < i1;
            const uint64_t key = valid ? S.key[from][i] : 0ull;
            const uint32_t d = (uint32_t)((key >> shift) & 255u);
            const unsigned peers = digit_peers(d, valid);
            const uint32_t base = valid ? S.cnt[warp][d] : 0u;
            __syncwarp();
            if (valid) {
                const uint32_t to = S.dsum[d] + base + (uint32_t)__popc(peers & ((1u << lane) - 1u));
                S.key[from ^ 1][to] = key;
                S.val[from ^ 1][to] = S.val[from][i];
                if (lane == __ffs(peers) - 1) S.cnt[warp][d] = (uint16_t)(base + __popc(peers));
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = tid; i < n; i += 1024) {
        kout[i] = S.key[passes & 1][i];
        vout[i] = S.val[passes & 1][i];
    }
}

static int radix_one(const uint64_t *kin, const int32_t *vin, uint64_t *kout, int32_t *vout, int64_t n, int bit0,
                     int passes, cudaStream_t st) {
    MG_CUDA(cudaFuncSetAttribute(k_radix_one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RsOneSmem)));
    k_radix_one<<<1, 1024, sizeof(RsOneSmem), st>>>(kin, vin, kout, vout, (int)n, bit0, passes);
    MG_CHECK_LAUNCH();
    return MG_OK;
}

// ---- slot-order positions -----------------------------------------------------

__global__ void k_slot_positions(const double *__restrict__ pos, int64_t n, int dim,
                                 const double *__restrict__ framep,
                                 const int32_t *__restrict__ order, int32_t *__restrict__ rank,
                                 float4 *__restrict__ hi, float4 *__restrict__ lo,
                                 double *__restrict__ pos64) {
    int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    Frame f = load_frame(framep);
    const int32_t p = order[s];
    rank[p] = (int32_t)s;
    double x[3] = {0.0, 0.0, 0.0};
    for (int a = 0; a < dim; ++a) x[a] = pos[(int64_t)p * dim + a];
    const double c[3] = {f.cx, f.cy, f.cz};
    float h[3], l[3];
    for (int a = 0; a < 3; ++a) {
        double r = x[a] - c[a];
        h[a] = (float)r;
        l[a] = (float)(r - (double)h[a]);
        pos64[s * 3 + a] = x[a];
    }
    hi[s] = make_float4(h[0], h[1], h[2], 0.0f);
    lo[s] = make_float4(l[0], l[1], l[2], 0.0f);
}

// ---- dense cell table ---------------------------------------------------------

__global__ void k_cell_count(const uint64_t *__restrict__ keys, int64_t n, int shift,
                             uint32_t *__restrict__ count) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint64_t c = i < n ? (keys[i] >> shift) : ~0ull;
    // sorted keys: a cell's particles are neighbouring lanes
    const uint64_t before = __shfl_up_sync(0xffffffffu, c, 1);
    const bool head = lane == 0 || c != before;
    const unsigned after = __ballot_sync(0xffffffffu, head) >> lane >> 1;  // heads above this lane
    if (head && i < n) atomicAdd(&count[c], (uint32_t)(after ? __ffs(after) : 32 - lane));
}

// ---- bricks: refinement tables below the dense level ----------------------------
// Level m bricks cover cells at level Lg + 3m holding more than T particles;
// each stores the first slots of its 512 descendants at level Lg + 3m + 3, the
// child brick of each descendant (-1: none) and its own slot range.  Built
// level by level without host synchronisation: lvl[2m], lvl[2m+1] hold the
// first brick id and the brick count of level m on the device.

inline int brick_levels(int Lg) {
    int m = 0;
    for (int l = Lg; l + 3 <= kMaxLevel; l += 3) ++m;
    return m;
}

// A warp sets up brick id over the slots [A, B): every first slot at the end of
// the range, no children.
__device__ __forceinline__ void brick_open(uint32_t *__restrict__ bricks, int id, uint32_t A, uint32_t B) {
    uint32_t *b = bricks + (size_t)id * kBrickWords;
    const int lane = threadIdx.x & 31;
    for (int s = lane; s < 513; s += 32) b[s] = B;
    for (int s = lane; s < 512; s += 32) b[kBrickChild + s] = 0xffffffffu;
    if (lane == 0) {
        b[kBrickRange] = A;
        b[kBrickRange + 1] = B;
    }
}

// Level 0: a brick for every dense cell over the threshold.  The bricks of a
// level are numbered in the order in which warps ask for them.
__global__ __launch_bounds__(256) void k_brick_top(const uint32_t *__restrict__ cs, int64_t ncell, int T, int cap,
                                                   int32_t *__restrict__ brick_of, uint32_t *__restrict__ bricks,
                                                   int32_t *__restrict__ lvl) {
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t A = 0, B = 0;
    if (c < ncell) {
        A = cs[c];
        B = cs[c + 1];
    }
    const bool big = B - A > (uint32_t)T;
    unsigned m = __ballot_sync(0xffffffffu, big);
    int base = 0;
    if (m && lane == 0) base = atomicAdd(&lvl[1], __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    const int id = base + __popc(m & ((1u << lane) - 1u));
    if (c < ncell) brick_of[c] = big && id < cap ? id : -1;
    while (m) {
        const int j = __ffs(m) - 1;
        m &= m - 1;
        const int idj = __shfl_sync(0xffffffffu, id, j);
        const uint32_t Aj = __shfl_sync(0xffffffffu, A, j), Bj = __shfl_sync(0xffffffffu, B, j);
        if (idj < cap) brick_open(bricks, idj, Aj, Bj);
    }
}

// particle p opens a descendant of its level-m brick: record the first slot
__global__ void k_brick_mark(const uint64_t *__restrict__ keys, int64_t n, int Lg, const int32_t *__restrict__ brick_of,
                             uint32_t *__restrict__ bricks, int m) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint64_t key = keys[p];
    int br = brick_of[key >> (3 * (kKeyBits - Lg))];
    for (int l = 0; l < m && br >= 0; ++l) {
        const uint32_t sub = (uint32_t)((key >> (3 * (kKeyBits - (Lg + 3 * (l + 1))))) & 511ull);
        br = (int)bricks[(size_t)br * kBrickWords + kBrickChild + sub];
    }
    if (br < 0) return;
    uint32_t *b = bricks + (size_t)br * kBrickWords;
    const int shift = 3 * (kKeyBits - (Lg + 3 * (m + 1)));
    const uint32_t sub = (uint32_t)((key >> shift) & 511ull);
    const bool first = (uint32_t)p == b[kBrickRange] || ((keys[p - 1] >> shift) & 511ull) != sub;
    if (first) b[sub] = (uint32_t)p;
}

// A warp per level-m brick: empty descendants start where the next non-empty one
// does (a suffix minimum over the 512, 32 at a time from the end), and with
// CHILDREN a brick of the next level is opened for each descendant over the
// threshold.  (A thread per brick walked the 512 twice, with a scan of
// the bricks' counts in between: 0.12 ms of 10^6 Plummer particles, and seven
// launches per level instead of two.)
template <bool CHILDREN>
__global__ __launch_bounds__(256) void k_brick_fill(uint32_t *__restrict__ bricks, int32_t *__restrict__ lvl, int m,
                                                    int T, int cap) {
    const int lane = threadIdx.x & 31;
    const int base = lvl[2 * m], nb = min(lvl[2 * m + 1], cap - base), nbase = base + nb;
    if (CHILDREN && blockIdx.x == 0 && threadIdx.x == 0) lvl[2 * (m + 1)] = nbase;
    const int nwarps = (int)(gridDim.x * (blockDim.x >> 5));
    for (int i = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); i < nb; i += nwarps) {
        uint32_t *b = bricks + (size_t)(base + i) * kBrickWords;
        uint32_t v[16];  // descendants lane, lane + 32, ..
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = b[32 * s + lane];
        uint32_t next[16], carry = b[512];  // first slot of the descendant after each
#pragma unroll
        for (int s = 15; s >= 0; --s) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_down_sync(0xffffffffu, v[s], o);
                if (lane + o < 32) v[s] = min(v[s], t);
            }
            v[s] = min(v[s], carry);
            const uint32_t t = __shfl_down_sync(0xffffffffu, v[s], 1);
            next[s] = lane < 31 ? t : carry;
            carry = __shfl_sync(0xffffffffu, v[s], 0);
            b[32 * s + lane] = v[s];
        }
        if (CHILDREN) {
            unsigned big = 0;
#pragma unroll
            for (int s = 0; s < 16; ++s) big |= next[s] - v[s] > (uint32_t)T ? 1u << s : 0u;
            const int n = __popc(big), inc = warp_incl_scan(n);
            int first = 0;
            const int all = __shfl_sync(0xffffffffu, inc, 31);
            if (all && lane == 0) first = atomicAdd(&lvl[2 * (m + 1) + 1], all);
            first = nbase + __shfl_sync(0xffffffffu, first, 0) + inc - n;
            // one descendant of each lane at a time
            while (__any_sync(0xffffffffu, big != 0u)) {
                const int s = big ? __ffs(big) - 1 : 0;
                uint32_t A = 0, B = 0;
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    A = u == s ? v[u] : A;
                    B = u == s ? next[u] : B;
                }
                const bool open = big != 0u && first < cap;
                if (open) b[kBrickChild + 32 * s + lane] = (uint32_t)first;
                unsigned mo = __ballot_sync(0xffffffffu, open);
                while (mo) {
                    const int j = __ffs(mo) - 1;
                    mo &= mo - 1;
                    const int id = __shfl_sync(0xffffffffu, first, j);
                    const uint32_t Aj = __shfl_sync(0xffffffffu, A, j), Bj = __shfl_sync(0xffffffffu, B, j);
                    brick_open(bricks, id, Aj, Bj);
                }
                if (big) {
                    big &= big - 1;
                    ++first;
                }
            }
        }
    }
}

}  // namespace mg

using namespace mg;

// ---- generic stable sort of (u64 key, i32 value) pairs by bits [bit0, bit0 + nbits)
namespace mg {

size_t radix_sort_workspace_bytes(int64_t n) {
    const int64_t nb = (n + kRsTile - 1) / kRsTile;
    return align_up(sizeof(uint64_t) * (size_t)n) + align_up(sizeof(int32_t) * (size_t)n) +
           align_up(sizeof(uint32_t) * 256 * (size_t)nb) + align_up(scan_workspace_bytes(256 * nb)) + 1024;
}

int radix_sort_pairs(uint64_t *keys, int32_t *vals, int64_t n, int bit0, int nbits, void *ws, size_t wsb,
                     cudaStream_t st) {
    if (n <= 1 || nbits <= 0) return MG_OK;
    if (n > 0x7fffffffll || wsb < radix_sort_workspace_bytes(n)) return MG_ERR_ARG;
    const int64_t nb = (n + kRsTile - 1) / kRsTile;
    Carve w(ws, wsb);
    uint64_t *kping = w.take<uint64_t>((size_t)n);
    int32_t *vping = w.take<int32_t>((size_t)n);
    uint32_t *counts = w.take<uint32_t>(256 * (size_t)nb);
    void *scan_ws = w.take<char>(scan_workspace_bytes(256 * nb));
    if (!w.ok()) return MG_ERR_ARG;
    uint64_t *kin = keys, *kout = kping;
    int32_t *vin = vals, *vout = vping;
    const int passes = (nbits + 7) / 8;
    if (n <= kRsOne) return radix_one(keys, vals, keys, vals, n, bit0, passes, st);  // reads all before it writes
    for (int p = 0; p < passes; ++p) {
        const int shift = bit0 + 8 * p;
        k_radix_hist<<<(unsigned)nb, kRsThreads, 0, st>>>(kin, n, shift, counts, (int)nb);
        MG_CHECK_LAUNCH();
        int rc = exclusive_scan_u32(counts, counts, 256 * nb, scan_ws, st);
        if (rc) return rc;
        k_radix_scatter<<<(unsigned)nb, kRsThreads, 0, st>>>(kin, vin, kout, vout, n, shift, counts, (int)nb);
        MG_CHECK_LAUNCH();
        uint64_t *tk = kin; kin = kout; kout = tk;
        int32_t *tv = vin; vin = vout; vout = tv;
    }
    if (kin != keys) {
        MG_CUDA(cudaMemcpyAsync(keys, kin, sizeof(uint64_t) * (size_t)n, cudaMemcpyDeviceToDevice, st));
        MG_CUDA(cudaMemcpyAsync(vals, vin, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, st));
    }
    return MG_OK;
}

}  // namespace mg

extern "C" int32_t mg_brick_capacity(int64_t n, int grid_level, int threshold) {
    if (n <= 0 || threshold < 1 || grid_level < 1) return 0;
    const int64_t lv = brick_levels(grid_level);
    int64_t cap = lv * (n / threshold) + 16;
    if (cap > (1 << 30)) cap = 1 << 30;
    return (int32_t)cap;
}

// Finest level with 8^(L+1) <= 4n (about 2-16 particles per dense cell), at
// most 9: measured best or within 2% of the best with level_bias 1 for
// Plummer, clump-mixture and uniform sets of 2^18..2^24 particles.
extern "C" int mg_default_grid_level(int64_t n) {
    int L = 1;
    while (L < 9 && (int64_t)1 << (3 * (L + 1)) <= 4 * n) ++L;
    return L;
}

static size_t cell_table_entries(int L) { return ((size_t)1 << (3 * L)) + 1; }

extern "C" size_t mg_build_cells_workspace_bytes(int64_t n, int grid_level) {
    if (n <= 0 || grid_level < 1 || grid_level > 9) return 0;
    const int64_t nb = (n + kRsTile - 1) / kRsTile;
    size_t b = 0;
    b += align_up(sizeof(uint64_t) * n);           // keys ping buffer
    b += align_up(sizeof(int32_t) * n);            // vals ping buffer
    b += align_up(sizeof(uint32_t) * 256 * nb);    // digit counts / offsets
    b += align_up(scan_workspace_bytes(256 * nb));
    b += align_up(scan_workspace_bytes(cell_table_entries(grid_level)));
    b += align_up(sizeof(double) * 6 * 1024);      // bbox partials
    // bricks: level table
    b += align_up(sizeof(int32_t) * 64);
    return b + 4096;
}

extern "C" int mg_build_cells(const double *pos, mg_cells *c, void *workspace,
                              size_t workspace_bytes, void *stream_) {
    if (!pos || !c || c->n <= 0 || c->dim < 1 || c->dim > 3 || c->grid_level < 1 ||
        c->grid_level > 9 || !c->frame || !c->keys || !c->order || !c->rank || !c->pos_hi ||
        !c->pos_lo || !c->pos64 || !c->cell_start)
        return MG_ERR_ARG;
    if (c->n >= ((int64_t)1 << 31) - 1) return MG_ERR_UNSUPPORTED;
    const int64_t n = c->n;
    const int dim = c->dim;
    cudaStream_t st = as_stream(stream_);
    if (workspace_bytes < mg_build_cells_workspace_bytes(n, c->grid_level)) return MG_ERR_ARG;
    Carve w(workspace, workspace_bytes);
    const int64_t nb = (n + kRsTile - 1) / kRsTile;
    uint64_t *kping = w.take<uint64_t>(n);
    int32_t *vping = w.take<int32_t>(n);
    uint32_t *counts = w.take<uint32_t>(256 * nb);
    void *scan_ws = w.take<char>(scan_workspace_bytes(256 * nb));
    void *scan_ws2 = w.take<char>(scan_workspace_bytes(cell_table_entries(c->grid_level)));
    double *partial = w.take<double>(6 * 1024);
    if (!w.ok()) return MG_ERR_ARG;

    int nparts = (int)((n + 255) / 256);
    if (nparts > 1024) nparts = 1024;
    k_bbox_partial<<<nparts, 256, 0, st>>>(pos, n, dim, partial);
    MG_CHECK_LAUNCH();
    k_frame<<<1, 256, 0, st>>>(partial, nparts, dim, c->boxsize, c->frame);
    MG_CHECK_LAUNCH();
    const int tb = 256;
    const int64_t gb = (n + tb - 1) / tb;
    // Keys land in the ping buffer; after an odd number of passes the sorted
    // result is in the caller's arrays.
    static_assert(kRsPasses % 2 == 1, "pass count parity decides the output buffer");
    k_keys<<<gb, tb, 0, st>>>(pos, n, dim, c->frame, kping, vping);
    MG_CHECK_LAUNCH();
    uint64_t *kin = kping, *kout = c->keys;
    int32_t *vin = vping, *vout = c->order;
    if (n <= kRsOne) {
        const int rc = radix_one(kin, vin, kout, vout, n, kSortLowBit, kRsPasses, st);
        if (rc) return rc;
    }
    for (int p = 0; p < kRsPasses && n > kRsOne; ++p) {
        const int shift = kSortLowBit + 8 * p;
        k_radix_hist<<<nb, kRsThreads, 0, st>>>(kin, n, shift, counts, (int)nb);
        MG_CHECK_LAUNCH();
        int rc = exclusive_scan_u32(counts, counts, 256 * nb, scan_ws, st);
        if (rc) return rc;
        k_radix_scatter<<<nb, kRsThreads, 0, st>>>(kin, vin, kout, vout, n, shift, counts, (int)nb);
        MG_CHECK_LAUNCH();
        uint64_t *tk = kin; kin = kout; kout = tk;
        int32_t *tv = vin; vin = vout; vout = tv;
    }
    k_slot_positions<<<gb, tb, 0, st>>>(pos, n, dim, c->frame, c->order, c->rank,
                                        reinterpret_cast<float4 *>(c->pos_hi),
                                        reinterpret_cast<float4 *>(c->pos_lo), c->pos64);
    MG_CHECK_LAUNCH();
    const size_t ncell = cell_table_entries(c->grid_level);
    MG_CUDA(cudaMemsetAsync(c->cell_start, 0, sizeof(uint32_t) * ncell, st));
    k_cell_count<<<gb, tb, 0, st>>>(c->keys, n, 3 * (kKeyBits - c->grid_level), c->cell_start);
    MG_CHECK_LAUNCH();
    int rc = exclusive_scan_u32(c->cell_start, c->cell_start, (int64_t)ncell, scan_ws2, st);
    if (rc) return rc;
    if (!c->brick_of || !c->bricks || c->brick_capacity <= 0) return MG_OK;
    // ---- bricks ----
    const int T = c->brick_threshold > 0 ? c->brick_threshold : 256;
    const int cap = c->brick_capacity;
    if (cap > mg_brick_capacity(n, c->grid_level, 64)) return MG_ERR_ARG;
    const int64_t ndense = (int64_t)ncell - 1;
    int32_t *lvl = w.take<int32_t>(64);  // first brick and bricks of each level
    if (!w.ok()) return MG_ERR_ARG;
    MG_CUDA(cudaMemsetAsync(lvl, 0, sizeof(int32_t) * 64, st));
    k_brick_top<<<(unsigned)((ndense + 255) / 256), 256, 0, st>>>(c->cell_start, ndense, T, cap, c->brick_of,
                                                                  c->bricks, lvl);
    MG_CHECK_LAUNCH();
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int levels = brick_levels(c->grid_level);
    const unsigned bb = (unsigned)std::min<int64_t>((int64_t)nsm * 8, ((int64_t)cap + 7) / 8);
    for (int m = 0; m < levels; ++m) {
        k_brick_mark<<<gb, tb, 0, st>>>(c->keys, n, c->grid_level, c->brick_of, c->bricks, m);
        MG_CHECK_LAUNCH();
        if (m + 1 < levels)
            k_brick_fill<true><<<bb, 256, 0, st>>>(c->bricks, lvl, m, T, cap);
        else
            k_brick_fill<false><<<bb, 256, 0, st>>>(c->bricks, lvl, m, T, cap);
        MG_CHECK_LAUNCH();
    }
    return MG_OK;
}

extern "C" const char *mg_status_string(int s) {
    switch (s) {
        case MG_OK: return "ok";
        case MG_ERR_ARG: return "invalid argument";
        case MG_ERR_CUDA: return "CUDA error";
        case MG_ERR_NOT_CONVERGED: return "search pass cap reached for some queries";
        case MG_ERR_UNSUPPORTED: return "unsupported size or parameter";
        case MG_ERR_NOALLOC_LIMIT:
            return "more queries than the fixed scratch of the no-allocation entry point holds "
                   "(MG_NOALLOC_MAX_QUERIES); use mg_grad_sweep with a workspace";
        default: return "unknown status";
    }
}

extern "C" int mg_version(void) { return 100; }

#include <atomic>
static std::atomic<long long> g_launches{0};
void mg::count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
extern "C" int64_t mg_launch_count(void) { return (int64_t)g_launches.load(std::memory_order_relaxed); }
