// segsort.cu -- per-tile sort of tile-bucketed instances for sm_103a.
//
// The reference sorts all (tile << 32 | depth bits) keys with a stable 64-bit
// radix sort (thrust::sort_by_key, src/GSSlam.cu:624-628).  A Gaussian has at
// most one instance per tile and instances are generated in Gaussian-index
// order, so inside a tile that stable order is exactly the order of the
// unique composite key (depth bits << 32 | Gaussian index).  Instances are
// therefore collected per tile and each tile is sorted on its own:
//  * full mode: the tile bucket was filled by the scatter (any order);
//  * incremental mode: the tile's previous sorted list, minus the members
//    that left the tile, with keys recomputed for the new pose, followed by
//    the entering instances -- nearly sorted;
//  * up to 8192 instances: one CTA of 512 threads sorts the tile in shared
//    memory by distribution (sort_tile);
//  * larger tiles (big maps, coarse pyramid levels) are listed by the first
//    kernel and sorted by a second one with 1024 threads: up to 16384 instances
//    the same way, beyond that split by key range -- 4096 sampled keys (or,
//    where they miss most of the tile, exact ranks) cut the tile into ranges,
//    each of which a CTA collects from the whole source list (reading it
//    twice, but all ranges at once and without exchange);
//  * tiles above 2^20 instances go to a merge sort through global memory.
//
// A list that has not changed (no member left or entered, keys still in
// order) is copied; one with a few descents is put in order by passes over
// overlapping blocks of eight keys.
//
// The sort by distribution: 127 keys of the tile, evenly spaced in its previous
// order, become splitters; a key's segment (binary search) and its linear
// place in it give one of 1024 or 2048 buckets of a few keys, in key order.
// Every key takes a slot of its bucket (shared-memory atomics), and after a
// scan its place is the bucket's start plus the number of smaller keys in the
// bucket.  That is about 100 operations a key and six barriers, whatever
// the order before; a merge sort needs 230 and more and a barrier per round.
// Between two Gauss-Newton steps the order changes a lot more than the
// membership: at 640x360 (room of 1 M Gaussians, steps of 5e-4 rad) a tile of
// 2,200 entries has 300 to 400 descents, and keys whose sign changes cross
// the whole list, so lists sorted by passes over neighbours do not get far.
//
// What bounds it: the latency of the gathers of the survivors' binning
// records (one 32-byte sector each) and then issue.  us per binning while
// tracking, room of 1 M Gaussians at 1280x720, levels 1 / 2 (2.05 M / 0.73 M
// instances): 43 / 33, before (256 threads, neighbour passes or merge sort,
// tiles above 4096 through global memory) 62 / 76; 2 M Gaussians, level 0
// (13.2 M instances, 3,673 a tile): 206, before 466, level 2 (6,000 a tile): 120,
// before 172.
// The output is the sorted Gaussian indices; the reference-format keys are
// rebuilt on request (make_keys_kernel) since the blending kernels only read
// ranges and indices.
#include <utility>

#include "fvgs_device.cuh"
#include "fvgs_launch.h"

namespace fvgs {

constexpr int kSegThreads = 512;                   // a tile's CTA
constexpr int kShortThreads = 256;                 // a tile's CTA where lists are short
constexpr int kLargeThreads = 1024;                // a listed tile's (or range's) CTA
constexpr int kSegItems = 16;                      // keys per thread at most
constexpr int kSmallItems = 8;                     // lists of up to half the capacity
constexpr int kSegments = 128;                     // splitters + 1
constexpr int kMaxBucket = 48;                     // above it: merge sort
constexpr int kFixBlock = 8;                       // keys of a block of the passes
constexpr int kFixMaxPasses = 4;
constexpr int kFixMaxDescents = 64;                // threads that saw one
constexpr int kPartSamples = 4096;                 // splitters of a large tile's ranges
// Mean entries per tile of the grid's last binning (known to the host from the
// call before) up to which a CTA reserves shared memory for half its capacity
// only (tiles above that are listed), which leaves the gathers more L1, and
// the listed tiles' kernel takes 512 threads: its CTAs, mostly idle, then fit
// beside the last tiles' and do not hold up the kernel after them.  Below
// half of that, tiles are sorted by 256 threads, twice as many on an SM (room of
// 400 k Gaussians at 1280x720, 747 a tile, unchanged lists: the call for outlier
// scores 444 -> 425 us; box of 50 k at 640x480: Jacobian 174 -> 168 us).
constexpr uint32_t kBriefMean = 2048, kShortMean = 1024;
constexpr int kGlobalMin = 1 << 20;                // from here: merge sort through global memory
template <int NT>
constexpr int seg_cap() { return NT * kSegItems; }
// A large tile's range: up to twice this.
template <int NT>
constexpr int part_keys() { return seg_cap<NT>() / 2; }
// Buckets of a sort: two a thread, twice that in the large tiles' kernel
// (whose ranges come in random order, so their segments differ more).
template <int NT>
constexpr int seg_buckets() { return (NT > kSegThreads ? 4 : 2) * NT; }
// Keys in the padded layout of the merge sort, bucket starts, splitters (as
// sampled, in order) and the segments' scale; cap: keys at most.
template <int NT>
constexpr size_t seg_smem(int cap = seg_cap<NT>()) {
    return sizeof(uint64_t) * (size_t)(cap + cap / 16) + sizeof(uint32_t) * (seg_buckets<NT>() + 4) +
           3 * sizeof(uint32_t) * kSegments;
}
// The large tiles' kernel: the same, with the ranges' counts.
template <int NT>
constexpr size_t large_smem() { return seg_smem<NT>() + sizeof(uint32_t) * (kPartSamples + 4); }
constexpr uint64_t kKeyInf = ~0ull;

__device__ __forceinline__ int spad(int i) { return i + (i >> 4); }  // one pad word per 16 keys

// Sort ITEMS keys in registers (bitonic network, ascending).
template <int ITEMS>
__device__ __forceinline__ void sort_items(uint64_t (&k)[ITEMS]) {
#pragma unroll
    for (int sz = 2; sz <= ITEMS; sz <<= 1)
#pragma unroll
        for (int j = sz >> 1; j > 0; j >>= 1)
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const int l = i ^ j;
                if (l > i) {
                    const bool up = (i & sz) == 0;
                    const uint64_t a = k[i], b = k[l];
                    if ((a > b) == up) {
                        k[i] = b;
                        k[l] = a;
                    }
                }
            }
}

// One merge-path round over runs of length L of s[0..m) (m a multiple of
// ITEMS): thread t produces outputs [ITEMS t, ITEMS (t + 1)) of the pair of runs
// containing them.
// Returns false when the pair is already in order (nothing to write).  Both
// run heads are re-read from shared memory each step (register-held heads
// measured slower: more registers, fewer resident CTAs).
template <int ITEMS>
__device__ __forceinline__ bool merge_round(const uint64_t* s, int t, int m, int L, uint64_t (&k)[ITEMS]) {
    const int per_pair = (2 * L) / ITEMS;
    const int ps = (t / per_pair) * 2 * L;
    const int d = (t % per_pair) * ITEMS;
    const int la = min(L, m - ps);
    const int lb = min(L, max(0, m - ps - L));
    if (lb == 0 || s[spad(ps + la - 1)] <= s[spad(ps + la)]) return false;
    int lo = max(0, d - lb), hi = min(d, la);
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (s[spad(ps + mid)] <= s[spad(ps + la + d - 1 - mid)])
            lo = mid + 1;
        else
            hi = mid;
    }
    int ai = lo, bj = d - lo;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint64_t a = ai < la ? s[spad(ps + ai)] : kKeyInf;
        const uint64_t b = bj < lb ? s[spad(ps + la + bj)] : kKeyInf;
        const bool ta = a <= b;
        k[r] = ta ? a : b;
        ai += ta ? 1 : 0;
        bj += ta ? 0 : 1;
    }
    return true;
}

// Sort s[0..m) (padded layout, m a multiple of ITEMS, at most ITEMS keys a
// thread) in shared memory with the CTA.  Threads >= m/ITEMS only take part in
// the barriers.  Lists of up to half the CTA's capacity use ITEMS = 8, so
// every thread sorts and merges instead of at most half of them.  While a merged pair spans at
// most one warp's 32 ITEMS keys the round touches only that warp's slice, so
// it synchronises the warp, not the CTA.
template <int ITEMS = kSegItems>
__device__ void block_merge_sort(uint64_t* s, int m) {
    const int t = threadIdx.x;
    const int active = m / ITEMS;
    uint64_t k[ITEMS];
    if (t < active) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) k[j] = s[spad(t * ITEMS + j)];
        bool sorted = true;
#pragma unroll
        for (int j = 0; j + 1 < ITEMS; ++j) sorted = sorted && k[j] <= k[j + 1];
        if (!sorted) {
            sort_items(k);
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) s[spad(t * ITEMS + j)] = k[j];
        }
    }
    __syncthreads();
    const bool desc = t + 1 < active && s[spad(t * ITEMS + ITEMS - 1)] > s[spad((t + 1) * ITEMS)];
    if (!__syncthreads_or(desc)) return;  // every run boundary already in order
    constexpr int kWarpSpan = 32 * ITEMS;
    for (int L = ITEMS; L < m; L <<= 1) {
        const bool warp_local = 2 * L <= kWarpSpan;
        bool wrote = false;
        if (t < active) wrote = merge_round(s, t, m, L, k);
        if (warp_local)
            __syncwarp();
        else
            __syncthreads();
        if (wrote) {
#pragma unroll
            for (int r = 0; r < ITEMS; ++r) s[spad(t * ITEMS + r)] = k[r];
        }
        if (4 * L <= kWarpSpan)
            __syncwarp();
        else
            __syncthreads();
    }
    __syncthreads();
}

__device__ __forceinline__ void write_sorted(uint64_t key, uint32_t dst, uint32_t* vals) {
    vals[dst] = (uint32_t)key;
}

// Incremental mode, tiles beyond shared memory: collect tile `tile`'s
// instances into dst (global memory) -- the members of the previous sorted
// list whose Gaussian's new rectangle still holds the tile, with the key for
// the new projection, and the entering instances, in any order.  Returns the
// number collected (the tile's count when consistent); writes stop at n_cap.
template <int NT>
__device__ int gather_tile(uint64_t* dst, uint32_t tile, int n_cap, const SegSortIncr& inc, uint32_t* s_count) {
    const int tx = (int)(tile % (uint32_t)inc.ntx), ty = (int)(tile / (uint32_t)inc.ntx);
    uint2 ro = inc.ranges_prev[tile];
    ro.y = (uint32_t)min((uint64_t)ro.y, inc.capacity);
    if (threadIdx.x == 0) *s_count = 0;
    __syncthreads();
    for (uint32_t i0 = ro.x; i0 < ro.y; i0 += NT) {
        const uint32_t i = i0 + threadIdx.x;
        const uint32_t g = i < ro.y ? inc.vals_prev[i] : 0xffffffffu;
        uint4 b0 = make_uint4(0, 0, 0, 0);
        float4 b1 = make_float4(0, 0, 0, 0);
        if (g < inc.n_gauss) {
            b0 = inc.bins[g].r;
            b1 = inc.bins[g].p;
        }
        const bool keep = g < inc.n_gauss && rect_contains(b0, tx, ty);
        const uint32_t bal = __ballot_sync(kFullMask, keep);
        uint32_t base = 0;
        if ((threadIdx.x & 31) == 0 && bal) base = atomicAdd(s_count, (uint32_t)__popc(bal));
        const int pos = (int)(__shfl_sync(kFullMask, base, 0) + (uint32_t)__popc(bal & lanemask_lt()));
        const float d = tile_depth(tx, ty, inc.tw, inc.th, b1.x, b1.y, b1.z, b1.w, b0.w);
        if (keep && pos < n_cap) dst[pos] = ((uint64_t)__float_as_uint(d) << 32) | g;
    }
    __syncthreads();
    const int kept = (int)*s_count;
    const uint2 re = inc.enter_ranges[tile];
    const int ne = (int)(re.y - re.x);
    for (int i = threadIdx.x; i < ne; i += NT)
        if (kept + i < n_cap) dst[kept + i] = inc.enter_keys[re.x + i];
    return kept + ne;
}

// Shared memory of sort_tile.
template <int NT>
struct SegShared {
    uint64_t* keys;     // seg_cap (padded for the merge sort)
    uint32_t* start;    // seg_buckets + 1 at most
    uint32_t* sample;   // kSegments
    uint32_t* split;    // kSegments
    float* scale;       // kSegments
    __device__ explicit SegShared(uint64_t* p, int cap = seg_cap<NT>()) {
        keys = p;
        start = reinterpret_cast<uint32_t*>(p + cap + cap / 16);
        sample = start + seg_buckets<NT>() + 4;
        split = sample + kSegments;
        scale = reinterpret_cast<float*>(split + kSegments);
    }
};

// Nearly sorted keys: passes over s[0..n) in blocks of kFixBlock, each sorted
// by one thread in registers when it is out of order, the blocks of every
// other pass shifted by half of one.  Every neighbouring pair lies inside a
// block of one of the two alignments, so the list is sorted once a pass after
// the first changed nothing (the pass before left the other alignment's
// blocks sorted).  Returns false (uniformly) when the passes run out first.
template <int NT>
__device__ bool block_fix(uint64_t* s, int n) {
    for (int pass = 0; pass < kFixMaxPasses; ++pass) {
        bool changed = false;
        const int off = (pass & 1) ? kFixBlock / 2 : 0;
        for (int i0 = off + kFixBlock * (int)threadIdx.x; i0 < n; i0 += kFixBlock * NT) {
            uint64_t k[kFixBlock];
            bool sorted = true;
#pragma unroll
            for (int j = 0; j < kFixBlock; ++j) k[j] = i0 + j < n ? s[spad(i0 + j)] : kKeyInf;
#pragma unroll
            for (int j = 0; j + 1 < kFixBlock; ++j) sorted = sorted && k[j] <= k[j + 1];
            if (!sorted) {
                sort_items(k);
#pragma unroll
                for (int j = 0; j < kFixBlock; ++j)
                    if (i0 + j < n) s[spad(i0 + j)] = k[j];
                changed = true;
            }
        }
        if (!__syncthreads_or(changed) && pass > 0) return true;
    }
    return false;
}

// Where a tile's keys come from: its bucket (full mode), its previous list and
// the entering instances (incremental), or the start of the CTA's own key
// buffer (a range of a large tile).
enum SegSource { kSrcBucket = 0, kSrcList = 1, kSrcShared = 2 };

// Sort the n keys of a tile (or of a range of one) that has at most ITEMS * NT
// source entries and write its indices from vals[dst0] on.  Thread t holds
// entries t, t + NT, ..., so neighbouring lanes read, and mostly write,
// neighbouring entries; an entering instance is one more key of the first
// threads.
template <int NT, int ITEMS, int SOURCE>
__device__ void sort_tile(const SegShared<NT>& sh, uint32_t* s_red, uint32_t tile, uint32_t dst0, int n, int n_src,
                          uint32_t src0, const uint64_t* __restrict__ comp, uint32_t* __restrict__ vals,
                          DevStatus* st, const SegSortIncr& inc) {
    constexpr int B = seg_buckets<NT>(), SUB = B / kSegments, PER = B / NT;
    constexpr int kStep = ITEMS % 4 == 0 ? 4 : (ITEMS % 3 == 0 ? 3 : 2);  // gathers in flight per thread
    static_assert(ITEMS % kStep == 0, "whole steps");
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    uint32_t dk[ITEMS], gk[ITEMS];  // depth bits and index of each key; index 0xffffffff: no key
    uint32_t* raw = reinterpret_cast<uint32_t*>(sh.keys);  // depth bits by source entry, until the keys are placed
    uint32_t ed = 0, eg = 0xffffffffu;  // the entering instance
    int ne = 0;
    if constexpr (SOURCE == kSrcList) {
        const int tx = (int)(tile % (uint32_t)inc.ntx), ty = (int)(tile / (uint32_t)inc.ntx);
        const uint2 re = inc.enter_ranges[tile];
        ne = (int)(re.y - re.x);
        if (t < ne && ne <= NT) {
            const uint64_t k = inc.enter_keys[re.x + t];
            ed = (uint32_t)(k >> 32);
            eg = (uint32_t)k;
        }
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            gk[q] = q * NT + t < n_src ? inc.vals_prev[src0 + q * NT + t] : 0xffffffffu;
            dk[q] = 0xffffffffu;
        }
#pragma unroll
        for (int q0 = 0; q0 < ITEMS; q0 += kStep) {
            if (q0 * NT < n_src) {
                uint4 b0[kStep];
                float4 b1[kStep];
#pragma unroll
                for (int j = 0; j < kStep; ++j) {
                    // both halves of the 32-byte record at once: one dependent step
                    b0[j] = make_uint4(0, 0, 0, 0);
                    b1[j] = make_float4(0, 0, 0, 0);
                    if (gk[q0 + j] < inc.n_gauss) {
                        b0[j] = inc.bins[gk[q0 + j]].r;
                        b1[j] = inc.bins[gk[q0 + j]].p;
                    }
                }
#pragma unroll
                for (int j = 0; j < kStep; ++j) {
                    const int q = q0 + j;
                    if (gk[q] < inc.n_gauss && rect_contains(b0[j], tx, ty))
                        dk[q] = __float_as_uint(tile_depth(tx, ty, inc.tw, inc.th, b1[j].x, b1[j].y, b1[j].z, b1[j].w,
                                                           b0[j].w));
                    else
                        gk[q] = 0xffffffffu;  // left the tile
                    if (q * NT + t < n_src) raw[q * NT + t] = dk[q];
                }
            }
        }
        if (ne == 0 && n == n_src) {
            // nothing left or entered (else the count would differ): in order still, or nearly
            __syncthreads();
            bool desc = false;
#pragma unroll
            for (int q = 0; q < ITEMS; ++q) {
                const int i = q * NT + t;
                if (i + 1 < n) desc = desc || raw[i + 1] <= dk[q];
            }
            const int n_desc = __syncthreads_count(desc);
            if (n_desc <= kFixMaxDescents) {
                if (n_desc) {
#pragma unroll
                    for (int q = 0; q < ITEMS; ++q)
                        if (q * NT + t < n) sh.keys[spad(q * NT + t)] = ((uint64_t)dk[q] << 32) | gk[q];
                    __syncthreads();
                }
                if (!n_desc || block_fix<NT>(sh.keys, n)) {
#pragma unroll
                    for (int q = 0; q < ITEMS; ++q) {
                        const int i = q * NT + t;
                        if (i < n) vals[dst0 + i] = n_desc ? (uint32_t)sh.keys[spad(i)] : gk[q];
                    }
                    return;
                }
                __syncthreads();
#pragma unroll
                for (int q = 0; q < ITEMS; ++q)
                    if (q * NT + t < n) raw[q * NT + t] = dk[q];
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const int i = q * NT + t;
            uint64_t k = kKeyInf;
            if (i < n_src) k = SOURCE == kSrcShared ? sh.keys[i] : comp[src0 + i];
            dk[q] = (uint32_t)(k >> 32);
            gk[q] = (uint32_t)k;
        }
        if (SOURCE == kSrcShared) __syncthreads();
#pragma unroll
        for (int q = 0; q < ITEMS; ++q)
            if (q * NT + t < n_src) raw[q * NT + t] = dk[q];
    }
    for (int b = t; b < B + 1; b += NT) sh.start[b] = 0;
    // the keys' range: the first segment's start and the last one's end
    uint32_t klo = 0xffffffffu, khi = 0;
#pragma unroll
    for (int q = 0; q < ITEMS; ++q)
        if (gk[q] != 0xffffffffu) {
            klo = min(klo, dk[q]);
            khi = max(khi, dk[q]);
        }
    if (eg != 0xffffffffu) {
        klo = min(klo, ed);
        khi = max(khi, ed);
    }
    klo = __reduce_min_sync(kFullMask, klo);
    khi = __reduce_max_sync(kFullMask, khi);
    if (lane == 0) {
        s_red[w] = klo;
        s_red[NT / 32 + w] = khi;
    }
    __syncthreads();
    klo = __reduce_min_sync(kFullMask, lane < NT / 32 ? s_red[lane] : 0xffffffffu);
    khi = __reduce_max_sync(kFullMask, lane < NT / 32 ? s_red[NT / 32 + lane] : 0u);
    // splitters: up to kSegments - 1 of the source entries, ranked by counting
    const int ns = min(n_src, kSegments - 1);
    if (t < kSegments) {
        sh.sample[t] = t < ns ? raw[(int)(((int64_t)t * n_src) / ns)] : 0xffffffffu;
        sh.split[t] = 0xffffffffu;
    }
    __syncthreads();
    if (t < ns) {
        const uint32_t d = sh.sample[t];
        int rank = 0;
        for (int k = 0; k < ns; ++k) {
            const uint32_t o = sh.sample[k];
            rank += (o < d || (o == d && k < t)) ? 1 : 0;
        }
        sh.split[rank] = d;
    }
    __syncthreads();
    if (t < kSegments) {
        // segment t: [split[t - 1], split[t]), within [klo, khi]
        const uint32_t lo = t ? sh.split[t - 1] : klo, hi = min(sh.split[t], khi);
        sh.scale[t] = hi > lo ? (float)SUB / (float)(hi - lo) : 0.0f;
    }
    __syncthreads();
    // a key's bucket, increasing with its depth bits, and its slot there
    auto place = [&](uint32_t d) -> uint32_t {
        int seg = 0;  // splitters at or below d
#pragma unroll
        for (int h = kSegments / 2; h > 0; h >>= 1)
            if (sh.split[seg + h - 1] <= d) seg += h;
        const uint32_t lo = seg ? sh.split[seg - 1] : klo;
        const int sub = min(SUB - 1, (int)((float)(d - lo) * sh.scale[seg]));
        const uint32_t b = (uint32_t)(seg * SUB + sub);
        return b | (atomicAdd(&sh.start[b], 1u) << 12);
    };
    static_assert(B <= 4096, "bucket number in 12 bits");
    uint32_t br[ITEMS], ebr = 0;
#pragma unroll
    for (int q = 0; q < ITEMS; ++q)
        if (gk[q] != 0xffffffffu) br[q] = place(dk[q]);
    if (eg != 0xffffffffu) ebr = place(ed);
    __syncthreads();
    // bucket starts, the largest bucket and the number of keys
    uint32_t c[PER], sum = 0, top = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        c[k] = sh.start[t * PER + k];
        sum += c[k];
        top = max(top, c[k]);
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += y;
    }
    top = __reduce_max_sync(kFullMask, top);
    if (lane == 31) s_red[w] = incl;
    if (lane == 0) s_red[NT / 32 + w] = top;
    __syncthreads();
    const uint32_t wsum = lane < NT / 32 ? s_red[lane] : 0u;
    const uint32_t wtop = lane < NT / 32 ? s_red[NT / 32 + lane] : 0u;
    uint32_t run = __reduce_add_sync(kFullMask, lane < w ? wsum : 0u) + incl - sum;
    const uint32_t total = __reduce_add_sync(kFullMask, wsum);
    top = __reduce_max_sync(kFullMask, wtop);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        sh.start[t * PER + k] = run;
        run += c[k];
    }
    if (t == NT - 1) sh.start[B] = total;
    if (ne > NT || top > (uint32_t)kMaxBucket) {
        // keys piled up (equal depths), or a tile of entering instances: merge sort
        __syncthreads();
        if (t == 0) s_red[0] = 0;
        __syncthreads();
        auto put = [&](uint32_t d, uint32_t g) {
            const uint32_t pos = atomicAdd(&s_red[0], 1u);
            if (pos < (uint32_t)n) sh.keys[spad((int)pos)] = ((uint64_t)d << 32) | g;
        };
#pragma unroll
        for (int q = 0; q < ITEMS; ++q)
            if (gk[q] != 0xffffffffu) put(dk[q], gk[q]);
        if constexpr (SOURCE == kSrcList) {
            const uint2 re = inc.enter_ranges[tile];
            for (int i = t; i < ne; i += NT) {
                const uint64_t k = inc.enter_keys[re.x + i];
                put((uint32_t)(k >> 32), (uint32_t)k);
            }
        }
        __syncthreads();
        const uint32_t got = s_red[0];
        if (got != (uint32_t)n) {
            if (t == 0) atomicOr(&st->flags, kErrBounds);
            return;
        }
        const int m = (n + kSegItems - 1) / kSegItems * kSegItems;
        if (t < m - n) sh.keys[spad(n + t)] = kKeyInf;
        __syncthreads();
        if (m <= NT * kSmallItems)
            block_merge_sort<kSmallItems>(sh.keys, (n + kSmallItems - 1) / kSmallItems * kSmallItems);
        else
            block_merge_sort<kSegItems>(sh.keys, m);
        for (int i = t; i < n; i += NT) write_sorted(sh.keys[spad(i)], dst0 + i, vals);
        return;
    }
    if (total != (uint32_t)n) {
        if (t == 0) atomicOr(&st->flags, kErrBounds);
        return;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ITEMS; ++q)
        if (gk[q] != 0xffffffffu)
            sh.keys[sh.start[br[q] & 0xfffu] + (br[q] >> 12)] = ((uint64_t)dk[q] << 32) | gk[q];
    if (eg != 0xffffffffu) sh.keys[sh.start[ebr & 0xfffu] + (ebr >> 12)] = ((uint64_t)ed << 32) | eg;
    __syncthreads();
    auto write = [&](uint32_t d, uint32_t g, uint32_t b) {
        const uint32_t b0 = sh.start[b], b1 = sh.start[b + 1];
        uint32_t pos = b0;
        if (b1 - b0 > 1) {
            const uint64_t key = ((uint64_t)d << 32) | g;
            for (uint32_t k = b0; k < b1; ++k) pos += sh.keys[k] < key ? 1u : 0u;
        }
        vals[dst0 + pos] = g;
    };
#pragma unroll
    for (int q = 0; q < ITEMS; ++q)
        if (gk[q] != 0xffffffffu) write(dk[q], gk[q], br[q] & 0xfffu);
    if (eg != 0xffffffffu) write(ed, eg, ebr & 0xfffu);
}

// Entries of a tile's source list: its previous sorted list (incremental) or
// its bucket.  Returns their number; src0: the first one.
__device__ __forceinline__ int tile_source(uint32_t tile, uint2 r, bool incr, const SegSortIncr& inc, uint32_t& src0) {
    if (!incr) {
        src0 = r.x;
        return (int)(r.y - r.x);
    }
    uint2 ro = inc.ranges_prev[tile];
    ro.y = (uint32_t)min((uint64_t)ro.y, inc.capacity);
    src0 = ro.x;
    return ro.y > ro.x ? (int)(ro.y - ro.x) : 0;
}

template <int NT, int SOURCE>
__device__ __forceinline__ void sort_tile_any(const SegShared<NT>& sh, uint32_t* s_red, uint32_t tile, uint32_t dst0,
                                              int n, int n_src, uint32_t src0, const uint64_t* __restrict__ comp,
                                              uint32_t* __restrict__ vals, DevStatus* st, const SegSortIncr& inc) {
    if (n_src <= 2 * NT)
        sort_tile<NT, 2, SOURCE>(sh, s_red, tile, dst0, n, n_src, src0, comp, vals, st, inc);
    else if (n_src <= 4 * NT)
        sort_tile<NT, 4, SOURCE>(sh, s_red, tile, dst0, n, n_src, src0, comp, vals, st, inc);
    else if (n_src <= 6 * NT)
        sort_tile<NT, 6, SOURCE>(sh, s_red, tile, dst0, n, n_src, src0, comp, vals, st, inc);
    else if (n_src <= 8 * NT)
        sort_tile<NT, 8, SOURCE>(sh, s_red, tile, dst0, n, n_src, src0, comp, vals, st, inc);
    else
        sort_tile<NT, 16, SOURCE>(sh, s_red, tile, dst0, n, n_src, src0, comp, vals, st, inc);
}

// cap: the most keys of a tile (the launch's shared memory); part: part_keys of
// the large tiles' kernel that follows.
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) segsort_kernel(const uint64_t* __restrict__ comp,
                                                                const uint2* __restrict__ ranges, uint32_t* vals,
                                                                SegSortWork w, DevStatus* st, int cap, int part,
                                                                SegSortIncr inc) {
    pdl_begin();
    extern __shared__ uint64_t s_keys[];
    __shared__ uint32_t s_red[2 * NT / 32];
    if (st->flags & kErrOverflow) return;
    const bool incr = st->mode == kBinIncremental;
    const uint32_t tile = blockIdx.x;
    const uint2 r = ranges[tile];
    const int n = (int)(r.y - r.x);
    if (n <= 0) return;
    uint32_t src0;
    const int n_src = tile_source(tile, r, incr, inc, src0);
    if (max(n, n_src) > cap) {
        // listed whole, or range by range
        const bool whole = max(n, n_src) <= 2 * part || n >= kGlobalMin;
        const uint32_t parts = whole ? 1u : (uint32_t)(n / part + 1);
        if (threadIdx.x == 0) s_red[0] = atomicAdd(&w.large_ctrl[0], parts);
        __syncthreads();
        for (uint32_t p = threadIdx.x; p < parts; p += NT) w.large_list[s_red[0] + p] = make_uint2(tile, p);
        return;
    }
    const SegShared<NT> sh(s_keys, cap);
    if (incr)
        sort_tile_any<NT, kSrcList>(sh, s_red, tile, r.x, n, n_src, src0, comp, vals, st, inc);
    else
        sort_tile_any<NT, kSrcBucket>(sh, s_red, tile, r.x, n, n_src, src0, comp, vals, st, inc);
}

// Key i of a large tile's source entries (the previous list, then the entering
// instances; or the bucket); false: no longer in the tile.
__device__ __forceinline__ bool source_key(const SegSortIncr& inc, const uint64_t* __restrict__ comp, bool incr,
                                           uint32_t src0, int n_src, uint32_t enter0, int tx, int ty, int i,
                                           uint64_t& key) {
    if (!incr) {
        key = comp[src0 + i];
        return true;
    }
    if (i >= n_src) {
        key = inc.enter_keys[enter0 + (i - n_src)];
        return true;
    }
    const uint32_t g = inc.vals_prev[src0 + i];
    if (g >= inc.n_gauss) return false;
    const uint4 b0 = inc.bins[g].r;
    const float4 b1 = inc.bins[g].p;
    key = ((uint64_t)__float_as_uint(tile_depth(tx, ty, inc.tw, inc.th, b1.x, b1.y, b1.z, b1.w, b0.w)) << 32) | g;
    return rect_contains(b0, tx, ty);
}

// A tile's cut number `part`: a key with at most part * kPart keys of the tile
// below it and fewer than kPart between it and that rank (`below`: the keys below
// the cut).  The keys' bits are followed from the top, 12 a pass, into the bin
// that holds the rank, until a bin holds at most kPart keys; its start is the cut.
// The bins of two cuts are the same or apart, so cuts come in order, and keys
// are unique, so the last bits leave one.  Whatever the keys and their order, two
// neighbouring cuts enclose fewer than 2 kPart keys.  hist: kPartSamples + 4 words.
// What bounds it: two to five more readings of the list for each of a range's
// two cuts.  One tile of 65,536 entries, carried over: 279 us of sort, where the
// samples serve 149; the binning repeated in full instead took 271 and could
// fail again.
template <int NT>
__device__ __noinline__ uint64_t rank_cut(uint32_t* hist, uint32_t* s_red, uint32_t part, int n, const uint64_t* comp,
                                          bool incr, const SegSortIncr& inc, uint32_t src0, int n_src, uint32_t enter0,
                                          int n_all, int tx, int ty, uint32_t& below) {
    constexpr int S = kPartSamples, PER = S / NT, kBits = 12;
    static_assert(S == 1 << kBits, "a counter per value of the bits of a pass");
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const uint32_t kPart = part_keys<NT>(), rank = part * kPart;
    uint32_t* bin = hist + S;  // [0] the bin, [1] keys below it, [2] keys in it
    uint64_t prefix = 0;       // the bin so far: keys with these bits above `shift`
    uint32_t count = (uint32_t)n;
    int shift = 64;
    below = 0;
    while (count > kPart && shift > 0) {
        const int bits = min(kBits, shift), down = shift - bits;
        for (int k = t; k < S; k += NT) hist[k] = 0;
        __syncthreads();
        for (int i = t; i < n_all; i += NT) {
            uint64_t key;
            if (source_key(inc, comp, incr, src0, n_src, enter0, tx, ty, i, key) &&
                (shift == 64 || key >> shift == prefix))
                atomicAdd(&hist[(uint32_t)(key >> down) & ((1u << bits) - 1u)], 1u);
        }
        __syncthreads();
        uint32_t sum = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) sum += hist[t * PER + k];
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_red[w] = incl;
        __syncthreads();
        uint32_t run = below + incl - sum;
        for (int k = 0; k < w; ++k) run += s_red[k];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const uint32_t c = hist[t * PER + k];
            if (rank >= run && rank - run < c) {
                bin[0] = (uint32_t)(t * PER + k);
                bin[1] = run;
                bin[2] = c;
            }
            run += c;
        }
        __syncthreads();
        prefix = prefix << bits | bin[0];
        below = bin[1];
        count = bin[2];
        shift = down;
        __syncthreads();  // the bin is read before the next pass writes it
    }
    return shift == 64 ? 0ull : prefix << shift;
}

// Range `part` of a large tile.  Every CTA of the tile samples and counts
// alike: kPartSamples source keys in order are the splitters, the exact counts
// between them give each segment's start, and range p holds the segments that
// start in [p, p + 1) kPart.  The samples stand at even places of the source
// list, so where its order repeats with their distance (layers that alternate
// from Gaussian to Gaussian) they miss most of the keys; a tile with a segment
// above kPart keys is cut by rank instead.
template <int NT>
__device__ void sort_part(uint64_t* s_keys, uint32_t* s_red, uint32_t tile, uint32_t part, uint2 r, bool incr,
                          const uint64_t* __restrict__ comp, uint32_t* __restrict__ vals, DevStatus* st,
                          const SegSortIncr& inc) {
    constexpr int S = kPartSamples, PER = S / NT, kPart = part_keys<NT>();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int n = (int)(r.y - r.x);
    uint32_t* hist = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(s_keys) + seg_smem<NT>());
    const int tx = (int)(tile % (uint32_t)inc.ntx), ty = (int)(tile / (uint32_t)inc.ntx);
    uint32_t src0, enter0 = 0;
    const int n_src = tile_source(tile, r, incr, inc, src0);
    int ne = 0;
    if (incr) {
        const uint2 re = inc.enter_ranges[tile];
        enter0 = re.x;
        ne = (int)(re.y - re.x);
    }
    const int n_all = n_src + ne;
    for (int k = t; k < S; k += NT) {
        uint64_t key = kKeyInf;
        if (!source_key(inc, comp, incr, src0, n_src, enter0, tx, ty, (int)(((int64_t)k * n_all) / S), key))
            key = kKeyInf;
        s_keys[spad(k)] = key;
        hist[k] = 0;
    }
    __syncthreads();
    block_merge_sort<PER>(s_keys, S);
    // pass over all keys: their number in each segment [sample k - 1, sample k); the last sample ends none
    for (int i0 = 0; i0 < n_all; i0 += 4 * NT) {
        uint64_t key[4];
        bool ok[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j * NT + t;
            ok[j] = i < n_all && source_key(inc, comp, incr, src0, n_src, enter0, tx, ty, i, key[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (ok[j]) {
                int seg = 0;  // samples at or below the key, the last one left out
#pragma unroll
                for (int h = S / 2; h > 0; h >>= 1)
                    if (s_keys[spad(seg + h - 1)] <= key[j]) seg += h;
                atomicAdd(&hist[seg], 1u);
            }
    }
    __syncthreads();
    uint32_t c[PER], sum = 0, top = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        c[k] = hist[t * PER + k];
        sum += c[k];
        top = max(top, c[k]);
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += y;
    }
    top = __reduce_max_sync(kFullMask, top);
    if (lane == 31) s_red[w] = incl;
    if (lane == 0) s_red[NT / 32 + w] = top;
    __syncthreads();
    const uint32_t wsum = lane < NT / 32 ? s_red[lane] : 0u;
    const uint32_t total = __reduce_add_sync(kFullMask, wsum);
    top = __reduce_max_sync(kFullMask, lane < NT / 32 ? s_red[NT / 32 + lane] : 0u);
    if (total != (uint32_t)n) {
        if (t == 0) atomicOr(&st->flags, kErrBounds);
        return;
    }
    uint32_t* first = hist + S;  // [0] first segment, [1] end segment, [2] first place, [3] keys collected
    uint32_t below;              // the range's keys: lo <= key < hi (open: no end), the first one's place
    uint64_t lo, hi = 0;
    bool open;
    if (top > (uint32_t)kPart) {
        if (part * (uint32_t)kPart >= (uint32_t)n) return;
        lo = rank_cut<NT>(hist, s_red, part, n, comp, incr, inc, src0, n_src, enter0, n_all, tx, ty, below);
        open = (part + 1) * (uint32_t)kPart >= (uint32_t)n;
        if (!open) {
            uint32_t next;
            hi = rank_cut<NT>(hist, s_red, part + 1, n, comp, incr, inc, src0, n_src, enter0, n_all, tx, ty, next);
        }
        if (t == 0) first[3] = 0;
    } else {
        // the range's first segment, its end and its first key's place
        uint32_t run = __reduce_add_sync(kFullMask, lane < w ? wsum : 0u) + incl - sum;
        __syncthreads();
        if (t == 0) {
            first[0] = S;
            first[1] = 0;
            first[2] = 0xffffffffu;
            first[3] = 0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (c[k] && run / kPart == part) {
                atomicMin(&first[0], (uint32_t)(t * PER + k));
                atomicMax(&first[1], (uint32_t)(t * PER + k + 1));
                atomicMin(&first[2], run);
            }
            run += c[k];
        }
        __syncthreads();
        const uint32_t s0 = first[0], s1 = first[1];
        if (s1 == 0) return;  // no segment starts in this range
        below = first[2];
        lo = s0 ? s_keys[spad((int)s0 - 1)] : 0ull;
        open = s1 >= (uint32_t)S;
        if (!open) hi = s_keys[spad((int)s1 - 1)];
    }
    __syncthreads();  // the samples make room for the keys
    for (int i0 = 0; i0 < n_all; i0 += 4 * NT) {
        uint64_t key[4];
        bool ok[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = i0 + j * NT + t;
            ok[j] = i < n_all && source_key(inc, comp, incr, src0, n_src, enter0, tx, ty, i, key[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool in = ok[j] && key[j] >= lo && (open || key[j] < hi);
            const uint32_t bal = __ballot_sync(kFullMask, in);
            uint32_t slot = 0;
            if (lane == 0 && bal) slot = atomicAdd(&first[3], (uint32_t)__popc(bal));
            slot = __shfl_sync(kFullMask, slot, 0) + (uint32_t)__popc(bal & lanemask_lt());
            if (in && slot < (uint32_t)seg_cap<NT>()) s_keys[slot] = key[j];
        }
    }
    __syncthreads();
    const int cnt = (int)first[3];
    if (cnt > seg_cap<NT>()) {  // a range holds below 2 kPart keys unless the lists do not agree
        if (t == 0) atomicOr(&st->flags, kErrBounds);
        return;
    }
    sort_tile<NT, kSegItems, kSrcShared>(SegShared<NT>(s_keys), s_red, tile, r.x + below, cnt, cnt, 0, comp, vals, st,
                                         inc);
}

// Large tiles: persistent CTAs take listed tiles and ranges.  From kGlobalMin
// on a tile is one item: chunks of shared memory's capacity sorted into tmp, then runs
// merged through global memory (every thread merges kSegItems outputs after
// its own merge-path search).
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) segsort_large_kernel(uint64_t* comp, uint64_t* tmp,
                                                                      const uint2* __restrict__ ranges, uint32_t* vals,
                                                                      SegSortWork w, DevStatus* st,
                                                                      const __grid_constant__ SegSortIncr inc) {
    // One CTA an SM with most of its registers, and usually no tile listed: let in
    // early, the blending kernel crowded onto the SMs that were left first.  Late
    // / early, us: frame of 50 k Gaussians VGA 2838 / 3124, of 1 M HD 3315 / 3395,
    // view of 75 k at 160x120 129 / 161.
    pdl_begin_late();
    constexpr int kCap = seg_cap<NT>();
    extern __shared__ uint64_t s_keys[];
    __shared__ uint32_t s_red[2 * NT / 32];
    __shared__ uint32_t s_idx;
    uint64_t* s = s_keys;
    if (st->flags & kErrOverflow) return;
    const bool incr = st->mode == kBinIncremental;
    for (;;) {
        if (threadIdx.x == 0) s_idx = atomicAdd(&w.large_ctrl[1], 1u);
        __syncthreads();
        const uint32_t idx = s_idx;
        __syncthreads();
        if (idx >= w.large_ctrl[0]) return;
        const uint32_t tile = w.large_list[idx].x;
        const uint2 r = ranges[tile];
        const int n = (int)(r.y - r.x);
        uint32_t src0;
        const int n_src = tile_source(tile, r, incr, inc, src0);
        if (max(n, n_src) <= kCap) {
            const SegShared<NT> sh(s_keys);
            if (incr)
                sort_tile<NT, kSegItems, kSrcList>(sh, s_red, tile, r.x, n, n_src, src0, comp, vals, st, inc);
            else
                sort_tile<NT, kSegItems, kSrcBucket>(sh, s_red, tile, r.x, n, n_src, src0, comp, vals, st, inc);
            __syncthreads();
            continue;
        }
        if (n < kGlobalMin) {
            sort_part<NT>(s_keys, s_red, tile, w.large_list[idx].y, r, incr, comp, vals, st, inc);
            __syncthreads();
            continue;
        }
        if (incr) {
            const int got = gather_tile<NT>(comp + r.x, tile, n, inc, s_red);
            if (got != n && threadIdx.x == 0) atomicOr(&st->flags, kErrBounds);
            __syncthreads();
        }
        uint64_t* src = tmp + r.x;
        uint64_t* dst = comp + r.x;
        // sorted chunks of kCap into src
        for (int c0 = 0; c0 < n; c0 += kCap) {
            const int cn = min(kCap, n - c0);
            for (int i = threadIdx.x; i < kCap; i += NT) s[spad(i)] = i < cn ? comp[r.x + c0 + i] : kKeyInf;
            __syncthreads();
            block_merge_sort(s, kCap);
            for (int i = threadIdx.x; i < cn; i += NT) src[c0 + i] = s[spad(i)];
            __syncthreads();
        }
        // merge passes src -> dst, runs of L doubling
        for (int L = kCap; L < n; L <<= 1) {
            for (int o = threadIdx.x * kSegItems; o < n; o += NT * kSegItems) {
                const int ps = (o / (2 * L)) * 2 * L;
                const int d = o - ps;
                const int la = min(L, n - ps);
                const int lb = max(0, min(L, n - ps - L));
                const uint64_t* A = src + ps;
                const uint64_t* B = src + ps + la;
                int lo = max(0, d - lb), hi = min(d, la);
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (A[mid] <= B[d - 1 - mid])
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                int ai = lo, bj = d - lo;
                const int outn = min(kSegItems, la + lb - d);
                for (int q = 0; q < outn; ++q) {
                    const uint64_t a = ai < la ? A[ai] : kKeyInf;
                    const uint64_t b = bj < lb ? B[bj] : kKeyInf;
                    const bool ta = a <= b;
                    dst[ps + d + q] = ta ? a : b;
                    ai += ta ? 1 : 0;
                    bj += ta ? 0 : 1;
                }
            }
            __syncthreads();
            uint64_t* tsw = src;
            src = dst;
            dst = tsw;
        }
        for (int i = threadIdx.x; i < n; i += NT) write_sorted(src[i], r.x + i, vals);
        __syncthreads();
    }
}

cudaError_t segsort_configure_device() {
    const std::pair<const void*, size_t> k[] = {
        {reinterpret_cast<const void*>(segsort_kernel<kShortThreads>), seg_smem<kShortThreads>()},
        {reinterpret_cast<const void*>(segsort_kernel<kSegThreads>), seg_smem<kSegThreads>()},
        {reinterpret_cast<const void*>(segsort_large_kernel<kSegThreads>), large_smem<kSegThreads>()},
        {reinterpret_cast<const void*>(segsort_large_kernel<kLargeThreads>), large_smem<kLargeThreads>()}};
    for (const auto& f : k) {
        const cudaError_t e = cudaFuncSetAttribute(f.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.second);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

size_t segsort_list_items(uint64_t max_instances, int num_tiles) {
    return (size_t)(max_instances / part_keys<kSegThreads>()) + (size_t)num_tiles;
}

cudaError_t launch_segsort(uint64_t* comp, uint64_t* tmp, const uint2* ranges, int num_tiles, uint32_t* vals,
                           SegSortWork w, const DevStatus* st, uint32_t n_hint, int num_sms, const SegSortIncr& inc,
                           cudaStream_t s) {
    if (num_tiles <= 0) return cudaSuccess;
    // the list counters were zeroed by the tile-offsets kernel of this binning
    const uint32_t mean = n_hint ? n_hint / (uint32_t)num_tiles : 0xffffffffu;
    const bool brief = mean <= kBriefMean;
    const int part = brief ? part_keys<kSegThreads>() : part_keys<kLargeThreads>();
    cudaError_t e;
    if (mean <= kShortMean) {
        constexpr int NT = kShortThreads, cap = seg_cap<NT>() / 2;
        e = launch_chained(segsort_kernel<NT>, dim3(num_tiles), dim3(NT), seg_smem<NT>(cap), s, comp, ranges, vals, w,
                           const_cast<DevStatus*>(st), cap, part, inc);
    } else {
        constexpr int NT = kSegThreads;
        const int cap = brief ? seg_cap<NT>() / 2 : seg_cap<NT>();
        e = launch_chained(segsort_kernel<NT>, dim3(num_tiles), dim3(NT), seg_smem<NT>(cap), s, comp, ranges, vals, w,
                           const_cast<DevStatus*>(st), cap, part, inc);
    }
    if (e != cudaSuccess) return e;
    if (brief)
        return launch_chained(segsort_large_kernel<kSegThreads>, dim3(num_sms), dim3(kSegThreads),
                              large_smem<kSegThreads>(), s, comp, tmp, ranges, vals, w, const_cast<DevStatus*>(st), inc);
    return launch_chained(segsort_large_kernel<kLargeThreads>, dim3(num_sms), dim3(kLargeThreads),
                          large_smem<kLargeThreads>(), s, comp, tmp, ranges, vals, w, const_cast<DevStatus*>(st), inc);
}

// One CTA per tile: key = tile << 32 | bits of the tile-centre depth of the
// Gaussian at each sorted position.
__global__ void __launch_bounds__(256) make_keys_kernel(const BinRec* __restrict__ bins,
                                                        const uint2* __restrict__ ranges,
                                                        const uint32_t* __restrict__ vals, uint32_t n_gauss, int ntx,
                                                        int tw, int th, const DevStatus* st, uint64_t* keys) {
    pdl_begin();
    if (st->flags & kErrOverflow) return;
    const uint32_t tile = blockIdx.x;
    const uint2 r = ranges[tile];
    const int tx = (int)(tile % (uint32_t)ntx), ty = (int)(tile / (uint32_t)ntx);
    for (uint32_t i = r.x + threadIdx.x; i < r.y; i += blockDim.x) {
        const uint32_t g = vals[i];
        if (g >= n_gauss) continue;
        const BinRec b = bins[g];
        const float d = tile_depth(tx, ty, tw, th, b.p.x, b.p.y, b.p.z, b.p.w, b.r.w);
        keys[i] = ((uint64_t)tile << 32) | __float_as_uint(d);
    }
}

cudaError_t launch_make_keys(const BinRec* bins, const uint2* ranges, const uint32_t* vals, uint32_t n_gauss,
                             int num_tiles, int ntx, int tw, int th, const DevStatus* st, uint64_t* keys,
                             cudaStream_t s) {
    if (num_tiles <= 0) return cudaSuccess;
    return launch_chained(make_keys_kernel, dim3(num_tiles), dim3(256), 0, s, bins, ranges, vals, n_gauss, ntx, tw,
                          th, st, keys);
}

}  // namespace fvgs
