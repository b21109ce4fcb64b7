// maintenance.cu -- map maintenance kernels for sm_103a: visibility and
// covisibility, outlier scores, prune marking, and stable compaction of the
// Gaussian planes.
//
// Reference: computeGaussiansVisibility_kernel, computeGaussiansCovisibility_
// kernel, pruneGaussians_kernel, computeOutliers_kernel and removeOutliers_
// kernel (src/GSCudaKernels.cu:1455-1739), driven by GSSlam::removeOutliers,
// GSSlam::prune and GSSlam::computeCovisibilityRatio (src/GSSlam.cu:1467-1904), which
// remove the marked Gaussians with thrust::sort_by_key on the 0 / 0xff states
// (survivors first, in order) and shrink the Gaussian count.
//
// Every blending kernel here reads the packed records of the binning (u,
// v, z, opacity; c.x, c.y, c.z, phat.x; phat.y, rgb; ...), where
// c is the inverse 2D covariance in the order the reference's tracking
// kernels consume it (c.y as the xy term, c.z as the yy term).  The
// reference's visibility and outlier kernels read the stored inverse the same
// way, so the same record serves both.
//
// Layout choices:
//  * visibility: one CTA per 16x16 tile, one thread per pixel, as the
//    reference (a pixel's transmittance depends on the Gaussians before it);
//    a Gaussian's flag is written once per tile, from a shared hit mask,
//    instead of once per pixel;
//  * outlier scores: the reference adds every (pixel, Gaussian) contribution
//    with two global atomics.  Here a lane takes one Gaussian of the tile
//    list, sums its contributions over the tile's pixels in a fixed order and
//    adds the tile's totals with one atomic per accumulator: the same sums,
//    one global update per (tile, Gaussian);
//  * compaction: mark (state + survivors per block) -> one-CTA scan of the
//    block counts -> scatter into the session's second set of planes, after
//    which the host swaps the plane pointers.  The source planes are never
//    written, so an aborted pass leaves the map as it was.
#include <cfloat>

#include "track_tile.cuh"

namespace fvgs {

constexpr int kMPix = 256;  // 16 x 16 pixels per tile
constexpr int kOutWarps = 4;  // warps per tile of the outlier scores

struct OutlierEntry {
    float u, v, z, lo2;
    float ca, cb, cc, phx, phy;
    uint32_t g;
};

__global__ void __launch_bounds__(kMPix) visibility_kernel(VisArgs a) {
    pdl_begin();
    // alpha = min(0.99, o exp(-q/2)) as one ex2.approx of log2(o) + the
    // conic pre-scaled by -log2(e)/2 (the tracking kernels' weight)
    __shared__ float4 sA[kMPix];  // u, v, log2(opacity), c'.x
    __shared__ float2 sB[kMPix];  // 2 c'.y, c'.z
    __shared__ int sHit[kMPix];
    const int tile = blockIdx.x;
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    const int tid = threadIdx.x;
    const int x = tx * 16 + (tid & 15), y = ty * 16 + (tid >> 4);
    const bool inside = x < a.W && y < a.H;
    uint2 range = a.ranges[tile];
    range.y = min(range.y, a.n_list);
    int n = range.y > range.x ? (int)(range.y - range.x) : 0;
    if (a.cap > 0) n = min(n, a.cap);
    const float px = (float)x, py = (float)y;
    float T = 1.f;
    bool done = !inside;
    for (int base = 0; base < n; base += kMPix) {
        if (__syncthreads_and(done)) break;
        const int li = base + tid;
        uint32_t g = 0xffffffffu;
        if (li < n) {
            g = a.indices[range.x + li];
            float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
            if (g < a.n_gauss) {
                r0 = a.rec[kRecQuads * (size_t)g];
                r1 = a.rec[kRecQuads * (size_t)g + 1];
            }
            constexpr float kNegHalfLog2e = -0.72134752044448170368f;
            sA[tid] = make_float4(r0.x, r0.y, log2_opacity(r0.w), kNegHalfLog2e * r1.x);
            sB[tid] = make_float2(2.0f * kNegHalfLog2e * r1.y, kNegHalfLog2e * r1.z);
        }
        sHit[tid] = 0;
        __syncthreads();
        const int cnt = min(kMPix, n - base);
        for (int j = 0; j < cnt && !done; ++j) {
            const float4 gA = sA[j];
            const float2 gB = sB[j];
            const float dx = gA.x - px, dy = gA.y - py;
            const float t = __fmaf_rn(dx, __fmaf_rn(gA.w, dx, __fmul_rn(gB.x, dy)),
                                      __fmaf_rn(__fmul_rn(gB.y, dy), dy, gA.z));
            float w;
            asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(t));
            const float alpha = fminf(0.99f, w);
            if (alpha < 1.0f / 255.0f) continue;
            sHit[j] = 1;
            T *= 1.0f - alpha;
            if (T < 0.5f) done = true;
        }
        __syncthreads();
        if (li < n && g < a.n_gauss && sHit[tid]) a.vis[g] = 1;
    }
}

// The entry's sums over the tile's pixels in row-major order.  FULL: all 16
// columns lie inside the image, and the pixels go two at a time with packed
// FP32 instructions, each lane of which rounds as the scalar form does.
// FRONT: dr > 0 at every pixel, so the pair's test of it is left out.
template <bool FULL, bool FRONT>
__device__ __forceinline__ float2 outlier_sums(const OutlierEntry& g, const float* __restrict__ lim, int x0, int y0,
                                               int bw, int bh) {
    float ta = 0.f, to = 0.f;
    // predicated sums: as a branch or as selects the tests cost more issue
    // than the rest of the pair
    auto add = [&](float alpha, float dr, float l) {
        if constexpr (FRONT) {
            asm("{\n\t.reg .pred p, q;\n\t"
                "setp.geu.f32 p, %2, 0f3b808081;\n\t"  // !(alpha < 1/255)
                "setp.lt.and.f32 q, %3, %4, p;\n\t"
                "@p add.f32 %0, %0, %2;\n\t"
                "@q add.f32 %1, %1, %2;\n\t}"
                : "+f"(ta), "+f"(to)
                : "f"(alpha), "f"(dr), "f"(l));
        } else {
            asm("{\n\t.reg .pred p, q;\n\t"
                "setp.geu.f32 p, %2, 0f3b808081;\n\t"
                "setp.gtu.and.f32 p, %3, 0f00000000, p;\n\t"  // !(dr <= 0)
                "setp.lt.and.f32 q, %3, %4, p;\n\t"
                "@p add.f32 %0, %0, %2;\n\t"
                "@q add.f32 %1, %1, %2;\n\t}"
                : "+f"(ta), "+f"(to)
                : "f"(alpha), "f"(dr), "f"(l));
        }
    };
    auto row = [&](int yy, float& dr_row, float& b_row, float& q_row) {
        const float dy = (float)(y0 + yy) - g.v;
        q_row = g.cc * dy * dy;
        b_row = 2.0f * g.cb * dy;
        dr_row = g.z + g.phy * dy;
    };
    if constexpr (FULL) {
        float2 dx[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) dx[k] = make_float2((float)(x0 + 2 * k) - g.u, (float)(x0 + 2 * k + 1) - g.u);
        const float2 ca = make_float2(g.ca, g.ca), ph = make_float2(g.phx, g.phx), lo = make_float2(g.lo2, g.lo2);
        const float2 kq = make_float2(kGaussScale, kGaussScale);
#pragma unroll 1
        for (int yy = 0; yy < bh; ++yy) {
            float dr_row, b_row, q_row;
            row(yy, dr_row, b_row, q_row);
            const float2 cb = make_float2(b_row, b_row), cc = make_float2(q_row, q_row), z = make_float2(dr_row, dr_row);
#pragma unroll
            for (int k = 0; k < 8; k += 2) {
                const float4 l = *reinterpret_cast<const float4*>(lim + yy * 16 + 2 * k);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float2 d = dx[k + h];
                    const float2 e = __ffma2_rn(__ffma2_rn(__ffma2_rn(ca, d, cb), d, cc), kq, lo);
                    const float2 dr = __ffma2_rn(ph, d, z);
                    add(ex2_approx(e.x), dr.x, h ? l.z : l.x);
                    add(ex2_approx(e.y), dr.y, h ? l.w : l.y);
                }
            }
        }
    } else {
        for (int yy = 0; yy < bh; ++yy) {
            float dr_row, b_row, q_row;
            row(yy, dr_row, b_row, q_row);
            for (int xx = 0; xx < bw; ++xx) {
                const float dx = (float)(x0 + xx) - g.u;
                const float q = __fmaf_rn(__fmaf_rn(g.ca, dx, b_row), dx, q_row);
                add(gauss_weight(g.lo2, q), __fmaf_rn(g.phx, dx, dr_row), lim[yy * 16 + xx]);
            }
        }
    }
    return make_float2(ta, to);
}

// A CTA per tile, whose four warps each take every fourth 32 entries of the
// list.  A warp queues the entries that reach alpha 1/255 somewhere in the
// tile (block_reject) and, once 32 are waiting, gives every lane one, over the
// tile's pixels in the same order in all lanes (a pixel's depth is a
// shared-memory broadcast); an entry's sums go out with one atomic each.
//
// What bounds it: issue (78 % of it), 10 instructions a pair with two pixels
// packed; 80 registers and 24 warps instead of 96 and 20 per SM change nothing.
// 400 k Gaussians, 1280x720 (2.69 M entries, 61 % of the pairs reach 1/255):
// 199 us, before (256 entries per CTA of 256 threads, no queue, a pixel at a
// time) 344; the 8 x 8 quarters with a queue each 294 (they drop 69 instead of
// 78 % of the pairs, at four times the tests and with the quarters' sums met
// in shared memory).
__global__ void __launch_bounds__(32 * kOutWarps) outliers_kernel(OutlierArgs a) {
    pdl_begin();
    __shared__ __align__(16) float lim[kMPix];
    __shared__ OutlierEntry queue[kOutWarps][64];
    const int tile = blockIdx.x;
    const int x0 = tile % a.ntx * 16, y0 = tile / a.ntx * 16;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < kMPix; k += 32 * kOutWarps) {
        const int x = x0 + (k & 15), y = y0 + (k >> 4);
        const float d_obs = (x < a.W && y < a.H) ? a.obs_depth[(size_t)y * a.W + x] : 0.f;
        // a pair counts as an outlier where d_obs > 0.1 and dr < 0.8 d_obs: one compare per pair
        lim[k] = d_obs > 0.1f ? 0.8f * d_obs : -INFINITY;
    }
    __syncthreads();
    uint2 range = a.ranges[tile];
    range.y = min(range.y, a.n_list);
    const uint32_t n = range.y > range.x ? range.y - range.x : 0u;
    const int bw = min(16, a.W - x0), bh = min(16, a.H - y0);  // the tile's pixels inside the image
    OutlierEntry* q = queue[w];
    int nq = 0;  // waiting entries
    for (uint32_t base = 32 * w;; base += 32 * kOutWarps) {
        const bool last = base >= n;
        if (!last) {
            uint32_t g = 0xffffffffu;
            if (base + lane < n) g = a.indices[range.x + base + lane];
            OutlierEntry e;
            bool keep = false;
            if (g < a.n_gauss) {
                const float4* rec = a.rec + kRecQuads * (size_t)g;
                const float4 r0 = rec[0], r1 = rec[1], r3 = rec[3];
                e.u = r0.x, e.v = r0.y, e.z = r0.z;
                e.lo2 = r3.x;  // log2 o; alpha = o exp(-q/2) = 2^(log2 o - q log2(e) / 2)
                e.ca = r1.x, e.cb = r1.y, e.cc = r1.z, e.phx = r1.w;
                e.phy = rec[2].x;
                e.g = g;
                // a finite bound also for opacity 0, so that non-finite records are kept
                const float vrej = fmaxf(r3.y, -FLT_MAX);
                keep = !(block_reject<16, 16>(e.u, e.v, e.ca, e.cb, e.cc, vrej, (float)x0, (float)y0) & kRejectAlpha);
            }
            const uint32_t bal = __ballot_sync(kFullMask, keep);
            if (keep) q[nq + __popc(bal & lanemask_lt())] = e;
            nq += __popc(bal);
            __syncwarp();
        }
        if (nq >= 32 || (last && nq > 0)) {
            const int m = min(nq, 32);
            nq -= m;  // the newest m: the queue is a stack, so nothing has to move
            OutlierEntry e = q[nq + min(lane, m - 1)];
            __syncwarp();
            // dr is rounded from products and sums that keep their order, so its
            // least value over the tile is at a corner
            bool front = true;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float dy = (float)(y0 + (c >> 1) * 15) - e.v, dx = (float)(x0 + (c & 1) * 15) - e.u;
                const float dr_row = e.z + e.phy * dy;
                front &= __fmaf_rn(e.phx, dx, dr_row) > 0.f;
            }
            const bool all_front = __all_sync(kFullMask, front);
            float2 sum;
            if (bw == 16)
                sum = all_front ? outlier_sums<true, true>(e, lim, x0, y0, bw, bh)
                                : outlier_sums<true, false>(e, lim, x0, y0, bw, bh);
            else
                sum = outlier_sums<false, false>(e, lim, x0, y0, bw, bh);
            if (lane < m) {
                if (sum.x != 0.f) atomicAdd(a.total_alpha + e.g, sum.x);
                if (sum.y != 0.f) atomicAdd(a.outlier_prob + e.g, sum.y);
            }
        }
        if (last) break;
    }
}

template <int MODE>
__global__ void __launch_bounds__(kCompactBlock) mark_kernel(MarkArgs a) {
    pdl_begin();
    const uint32_t i = blockIdx.x * kCompactBlock + threadIdx.x;
    bool remove = false;
    if (i < a.n) {
        if (MODE == kMarkPrune) {
            const float alpha = a.col[i].w;
            const float4 sc = a.scale[i];
            if (alpha < a.alpha_thr) {
                remove = true;
            } else {
                const float smax = fmaxf(sc.x, fmaxf(sc.y, sc.z));
                const float smin = fminf(sc.x, fminf(sc.y, sc.z));
                const float smed = __fsub_rn(__fsub_rn(__fadd_rn(__fadd_rn(sc.x, sc.y), sc.z), smax), smin);
                remove = __fdiv_rn(smed, smax) < a.ratio_thr || smax < a.min_scale;
            }
        } else {
            const float tot = a.total_alpha[i];
            remove = tot > 1.0f && __fdiv_rn(a.outlier_prob[i], tot) > a.threshold;
        }
        a.states[i] = remove ? 0xff : 0;
    }
    const int keep = __syncthreads_count(i < a.n && !remove);
    if (threadIdx.x == 0) a.block_keep[blockIdx.x] = (uint32_t)keep;
}

// Exclusive scan of the per-block survivor counts (one CTA); counters[0] =
// survivors, counters[1] = removed.
__global__ void __launch_bounds__(1024) compact_scan_kernel(const uint32_t* __restrict__ block_keep, int nb,
                                                            uint32_t n, uint32_t* __restrict__ block_base,
                                                            uint32_t* __restrict__ counters) {
    pdl_begin();
    __shared__ uint32_t warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < nb ? block_keep[i] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            uint32_t ws = warp_sum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, ws, o);
                if (lane >= o) ws += t;
            }
            warp_sum[lane] = ws;  // inclusive over warps
        }
        __syncthreads();
        const uint32_t before = warp > 0 ? warp_sum[warp - 1] : 0u;
        if (i < nb) block_base[i] = carry + before + incl - v;
        carry += warp_sum[31];
        __syncthreads();  // warp_sum is rewritten by the next round
    }
    if (threadIdx.x == 0) {
        counters[0] = carry;
        counters[1] = n - carry;
    }
}

__global__ void __launch_bounds__(kCompactBlock) compact_scatter_kernel(CompactArgs a) {
    pdl_begin();
    if (a.counters[1] == 0) return;  // nothing removed: the host keeps the current planes
    __shared__ uint32_t wk[kCompactBlock / 32], wr[kCompactBlock / 32];
    const uint32_t i = blockIdx.x * kCompactBlock + threadIdx.x;
    const bool valid = i < a.n;
    const bool keep = valid && a.states[i] == 0;
    const unsigned bk = __ballot_sync(0xffffffffu, keep), brm = __ballot_sync(0xffffffffu, valid && !keep);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        wk[warp] = __popc(bk);
        wr[warp] = __popc(brm);
    }
    __syncthreads();
    if (!valid) return;
    uint32_t k_before = 0, r_before = 0;
    for (int w = 0; w < warp; ++w) {
        k_before += wk[w];
        r_before += wr[w];
    }
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t base_keep = a.block_base[blockIdx.x];
    // every block before this one is full, so the removed items before it are
    // its start minus the survivors before it; they follow all survivors
    const uint32_t base_rem = a.counters[0] + (blockIdx.x * (uint32_t)kCompactBlock - base_keep);
    const uint32_t dst = keep ? base_keep + k_before + __popc(bk & lt) : base_rem + r_before + __popc(brm & lt);
    a.pos_out[dst] = a.pos[i];
    a.scale_out[dst] = a.scale[i];
    a.rot_out[dst] = a.rot[i];
    a.col_out[dst] = a.col[i];
    if (a.adam) {
        const size_t cap = a.cap;
#pragma unroll
        for (int p = 0; p < 9; ++p) a.adam_out[p * cap + dst] = a.adam[p * cap + i];
    }
}

// Counts over two visibility masks: counters[0] += |a & b|, counters[1] += |a | b|.
__global__ void __launch_bounds__(256) covis_count_kernel(const uint8_t* __restrict__ va, const uint8_t* __restrict__ vb,
                                                          uint32_t n, uint32_t* __restrict__ counters) {
    pdl_begin();
    uint32_t inter = 0, uni = 0;
    const uint32_t n16 = n / 16;
    const uint4* a4 = reinterpret_cast<const uint4*>(va);
    const uint4* b4 = reinterpret_cast<const uint4*>(vb);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n16; k += stride) {
        const uint4 x = a4[k], y = b4[k];
        const uint32_t xa[4] = {x.x, x.y, x.z, x.w}, ya[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint32_t p = (xa[c] >> (8 * b)) & 0xffu, q = (ya[c] >> (8 * b)) & 0xffu;
                inter += (p & q) != 0u;
                uni += (p | q) != 0u;
            }
        }
    }
    for (uint32_t k = n16 * 16 + blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        inter += (va[k] & vb[k]) != 0;
        uni += (va[k] | vb[k]) != 0;
    }
    inter = __reduce_add_sync(0xffffffffu, inter);
    uni = __reduce_add_sync(0xffffffffu, uni);
    if ((threadIdx.x & 31) == 0 && (inter | uni)) {
        atomicAdd(counters, inter);
        atomicAdd(counters + 1, uni);
    }
}

cudaError_t launch_visibility(const VisArgs& a, cudaStream_t s) {
    const int T = a.ntx * a.nty;
    if (T <= 0) return cudaSuccess;
    return launch_chained(visibility_kernel, dim3(T), dim3(kMPix), 0, s, a);
}

cudaError_t launch_outliers(const OutlierArgs& a, cudaStream_t s) {
    const int T = a.ntx * a.nty;
    if (T <= 0) return cudaSuccess;
    return launch_chained(outliers_kernel, dim3(T), dim3(32 * kOutWarps), 0, s, a);
}

static unsigned compact_blocks(uint32_t n) { return (n + kCompactBlock - 1) / kCompactBlock; }

cudaError_t launch_mark(MarkMode mode, const MarkArgs& a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    const dim3 grid(compact_blocks(a.n));
    return mode == kMarkPrune ? launch_chained(mark_kernel<kMarkPrune>, grid, dim3(kCompactBlock), 0, s, a)
                              : launch_chained(mark_kernel<kMarkOutliers>, grid, dim3(kCompactBlock), 0, s, a);
}

cudaError_t launch_compact_scan(const uint32_t* block_keep, uint32_t n, uint32_t* block_base, uint32_t* counters,
                                cudaStream_t s) {
    return launch_chained(compact_scan_kernel, dim3(1), dim3(1024), 0, s, block_keep, (int)compact_blocks(n), n,
                          block_base, counters);
}

cudaError_t launch_compact_scatter(const CompactArgs& a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    return launch_chained(compact_scatter_kernel, dim3(compact_blocks(a.n)), dim3(kCompactBlock), 0, s, a);
}

cudaError_t launch_covis_count(const uint8_t* va, const uint8_t* vb, uint32_t n, uint32_t* counters,
                               cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const unsigned want = (n / 16 + 255) / 256 + 1;
    const unsigned grid = want < 4u * 152u ? want : 4u * 152u;
    return launch_chained(covis_count_kernel, dim3(grid), dim3(256), 0, s, va, vb, n, counters);
}

}  // namespace fvgs
