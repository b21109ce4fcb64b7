// render.cu -- render-form forward pass (the viewer's image) for sm_103a.
//
// Reference: forwardPassTileKernel (src/GSCudaKernels.cu:710-859) launched by
// GSSlam::rasterize / renderView (src/GSSlam.cu:648-799).  Its semantics
// differ from the tracking kernel's forward blend:
//  * the inverse 2D covariance is taken in its true (xx, xy, yy) layout (the
//    kernel inverts Sigma2D itself, 817, so the stored-layout swap of the
//    tracking kernels does not apply);
//  * every Gaussian of the tile list blends with w = opacity *
//    exp(-0.5 (ixx dx^2 + iyy dy^2 + 2 ixy dx dy)), d = pixel - mean: no 0.99
//    clamp, no 1/255 threshold, no v <= 0 skip (a negative opacity blends a
//    negative weight, as there);
//  * colour += (1 - A) w c, A += (1 - A) w; a pixel stops once A >= 0.99
//    (the transmittance 1 - A is carried here as T <- T (1 - w), the same
//    quantity without the cancellation of 1 - A near A = 0.99);
//  * median depth z + phat . d at the first crossing of 1 - A through 0.5,
//    1e10 where there is none; no background colour.
// The reference writes its float3 colour into an 8-bit, 3-channel image (an
// overrun); here the image is a float RGB buffer, with an optional 8-bit copy
// (round(255 c), saturated).
#include <type_traits>

#include "track_tile.cuh"

namespace fvgs {

// One warp's staged list entries.  The colours and c'xx stand twice, as the
// packed FP32 instructions take them.
struct ViewStage {
    float4 A[kRound];     // u, v, log2|opacity|, z
    float4 B[kRound];     // 2 c'xy, c'yy, phat.x, phat.y
    float4 C[kRound];     // r, r, g, g
    float4 D[kRound];     // b, b, c'xx, c'xx
    float S[kRound];      // sign of the opacity (read only by rounds with an odd record)
    RecordStage R;        // the next round's records, in flight
};

// w = o exp(-q/2) as 2^t with t = log2|o| + c'xx dx^2 + 2 c'xy dx dy +
// c'yy dy^2, the inverse covariance pre-scaled by -log2(e)/2 once per staged
// Gaussian: five FP32 ops and the PTX ex2.approx per pair (the tracking
// kernels' weight, without their thresholds).  The exponent's FP32 rounding
// adds about 1.4e-7 |t| relative error to w, so under 3e-6 wherever
// w > 2^-20.  Opacity zero gives w = 0, NaN gives NaN, as o exp(..) does.
//
// Two warps a CTA, each an 8 x 8 pixel quarter of a 16 x 16 tile on its own
// (no barrier; a warp ends when its 64 pixels have), two neighbouring pixels
// of a row a lane with packed FP32 instructions, whose halves round as the
// scalar ones do.  A pixel's next event is the level th its T has to fall to:
// 0.5 (the depth), then 0.01 (the end), then none; so a pair costs one compare
// a pixel.  An ended pixel goes on with off = -inf, that is w = 0.  A round of
// 32 entries that holds a negative opacity or a value above 1e8 or not finite
// (where w = 0 could not be relied on) takes the plain loop.
//
// What bounds it: issue (59 %) and shared-memory wavefronts (68 %).  1 M
// Gaussians, 1280x720 (6.7 M entries): 66 us,
// before (a CTA per tile, a pixel a lane, 256 entries between barriers) 72.
__global__ void __launch_bounds__(64) render_view_kernel(RenderArgs a) {
    pdl_begin();
    __shared__ ViewStage stage[2];
    const int lane = threadIdx.x & 31;
    ViewStage& ws = stage[threadIdx.x >> 5];
    const int tile = blockIdx.x >> 1, quarter = (blockIdx.x & 1) * 2 + (threadIdx.x >> 5);
    const int x = tile % a.ntx * 16 + (quarter & 1) * 8 + 2 * (lane & 3);
    const int y = tile / a.ntx * 16 + (quarter >> 1) * 8 + (lane >> 2);
    uint2 range = a.ranges[tile];
    range.y = min(range.y, a.n_list);
    const int n = range.y > range.x ? (int)(range.y - range.x) : 0;
    const bool swap = (a.quirks & FVGS_Q_INVSIGMA_SWAP) != 0;
    const float2 px = make_float2((float)x, (float)(x + 1));
    const float py = (float)y;
    float2 cr = make_float2(0.f, 0.f), cg = cr, cb = cr, T = make_float2(1.f, 1.f);
    float depth[2] = {1e10f, 1e10f}, th[2];
    float2 off;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const bool inside = x + k < a.W && y < a.H;
        th[k] = inside ? 0.5f : -1.f;
        (k ? off.y : off.x) = inside ? 0.f : -INFINITY;
    }
    bool done = th[0] < 0.f && th[1] < 0.f;

    // T has fallen to th
    auto event = [&](int j, int k, float& t, float& o, float dx, float dy) {
        if (th[k] == 0.5f) {
            const float4 gB = ws.B[j];
            depth[k] = ws.A[j].w + gB.z * dx + gB.w * dy;
            th[k] = 0.01f;
        }
        if (t <= 0.01f) {  // A >= 0.99
            th[k] = -1.f;
            t = 0.f;
            o = -INFINITY;
        }
        done = th[0] < 0.f && th[1] < 0.f;
    };
    auto weight = [&](int j, float& dy, float2& dx) {
        const float4 gA = ws.A[j];
        const float2 gB = *reinterpret_cast<const float2*>(&ws.B[j]), gD = *reinterpret_cast<const float2*>(&ws.D[j].z);
        dy = py - gA.y;
        dx = __fadd2_rn(px, make_float2(-gA.x, -gA.x));
        const float by = __fmul_rn(gB.x, dy), cc = __fmaf_rn(__fmul_rn(gB.y, dy), dy, gA.z);
        const float2 t = __ffma2_rn(dx, __ffma2_rn(gD, dx, make_float2(by, by)),
                                    __fadd2_rn(make_float2(cc, cc), off));
        return make_float2(ex2_approx(t.x), ex2_approx(t.y));
    };
    auto blend = [&](int j, float2 w, float dy, float2 dx) {
        const float4 gC = ws.C[j];
        const float2 gD = *reinterpret_cast<const float2*>(&ws.D[j]);
        const float2 Tw = __fmul2_rn(T, w);
        cr = __ffma2_rn(Tw, make_float2(gC.x, gC.y), cr);
        cg = __ffma2_rn(Tw, make_float2(gC.z, gC.w), cg);
        cb = __ffma2_rn(Tw, gD, cb);
        // 1 - A of the reference, without the cancellation
        T = __fmul2_rn(T, __fadd2_rn(make_float2(1.f, 1.f), make_float2(-w.x, -w.y)));
        if (T.x <= th[0] || T.y <= th[1]) {
            if (T.x <= th[0]) event(j, 0, T.x, off.x, dx.x, dy);
            if (T.y <= th[1]) event(j, 1, T.y, off.y, dx.y, dy);
        }
    };
    // any record: the weight takes the sign of the Gaussian's opacity, and an
    // ended pixel is passed by
    auto blend_odd = [&](int j, int k) {
        if (th[k] < 0.f) return;
        float& t = k ? T.y : T.x;
        const float4 gA = ws.A[j], gB = ws.B[j], gC = ws.C[j], gD = ws.D[j];
        const float dx = (k ? px.y : px.x) - gA.x, dy = py - gA.y;
        const float w = ws.S[j] * ex2_approx(__fmaf_rn(dx, __fmaf_rn(gD.z, dx, __fmul_rn(gB.x, dy)),
                                                       __fmaf_rn(__fmul_rn(gB.y, dy), dy, gA.z)));
        const float Tw = t * w;
        (k ? cr.y : cr.x) += Tw * gC.x;
        (k ? cg.y : cg.x) += Tw * gC.z;
        (k ? cb.y : cb.x) += Tw * gD.x;
        t *= 1.0f - w;
        if (t <= th[k]) event(j, k, t, k ? off.y : off.x, dx, dy);
    };

    // the records of the next round travel while this one's are blended
    auto fetch = [&](uint32_t g) { fetch_records(ws.R, a.rec, g, a.n_gauss); };
    uint32_t g = lane < n ? a.indices[range.x + lane] : 0xffffffffu;
    if (!__all_sync(kFullMask, done)) {
        fetch(g);
        for (int base = 0; base < n; base += kRound) {
            const int li = base + lane;
            const uint32_t g_next = li + kRound < n ? a.indices[range.x + li + kRound] : 0xffffffffu;
            float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
            cp_async_wait<0>();
            __syncwarp();  // four lanes brought each record
            if (g < a.n_gauss) {
                r0 = record_quad(ws.R, lane, 0);
                r1 = record_quad(ws.R, lane, 1);
                r2 = record_quad(ws.R, lane, 2);
            }
            // the packed record holds the inverse in the tracking kernels'
            // consumed order; undo the swap for the true layout
            const float cxx = kGaussScale * r1.x, cxy = 2.0f * kGaussScale * (swap ? r1.z : r1.y),
                        cyy = kGaussScale * (swap ? r1.y : r1.z);
            ws.A[lane] = make_float4(r0.x, r0.y, log2f(fabsf(r0.w)), r0.z);
            ws.B[lane] = make_float4(cxy, cyy, r1.w, r2.x);
            ws.C[lane] = make_float4(r2.y, r2.y, r2.z, r2.z);
            ws.D[lane] = make_float4(r2.w, r2.w, cxx, cxx);
            ws.S[lane] = r0.w < 0.f ? -1.0f : 1.0f;
            const float sum = fabsf(r0.x) + fabsf(r0.y) + r0.w + fabsf(cxx) + fabsf(cxy) + fabsf(cyy) + fabsf(r2.y) +
                              fabsf(r2.z) + fabsf(r2.w);
            const bool odd = __any_sync(kFullMask, r0.w < 0.f || !(sum < 1e8f));
            __syncwarp();
            g = g_next;
            fetch(g);
            const int cnt = min(kRound, n - base);
            if (!odd) {
                // the slots beyond the list's end hold w = 0
                for (int j = 0; j < cnt; j += 2) {
                    float dy0, dy1;
                    float2 dx0, dx1;
                    const float2 w0 = weight(j, dy0, dx0), w1 = weight(j + 1, dy1, dx1);
                    blend(j, w0, dy0, dx0);
                    // a pixel that ended with the first entry
                    blend(j + 1, make_float2(th[0] < 0.f ? 0.f : w1.x, th[1] < 0.f ? 0.f : w1.y), dy1, dx1);
                    if (__all_sync(kFullMask, done)) break;
                }
            } else {
                for (int j = 0; j < cnt && !done; ++j) {
                    blend_odd(j, 0);
                    blend_odd(j, 1);
                }
            }
            if (__all_sync(kFullMask, done)) break;
            __syncwarp();  // every lane is through with the staged entries
        }
        cp_async_wait<0>();
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (x + k >= a.W || y >= a.H) continue;
        const size_t p = (size_t)y * a.W + x + k;
        const float c[3] = {k ? cr.y : cr.x, k ? cg.y : cg.x, k ? cb.y : cb.x};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a.out_rgb[3 * p + i] = c[i];
            if (a.out_rgb8) a.out_rgb8[3 * p + i] = (uint8_t)__float2int_rn(__saturatef(c[i]) * 255.0f);
        }
        a.out_depth[p] = depth[k];
    }
}

// The form for small images: a CTA per tile, a pixel a lane, 256 entries staged
// by the whole CTA.  It has twice the warps a tile, and its long lists (few
// tiles: each holds much of the map) are staged eight times as deep.
constexpr int kRPix = 256;  // 16 x 16 pixels per tile
__global__ void __launch_bounds__(kRPix) render_view_tile_kernel(RenderArgs a) {
    pdl_begin();
    __shared__ float4 sA[kRPix];  // u, v, log2|opacity|, z
    __shared__ float4 sB[kRPix];  // c'xx, 2 c'xy, c'yy, phat.x
    __shared__ float4 sC[kRPix];  // phat.y, r, g, b
    __shared__ float sS[kRPix];   // sign of the opacity (read only by batches with a negative one)
    const int tile = blockIdx.x;
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    const int tid = threadIdx.x;
    const int x = tx * 16 + (tid & 15), y = ty * 16 + (tid >> 4);
    const bool inside = x < a.W && y < a.H;
    uint2 range = a.ranges[tile];
    range.y = min(range.y, a.n_list);
    const int n = range.y > range.x ? (int)(range.y - range.x) : 0;
    const bool swap = (a.quirks & FVGS_Q_INVSIGMA_SWAP) != 0;
    const float px = (float)x, py = (float)y;
    float cr = 0.f, cg = 0.f, cb = 0.f, T = 1.f, depth = 1e10f;
    bool has_depth = false, done = !inside;

    // one pair; NEG: the weight takes the sign of the Gaussian's opacity
    auto blend = [&](int j, auto neg_tag) {
        constexpr bool NEG = decltype(neg_tag)::value;
        const float4 gA = sA[j];
        const float4 gB = sB[j];
        const float dx = px - gA.x, dy = py - gA.y;
        const float t = __fmaf_rn(dx, __fmaf_rn(gB.x, dx, __fmul_rn(gB.y, dy)),
                                  __fmaf_rn(__fmul_rn(gB.z, dy), dy, gA.z));
        float w = ex2_approx(t);
        if (NEG) w *= sS[j];
        const float Tb = T;
        const float Tw = Tb * w;
        const float4 gC = sC[j];
        cr += Tw * gC.y;
        cg += Tw * gC.z;
        cb += Tw * gC.w;
        T = Tb * (1.0f - w);  // 1 - A of the reference, without the cancellation
        if (!has_depth && Tb > 0.5f && T <= 0.5f) {
            depth = gA.w + gB.w * dx + gC.x * dy;
            has_depth = true;
        }
        if (T <= 0.01f) done = true;  // A >= 0.99
    };

    for (int base = 0; base < n; base += kRPix) {
        if (__syncthreads_and(done)) break;
        const int li = base + tid;
        bool neg = false;
        if (li < n) {
            const uint32_t g = a.indices[range.x + li];
            float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0;
            if (g < a.n_gauss) {
                const float4* rec = a.rec + kRecQuads * (size_t)g;
                r0 = rec[0];
                r1 = rec[1];
                r2 = rec[2];
            }
            // the packed record holds the inverse in the tracking kernels'
            // consumed order; undo the swap for the true layout
            const float ixy = swap ? r1.z : r1.y, iyy = swap ? r1.y : r1.z;
            neg = r0.w < 0.f;
            sA[tid] = make_float4(r0.x, r0.y, log2f(fabsf(r0.w)), r0.z);
            sB[tid] = make_float4(kGaussScale * r1.x, 2.0f * kGaussScale * ixy, kGaussScale * iyy, r1.w);
            sC[tid] = r2;
            sS[tid] = neg ? -1.0f : 1.0f;
        }
        const bool any_neg = __syncthreads_or(neg);
        const int cnt = min(kRPix, n - base);
        if (!any_neg) {
            for (int j = 0; j < cnt && !done; ++j) blend(j, std::false_type{});
        } else {
            for (int j = 0; j < cnt && !done; ++j) blend(j, std::true_type{});
        }
    }
    if (!inside) return;
    const size_t p = (size_t)y * a.W + x;
    a.out_rgb[3 * p] = cr;
    a.out_rgb[3 * p + 1] = cg;
    a.out_rgb[3 * p + 2] = cb;
    a.out_depth[p] = depth;
    if (a.out_rgb8) {
        a.out_rgb8[3 * p] = (uint8_t)__float2int_rn(__saturatef(cr) * 255.0f);
        a.out_rgb8[3 * p + 1] = (uint8_t)__float2int_rn(__saturatef(cg) * 255.0f);
        a.out_rgb8[3 * p + 2] = (uint8_t)__float2int_rn(__saturatef(cb) * 255.0f);
    }
}

// Up to kSmallTiles tiles per SM the warps of two pixels a lane are too few to
// hide each other's latency.  Kernel, us, that form / the tile's: 107x82 (42
// tiles) 39 / 29, 160x120 (80) 94 / 66, 240x160 (150) 43 / 31, 398x313 (500) 37 /
// 37, 500x400 (800) 37 / 39, 640x480 (1200) 41 / 45, 900x600 (2166) 45 / 50,
// 1280x720 (3600) 64 / 74.
constexpr int kSmallTiles = 3;

cudaError_t launch_render_view(const RenderArgs& a, int num_sms, cudaStream_t s) {
    const int T = a.ntx * a.nty;
    if (T <= 0) return cudaSuccess;
    if (T <= kSmallTiles * num_sms) return launch_chained(render_view_tile_kernel, dim3(T), dim3(kRPix), 0, s, a);
    return launch_chained(render_view_kernel, dim3(2 * T), dim3(64), 0, s, a);
}

}  // namespace fvgs
