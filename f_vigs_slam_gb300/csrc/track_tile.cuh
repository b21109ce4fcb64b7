// track_tile.cuh -- the per-tile body of the fused tracking kernel (forward
// blend + RGB-D pose Jacobian + per-tile J^T J / J^T r reduction) and its
// helpers, shared by the per-frame kernel (track.cu) and the persistent
// kernel that runs the tiles of many sessions in one launch (track_batch.cu).
//
// Reference: getRgbdPoseJacobians (src/GSCudaKernels.cu:922-1392); the
// arithmetic and its reorganisation are described at the top of track.cu.
#pragma once

#include "fvgs_device.cuh"
#include "fvgs_launch.h"

namespace fvgs {

// The default tile (16 x 16, one thread per pixel): the reference's TILE_SIZE
// (src/GSCudaKernels.cu:6).
constexpr int kTW = 16, kTH = 16, kPix = kTW * kTH;
constexpr float kInv255 = 1.0f / 255.0f;

// Error-free difference: hi + lo == a - b exactly (TwoSum).
__device__ __forceinline__ void two_diff(float a, float b, float& hi, float& lo) {
    hi = __fsub_rn(a, b);
    const float bb = __fsub_rn(hi, a);
    lo = __fadd_rn(__fsub_rn(a, __fsub_rn(hi, bb)), __fsub_rn(-b, bb));
}

// z + dx*phx + dy*phy, dx = u - x and dy = v - y taken exactly, with
// compensated arithmetic (error-free differences and products via TwoSum and
// FMA, error-free sums via TwoSum): the per-Gaussian depth cancels to values
// near zero for distant pixels, and its reciprocal enters the Jacobian, so a
// plain FP32 evaluation -- or one that rounds dx, which happens when |dx|
// exceeds |u| -- would cost several digits there.
__device__ __forceinline__ float depth_at(float z, float u, float x, float phx, float v, float y, float phy) {
    float dx, dxl, dy, dyl;
    two_diff(u, x, dx, dxl);
    two_diff(v, y, dy, dyl);
    const float p1 = __fmul_rn(dx, phx);
    const float e1 = __fmaf_rn(dx, phx, -p1);
    const float p2 = __fmul_rn(dy, phy);
    const float e2 = __fmaf_rn(dy, phy, -p2);
    const float s1 = __fadd_rn(z, p1);
    const float b1 = __fsub_rn(s1, z);
    const float r1 = __fadd_rn(__fsub_rn(z, __fsub_rn(s1, b1)), __fsub_rn(p1, b1));
    const float s2 = __fadd_rn(s1, p2);
    const float b2 = __fsub_rn(s2, s1);
    const float r2 = __fadd_rn(__fsub_rn(s1, __fsub_rn(s2, b2)), __fsub_rn(p2, b2));
    const float lo = __fmaf_rn(dxl, phx, __fmul_rn(dyl, phy));
    return __fadd_rn(s2, __fadd_rn(__fadd_rn(r1, r2), __fadd_rn(__fadd_rn(e1, e2), lo)));
}

// z + dx*phx + dy*phy by two FMAs on the rounded dx = u - x, dy = v - y when
// that is accurate, else depth_at.  Each FMA rounds once and dx, dy carry at
// most half an ulp each, so the error is at most 2^-24 (|t| + |s| + |dx phx|
// + |dy phy|) with t the first FMA's result and s the second's; when |t|, |dx
// phx| and |dy phy| are all within 8 |s| that is under 1.2e-6 |s|.
// Cancellation and non-finite values take the compensated path.
__device__ __forceinline__ float depth_fast(float z, float dx, float phx, float dy, float phy, float u, float x,
                                           float v, float y) {
    const float t = __fmaf_rn(dx, phx, z);
    const float s = __fmaf_rn(dy, phy, t);
    const float m = 8.0f * fabsf(s);
    if (fabsf(t) <= m && fabsf(dx * phx) <= m && fabsf(dy * phy) <= m) return s;
    return depth_at(z, u, x, phx, v, y, phy);
}

__device__ __forceinline__ void rank1_update(float A[21], float w, float a0, float a1, float a2, float d,
                                             float r0, float r1, float r2) {
    // u = (a, d * (r x a))
    const float u[6] = {a0, a1, a2, d * (r1 * a2 - r2 * a1), d * (r2 * a0 - r0 * a2), d * (r0 * a1 - r1 * a0)};
    int idx = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const float wu = w * u[i];
#pragma unroll
        for (int j = i; j < 6; ++j) A[idx++] += wu * u[j];
    }
}

// Kahan-compensated s += x: c carries the running rounding error.
__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}

// Error-free sum: hi + lo == a + b exactly (TwoSum).
__device__ __forceinline__ void two_sum(float a, float b, float& hi, float& lo) {
    hi = __fadd_rn(a, b);
    const float bb = __fsub_rn(hi, a);
    lo = __fadd_rn(__fsub_rn(a, __fsub_rn(hi, bb)), __fsub_rn(b, bb));
}

// Butterfly reduce-scatter of 32 values over a warp: lane l ends with the warp
// sum of value l.
__device__ __forceinline__ float warp_reduce_scatter32(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < o; ++k) {
            const float send = upper ? v[k] : v[k + o];
            const float keep = upper ? v[k + o] : v[k];
            v[k] = keep + __shfl_xor_sync(kFullMask, send, o);
        }
    }
    return v[0];
}

// The same with every value an unevaluated sum v + e (precision form): each
// add is a TwoSum whose error joins the low parts, so the warp sum of value l
// is returned as hi + lo with the rounding of the butterfly compensated.
__device__ __forceinline__ void warp_reduce_scatter32_comp(float (&v)[32], float (&e)[32], float& hi, float& lo) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool upper = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < o; ++k) {
            const float send = upper ? v[k] : v[k + o], send_e = upper ? e[k] : e[k + o];
            const float keep = upper ? v[k + o] : v[k], keep_e = upper ? e[k + o] : e[k];
            const float rv = __shfl_xor_sync(kFullMask, send, o), re = __shfl_xor_sync(kFullMask, send_e, o);
            float err;
            two_sum(keep, rv, v[k], err);
            e[k] = __fadd_rn(__fadd_rn(keep_e, re), err);
        }
    }
    hi = v[0];
    lo = e[0];
}

// One Gaussian's blending record built from the reference's separate
// screen-space buffers.
__device__ __forceinline__ void load_ref_record(const TrackArgs& a, uint32_t g, float4& r0, float4& r1, float4& r2) {
    const float2 uv = reinterpret_cast<const float2*>(a.ref_uv)[g];
    const float ixx = a.ref_inv[3 * (size_t)g], iyy = a.ref_inv[3 * (size_t)g + 1], ixy = a.ref_inv[3 * (size_t)g + 2];
    const float2 ph = reinterpret_cast<const float2*>(a.ref_phat)[g];
    const bool swap = (a.quirks & FVGS_Q_INVSIGMA_SWAP) != 0;
    r0 = make_float4(uv.x, uv.y, a.ref_depth[g], a.ref_opa[g]);
    r1 = make_float4(ixx, swap ? iyy : ixy, swap ? ixy : iyy, ph.x);
    r2 = make_float4(ph.y, a.ref_col[3 * (size_t)g], a.ref_col[3 * (size_t)g + 1], a.ref_col[3 * (size_t)g + 2]);
}

// Rejection of a Gaussian by a warp's COLS x ROWS pixel block, once per staged
// Gaussian.  A pixel skips a Gaussian when v > vreject (alpha < 1/255, both
// passes) or, in the forward pass only, when v <= 0.  If the extremes of v
// over the block prove one of these for every pixel -- kRejectAlpha: min v >
// vreject, kRejectSign: max v < 0 -- with a margin covering FP32 rounding at
// the magnitude of the terms, the Gaussian is dropped.  Kept Gaussians carry
// their list index, so contributor counts and all results are unchanged.
// Non-finite records are always kept.
//
// Positive definite forms (all of them unless the reference's swapped storage
// of the inverse covariance is on) take a short way: v >= 0, and over a
// rectangle without the mean the minimum lies on an edge that faces the mean
// (the straight line from the minimum to the mean falls, so it leaves the
// rectangle at once).  Those are the edge X = the rectangle's dx nearest to 0
// and the edge Y = its dy nearest to 0; where such an edge does not face the
// mean its candidate is still a point of the rectangle, so the smaller of the
// two is the minimum.  Any other form has its extremes at the corners or, on
// an edge, at the clamped stationary point of the 1-D quadratic there (a
// minimum where it is convex, else a maximum).  The stationary points come
// from rcp.approx: one ulp off changes v by 1e-14 of its terms.
constexpr uint32_t kRejectAlpha = 1u, kRejectSign = 2u;
template <int ROWS = 4, int COLS = 8>
__device__ __forceinline__ uint32_t block_reject(float u, float v, float ca, float cb, float cc, float vrej, float x0,
                                                 float y0) {
    if (vrej == -INFINITY) return kRejectAlpha;  // zero opacity: alpha is 0 everywhere
    if (!(isfinite(u) && isfinite(v) && isfinite(ca) && isfinite(cb) && isfinite(cc) && isfinite(vrej))) return 0u;
    const float dxlo = u - (x0 + (float)(COLS - 1)), dxhi = u - x0;
    const float dylo = v - (y0 + (float)(ROWS - 1)), dyhi = v - y0;
    const float mx = fmaxf(fabsf(dxlo), fabsf(dxhi)), my = fmaxf(fabsf(dylo), fabsf(dyhi));
    const float margin = 1e-5f * (fabsf(ca) * mx * mx + 2.0f * fabsf(cb) * mx * my + fabsf(cc) * my * my) + 1e-3f;
    auto q = [&](float dx, float dy) { return ca * dx * dx + 2.0f * cb * dx * dy + cc * dy * dy; };
    const float sy = -cb * rcp_approx(cc), sx = -cb * rcp_approx(ca);
    auto on_x = [&](float X) { return q(X, fminf(fmaxf(sy * X, dylo), dyhi)); };
    auto on_y = [&](float Y) { return q(fminf(fmaxf(sx * Y, dxlo), dxhi), Y); };
    if (ca > 0.f && cc > 0.f && ca * cc - cb * cb > 0.f) {
        const float X = fminf(fmaxf(0.f, dxlo), dxhi), Y = fminf(fmaxf(0.f, dylo), dyhi);
        return fminf(on_x(X), on_y(Y)) > vrej + margin ? kRejectAlpha : 0u;
    }
    const float q00 = q(dxlo, dylo), q01 = q(dxlo, dyhi), q10 = q(dxhi, dylo), q11 = q(dxhi, dyhi);
    float lo = fminf(fminf(q00, q01), fminf(q10, q11)), hi = fmaxf(fmaxf(q00, q01), fmaxf(q10, q11));
    // a form that is 0 in both squares has no stationary point on an edge
    if (cc != 0.f) {
        const float e0 = on_x(dxlo), e1 = on_x(dxhi);
        lo = fminf(lo, fminf(e0, e1));
        hi = fmaxf(hi, fmaxf(e0, e1));
    }
    if (ca != 0.f) {
        const float e0 = on_y(dylo), e1 = on_y(dyhi);
        lo = fminf(lo, fminf(e0, e1));
        hi = fmaxf(hi, fmaxf(e0, e1));
    }
    return (lo > vrej + margin ? kRejectAlpha : 0u) | (hi < -margin ? kRejectSign : 0u);
}

// One warp's staged Gaussians: the survivors of 32 list entries, repacked so a
// rejected pair needs two loads: A = (u, v, c.x, c.y), B = (c.z, vreject,
// log2(opacity), z), C = (phat.x, phat.y, r, g), E = (b, list index), G =
// Gaussian index; for the Jacobians also X: the reference Jacobian stages
// X[j][0] = (rgx, rgy, -fx rgx, -fy rgy), the mean's normalised ray and the
// third row of the projection Jacobian without 1/d; the analytic Jacobian the
// eight vectors of pose_derivs.  An odd count is filled up with an entry that
// every pixel rejects, so the entries are taken in pairs.
constexpr int kRound = 32;  // list entries a warp stages at a time
constexpr int kMaskRounds = 32;
using RecordStage = float4[kRound][kRecQuads];
template <int NX>
struct WarpStage {
    float4 A[kRound];
    float4 B[kRound];
    float4 C[kRound];
    float4 X[NX ? kRound : 1][NX ? NX : 1];
    float2 E[kRound];
    uint32_t G[kRound];
    RecordStage R;            // the next round's records
    uint32_t M[kMaskRounds];  // reference Jacobian: the second pass's survivors of each round
};

// What a staging round stores besides the blending record.
enum StageExtra { kStageNone = 0, kStageRay = 1, kStageDeriv = 2, kStageIndex = 3 };

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// The records of a warp's 32 Gaussians (lane l's g; >= n: none) on their way to
// shared memory, four lanes a record: a 128-byte line serves eight lanes of a
// copy instead of two.  Quad c of record s lies at column c ^ (s / 2 % 4), so
// that the 32 lanes' reads of their own records meet no bank conflict.  Frames of
// 20 iterations against three planes and a lane a record: 1 M Gaussians, HD
// 3400 -> 3321 us; VGA 3329 -> 3221.
__device__ __forceinline__ void fetch_records(RecordStage& R, const float4* __restrict__ rec, uint32_t g, uint32_t n) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < kRecQuads; ++k) {
        const int s = 8 * k + (lane >> 2), c = lane & 3;
        const uint32_t gs = __shfl_sync(kFullMask, g, s);
        if (gs < n) cp_async16(&R[s][c ^ ((s >> 1) & 3)], rec + kRecQuads * (size_t)gs + c);
    }
    cp_async_commit();
}
__device__ __forceinline__ float4 record_quad(const RecordStage& R, int s, int c) { return R[s][c ^ ((s >> 1) & 3)]; }

// Walk the first n entries of the tile's list for one warp's 8 x ROWS pixel
// block with corner (x0, y0), front to back, until every lane is done.  The
// warp stages kRound entries at a time on its own -- each lane takes one
// entry, drops it when the block cannot see it, and the survivors are
// compacted in list order -- so no barrier ties it to the tile's other warps:
// a warp stops as soon as its own 32 pixels are opaque, and the tile's slowest
// block delays nobody.  The next round's records are loaded while this
// one's are blended.  pair(j, A, B, dx, dy, dl0, dl1, v, raw): one staged
// Gaussian for every lane; round_end(): after each round.
// MASKS: this walk's use of the kept survivors of the second pass (the
// reference Jacobian's rejection test costs more than the rest of its staging,
// and the first pass has both answers at hand).
// kMasksSecond: the second pass's survivors, without masks from a first.
enum WalkMasks { kMasksNone = 0, kMasksKeep = 1, kMasksUse = 2, kMasksSecond = 3 };
template <bool REF_LAYOUT, int MASKS, int STAGE, int ROWS = 4, class Args, int NX, class Pair, class RoundEnd>
__device__ __forceinline__ void walk_list(const Args& a, WarpStage<NX>& ws, uint32_t list0, int n, float x0,
                                          float y0, float xf, float yf, bool& done, Pair&& pair,
                                          RoundEnd&& round_end) {
    const int lane = threadIdx.x & 31;
    if (__all_sync(kFullMask, done)) return;
    __syncwarp();  // the staging area may still be read from an earlier walk
    // the packed records travel to shared memory while the round before is
    // blended (in registers they would be spilled around the pair loop)
    auto fetch = [&](uint32_t gi) {
        if constexpr (!REF_LAYOUT) fetch_records(ws.R, a.rec, gi, a.n_gauss);
    };
    uint32_t g = lane < n ? a.indices[list0 + lane] : 0xffffffffu;
    fetch(g);
    for (int base = 0; base < n; base += kRound) {
        const int li = base + lane;
        const uint32_t g_next = li + kRound < n ? a.indices[list0 + li + kRound] : 0xffffffffu;
        bool keep = false;
        uint32_t rej = kRejectAlpha;
        float vrej = 0.f, lo2 = 0.f;
        float4 r0, r1, r2;
        if constexpr (!REF_LAYOUT) {
            cp_async_wait<0>();
            __syncwarp();  // four lanes brought each record
        }
        if (g < a.n_gauss) {
            if constexpr (REF_LAYOUT) {
                load_ref_record(a, g, r0, r1, r2);
                lo2 = log2_opacity(r0.w);
                vrej = reject_bound(r0.w, lo2);
            } else {
                r0 = record_quad(ws.R, lane, 0);
                r1 = record_quad(ws.R, lane, 1);
                r2 = record_quad(ws.R, lane, 2);
                const float4 r3 = record_quad(ws.R, lane, 3);
                lo2 = r3.x;
                vrej = r3.y;
            }
            if (MASKS == kMasksUse && base < kRound * kMaskRounds)
                keep = (ws.M[base / kRound] >> lane) & 1u;
            else {
                rej = block_reject<ROWS>(r0.x, r0.y, r1.x, r1.y, r1.z, vrej, x0, y0);
                keep = MASKS >= kMasksUse ? !(rej & kRejectAlpha) : rej == 0u;
            }
        }
        if constexpr (MASKS == kMasksKeep) {
            const uint32_t m = __ballot_sync(kFullMask, !(rej & kRejectAlpha));
            if (lane == 0 && base < kRound * kMaskRounds) ws.M[base / kRound] = m;
        }
        const uint32_t bal = __ballot_sync(kFullMask, keep);
        const int cnt = __popc(bal);
        if (keep) {
            const int pos = __popc(bal & lanemask_lt());
            ws.A[pos] = make_float4(r0.x, r0.y, r1.x, r1.y);
            ws.B[pos] = make_float4(r1.z, vrej, lo2, r0.z);
            ws.C[pos] = make_float4(r1.w, r2.x, r2.y, r2.z);
            ws.E[pos] = make_float2(r2.w, __int_as_float(li));
            if constexpr (STAGE == kStageDeriv || STAGE == kStageIndex) ws.G[pos] = g;
            if constexpr (STAGE == kStageRay) {
                const float rgx = (r0.x - a.K.cx) * __frcp_rn(a.K.fx), rgy = (r0.y - a.K.cy) * __frcp_rn(a.K.fy);
                ws.X[pos][0] = make_float4(rgx, rgy, -a.K.fx * rgx, -a.K.fy * rgy);
            }
        }
        if (lane == 0 && (cnt & 1)) {
            ws.A[cnt] = make_float4(0.f, 0.f, 0.f, 0.f);
            ws.B[cnt] = make_float4(0.f, -INFINITY, -INFINITY, 0.f);
        }
        __syncwarp();
        if constexpr (STAGE == kStageDeriv) {
            // eight lanes bring one survivor's 128 bytes
            static_assert(NX == 8, "the analytic Jacobian stages eight derivative vectors");
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int slot = 4 * k + (lane >> 3);
                if (slot < cnt) cp_async16(&ws.X[slot][lane & 7], a.deriv + 8 * (size_t)ws.G[slot] + (lane & 7));
            }
            cp_async_commit();
        }
        g = g_next;
        fetch(g);
        if constexpr (STAGE == kStageDeriv) {
            cp_async_wait<1>();  // the derivatives; the records stay in flight
            __syncwarp();
        }
        // two entries per step: both quadratic forms and weights are
        // evaluated before the branches, in list order
        for (int j = 0; j < cnt; j += 2) {
            const float4 A0 = ws.A[j], A1 = ws.A[j + 1];
            const float4 B0 = ws.B[j], B1 = ws.B[j + 1];
            const float dx0 = A0.x - xf, dy0 = A0.y - yf, dx1 = A1.x - xf, dy1 = A1.y - yf;
            float l00, l01, l10, l11;
            const float v0 = conic_form(A0.z, A0.w, B0.x, dx0, dy0, l00, l01);
            const float v1 = conic_form(A1.z, A1.w, B1.x, dx1, dy1, l10, l11);
            const float w0 = gauss_weight(B0.z, v0), w1 = gauss_weight(B1.z, v1);
            pair(j, A0, B0, dx0, dy0, l00, l01, v0, w0);
            pair(j + 1, A1, B1, dx1, dy1, l10, l11, v1, w1);
            if (__all_sync(kFullMask, done)) break;
        }
        round_end();
        if (__all_sync(kFullMask, done)) break;
        __syncwarp();  // every lane is through with the staged entries
    }
    if constexpr (!REF_LAYOUT) cp_async_wait<0>();
}

// The derivatives of pose-coordinate pair m (2m, 2m + 1) of staged Gaussian
// j (pose_derivs' layout): du, dv, da, db, dc as float2 (register pairs).
struct DerivPair {
    float2 du, dv, da, db, dc;
};
// One pair at a time (three or two 16-byte and one 8-byte shared load), so
// the fused pass holds one pair's ten values rather than all thirty.
__device__ __forceinline__ DerivPair deriv_pair(const float4 (&X)[8], int m) {
    auto lo = [&](int plane) { return *reinterpret_cast<const float2*>(&X[plane].x); };
    auto hi = [&](int plane) { return *reinterpret_cast<const float2*>(&X[plane].z); };
    if (m == 0) {
        const float4 p0 = X[0], p1 = X[1];
        return {make_float2(p0.x, p0.y), make_float2(p0.z, p0.w), make_float2(p1.x, p1.y), make_float2(p1.z, p1.w),
                lo(2)};
    }
    if (m == 1) {
        const float4 p3 = X[3], p4 = X[4];
        return {hi(2), make_float2(p3.x, p3.y), make_float2(p3.z, p3.w), make_float2(p4.x, p4.y),
                make_float2(p4.z, p4.w)};
    }
    const float4 p5 = X[5], p6 = X[6];
    return {make_float2(p5.x, p5.y), make_float2(p5.z, p5.w), make_float2(p6.x, p6.y), make_float2(p6.z, p6.w),
            lo(7)};
}

// Depth weight of a pixel's depth residual: the reference's
// (|e| < thr ? 1 : thr / |e|) / z_obs (src/GSCudaKernels.cu:1120-1121) with
// FVGS_Q_DEPTH_HUBER, else Tukey's biweight (1 - (e / thr)^2)^2 / z_obs, zero
// beyond thr.
__device__ __forceinline__ float depth_weight(float derr, float thr, float z_obs, bool huber) {
    const float ld = fabsf(derr);
    float w;
    if (huber) {
        w = (ld < thr) ? 1.0f : thr / ld;
    } else {
        const float r = ld / thr, t = 1.0f - r * r;
        w = (ld < thr) ? t * t : 0.0f;
    }
    return w / z_obs;
}

// Dynamic shared memory of one CTA running the body: a staging area per warp.
template <int TW, int TH, bool ANALYTIC>
using BodyStage = WarpStage<ANALYTIC ? 8 : 1>;
template <int TW, int TH, bool ANALYTIC>
constexpr size_t body_smem_bytes() {
    return sizeof(BodyStage<TW, TH, ANALYTIC>) * (TW * TH / 32);
}

// One tile of the fused tracking kernel, run by a CTA of TW * TH threads (one
// per pixel; each warp covers an 8 x 4 pixel block).  Tile shapes: 16 x 16
// (the reference's), 8 x 8 and 32 x 8; the binning must use the same shape,
// except that a 16 x 16 list tile may be split over a.split CTAs of 16 x 8
// or 8 x 8 pixels (CTA `tile` covers part (tile % split) of list tile
// tile / split).  Ends with the CTA's 27 partials written to
// a.tile_out[tile]: the sum over its warps in the order of tile_partial_sum.
// COMP (precision form, analytic Jacobian only): the forward blend's colour
// accumulated with Kahan summation, and the in-tile sums of the 27 J^T J /
// J^T r partials compensated (warp_reduce_scatter32_comp, then TwoSum across
// warps); the tile-to-frame sum is compensated in every form.
// The sum of a CTA's warp partials (column col of s_red).  16 pixels wide:
// per 8-row band, (left 8 x 8 quadrant + right quadrant), each quadrant its
// upper + lower warp, then band 0 + band 1 -- so a 16 x 16 tile's sum is
// ((q00 + q10) + (q01 + q11)) whether one CTA forms it or the frame
// reduction adds the partials of 16 x 8 or 8 x 8 CTAs (tile_partial_sum).
// Other widths: the warps in order.
template <int TW, int TH>
__device__ __forceinline__ float cta_partial_sum(const float (*s_red)[32], int col) {
    constexpr int NW = TW * TH / 32;
    if constexpr (TW == 16) {
        float s = __fadd_rn(__fadd_rn(s_red[0][col], s_red[2][col]), __fadd_rn(s_red[1][col], s_red[3][col]));
        if constexpr (TH == 16)
            s = __fadd_rn(s, __fadd_rn(__fadd_rn(s_red[4][col], s_red[6][col]),
                                       __fadd_rn(s_red[5][col], s_red[7][col])));
        return s;
    } else if constexpr (TW == 8 && TH == 8) {
        return __fadd_rn(s_red[0][col], s_red[1][col]);
    } else {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) s += s_red[w][col];
        return s;
    }
}

template <int TW, int TH, bool RENDER_ONLY, bool REF_LAYOUT, bool ANALYTIC, bool COMP = false>
__device__ __forceinline__ void track_tile_body(const TrackArgs& a, int tile, unsigned char* dyn) {
    constexpr int NT = TW * TH;
    static_assert(!COMP || ANALYTIC, "compensated accumulation: analytic Jacobian");
    static_assert(TW % 8 == 0 && TH % 4 == 0 && NT % 32 == 0 && NT <= 256, "tile of 8 x 4 pixel warps");
    static_assert(TW != 16 || TH == 8 || TH == 16, "16-wide CTAs: 8-row bands");
    static_assert(!ANALYTIC || !REF_LAYOUT, "analytic Jacobian: packed records");
    using Stage = BodyStage<TW, TH, ANALYTIC>;
    Stage& ws = reinterpret_cast<Stage*>(dyn)[threadIdx.x >> 5];
    __shared__ float s_red[NT / 32][32];
    __shared__ float s_red_lo[COMP ? NT / 32 : 1][32];

    // the list tile and this CTA's pixel block in it
    const int split = a.split > 1 ? a.split : 1;
    const int lt = split == 1 ? tile : tile / split;
    int bx = 0, by = 0, ltw = TW, lth = TH;
    if (split > 1) {
        const int sub = tile - lt * split;
        bx = (sub % (16 / TW)) * TW;
        by = (sub / (16 / TW)) * TH;
        ltw = lth = 16;
    }
    const int tx = lt % a.ntx, ty = lt / a.ntx;
    const int px0 = tx * ltw + bx, py0 = ty * lth + by;
    const int tid = threadIdx.x;
    // each warp covers an 8 x 4 pixel block (compact footprint: less divergence)
    const int wq = tid >> 5, lq = tid & 31;
    const int wx0 = px0 + (wq % (TW / 8)) * 8, wy0 = py0 + (wq / (TW / 8)) * 4;
    const int x = wx0 + (lq & 7), y = wy0 + (lq >> 3);
    const float x0 = (float)wx0, y0 = (float)wy0;
    const bool in_bounds = (x < a.W && y < a.H);
    const size_t p = (size_t)y * a.W + x;
    uint2 range = a.ranges[lt];
    range.y = min(range.y, a.n_list);
    const int n = range.y > range.x ? (int)(range.y - range.x) : 0;
    const float xf = (float)x, yf = (float)y;

    float img_depth = 0.f;
    if (!RENDER_ONLY && in_bounds) img_depth = a.obs_depth[p];
    const bool inside = RENDER_ONLY ? in_bounds : (in_bounds && img_depth > 0.1f);

    // ------------------------- pass 1: forward blend -------------------------
    // FUSED (analytic Jacobian): the colour and depth Jacobians are
    // accumulated in this pass, so there is no second pass over the list.
    // Each blended Gaussian contributes
    //   kf (c T - (C - A) / (1 - alpha)) dv/dpose
    // per channel (A: colour accumulated up to and including it, C: the final
    // colour with background, kf = dalpha/dv = -alpha / 2, 0 where alpha is
    // clamped at 0.99); C is known only at the end, so with it factored out
    //   S1 += (kf c T + kf A / (1 - alpha)) dv/dpose,  S2 += kf / (1 - alpha) dv/dpose,
    // and the colour Jacobian is S1 - C S2.  (The reference's second pass
    // walks the list again with the remaining colour C - A.)
    constexpr bool FUSED = ANALYTIC && !RENDER_ONLY;
    float T = 1.f, cr = 0.f, cg = 0.f, cb = 0.f, depth = 0.f;
    float ccr = 0.f, ccg = 0.f, ccb = 0.f;  // Kahan carries of the colour (COMP)
    uint32_t last = 0;
    bool done = !inside;
    float final_T = 1.f;
    uint32_t n_contrib = 0;
    float2 fs1[3][3], fs2[3];  // FUSED: S1 (channel, pose pair) and S2 (pose pair)
#pragma unroll
    for (int m = 0; m < 3; ++m) fs1[0][m] = fs1[1][m] = fs1[2][m] = fs2[m] = make_float2(0.f, 0.f);
    // FUSED: the depth Jacobian, written once where T crosses 0.5 (each
    // thread its own column: no barrier needed)
    __shared__ float s_jd[FUSED ? 6 : 1][FUSED ? NT : 1];
    if constexpr (FUSED) {
#pragma unroll
        for (int k = 0; k < 6; ++k) s_jd[k][tid] = 0.f;
    }
    if (n > 0) {
        int last_j = -1;  // staged slot of the last blended Gaussian of this round
        auto round_end = [&]() {
            if (last_j >= 0) last = (uint32_t)__float_as_int(ws.E[last_j].y) + 1u;
            last_j = -1;
        };
        if constexpr (FUSED) {
            // one staged Gaussian with its conic-form gradient (dl0, dl1)
            auto blend_jac = [&](int j, const float4& rA, const float4& rB, float dx, float dy, float dl0, float dl1, float v,
                                 float raw) {
                const float alpha = fminf(0.99f, raw);
                if (done || v > rB.y || v <= 0.0f || alpha < kInv255) return;
                const float test_T = T * (1.0f - alpha);
                if (test_T < 0.0001f) {
                    done = true;
                    return;
                }
                const float4 rC = ws.C[j];
                const float cB = ws.E[j].x;
                const float aT = alpha * T;
                if constexpr (COMP) {
                    kahan_add(cr, ccr, rC.z * aT);
                    kahan_add(cg, ccg, rC.w * aT);
                    kahan_add(cb, ccb, cB * aT);
                } else {
                    cr += rC.z * aT;
                    cg += rC.w * aT;
                    cb += cB * aT;
                }
                const float inv1m = rcp_approx(1.0f - alpha);
                const float kf = (raw > 0.99f) ? 0.0f : -0.5f * alpha;
                const float kfi = kf * inv1m;
                const float kT = kf * T;
                const float2 w0 = make_float2(kT * rC.z + kfi * cr, kT * rC.z + kfi * cr);
                const float2 w1 = make_float2(kT * rC.w + kfi * cg, kT * rC.w + kfi * cg);
                const float2 w2 = make_float2(kT * cB + kfi * cb, kT * cB + kfi * cb);
                const float2 wi = make_float2(kfi, kfi);
                const float cu = 2.0f * dl0, cv = 2.0f * dl1, ca = dx * dx, cb2 = 2.0f * dx * dy, cc = dy * dy;
                const float2 cu2 = make_float2(cu, cu), cv2 = make_float2(cv, cv), ca2 = make_float2(ca, ca),
                             cb22 = make_float2(cb2, cb2), cc2 = make_float2(cc, cc);
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    // dv/dpose = cu du + cv dv + ca da + cb2 db + cc dc for pose pair m
                    const DerivPair d = deriv_pair(ws.X[j], m);
                    float2 gv = __fmul2_rn(cu2, d.du);
                    gv = __ffma2_rn(cv2, d.dv, gv);
                    gv = __ffma2_rn(ca2, d.da, gv);
                    gv = __ffma2_rn(cb22, d.db, gv);
                    gv = __ffma2_rn(cc2, d.dc, gv);
                    fs1[0][m] = __ffma2_rn(w0, gv, fs1[0][m]);
                    fs1[1][m] = __ffma2_rn(w1, gv, fs1[1][m]);
                    fs1[2][m] = __ffma2_rn(w2, gv, fs1[2][m]);
                    fs2[m] = __ffma2_rn(wi, gv, fs2[m]);
                }
                if (T > 0.5f && test_T < 0.5f) {
                    depth = depth_at(rB.w, rA.x, xf, rC.x, rA.y, yf, rC.y);
                    // d depth = d z + phat . d(dx, dy) + (dx, dy) . d phat, with
                    // d phat = (dp_x / z^2 - 2 x dp_z / z^3, dp_y / z^2 - 2 y dp_z / z^3)
                    const float z = rB.w, x = ws.X[j][7].z, y = ws.X[j][7].w;
                    const float iz = __frcp_rn(z), iz2 = iz * iz, iz3 = iz2 * iz;
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        const float dpx = k == 0 ? -1.f : (k == 4 ? -z : (k == 5 ? y : 0.f));
                        const float dpy = k == 1 ? -1.f : (k == 3 ? z : (k == 5 ? -x : 0.f));
                        const float dpz = k == 2 ? -1.f : (k == 3 ? -y : (k == 4 ? x : 0.f));
                        const float dphx = dpx * iz2 - 2.f * x * iz3 * dpz;
                        const float dphy = dpy * iz2 - 2.f * y * iz3 * dpz;
                        const DerivPair d = deriv_pair(ws.X[j], k >> 1);
                        const float du_k = (k & 1) ? d.du.y : d.du.x;
                        const float dv_k = (k & 1) ? d.dv.y : d.dv.x;
                        s_jd[k][tid] = dpz + rC.x * du_k + dx * dphx + rC.y * dv_k + dy * dphy;
                    }
                }
                T = test_T;
                last_j = j;
            };
            walk_list<REF_LAYOUT, kMasksNone, kStageDeriv>(a, ws, range.x, n, x0, y0, xf, yf, done, blend_jac, round_end);
        } else {
            auto blend = [&](int j, const float4& rA, const float4& rB, float dx, float dy, float, float, float v, float raw) {
                const float alpha = fminf(0.99f, raw);
                if (done || v > rB.y || v <= 0.0f || alpha < kInv255) return;
                const float test_T = T * (1.0f - alpha);
                if (test_T < 0.0001f) {
                    done = true;
                    return;
                }
                const float4 rC = ws.C[j];
                const float aT = alpha * T;
                cr += rC.z * aT;
                cg += rC.w * aT;
                cb += ws.E[j].x * aT;
                if (T > 0.5f && test_T < 0.5f) depth = depth_at(rB.w, rA.x, xf, rC.x, rA.y, yf, rC.y);
                T = test_T;
                last_j = j;
            };
            walk_list<REF_LAYOUT, RENDER_ONLY ? kMasksNone : kMasksKeep, kStageNone>(a, ws, range.x, n, x0, y0, xf, yf, done, blend, round_end);
        }
        if (inside) {
            final_T = T;
            n_contrib = last;
            cr += T * a.bg[0];
            cg += T * a.bg[1];
            cb += T * a.bg[2];
        }
    }
    if (a.img_color && in_bounds) {
        a.img_color[3 * p] = cr;
        a.img_color[3 * p + 1] = cg;
        a.img_color[3 * p + 2] = cb;
        a.img_depth[p] = depth;
        a.img_T[p] = final_T;
        a.img_nc[p] = n_contrib;
    }
    if (RENDER_ONLY) return;

    // ------------------------- per-pixel term -------------------------------
    const bool do_jac = inside && (final_T < a.alpha_thresh);
    float A[21];
    float bv[6];
#pragma unroll
    for (int k = 0; k < 21; ++k) A[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 6; ++k) bv[k] = 0.f;
    const float fx = a.K.fx, fy = a.K.fy, cx = a.K.cx, cy = a.K.cy;
    const bool huber = (a.quirks & FVGS_Q_DEPTH_HUBER) != 0;
    float e0 = 0.f, e1 = 0.f, e2 = 0.f, wc = 0.f, derr = 0.f, wd = 0.f;
    if (ANALYTIC && do_jac) {
        e0 = cr - a.obs_rgb[3 * p];
        e1 = cg - a.obs_rgb[3 * p + 1];
        e2 = cb - a.obs_rgb[3 * p + 2];
        derr = depth - img_depth;
        const float closs = sqrtf(e0 * e0 + e1 * e1 + e2 * e2);
        wc = (closs < a.color_thresh) ? 1.0f : a.color_thresh / closs;
        wd = depth_weight(derr, a.depth_thresh, img_depth, huber);
    }
    if (!ANALYTIC && do_jac) {
        e0 = cr - a.obs_rgb[3 * p];
        e1 = cg - a.obs_rgb[3 * p + 1];
        e2 = cb - a.obs_rgb[3 * p + 2];
        derr = (img_depth > 0.1f) ? (depth - img_depth) : 0.0f;
        const float closs = sqrtf(e0 * e0 + e1 * e1 + e2 * e2);
        wc = (closs < a.color_thresh) ? 1.0f : a.color_thresh / closs;
        const float rx = (xf - cx) / fx, ry = (yf - cy) / fy;
        const float inv_id = __frcp_rn(img_depth);
        const float j0 = fx * inv_id, j3 = fy * inv_id, j4 = -fx * rx * inv_id, j5 = -fy * ry * inv_id;
        const float gX[3] = {a.gx[3 * p], a.gx[3 * p + 1], a.gx[3 * p + 2]};
        const float gY[3] = {a.gy[3 * p], a.gy[3 * p + 1], a.gy[3 * p + 2]};
        const float ee[3] = {e0, e1, e2};
        float Jr0 = 0.f, Jr1 = 0.f, Jr2 = 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float c0 = j0 * gX[k], c1 = j3 * gY[k], c2 = j4 * gX[k] + j5 * gY[k];
            rank1_update(A, wc, c0, c1, c2, img_depth, rx, ry, 1.0f);
            Jr0 += c0 * ee[k];
            Jr1 += c1 * ee[k];
            Jr2 += c2 * ee[k];
        }
        Jr0 *= -wc;
        Jr1 *= -wc;
        Jr2 *= -wc;
        wd = depth_weight(derr, a.depth_thresh, img_depth, huber);
        // wd * ray ray^T: the rotation block gets ray x ray = 0
        {
            const float r[3] = {rx, ry, 1.0f};
            int idx = 0;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
#pragma unroll
                for (int j = i; j < 6; ++j) {
                    if (j < 3) A[idx] += wd * r[i] * r[j];
                    ++idx;
                }
            }
        }
        Jr0 += wd * derr * rx;
        Jr1 += wd * derr * ry;
        Jr2 += wd * derr;
        bv[0] += Jr0;
        bv[1] += Jr1;
        bv[2] += Jr2;
        bv[3] += img_depth * (ry * Jr2 - 1.0f * Jr1);
        bv[4] += img_depth * (1.0f * Jr0 - rx * Jr2);
        bv[5] += img_depth * (rx * Jr1 - ry * Jr0);
    }

    // ------------------- pass 2 (reference Jacobian): per-Gaussian terms ---
    if constexpr (ANALYTIC) {
        // Colour Jacobian jc (3 x 6) of the pixel from the fused pass's sums:
        // jc = S1 - C S2 (C: the final colour with background); jd: the depth
        // Jacobian of the Gaussian where T crossed 0.5.  Pose coordinates in
        // pairs (2m, 2m + 1), packed FP32 FMAs (two IEEE round-to-nearest
        // FMAs each, the results of __fmaf_rn).
        float2 jc2[3][3];
        const float2 nr = make_float2(-cr, -cr), ng = make_float2(-cg, -cg), nb = make_float2(-cb, -cb);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            jc2[0][m] = __ffma2_rn(nr, fs2[m], fs1[0][m]);
            jc2[1][m] = __ffma2_rn(ng, fs2[m], fs1[1][m]);
            jc2[2][m] = __ffma2_rn(nb, fs2[m], fs1[2][m]);
        }
        float jd[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) jd[k] = s_jd[k][tid];
        if (do_jac) {
            float jc[3][6];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int m = 0; m < 3; ++m) {
                    jc[c][2 * m] = jc2[c][m].x;
                    jc[c][2 * m + 1] = jc2[c][m].y;
                }
            int idx = 0;
#pragma unroll
            for (int i = 0; i < 6; ++i) {
#pragma unroll
                for (int k = i; k < 6; ++k)
                    A[idx++] = wc * (jc[0][i] * jc[0][k] + jc[1][i] * jc[1][k] + jc[2][i] * jc[2][k]) +
                               wd * jd[i] * jd[k];
                bv[i] = -(wc * (jc[0][i] * e0 + jc[1][i] * e1 + jc[2][i] * e2) + wd * jd[i] * derr);
            }
        }
    } else {
        // rem = final colour minus the colour accumulated so far (running)
        float prod_alpha = 1.f, remr = cr, remg = cg, remb = cb;
        bool depth_pending = img_depth > 0.5f;  // the depth term is added once, where T first falls to 0.5
        bool done2 = !do_jac || n_contrib == 0;
        // the entries past the last contributor of the warp's pixels are not needed
        const int nmax = (int)min((uint32_t)n, __reduce_max_sync(kFullMask, do_jac ? n_contrib : 0u));
        auto rank_one = [&](int j, const float4& rA, const float4& rB, float dx, float dy, float dl0, float dl1, float v,
                            float raw) {
            if (done2) return;
            if (rB.y != -INFINITY && __float_as_int(ws.E[j].y) >= (int)n_contrib) {
                done2 = true;
                return;
            }
            const float alpha = fminf(0.99f, raw);
            if (v > rB.y || alpha < kInv255) return;
            const float4 rC = ws.C[j];
            const float4 rE = ws.X[j][0];
            const float d = depth_fast(rB.w, dx, rC.x, dy, rC.y, rA.x, xf, rA.y, yf);
            float da0 = rC.z * prod_alpha, da1 = rC.w * prod_alpha, da2 = ws.E[j].x * prod_alpha;
            remr -= alpha * da0;
            remg -= alpha * da1;
            remb -= alpha * da2;
            const float inv1m = rcp_approx(1.0f - alpha);
            da0 -= remr * inv1m;
            da1 -= remg * inv1m;
            da2 -= remb * inv1m;
            // The reference's per-Gaussian row is u = (jt, d (r x jt)) with
            // jt = g / d, g = (fx dl0, fy dl1, -fx rgx dl0 - fy rgy dl1) and
            // r = (rgx, rgy, 1): the same vector as (g / d, r x g).
            const float g0 = fx * dl0, g1 = fy * dl1, g2 = rE.z * dl0 + rE.w * dl1;
            const float inv_d = rcp_approx(d);
            const float u0 = g0 * inv_d, u1 = g1 * inv_d, u2 = g2 * inv_d;
            const float u3 = rE.y * g2 - g1, u4 = g0 - rE.x * g2, u5 = rE.x * g1 - rE.y * g0;
            const float w = wc * alpha * alpha * (da0 * da0 + da1 * da1 + da2 * da2);
            {
                const float u[6] = {u0, u1, u2, u3, u4, u5};
                int idx = 0;
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    const float wu = w * u[i];
#pragma unroll
                    for (int k = i; k < 6; ++k) A[idx++] += wu * u[k];
                }
            }
            const float coef = -wc * alpha * (da0 * e0 + da1 * e1 + da2 * e2);
            bv[0] += coef * u0;
            bv[1] += coef * u1;
            bv[2] += coef * u2;
            bv[3] += coef * u3;
            bv[4] += coef * u4;
            bv[5] += coef * u5;
            prod_alpha *= (1.0f - alpha);
            if (depth_pending && prod_alpha <= 0.5f) {
                // the depth term wd * derr * r: its rotation part d (r x r) is zero
                depth_pending = false;
                const float r[3] = {rE.x, rE.y, 1.0f};
                int idx = 0;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
#pragma unroll
                    for (int jj = i; jj < 6; ++jj) {
                        if (jj < 3) A[idx] += wd * r[i] * r[jj];
                        ++idx;
                    }
                }
                bv[0] += wd * derr * rE.x;
                bv[1] += wd * derr * rE.y;
                bv[2] += wd * derr;
            }
            if (prod_alpha < 0.001f) done2 = true;
        };
        if (nmax > 0)
            walk_list<REF_LAYOUT, kMasksUse, kStageRay>(a, ws, range.x, nmax, x0, y0, xf, yf, done2, rank_one, [] {});
    }

    // --------------------------- tile reduction ------------------------------
    float vals[32];
#pragma unroll
    for (int k = 0; k < 6; ++k) vals[k] = bv[k];
#pragma unroll
    for (int k = 0; k < 21; ++k) vals[6 + k] = A[k];
#pragma unroll
    for (int k = 27; k < 32; ++k) vals[k] = 0.f;
    if constexpr (COMP) {
        float errs[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) errs[k] = 0.f;
        float hi, lo;
        warp_reduce_scatter32_comp(vals, errs, hi, lo);
        s_red[tid >> 5][tid & 31] = hi;
        s_red_lo[tid >> 5][tid & 31] = lo;
        __syncthreads();
        if (tid < FVGS_POSEDATA_FLOATS) {
            float s = 0.f, e = 0.f;
#pragma unroll
            for (int w = 0; w < NT / 32; ++w) {
                float err;
                two_sum(s, s_red[w][tid], s, err);
                e = __fadd_rn(e, __fadd_rn(err, s_red_lo[w][tid]));
            }
            a.tile_out[(size_t)tile * FVGS_POSEDATA_FLOATS + tid] = __fadd_rn(s, e);
        }
    } else {
        const float mine = warp_reduce_scatter32(vals);
        s_red[tid >> 5][tid & 31] = mine;
        __syncthreads();
        if (tid < FVGS_POSEDATA_FLOATS)
            a.tile_out[(size_t)tile * FVGS_POSEDATA_FLOATS + tid] = cta_partial_sum<TW, TH>(s_red, tid);
    }
}

}  // namespace fvgs
