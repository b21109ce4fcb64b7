// map.cu -- mapping step (forward, backward,
// 2D->3D chain rule and Adam) for sm_103a.
//
// Reference: GSSlam::optimizeGaussiansKeyframe (src/GSSlam.cu:1083-1320) with
// perTileBucketCount (src/GSCudaKernels.cu:2074-2090),
// optimizeGaussiansForwardPass (2092-2263), optimizeGaussiansPerGaussianPass
// (2265-2502), computeDeltaGaussians3D_kernel (2504-2720) and
// updateGaussiansParametersAdam_kernel (2722-2882).
//
// GPU structure:
//  * forward and backward: every warp walks its tile's list for its own 8 x 4
//    pixels (walk_list, as the tracking kernel), a lane per pixel.  The
//    backward pass carries the pixel's T and accumulated colour along the list
//    again, so the forward pass leaves no checkpoints; the reference's restart
//    from a checkpoint every 32 list entries is the forward pass's state,
//    carried beside.  A Gaussian's twelve sums are added over the warp by a
//    butterfly and go to memory with one reduction of 12 lanes;
//  * 2D->3D and Adam are fused: the 3D deltas never go to memory.
#include <algorithm>

#include "track_tile.cuh"

namespace fvgs {

constexpr int kMapCap = 256;  // list entries that receive gradients with MAP_CAP256

// Two warps a CTA, each an 8 x 8 pixel quarter of a 16 x 16 tile, two pixels a
// lane (rows y and y + 4): a staged Gaussian is read, and its sums are added
// over the warp, once for 64 pixels.
struct MapBlock {
    int x0, y0, x, y[2], n;
    uint32_t list0;
    bool inside[2];
    __device__ explicit MapBlock(const MapArgs& a) {
        const int tile = blockIdx.x >> 1, quarter = (blockIdx.x & 1) * 2 + (threadIdx.x >> 5);
        const int lane = threadIdx.x & 31;
        x0 = (tile % a.ntx) * 16 + (quarter & 1) * 8;
        y0 = (tile / a.ntx) * 16 + (quarter >> 1) * 8;
        x = x0 + (lane & 7);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            y[k] = y0 + (lane >> 3) + 4 * k;
            inside[k] = x < a.W && y[k] < a.H;
        }
        uint2 range = a.ranges[tile];
        range.y = min(range.y, a.n_list);
        list0 = range.x;
        n = range.y > range.x ? (int)(range.y - range.x) : 0;
    }
};

// Forward pass.  What bounds it: issue; 1 M Gaussians, 1280x720: 125 us, before
// (a CTA per tile, every list entry evaluated by every pixel, checkpoints)
// 187.
__global__ void __launch_bounds__(64) map_forward_kernel(MapArgs a) {
    pdl_begin();
    __shared__ WarpStage<0> stage[2];
    WarpStage<0>& ws = stage[threadIdx.x >> 5];
    const MapBlock blk(a);
    const float xf = (float)blk.x;
    float T[2], cr[2], cg[2], cb[2], depth[2];
    uint32_t last[2];
    int last_j[2];  // staged slot of the last blended Gaussian of this round
    bool end[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        T[k] = 1.f;
        cr[k] = cg[k] = cb[k] = depth[k] = 0.f;
        last[k] = 0;
        last_j[k] = -1;
        end[k] = !blk.inside[k];
    }
    bool done = end[0] && end[1];
    auto blend = [&](int j, const float4& rA, const float4& rB, float dxm, float dy0, float, float, float v0,
                     float raw0) {
        const float dy1 = rA.y - (float)blk.y[1];
        float q0, q1;
        const float v1 = conic_form(rA.z, rA.w, rB.x, dxm, dy1, q0, q1);
        const float raw1 = gauss_weight(rB.z, v1);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float v = k ? v1 : v0, dym = k ? dy1 : dy0;
            const float alpha = fminf(0.99f, k ? raw1 : raw0);
            if (!(end[k] || v > rB.y || v <= 0.0f || alpha < kInv255)) {
                const float4 rC = ws.C[j];
                cr[k] += T[k] * alpha * rC.z;
                cg[k] += T[k] * alpha * rC.w;
                cb[k] += T[k] * alpha * ws.E[j].x;
                const float test_T = T[k] * (1.0f - alpha);
                if (T[k] > 0.5f && test_T <= 0.5f) {
                    const float dx = -dxm, dy = -dym;  // pixel - mean
                    depth[k] = rB.w + rC.x * dx + rC.y * dy;
                }
                T[k] = test_T;
                last_j[k] = j;
                if (test_T < 0.0001f) end[k] = true;
            }
        }
        done = end[0] && end[1];
    };
    auto round_end = [&]() {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (last_j[k] >= 0) last[k] = (uint32_t)__float_as_int(ws.E[last_j[k]].y) + 1u;
            last_j[k] = -1;
        }
    };
    walk_list<false, kMasksNone, kStageNone, 8>(a, ws, blk.list0, blk.n, (float)blk.x0, (float)blk.y0, xf,
                                                (float)blk.y[0], done, blend, round_end);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (!blk.inside[k]) continue;
        const size_t p = (size_t)blk.y[k] * a.W + blk.x;
        a.final_T[p] = T[k];
        a.n_contrib[p] = last[k];
        cr[k] += T[k] * a.bg[0];
        cg[k] += T[k] * a.bg[1];
        cb[k] += T[k] * a.bg[2];
        a.color[3 * p] = cr[k];
        a.color[3 * p + 1] = cg[k];
        a.color[3 * p + 2] = cb[k];
        a.depth[p] = depth[k];
        a.color_err[3 * p] = cr[k] - a.obs_rgb[3 * p];
        a.color_err[3 * p + 1] = cg[k] - a.obs_rgb[3 * p + 1];
        a.color_err[3 * p + 2] = cb[k] - a.obs_rgb[3 * p + 2];
    }
}

// Sum of 12 values over the warp: the lane whose bit 0 is clear and whose
// slot() is below 12 returns the sum of v[slot()].
struct WarpSum12 {
    // bit 4 picks a half, bit 3 a quarter, bits 2 and 1 one of three
    static __device__ __forceinline__ int slot(int lane) {
        const int k = ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
        return (lane & 1) || k > 2 ? 12 : ((lane >> 4) & 1) * 6 + ((lane >> 3) & 1) * 3 + k;
    }
    static __device__ __forceinline__ float run(const float (&v)[12], int lane) {
        float a[6], b[4], c[2];
        const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4, h1 = lane & 2;
#pragma unroll
        for (int k = 0; k < 6; ++k) a[k] = (h4 ? v[k + 6] : v[k]) + __shfl_xor_sync(kFullMask, h4 ? v[k] : v[k + 6], 16);
#pragma unroll
        for (int k = 0; k < 3; ++k) b[k] = (h3 ? a[k + 3] : a[k]) + __shfl_xor_sync(kFullMask, h3 ? a[k] : a[k + 3], 8);
        b[3] = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) c[k] = (h2 ? b[k + 2] : b[k]) + __shfl_xor_sync(kFullMask, h2 ? b[k] : b[k + 2], 4);
        const float d = (h1 ? c[1] : c[0]) + __shfl_xor_sync(kFullMask, h1 ? c[0] : c[1], 2);
        return d + __shfl_xor_sync(kFullMask, d, 1);
    }
};

// Backward pass.  n_max: list entries that receive gradients.  What bounds it:
// issue -- about 60 instructions of gradient a pixel and 55 of warp sum for a
// visited block and Gaussian (one pixel a lane: 437 us).  1 M Gaussians, 1280x720: 360 us, before (a lane per
// Gaussian, pixels passed from lane to lane in list order, one step per pixel
// and bucket of 32 entries whether they meet or not) 652.
__global__ void __launch_bounds__(64, 8) map_backward_kernel(MapArgs a, int n_max) {
    pdl_begin();
    __shared__ WarpStage<0> stage[2];
    WarpStage<0>& ws = stage[threadIdx.x >> 5];
    const MapBlock blk(a);
    const int lane = threadIdx.x & 31, slot = WarpSum12::slot(lane);
    const float xf = (float)blk.x;
    uint32_t nc[2] = {0u, 0u};
    float4 pc[2], pe[2];             // final colour and depth; colour error, observed depth
    float T[2], a0[2], a1[2], a2[2];  // this pass's state
    float Tf[2], f0[2], f1[2], f2[2];  // the forward pass's state
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        pc[k] = pe[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (blk.inside[k]) {
            const size_t p = (size_t)blk.y[k] * a.W + blk.x;
            nc[k] = a.n_contrib[p];
            pc[k] = make_float4(a.color[3 * p], a.color[3 * p + 1], a.color[3 * p + 2], a.depth[p]);
            pe[k] = make_float4(a.color_err[3 * p], a.color_err[3 * p + 1], a.color_err[3 * p + 2], a.obs_depth[p]);
        }
        T[k] = Tf[k] = 1.f;
        a0[k] = a1[k] = a2[k] = f0[k] = f1[k] = f2[k] = 0.f;
    }
    const uint32_t nc_max = max(nc[0], nc[1]);
    const int n = min(min(blk.n, n_max), (int)__reduce_max_sync(kFullMask, nc_max));
    const float w_depth = a.w_depth, w_dist = a.w_dist;
    bool done = nc_max == 0;
    auto grad = [&](int j, const float4& rA, const float4& rB, float dx, float dy0, float l00, float l01, float v0,
                    float raw0) {
        const float2 rE = ws.E[j];
        const float dy1 = rA.y - (float)blk.y[1];
        float l10, l11;
        const float v1 = conic_form(rA.z, rA.w, rB.x, dx, dy1, l10, l11);
        const float al[2] = {fminf(0.99f, raw0), fminf(0.99f, gauss_weight(rB.z, v1))};
        const uint32_t li = (uint32_t)__float_as_int(rE.y);
        // (the entry that fills up an odd count has v > rB.y, whatever its list index)
        const bool on[2] = {li < nc[0] && !(v0 > rB.y || al[0] < kInv255), li < nc[1] && !(v1 > rB.y || al[1] < kInv255)};
        const uint32_t hit0 = __ballot_sync(kFullMask, on[0]), hit1 = __ballot_sync(kFullMask, on[1]);
        if (rB.y != -INFINITY && li >= nc_max) done = true;
        if ((hit0 | hit1) == 0u) return;
        const float4 rC = ws.C[j];
        float s[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) s[k] = 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (on[k]) {
                const float alpha = al[k], dy = k ? dy1 : dy0;
                float d0 = rC.z * T[k], d1 = rC.w * T[k], d2 = rE.x * T[k];
                a0[k] += d0 * alpha;
                a1[k] += d1 * alpha;
                a2[k] += d2 * alpha;
                const float inv1m = rcp_approx(1.0f - alpha);
                d0 = (d0 - (pc[k].x - a0[k]) * inv1m) * -pe[k].x;
                d1 = (d1 - (pc[k].y - a1[k]) * inv1m) * -pe[k].y;
                d2 = (d2 - (pc[k].z - a2[k]) * inv1m) * -pe[k].z;
                const float aG = alpha * (d0 + d1 + d2);
                const float aT = alpha * T[k];
                const float haG = 0.5f * aG;
                const float test_T = T[k] * (1.0f - alpha);
                const float di = rB.w + dx * rC.x + dy * rC.y;
                float dc = w_dist * alpha * T[k] * (di - pc[k].w);
                if (T[k] > 0.5f && test_T <= 0.5f) {
                    const float derr = (pe[k].w > 0.1f) ? (pc[k].w - pe[k].w) : 0.0f;
                    dc += w_depth * derr;
                }
                s[0] -= aG * (k ? l10 : l00) + dc * rC.x;
                s[1] -= aG * (k ? l11 : l01) + dc * rC.y;
                s[2] -= haG * dx * dx;
                s[3] -= haG * dx * dy;
                s[4] -= haG * dy * dy;
                s[5] -= aT * pe[k].x;
                s[6] -= aT * pe[k].y;
                s[7] -= aT * pe[k].z;
                s[8] -= dc;
                s[9] -= aG;
                s[10] -= dc * dx;
                s[11] -= dc * dy;
                T[k] = test_T;
                if ((k ? v1 : v0) > 0.0f) {
                    f0[k] += Tf[k] * alpha * rC.z;
                    f1[k] += Tf[k] * alpha * rC.w;
                    f2[k] += Tf[k] * alpha * rE.x;
                    Tf[k] *= 1.0f - alpha;
                }
            }
        }
        const float sum = WarpSum12::run(s, lane);
        float* D = a.delta2d + (size_t)ws.G[j] * 16;
        if (slot < 12) atomicAdd(D + slot, sum);
        if (lane == 31) atomicAdd(reinterpret_cast<uint32_t*>(D + 12), (uint32_t)(__popc(hit0) + __popc(hit1)));
    };
    auto round_end = [&]() {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            T[k] = Tf[k];
            a0[k] = f0[k];
            a1[k] = f1[k];
            a2[k] = f2[k];
        }
    };
    walk_list<false, kMasksSecond, kStageIndex, 8>(a, ws, blk.list0, n, (float)blk.x0, (float)blk.y0, xf,
                                                   (float)blk.y[0], done, grad, round_end);
}

// ----------------------- 2D -> 3D chain rule + Adam ------------------------
struct Q4 {
    float x, y, z, w;
};
// Eigen's quaternion-vector product: uv = 2 vec x v; v + w uv + vec x uv.
__device__ __forceinline__ float3 qapply(const Q4& q, float3 v) {
    float3 uv = make_float3(q.y * v.z - q.z * v.y, q.z * v.x - q.x * v.z, q.x * v.y - q.y * v.x);
    uv.x += uv.x;
    uv.y += uv.y;
    uv.z += uv.z;
    const float3 c = make_float3(q.y * uv.z - q.z * uv.y, q.z * uv.x - q.x * uv.z, q.x * uv.y - q.y * uv.x);
    return make_float3(v.x + q.w * uv.x + c.x, v.y + q.w * uv.y + c.y, v.z + q.w * uv.z + c.z);
}
__device__ __forceinline__ void qmat(const Q4& q, float R[3][3]) {
    const float tx = 2 * q.x, ty = 2 * q.y, tz = 2 * q.z;
    const float twx = tx * q.w, twy = ty * q.w, twz = tz * q.w;
    const float txx = tx * q.x, txy = ty * q.x, txz = tz * q.x;
    const float tyy = ty * q.y, tyz = tz * q.y, tzz = tz * q.z;
    R[0][0] = 1 - (tyy + tzz); R[0][1] = txy - twz; R[0][2] = txz + twy;
    R[1][0] = txy + twz; R[1][1] = 1 - (txx + tzz); R[1][2] = tyz - twx;
    R[2][0] = txz - twy; R[2][1] = tyz + twx; R[2][2] = 1 - (txx + tyy);
}
__device__ __forceinline__ void mm3(const float A[3][3], const float B[3][3], float C[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) C[i][j] = A[i][0] * B[0][j] + A[i][1] * B[1][j] + A[i][2] * B[2][j];
}

__device__ __forceinline__ float adam_step(float& m, float& v, float g, float eta, float a1, float b1, float b1t,
                                           float a2, float b2, float b2t, float eps) {
    m = a1 * g + b1 * m;
    v = a2 * g * g + b2 * v;
    return eta * (b1t * m) * rsqrtf(b2t * v + eps);
}

// One Gaussian with a gradient (nn contributing pixels).
__device__ __forceinline__ void update_one(const MapUpdateArgs& a, int i) {
    const float4* D4 = reinterpret_cast<const float4*>(a.delta2d + (size_t)i * 16);
    const uint32_t nn = __float_as_uint(D4[3].x);
    if (nn == 0) return;
    const float4 q0 = D4[0], q1 = D4[1], q2 = D4[2];
    const float d_mean[2] = {q0.x, q0.y};
    const float d_inv[3] = {q0.z, q0.w, q1.x};
    const float d_col[3] = {q1.y, q1.z, q1.w};
    const float d_depth = q2.x, d_alpha = q2.y;
    const float d_ph[2] = {q2.z, q2.w};
    const float eta_n = 1.0f / (5.0f + (float)nn);
    const float fx = a.K.fx, fy = a.K.fy;
    const DevPose* P = a.pose;
    const Q4 qcw{P->q[0], P->q[1], P->q[2], P->q[3]};
    const float n2q = qcw.x * qcw.x + qcw.y * qcw.y + qcw.z * qcw.z + qcw.w * qcw.w;
    const Q4 qinv = (n2q > 0.f) ? Q4{-qcw.x / n2q, -qcw.y / n2q, -qcw.z / n2q, qcw.w / n2q} : Q4{0, 0, 0, 0};
    float Rcw[3][3];
    qmat(qinv, Rcw);
    const float4 pw = a.pos[i];
    const float4 sw = a.scale[i];
    const float4 rw = a.rot[i];
    float4 cw = a.col[i];
    const float3 mc = qapply(qinv, make_float3(pw.x - P->t[0], pw.y - P->t[1], pw.z - P->t[2]));
    const float z = mc.z;
    const float J[3][3] = {{fx / z, 0.f, -fx * mc.x / (z * z)}, {0.f, fy / z, -fy * mc.y / (z * z)}, {0.f, 0.f, 1.f}};
    const Q4 qg{rw.x, rw.y, rw.z, rw.w};
    float Rg[3][3];
    qmat(qg, Rg);
    const float s[3] = {sw.x, sw.y, sw.z};
    float Tm[3][3], RS[3][3], M[3][3], Sp[3][3];
    mm3(J, Rcw, Tm);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) RS[r][c] = Rg[r][c] * s[c];
    mm3(Tm, RS, M);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) Sp[r][c] = M[r][0] * M[c][0] + M[r][1] * M[c][1] + M[r][2] * M[c][2];
    // 3x3 inverse by cofactors
    float Spi[3][3];
    {
        const float c00 = Sp[1][1] * Sp[2][2] - Sp[1][2] * Sp[2][1];
        const float c01 = Sp[1][2] * Sp[2][0] - Sp[1][0] * Sp[2][2];
        const float c02 = Sp[1][0] * Sp[2][1] - Sp[1][1] * Sp[2][0];
        const float id = 1.0f / (Sp[0][0] * c00 + Sp[0][1] * c01 + Sp[0][2] * c02);
        Spi[0][0] = c00 * id;
        Spi[1][0] = c01 * id;
        Spi[2][0] = c02 * id;
        Spi[0][1] = (Sp[0][2] * Sp[2][1] - Sp[0][1] * Sp[2][2]) * id;
        Spi[1][1] = (Sp[0][0] * Sp[2][2] - Sp[0][2] * Sp[2][0]) * id;
        Spi[2][1] = (Sp[0][1] * Sp[2][0] - Sp[0][0] * Sp[2][1]) * id;
        Spi[0][2] = (Sp[0][1] * Sp[1][2] - Sp[0][2] * Sp[1][1]) * id;
        Spi[1][2] = (Sp[0][2] * Sp[1][0] - Sp[0][0] * Sp[1][2]) * id;
        Spi[2][2] = (Sp[0][0] * Sp[1][1] - Sp[0][1] * Sp[1][0]) * id;
    }
    float3 tmp;
    tmp.x = J[0][0] * d_mean[0] + J[1][0] * d_mean[1] + d_depth * (mc.x / z);
    tmp.y = J[0][1] * d_mean[0] + J[1][1] * d_mean[1] + d_depth * (mc.y / z);
    tmp.z = J[0][2] * d_mean[0] + J[1][2] * d_mean[1] + d_depth;
    float3 dmu3 = qapply(qcw, tmp);
    const float n2 = mc.x * mc.x + mc.y * mc.y + mc.z * mc.z;
    const float nm = sqrtf(n2);
    const float in3 = 1.0f / (n2 * nm);
    {
        const float fac = (Spi[2][0] * d_ph[0] + Spi[2][1] * d_ph[1]) / Spi[2][2];
        const float3 w = qapply(qcw, make_float3(-mc.x * mc.z * in3 * fac, -mc.y * mc.z * in3 * fac,
                                                 (mc.x * mc.x + mc.y * mc.y) * in3 * fac));
        dmu3.x += w.x;
        dmu3.y += w.y;
        dmu3.z += w.z;
    }
    const float sxx = Sp[0][0] + 0.001f, sxy = Sp[1][0], syy = Sp[1][1] + 0.001f;
    const float den = sxx * syy - sxy * sxy;
    const float d2i = 1.0f / ((den * den) + 0.0000001f);
    const float dSxx = d2i * (-syy * syy * d_inv[0] + 2 * sxy * syy * d_inv[1] + (den - sxx * syy) * d_inv[2]);
    const float dSyy = d2i * (-sxx * sxx * d_inv[2] + 2 * sxx * sxy * d_inv[1] + (den - sxx * syy) * d_inv[0]);
    const float dSxy = d2i * 2 * (sxy * syy * d_inv[0] - (den + 2 * sxy * sxy) * d_inv[1] + sxx * sxy * d_inv[2]);
    float S3[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) S3[r][c] = RS[r][0] * RS[c][0] + RS[r][1] * RS[c][1] + RS[r][2] * RS[c][2];
    float dT[2][3];
#pragma unroll
    for (int jj = 0; jj < 3; ++jj) {
        const float t0 = Tm[0][0] * S3[jj][0] + Tm[0][1] * S3[jj][1] + Tm[0][2] * S3[jj][2];
        const float t1 = Tm[1][0] * S3[jj][0] + Tm[1][1] * S3[jj][1] + Tm[1][2] * S3[jj][2];
        dT[0][jj] = 2 * t0 * dSxx + t1 * dSxy;
        dT[1][jj] = 2 * t1 * dSyy + t0 * dSxy;
    }
    const float zt = z / nm;
    const float av = 0.5f * zt * d_ph[0] / Spi[2][2];
    const float bv = 0.5f * zt * d_ph[1] / Spi[2][2];
    const float cv = -zt * (d_ph[0] * Spi[2][0] + d_ph[1] * Spi[2][1]) / (Spi[2][2] * Spi[2][2]);
    const float dLSi[3][3] = {{0.f, 0.f, av}, {0.f, 0.f, bv}, {av, bv, cv}};
    float t1m[3][3], dSp[3][3];
    mm3(Spi, dLSi, t1m);
    mm3(t1m, Spi, dSp);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) dSp[r][c] = -dSp[r][c];
    float TS[3][3];
    mm3(Tm, S3, TS);
#pragma unroll
    for (int aa = 0; aa < 2; ++aa)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
            float s1 = 0.f, s2 = 0.f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                s1 += TS[k][jj] * dSp[k][aa];
                // (S3 T^T)[jj][k] = S3 row jj . T row k
                s2 += (S3[jj][0] * Tm[k][0] + S3[jj][1] * Tm[k][1] + S3[jj][2] * Tm[k][2]) * dSp[aa][k];
            }
            dT[aa][jj] += s1 + s2;
        }
    const float dJ00 = Rcw[0][0] * dT[0][0] + Rcw[0][1] * dT[0][1] + Rcw[0][2] * dT[0][2];
    const float dJ02 = Rcw[2][0] * dT[0][0] + Rcw[2][1] * dT[0][1] + Rcw[2][2] * dT[0][2];
    const float dJ11 = Rcw[1][0] * dT[1][0] + Rcw[1][1] * dT[1][1] + Rcw[1][2] * dT[1][2];
    const float dJ12 = Rcw[2][0] * dT[1][0] + Rcw[2][1] * dT[1][1] + Rcw[2][2] * dT[1][2];
    const float iz = 1.0f / z, iz2 = iz * iz, iz3 = iz2 * iz;
    {
        const float3 w = qapply(qcw, make_float3(-fx * iz2 * dJ02, -fy * iz2 * dJ12,
                                                 -fx * iz2 * dJ00 - fy * iz2 * dJ11 + (2 * fx * mc.x) * iz3 * dJ02 +
                                                     (2 * fy * mc.y) * iz3 * dJ12));
        dmu3.x += w.x;
        dmu3.y += w.y;
        dmu3.z += w.z;
    }
    float dS3[3][3];
    dS3[0][0] = Tm[0][0] * Tm[0][0] * dSxx + Tm[0][0] * Tm[1][0] * dSxy + Tm[1][0] * Tm[1][0] * dSyy;
    dS3[1][1] = Tm[0][1] * Tm[0][1] * dSxx + Tm[0][1] * Tm[1][1] * dSxy + Tm[1][1] * Tm[1][1] * dSyy;
    dS3[2][2] = Tm[0][2] * Tm[0][2] * dSxx + Tm[0][2] * Tm[1][2] * dSxy + Tm[1][2] * Tm[1][2] * dSyy;
    dS3[1][0] = dS3[0][1] = Tm[0][0] * Tm[0][1] * dSxx + 0.5f * (Tm[0][0] * Tm[1][1] + Tm[0][1] * Tm[1][0]) * dSxy +
                            Tm[1][0] * Tm[1][1] * dSyy;
    dS3[2][0] = dS3[0][2] = Tm[0][0] * Tm[0][2] * dSxx + 0.5f * (Tm[0][0] * Tm[1][2] + Tm[0][2] * Tm[1][0]) * dSxy +
                            Tm[1][0] * Tm[1][2] * dSyy;
    dS3[2][1] = dS3[1][2] = Tm[0][2] * Tm[0][1] * dSxx + 0.5f * (Tm[0][1] * Tm[1][2] + Tm[0][2] * Tm[1][1]) * dSxy +
                            Tm[1][1] * Tm[1][2] * dSyy;
    {
        float TtD[3][3], add[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) TtD[r][c] = Tm[0][r] * dSp[0][c] + Tm[1][r] * dSp[1][c] + Tm[2][r] * dSp[2][c];
        mm3(TtD, Tm, add);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) dS3[r][c] += add[r][c];
    }
    float dM[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) dM[r][c] = 2.0f * (RS[0][r] * dS3[0][c] + RS[1][r] * dS3[1][c] + RS[2][r] * dS3[2][c]);
    float dLds[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) dLds[k] = Rg[0][k] * dM[k][0] + Rg[1][k] * dM[k][1] + Rg[2][k] * dM[k][2];
    {
        const float ms = (s[0] + s[1] + s[2]) / 3.f;
        const float l0 = s[0] - ms, l1 = s[1] - ms, l2 = s[2] - ms;
        const float li = a.lambda_iso * (1.f / 3.f);
        dLds[0] -= li * (2.f * l0 - l1 - l2);
        dLds[1] -= li * (-l0 + 2.f * l1 - l2);
        dLds[2] -= li * (-l0 - l1 + 2.f * l2);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) dM[r][c] *= s[r];
    float th0 = 0.f, th1 = 0.f, th2 = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float b0 = dM[0][r], b1 = dM[1][r], b2 = dM[2][r];
        th0 += Rg[r][1] * b2 - Rg[r][2] * b1;
        th1 += Rg[r][2] * b0 - Rg[r][0] * b2;
        th2 += Rg[r][0] * b1 - Rg[r][1] * b0;
    }
    float d3[14];
    d3[0] = eta_n * dmu3.x;
    d3[1] = eta_n * dmu3.y;
    d3[2] = eta_n * dmu3.z;
    d3[3] = eta_n * dLds[0];
    d3[4] = eta_n * dLds[1];
    d3[5] = eta_n * dLds[2];
    d3[6] = -eta_n * th0;
    d3[7] = -eta_n * th1;
    d3[8] = -eta_n * th2;
    d3[9] = d_col[0] * eta_n;
    d3[10] = d_col[1] * eta_n;
    d3[11] = d_col[2] * eta_n;
    d3[12] = d_alpha * eta_n;
    d3[13] = (float)nn;
    if (a.dbg_delta3d) {
        for (int k = 0; k < 14; ++k) a.dbg_delta3d[(size_t)i * 16 + k] = d3[k];
        a.dbg_delta3d[(size_t)i * 16 + 14] = 0.f;
        a.dbg_delta3d[(size_t)i * 16 + 15] = 0.f;
    }

    // --------------------------------- Adam ---------------------------------
    // state planes (float4 per Gaussian): 0 m_pos,1 v_pos,2 m_scl,3 v_scl,
    // 4 m_rot,5 v_rot,6 m_col,7 v_col,8 (m_alpha, v_alpha, k, -)
    float4* S = a.adam;
    const size_t NN = (size_t)a.cap;
    float4 mp = S[0 * NN + i], vp = S[1 * NN + i], ms = S[2 * NN + i], vs = S[3 * NN + i];
    float4 mr = S[4 * NN + i], vr = S[5 * NN + i], mcl = S[6 * NN + i], vcl = S[7 * NN + i];
    float4 mal = S[8 * NN + i];
    mal.z += 1.f;
    const float b1 = a.beta1, b2 = a.beta2, eps = a.eps, eta = a.eta;
    const float a1 = 1.f - b1, a2 = 1.f - b2;
    const float b1t = 1.0f / (1.f - powf(b1, mal.z));
    const float b2t = 1.0f / (1.f - powf(b2, mal.z));
    float4 np = pw;
    np.x += adam_step(mp.x, vp.x, d3[0], eta, a1, b1, b1t, a2, b2, b2t, eps);
    np.y += adam_step(mp.y, vp.y, d3[1], eta, a1, b1, b1t, a2, b2, b2t, eps);
    np.z += adam_step(mp.z, vp.z, d3[2], eta, a1, b1, b1t, a2, b2, b2t, eps);
    const float dq0 = adam_step(mr.x, vr.x, d3[6], eta, a1, b1, b1t, a2, b2, b2t, eps);
    const float dq1 = adam_step(mr.y, vr.y, d3[7], eta, a1, b1, b1t, a2, b2, b2t, eps);
    const float dq2 = adam_step(mr.z, vr.z, d3[8], eta, a1, b1, b1t, a2, b2, b2t, eps);
    float4 nr;
    {
        const float bx = 0.5f * dq0, by = 0.5f * dq1, bz = 0.5f * dq2;
        float x = rw.w * bx + rw.x + (rw.y * bz - rw.z * by);
        float y = rw.w * by + rw.y + (rw.z * bx - rw.x * bz);
        float zq = rw.w * bz + rw.z + (rw.x * by - rw.y * bx);
        float w = rw.w - (rw.x * bx + rw.y * by + rw.z * bz);
        const float nq = sqrtf(x * x + y * y + zq * zq + w * w);
        if (nq > 0.f) {
            const float inq = 1.0f / nq;
            x *= inq;
            y *= inq;
            zq *= inq;
            w *= inq;
        }
        nr = make_float4(x, y, zq, w);
    }
    float4 ns = sw;
    ns.x += adam_step(ms.x, vs.x, d3[3], eta, a1, b1, b1t, a2, b2, b2t, eps);
    ns.y += adam_step(ms.y, vs.y, d3[4], eta, a1, b1, b1t, a2, b2, b2t, eps);
    ns.z += adam_step(ms.z, vs.z, d3[5], eta, a1, b1, b1t, a2, b2, b2t, eps);
    cw.x += adam_step(mcl.x, vcl.x, d3[9], eta, a1, b1, b1t, a2, b2, b2t, eps);
    cw.y += adam_step(mcl.y, vcl.y, d3[10], eta, a1, b1, b1t, a2, b2, b2t, eps);
    cw.z += adam_step(mcl.z, vcl.z, d3[11], eta, a1, b1, b1t, a2, b2, b2t, eps);
    const float dalpha = adam_step(mal.x, mal.y, d3[12], eta, a1, b1, b1t, a2, b2, b2t, eps);
    {
        const float al = cw.w;
        const float as = logf(al / (1.f - al)) + dalpha / (al - al * al);
        cw.w = fmaxf(0.01f, fminf(0.99f, 1.f / (1.f + expf(-as))));
    }
    ns.x = fmaxf(0.001f, ns.x);
    ns.y = fmaxf(0.001f, ns.y);
    ns.z = fmaxf(0.001f, ns.z);
    cw.x = fminf(1.f, fmaxf(0.f, cw.x));
    cw.y = fminf(1.f, fmaxf(0.f, cw.y));
    cw.z = fminf(1.f, fmaxf(0.f, cw.z));
    a.pos[i] = np;
    a.scale[i] = ns;
    a.rot[i] = nr;
    a.col[i] = cw;
    if (a.attr_sr) {
        a.attr_sr[i] = pack_sr(ns, nr);
        a.attr_c[i] = pack_c(cw);
    }
    S[0 * NN + i] = mp;
    S[1 * NN + i] = vp;
    S[2 * NN + i] = ms;
    S[3 * NN + i] = vs;
    S[4 * NN + i] = mr;
    S[5 * NN + i] = vr;
    S[6 * NN + i] = mcl;
    S[7 * NN + i] = vcl;
    S[8 * NN + i] = mal;
}

// A CTA takes kUpdThreads * per Gaussians: first their instance counts, the
// ones with instances queued in shared memory, then the queue with full warps
// -- most of a large map is out of view, so in index order only a few lanes
// of a warp would run the chain rule and Adam.  per spreads a small map over
// all SMs (1) and gives a large one full queues (8).  What bounds it: the
// latency of the queued Gaussians' state (464 bytes each).  1 M Gaussians, 86 k
// in view: 33 us, before (a thread per Gaussian, its gradient count read from
// the 64-byte record) 74.
constexpr int kUpdThreads = 256, kUpdMost = 8;
__global__ void __launch_bounds__(kUpdThreads) map_update_kernel(MapUpdateArgs a, int per, const DevStatus* st) {
    pdl_begin();
    __shared__ uint32_t q_i[kUpdThreads * kUpdMost];
    __shared__ int q_n;
    const int t = threadIdx.x, lane = t & 31;
    if (blockIdx.x == 0 && t < a.n_cst && a.cst) a.cst[t].valid = 0;
    // After an instance overflow, or where a tile's list was not written, the
    // host repeats the step or reports the error: the parameters stay untouched.
    if (st->flags) return;
    if (t == 0) q_n = 0;
    __syncthreads();
    const int base = blockIdx.x * kUpdThreads * per;
    uint32_t c[kUpdMost];
#pragma unroll
    for (int k = 0; k < kUpdMost; ++k) {
        const int i = base + k * kUpdThreads + t;
        c[k] = k < per && i < a.n ? a.counts[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kUpdMost; ++k) {
        const int i = base + k * kUpdThreads + t;
        const uint32_t bal = __ballot_sync(kFullMask, c[k] != 0u);
        if (bal) {
            int slot = 0;
            if (lane == 0) slot = atomicAdd(&q_n, __popc(bal));
            slot = __shfl_sync(kFullMask, slot, 0) + __popc(bal & lanemask_lt());
            if (c[k]) q_i[slot] = (uint32_t)i;
        }
        if (a.dbg_delta3d && k < per && i < a.n)
            for (int w = 0; w < 16; ++w) a.dbg_delta3d[(size_t)i * 16 + w] = 0.f;
    }
    __syncthreads();
    const int n = q_n;
    for (int k = t; k < n; k += kUpdThreads) update_one(a, (int)q_i[k]);
}

cudaError_t launch_map_forward(const MapArgs& a, cudaStream_t s) {
    return launch_chained(map_forward_kernel, dim3(2 * a.ntx * a.nty), dim3(64), 0, s, a);
}

cudaError_t launch_map_backward(const MapArgs& a, bool cap, cudaStream_t s) {
    return launch_chained(map_backward_kernel, dim3(2 * a.ntx * a.nty), dim3(64), 0, s, a,
                          cap ? kMapCap : 0x7fffffff);
}

cudaError_t launch_map_update(const MapUpdateArgs& a, const DevStatus* st, int num_sms, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    // two CTAs an SM: as many Gaussians each as fill them once
    const int per = std::max(1, std::min(kUpdMost, a.n / (2 * num_sms * kUpdThreads)));
    const int chunk = per * kUpdThreads;
    return launch_chained(map_update_kernel, dim3((a.n + chunk - 1) / chunk), dim3(kUpdThreads), 0, s, a, per, st);
}

__global__ void pack_reduced_kernel(const float4* __restrict__ scale, const float4* __restrict__ rot,
                                    const float4* __restrict__ col, uint32_t n, uint4* __restrict__ sr,
                                    uint2* __restrict__ c) {
    pdl_begin();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    sr[i] = pack_sr(scale[i], rot[i]);
    c[i] = pack_c(col[i]);
}

cudaError_t launch_pack_reduced(const float4* scale, const float4* rot, const float4* col, uint32_t n, uint4* sr,
                                uint2* c, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    return launch_chained(pack_reduced_kernel, dim3((n + 255) / 256), dim3(256), 0, s, scale, rot, col, n, sr, c);
}

}  // namespace fvgs
