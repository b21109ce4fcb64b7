// pose_derivs.cuh -- derivatives of a Gaussian's screen-space quantities with
// respect to the camera pose (analytic pose Jacobian).
#pragma once

#include "fvgs_device.cuh"

namespace fvgs {

// Derivatives of one Gaussian's screen mean (u, v) and consumed conic slots
// (a, b, c) with respect to the camera-frame pose update delta = (dp_c,
// dtheta): t' = t + R dp_c, R' = R exp(dtheta), so d p_cam / d dp_c = -I,
// d p_cam / d dtheta = [p_cam]x and d Sigma_cam / d dtheta_j =
// -[e_j]x Sigma_cam + Sigma_cam [e_j]x.  With J the projection's Jacobian
// (rows J0, J1), M = Sigma_cam J^T and Q = Sigma2D^-1:
//   d Sigma2D = dJ M + (dJ M)^T (+ the rotated-covariance terms
//   2 J0 x M0, J0 x M1 + J1 x M0, 2 J1 x M1 for dtheta), dQ = -Q dSigma2D Q.
// r0, r1: the blending record; g0, g1: the geometry record (camera-frame
// covariance and mean).  out: du, dv, da, db, dc grouped by pairs of pose
// coordinates (2m, 2m + 1), each quantity's pair adjacent (the order the
// tracking kernel reads them in, deriv_pair), then the mean's x, y.
__device__ __forceinline__ void pose_derivs(float fx, float fy, bool swap, const float4& r0, const float4& r1,
                                            const float4& g0, const float4& g1, float4* __restrict__ out) {
    const float z = r0.z, x = g1.z, y = g1.w;
    const float sxx = g0.x, sxy = g0.y, sxz = g0.z, syy = g0.w, syz = g1.x, szz = g1.y;
    const float q00 = r1.x, q01 = swap ? r1.z : r1.y, q11 = swap ? r1.y : r1.z;
    const float iz = __frcp_rn(z), iz2 = iz * iz, iz3 = iz2 * iz;
    // J0 = (j00, 0, j02), J1 = (0, j11, j12)
    const float j00 = fx * iz, j02 = -fx * x * iz2, j11 = fy * iz, j12 = -fy * y * iz2;
    const float m0x = sxx * j00 + sxz * j02, m0y = sxy * j00 + syz * j02, m0z = sxz * j00 + szz * j02;
    const float m1x = sxy * j11 + sxz * j12, m1y = syy * j11 + syz * j12, m1z = syz * j11 + szz * j12;
    // rotated-covariance terms: w00 = 2 J0 x M0, w01 = J0 x M1 + J1 x M0, w11 = 2 J1 x M1
    const float w00[3] = {2.f * (-j02 * m0y), 2.f * (j02 * m0x - j00 * m0z), 2.f * (j00 * m0y)};
    const float w01[3] = {-j02 * m1y + (j11 * m0z - j12 * m0y), (j02 * m1x - j00 * m1z) + j12 * m0x,
                          j00 * m1y - j11 * m0x};
    const float w11[3] = {2.f * (j11 * m1z - j12 * m1y), 2.f * (j12 * m1x), 2.f * (-j11 * m1x)};
    const float qa = q00 * q00, qb = 2.f * q00 * q01, qc = q01 * q01;
    const float qd = q00 * q01, qe = q00 * q11 + q01 * q01, qf = q01 * q11;
    const float qg = 2.f * q01 * q11, qh = q11 * q11;
    float du[6], dv[6], da[6], db[6], dc[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        // d p_cam for tangent direction k
        const float dpx = k == 0 ? -1.f : (k == 4 ? -z : (k == 5 ? y : 0.f));
        const float dpy = k == 1 ? -1.f : (k == 3 ? z : (k == 5 ? -x : 0.f));
        const float dpz = k == 2 ? -1.f : (k == 3 ? -y : (k == 4 ? x : 0.f));
        const float dj00 = -fx * iz2 * dpz;
        const float dj02 = -fx * iz2 * dpx + 2.f * fx * x * iz3 * dpz;
        const float dj11 = -fy * iz2 * dpz;
        const float dj12 = -fy * iz2 * dpy + 2.f * fy * y * iz3 * dpz;
        float ds00 = 2.f * (dj00 * m0x + dj02 * m0z);
        float ds01 = (dj00 * m1x + dj02 * m1z) + (dj11 * m0y + dj12 * m0z);
        float ds11 = 2.f * (dj11 * m1y + dj12 * m1z);
        if (k >= 3) {
            ds00 += w00[k - 3];
            ds01 += w01[k - 3];
            ds11 += w11[k - 3];
        }
        const float dq00 = -(qa * ds00 + qb * ds01 + qc * ds11);
        const float dq01 = -(qd * ds00 + qe * ds01 + qf * ds11);
        const float dq11 = -(qc * ds00 + qg * ds01 + qh * ds11);
        du[k] = j00 * dpx + j02 * dpz;
        dv[k] = j11 * dpy + j12 * dpz;
        da[k] = dq00;
        db[k] = swap ? dq11 : dq01;
        dc[k] = swap ? dq01 : dq11;
    }
    store_pair(out, make_float4(du[0], du[1], dv[0], dv[1]),
               make_float4(da[0], da[1], db[0], db[1]));
    store_pair(out + 2, make_float4(dc[0], dc[1], du[2], du[3]),
               make_float4(dv[2], dv[3], da[2], da[3]));
    store_pair(out + 4, make_float4(db[2], db[3], dc[2], dc[3]),
               make_float4(du[4], du[5], dv[4], dv[5]));
    store_pair(out + 6, make_float4(da[4], da[5], db[4], db[5]),
               make_float4(dc[4], dc[5], x, y));
}

}  // namespace fvgs
