// sphmp_features.cuh — the learned corrector's per-particle features, as an
// accumulator over the neighbours the force pass visits (the force pass of a
// corrected large step also fills the features, so that the neighbours are
// gathered once).
//
// Features of an in-grid fluid particle, from the state after the density pass
// of a step (pos, vel, 1/rho and p, fractions and rest density, g - a of the
// last advance) over its neighbours closer than h. With w = (1 - r^2/h^2)^3,
// g = (1 - r/h)^2, x_ij = x_i - x_j (metres), u = unit x_ij, vs = sqrt(|g| h):
//   0-2  v_i / vs                     3   rho_i / rho0_i - 1
//   4    p_i / (rho0_i vs^2)          5-7 alpha_i
//   8-10 (g - a)_i dt_large / vs      11  sum_fluid w
//   12-14 sum_fluid w x_ij / h        15-17 sum_fluid w (v_j - v_i) / vs
//   18   sum_fluid w (rho_j/rho0_j - rho_i/rho0_i)
//   19   sum_fluid w (p_j - p_i) / (rho0_i vs^2)
//   20-22 sum_fluid w (alpha_j - alpha_i)
//   23-28 sum_fluid w x x^T / h^2 (xx, yy, zz, xy, xz, yz)
//   29-31 sum_fluid g u               32  sum_fluid g (v_j - v_i).u / vs
//   33-35 sum_fluid g ((v_j - v_i) x u) / vs
//   36-38 sum_fluid g (p_i + p_j) u / (rho0_i vs^2)
//   39   fluid neighbours / 32        40  sum_boundary w
//   41-43 sum_boundary w x_ij / h     44  boundary neighbours / 32
//   45-47 sum_fluid g (alpha_j0 - alpha_i0) u
#pragma once

#include "sphmp_internal.h"

namespace sphmp {
namespace dev {

constexpr int kLearnedFeatures = 48;

// Only what the neighbour walk needs stays in registers: the particle's own features
// (0 .. 10) go to memory before it, and the sums take their scale in store().
struct LearnedFeatures {
    float f[kLearnedFeatures];  // 11 .. 47: the sums
    float4 pi, vi, ai;
    float pres_i, reli;

    __device__ __forceinline__ static float pressure_scale(float4 ai, float vs) { return 1.f / (ai.w * vs * vs); }

    // pi, vi, ai, di: this particle's pos4, vel4, alpha4, (1/rho, p); features 0 .. 7 into row
    __device__ __forceinline__ void init(const DevParams& P, float4 pi_, float4 vi_, float4 ai_, float2 di, float vs,
                                         float* row) {
        pi = pi_;
        vi = vi_;
        ai = ai_;
        pres_i = di.y;
        const float rhoi = 1.f / di.x;
        reli = rhoi / ai.w;
        const float ivs = 1.f / vs;
#pragma unroll
        for (int k = 11; k < kLearnedFeatures; k++) f[k] = 0.f;
        float4* out = reinterpret_cast<float4*>(row);
        out[0] = make_float4(vi.x * ivs, vi.y * ivs, vi.z * ivs, reli - 1.f);
        out[1] = make_float4(di.y * pressure_scale(ai, vs), ai.x, P.nphase > 1 ? ai.y : 0.f, P.nphase > 2 ? ai.z : 0.f);
    }

    // neighbour j: pos4, (1/rho, p), vel4, alpha4
    __device__ __forceinline__ void pair(const DevParams& P, const float4 pj, const float2 dj, const float4 vj,
                                         const float4 aj) {
        const float dx = (pi.x - pj.x) * P.ss, dy = (pi.y - pj.y) * P.ss, dz = (pi.z - pj.z) * P.ss;
        const float dsq = dx * dx + dy * dy + dz * dz;
        if (!(dsq < P.r2 && dsq > 0.f)) return;
        const float rinv = rsqrtf(dsq);
        const float q1 = 1.f - dsq * P.ir2, q = 1.f - dsq * rinv * P.ih;
        const float w = q1 * q1 * q1, g = q * q;
        const float wx = w * dx, wy = w * dy, wz = w * dz;
        if (pj.w < 0.f) {  // boundary
            f[40] += w;
            f[41] += wx; f[42] += wy; f[43] += wz;
            f[44] += 1.f / 32.f;
            return;
        }
        const float dvx = vj.x - vi.x, dvy = vj.y - vi.y, dvz = vj.z - vi.z;
        f[11] += w;
        f[12] += wx; f[13] += wy; f[14] += wz;
        f[15] += w * dvx; f[16] += w * dvy; f[17] += w * dvz;
        f[18] += w * (__fdividef(1.f, dj.x * aj.w) - reli);
        f[19] += w * (dj.y - pres_i);
        f[20] += w * (aj.x - ai.x);
        f[21] += w * (P.nphase > 1 ? aj.y - ai.y : 0.f);
        f[22] += w * (P.nphase > 2 ? aj.z - ai.z : 0.f);
        f[23] += wx * dx; f[24] += wy * dy; f[25] += wz * dz;
        f[26] += wx * dy; f[27] += wx * dz; f[28] += wy * dz;
        const float gr = g * rinv, gx = gr * dx, gy = gr * dy, gz = gr * dz;
        f[29] += gx; f[30] += gy; f[31] += gz;
        f[32] += dvx * gx + dvy * gy + dvz * gz;
        f[33] += dvy * gz - dvz * gy;
        f[34] += dvz * gx - dvx * gz;
        f[35] += dvx * gy - dvy * gx;
        const float pp = pres_i + dj.y;
        f[36] += pp * gx; f[37] += pp * gy; f[38] += pp * gz;
        f[39] += 1.f / 32.f;
        const float da = aj.x - ai.x;
        f[45] += da * gx; f[46] += da * gy; f[47] += da * gz;
    }

    // Features 8 .. 47 into row; gi: this particle's aprev4.
    __device__ __forceinline__ void store(const DevParams& P, float4 gi, float vs, float dt_large, float* row) {
        const float ivs = 1.f / vs, ih = P.ih, ih2 = ih * ih, ips = pressure_scale(ai, vs);
        auto scale = [&](int from, int to, float k) {
#pragma unroll
            for (int i = from; i <= to; i++) f[i] *= k;
        };
        f[8] = gi.x * dt_large * ivs; f[9] = gi.y * dt_large * ivs; f[10] = gi.z * dt_large * ivs;
        scale(12, 14, ih);
        scale(15, 17, ivs);
        scale(19, 19, ips);
        scale(23, 28, ih2);
        scale(32, 35, ivs);
        scale(36, 38, ips);
        scale(41, 43, ih);
        float4* out = reinterpret_cast<float4*>(row);
#pragma unroll
        for (int i = 2; i < kLearnedFeatures / 4; i++)
            out[i] = make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
    }
};

// A particle without features (boundary or out of the grid): zeros, id -1.
__device__ __forceinline__ void store_no_features(float* row, int32_t* id) {
    float4* out = reinterpret_cast<float4*>(row);
#pragma unroll
    for (int i = 0; i < kLearnedFeatures / 4; i++) out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    *id = -1;
}

}  // namespace dev
}  // namespace sphmp
