// The Hasimoto/RPY Green's function of the wave-space mobility on the spectra
// of the 11 real grids (Mobility_WaveSpace_Green_kernel, Mobility.cu:315).
// Spectra order: X Y Z XX XY XZ YX YY YZ ZX ZY (force then couplet on input,
// velocity then velocity gradient on output).
#pragma once

#include <cuda_runtime.h>

namespace fsd {

// Scalar factors of the operator at one wave vector: uf scales the
// (I - kk) F and (with the imaginary unit) df the force-gradient couplings,
// dc the couplet's velocity gradient; ik2 = 1 / k^2.
struct GreenFactors {
    float uf, df, dc, ik2;
};

__device__ __forceinline__ GreenFactors green_factors(const float4 tk) {
    const float ksq = tk.x * tk.x + tk.y * tk.y + tk.z * tk.z;
    const float k = sqrtf(ksq);
    const float sk = sinf(k), ck = cosf(k);
    const float j0 = sk / k;
    const float j1k = (sk - k * ck) / (ksq * k);
    GreenFactors g;
    g.uf = tk.w * j0 * j0;
    g.df = (float)((double)(tk.w * j0) * (3.0 * (double)(sk - k * ck) / (double)(ksq * k)));
    g.dc = (float)((double)tk.w * 9.0 * (double)j1k * (double)j1k);
    g.ik2 = 1.0f / ksq;
    return g;
}

// o = operator(k) f.  sgn = +1 applies the operator at k; sgn = -1 conjugates
// its imaginary-unit couplings (used to average with the mirror point on
// Nyquist planes).
__device__ __forceinline__ void green_apply(const float kx, const float ky, const float kz, const GreenFactors g,
                                            const float2* f, float2* o, float sgn) {
    const float2 fX = f[0], fY = f[1], fZ = f[2];
    const float2 cXX = f[3], cXY = f[4], cXZ = f[5], cYX = f[6], cYY = f[7], cYZ = f[8], cZX = f[9], cZY = f[10];
    const float2 cZZ = make_float2(-(cXX.x + cYY.x), -(cXX.y + cYY.y));
    const float2 kdF = make_float2((kx * fX.x + ky * fY.x + kz * fZ.x) * g.ik2,
                                   (kx * fX.y + ky * fY.y + kz * fZ.y) * g.ik2);
    const float2 Cdkx = make_float2(cXX.x * kx + cXY.x * ky + cXZ.x * kz, cXX.y * kx + cXY.y * ky + cXZ.y * kz);
    const float2 Cdky = make_float2(cYX.x * kx + cYY.x * ky + cYZ.x * kz, cYX.y * kx + cYY.y * ky + cYZ.y * kz);
    const float2 Cdkz = make_float2(cZX.x * kx + cZY.x * ky + cZZ.x * kz, cZX.y * kx + cZY.y * ky + cZZ.y * kz);
    const float2 kdcdk = make_float2((Cdkx.x * kx + Cdky.x * ky + Cdkz.x * kz) * g.ik2,
                                     (Cdkx.y * kx + Cdky.y * ky + Cdkz.y * kz) * g.ik2);
    // UF: (I - kk) F, real scale.
    o[0] = make_float2((fX.x - kx * kdF.x) * g.uf, (fX.y - kx * kdF.y) * g.uf);
    o[1] = make_float2((fY.x - ky * kdF.x) * g.uf, (fY.y - ky * kdF.y) * g.uf);
    o[2] = make_float2((fZ.x - kz * kdF.x) * g.uf, (fZ.y - kz * kdF.y) * g.uf);
    // UC: imaginary scale, minus that of DF.
    const float Bdf = sgn * g.df, Buc = -Bdf;
    o[0].x += -(Cdkx.y - kx * kdcdk.y) * Buc;
    o[1].x += -(Cdky.y - ky * kdcdk.y) * Buc;
    o[2].x += -(Cdkz.y - kz * kdcdk.y) * Buc;
    o[0].y += (Cdkx.x - kx * kdcdk.x) * Buc;
    o[1].y += (Cdky.x - ky * kdcdk.x) * Buc;
    o[2].y += (Cdkz.x - kz * kdcdk.x) * Buc;
    // DF: imaginary scale, D_ab = i B (F_a k_b - k_a k_b k.F/k^2); DC: real scale.
    const float fa[3][2] = {{fX.x, fX.y}, {fY.x, fY.y}, {fZ.x, fZ.y}};
    const float kv[3] = {kx, ky, kz};
    const float2 Cdk[3] = {Cdkx, Cdky, Cdkz};
    const int ia[8] = {0, 0, 0, 1, 1, 1, 2, 2};
    const int ib[8] = {0, 1, 2, 0, 1, 2, 0, 1};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float kk = kv[ia[c]] * kv[ib[c]];
        const float Fkr = fa[ia[c]][0] * kv[ib[c]], Fki = fa[ia[c]][1] * kv[ib[c]];
        o[3 + c] = make_float2(-(Fki - kk * kdF.y) * Bdf + (Cdk[ia[c]].x * kv[ib[c]] - kk * kdcdk.x) * g.dc,
                               (Fkr - kk * kdF.x) * Bdf + (Cdk[ia[c]].y * kv[ib[c]] - kk * kdcdk.y) * g.dc);
    }
}

__device__ __forceinline__ void green_apply(const float4 tk, const float2* f, float2* o, float sgn) {
    green_apply(tk.x, tk.y, tk.z, green_factors(tk), f, o, sgn);
}

// Packed pair p holds spectra (packA(p), packB(p)); compile-time so that the
// unrolled loops keep the spectra in registers.
__host__ __device__ constexpr int packA(int p) { return p == 0 ? 0 : p == 1 ? 3 : p == 2 ? 5 : p == 3 ? 7 : p == 4 ? 9 : 2; }
__host__ __device__ constexpr int packB(int p) { return p == 0 ? 1 : p == 1 ? 4 : p == 2 ? 6 : p == 3 ? 8 : p == 4 ? 10 : -1; }

}  // namespace fsd
