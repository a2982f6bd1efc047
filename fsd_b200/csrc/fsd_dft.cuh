// Small complex DFTs in registers: radices 2, 3, 4 and 5 by their
// factored forms, the composites A*B from them by one Cooley-Tukey step with
// compile-time roots.  INV = false uses exp(-2 pi i / R), true its conjugate.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace fsd {

// cos and sin of 2 pi m / n in double at compile time: the argument is folded
// to [0, pi/4] and the Taylor series summed to the rounding level.
__host__ __device__ constexpr double trig_series(double x, bool sine) {
    double term = sine ? x : 1.0, sum = term;
    for (int k = 1; k < 14; ++k) {
        const double a = 2.0 * k - (sine ? 0.0 : 1.0);
        term *= -x * x / (a * (a + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double cos_turn(int m, int n) {  // cos(2 pi m / n)
    m %= n;
    if (m < 0) m += n;
    if (2 * m > n) m = n - m;                                   // [0, 1/2] turn
    const bool neg = 4 * m > n;                                 // (1/4, 1/2]: -cos(pi - x)
    const double u = neg ? 0.5 - (double)m / n : (double)m / n;  // [0, 1/4] turn
    const double two_pi = 6.283185307179586476925286766559;
    if (4 * m == n) return 0.0;
    const double v = u <= 0.125 ? trig_series(two_pi * u, false) : trig_series(two_pi * (0.25 - u), true);
    return neg ? -v : v;
}
__host__ __device__ constexpr double sin_turn(int m, int n) {  // sin(2 pi m / n) = cos(2 pi (m/n - 1/4))
    return cos_turn(4 * m - n, 4 * n);
}

__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a + s i d with s = +1 or -1 (a compile-time sign)
template <bool PLUS>
__device__ __forceinline__ float2 c_add_i(float2 a, float2 d) {
    return PLUS ? make_float2(a.x - d.y, a.y + d.x) : make_float2(a.x + d.y, a.y - d.x);
}
// a times w (INV: times its conjugate)
template <bool INV>
__device__ __forceinline__ float2 c_twiddle(float2 a, float2 w) {
    return INV ? make_float2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y)
               : make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}

template <int R>
struct DftSplit {  // R = A * B; 0: a base radix
    static constexpr int A = R == 6 ? 2 : R == 8 ? 2 : R == 9 ? 3 : R == 10 ? 2 : R == 12 ? 3 : R == 15 ? 3 : R == 16 ? 4 : 0;
    static constexpr int B = A ? R / A : 0;
};

template <int R, bool INV>
__device__ __forceinline__ void dft(float2* y);

// v times w_R^M (INV: its conjugate)
template <int R, bool INV, int M>
__device__ __forceinline__ float2 root_mul(float2 v) {
    if constexpr (M == 0) {
        return v;
    } else if constexpr (4 * M == R) {  // -i (forward)
        return INV ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
    } else if constexpr (2 * M == R) {
        return make_float2(-v.x, -v.y);
    } else {
        constexpr float c = (float)cos_turn(M, R), s = (float)sin_turn(M, R);
        return INV ? make_float2(v.x * c - v.y * s, v.y * c + v.x * s)
                   : make_float2(v.x * c + v.y * s, v.y * c - v.x * s);
    }
}

// Second step of a composite DFT for one k2: roots w_R^(r k2), then the
// A-point DFT over r.
template <int R, bool INV, int K2, int... r>
__device__ __forceinline__ void dft_column(float2 (*z)[DftSplit<R>::B], float2* y, std::integer_sequence<int, r...>) {
    float2 u[sizeof...(r)] = {root_mul<R, INV, r * K2>(z[r][K2])...};
    dft<(int)sizeof...(r), INV>(u);
    ((y[K2 + DftSplit<R>::B * r] = u[r]), ...);
}
template <int R, bool INV, int... k2>
__device__ __forceinline__ void dft_columns(float2 (*z)[DftSplit<R>::B], float2* y, std::integer_sequence<int, k2...>) {
    (dft_column<R, INV, k2>(z, y, std::make_integer_sequence<int, DftSplit<R>::A>{}), ...);
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2* y) {
    if constexpr (R == 2) {
        const float2 a = y[0], b = y[1];
        y[0] = c_add(a, b);
        y[1] = c_sub(a, b);
    } else if constexpr (R == 3) {
        constexpr float s3 = (float)sin_turn(1, 3);
        const float2 t = c_add(y[1], y[2]);
        float2 d = c_sub(y[1], y[2]);
        d = make_float2(d.x * s3, d.y * s3);
        const float2 a = make_float2(fmaf(-0.5f, t.x, y[0].x), fmaf(-0.5f, t.y, y[0].y));
        y[0] = c_add(y[0], t);
        y[1] = c_add_i<INV>(a, d);
        y[2] = c_add_i<!INV>(a, d);
    } else if constexpr (R == 4) {
        const float2 a = c_add(y[0], y[2]), b = c_sub(y[0], y[2]);
        const float2 c = c_add(y[1], y[3]), d = c_sub(y[1], y[3]);
        y[0] = c_add(a, c);
        y[2] = c_sub(a, c);
        y[1] = c_add_i<INV>(b, d);
        y[3] = c_add_i<!INV>(b, d);
    } else if constexpr (R == 5) {
        constexpr float c1 = (float)cos_turn(1, 5), c2 = (float)cos_turn(2, 5);
        constexpr float s1 = (float)sin_turn(1, 5), s2 = (float)sin_turn(2, 5);
        const float2 t1 = c_add(y[1], y[4]), t2 = c_add(y[2], y[3]);
        const float2 t3 = c_sub(y[1], y[4]), t4 = c_sub(y[2], y[3]);
        const float2 a = make_float2(fmaf(c1, t1.x, fmaf(c2, t2.x, y[0].x)), fmaf(c1, t1.y, fmaf(c2, t2.y, y[0].y)));
        const float2 b = make_float2(fmaf(c2, t1.x, fmaf(c1, t2.x, y[0].x)), fmaf(c2, t1.y, fmaf(c1, t2.y, y[0].y)));
        const float2 d = make_float2(fmaf(s1, t3.x, s2 * t4.x), fmaf(s1, t3.y, s2 * t4.y));
        const float2 e = make_float2(fmaf(s2, t3.x, -s1 * t4.x), fmaf(s2, t3.y, -s1 * t4.y));
        y[0] = c_add(y[0], c_add(t1, t2));
        y[1] = c_add_i<INV>(a, d);
        y[4] = c_add_i<!INV>(a, d);
        y[2] = c_add_i<INV>(b, e);
        y[3] = c_add_i<!INV>(b, e);
    } else {
        // n = r + A s: B-point DFTs over s, roots w_R^(r k2), A-point DFTs over r; k = k2 + B k1
        constexpr int A = DftSplit<R>::A, B = DftSplit<R>::B;
        static_assert(A > 1, "unsupported radix");
        float2 z[A][B];
#pragma unroll
        for (int r = 0; r < A; ++r) {
#pragma unroll
            for (int s = 0; s < B; ++s) z[r][s] = y[r + A * s];
            dft<B, INV>(z[r]);
        }
dft_columns<R, INV>(z, y, std::make_integer_sequence<int, B>{});
    }
}

}  // namespace fsd
