// In-register DFTs of 2..16 points for the mixed-radix FourierTrans kernel (fft_mixed.cu).
// Composite lengths are Cooley-Tukey products of the lengths below them, primes use the conjugate symmetry of
// the roots; every constant is evaluated at compile time from its Taylor series in double.
#pragma once
#include "common.cuh"

namespace cnb_mixed {

constexpr double kPi = 3.14159265358979323846;

// |x| <= pi; the 14th term is below 1e-15 there
__host__ __device__ constexpr double sin_series(double x) {
    double t = x, s = x;
    for (int k = 1; k < 14; ++k) { t *= -x * x / ((2 * k) * (2 * k + 1)); s += t; }
    return s;
}
__host__ __device__ constexpr double cos_series(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 14; ++k) { t *= -x * x / ((2 * k - 1) * (2 * k)); s += t; }
    return s;
}
// cos and sin of 2 pi p / q, angle brought to (-pi, pi]
__host__ __device__ constexpr double root_angle(int p, int q) {
    p %= q;
    return 2.0 * kPi * (2 * p > q ? p - q : p) / q;
}
__host__ __device__ constexpr float root_cos(int p, int q) { return (float) cos_series(root_angle(p, q)); }
__host__ __device__ constexpr float root_sin(int p, int q) { return (float) sin_series(root_angle(p, q)); }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

// v * e^{-2 pi i P / Q}; quarter turns cost nothing
template <int P, int Q> __device__ __forceinline__ float2 rotate(float2 v) {
    constexpr int p = P % Q;
    if constexpr (p == 0) return v;
    else if constexpr (4 * p == Q) return make_float2(v.y, -v.x);
    else if constexpr (2 * p == Q) return make_float2(-v.x, -v.y);
    else if constexpr (4 * p == 3 * Q) return make_float2(-v.y, v.x);
    else {
        constexpr float c = root_cos(p, Q), s = root_sin(p, Q);
        return make_float2(v.x * c + v.y * s, v.y * c - v.x * s);
    }
}

template <int R> __host__ __device__ constexpr int first_factor() {        // the A of R = A * B; 0 for a base length
    return R == 6 ? 2 : R == 8 ? 2 : R == 9 ? 3 : R == 10 ? 2 : R == 12 ? 4 : R == 14 ? 2 : R == 15 ? 3 : R == 16 ? 4 : 0;
}

template <int R> __device__ __forceinline__ void dft(float2 (&v)[R]);

// a += sum_k sum[k] cos(2 pi M k / R), b += sum_k dif[k] sin(2 pi M k / R)
template <int R, int M, int K> struct PrimeTerm {
    static __device__ __forceinline__ void all(const float2 (&sum)[(R - 1) / 2], const float2 (&dif)[(R - 1) / 2], float2& a, float2& b) {
        constexpr float c = root_cos(M * K, R), s = root_sin(M * K, R);
        a.x += sum[K - 1].x * c; a.y += sum[K - 1].y * c;
        b.x += dif[K - 1].x * s; b.y += dif[K - 1].y * s;
        if constexpr (2 * (K + 1) < R) PrimeTerm<R, M, K + 1>::all(sum, dif, a, b);
    }
};

template <int R, int M> struct PrimeOut {
    static __device__ __forceinline__ void all(float2 (&v)[R], float2 v0, const float2 (&sum)[(R - 1) / 2], const float2 (&dif)[(R - 1) / 2]) {
        float2 a = v0, b = make_float2(0.f, 0.f);
        PrimeTerm<R, M, 1>::all(sum, dif, a, b);
        v[M] = make_float2(a.x + b.y, a.y - b.x);                            // a - i b
        v[R - M] = make_float2(a.x - b.y, a.y + b.x);
        if constexpr (2 * (M + 1) < R) PrimeOut<R, M + 1>::all(v, v0, sum, dif);
    }
};

template <int R> __device__ __forceinline__ void dft_prime(float2 (&v)[R]) {
    constexpr int H = (R - 1) / 2;
    float2 sum[H], dif[H];
    float2 z = v[0];
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        sum[k - 1] = make_float2(v[k].x + v[R - k].x, v[k].y + v[R - k].y);
        dif[k - 1] = make_float2(v[k].x - v[R - k].x, v[k].y - v[R - k].y);
        z.x += sum[k - 1].x; z.y += sum[k - 1].y;
    }
    const float2 v0 = v[0];
    v[0] = z;
    PrimeOut<R, 1>::all(v, v0, sum, dif);
}

template <int A, int B, int N2, int K1> struct Twist {
    static __device__ __forceinline__ void all(float2 (&t)[A], float2 (&u)[A][B]) {
        u[K1][N2] = rotate<N2 * K1, A * B>(t[K1]);
        if constexpr (K1 + 1 < A) Twist<A, B, N2, K1 + 1>::all(t, u);
    }
};

template <int A, int B, int N2> struct Columns {
    static __device__ __forceinline__ void all(const float2 (&v)[A * B], float2 (&u)[A][B]) {
        float2 t[A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + N2];
        dft<A>(t);
        Twist<A, B, N2, 0>::all(t, u);
        if constexpr (N2 + 1 < B) Columns<A, B, N2 + 1>::all(v, u);
    }
};

// natural order in and out, sign e^{-2 pi i jk/R}
template <int R> __device__ __forceinline__ void dft(float2 (&v)[R]) {
    if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = make_float2(a.x + b.x, a.y + b.y);
        v[1] = make_float2(a.x - b.x, a.y - b.y);
    } else if constexpr (R == 4) {
        const float2 a = make_float2(v[0].x + v[2].x, v[0].y + v[2].y), b = make_float2(v[0].x - v[2].x, v[0].y - v[2].y);
        const float2 c = make_float2(v[1].x + v[3].x, v[1].y + v[3].y), d = make_float2(v[1].x - v[3].x, v[1].y - v[3].y);
        v[0] = make_float2(a.x + c.x, a.y + c.y);
        v[1] = make_float2(b.x + d.y, b.y - d.x);
        v[2] = make_float2(a.x - c.x, a.y - c.y);
        v[3] = make_float2(b.x - d.y, b.y + d.x);
    } else if constexpr (first_factor<R>() != 0) {
        constexpr int A = first_factor<R>(), B = R / A;
        float2 u[A][B];
        Columns<A, B, 0>::all(v, u);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            dft<B>(u[k1]);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = u[k1][k2];
        }
    } else {
        dft_prime<R>(v);
    }
}

}  // namespace cnb_mixed
