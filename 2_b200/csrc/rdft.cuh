// rdft.cuh -- DFTs of short lengths that are not powers of two, in registers.
//
// An odd prime length P pairs the inputs n and P-n: with s_n = a_n + a_{P-n} and
// d_n = a_n - a_{P-n}, X_k and X_{P-k} are A_k +- i B_k, A_k = a_0 + sum s_n cos(2 pi n k/P),
// B_k = sum d_n sin(2 pi n k/P): (P-1)^2 real multiply-adds where the plain sum takes
// 4 P (P-1).  A composite length A*B is the two-step decomposition
// X[k1 + A k2] = sum_r W_B^(r k2) W_P^(r k1) sum_n a[B n + r] W_A^(n k1).  The constants are
// evaluated at compile time in FP64 from the Taylor series and rounded once.
#pragma once
#include "fft4.cuh"

namespace mmfft {

// cos(2 pi num/den) and sin(2 pi num/den), 0 <= num <= den, at compile time
__host__ __device__ constexpr double turn_series(double x, int first) {
    double term = first ? x : 1.0, sum = term;
    for (int k = first + 1; k < 60; k += 2) {
        term *= -x * x / ((double)k * (double)(k + 1));
        sum += term;
    }
    return sum;
}
template <int P>
struct TurnTable {
    float c[P], s[P];
    __host__ __device__ constexpr TurnTable() : c(), s() {
        for (int n = 0; n < P; n++) {
            // the angle reduced to [-pi, pi]
            const double a = 6.283185307179586476925286766559 * (2 * n > P ? n - P : n) / P;
            c[n] = (float)turn_series(a, 0);
            s[n] = (float)turn_series(a, 1);
        }
    }
};

template <int P, int SIGN>
__device__ __forceinline__ void dft_prime(float2* a) {
    constexpr TurnTable<P> T{};
    constexpr int H = (P - 1) / 2;
    float2 s[H + 1], d[H + 1];
    float2 sum = a[0];
#pragma unroll
    for (int n = 1; n <= H; n++) {
        s[n] = cadd(a[n], a[P - n]);
        d[n] = csub(a[n], a[P - n]);
        sum = cadd(sum, s[n]);
    }
    const float2 a0 = a[0];
    a[0] = sum;
#pragma unroll
    for (int k = 1; k <= H; k++) {
        float2 A = a0, B = make_float2(0.f, 0.f);
#pragma unroll
        for (int n = 1; n <= H; n++) {
            const float c = T.c[(n * k) % P], q = T.s[(n * k) % P];
            A.x += c * s[n].x;
            A.y += c * s[n].y;
            B.x += q * d[n].x;
            B.y += q * d[n].y;
        }
        const float2 iB = mul_si<SIGN>(B);
        a[k] = cadd(A, iB);
        a[P - k] = csub(A, iB);
    }
}

template <int A, int B, int SIGN>
__device__ __forceinline__ void dft_composite(float2* a) {
    constexpr int P = A * B;
    constexpr TurnTable<P> T{};
    float2 t[B][A];
#pragma unroll
    for (int r = 0; r < B; r++) {
#pragma unroll
        for (int n = 0; n < A; n++) t[r][n] = a[B * n + r];
        RDft<A, SIGN>::run(t[r]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
        float2 u[B];
#pragma unroll
        for (int r = 0; r < B; r++) {
            const float c = T.c[(r * k1) % P], q = SIGN > 0 ? T.s[(r * k1) % P] : -T.s[(r * k1) % P];
            u[r] = r * k1 == 0 ? t[r][k1] : cmul(t[r][k1], make_float2(c, q));
        }
        RDft<B, SIGN>::run(u);
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) a[k1 + A * k2] = u[k2];
    }
}

#define MM_RDFT_PRIME(P) \
    template <int SIGN> struct RDft<P, SIGN> { static __device__ __forceinline__ void run(float2* a) { dft_prime<P, SIGN>(a); } };
#define MM_RDFT_COMP(P, A, B) \
    template <int SIGN> struct RDft<P, SIGN> { static __device__ __forceinline__ void run(float2* a) { dft_composite<A, B, SIGN>(a); } };
MM_RDFT_PRIME(3)
MM_RDFT_PRIME(5)
MM_RDFT_PRIME(7)
MM_RDFT_PRIME(11)
MM_RDFT_PRIME(13)
MM_RDFT_COMP(6, 3, 2)
MM_RDFT_COMP(9, 3, 3)
MM_RDFT_COMP(10, 5, 2)
MM_RDFT_COMP(12, 4, 3)
MM_RDFT_COMP(14, 7, 2)
MM_RDFT_COMP(15, 5, 3)
#undef MM_RDFT_PRIME
#undef MM_RDFT_COMP

}  // namespace mmfft
