// colmix.cuh -- in-place transforms of many lines at once in shared memory, any length with
// prime factors up to 31: the stages that the column passes (colmix.cu) and the row passes of
// lengths that are not powers of two (mixed.cu, rhs.cu) share.
//
// TC lines lie side by side, [element][line]; a half-warp takes adjacent lines, so no stride
// of a stage causes bank conflicts and the lanes of a line group share their twiddles.
#pragma once
#include "mixed.cuh"
#include "rdft.cuh"

namespace mm {
using namespace mmfft;

constexpr int MC_MAXST = 12;

struct ColPlan {
    int N, NP, nst;
    int r[MC_MAXST];  // radices in the order of the forward stages; the last one is the smallest
    int nq;           // N / r[nst - 1]
    int tws;          // W_L^m = tw[m * tws]
    int big;          // a radix above 10 (the row passes' run-time radix)
    int tc;           // lines per block (TC)
    int sh;           // log2 of TC where it is a power of two
    unsigned rcp;     // 0 there, else ceil(2^32 / TC): element / TC without a division
    int pitch;        // shared-memory distance of a line's elements: TC, odd where rows are transposed
};

// split(e): e = q * TC + line
__device__ __forceinline__ int line_of(const ColPlan& P, int e, int& q) {
    q = P.rcp ? (int)__umulhi((unsigned)e, P.rcp) : e >> P.sh;
    return e - q * P.tc;
}

// a run-time radix 17..31 (prime): the paired sums of dft_prime on a local array, constants
// from the twiddle table (W_R^m = tw[m * step])
template <int SIGN>
__device__ __noinline__ void dft_any(float2* a, int R, const float2* __restrict__ tw, int step) {
    const int H = (R - 1) / 2;
    float2 s[16], d[16];
    float2 sum = a[0];
    for (int n = 1; n <= H; n++) {
        s[n] = cadd(a[n], a[R - n]);
        d[n] = csub(a[n], a[R - n]);
        sum = cadd(sum, s[n]);
    }
    const float2 a0 = a[0];
    a[0] = sum;
    for (int k = 1; k <= H; k++) {
        float2 A = a0, B = make_float2(0.f, 0.f);
        int m = 0;
        for (int n = 1; n <= H; n++) {
            m += k;
            if (m >= R) m -= R;
            const float2 w = tw[m * step];  // cos, -sin
            A.x += w.x * s[n].x;
            A.y += w.x * s[n].y;
            B.x -= w.y * d[n].x;
            B.y -= w.y * d[n].y;
        }
        const float2 iB = mul_si<SIGN>(B);
        a[k] = cadd(A, iB);
        a[R - k] = csub(A, iB);
    }
}

// R = 0: the run-time radix `rad`
template <int R, int SIGN>
__device__ __forceinline__ void dft_r(float2* v, int rad, const ColPlan& P, const float2* __restrict__ tw) {
    if constexpr (R > 0) RDft<R, SIGN>::run(v);
    else dft_any<SIGN>(v, rad, tw, P.NP * P.N / rad * P.tws);
}
template <int R> struct RegLen { static constexpr int n = R > 0 ? R : 31; };

template <int SIGN>
__device__ __forceinline__ float2 tw_l(const ColPlan& P, const float2* __restrict__ tw, int m) {
    const float2 w = __ldg(tw + m * P.tws);
    return SIGN > 0 ? make_float2(w.x, -w.y) : w;
}

#define MC_EACH(r, rad) _Pragma("unroll") for (int r = 0; r < (R > 0 ? R : rad); r++)
#define MC_SWITCH(rad, CALL)                                                                                   \
    switch (rad) {                                                                                             \
        case 1: CALL(1); break;                                                                                \
        case 2: CALL(2); break;                                                                                \
        case 3: CALL(3); break;                                                                                \
        case 4: CALL(4); break;                                                                                \
        case 5: CALL(5); break;                                                                                \
        case 6: CALL(6); break;                                                                                \
        case 7: CALL(7); break;                                                                                \
        case 8: CALL(8); break;                                                                                \
        case 9: CALL(9); break;                                                                                \
        case 10: CALL(10); break;                                                                              \
        case 12: CALL(12); break;                                                                              \
        case 15: CALL(15); break;                                                                              \
        case 16: CALL(16); break;                                                                              \
        default: CALL(0); break;                                                                               \
    }

// The row passes' radices: at most 10, and the run-time radix only in the kernels of lengths that
// need it (BIG): its local array and body cost every other length registers and instruction
// fetches.
#define MC_SWITCH_ROW(rad, CALL)                                                                               \
    switch (rad) {                                                                                             \
        case 1: CALL(1); break;                                                                                \
        case 2: CALL(2); break;                                                                                \
        case 3: CALL(3); break;                                                                                \
        case 4: CALL(4); break;                                                                                \
        case 5: CALL(5); break;                                                                                \
        case 6: CALL(6); break;                                                                                \
        case 7: CALL(7); break;                                                                                \
        case 8: CALL(8); break;                                                                                \
        case 9: CALL(9); break;                                                                                \
        case 10: CALL(10); break;                                                                              \
        default:                                                                                               \
            if constexpr (BIG) { CALL(0); }                                                                    \
            break;                                                                                             \
    }

// ---- a middle stage of sub-blocks of ncur elements (forward, or its mirror image)
template <int R, int SIGN>
__device__ __forceinline__ void mid_stage(const ColPlan& P, int rad, int ncur, float2* sm, int lines,
                                          const float2* __restrict__ tw) {
    const int M = ncur / rad, per = P.N / rad * P.tc, ts = P.N / ncur * P.NP;
    for (int i = threadIdx.x; i < lines * per; i += blockDim.x) {
        const int l = lines == 1 ? 0 : i / per;
        int q;
        const int col = line_of(P, i - l * per, q);
        const int blk = q / M, j = q - blk * M;
        float2* x = sm + (l * P.N + blk * ncur + j) * P.pitch + col;
        float2 v[RegLen<R>::n];
        MC_EACH(r, rad) {
            v[r] = x[r * M * P.pitch];
            if (SIGN > 0 && j * r) v[r] = cmul(v[r], tw_l<+1>(P, tw, j * r * ts));
        }
        dft_r<R, SIGN>(v, rad, P, tw);
        MC_EACH(k, rad) x[k * M * P.pitch] = (SIGN < 0 && j * k) ? cmul(v[k], tw_l<-1>(P, tw, j * k * ts)) : v[k];
    }
}

// frequency of slot q of the last stage's sub-block: digits of q, most significant = stage 0
__device__ __forceinline__ int slot_freq(const ColPlan& P, int q) {
    if (P.nst <= 2) return q;
    int f = 0, rest = P.nq, base = 1;
    for (int s = 0; s < P.nst - 1; s++) {
        rest /= P.r[s];
        const int d = q / rest;
        q -= d * rest;
        f += d * base;
        base *= P.r[s];
    }
    return f;
}

// slot of frequency k after the forward stages
__device__ __forceinline__ int freq_slot(const ColPlan& P, int k) {
    int slot = 0, n = P.N;
    for (int s = 0; s < P.nst; s++) {
        const int d = k % P.r[s];
        k /= P.r[s];
        n /= P.r[s];
        slot += d * n;
    }
    return slot;
}

// The whole transform of the block's TC lines in shared memory: forward (natural order in,
// digit-reversed slots out) or its mirror image.  Synchronises the block after each stage.
// Inlined: as a called function it made every epilogue spill 128-640 bytes at 80 registers, and
// small grids wait for its instructions (256 rows of 192 cells, C2R + epilogue 18.1 -> 14.4 us).
template <int SIGN, bool BIG>
__device__ __forceinline__ void lines_fft(const ColPlan& P, float2* sm, const float2* __restrict__ tw) {
    int ncur = SIGN < 0 ? P.N : 1;
    for (int i = 0; i < P.nst; i++) {
        const int rad = P.r[SIGN < 0 ? i : P.nst - 1 - i];
        if (SIGN > 0) ncur *= rad;
#define CALL(R) mid_stage<R, SIGN>(P, rad, ncur, sm, 1, tw)
        MC_SWITCH_ROW(rad, CALL)
#undef CALL
        if (SIGN < 0) ncur /= rad;
        __syncthreads();
    }
}

// slot[k] of every frequency k < N, filled by the block
__device__ __forceinline__ void fill_slots(const ColPlan& P, unsigned short* slot) {
    for (int k = threadIdx.x; k < P.N; k += blockDim.x) slot[k] = (unsigned short)freq_slot(P, k);
}

// Real-to-complex post-processing of one transformed line (the packed sequence
// x[2n] + i x[2n+1], element e at line[e * pitch]): X[k] = E[k] + W_2M^k O[k], k <= M, to dst,
// for k0, k0 + kstep ... up to M / 2 and their mirror images.
__device__ __forceinline__ void r2c_line(const ColPlan& P, const float2* line, const unsigned short* slot,
                                         const float2* __restrict__ tw2M, int k0, int kstep, float2* dst) {
    const int M = P.N;
    for (int k = k0; k <= M / 2; k += kstep) {
        const float2 zk = line[slot[k] * P.pitch];
        const float2 zm = line[slot[k ? M - k : 0] * P.pitch];
        const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 od = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));  // (Z[k] - conj Z[M-k]) / 2i
        const float2 w = __ldg(tw2M + k);
        dst[k] = cadd(e, cmul(w, od));
        if (k != M - k) dst[M - k] = cadd(cconj(e), cmul(make_float2(-w.x, w.y), cconj(od)));
    }
}

// Complex-to-real pre-processing of one spectrum row, into the slots that the inverse starts
// from: Z[k] = (X[k] + conj X[M-k]) + i W_2M^-k (X[k] - conj X[M-k]), k = k0, k0 + kstep ... < M.
__device__ __forceinline__ void c2r_line(const ColPlan& P, float2* line, const unsigned short* slot,
                                         const float2* __restrict__ tw2M, int k0, int kstep, const float2* src) {
    const int M = P.N;
    for (int k = k0; k < M; k += kstep) {
        const float2 a = src[k], b = src[M - k];
        const float2 s = make_float2(a.x + b.x, a.y - b.y);
        const float2 d = make_float2(a.x - b.x, a.y + b.y);
        const float2 w0 = __ldg(tw2M + k);
        const float2 wd = cmul(make_float2(w0.x, -w0.y), d);
        line[slot[k] * P.pitch] = make_float2(s.x - wd.y, s.y + wd.x);
    }
}

// shared memory of tc transposed lines of length M with their slot table
inline size_t lines_smem(int M, int tc) {
    return (size_t)M * (tc | 1) * sizeof(float2) + (size_t)(M + 3) / 4 * 4 * sizeof(unsigned short);
}
// tc lines per block in the plan of a row pass; an odd pitch
inline void set_lines(ColPlan* P, int tc) {
    P->tc = tc;
    P->sh = 0;
    while (1 << P->sh < tc) P->sh++;
    P->rcp = 1 << P->sh == tc ? 0u : (unsigned)((((unsigned long long)1 << 32) + tc - 1) / tc);
    P->pitch = tc | 1;
}

// Host: the stages of length L (split: as two half-length transforms by parity, NP = 2) from
// radices of at most `cap` (and primes up to 31), the last at most `cap_last` or prime; and the
// twiddle table of length L: entries of the 4096-entry table for powers of two, else the
// prepared table (mr_prepare).  false if the length is not served.
bool col_plan(int L, bool split, int cap, int cap_last, const float2* tw_pow2, ColPlan* P, const float2** tw);

}  // namespace mm
