// colmix.cu -- column passes for any transform length with prime factors up to 31.
//
// A block holds TC adjacent kx columns in shared memory as [element][column], so every
// access of a half-warp is to consecutive columns (no bank conflicts at any stride), all
// lanes of a column group share their twiddles, and global rows move TC*8 contiguous bytes.
//
// Zero padding: with at most N = L/2 non-zero rows the length-L transform splits by the
// parity of the frequency, X[2k] = DFT_N(x)[k] and X[2k+1] = DFT_N(x W_L^n)[k], and the
// inverse's first N rows are the sum of the two length-N inverses (the odd one times
// W_L^-n).  NP = 2 then; periodic axes have NP = 1, N = L.
//
// The length-N transform is in place with few, large radices (at most 16; 2-3 stages up to
// N = 4096): the forward stages decimate in frequency and leave the frequencies in
// digit-reversed slots, the inverse stages are their mirror images, so nothing is reordered
// and the last forward stage, the kernel multiply and the first inverse stage work on the
// same slots in registers (Gentleman & Sande 1966).  The first stage reads global memory and
// the last one writes it: a 3x3 multiply of two-stage columns needs two barriers.
#include <algorithm>

#include "colmix.cuh"
#include "kernel_view.cuh"
#include "mm_internal.h"
#include "pdl.cuh"
#include "tiles.h"

namespace mm {
using namespace mmfft;

namespace {

// the multiply's radices: three components in registers
#define MC_SWITCH_MUL(rad, CALL)                                                                               \
    switch (rad) {                                                                                             \
        case 1: CALL(1); break;                                                                                \
        case 2: CALL(2); break;                                                                                \
        case 3: CALL(3); break;                                                                                \
        case 4: CALL(4); break;                                                                                \
        case 5: CALL(5); break;                                                                                \
        case 6: CALL(6); break;                                                                                \
        case 7: CALL(7); break;                                                                                \
        case 8: CALL(8); break;                                                                                \
        default: CALL(0); break;                                                                               \
    }

// ---- forward stage 0: rows n < n_in of column `col` of component c (global) into the lines
// (c, parity p), at (c*np + p)*N*TC.
template <int R>
__device__ __forceinline__ void first_fwd(const ColPlan& P, int rad, float2* sm, const float2* base,
                                          long long comp_stride, long long ls, int n_in, int nh, int comps, int np, const float2* __restrict__ tw) {
    const int TC = 1 << P.sh;
    const int M = P.N / rad, per = M * TC;
    for (int i = threadIdx.x; i < comps * per; i += blockDim.x) {
        const int c = comps == 1 ? 0 : i / per, e = i - c * per;
        const int col = e & (TC - 1), j = e >> P.sh;
        const float2* g = base + c * comp_stride + col;
        float2 x[RegLen<R>::n];
        MC_EACH(r, rad) {
            const int n = j + r * M;
            x[r] = (col < nh && n < n_in) ? g[n * ls] : make_float2(0.f, 0.f);
        }
        for (int p = 0; p < np; p++) {
            float2 v[RegLen<R>::n];
            MC_EACH(r, rad) v[r] = p ? cmul(x[r], tw_l<-1>(P, tw, j + r * M)) : x[r];
            dft_r<R, -1>(v, rad, P, tw);
            float2* dst = sm + ((c * np + p) * P.N + j) * TC + col;
            MC_EACH(k, rad) dst[k * M * TC] = j * k == 0 ? v[k] : cmul(v[k], tw_l<-1>(P, tw, j * k * P.NP));
        }
    }
}

// ---- last forward stage to global rows (row NP*k + parity, rows < n_out)
template <int R>
__device__ __forceinline__ void last_fwd(const ColPlan& P, int rad, const float2* sm, float2* base, long long ls,
                                         int n_out, int nh, int p0, const float2* __restrict__ tw) {
    const int TC = 1 << P.sh;
    for (int i = threadIdx.x; i < P.nq * TC; i += blockDim.x) {
        const int col = i & (TC - 1), q = i >> P.sh;
        float2 v[RegLen<R>::n];
        MC_EACH(r, rad) v[r] = sm[(q * rad + r) * TC + col];
        dft_r<R, -1>(v, rad, P, tw);
        const int f = slot_freq(P, q);
        if (col >= nh) continue;
        MC_EACH(k, rad) {
            const int row = P.NP * (f + k * P.nq) + p0;
            if (row < n_out) base[row * ls + col] = v[k];
        }
    }
}

// ---- first inverse stage from global rows (< n_in) into the np parity lines
template <int R>
__device__ __forceinline__ void first_inv(const ColPlan& P, int rad, float2* sm, const float2* base, long long ls,
                                          int n_in, int nh, const float2* __restrict__ tw) {
    const int TC = 1 << P.sh;
    const int per = P.nq * TC;
    for (int i = threadIdx.x; i < P.NP * per; i += blockDim.x) {
        const int p = P.NP == 1 ? 0 : i / per, e = i - p * per;
        const int col = e & (TC - 1), q = e >> P.sh;
        const int f = slot_freq(P, q);
        float2 v[RegLen<R>::n];
        MC_EACH(k, rad) {
            const int row = P.NP * (f + k * P.nq) + p;
            v[k] = (col < nh && row < n_in) ? base[row * ls + col] : make_float2(0.f, 0.f);
        }
        dft_r<R, +1>(v, rad, P, tw);
        MC_EACH(r, rad) sm[(p * P.N + q * rad + r) * TC + col] = v[r];
    }
}

// ---- last inverse stage: the parities' sum to global rows n < n_out
template <int R>
__device__ __forceinline__ void last_inv(const ColPlan& P, int rad, const float2* sm, float2* base,
                                         long long comp_stride, long long ls, int n_out, int nh, int comps,
                                         const float2* __restrict__ tw) {
    const int TC = 1 << P.sh;
    const int M = P.N / rad, per = M * TC;
    for (int i = threadIdx.x; i < comps * per; i += blockDim.x) {
        const int c = comps == 1 ? 0 : i / per, e = i - c * per;
        const int col = e & (TC - 1), j = e >> P.sh;
        float2 acc[RegLen<R>::n];
        for (int p = 0; p < P.NP; p++) {
            const float2* x = sm + ((c * P.NP + p) * P.N + j) * TC + col;
            float2 v[RegLen<R>::n];
            MC_EACH(k, rad) v[k] = j * k == 0 ? x[k * M * TC] : cmul(x[k * M * TC], tw_l<+1>(P, tw, j * k * P.NP));
            dft_r<R, +1>(v, rad, P, tw);
            MC_EACH(r, rad) acc[r] = p ? cadd(acc[r], cmul(v[r], tw_l<+1>(P, tw, j + r * M))) : v[r];
        }
        if (col >= nh) continue;
        MC_EACH(r, rad) {
            const int n = j + r * M;
            if (n < n_out) base[c * comp_stride + n * ls + col] = acc[r];
        }
    }
}

// ---- last forward stage of the three components, H = K M, first inverse stage
template <int R>
__device__ __forceinline__ void mul_stage(const ColPlan& P, int rad, float2* sm, const KernelView& K, int kaxis, int o,
                                          int kx0, int nh, float scale, const float2* __restrict__ tw) {
    const int TC = 1 << P.sh;
    const int per = P.nq * TC, cs = P.NP * P.N * TC;
    for (int i = threadIdx.x; i < P.NP * per; i += blockDim.x) {
        const int p = P.NP == 1 ? 0 : i / per, e = i - p * per;
        const int col = e & (TC - 1), q = e >> P.sh;
        if (col >= nh) continue;
        float2* x = sm + (p * P.N + q * rad) * TC + col;
        float2 a[RegLen<R>::n], b[RegLen<R>::n], c[RegLen<R>::n];
        MC_EACH(r, rad) {
            a[r] = x[r * TC];
            b[r] = x[cs + r * TC];
            c[r] = x[2 * cs + r * TC];
        }
        dft_r<R, -1>(a, rad, P, tw);
        dft_r<R, -1>(b, rad, P, tw);
        dft_r<R, -1>(c, rad, P, tw);
        const int f = slot_freq(P, q);
        MC_EACH(k, rad) {
            const int fr = P.NP * (f + k * P.nq) + p;
            float kk[6];
            if (kaxis == 0) kernel_at(K, fr, o, kx0 + col, kk);
            else kernel_at(K, 0, fr, kx0 + col, kk);
            const float2 m0 = a[k], m1 = b[k], m2 = c[k];
            // q: 0 xx, 1 yy, 2 zz, 3 yz, 4 xz, 5 xy
            a[k] = make_float2(scale * (kk[0] * m0.x + kk[5] * m1.x + kk[4] * m2.x),
                               scale * (kk[0] * m0.y + kk[5] * m1.y + kk[4] * m2.y));
            b[k] = make_float2(scale * (kk[5] * m0.x + kk[1] * m1.x + kk[3] * m2.x),
                               scale * (kk[5] * m0.y + kk[1] * m1.y + kk[3] * m2.y));
            c[k] = make_float2(scale * (kk[4] * m0.x + kk[3] * m1.x + kk[2] * m2.x),
                               scale * (kk[4] * m0.y + kk[3] * m1.y + kk[2] * m2.y));
        }
        dft_r<R, +1>(a, rad, P, tw);
        dft_r<R, +1>(b, rad, P, tw);
        dft_r<R, +1>(c, rad, P, tw);
        MC_EACH(r, rad) {
            x[r * TC] = a[r];
            x[cs + r * TC] = b[r];
            x[2 * cs + r * TC] = c[r];
        }
    }
}

template <int SIGN>
__device__ __forceinline__ void mid_stages(const ColPlan& P, float2* sm, int lines, const float2* __restrict__ tw) {
    if (SIGN < 0) {
        int ncur = P.N / P.r[0];
        for (int s = 1; s < P.nst - 1; s++) {
#define CALL(R) mid_stage<R, -1>(P, P.r[s], ncur, sm, lines, tw)
            MC_SWITCH(P.r[s], CALL)
#undef CALL
            ncur /= P.r[s];
            __syncthreads();
        }
    } else {
        int ncur = P.r[P.nst - 1];
        for (int s = P.nst - 2; s > 0; s--) {
            ncur *= P.r[s];
#define CALL(R) mid_stage<R, +1>(P, P.r[s], ncur, sm, lines, tw)
            MC_SWITCH(P.r[s], CALL)
#undef CALL
            __syncthreads();
        }
    }
}

// One component per line; block: outer index o, tile of TC columns.  192x192x8 cells (N = 192
// in stages of 16 and 12): forward 32 -> 22 us, inverse 35 -> 26 (21 MB each); bound by the
// twiddle loads and arithmetic of two blocks of 256 threads per SM (128 registers, which also
// lets one block have 512).
template <int SIGN>
__global__ void __launch_bounds__(512) colmix_fft_kernel(float2* __restrict__ S, int ncols, long long outer_stride,
                                                         long long ls, int n_in, int n_out, const __grid_constant__ ColPlan P,
                                                         const float2* __restrict__ tw, const DevCtl* ctl,
                                                         int skip_retry, long long sim_stride) {
    pdl_begin();
    if (ctl) ctl += blockIdx.y;
    if (conv_skip(ctl, skip_retry)) return;
    S += blockIdx.y * sim_stride;
    const int TC = 1 << P.sh;
    extern __shared__ unsigned char smem_raw[];
    float2* sm = reinterpret_cast<float2*>(smem_raw);
    const int ntiles = (ncols + TC - 1) / TC;
    const int o = blockIdx.x / ntiles;
    const int kx0 = (blockIdx.x - o * ntiles) * TC;
    const int nh = min(TC, ncols - kx0);
    float2* base = S + (long long)o * outer_stride + kx0;
    const int first = P.r[0], last = P.r[P.nst - 1];
    if (SIGN < 0) {
#define CALL(R) first_fwd<R>(P, first, sm, base, 0, ls, n_in, nh, 1, P.NP, tw)
        MC_SWITCH(first, CALL)
#undef CALL
        __syncthreads();
        mid_stages<-1>(P, sm, P.NP, tw);
        for (int p = 0; p < P.NP; p++) {
#define CALL(R) last_fwd<R>(P, last, sm + p * P.N * TC, base, ls, n_out, nh, p, tw)
            MC_SWITCH(last, CALL)
#undef CALL
        }
    } else {
#define CALL(R) first_inv<R>(P, last, sm, base, ls, n_in, nh, tw)
        MC_SWITCH(last, CALL)
#undef CALL
        __syncthreads();
        mid_stages<+1>(P, sm, P.NP, tw);
#define CALL(R) last_inv<R>(P, first, sm, base, 0, ls, n_out, nh, 1, tw)
        MC_SWITCH(first, CALL)
#undef CALL
    }
}

// Three components per column: forward, symmetric kernel multiply, inverse.  kaxis 0: lines
// along z (ky = o), 1: along y (kz = 0).  Bound by registers and shared memory (few warps: one
// block of 512 threads per SM or two of 256); lengths that are powers of two up to 1024 have faster
// four-step passes (conv.cu).
__global__ void __launch_bounds__(512) colmix_mul_kernel(float2* __restrict__ S, KernelView K, int ncols,
                                                         long long comp_stride, long long outer_stride, long long ls,
                                                         int n_in, int kaxis, float scale, const __grid_constant__ ColPlan P,
                                                         const float2* __restrict__ tw, const DevCtl* ctl,
                                                         int skip_retry, long long sim_stride,
                                                         const float* __restrict__ sim_scale) {
    pdl_begin();
    if (ctl) ctl += blockIdx.y;
    if (conv_skip(ctl, skip_retry)) return;
    S += blockIdx.y * sim_stride;
    if (sim_scale) scale = sim_scale[blockIdx.y];
    const int TC = 1 << P.sh;
    extern __shared__ unsigned char smem_raw[];
    float2* sm = reinterpret_cast<float2*>(smem_raw);
    const int ntiles = (ncols + TC - 1) / TC;
    const int o = blockIdx.x / ntiles;
    const int kx0 = (blockIdx.x - o * ntiles) * TC;
    const int nh = min(TC, ncols - kx0);
    float2* base = S + (long long)o * outer_stride + kx0;
    const int first = P.r[0], last = P.r[P.nst - 1];
#define CALL(R) first_fwd<R>(P, first, sm, base, comp_stride, ls, n_in, nh, 3, P.NP, tw)
    MC_SWITCH(first, CALL)
#undef CALL
    __syncthreads();
    mid_stages<-1>(P, sm, 3 * P.NP, tw);
#define CALL(R) mul_stage<R>(P, last, sm, K, kaxis, o, kx0, nh, scale, tw)
    MC_SWITCH_MUL(last, CALL)
#undef CALL
    __syncthreads();
    mid_stages<+1>(P, sm, 3 * P.NP, tw);
#define CALL(R) last_inv<R>(P, first, sm, base, comp_stride, ls, n_in, nh, 3, tw)
    MC_SWITCH(first, CALL)
#undef CALL
}

bool mc_prime(int r) { return r == 11 || r == 13 || r > 16; }

// `left` radices in descending order with product n, the smallest possible first one
bool radix_search(int n, int left, int most, int cap, int* out, int depth, int* best) {
    if (left == 0) {
        if (n != 1) return false;
        for (int i = 0; i < depth; i++) best[i] = out[i];
        return true;
    }
    for (int r = 2; r <= most; r++) {
        const bool ok = (r <= cap && r != 14) || r == 11 || r == 13 || r == 17 || r == 19 || r == 23 || r == 29 || r == 31;
        if (!ok || n % r) continue;
        out[depth] = r;
        if (radix_search(n / r, left - 1, r, cap, out, depth + 1, best)) return true;
    }
    return false;
}

int pick_threads(int work, int most) { return std::min(most, std::max(64, (work + 31) / 32 * 32)); }

}  // namespace

// The fewest stages, then the smallest largest radix; at least two stages (a short composite
// length in two, a prime one with a trivial second stage).
bool col_plan(int L, bool split, int cap, int cap_last, const float2* tw_pow2, ColPlan* P, const float2** tw) {
    P->NP = split ? 2 : 1;
    P->N = L / P->NP;
    int out[MC_MAXST], best[MC_MAXST] = {0};
    P->nst = 0;
    if (P->N == 1) {
        best[0] = best[1] = 1;
        P->nst = 2;
    }
    for (int k = 1; k < MC_MAXST && !P->nst; k++)
        if (radix_search(P->N, k, 31, cap, out, 0, best)) P->nst = k;
    if (!P->nst) return false;
    if (P->nst == 1) {
        if (radix_search(P->N, 2, 31, cap, out, 0, best)) P->nst = 2;
        else best[P->nst++] = 1;
    }
    // a composite last radix always splits further
    while (best[P->nst - 1] > cap_last && !mc_prime(best[P->nst - 1])) {
        if (!radix_search(P->N, P->nst + 1, 31, cap, out, 0, best)) return false;
        P->nst++;
    }
    for (int s = 0; s < P->nst; s++) P->r[s] = best[s];
    P->nq = P->N / P->r[P->nst - 1];
    P->big = best[0] > 10;  // descending order
    set_lines(P, 1);
    if (mr_pow2(L)) {
        P->tws = TWN / L;
        *tw = tw_pow2;
        return true;
    }
    P->tws = 1;
    return mr_tables(L, tw, nullptr);
}

cudaError_t launch_colmix_fft(int L, int sign, float2* S, int ncols, int nouter, long long outer_stride,
                              long long line_stride, int n_in, int n_out, const float2* tw_pow2, const DevCtl* ctl,
                              int skip_retry, cudaStream_t st, int nsim, long long sim_stride) {
    ColPlan P;
    const float2* tw = nullptr;
    if (!col_plan(L, L % 2 == 0 && 2 * std::min(n_in, n_out) <= L, 16, 16, tw_pow2, &P, &tw)) return cudaErrorInvalidValue;
    const size_t line = (size_t)P.NP * P.N * sizeof(float2);
    const ColTile tile = col_tiles(line, ncols, (long long)nouter * nsim);
    const int tc = tile.tc;
    const size_t smem = line * tc;
    set_lines(&P, tc);
    P.pitch = tc;
    const int threads = pick_threads(P.NP * P.nq * tc, tile.threads);
    const dim3 grid((unsigned)(nouter * ((ncols + tc - 1) / tc)), (unsigned)nsim);
    cudaError_t e;
    auto kern = sign < 0 ? colmix_fft_kernel<-1> : colmix_fft_kernel<1>;
    if ((e = allow_smem(kern, smem)) != cudaSuccess) return e;
    return launch_pdl(kern, grid, dim3(threads), smem, st, S, ncols, outer_stride, line_stride, n_in, n_out, P, tw, ctl,
                      skip_retry, sim_stride);
}

cudaError_t launch_colmix_mul(int L, float2* S, const KernelView& K, int ncols, int nouter, long long comp_stride,
                              long long outer_stride, long long line_stride, int n_in, int kaxis, float scale,
                              const float2* tw_pow2, const DevCtl* ctl, int skip_retry, cudaStream_t st, int nsim,
                              long long sim_stride, const float* sim_scale, int tile) {
    ColPlan P;
    const float2* tw = nullptr;
    if (!col_plan(L, L % 2 == 0 && 2 * n_in <= L, 16, 8, tw_pow2, &P, &tw)) return cudaErrorInvalidValue;
    const size_t line = (size_t)3 * P.NP * P.N * sizeof(float2);
    const ColTile shape = col_tiles(line, ncols, (long long)nouter * nsim);
    int tc = shape.tc;
    if (tile < 0 && tc > 1) tc /= 2;
    if (tile > 0 && tc < 16 && line * tc * 2 <= 200 * 1024) tc *= 2;
    const size_t smem = line * tc;
    set_lines(&P, tc);
    P.pitch = tc;
    if (smem > 220 * 1024) return cudaErrorNotSupported;
    const int threads = pick_threads(std::max(P.NP * P.nq, 3 * P.N / P.r[0]) * tc, shape.threads);
    const dim3 grid((unsigned)(nouter * ((ncols + tc - 1) / tc)), (unsigned)nsim);
    cudaError_t e;
    if ((e = allow_smem(colmix_mul_kernel, smem)) != cudaSuccess) return e;
    return launch_pdl(colmix_mul_kernel, grid, dim3(threads), smem, st, S, K, ncols, comp_stride, outer_stride,
                      line_stride, n_in, kaxis, scale, P, tw, ctl, skip_retry, sim_stride, sim_scale);
}

}  // namespace mm
