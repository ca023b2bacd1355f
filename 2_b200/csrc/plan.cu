// plan.cu -- plan object, time stepper and the fused-tier C-ABI (include/mm_b200.h).
//
// A plan owns every device buffer the hot path needs (spectrum, demag kernel octant,
// Runge-Kutta stages, control block, reduction partials), allocated once at
// mm_plan_create: nothing is allocated in a step (the reference allocates per call in
// maxwell_convolution.go:251 and solve_heun.go:47).
//
// Time stepping follows Solver.Step (src/mumax/engine/solver.go:14-17).  Each step
// attempt is a fixed sequence of launches whose pointers are resolved on the device
// from the control block (accepted-state ping-pong, retry and done flags), so attempts
// can be queued back to back, or replayed from a CUDA graph, without a host round trip.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "fft.cuh"
#include "mm_internal.h"
#include "mixed.cuh"
#include "pdl.cuh"

namespace mm {
int build_demag_kernel(const int L[3], const double cell[3], const int pbc[3], int kind, int accuracy, float* khat,
                       const int kd[3], int nz[6], cudaStream_t st, char* err, int errlen);
int build_exchange_kernel(const int L[3], const double cell[3], float* kex, const int kd[3], cudaStream_t st,
                          char* err, int errlen);
int combine_dex(const float* kd, const float* kex, long long oct, double c, float* khat, cudaStream_t st);
int fill_demag_tensor(const int L[3], const double cell[3], const int pbc[3], int kind, int accuracy, double* K,
                      cudaStream_t st);
}

using namespace mm;

static thread_local std::string g_err;
static int set_err(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}
namespace mm {
// lets other translation units report through mm_last_error()
int report_error(int code, const char* msg) { return set_err(code, "%s", msg); }
}  // namespace mm

#define CUCHK(...)                                                                                            \
    do {                                                                                                      \
        cudaError_t e_ = (__VA_ARGS__);                                                                               \
        if (e_ != cudaSuccess) return set_err(MM_ERR_CUDA, "%s: %s (%s:%d)", #__VA_ARGS__, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

static const double PI = 3.14159265358979323846264338327950288;
static const double MU0 = 4.0 * PI * 1e-7;
static const double KB = 1.380650424E-23;
static const double MUB = 9.2740091523E-24;
static const double QE = 1.60217646E-19;
static const double HBAR = 1.054571726E-34;

// ---------------------------------------------------------------- device helpers
// All per-cell kernels take the simulation from blockIdx.y; bstride = 3N floats between
// simulations, mask_bstride = 0 (shared masks) or N.
__global__ void normalize_kernel(float* m, const float* msat_mask, long long N, long long bstride,
                                 long long mask_bstride) {
    m += blockIdx.y * bstride;
    if (msat_mask) msat_mask += blockIdx.y * mask_bstride;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        float norm = msat_mask ? msat_mask[i] : 1.0f;
        float x = m[i], y = m[N + i], z = m[2 * N + i];
        float mn = sqrtf(x * x + y * y + z * z);
        float sc = (norm == 0.0f) ? 0.0f : 1.0f;
        sc = (mn != 0.0f) ? sc / mn : 0.0f;
        m[i] = x * sc;
        m[N + i] = y * sc;
        m[2 * N + i] = z * sc;
    }
}

// next = normalise(base + h * sum_j a_j K_j); h from the simulation's control block.
__global__ void combine_kernel(CombineArgs A) {
    const DevCtl* ctl = A.ctl + blockIdx.y;
    if (ctl->done) return;
    const int cur = ctl->cur;
    const long long off = blockIdx.y * A.bstride;
    const float* base = A.base.get(cur) + off;
    float* next = A.next.get(cur) + off;
    const float* msk = A.msat_mask ? A.msat_mask + blockIdx.y * A.mask_bstride : nullptr;
    const float* kp[MM_MAXK];
    float ak[MM_MAXK];
#pragma unroll
    for (int j = 0; j < MM_MAXK; j++) {
        kp[j] = j < A.nk ? A.kp[j].get(cur) + off : nullptr;
        ak[j] = j < A.nk ? (float)(A.ak[j] * ctl->h) : 0.f;
    }
    const long long N = A.N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        float x = base[i], y = base[N + i], z = base[2 * N + i];
#pragma unroll
        for (int j = 0; j < MM_MAXK; j++) {
            if (j >= A.nk) break;
            x += ak[j] * kp[j][i];
            y += ak[j] * kp[j][N + i];
            z += ak[j] * kp[j][2 * N + i];
        }
        float sc = 1.0f;
        if (!A.no_norm) {
            float norm = msk ? msk[i] : 1.0f;
            float mn = sqrtf(x * x + y * y + z * z);
            sc = (norm == 0.0f) ? 0.0f : 1.0f;
            sc = (mn != 0.0f) ? sc / mn : 0.0f;
        }
        next[i] = x * sc;
        next[N + i] = y * sc;
        next[2 * N + i] = z * sc;
    }
}

// Step controller of solve_rk12.go:156-210, generalised to error order q (RK12: q=1),
// for one simulation.
__device__ void control_one(DevCtl* c, int adaptive, int q, int fsal, int nevals, int first_skippable) {
    if (c->done) return;
    c->attempts++;
    c->evals += nevals - ((first_skippable && c->tries > 0) ? 1 : 0);
    const double dt_used = c->dt;
    bool accept = true;
    if (adaptive) {
        const double err = (double)__uint_as_float(c->err_bits) * c->h;
        c->err = err;
        const double maxErr = c->maxerr;
        const bool bad = err > maxErr;
        if (bad) c->badsteps++;
        if ((!bad || c->tries == 10 - 1) && err > c->peakerr) c->peakerr = err;
        double factor = bad ? pow(maxErr / err, 1.0 / (q + 2)) : pow(maxErr / err, 1.0 / (q + 1));
        factor *= c->headroom;
        if (factor > 1.5) factor = 1.5;
        if (factor < 0.1) factor = 0.1;
        double newDt = dt_used * factor;
        if (newDt < c->mindt) newDt = c->mindt;
        if (newDt > c->maxdt) newDt = c->maxdt;
        c->dt = newDt;
        accept = !bad || newDt == c->mindt;
        if (!accept) {
            if (c->tries > 10) {
                c->status = MM_ERR_NOT_CONVERGED;
                c->done = 1;
            }
            c->tries++;
        }
    }
    c->err_bits = 0u;
    if (accept) {
        c->t += dt_used;
        c->step++;
        c->noise_step++;
        c->cur ^= 1;
        c->tries = 0;
        if (fsal) {
            c->fsal_valid = 1;
            c->maxtorque = sqrt((double)__uint_as_float(c->tq_bits)) * c->gamma;
            if (c->torque_thr > 0 && c->maxtorque < c->torque_thr) c->done = 1;
        }
        if (c->t >= c->t_end) c->done = 1;
        if (c->step >= c->step_end) c->done = 1;
        if (c->tab_period > 0 && c->t - (double)c->tab_count * c->tab_period >= c->tab_period) {
            if (c->tab_n < c->tab_cap) c->tab_pending = 1;
            else c->tab_lost++;
            c->tab_count++;
        }
        if (c->save_period > 0 && (c->t - c->save_start) - (double)c->save_count * c->save_period >= c->save_period) {
            if (c->save_n < c->save_cap) c->save_pending = 1;
            else c->save_lost++;
            c->save_count++;
        }
    }
    if (!fsal && c->tq_bits) c->maxtorque = sqrt((double)__uint_as_float(c->tq_bits)) * c->gamma;
    c->tq_bits = 0u;
    if (c->status != MM_OK) c->done = 1;
    c->h = c->dt * c->gamma;
}

// Summary of nsim control blocks for the host: active count, first error, and the most
// accepted steps any active simulation still needs.  One block; `mode` selects what is
// done to each block first (0: nothing, 1: control_one, 2: torque check).
__device__ void summarise(const DevCtl* c, int nsim, CtlSummary* sum, int active, int bad, long long left) {
    __shared__ int s_active[32], s_bad[32];
    __shared__ long long s_left[32];
    for (int o = 16; o > 0; o >>= 1) {
        active += __shfl_xor_sync(0xffffffffu, active, o);
        bad = min(bad, __shfl_xor_sync(0xffffffffu, bad, o));
        left = max(left, __shfl_xor_sync(0xffffffffu, left, o));
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) { s_active[w] = active; s_bad[w] = bad; s_left[w] = left; }
    __syncthreads();
    if (threadIdx.x == 0) {
        int a = 0, b = 0x7fffffff;
        long long l = 0;
        for (int i = 0; i < nw; i++) { a += s_active[i]; b = min(b, s_bad[i]); l = max(l, s_left[i]); }
        sum->active = a;
        sum->bad_sim = (b == 0x7fffffff) ? -1 : b;
        sum->status = (b == 0x7fffffff) ? MM_OK : c[b].status;
        sum->step = (b == 0x7fffffff) ? 0 : c[b].step;
        sum->max_left = l;
    }
}

__global__ void controller_kernel(DevCtl* ctl, int nsim, CtlSummary* sum, int mode, int adaptive, int q, int fsal,
                                  int nevals, int first_skippable) {
    pdl_begin();
    int active = 0, bad = 0x7fffffff;
    long long left = 0;
    for (int b = threadIdx.x; b < nsim; b += blockDim.x) {
        // a local copy: one round trip for the block's fields, then one for the stores, where
        // working in place takes one for each group of fields that a branch waits for
        DevCtl local = ctl[b];
        DevCtl* c = &local;
        if (mode == 1) control_one(c, adaptive, q, fsal, nevals, first_skippable);
        if (mode == 2 && !c->done) {
            // run_until_smaller for non-FSAL solvers: the torque k0 of the current state is
            // known after the first evaluation of an attempt (api.go:122-131 checks before
            // each step)
            if (c->tries == 0) {
                c->maxtorque = sqrt((double)__uint_as_float(c->tq_bits)) * c->gamma;
                if (c->torque_thr > 0 && c->maxtorque < c->torque_thr) c->done = 1;
            }
            c->tq_bits = 0u;
        }
        if (mode != 0) ctl[b] = local;
        if (!c->done) {
            active++;
            left = max(left, c->step_end - c->step);
        }
        if (c->status != MM_OK) bad = min(bad, b);
    }
    summarise(ctl, nsim, sum, active, bad, left);
}

// For each simulation whose accepted state sits in the second ping-pong buffer, copy
// state and FSAL derivative to the first (cur is reset afterwards by reset_cur_kernel).
__global__ void canonical_copy_kernel(float* Y0, const float* Y1, float* K0, const float* K1, const DevCtl* ctl,
                                      long long n3) {
    if (ctl[blockIdx.y].cur == 0) return;
    const long long off = blockIdx.y * n3;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3; i += (long long)gridDim.x * blockDim.x) {
        Y0[off + i] = Y1[off + i];
        K0[off + i] = K1[off + i];
    }
}
__global__ void reset_cur_kernel(DevCtl* ctl, int nsim) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nsim; b += gridDim.x * blockDim.x) ctl[b].cur = 0;
}

// deterministic compensated finish of block partials: out[sim*4 + q] from
// red[(sim*nblocks + b)*8 + 2q (+1)]
__global__ void energy_finish_kernel(const float* red, int nblocks, double* out, int nsim) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nsim * 4) return;
    const int sim = g >> 2, q = g & 3;
    const float* rs = red + (long long)sim * nblocks * 8;
    float fs = 0.f, fc = 0.f;  // partial pairs are folded in fixed block order
    for (int b = 0; b < nblocks; b++) {
        float v = rs[b * 8 + 2 * q];
        float t = fs + v;
        if (fabsf(fs) >= fabsf(v)) fc += (fs - t) + v;
        else fc += (v - t) + fs;
        fs = t;
        fc += rs[b * 8 + 2 * q + 1];
    }
    out[g] = (double)fs + (double)fc;
}

// compensated per-component sums of one simulation's state m into the block's slot of red
__device__ void sum3_block(const float* m, long long N, float* red) {
    float s[3] = {0.f, 0.f, 0.f}, c[3] = {0.f, 0.f, 0.f};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
        for (int q = 0; q < 3; q++) {
            float v = m[q * N + i];
            float t = s[q] + v;
            if (fabsf(s[q]) >= fabsf(v)) c[q] += (s[q] - t) + v;
            else c[q] += (v - t) + s[q];
            s[q] = t;
        }
    }
    __shared__ float sh[6][256];
    for (int q = 0; q < 3; q++) { sh[2 * q][threadIdx.x] = s[q]; sh[2 * q + 1][threadIdx.x] = c[q]; }
    __syncthreads();
    if (threadIdx.x < 3) {
        int q = threadIdx.x;
        float fs = 0.f, fc = 0.f;
        for (int t = 0; t < blockDim.x; t++) {
            float v = sh[2 * q][t];
            float tt = fs + v;
            if (fabsf(fs) >= fabsf(v)) fc += (fs - tt) + v;
            else fc += (v - tt) + fs;
            fs = tt;
            fc += sh[2 * q + 1][t];
        }
        const long long slot = (long long)blockIdx.y * gridDim.x + blockIdx.x;
        red[slot * 8 + 2 * q] = fs;
        red[slot * 8 + 2 * q + 1] = fc;
    }
}

// <m> partial sums, one row of blocks per simulation
__global__ void sum3_kernel(const float* m, long long N, long long bstride, float* red) {
    sum3_block(m + blockIdx.y * bstride, N, red);
}

// autotabulate: partial sums of the just-accepted state of simulations with a record due
__global__ void tab_sum_kernel(const float* Y0, const float* Y1, const DevCtl* ctl, long long N, long long bstride,
                               float* red) {
    const DevCtl* c = ctl + blockIdx.y;
    if (!c->tab_pending) return;
    sum3_block((c->cur ? Y1 : Y0) + blockIdx.y * bstride, N, red);
}

// autosave: copy of the just-accepted state of simulations with a save due into their
// next ring slot
__global__ void save_copy_kernel(const float* Y0, const float* Y1, const DevCtl* ctl, long long n3, float* ring,
                                 double* ring_t) {
    const DevCtl* c = ctl + blockIdx.y;
    if (!c->save_pending) return;
    const float* src = (c->cur ? Y1 : Y0) + blockIdx.y * n3;
    const long long slot = (long long)blockIdx.y * c->save_cap + c->save_n;
    float* dst = ring + slot * n3;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n3; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) ring_t[slot] = c->t;
}

// autotabulate / autosave bookkeeping, one thread per simulation: folds the <m>
// partials (fixed order, compensated) and appends the row (t, <m>_0, <m>_1, <m>_2,
// maxtorque, dt, step, 0); counts the saved state
__global__ void tab_finish_kernel(const float* red, int nblocks, DevCtl* ctl, int nsim, double* rec, long long N) {
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nsim; b += gridDim.x * blockDim.x) {
        DevCtl* c = ctl + b;
        if (c->save_pending) {
            c->save_n++;
            c->save_pending = 0;
        }
        if (!c->tab_pending) continue;
        double avg[3];
        for (int q = 0; q < 3; q++) {
            const float* rs = red + (long long)b * nblocks * 8;
            float fs = 0.f, fc = 0.f;
            for (int k = 0; k < nblocks; k++) {
                float v = rs[k * 8 + 2 * q];
                float t = fs + v;
                if (fabsf(fs) >= fabsf(v)) fc += (fs - t) + v;
                else fc += (v - t) + fs;
                fs = t;
                fc += rs[k * 8 + 2 * q + 1];
            }
            avg[q] = ((double)fs + (double)fc) / (double)N;
        }
        double* row = rec + ((long long)b * c->tab_cap + c->tab_n) * 8;
        row[0] = c->t;
        row[1] = avg[0];
        row[2] = avg[1];
        row[3] = avg[2];
        row[4] = c->maxtorque;
        row[5] = c->dt;
        row[6] = (double)c->step;
        row[7] = 0.0;
        c->tab_n++;
        c->tab_pending = 0;
    }
}

// ---------------------------------------------------------------- plan
struct mm_plan_s {
    int device = 0;
    mm_problem prob;
    int nsim = 1;
    int masks_per_sim = 0;
    std::vector<mm_sim> sims;        // per-simulation scalars (host copy)
    ConvGeom g;
    FieldParams P;
    bool demag = false;
    float* khat = nullptr;
    float* khat_d = nullptr;         // demagexch: pure demag octant (khat holds the sum)
    float* khat_ex = nullptr;        // demagexch: Laplacian octant
    float2* tw = nullptr;            // FP32 twiddle table exp(-2 pi i k / 4096)
    KernelView kv;
    float2* S = nullptr;
    SimScalars* d_sims = nullptr;    // nsim > 1: per-simulation scalars
    float* d_sim_msat = nullptr;     // nsim > 1: demag scale of each simulation
    // solver state (every per-cell buffer holds nsim blocks of 3N floats)
    int solver = -1;
    float* Y[2] = {nullptr, nullptr};
    float* K1[2] = {nullptr, nullptr};
    float* Kst[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    float* Ma = nullptr;
    float* Mb = nullptr;
    float* Mtmp = nullptr;
    DevCtl* ctl = nullptr;           // nsim control blocks
    DevCtl* ctl_host = nullptr;      // pinned mirror
    CtlSummary* dsum = nullptr;
    CtlSummary* hsum = nullptr;      // pinned
    float* red = nullptr;            // [nsim][red_blocks][8]
    int red_blocks = 0;
    double* dres = nullptr;          // [nsim][8]
    unsigned int* tq = nullptr;      // [nsim]
    bool state_set = false;
    bool run_until = false;
    long long launches = 0;          // kernels enqueued by this plan (graph replays counted per node)
    int graph_nodes = 0;
    cudaGraphExec_t graph = nullptr;
    int graph_solver = -1;
    bool graph_run_until = false;
    long long version = 0;           // bumped whenever captured launches would change
    double* tab[2] = {nullptr, nullptr};  // SetPointwise tables (device rows t v0 v1 v2)
    int tab_n[2] = {0, 0};
    int tab_cap[2] = {0, 0};
    std::vector<double> tab_host[2];
    double t_eval = 0.0;             // time of standalone evaluations
    double dt0 = 1e-15;              // initial dt of the solver (mm_batch_restart)
    // asynchronous snapshots (mm_save_async): device staging is Mtmp; pinned host copy,
    // side stream, events and the writer thread are made on first use
    float* snap_host = nullptr;
    double* snap_t_host = nullptr;
    double* snap_t_dev = nullptr;
    cudaStream_t snap_stream = nullptr;
    cudaEvent_t snap_ready = nullptr, snap_copied = nullptr;
    std::thread snap_writer;
    int snap_rc = MM_OK;
    double* rec = nullptr;           // autotabulate rows [nsim][rec_cap][8]
    int rec_cap = 0;
    bool tab_on = false;
    float* ring = nullptr;           // autosave states [nsim][ring_cap][3N]
    double* ring_t = nullptr;        // their times [nsim][ring_cap]
    int ring_cap = 0;
    bool save_on = false;
    long long bytes = 0;
    // autotuned tile variants (-1, 0, +1) of the row, column and epilogue passes, and the
    // evaluation time measured with them (0 if not tuned)
    int tiles[4] = {0, 0, 0, 0};     // [3]: fused single-layer evaluation (fused2d_kernel)
    float tuned_us = 0.f;
    // the epilogue of a stage that forms the next stage state also writes its R2C rows
    // (MM_EPI_R2C=0 in the environment at plan creation turns this off)
    bool epi_r2c = true;
    // programmatic dependent launch for this plan's passes and controller, on plans of at
    // least 2^18 cells in all (RK23 step of 256 films of 64x64: 471 -> 454 us); on smaller
    // ones the programmatic edges cost more than they hide (SP4 film 161 -> 183 us,
    // 16 films of 64x64 93 -> 103 us per step)
    bool pdl = false;
    long long n3() const { return 3 * g.N; }
    long long spec_bstride() const { return 3LL * g.n[0] * g.L[1] * g.hp; }
};

static int dalloc(mm_plan p, void** ptr, size_t bytes) {
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e != cudaSuccess) return set_err(MM_ERR_CUDA, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
    p->bytes += (long long)bytes;
    return MM_OK;
}

static bool pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }

// Folds one simulation's multipliers the way the reference's updaters do on the host
// (mod_exchange6.go:47, mod_uniaxialanisotropy.go:49-53, mod_temperature.go:100-112,
// mod_zhang-li.go:60-64, mod_slonczewski.go:77-79).
static SimScalars fold_scalars(const mm_problem& q, const mm_sim& m) {
    SimScalars s;
    memset(&s, 0, sizeof s);
    s.msat = (float)m.msat;
    s.ex_pre = (float)(2.0 * m.aex / (MU0 * m.msat));
    s.alpha = (float)m.alpha;
    for (int i = 0; i < 3; i++) s.hz[i] = (float)(m.bext[i] / MU0);
    s.kmul = (float)(2.0 * m.ku / (MU0 * m.msat));
    for (int i = 0; i < 3; i++) s.anisu[i] = (float)m.anisu[i];
    s.therm_num = (float)(m.alpha * KB * 2.0 * m.temp);
    s.therm_den = MU0 * (q.cell[0] * q.cell[1] * q.cell[2]) * q.gamma * m.msat;
    s.seed = m.seed;
    s.zl_pre = (float)(q.zl_pol * MUB / (QE * m.msat));
    const double beta = HBAR * q.gamma / (MU0 * QE * m.msat);
    s.sl_beta_prime = (float)(q.sl_pol * beta);
    s.sl_pre_fld = (float)(beta * q.eps_prime);
    for (int i = 0; i < 3; i++) s.jmul[i] = (float)q.j[i];
    return s;
}

static mm_sim sim_of(const mm_problem& q) {
    mm_sim m;
    m.msat = q.msat;
    m.aex = q.aex;
    m.alpha = q.alpha;
    for (int i = 0; i < 3; i++) { m.bext[i] = q.bext[i]; m.anisu[i] = q.anisu[i]; }
    m.ku = q.ku;
    m.temp = q.temp;
    m.seed = q.seed;
    return m;
}

static void fill_params(mm_plan p) {
    const mm_problem& q = p->prob;
    FieldParams& P = p->P;
    memset(&P, 0, sizeof P);
    P.demag = q.demag;
    P.exchange = q.exchange && !q.demag_exchange;
    P.anis = q.anis;
    P.zeeman = q.zeeman;
    bool hot = false;
    for (const mm_sim& m : p->sims) hot = hot || m.temp != 0.0;
    P.thermal = q.thermal && hot;
    P.zhangli = q.zhangli;
    P.slonczewski = q.slonczewski;
    for (int i = 0; i < 3; i++) { P.n[i] = q.n[i]; P.pbc[i] = q.pbc[i]; }
    P.N = (long long)q.n[0] * q.n[1] * q.n[2];
    P.s = fold_scalars(q, p->sims[0]);
    P.sims = p->nsim > 1 ? p->d_sims : nullptr;
    P.bstride = 3 * P.N;
    P.mask_bstride = p->masks_per_sim ? P.N : 0;
    for (int i = 0; i < 3; i++) P.cinv2[i] = (float)(1.0 / ((double)q.cell[i] * (double)q.cell[i]));
    P.xi = (float)q.xi;
    for (int i = 0; i < 3; i++) {
        P.c12inv[i] = 1.0f / (12.0f * (float)q.cell[i]);
        P.p[i] = (float)q.p[i];
    }
    P.lambda = (float)q.lambda;
    P.t_fl = (float)q.t_fl;
    P.inv_gamma = (float)(1.0 / q.gamma);
    P.msat_mask = q.msat_mask;
    P.aex_mask = q.aex_mask;
    P.alpha_mask = q.alpha_mask;
    P.ku_mask = q.ku_mask;
    for (int i = 0; i < 3; i++) {
        P.anisu_mask[i] = q.anisu_mask[i];
        P.bext_mask[i] = q.bext_mask[i];
        P.j_mask[i] = q.j_mask[i];
        P.p_mask[i] = q.p_mask[i];
    }
    P.temp_mask = q.temp_mask;
    P.xi_mask = q.xi_mask;
    P.zl_pol_mask = q.zl_pol_mask;
    P.sl_pol_mask = q.sl_pol_mask;
    P.lambda_mask = q.lambda_mask;
    P.eps_prime_mask = q.eps_prime_mask;
    P.t_fl_mask = q.t_fl_mask;
    for (int w = 0; w < 2; w++) {
        P.tab[w].rows = p->tab[w];
        P.tab[w].n = p->tab_n[w];
    }
}

// Uploads the per-simulation scalars (nsim > 1) and refreshes the parameter block.
static int upload_sims(mm_plan p) {
    fill_params(p);
    if (p->nsim == 1) return MM_OK;
    std::vector<SimScalars> h(p->nsim);
    std::vector<float> ms(p->nsim);
    for (int b = 0; b < p->nsim; b++) {
        h[b] = fold_scalars(p->prob, p->sims[b]);
        ms[b] = (float)p->sims[b].msat;
    }
    if (cudaMemcpy(p->d_sims, h.data(), sizeof(SimScalars) * p->nsim, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(p->d_sim_msat, ms.data(), sizeof(float) * p->nsim, cudaMemcpyHostToDevice) != cudaSuccess)
        return set_err(MM_ERR_CUDA, "upload of the per-simulation scalars failed");
    return MM_OK;
}

static int check_sims(const mm_sim* sims, int nsim) {
    for (int b = 0; b < nsim; b++)
        if (!(sims[b].msat != 0.0)) return set_err(MM_ERR_ARG, "Msat of simulation %d must be non-zero", b);
    return MM_OK;
}

static int read_ctl(mm_plan p, cudaStream_t st);
static int write_ctl(mm_plan p, cudaStream_t st);

static void free_graph(mm_plan p) {
    if (p->graph) {
        cudaGraphExecDestroy(p->graph);
        p->graph = nullptr;
    }
    p->version++;
}

extern "C" MM_API const char* mm_last_error(void) { return g_err.c_str(); }
extern "C" MM_API const char* mm_version(void) { return "mm_b200 0.2 (sm_100a)"; }

static int autotune(mm_plan p);

extern "C" MM_API int mm_plan_create_batch(const mm_problem* prob, int nsim, const mm_sim* sims, int masks_per_sim,
                                           mm_plan* out) {
    if (!prob || !out) return set_err(MM_ERR_ARG, "null argument");
    *out = nullptr;
    if (nsim < 1 || nsim > 65535) return set_err(MM_ERR_ARG, "nsim must be in 1..65535 (got %d)", nsim);
    for (int i = 0; i < 3; i++) {
        if (prob->n[i] < 1) return set_err(MM_ERR_ARG, "grid size must be >= 1");
        if (!(prob->cell[i] > 0)) return set_err(MM_ERR_ARG, "cell size must be > 0");
    }
    if (!(prob->gamma != 0.0)) return set_err(MM_ERR_ARG, "gamma should be non-zero");
    if (sims) {
        int rc = check_sims(sims, nsim);
        if (rc) return rc;
    } else if (!(prob->msat != 0.0)) {
        return set_err(MM_ERR_ARG, "Msat multiplier must be non-zero");
    }
    mm_plan p = new mm_plan_s();
    cudaGetDevice(&p->device);
    p->prob = *prob;
    p->nsim = nsim;
    p->masks_per_sim = masks_per_sim ? 1 : 0;
    p->sims.resize(nsim);
    for (int b = 0; b < nsim; b++) p->sims[b] = sims ? sims[b] : sim_of(*prob);
    if (sims) {
        // the problem's own scalars follow simulation 0 (what single-simulation paths read)
        const mm_sim& m0 = sims[0];
        p->prob.msat = m0.msat;
        p->prob.aex = m0.aex;
        p->prob.alpha = m0.alpha;
        p->prob.ku = m0.ku;
        p->prob.temp = m0.temp;
        p->prob.seed = m0.seed;
        for (int i = 0; i < 3; i++) { p->prob.bext[i] = m0.bext[i]; p->prob.anisu[i] = m0.anisu[i]; }
    }
    if (prob->demag_tensor != MM_TENSOR_ARNE && prob->demag_tensor != MM_TENSOR_NEWELL)
        return set_err(MM_ERR_ARG, "demag_tensor must be MM_TENSOR_ARNE (0) or MM_TENSOR_NEWELL (1), got %d",
                       prob->demag_tensor);
    if (prob->demag_exchange && (!prob->demag || prob->aex_mask || nsim != 1)) {
        delete p;
        return set_err(MM_ERR_ARG, "demag_exchange needs demag = 1, a uniform Aex (no mask) and one simulation");
    }
    ConvGeom& g = p->g;
    for (int i = 0; i < 3; i++) {
        g.n[i] = prob->n[i];
        g.L[i] = (prob->n[i] > 1 && prob->pbc[i] == 0) ? 2 * prob->n[i] : prob->n[i];
    }
    g.N = (long long)g.n[0] * g.n[1] * g.n[2];
    p->demag = prob->demag != 0;
    int rc = MM_OK;
    if (nsim > 1) {
        if ((rc = dalloc(p, (void**)&p->d_sims, sizeof(SimScalars) * nsim))) { delete p; return rc; }
        if ((rc = dalloc(p, (void**)&p->d_sim_msat, sizeof(float) * nsim))) { mm_plan_destroy(p); return rc; }
    }
    if ((rc = upload_sims(p))) { mm_plan_destroy(p); return rc; }
    if (p->demag) {
        // Kernel_Arne's sanity checks (kernel_magnetostatic.go:36-45)
        if (!(g.L[1] > 1 && g.L[2] > 1 && g.L[1] % 2 == 0 && g.L[2] % 2 == 0 && (g.L[0] == 1 || g.L[0] % 2 == 0))) {
            mm_plan_destroy(p);
            return set_err(MM_ERR_ARG, "demag needs even padded sizes > 1 in y and x (got %d %d %d)", g.L[0], g.L[1],
                           g.L[2]);
        }
        // transform lengths: powers of two go to the power-of-two passes, every other length
        // up to 4096 with prime factors <= 31 to the mixed-radix ones (the reference takes
        // any size through cuFFT, fftplanX.go:59-64; gridsize.go:16-33 recommends
        // 2^n * {1, 3, 5, 7})
        {
            const int lens[4] = {g.L[0], g.L[1], g.L[2] / 2, g.L[2]};
            for (int q = 0; q < 4; q++) {
                const int len = lens[q];
                if (len <= 1 || pow2(len)) {
                    if (len > 4096) {
                        mm_plan_destroy(p);
                        return set_err(MM_ERR_ARG, "demag transform sizes must be <= 4096 (got %d %d %d)", g.L[0],
                                       g.L[1], g.L[2]);
                    }
                    continue;
                }
                MrLine f;
                if (!mr_factor(len, &f)) {
                    mm_plan_destroy(p);
                    return set_err(MM_ERR_ARG,
                                   "demag transform size %d (padded %d %d %d) is above 4096 or has a prime factor "
                                   "above 31; use sizes 2^n * {1, 3, 5, 7}",
                                   len, g.L[0], g.L[1], g.L[2]);
                }
                if ((rc = mr_prepare(len)) != MM_OK) {
                    mm_plan_destroy(p);
                    return set_err(rc, "twiddle tables of length %d could not be built", len);
                }
            }
        }
        if (nsim > 1 && pow2(g.L[2]) && (g.L[2] < 8 || g.L[2] > 2048)) {
            mm_plan_destroy(p);
            return set_err(MM_ERR_ARG, "batched plans with demag need 8 <= padded L2 <= 2048 (got %d)", g.L[2]);
        }
        g.M = g.L[2] / 2;
        g.h = g.M + 1;
        g.hp = (g.h + 3) & ~3;
        g.kd[0] = g.L[0] / 2 + 1;
        g.kd[1] = g.L[1] / 2 + 1;
        g.kd[2] = g.L[2] / 2 + 1;
        const long long oct = (long long)g.kd[0] * g.kd[1] * g.kd[2];
        if ((rc = dalloc(p, (void**)&p->khat, sizeof(float) * 6 * oct))) { mm_plan_destroy(p); return rc; }
        if ((rc = dalloc(p, (void**)&p->tw, sizeof(float2) * mmfft::TWN))) { mm_plan_destroy(p); return rc; }
        {
            std::vector<float2> h(mmfft::TWN);
            mmfft::make_twiddle_table(h.data());
            if (cudaMemcpy(p->tw, h.data(), sizeof(float2) * mmfft::TWN, cudaMemcpyHostToDevice) != cudaSuccess) {
                mm_plan_destroy(p);
                return set_err(MM_ERR_CUDA, "twiddle table upload failed");
            }
        }
        if ((rc = dalloc(p, (void**)&p->S, sizeof(float2) * (size_t)p->spec_bstride() * nsim))) {
            mm_plan_destroy(p);
            return rc;
        }
        cudaStream_t st;
        cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        char err[512] = {0};
        int nz[6];
        if (prob->demag_exchange) {
            if (!(rc = dalloc(p, (void**)&p->khat_d, sizeof(float) * 6 * oct)) &&
                !(rc = dalloc(p, (void**)&p->khat_ex, sizeof(float) * oct))) {
                rc = build_demag_kernel(g.L, prob->cell, prob->pbc, prob->demag_tensor, prob->demag_accuracy, p->khat_d,
                                        g.kd, nz, st, err, sizeof err);
                if (rc == MM_OK) rc = build_exchange_kernel(g.L, prob->cell, p->khat_ex, g.kd, st, err, sizeof err);
                if (rc == MM_OK)
                    rc = combine_dex(p->khat_d, p->khat_ex, oct, 2.0 * prob->aex / (MU0 * prob->msat * prob->msat),
                                     p->khat, st);
                for (int q = 0; q < 3; q++) nz[q] = 1;
            }
        } else {
            rc = build_demag_kernel(g.L, prob->cell, prob->pbc, prob->demag_tensor, prob->demag_accuracy, p->khat, g.kd,
                                    nz, st, err, sizeof err);
        }
        if (rc == MM_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = MM_ERR_CUDA;
        cudaStreamDestroy(st);
        if (rc != MM_OK) {
            mm_plan_destroy(p);
            return set_err(rc, "demag kernel: %s", err);
        }
        p->kv.k = p->khat;
        p->kv.kd0 = g.kd[0];
        p->kv.kd1 = g.kd[1];
        p->kv.kd2 = g.kd[2];
        p->kv.L0 = g.L[0];
        p->kv.L1 = g.L[1];
        for (int q = 0; q < 6; q++) p->kv.nz[q] = nz[q];
    }
    const size_t vb = sizeof(float) * (size_t)p->n3() * nsim;
    void** bufs[] = {(void**)&p->Y[0], (void**)&p->Y[1], (void**)&p->K1[0], (void**)&p->K1[1], (void**)&p->Ma,
                     (void**)&p->Mb, (void**)&p->Mtmp};
    for (auto b : bufs)
        if ((rc = dalloc(p, b, vb))) { mm_plan_destroy(p); return rc; }
    for (int i = 0; i < 6; i++)
        if ((rc = dalloc(p, (void**)&p->Kst[i], vb))) { mm_plan_destroy(p); return rc; }
    if ((rc = dalloc(p, (void**)&p->ctl, sizeof(DevCtl) * nsim))) { mm_plan_destroy(p); return rc; }
    if ((rc = dalloc(p, (void**)&p->dsum, sizeof(CtlSummary)))) { mm_plan_destroy(p); return rc; }
    if (cudaMallocHost(&p->ctl_host, sizeof(DevCtl) * nsim) != cudaSuccess ||
        cudaMallocHost(&p->hsum, sizeof(CtlSummary)) != cudaSuccess) {
        mm_plan_destroy(p);
        return set_err(MM_ERR_CUDA, "cudaMallocHost failed");
    }
    p->red_blocks = std::max(p->demag ? xinv_blocks(g.M, g.n[0] * g.n[1]) : 0, local_blocks(g.N, nsim));
    if (nsim == 1) p->red_blocks = std::max(p->red_blocks, 148 * 4);
    if ((rc = dalloc(p, (void**)&p->red, sizeof(float) * 8 * (size_t)p->red_blocks * nsim))) {
        mm_plan_destroy(p);
        return rc;
    }
    if ((rc = dalloc(p, (void**)&p->dres, sizeof(double) * 8 * nsim))) { mm_plan_destroy(p); return rc; }
    if ((rc = dalloc(p, (void**)&p->tq, sizeof(unsigned int) * std::max(4, nsim)))) { mm_plan_destroy(p); return rc; }
    DevCtl c;
    memset(&c, 0, sizeof c);
    c.t_end = 1e300;
    c.step_end = (1LL << 62);
    c.maxerr = 1.0 / 2000;
    c.mindt = 1e-38;
    c.maxdt = 1e38;
    c.headroom = 0.8;
    c.dt = 1e-15;
    c.gamma = prob->gamma;
    c.h = c.dt * c.gamma;
    c.done = 1;
    for (int b = 0; b < nsim; b++) p->ctl_host[b] = c;
    if (cudaMemcpy(p->ctl, p->ctl_host, sizeof(DevCtl) * nsim, cudaMemcpyHostToDevice) != cudaSuccess) {
        mm_plan_destroy(p);
        return set_err(MM_ERR_CUDA, "ctl init failed");
    }
    {
        const char* e = getenv("MM_EPI_R2C");
        p->epi_r2c = !(e && e[0] == '0');
    }
    p->pdl = (long long)nsim * p->g.N >= (1LL << 18);
    if ((rc = autotune(p))) {
        mm_plan_destroy(p);
        return rc;
    }
    *out = p;
    return MM_OK;
}

extern "C" MM_API int mm_plan_create(const mm_problem* prob, mm_plan* out) {
    return mm_plan_create_batch(prob, 1, nullptr, 0, out);
}

extern "C" MM_API int mm_plan_nsim(mm_plan p) { return p ? p->nsim : 0; }

extern "C" MM_API int mm_save_wait(mm_plan p);

extern "C" MM_API int mm_plan_destroy(mm_plan p) {
    if (!p) return MM_OK;
    mm_save_wait(p);
    if (p->snap_host) cudaFreeHost(p->snap_host);
    if (p->snap_t_host) cudaFreeHost(p->snap_t_host);
    if (p->snap_t_dev) cudaFree(p->snap_t_dev);
    if (p->snap_stream) cudaStreamDestroy(p->snap_stream);
    if (p->snap_ready) cudaEventDestroy(p->snap_ready);
    if (p->snap_copied) cudaEventDestroy(p->snap_copied);
    if (p->graph) cudaGraphExecDestroy(p->graph);
    void* bufs[] = {p->ring, p->ring_t, p->rec, p->tab[0], p->tab[1], p->khat, p->khat_d, p->khat_ex, p->tw, p->S, p->d_sims, p->d_sim_msat, p->Y[0], p->Y[1], p->K1[0], p->K1[1], p->Ma,
                    p->Mb, p->Mtmp, p->ctl, p->dsum, p->red, p->dres, p->tq};
    for (void* b : bufs)
        if (b) cudaFree(b);
    for (int i = 0; i < 6; i++)
        if (p->Kst[i]) cudaFree(p->Kst[i]);
    if (p->ctl_host) cudaFreeHost(p->ctl_host);
    if (p->hsum) cudaFreeHost(p->hsum);
    delete p;
    return MM_OK;
}

extern "C" MM_API int mm_batch_set_sims(mm_plan p, const mm_sim* sims) {
    if (!p || !sims) return set_err(MM_ERR_ARG, "null argument");
    int rc = check_sims(sims, p->nsim);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) p->sims[b] = sims[b];
    const mm_sim& m0 = sims[0];
    p->prob.msat = m0.msat;
    p->prob.aex = m0.aex;
    p->prob.alpha = m0.alpha;
    p->prob.ku = m0.ku;
    p->prob.temp = m0.temp;
    p->prob.seed = m0.seed;
    for (int i = 0; i < 3; i++) { p->prob.bext[i] = m0.bext[i]; p->prob.anisu[i] = m0.anisu[i]; }
    free_graph(p);
    if ((rc = upload_sims(p))) return rc;
    if ((rc = read_ctl(p, 0))) return rc;
    for (int b = 0; b < p->nsim; b++) p->ctl_host[b].fsal_valid = 0;
    return write_ctl(p, 0);
}

extern "C" MM_API int mm_plan_set_problem(mm_plan p, const mm_problem* prob) {
    if (!p || !prob) return set_err(MM_ERR_ARG, "null argument");
    for (int i = 0; i < 3; i++)
        if (prob->n[i] != p->prob.n[i] || prob->cell[i] != p->prob.cell[i] || prob->pbc[i] != p->prob.pbc[i])
            return set_err(MM_ERR_ARG, "geometry of a plan cannot change");
    if ((prob->demag != 0) != p->demag) return set_err(MM_ERR_ARG, "demag on/off cannot change after plan creation");
    if ((prob->demag_exchange != 0) != (p->khat_d != nullptr))
        return set_err(MM_ERR_ARG, "demag_exchange on/off cannot change after plan creation");
    if (prob->demag_exchange && prob->aex_mask) return set_err(MM_ERR_ARG, "demag_exchange needs a uniform Aex");
    if (prob->demag_tensor != p->prob.demag_tensor)
        return set_err(MM_ERR_ARG, "the demag tensor kind cannot change after plan creation");
    if (!(prob->gamma != 0.0)) return set_err(MM_ERR_ARG, "gamma must be non-zero");
    if (p->nsim == 1 && !(prob->msat != 0.0)) return set_err(MM_ERR_ARG, "Msat must be non-zero");
    p->prob = *prob;
    if (p->nsim == 1) p->sims[0] = sim_of(*prob);   // batched plans keep their mm_sim scalars
    free_graph(p);
    int rc = upload_sims(p);
    if (rc) return rc;
    if (p->khat_d) {  // the demag+exchange kernel depends on Aex and Ms
        const long long oct = (long long)p->g.kd[0] * p->g.kd[1] * p->g.kd[2];
        if ((rc = combine_dex(p->khat_d, p->khat_ex, oct, 2.0 * prob->aex / (MU0 * prob->msat * prob->msat), p->khat,
                              0)))
            return set_err(rc, "demag+exchange kernel update failed");
    }
    // gamma is part of h = dt*gamma on the device
    if ((rc = read_ctl(p, 0))) return rc;
    for (int b = 0; b < p->nsim; b++) {
        p->ctl_host[b].gamma = prob->gamma;
        p->ctl_host[b].h = p->ctl_host[b].dt * prob->gamma;
        p->ctl_host[b].fsal_valid = 0;
    }
    return write_ctl(p, 0);
}

extern "C" MM_API int mm_plan_kernel_nonzero(mm_plan p, int out6[6]) {
    if (!p || !out6) return set_err(MM_ERR_ARG, "null argument");
    for (int q = 0; q < 6; q++) out6[q] = p->demag ? p->kv.nz[q] : 0;
    return MM_OK;
}

extern "C" MM_API long long mm_plan_device_bytes(mm_plan p) { return p ? p->bytes : 0; }

// the register z-multiply applies when z is zero-padded (L0 = 2 N0) with N0 <= 16
static bool zreg_ok(const ConvGeom& g) {
    const int n0 = g.n[0];
    return g.L[0] == 2 * n0 && n0 <= 16;
}

// ---------------------------------------------------------------- one evaluation
// Launches of the five (3-D) or three (2-D) convolution passes for all simulations;
// `ev` (optional) receives an event record after each pass.
// rows_ready: the R2C rows of m_in are already in the spectrum (written by the epilogue
// of the evaluation that formed m_in), so the row pass is left out.
static int launch_conv(mm_plan p, PP m_in, const DevCtl* ctl, int skip_retry, cudaStream_t st,
                       const std::vector<cudaEvent_t>* ev = nullptr, bool rows_ready = false) {
    PdlScope pdl_scope(p->pdl);
    const ConvGeom& g = p->g;
    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
    const int L0 = g.L[0], L1 = g.L[1];
    const int ns = p->nsim;
    const long long plane = (long long)L1 * g.hp;
    const long long sb = p->spec_bstride();
    const float scale = (float)p->prob.msat;
    const float* sim_scale = ns > 1 ? p->d_sim_msat : nullptr;
    int k = 1;
    auto mark = [&]() -> int {
        if (ev) CUCHK(cudaEventRecord((*ev)[k++], st));
        return MM_OK;
    };
    int rc;
    // demagexch convolves m itself (mod_demagexchange.go:207-209), demag convolves Ms_mask m
    const float* in_mask = p->khat_d ? nullptr : p->P.msat_mask;
    if (!rows_ready) {
        CUCHK(launch_xfwd<float2, float>(g.M, nullptr, m_in, in_mask, p->S, 3 * n0 * n1, n0, n1, L1, n2, n2, g.hp,
                                         p->tw, ctl, skip_retry, st, ns, p->n3(), sb, p->P.mask_bstride, p->tiles[0]));
        p->launches++;
    }
    if ((rc = mark())) return rc;
    if (L0 == 1) {
        CUCHK(launch_colmul(L1, p->S, p->kv, g.h, 1, plane, 0, g.hp, n1, 1, scale, p->tw, ctl, skip_retry, st, ns, sb,
                            sim_scale, p->tiles[1]));
        if ((rc = mark())) return rc;
    } else {
        CUCHK(launch_colfft<float2>(L1, -1, p->S, g.h, 3 * n0, plane, g.hp, n1, L1, p->tw, ctl, skip_retry, st, ns,
                                    sb, p->tiles[1]));
        if ((rc = mark())) return rc;
        if (zreg_ok(g))
            CUCHK(launch_zmul_reg(n0, p->S, p->kv, L1, g.h, g.hp, (long long)n0 * plane, plane, scale, p->tw, ctl,
                                  skip_retry, st, ns, sb, sim_scale));
        else
            CUCHK(launch_colmul(L0, p->S, p->kv, g.h, L1, (long long)n0 * plane, g.hp, plane, n0, 0, scale, p->tw,
                                ctl, skip_retry, st, ns, sb, sim_scale));
        if ((rc = mark())) return rc;
        CUCHK(launch_colfft<float2>(L1, +1, p->S, g.h, 3 * n0, plane, g.hp, L1, n1, p->tw, ctl, skip_retry, st, ns,
                                    sb, p->tiles[1]));
        if ((rc = mark())) return rc;
    }
    p->launches += (L0 == 1) ? 1 : 3;
    return MM_OK;
}

// Whether an evaluation of this plan can hand the R2C rows of the next stage state to
// the following evaluation: the four-step row and epilogue passes, not the fused
// single-layer kernel.
static bool epi_r2c_ok(mm_plan p) {
    return p->epi_r2c && p->demag && epi_r2c_supported(p->g.M) && !(p->tiles[3] && fused2d_ok(p->g.n));
}

// Launches the convolution passes (if demag) and the epilogue for one StageOp.
// fwd: EVAL_EMIT_ROWS = the epilogue also writes the R2C rows of op.next (the m_in of the
// evaluation that follows); EVAL_ROWS_READY = the R2C rows of op.m_in are in the spectrum.
// Both only where epi_r2c_ok(p).
enum { EVAL_EMIT_ROWS = 1, EVAL_ROWS_READY = 2 };
static int launch_eval(mm_plan p, const StageOp& op, DevCtl* ctl, int skip_retry, float* const* dbg,
                       long long noise_step, double dt_thermal, float* red, unsigned int* tq_out, cudaStream_t st,
                       int* nblocks_out, int fwd = 0) {
    PdlScope pdl_scope(p->pdl);
    const ConvGeom& g = p->g;
    EpiArgs A;
    memset(&A, 0, sizeof A);
    A.P = p->P;
    A.op = op;
    A.ctl = ctl;
    A.noise_step = noise_step;
    A.dt_thermal = dt_thermal;
    bool terms = op.want_energy != 0;
    for (int i = 0; i < 6; i++) {
        A.dbg[i] = dbg ? dbg[i] : nullptr;
        if (A.dbg[i]) terms = true;
    }
    A.red = red;
    A.tq_out = tq_out;
    A.skip_retry = skip_retry;
    A.spec_bstride = p->spec_bstride();
    A.t_eval = p->t_eval;
    if (fwd && (terms || !epi_r2c_ok(p))) fwd = 0;  // the per-term epilogue has no row output
    if ((fwd & EVAL_EMIT_ROWS) && op.do_combine) {
        A.fwd = p->S;
        A.fwd_mask = p->khat_d ? 0 : 1;
    }
    int nb = 0, rc;
    if (p->demag && p->tiles[3] && !terms && fused2d_ok(g.n)) {
        const float* in_mask = p->khat_d ? nullptr : p->P.msat_mask;
        CUCHK(launch_fused2d(in_mask, p->P.mask_bstride, p->kv, (float)p->prob.msat,
                             p->nsim > 1 ? p->d_sim_msat : nullptr, p->tw, A, st, &nb, p->nsim));
        p->launches += 1;
        if (nblocks_out) *nblocks_out = nb;
        return MM_OK;
    }
    if (p->demag) {
        if ((rc = launch_conv(p, op.m_in, ctl, skip_retry, st, nullptr, (fwd & EVAL_ROWS_READY) != 0))) return rc;
        CUCHK(launch_xinv_epi(g.M, p->S, g.hp, g.L[1], p->tw, A, terms, st, &nb, p->nsim, p->tiles[2]));
    } else {
        CUCHK(launch_local_epi(A, terms, st, &nb, p->nsim));
    }
    p->launches += 1;
    if (nblocks_out) *nblocks_out = nb;
    return MM_OK;
}

static PP fixed(float* q) { return PP{q, nullptr, 0}; }
static PP cur_of(float* const* q) { return PP{q[0], q[1], 1}; }
static PP oth_of(float* const* q) { return PP{q[0], q[1], 2}; }
static PP none() { return PP{nullptr, nullptr, 0}; }

static StageOp op_blank() {
    StageOp o;
    memset(&o, 0, sizeof o);
    o.kcur = -1;
    o.ecur = -1;
    return o;
}

// ---------------------------------------------------------------- tile autotuner
// Times whole field evaluations (torque of a zeroed state, the plan's own buffers and
// masks) for the tile variants of the four-step passes: rows per block of the R2C row
// pass (1/2, 1, 2 x default), columns per block of the column passes (the y FFTs of 3-D
// grids, the y FFT + kernel multiply of single-layer films; 1/2, 1, 2 x) and rows per
// block of the C2R + epilogue pass (1/2, 1 x).  One pass at a time from the
// defaults (coordinate descent); a variant replaces the current choice only when it is
// more than 2 % faster.  Single-layer films whose half spectrum fits in shared memory also
// try the fused evaluation (fused2d_kernel: convolution and epilogue in one launch).
// Runs once at plan creation; MM_AUTOTUNE=0 in the environment keeps the defaults.  Tile variants change the block decomposition only: every cell's
// arithmetic is the same, and so are the fields, torques and step sequences.
// Tuning results are kept per device and plan shape for the life of the process, so
// that plans of a shape tuned before (the slots of a relaxation pool, an engine that
// rebuilds its plan, the plans of an ensemble's grid classes) take the earlier choice
// without timing again.  The shape covers everything the passes' launch configuration and
// work depend on: grid, padded sizes, simulations, which terms and masks are present.
namespace {
struct TuneKey {
    int v[24];
    bool operator<(const TuneKey& o) const { return std::lexicographical_compare(v, v + 24, o.v, o.v + 24); }
};
struct TuneVal {
    int tiles[4];
    float us;
};
std::mutex g_tune_mu;
std::map<TuneKey, TuneVal> g_tune;
long long g_tune_runs = 0;
}  // namespace

static TuneKey tune_key(mm_plan p) {
    TuneKey k;
    memset(k.v, 0, sizeof k.v);
    const FieldParams& P = p->P;
    int i = 0;
    k.v[i++] = p->device;
    for (int d = 0; d < 3; d++) { k.v[i++] = p->g.n[d]; k.v[i++] = p->g.L[d]; }
    k.v[i++] = p->nsim;
    k.v[i++] = p->masks_per_sim;
    k.v[i++] = p->khat_d ? 1 : 0;
    k.v[i++] = P.exchange | P.anis << 1 | P.zeeman << 2 | P.thermal << 3 | P.zhangli << 4 | P.slonczewski << 5;
    const void* masks[] = {P.msat_mask, P.aex_mask, P.alpha_mask, P.ku_mask, P.anisu_mask[0], P.bext_mask[0],
                           P.j_mask[0], P.temp_mask, P.xi_mask, P.zl_pol_mask, P.p_mask[0], P.sl_pol_mask,
                           P.lambda_mask, P.eps_prime_mask, P.t_fl_mask};
    int bits = 0;
    for (int q = 0; q < 15; q++) bits |= (masks[q] ? 1 : 0) << q;
    k.v[i++] = bits;
    k.v[i++] = (P.tab[0].n ? 1 : 0) | (P.tab[1].n ? 2 : 0);
    k.v[i++] = p->pdl ? 1 : 0;
    return k;
}

extern "C" MM_API long long mm_autotune_runs(void) {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    return g_tune_runs;
}

static int autotune_run(mm_plan p);

static int autotune(mm_plan p) {
    if (!p->demag) return MM_OK;
    // the tiles are those of the power-of-two passes
    if (!pow2(p->g.L[0]) || !pow2(p->g.L[1]) || !pow2(p->g.L[2])) return MM_OK;
    const char* env = getenv("MM_AUTOTUNE");
    if (env && env[0] == '0') return MM_OK;
    const TuneKey key = tune_key(p);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune.find(key);
        if (it != g_tune.end()) {
            for (int d = 0; d < 4; d++) p->tiles[d] = it->second.tiles[d];
            p->tuned_us = it->second.us;
            return MM_OK;
        }
    }
    const int rc = autotune_run(p);
    if (rc == MM_OK && p->tuned_us > 0.f) {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        TuneVal v;
        for (int d = 0; d < 4; d++) v.tiles[d] = p->tiles[d];
        v.us = p->tuned_us;
        g_tune[key] = v;
        g_tune_runs++;
    }
    return rc;
}

static int autotune_run(mm_plan p) {
    cudaStream_t st = nullptr;
    const long long launches = p->launches;
    CUCHK(cudaMemsetAsync(p->Y[0], 0, sizeof(float) * (size_t)p->n3() * p->nsim, st));
    StageOp o = op_blank();
    o.m_in = fixed(p->Y[0]);
    o.k_out = fixed(p->K1[0]);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    CUCHK(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return set_err(MM_ERR_CUDA, "cudaEventCreate failed");
    }
    int rc = MM_OK;
    int reps = 5;
    auto time_eval = [&](float* us) -> int {
        int r;
        for (int i = 0; i < 2; i++)
            if ((r = launch_eval(p, o, nullptr, 0, nullptr, 0, 0, nullptr, nullptr, st, nullptr))) return r;
        CUCHK(cudaEventRecord(e0, st));
        for (int i = 0; i < reps; i++)
            if ((r = launch_eval(p, o, nullptr, 0, nullptr, 0, 0, nullptr, nullptr, st, nullptr))) return r;
        CUCHK(cudaEventRecord(e1, st));
        CUCHK(cudaEventSynchronize(e1));
        float ms = 0.f;
        CUCHK(cudaEventElapsedTime(&ms, e0, e1));
        *us = 1000.f * ms / reps;
        return MM_OK;
    };
    float best = 0.f;
    if (!(rc = time_eval(&best))) {
        // about 2 ms of timing per variant
        reps = std::max(5, std::min(200, (int)(2000.f / std::max(best, 1.f))));
        rc = time_eval(&best);
    }
    // a variant whose launch fails (a refused shared-memory size, say) is dropped: its
    // error is not sticky, so it is cleared and the previous choice kept
    auto try_variant = [&](float* t) -> bool {
        if (time_eval(t) == MM_OK) return true;
        cudaGetLastError();
        cudaStreamSynchronize(st);
        return false;
    };
    const int lo[3] = {-1, -1, -1}, hi[3] = {1, 1, 0};
    for (int d = 0; d < 3 && !rc; d++) {
        int keep = p->tiles[d];
        for (int v = lo[d]; v <= hi[d]; v++) {
            if (v == keep) continue;
            p->tiles[d] = v;
            float t = 0.f;
            if (try_variant(&t) && t < 0.98f * best) {
                best = t;
                keep = v;
            }
        }
        p->tiles[d] = keep;
    }
    // single-layer films whose spectrum fits in shared memory: the fused evaluation
    if (!rc && fused2d_ok(p->g.n)) {
        p->tiles[3] = 1;
        float t = 0.f;
        if (try_variant(&t) && t < 0.98f * best) best = t;
        else p->tiles[3] = 0;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    p->tuned_us = rc ? 0.f : best;
    p->launches = launches;
    return rc;
}

extern "C" MM_API int mm_plan_demag_kernel(mm_plan p, float* out, int kd[3]) {
    if (!p || !kd) return set_err(MM_ERR_ARG, "null argument");
    if (!p->demag || !p->khat) return set_err(MM_ERR_STATE, "the plan has no demag kernel");
    for (int i = 0; i < 3; i++) kd[i] = p->g.kd[i];
    if (!out) return MM_OK;
    const long long oct = (long long)p->g.kd[0] * p->g.kd[1] * p->g.kd[2];
    const float* src = p->khat_d ? p->khat_d : p->khat;
    CUCHK(cudaMemcpy(out, src, sizeof(float) * 6 * (size_t)oct, cudaMemcpyDeviceToHost));
    return MM_OK;
}

extern "C" MM_API int mm_demag_tensor(const int L[3], const double cell[3], const int pbc[3], int kind, int accuracy,
                                      double* out, mm_stream stream) {
    if (!L || !cell || !pbc || !out) return set_err(MM_ERR_ARG, "null argument");
    if (kind != MM_TENSOR_ARNE && kind != MM_TENSOR_NEWELL) return set_err(MM_ERR_ARG, "unknown tensor kind %d", kind);
    for (int i = 0; i < 3; i++) {
        if (L[i] < 1 || L[i] > 65536) return set_err(MM_ERR_ARG, "padded size %d out of range", L[i]);
        if (!(cell[i] > 0)) return set_err(MM_ERR_ARG, "cell size must be > 0");
    }
    if (kind == MM_TENSOR_ARNE && !(L[1] > 1 && L[2] > 1 && L[1] % 2 == 0 && L[2] % 2 == 0 &&
                                    (L[0] == 1 || L[0] % 2 == 0)))
        return set_err(MM_ERR_ARG, "Kernel_Arne needs even padded sizes > 1 in y and x (got %d %d %d)", L[0], L[1],
                       L[2]);
    const int rc = fill_demag_tensor(L, cell, pbc, kind, accuracy, out, (cudaStream_t)stream);
    if (rc != MM_OK) return set_err(rc, "demag tensor launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    return MM_OK;
}

extern "C" MM_API int mm_plan_tiles(mm_plan p, int* tiles, double* eval_us) {
    if (!p || !tiles) return set_err(MM_ERR_ARG, "null argument");
    for (int d = 0; d < 4; d++) tiles[d] = p->tiles[d];
    if (eval_us) *eval_us = p->tuned_us;
    return MM_OK;
}

extern "C" MM_API int mm_plan_set_tiles(mm_plan p, const int* tiles) {
    if (!p || !tiles) return set_err(MM_ERR_ARG, "null argument");
    for (int d = 0; d < 3; d++)
        if (tiles[d] < -1 || tiles[d] > (d == 2 ? 0 : 1)) return set_err(MM_ERR_ARG, "tile %d out of range", d);
    if (tiles[3] != 0 && tiles[3] != 1) return set_err(MM_ERR_ARG, "tile 3 must be 0 or 1");
    if (tiles[3] && !fused2d_ok(p->g.n))
        return set_err(MM_ERR_ARG, "the fused evaluation does not serve this geometry");
    for (int d = 0; d < 4; d++) p->tiles[d] = tiles[d];
    free_graph(p);
    return MM_OK;
}

// host copy of the device table lookup (update_pointwise.go:30-88); false past the end
static bool host_table_ok(const std::vector<double>& rows, double t) {
    const size_t n = rows.size() / 4;
    return n == 0 || rows[4 * (n - 1)] >= t;
}

// Standalone evaluations happen at simulation 0's time when time tables are set.
static int standalone_time(mm_plan p, cudaStream_t st) {
    if (!p->tab_n[0] && !p->tab_n[1]) return MM_OK;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    p->t_eval = p->ctl_host[0].t;
    for (int w = 0; w < 2; w++)
        if (!host_table_ok(p->tab_host[w], p->t_eval))
            return set_err(MM_ERR_RANGE, "time %g s is past the end of the %s table", p->t_eval,
                           w == 0 ? "B_ext" : "j");
    return MM_OK;
}

extern "C" MM_API int mm_set_table(mm_plan p, int quantity, int npoints, const double* rows) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (quantity != MM_TABLE_BEXT && quantity != MM_TABLE_J) return set_err(MM_ERR_ARG, "unknown table %d", quantity);
    if (npoints < 0 || npoints == 1) return set_err(MM_ERR_ARG, "a time table needs at least two points");
    if (npoints > 0 && !rows) return set_err(MM_ERR_ARG, "null rows");
    for (int i = 1; i < npoints; i++)
        if (!(rows[4 * i] >= rows[4 * (i - 1)])) return set_err(MM_ERR_ARG, "table times must be non-decreasing");
    const int w = quantity;
    if (npoints > p->tab_cap[w]) {
        if (p->tab[w]) cudaFree(p->tab[w]);
        p->tab[w] = nullptr;
        p->tab_cap[w] = 0;
        int rc = dalloc(p, (void**)&p->tab[w], sizeof(double) * 4 * (size_t)npoints);
        if (rc) return rc;
        p->tab_cap[w] = npoints;
    }
    if (npoints > 0) CUCHK(cudaMemcpy(p->tab[w], rows, sizeof(double) * 4 * (size_t)npoints, cudaMemcpyHostToDevice));
    p->tab_host[w].assign(rows, rows + 4 * (size_t)npoints);
    p->tab_n[w] = npoints;
    fill_params(p);
    free_graph(p);
    return MM_OK;
}

extern "C" MM_API int mm_tabulate(mm_plan p, double period, int capacity) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (period > 0 && capacity < 1) return set_err(MM_ERR_ARG, "capacity must be >= 1");
    if (period > 0 && capacity > p->rec_cap) {
        if (p->rec) cudaFree(p->rec);
        p->rec = nullptr;
        p->rec_cap = 0;
        int rc = dalloc(p, (void**)&p->rec, sizeof(double) * 8 * (size_t)capacity * p->nsim);
        if (rc) return rc;
        p->rec_cap = capacity;
    }
    int rc = read_ctl(p, 0);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        c.tab_period = period > 0 ? period : 0.0;
        c.tab_count = 0;
        c.tab_lost = 0;
        c.tab_n = 0;
        c.tab_cap = period > 0 ? capacity : 0;
        c.tab_pending = 0;
    }
    p->tab_on = period > 0;
    free_graph(p);
    return write_ctl(p, 0);
}

extern "C" MM_API int mm_autosave(mm_plan p, double period, int capacity) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (period > 0 && capacity < 1) return set_err(MM_ERR_ARG, "capacity must be >= 1");
    if (period > 0 && capacity > p->ring_cap) {
        if (p->ring) cudaFree(p->ring);
        if (p->ring_t) cudaFree(p->ring_t);
        p->ring = nullptr;
        p->ring_t = nullptr;
        p->ring_cap = 0;
        int rc = dalloc(p, (void**)&p->ring, sizeof(float) * (size_t)p->n3() * capacity * p->nsim);
        if (!rc) rc = dalloc(p, (void**)&p->ring_t, sizeof(double) * (size_t)capacity * p->nsim);
        if (rc) return rc;
        p->ring_cap = capacity;
    }
    int rc = read_ctl(p, 0);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        c.save_period = period > 0 ? period : 0.0;
        c.save_start = c.t;
        c.save_count = 0;
        c.save_lost = 0;
        c.save_n = 0;
        c.save_cap = period > 0 ? capacity : 0;
        c.save_pending = 0;
    }
    p->save_on = period > 0;
    free_graph(p);
    return write_ctl(p, 0);
}

extern "C" MM_API int mm_autosave_read(mm_plan p, float* states, double* times, int* counts, long long* lost,
                                       mm_stream stream) {
    if (!p || !states || !times || !counts) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        const int n = p->ctl_host[b].save_n;
        const size_t off = (size_t)b * p->ring_cap;
        if (n > 0) {
            CUCHK(cudaMemcpyAsync(states + off * p->n3(), p->ring + off * p->n3(), sizeof(float) * p->n3() * n,
                                  cudaMemcpyDeviceToHost, st));
            CUCHK(cudaMemcpyAsync(times + off, p->ring_t + off, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
        }
        counts[b] = n;
        if (lost) lost[b] = p->ctl_host[b].save_lost;
        p->ctl_host[b].save_n = 0;
        p->ctl_host[b].save_lost = 0;
    }
    CUCHK(cudaStreamSynchronize(st));
    return write_ctl(p, st);
}

extern "C" MM_API int mm_tabulate_read(mm_plan p, double* out, int* counts, long long* lost, mm_stream stream) {
    if (!p || !out || !counts) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    if (p->rec_cap > 0)
        CUCHK(cudaMemcpyAsync(out, p->rec, sizeof(double) * 8 * (size_t)p->rec_cap * p->nsim, cudaMemcpyDeviceToHost,
                              st));
    CUCHK(cudaStreamSynchronize(st));
    for (int b = 0; b < p->nsim; b++) {
        counts[b] = p->ctl_host[b].tab_n;
        if (lost) lost[b] = p->ctl_host[b].tab_lost;
        p->ctl_host[b].tab_n = 0;
        p->ctl_host[b].tab_lost = 0;
    }
    return write_ctl(p, st);
}

extern "C" MM_API int mm_fields(mm_plan p, const float* m, long long noise_step, double dt_thermal, float* h_demag,
                                float* h_ex, float* h_anis, float* h_zee, float* h_therm, float* h_eff,
                                mm_stream stream) {
    if (!p || !m) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = standalone_time(p, st);
    if (rc) return rc;
    StageOp op = op_blank();
    op.m_in = fixed(const_cast<float*>(m));
    float* dbg[6] = {h_demag, h_ex, h_anis, h_zee, h_therm, h_eff};
    return launch_eval(p, op, nullptr, 0, dbg, noise_step, dt_thermal, nullptr, nullptr, st, nullptr);
}

static int normalize_launch(mm_plan p, float* m, cudaStream_t st) {
    const dim3 grid((unsigned)local_blocks(p->g.N, p->nsim), (unsigned)p->nsim);
    normalize_kernel<<<grid, 256, 0, st>>>(m, p->P.msat_mask, p->g.N, p->n3(), p->P.mask_bstride);
    CUCHK(cudaGetLastError());
    return MM_OK;
}

extern "C" MM_API int mm_torque(mm_plan p, float* m, long long noise_step, double dt_thermal, float* torque,
                                mm_stream stream) {
    if (!p || !m || !torque) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = standalone_time(p, st);
    if (rc) return rc;
    if ((rc = normalize_launch(p, m, st))) return rc;
    StageOp op = op_blank();
    op.m_in = fixed(m);
    op.k_out = fixed(torque);
    return launch_eval(p, op, nullptr, 0, nullptr, noise_step, dt_thermal, nullptr, nullptr, st, nullptr);
}

// ---------------------------------------------------------------- solvers
// Butcher tableaux.  Bogacki-Shampine 3(2) and Dormand-Prince 5(4), both FSAL.
static const double BS_A[4][4] = {{0, 0, 0, 0}, {0.5, 0, 0, 0}, {0, 0.75, 0, 0}, {2. / 9, 1. / 3, 4. / 9, 0}};
static const double BS_E[4] = {2. / 9 - 7. / 24, 1. / 3 - 1. / 4, 4. / 9 - 1. / 3, -1. / 8};
static const double DP_A[7][7] = {
    {0, 0, 0, 0, 0, 0, 0},
    {1. / 5, 0, 0, 0, 0, 0, 0},
    {3. / 40, 9. / 40, 0, 0, 0, 0, 0},
    {44. / 45, -56. / 15, 32. / 9, 0, 0, 0, 0},
    {19372. / 6561, -25360. / 2187, 64448. / 6561, -212. / 729, 0, 0, 0},
    {9017. / 3168, -355. / 33, 46732. / 5247, 49. / 176, -5103. / 18656, 0, 0},
    {35. / 384, 0, 500. / 1113, 125. / 192, -2187. / 6784, 11. / 84, 0}};
static const double DP_E[7] = {35. / 384 - 5179. / 57600, 0, 500. / 1113 - 7571. / 16695,
                               125. / 192 - 393. / 640, -2187. / 6784 + 92097. / 339200,
                               11. / 84 - 187. / 2100, -1. / 40};

static CombineArgs combine_args(mm_plan p, PP base, PP next, int nk, const PP* kp, const double* ak, int no_norm) {
    CombineArgs A;
    memset(&A, 0, sizeof A);
    A.no_norm = no_norm;
    A.base = base;
    A.next = next;
    A.nk = 0;
    for (int j = 0; j < nk; j++) {
        if (ak[j] == 0.0) continue;
        A.kp[A.nk] = kp[j];
        A.ak[A.nk] = ak[j];
        A.nk++;
    }
    A.msat_mask = p->P.msat_mask;
    A.N = p->g.N;
    A.bstride = p->n3();
    A.mask_bstride = p->P.mask_bstride;
    A.ctl = p->ctl;
    return A;
}

static int launch_combine(mm_plan p, PP base, PP next, int nk, const PP* kp, const double* ak, cudaStream_t st,
                          int no_norm = 0) {
    const CombineArgs A = combine_args(p, base, next, nk, kp, ak, no_norm);
    combine_kernel<<<dim3((unsigned)local_blocks(p->g.N, p->nsim), (unsigned)p->nsim), 256, 0, st>>>(A);
    CUCHK(cudaGetLastError());
    p->launches++;
    return MM_OK;
}

// The same stage state, also written as its R2C rows into the spectrum (where
// epi_r2c_ok(p)), so that the evaluation at `next` starts at its column pass
// (launch_eval with EVAL_ROWS_READY).
static int enqueue_combine_rows(mm_plan p, PP base, PP next, int nk, const PP* kp, const double* ak, cudaStream_t st) {
    PdlScope pdl_scope(p->pdl);
    const CombineArgs A = combine_args(p, base, next, nk, kp, ak, 0);
    CUCHK(launch_combine_rows(p->g.M, A, p->g.n, p->S, p->g.hp, p->g.L[1], p->spec_bstride(), p->tw,
                              p->khat_d ? 0 : 1, p->nsim, st));
    p->launches++;
    return MM_OK;
}

// One block over the plan's control blocks (see controller_kernel); also refreshes the
// summary the host polls.
static cudaError_t launch_controller(mm_plan p, cudaStream_t st, int mode, int adaptive, int q, int fsal, int nevals,
                                     int first_skippable) {
    PdlScope pdl_scope(p->pdl);
    const int threads = p->nsim >= 256 ? 256 : ((p->nsim + 31) / 32) * 32;
    return launch_pdl(controller_kernel, dim3(1), dim3(threads), 0, st, p->ctl, p->nsim, p->dsum, mode, adaptive, q,
                      fsal, nevals, first_skippable);
}

// blocks per simulation of the record sums
static int tab_blocks(mm_plan p) { return std::min(p->red_blocks, std::max(1, (148 * 2 + p->nsim - 1) / p->nsim)); }

// The autotabulate / autosave record kernels (no-ops unless a record is due).
static int launch_records(mm_plan p, cudaStream_t st) {
    if (!p->tab_on && !p->save_on) return MM_OK;
    const int nb = tab_blocks(p);
    if (p->tab_on) {
        tab_sum_kernel<<<dim3((unsigned)nb, (unsigned)p->nsim), 256, 0, st>>>(p->Y[0], p->Y[1], p->ctl, p->g.N,
                                                                              p->n3(), p->red);
        CUCHK(cudaGetLastError());
        p->launches++;
    }
    if (p->save_on) {
        save_copy_kernel<<<dim3((unsigned)local_blocks(p->n3(), p->nsim), (unsigned)p->nsim), 256, 0, st>>>(
            p->Y[0], p->Y[1], p->ctl, p->n3(), p->ring, p->ring_t);
        CUCHK(cudaGetLastError());
        p->launches++;
    }
    tab_finish_kernel<<<(p->nsim + 127) / 128, 128, 0, st>>>(p->red, nb, p->ctl, p->nsim, p->rec, p->g.N);
    CUCHK(cudaGetLastError());
    p->launches++;
    return MM_OK;
}

// One attempt of solver/am12 (am12.cu).  Buffers: y0 = Y[cur] (accepted state), the
// iterate y = Y[other] (accepted by flipping cur), dy0 = Kst[0], dy = Kst[1], the RHS at
// the Euler point = Kst[2], the predictor y1 = Ma.
static int enqueue_am12(mm_plan p, cudaStream_t st) {
    DevCtl* ctl = p->ctl;
    const int ns = p->nsim, bps = local_blocks(p->g.N, ns);
    const long long N = p->g.N;
    int rc;
    auto normalize = [&](PP m, int skip) -> int {
        CUCHK(am_normalize(m, p->P.msat_mask, ctl, N, p->P.mask_bstride, ns, bps, skip, st));
        p->launches++;
        return MM_OK;
    };
    auto eval = [&](PP m_in, float* k_out, int skip, double c_time, int want_tq) -> int {
        StageOp o = op_blank();
        o.m_in = m_in;
        o.k_out = fixed(k_out);
        o.want_tq = want_tq;
        o.c_time = c_time;
        return launch_eval(p, o, ctl, skip, nullptr, 0, 0, nullptr, nullptr, st, nullptr);
    };
    // dy0 = f(y0) at the start of the step (pulling m normalises it); reused by retries
    if ((rc = normalize(cur_of(p->Y), 1))) return rc;
    if ((rc = eval(cur_of(p->Y), p->Kst[0], 1, 0.0, 1))) return rc;
    if (p->run_until) {
        CUCHK(launch_controller(p, st, 2, 0, 0, 0, 0, 0));
        p->launches++;
    }
    CUCHK(am_begin(ctl, ns, st));
    p->launches++;
    // explicit Euler start y = y0 + h dy0 (not normalised), then f at t0 + dt
    {
        PP kp[1] = {fixed(p->Kst[0])};
        double ak[1] = {1.0};
        if ((rc = launch_combine(p, cur_of(p->Y), oth_of(p->Y), 1, kp, ak, st, 1))) return rc;
    }
    if ((rc = normalize(oth_of(p->Y), 2))) return rc;
    if ((rc = eval(oth_of(p->Y), p->Kst[1], 2, 1.0, 0))) return rc;
    CUCHK(am_copy(fixed(p->Kst[1]), fixed(p->Kst[2]), ctl, p->n3(), ns, bps, st));
    p->launches++;
    for (int loop = 0; loop < 2; loop++) {  // 0: implicit Euler predictor, 1: trapezoidal corrector
        if (loop == 1) {
            CUCHK(am_copy(oth_of(p->Y), fixed(p->Ma), ctl, p->n3(), ns, bps, st));
            CUCHK(am_copy(fixed(p->Kst[2]), fixed(p->Kst[1]), ctl, p->n3(), ns, bps, st));
            p->launches += 2;
        }
        for (int it = 0; it < 6; it++) {
            CUCHK(am_update(cur_of(p->Y), oth_of(p->Y), p->Kst[1], p->Kst[0], nullptr, ctl, N, ns, bps,
                            loop == 0 ? 0 : 1, st));
            CUCHK(am_test(ctl, ns, loop == 0, st));
            p->launches += 2;
            if (it < 5) {
                if ((rc = normalize(oth_of(p->Y), 2))) return rc;
                if ((rc = eval(oth_of(p->Y), p->Kst[1], 2, 1.0, 0))) return rc;
            }
        }
        CUCHK(am_between(ctl, ns, loop == 0, st));
        p->launches++;
    }
    CUCHK(am_update(cur_of(p->Y), oth_of(p->Y), nullptr, nullptr, p->Ma, ctl, N, ns, bps, 2, st));
    CUCHK(am_final(ctl, ns, st));
    p->launches += 2;
    CUCHK(launch_controller(p, st, 0, 0, 0, 0, 0, 0));
    p->launches++;
    return launch_records(p, st);
}

// Enqueues one step attempt of the configured solver (no host synchronisation).
static int enqueue_attempt(mm_plan p, cudaStream_t st) {
    DevCtl* ctl = p->ctl;
    int rc;
    const int s = p->solver;
    if (s == MM_AM12) return enqueue_am12(p, st);
    if (s == MM_EULER || s == MM_HEUN || s == MM_RK12) {
        // eval k0 at the accepted state
        StageOp o0 = op_blank();
        o0.m_in = cur_of(p->Y);
        o0.k_out = fixed(p->Kst[0]);
        o0.want_tq = 1;
        if (s == MM_EULER) {
            o0.do_combine = 1;
            o0.base_is_cur = 1;
            o0.next = oth_of(p->Y);
            o0.nk = 1;
            o0.kcur = 0;
            o0.kp[0] = fixed(p->Kst[0]);
            o0.ak[0] = 1.0;
        } else if (s == MM_HEUN) {
            o0.do_combine = 1;
            o0.base_is_cur = 1;
            o0.next = fixed(p->Ma);
            o0.nk = 1;
            o0.kcur = 0;
            o0.kp[0] = fixed(p->Kst[0]);
            o0.ak[0] = 1.0;
        }
        const int skip = (s == MM_RK12) ? 1 : 0;
        o0.c_time = 0.0;
        // Heun's predictor Ma is the corrector's input: its rows come from this epilogue
        const int fwd0 = (s == MM_HEUN) ? EVAL_EMIT_ROWS : 0;
        if ((rc = launch_eval(p, o0, ctl, skip, nullptr, 0, 0, nullptr, nullptr, st, nullptr, fwd0))) return rc;
        if (p->run_until) {
            CUCHK(launch_controller(p, st, 2, 0, 0, 0, 0, 0));
            p->launches++;
        }
        // RK12: the corrector's input, the Euler predictor, comes with its R2C rows
        const bool rows12 = (s == MM_RK12) && epi_r2c_ok(p);
        if (s == MM_RK12) {
            // Euler predictor from the saved k0 (solve_rk12.go:133), also on retries
            PP kp[1] = {fixed(p->Kst[0])};
            double ak[1] = {1.0};
            if ((rc = rows12 ? enqueue_combine_rows(p, cur_of(p->Y), fixed(p->Ma), 1, kp, ak, st)
                             : launch_combine(p, cur_of(p->Y), fixed(p->Ma), 1, kp, ak, st)))
                return rc;
        }
        if (s == MM_HEUN || s == MM_RK12) {
            // corrector: y = y_pred + h/2 k1 - h/2 k0 (solve_rk12.go:154, solve_heun.go:63)
            StageOp o1 = op_blank();
            o1.m_in = fixed(p->Ma);
            o1.c_time = 1.0;  // the corrector is evaluated at t + dt (solve_rk12.go:138, solve_heun.go:56)
            o1.do_combine = 1;
            o1.base_is_cur = 1;
            o1.next = oth_of(p->Y);
            o1.nk = 2;
            o1.kcur = 0;
            o1.kp[0] = none();
            o1.ak[0] = 0.5;
            o1.kp[1] = fixed(p->Kst[0]);
            o1.ak[1] = -0.5;
            if (s == MM_RK12) {
                o1.ne = 2;
                o1.ecur = 0;
                o1.ep[0] = none();
                o1.ek[0] = 1.0;
                o1.ep[1] = fixed(p->Kst[0]);
                o1.ek[1] = -1.0;
            }
            const int fwd1 = (s == MM_HEUN || rows12) ? EVAL_ROWS_READY : 0;
            if ((rc = launch_eval(p, o1, ctl, 0, nullptr, 0, 0, nullptr, nullptr, st, nullptr, fwd1))) return rc;
        }
        CUCHK(launch_controller(p, st, 1, s == MM_RK12 ? 1 : 0, 1, 0, s == MM_EULER ? 1 : 2, s == MM_RK12));
        p->launches++;
        return launch_records(p, st);
    }
    // RK23 / RK45 (FSAL): K1[cur] = f(Y[cur]) is valid
    const bool dp = (s == MM_RK45);
    const int S = dp ? 7 : 4;
    auto A = [&](int i, int j) { return dp ? DP_A[i][j] : BS_A[i][j]; };
    const double* E = dp ? DP_E : BS_E;
    // k-buffer of stage j: stage 0 = K1[cur], stages 1..S-2 = Kst[j-1], stage S-1 = K1[other]
    auto kbuf = [&](int j) -> PP {
        if (j == 0) return cur_of(p->K1);
        if (j == S - 1) return oth_of(p->K1);
        return fixed(p->Kst[j - 1]);
    };
    // stage-state buffer of stage i (1..S-1): alternate Ma/Mb, the last is Y[other]
    auto mbuf = [&](int i) -> PP {
        if (i == S - 1) return oth_of(p->Y);
        return fixed((i & 1) ? p->Ma : p->Mb);
    };
    // the first stage state, with its R2C rows where the plan allows
    const bool rows1 = epi_r2c_ok(p);
    {
        PP kp[1] = {kbuf(0)};
        double ak[1] = {A(1, 0)};
        if ((rc = rows1 ? enqueue_combine_rows(p, cur_of(p->Y), mbuf(1), 1, kp, ak, st)
                        : launch_combine(p, cur_of(p->Y), mbuf(1), 1, kp, ak, st)))
            return rc;
    }
    for (int i = 1; i < S; i++) {
        StageOp o = op_blank();
        o.m_in = mbuf(i);
        o.k_out = kbuf(i);
        for (int j = 0; j < i; j++) o.c_time += A(i, j);  // stage time t + c_i dt
        if (i + 1 < S) {
            o.do_combine = 1;
            o.base = cur_of(p->Y);
            o.next = mbuf(i + 1);
            o.nk = 0;
            for (int j = 0; j <= i; j++) {
                double a = A(i + 1, j);
                if (a == 0.0) continue;
                if (j == i) o.kcur = o.nk;
                o.kp[o.nk] = (j == i) ? none() : kbuf(j);
                o.ak[o.nk] = a;
                o.nk++;
            }
        } else {
            o.want_tq = 1;
            o.ne = 0;
            for (int j = 0; j < S; j++) {
                if (E[j] == 0.0) continue;
                if (j == i) o.ecur = o.ne;
                o.ep[o.ne] = (j == i) ? none() : kbuf(j);
                o.ek[o.ne] = E[j];
                o.ne++;
            }
        }
        // stage i + 1 reads mbuf(i + 1), which this epilogue forms: its rows come from here
        int fwd = (i + 1 < S) ? EVAL_EMIT_ROWS : 0;
        if (i > 1 || rows1) fwd |= EVAL_ROWS_READY;
        if ((rc = launch_eval(p, o, ctl, 0, nullptr, 0, 0, nullptr, nullptr, st, nullptr, fwd))) return rc;
    }
    CUCHK(launch_controller(p, st, 1, 1, dp ? 4 : 2, 1, S - 1, 0));
    p->launches++;
    return launch_records(p, st);
}

static int read_ctl(mm_plan p, cudaStream_t st) {
    CUCHK(cudaMemcpyAsync(p->ctl_host, p->ctl, sizeof(DevCtl) * p->nsim, cudaMemcpyDeviceToHost, st));
    CUCHK(cudaStreamSynchronize(st));
    return MM_OK;
}
static int write_ctl(mm_plan p, cudaStream_t st) {
    CUCHK(cudaMemcpyAsync(p->ctl, p->ctl_host, sizeof(DevCtl) * p->nsim, cudaMemcpyHostToDevice, st));
    CUCHK(cudaStreamSynchronize(st));
    return MM_OK;
}

extern "C" MM_API int mm_solver_init(mm_plan p, int solver, double dt, double mindt, double maxdt, double maxerr) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (solver < MM_EULER || solver > MM_AM12) return set_err(MM_ERR_ARG, "unknown solver %d", solver);
    if (!(dt > 0) || !(mindt > 0) || !(maxdt > 0) || !(maxerr > 0)) return set_err(MM_ERR_ARG, "dt, mindt, maxdt, maxerr must be > 0");
    p->solver = solver;
    free_graph(p);
    int rc = read_ctl(p, 0);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        c.dt = dt;
        p->dt0 = dt;
        c.mindt = mindt;
        c.maxdt = maxdt;
        c.maxerr = maxerr;
        c.headroom = 0.8;
        c.gamma = p->prob.gamma;
        c.h = dt * c.gamma;
        c.fsal_valid = 0;
        c.tries = 0;
        c.status = MM_OK;
        if (c.am_abs_err <= 0) c.am_abs_err = 1e-4;  // solve_am01.go:355-358 defaults
        if (c.am_rel_err <= 0) c.am_rel_err = 1e-3;
        c.am_restrict = 0;
    }
    return write_ctl(p, 0);
}

extern "C" MM_API int mm_solver_am12_tolerances(mm_plan p, double abs_err, double rel_err) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (!(abs_err > 0) || !(rel_err > 0)) return set_err(MM_ERR_ARG, "tolerances must be > 0");
    int rc = read_ctl(p, 0);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        p->ctl_host[b].am_abs_err = abs_err;
        p->ctl_host[b].am_rel_err = rel_err;
    }
    return write_ctl(p, 0);
}

// Batched plans keep every accepted state in the first ping-pong buffer between runs, so
// that state transfers and reductions see one layout.
static int canonicalise(mm_plan p, cudaStream_t st) {
    if (p->nsim == 1) return MM_OK;
    const dim3 grid((unsigned)local_blocks(p->g.N, p->nsim), (unsigned)p->nsim);
    canonical_copy_kernel<<<grid, 256, 0, st>>>(p->Y[0], p->Y[1], p->K1[0], p->K1[1], p->ctl, p->n3());
    CUCHK(cudaGetLastError());
    reset_cur_kernel<<<(p->nsim + 255) / 256, 256, 0, st>>>(p->ctl, p->nsim);
    CUCHK(cudaGetLastError());
    return MM_OK;
}

// device pointer of the accepted state (read_ctl must have run)
static float* state_ptr(mm_plan p) { return p->Y[p->ctl_host[0].cur]; }

extern "C" MM_API int mm_set_state(mm_plan p, const float* m, int from_host, mm_stream stream) {
    if (!p || !m) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    if (p->nsim > 1)
        for (int b = 0; b < p->nsim; b++) p->ctl_host[b].cur = 0;
    float* dst = state_ptr(p);
    CUCHK(cudaMemcpyAsync(dst, m, sizeof(float) * p->n3() * p->nsim,
                          from_host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
    if ((rc = normalize_launch(p, dst, st))) return rc;
    for (int b = 0; b < p->nsim; b++) p->ctl_host[b].fsal_valid = 0;
    p->state_set = true;
    return write_ctl(p, st);
}

extern "C" MM_API int mm_get_state(mm_plan p, float* m, int to_host, mm_stream stream) {
    if (!p || !m) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    CUCHK(cudaMemcpyAsync(m, state_ptr(p), sizeof(float) * p->n3() * p->nsim,
                          to_host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, st));
    CUCHK(cudaStreamSynchronize(st));
    return MM_OK;
}

extern "C" MM_API int mm_set_time(mm_plan p, double t, double dt) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    int rc = read_ctl(p, 0);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        p->ctl_host[b].t = t;
        if (dt > 0) {
            p->ctl_host[b].dt = dt;
            p->ctl_host[b].h = dt * p->ctl_host[b].gamma;
        }
    }
    return write_ctl(p, 0);
}

extern "C" MM_API int mm_set_thermal_dt(mm_plan p, double dt_thermal) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    int rc = read_ctl(p, 0);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) p->ctl_host[b].dt_thermal = dt_thermal;
    return write_ctl(p, 0);
}

// FSAL solvers need f(Y[cur]) before the first attempt.
static int ensure_fsal(mm_plan p, cudaStream_t st) {
    if (p->solver != MM_RK23 && p->solver != MM_RK45) return MM_OK;
    bool all = true;
    for (int b = 0; b < p->nsim; b++) all = all && p->ctl_host[b].fsal_valid;
    if (all) return MM_OK;
    // a standalone evaluation with the control blocks (done = 0 at this point)
    StageOp o = op_blank();
    o.m_in = cur_of(p->Y);
    o.k_out = cur_of(p->K1);
    o.want_tq = 1;
    int rc = launch_eval(p, o, p->ctl, 0, nullptr, 0, 0, nullptr, nullptr, st, nullptr);
    if (rc) return rc;
    if ((rc = read_ctl(p, st))) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        float tqv;
        memcpy(&tqv, &c.tq_bits, sizeof tqv);
        c.maxtorque = sqrt((double)tqv) * c.gamma;
        c.tq_bits = 0;
        c.fsal_valid = 1;
    }
    return write_ctl(p, st);
}

static int capture_attempt(mm_plan p) {
    if (p->graph && p->graph_solver == p->solver && p->graph_run_until == p->run_until) return MM_OK;
    free_graph(p);
    cudaStream_t cs;
    CUCHK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaGraph_t gr;
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) { cudaStreamDestroy(cs); return set_err(MM_ERR_CUDA, "begin capture: %s", cudaGetErrorString(e)); }
    const long long before = p->launches;
    int rc = enqueue_attempt(p, cs);
    p->graph_nodes = (int)(p->launches - before);
    p->launches = before;
    e = cudaStreamEndCapture(cs, &gr);
    cudaStreamDestroy(cs);
    if (rc) return rc;
    if (e != cudaSuccess) return set_err(MM_ERR_CUDA, "end capture: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(&p->graph, gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) { p->graph = nullptr; return set_err(MM_ERR_CUDA, "instantiate: %s", cudaGetErrorString(e)); }
    p->graph_solver = p->solver;
    p->graph_run_until = p->run_until;
    return MM_OK;
}

extern "C" MM_API int mm_queue_attempts(mm_plan p, int attempts, mm_stream stream) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (p->solver < 0) return set_err(MM_ERR_STATE, "no solver: call mm_solver_init");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = capture_attempt(p);
    if (rc) return rc;
    for (int a = 0; a < attempts; a++) CUCHK(cudaGraphLaunch(p->graph, st));
    p->launches += (long long)attempts * p->graph_nodes;
    return MM_OK;
}

static int read_summary(mm_plan p, cudaStream_t st) {
    CUCHK(cudaMemcpyAsync(p->hsum, p->dsum, sizeof(CtlSummary), cudaMemcpyDeviceToHost, st));
    CUCHK(cudaStreamSynchronize(st));
    return MM_OK;
}

static int summary_status(mm_plan p) {
    const CtlSummary& s = *p->hsum;
    if (s.status == MM_OK) return MM_OK;
    const char* who = p->nsim > 1 ? " of simulation " : "";
    char num[32] = "";
    if (p->nsim > 1) snprintf(num, sizeof num, "%d", s.bad_sim);
    if (s.status == MM_ERR_NAN) return set_err(MM_ERR_NAN, "NaN in the torque at step %lld%s%s", s.step, who, num);
    if (s.status == MM_ERR_RANGE)
        return set_err(MM_ERR_RANGE, "time past the end of a time table (step %lld%s%s)", s.step, who, num);
    return set_err(s.status, "solver cannot converge after 10 bad steps (step %lld%s%s)", s.step, who, num);
}

// Attempts to queue next: no more than the largest number of accepted steps an active
// simulation still needs (so fixed-count runs launch no no-op attempts), doubling from 4
// up to 64 while the end is not known in steps.
static int next_batch(long long max_left, int grow) {
    long long b = grow;
    if (max_left > 0 && max_left < b) b = max_left;
    return (int)std::max(1LL, b);
}

// Runs attempts until the device sets `done` for every simulation.  The host only polls
// the summary between batches of queued attempts.
static int drive(mm_plan p, cudaStream_t st, long long max_attempts, int target_active = 0) {
    int grow = 4;
    long long launched = 0;
    long long max_left = 0;
    for (int b = 0; b < p->nsim; b++)
        if (!p->ctl_host[b].done) max_left = std::max(max_left, p->ctl_host[b].step_end - p->ctl_host[b].step);
    for (;;) {
        const int batch = next_batch(max_left, grow);
        int rc = mm_queue_attempts(p, batch, (mm_stream)st);
        if (rc) return rc;
        launched += batch;
        if ((rc = read_summary(p, st))) return rc;
        if ((rc = summary_status(p))) return rc;
        if (p->hsum->active <= target_active) return MM_OK;
        if (max_attempts > 0 && launched >= max_attempts) return set_err(MM_ERR_TIMEOUT, "attempt limit reached");
        max_left = p->hsum->max_left;
        if (grow < 64) grow *= 2;
    }
}

// Sets every simulation's stop condition: t_end = t + duration (duration > 0), or
// step_end = step + nsteps (nsteps > 0), or maxtorque < thr (thr_sim[b] if given).
static int start_run(mm_plan p, cudaStream_t st, double duration, long long nsteps, double thr,
                     long long max_steps, const double* thr_sim = nullptr) {
    if (p->solver < 0) return set_err(MM_ERR_STATE, "no solver: call mm_solver_init");
    if (!p->state_set) return set_err(MM_ERR_STATE, "no state: call mm_set_state");
    int rc = read_ctl(p, st);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        c.done = 0;
        c.status = MM_OK;
        c.tries = 0;
        c.t_end = duration > 0 ? c.t + duration : 1e300;
        c.step_end = nsteps > 0 ? c.step + nsteps : (max_steps > 0 ? c.step + max_steps : (1LL << 62));
        c.torque_thr = thr_sim ? thr_sim[b] : thr;
        c.err_bits = 0;
        c.tq_bits = 0;
        c.gamma = p->prob.gamma;
        c.h = c.dt * c.gamma;
        if (duration > 0 && !(c.t < c.t_end)) c.done = 1;
    }
    p->run_until = thr > 0;
    if ((rc = write_ctl(p, st))) return rc;
    if ((rc = ensure_fsal(p, st))) return rc;
    if (thr > 0 && (p->solver == MM_RK23 || p->solver == MM_RK45)) {
        if ((rc = read_ctl(p, st))) return rc;
        for (int b = 0; b < p->nsim; b++)
            if (p->ctl_host[b].maxtorque < p->ctl_host[b].torque_thr) p->ctl_host[b].done = 1;
        return write_ctl(p, st);
    }
    return MM_OK;
}

static int finish_run(mm_plan p, cudaStream_t st) {
    int rc = canonicalise(p, st);
    if (rc) return rc;
    if (p->solver == MM_AM12) {
        // AM12 leaves its last iterate unnormalised; reading m normalises it
        CUCHK(am_normalize(cur_of(p->Y), p->P.msat_mask, p->ctl, p->g.N, p->P.mask_bstride, p->nsim,
                           local_blocks(p->g.N, p->nsim), 0, st));
    }
    if ((rc = read_ctl(p, st))) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        c.done = 1;
        c.t_end = 1e300;
        c.step_end = (1LL << 62);
        c.torque_thr = 0;
    }
    p->run_until = false;
    return write_ctl(p, st);
}

static bool any_active(mm_plan p) {
    for (int b = 0; b < p->nsim; b++)
        if (!p->ctl_host[b].done) return true;
    return false;
}

static int run_plan(mm_plan p, cudaStream_t st, double duration, long long nsteps, double thr, long long max_steps,
                    const double* thr_sim = nullptr) {
    int rc = start_run(p, st, duration, nsteps, thr, max_steps, thr_sim);
    if (rc) return rc;
    if (any_active(p)) rc = drive(p, st, 0);
    int rc2 = finish_run(p, st);
    return rc ? rc : rc2;
}

extern "C" MM_API int mm_run(mm_plan p, double duration, mm_stream stream) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (!(duration > 0)) return MM_OK;
    return run_plan(p, (cudaStream_t)stream, duration, 0, 0, 0);
}

extern "C" MM_API int mm_steps(mm_plan p, long long n, mm_stream stream) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (n <= 0) return MM_OK;
    return run_plan(p, (cudaStream_t)stream, 0, n, 0, 0);
}

extern "C" MM_API int mm_step(mm_plan p, mm_stream stream) { return mm_steps(p, 1, stream); }

extern "C" MM_API int mm_run_until_maxtorque(mm_plan p, double thr, long long max_steps, mm_stream stream) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (!(thr > 0)) return set_err(MM_ERR_ARG, "threshold must be > 0");
    return run_plan(p, (cudaStream_t)stream, 0, 0, thr, max_steps);
}

extern "C" MM_API int mm_batch_run_until_maxtorque(mm_plan p, const double* thr, long long max_steps,
                                                   mm_stream stream) {
    if (!p || !thr) return set_err(MM_ERR_ARG, "null argument");
    for (int b = 0; b < p->nsim; b++)
        if (!(thr[b] > 0)) return set_err(MM_ERR_ARG, "threshold of simulation %d must be > 0", b);
    return run_plan(p, (cudaStream_t)stream, 0, 0, 1.0, max_steps, thr);
}

static void stats_of(const DevCtl& c, mm_stats* out) {
    out->t = c.t;
    out->dt = c.dt;
    out->err = c.err;
    out->peakerr = c.peakerr;
    out->maxtorque = c.maxtorque;
    out->step = c.step;
    out->badsteps = c.badsteps;
    out->attempts = c.attempts;
    out->evals = c.evals;
    out->status = c.status;
    out->done = c.done;
    out->iterations = c.am_iterations;
}

static int single(mm_plan p) {
    if (p->nsim != 1)
        return set_err(MM_ERR_ARG, "plan holds %d simulations: use the mm_batch_* variant", p->nsim);
    return MM_OK;
}

extern "C" MM_API int mm_batch_stats(mm_plan p, mm_stats* out, mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    int rc = read_ctl(p, (cudaStream_t)stream);
    if (rc) return rc;
    for (int b = 0; b < p->nsim; b++) stats_of(p->ctl_host[b], out + b);
    return MM_OK;
}

extern "C" MM_API int mm_get_stats(mm_plan p, mm_stats* out, mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    int rc = single(p);
    return rc ? rc : mm_batch_stats(p, out, stream);
}

// ---------------------------------------------------------------- reductions of the state
extern "C" MM_API int mm_batch_maxtorque(mm_plan p, double* out, mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    const DevCtl& c0 = p->ctl_host[0];
    if ((rc = standalone_time(p, st))) return rc;
    CUCHK(cudaMemsetAsync(p->tq, 0, sizeof(unsigned int) * p->nsim, st));
    StageOp o = op_blank();
    o.m_in = fixed(state_ptr(p));
    o.k_out = fixed(p->Mtmp);
    o.want_tq = 1;
    if ((rc = launch_eval(p, o, nullptr, 0, nullptr, c0.noise_step, c0.dt_thermal > 0 ? c0.dt_thermal : c0.dt,
                          nullptr, p->tq, st, nullptr)))
        return rc;
    std::vector<unsigned int> bits(p->nsim);
    CUCHK(cudaMemcpyAsync(bits.data(), p->tq, sizeof(unsigned int) * p->nsim, cudaMemcpyDeviceToHost, st));
    CUCHK(cudaStreamSynchronize(st));
    for (int b = 0; b < p->nsim; b++) {
        float v;
        memcpy(&v, &bits[b], sizeof v);
        out[b] = sqrt((double)v) * p->prob.gamma;
    }
    return MM_OK;
}

extern "C" MM_API int mm_maxtorque(mm_plan p, double* out, mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    int rc = single(p);
    return rc ? rc : mm_batch_maxtorque(p, out, stream);
}

extern "C" MM_API int mm_batch_average(mm_plan p, double* out, mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    const int nb = std::min(p->red_blocks, std::max(1, (148 * 2 + p->nsim - 1) / p->nsim));
    sum3_kernel<<<dim3((unsigned)nb, (unsigned)p->nsim), 256, 0, st>>>(state_ptr(p), p->g.N, p->n3(), p->red);
    CUCHK(cudaGetLastError());
    energy_finish_kernel<<<(p->nsim * 4 + 127) / 128, 128, 0, st>>>(p->red, nb, p->dres, p->nsim);
    CUCHK(cudaGetLastError());
    std::vector<double> r(4 * (size_t)p->nsim);
    CUCHK(cudaMemcpyAsync(r.data(), p->dres, sizeof(double) * r.size(), cudaMemcpyDeviceToHost, st));
    CUCHK(cudaStreamSynchronize(st));
    for (int b = 0; b < p->nsim; b++)
        for (int c = 0; c < 3; c++) out[3 * b + c] = r[4 * b + c] / (double)p->g.N;
    return MM_OK;
}

extern "C" MM_API int mm_average(mm_plan p, double out[3], mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    int rc = single(p);
    return rc ? rc : mm_batch_average(p, out, stream);
}

extern "C" MM_API int mm_batch_energy(mm_plan p, double* out, mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    if ((rc = standalone_time(p, st))) return rc;
    StageOp o = op_blank();
    o.m_in = fixed(state_ptr(p));
    o.want_energy = 1;
    // thermal noise does not enter the energy terms
    int nb = 0;
    if ((rc = launch_eval(p, o, nullptr, 0, nullptr, 0, 1.0, p->red, nullptr, st, &nb))) return rc;
    energy_finish_kernel<<<(p->nsim * 4 + 127) / 128, 128, 0, st>>>(p->red, nb, p->dres, p->nsim);
    CUCHK(cudaGetLastError());
    std::vector<double> r(4 * (size_t)p->nsim);
    CUCHK(cudaMemcpyAsync(r.data(), p->dres, sizeof(double) * r.size(), cudaMemcpyDeviceToHost, st));
    CUCHK(cudaStreamSynchronize(st));
    const mm_problem& q = p->prob;
    const double V = q.cell[0] * q.cell[1] * q.cell[2];
    for (int b = 0; b < p->nsim; b++) {
        const double ms = p->sims[b].msat;
        double* e = out + 5 * b;
        const double* rb = r.data() + 4 * b;
        e[0] = q.zeeman ? -V * rb[0] * ms : 0.0;
        e[1] = q.exchange ? -0.5 * V * MU0 * rb[1] * ms : 0.0;
        e[2] = q.demag ? -0.5 * V * MU0 * rb[2] * ms : 0.0;
        e[3] = q.anis ? -0.5 * V * MU0 * rb[3] * ms : 0.0;
        e[4] = e[0] + e[1] + e[2] + e[3];
    }
    return MM_OK;
}

extern "C" MM_API int mm_energy(mm_plan p, double out[5], mm_stream stream) {
    if (!p || !out) return set_err(MM_ERR_ARG, "null argument");
    int rc = single(p);
    return rc ? rc : mm_batch_energy(p, out, stream);
}

extern "C" MM_API long long mm_plan_launch_count(mm_plan p) { return p ? p->launches : 0; }

// Times each pass of one right-hand-side evaluation (at the accepted state, result
// discarded) with CUDA events recorded on the launching stream between the passes;
// ms_out[i] = average duration of pass i over `reps` evaluations.  Pass order:
// 3-D: xfwd, y fwd, z mul, y inv, x inv + epilogue; 2-D: xfwd, y mul, x inv + epilogue;
// no demag: epilogue only.  Batched plans time all simulations together.
extern "C" MM_API int mm_profile_eval(mm_plan p, int reps, double* ms_out, int* npass, mm_stream stream) {
    if (!p || !ms_out || !npass || reps < 1) return set_err(MM_ERR_ARG, "bad argument");
    PdlScope pdl_scope(p->pdl);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    const ConvGeom& g = p->g;
    StageOp op = op_blank();
    op.m_in = fixed(state_ptr(p));
    op.k_out = fixed(p->Mtmp);
    EpiArgs A;
    memset(&A, 0, sizeof A);
    A.P = p->P;
    A.op = op;
    A.spec_bstride = p->spec_bstride();
    const int np = p->demag ? (g.L[0] == 1 ? 3 : 5) : 1;
    *npass = np;
    std::vector<cudaEvent_t> ev(np + 1);
    for (auto& e : ev) CUCHK(cudaEventCreate(&e));
    std::vector<double> acc(np, 0.0);
    const long long launches0 = p->launches;
    for (int r = -1; r < reps; r++) {  // r = -1: untimed warm-up evaluation
        CUCHK(cudaEventRecord(ev[0], st));
        int nb = 0;
        if (p->demag) {
            if ((rc = launch_conv(p, op.m_in, nullptr, 0, st, &ev))) return rc;
            CUCHK(launch_xinv_epi(g.M, p->S, g.hp, g.L[1], p->tw, A, false, st, &nb, p->nsim));
        } else {
            CUCHK(launch_local_epi(A, false, st, &nb, p->nsim));
        }
        CUCHK(cudaEventRecord(ev[np], st));
        CUCHK(cudaEventSynchronize(ev[np]));
        if (r < 0) continue;
        for (int i = 0; i < np; i++) {
            float ms = 0.f;
            CUCHK(cudaEventElapsedTime(&ms, ev[i], ev[i + 1]));
            acc[i] += ms;
        }
    }
    p->launches = launches0 + (long long)(reps + 1) * np;
    for (int i = 0; i < np; i++) ms_out[i] = acc[i] / reps;
    for (auto& e : ev) cudaEventDestroy(e);
    return MM_OK;
}

// Geometry of the plan's transform: L[3], M, h, hp, kd[3], nonzero kernel components.
extern "C" MM_API int mm_plan_geometry(mm_plan p, int* out12) {
    if (!p || !out12) return set_err(MM_ERR_ARG, "bad argument");
    const ConvGeom& g = p->g;
    int v[12] = {g.L[0], g.L[1], g.L[2], g.M, g.h, g.hp, g.kd[0], g.kd[1], g.kd[2], 0, 0, 0};
    int nzc = 0;
    for (int q = 0; q < 6; q++) nzc += p->demag ? p->kv.nz[q] : 0;
    v[9] = nzc;
    v[10] = p->demag ? 1 : 0;
    v[11] = p->nsim;
    memcpy(out12, v, sizeof v);
    return MM_OK;
}

// ---------------------------------------------------------------- ensembles
// Plans of different geometry stepped together: one CUDA graph whose branches (one per
// plan, forked from and joined to the capture stream) each replay K attempts of that
// plan.  Branches share no buffers, so the GPU overlaps the small plans' launches.
struct mm_ensemble_s {
    std::vector<mm_plan> plans;
    int K = 16;
    std::vector<cudaStream_t> streams;
    cudaEvent_t fork = nullptr;
    std::vector<cudaEvent_t> joins;
    cudaGraphExec_t graph = nullptr;
    std::vector<long long> versions;  // plan versions the graph was captured from
    long long nodes = 0;
    long long launches = 0;
};

extern "C" MM_API int mm_ensemble_destroy(mm_ensemble e) {
    if (!e) return MM_OK;
    if (e->graph) cudaGraphExecDestroy(e->graph);
    for (auto s : e->streams) cudaStreamDestroy(s);
    for (auto j : e->joins) cudaEventDestroy(j);
    if (e->fork) cudaEventDestroy(e->fork);
    delete e;
    return MM_OK;
}

extern "C" MM_API int mm_ensemble_create(const mm_plan* plans, int nplans, int attempts_per_launch,
                                         mm_ensemble* out) {
    if (!plans || !out || nplans < 1) return set_err(MM_ERR_ARG, "need at least one plan");
    if (attempts_per_launch < 1 || attempts_per_launch > 1024) return set_err(MM_ERR_ARG, "attempts_per_launch in 1..1024");
    *out = nullptr;
    for (int i = 0; i < nplans; i++) {
        if (!plans[i]) return set_err(MM_ERR_ARG, "plan %d is null", i);
        for (int j = 0; j < i; j++)
            if (plans[j] == plans[i]) return set_err(MM_ERR_ARG, "plan %d appears twice", i);
    }
    mm_ensemble e = new mm_ensemble_s();
    e->plans.assign(plans, plans + nplans);
    e->K = attempts_per_launch;
    e->streams.resize(nplans, nullptr);
    e->joins.resize(nplans, nullptr);
    cudaError_t err = cudaEventCreateWithFlags(&e->fork, cudaEventDisableTiming);
    for (int i = 0; i < nplans && err == cudaSuccess; i++) {
        err = cudaStreamCreateWithFlags(&e->streams[i], cudaStreamNonBlocking);
        if (err == cudaSuccess) err = cudaEventCreateWithFlags(&e->joins[i], cudaEventDisableTiming);
    }
    if (err != cudaSuccess) {
        mm_ensemble_destroy(e);
        return set_err(MM_ERR_CUDA, "ensemble streams/events: %s", cudaGetErrorString(err));
    }
    *out = e;
    return MM_OK;
}

static int ensemble_capture(mm_ensemble e) {
    bool fresh = e->graph != nullptr && e->versions.size() == e->plans.size();
    for (size_t i = 0; fresh && i < e->plans.size(); i++) fresh = e->versions[i] == e->plans[i]->version;
    if (fresh) return MM_OK;
    if (e->graph) { cudaGraphExecDestroy(e->graph); e->graph = nullptr; }
    cudaStream_t cs;
    CUCHK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaError_t err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (err != cudaSuccess) { cudaStreamDestroy(cs); return set_err(MM_ERR_CUDA, "begin capture: %s", cudaGetErrorString(err)); }
    int rc = MM_OK;
    long long nodes = 0;
    err = cudaEventRecord(e->fork, cs);
    for (size_t i = 0; i < e->plans.size() && rc == MM_OK && err == cudaSuccess; i++) {
        mm_plan p = e->plans[i];
        err = cudaStreamWaitEvent(e->streams[i], e->fork, 0);
        const long long before = p->launches;
        for (int k = 0; k < e->K && rc == MM_OK && err == cudaSuccess; k++) rc = enqueue_attempt(p, e->streams[i]);
        nodes += p->launches - before;
        p->launches = before;
        if (err == cudaSuccess) err = cudaEventRecord(e->joins[i], e->streams[i]);
        if (err == cudaSuccess) err = cudaStreamWaitEvent(cs, e->joins[i], 0);
    }
    cudaGraph_t gr = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(cs, &gr);
    cudaStreamDestroy(cs);
    if (rc) { if (gr) cudaGraphDestroy(gr); return rc; }
    if (err != cudaSuccess || e2 != cudaSuccess) {
        if (gr) cudaGraphDestroy(gr);
        return set_err(MM_ERR_CUDA, "ensemble capture: %s", cudaGetErrorString(err != cudaSuccess ? err : e2));
    }
    err = cudaGraphInstantiate(&e->graph, gr, 0);
    cudaGraphDestroy(gr);
    if (err != cudaSuccess) { e->graph = nullptr; return set_err(MM_ERR_CUDA, "instantiate: %s", cudaGetErrorString(err)); }
    e->nodes = nodes;
    e->versions.resize(e->plans.size());
    for (size_t i = 0; i < e->plans.size(); i++) e->versions[i] = e->plans[i]->version;
    return MM_OK;
}

static int ensemble_drive(mm_ensemble e, cudaStream_t st, double duration, long long nsteps) {
    int rc = MM_OK;
    size_t started = 0;
    for (; started < e->plans.size() && rc == MM_OK; started++) {
        mm_plan p = e->plans[started];
        rc = start_run(p, st, duration, nsteps, 0, 0);
        if (rc == MM_OK && p->run_until) rc = set_err(MM_ERR_STATE, "internal: run_until set");
    }
    if (rc == MM_OK) rc = ensemble_capture(e);
    while (rc == MM_OK) {
        bool active = false;
        for (mm_plan p : e->plans) active = active || any_active(p);
        if (!active) break;
        CUCHK(cudaGraphLaunch(e->graph, st));
        e->launches += e->nodes;
        for (size_t i = 0; i < e->plans.size() && rc == MM_OK; i++) {
            mm_plan p = e->plans[i];
            CUCHK(cudaMemcpyAsync(p->hsum, p->dsum, sizeof(CtlSummary), cudaMemcpyDeviceToHost, st));
        }
        CUCHK(cudaStreamSynchronize(st));
        for (size_t i = 0; i < e->plans.size() && rc == MM_OK; i++) {
            mm_plan p = e->plans[i];
            rc = summary_status(p);
            for (int b = 0; b < p->nsim; b++) p->ctl_host[b].done = p->hsum->active == 0 ? 1 : 0;
        }
    }
    for (size_t i = 0; i < started; i++) {
        int rc2 = finish_run(e->plans[i], st);
        if (rc == MM_OK) rc = rc2;
    }
    return rc;
}

extern "C" MM_API int mm_ensemble_steps(mm_ensemble e, long long n, mm_stream stream) {
    if (!e) return set_err(MM_ERR_ARG, "null ensemble");
    if (n <= 0) return MM_OK;
    return ensemble_drive(e, (cudaStream_t)stream, 0, n);
}

extern "C" MM_API int mm_ensemble_run(mm_ensemble e, double duration, mm_stream stream) {
    if (!e) return set_err(MM_ERR_ARG, "null ensemble");
    if (!(duration > 0)) return MM_OK;
    return ensemble_drive(e, (cudaStream_t)stream, duration, 0);
}

extern "C" MM_API long long mm_ensemble_launch_count(mm_ensemble e) { return e ? e->launches : 0; }

// ---------------------------------------------------------------- asynchronous snapshots
extern "C" MM_API int mm_write_field(const char* path, int format, const float* data, int ncomp, const int n[3],
                                     const double cell[3], double time, const char* name, const char* unit);

// copies the accepted state (resolved on the device) and the time to the staging buffers
__global__ void snapshot_kernel(PP y, const DevCtl* ctl, float* dst, long long n, double* t_out) {
    const float* src = y.get(ctl->cur);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = src[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) *t_out = ctl->t;
}

extern "C" MM_API int mm_save_wait(mm_plan p) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (p->snap_writer.joinable()) p->snap_writer.join();
    const int rc = p->snap_rc;
    p->snap_rc = MM_OK;
    return rc;
}

extern "C" MM_API int mm_save_async(mm_plan p, const char* path, int format, mm_stream stream) {
    if (!p || !path) return set_err(MM_ERR_ARG, "null argument");
    if (format < MM_FMT_OVF2_BIN4 || format > MM_FMT_DUMP) return set_err(MM_ERR_ARG, "unknown format %d", format);
    if (p->nsim > 1 && format != MM_FMT_DUMP)
        return set_err(MM_ERR_ARG, "a batched plan saves dump frames (one per simulation)");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t n3 = (size_t)p->n3() * p->nsim;
    if (!p->snap_host) {
        CUCHK(cudaMallocHost(&p->snap_host, sizeof(float) * n3));
        CUCHK(cudaMallocHost(&p->snap_t_host, sizeof(double)));
        CUCHK(cudaMalloc(&p->snap_t_dev, sizeof(double)));
        CUCHK(cudaStreamCreateWithFlags(&p->snap_stream, cudaStreamNonBlocking));
        CUCHK(cudaEventCreateWithFlags(&p->snap_ready, cudaEventDisableTiming));
        CUCHK(cudaEventCreateWithFlags(&p->snap_copied, cudaEventDisableTiming));
    }
    // one snapshot in flight at a time: the previous writer releases the pinned buffer
    if (p->snap_writer.joinable()) p->snap_writer.join();
    // batched plans keep every accepted state in Y[0] between runs, so simulation 0's
    // control block selects the buffer for all of them
    snapshot_kernel<<<local_blocks((long long)n3), 256, 0, st>>>(cur_of(p->Y), p->ctl, p->Mtmp, (long long)n3,
                                                                  p->snap_t_dev);
    CUCHK(cudaGetLastError());
    CUCHK(cudaEventRecord(p->snap_ready, st));
    CUCHK(cudaStreamWaitEvent(p->snap_stream, p->snap_ready, 0));
    CUCHK(cudaMemcpyAsync(p->snap_host, p->Mtmp, sizeof(float) * n3, cudaMemcpyDeviceToHost, p->snap_stream));
    CUCHK(cudaMemcpyAsync(p->snap_t_host, p->snap_t_dev, sizeof(double), cudaMemcpyDeviceToHost, p->snap_stream));
    CUCHK(cudaEventRecord(p->snap_copied, p->snap_stream));
    // later work on the caller's stream may reuse the staging buffer: it waits for the copy
    CUCHK(cudaStreamWaitEvent(st, p->snap_copied, 0));
    const std::string file(path);
    const int device = p->device;
    p->snap_writer = std::thread([p, file, format, device]() {
        cudaSetDevice(device);
        if (cudaEventSynchronize(p->snap_copied) != cudaSuccess) {
            p->snap_rc = MM_ERR_CUDA;
            return;
        }
        const int n[3] = {p->g.n[0], p->g.n[1], p->g.n[2]};
        for (int b = 0; b < p->nsim && p->snap_rc == MM_OK; b++) {
            const int rc = mm_write_field(file.c_str(), format, p->snap_host + (size_t)b * p->n3(), 3, n,
                                          p->prob.cell, *p->snap_t_host, "m", "");
            if (rc != MM_OK) p->snap_rc = rc;
        }
    });
    return MM_OK;
}

// ---------------------------------------------------------------- continuous batching
// A batched plan as a pool of slots: finished simulations are replaced by new problems
// while the others keep their state, so the GPU never waits for a batch's slowest member.

// Stops the simulations in slots idx (their state and statistics stay as they are; the
// slot counts as done until mm_batch_restart puts a new problem into it).
extern "C" MM_API int mm_batch_cancel(mm_plan p, int count, const int* idx, mm_stream stream) {
    if (!p || count < 0 || (count > 0 && !idx)) return set_err(MM_ERR_ARG, "bad argument");
    for (int k = 0; k < count; k++)
        if (idx[k] < 0 || idx[k] >= p->nsim) return set_err(MM_ERR_ARG, "slot %d out of range", idx[k]);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = canonicalise(p, st);
    if (rc) return rc;
    if ((rc = read_ctl(p, st))) return rc;
    for (int k = 0; k < count; k++) p->ctl_host[idx[k]].done = 1;
    return write_ctl(p, st);
}

extern "C" MM_API int mm_batch_restart(mm_plan p, int count, const int* idx, const float* m, int from_host,
                                       const mm_sim* sims, const double* thr, long long max_steps,
                                       mm_stream stream) {
    if (!p || count < 0 || (count > 0 && (!idx || !m || !thr))) return set_err(MM_ERR_ARG, "bad argument");
    if (p->solver < 0) return set_err(MM_ERR_STATE, "no solver: call mm_solver_init");
    cudaStream_t st = (cudaStream_t)stream;
    for (int k = 0; k < count; k++) {
        if (idx[k] < 0 || idx[k] >= p->nsim) return set_err(MM_ERR_ARG, "slot %d out of range", idx[k]);
        if (!(thr[k] > 0)) return set_err(MM_ERR_ARG, "threshold must be > 0");
    }
    if (sims) {
        int rc = check_sims(sims, count);
        if (rc) return rc;
    }
    int rc = canonicalise(p, st);
    if (rc) return rc;
    if ((rc = read_ctl(p, st))) return rc;
    std::vector<int> was_done(p->nsim);
    for (int b = 0; b < p->nsim; b++) was_done[b] = p->ctl_host[b].done;
    std::vector<char> restarted(p->nsim, 0);
    const size_t n3 = (size_t)p->n3();
    for (int k = 0; k < count; k++) {
        const int b = idx[k];
        restarted[b] = 1;
        if (sims) p->sims[b] = sims[k];
        CUCHK(cudaMemcpyAsync(p->Y[0] + b * n3, m + k * n3, sizeof(float) * n3,
                              from_host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
        normalize_kernel<<<local_blocks(p->g.N), 256, 0, st>>>(
            p->Y[0] + b * n3, p->P.msat_mask ? p->P.msat_mask + b * p->P.mask_bstride : nullptr, p->g.N, 0, 0);
        CUCHK(cudaGetLastError());
        DevCtl& c = p->ctl_host[b];
        const DevCtl keep = c;
        memset(&c, 0, sizeof c);
        c.dt = p->dt0;
        c.mindt = keep.mindt;
        c.maxdt = keep.maxdt;
        c.maxerr = keep.maxerr;
        c.headroom = keep.headroom;
        c.gamma = keep.gamma;
        c.h = c.dt * c.gamma;
        c.dt_thermal = keep.dt_thermal;
        c.t_end = 1e300;
        c.step_end = max_steps > 0 ? max_steps : (1LL << 62);
        c.torque_thr = thr[k];
        c.am_abs_err = keep.am_abs_err;
        c.am_rel_err = keep.am_rel_err;
    }
    if (sims) {
        if ((rc = upload_sims(p))) return rc;
        if (p->nsim == 1) free_graph(p);  // a single plan's scalars live in the captured parameters
    }
    // the FSAL derivative of the new states: the other slots sit out this evaluation
    for (int b = 0; b < p->nsim; b++) p->ctl_host[b].done = restarted[b] ? 0 : 1;
    if ((rc = write_ctl(p, st))) return rc;
    if (p->solver == MM_RK23 || p->solver == MM_RK45) {
        StageOp o = op_blank();
        o.m_in = cur_of(p->Y);
        o.k_out = cur_of(p->K1);
        o.want_tq = 1;
        if ((rc = launch_eval(p, o, p->ctl, 0, nullptr, 0, 0, nullptr, nullptr, st, nullptr))) return rc;
    }
    if ((rc = read_ctl(p, st))) return rc;
    for (int b = 0; b < p->nsim; b++) {
        DevCtl& c = p->ctl_host[b];
        if (!restarted[b]) {
            c.done = was_done[b];
            continue;
        }
        if (p->solver == MM_RK23 || p->solver == MM_RK45) {
            float tqv;
            memcpy(&tqv, &c.tq_bits, sizeof tqv);
            c.maxtorque = sqrt((double)tqv) * c.gamma;
            c.fsal_valid = 1;
            if (c.maxtorque < c.torque_thr) c.done = 1;
        }
        c.tq_bits = 0;
    }
    p->state_set = true;
    return write_ctl(p, st);
}

extern "C" MM_API int mm_batch_drive(mm_plan p, int target_active, long long max_attempts, mm_stream stream) {
    if (!p) return set_err(MM_ERR_ARG, "null plan");
    if (p->solver < 0) return set_err(MM_ERR_STATE, "no solver: call mm_solver_init");
    cudaStream_t st = (cudaStream_t)stream;
    p->run_until = true;
    int rc = read_ctl(p, st);
    if (rc) return rc;
    if (any_active(p)) rc = drive(p, st, max_attempts, target_active);
    int rc2 = canonicalise(p, st);
    int rc3 = read_ctl(p, st);
    return rc ? rc : (rc2 ? rc2 : rc3);
}
