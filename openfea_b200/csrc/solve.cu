// On-device Krylov solvers: the B200 replacement of the direct solves behind
// solution_api / solution_nl_api (src/linear_solution.cpp:17-137, MKL Pardiso /
// SuperLU dgssv).
//
// PCG64 (plain): FP64 conjugate gradients with 3x3 block-Jacobi.  Two fused
// kernels per iteration over the BSELL-32 matrix (sell.cuh):
//   A: p <- z + beta p (neighbour values formed on the fly, the owner writes
//      p), q = K p, per-CTA partial of p.q
//   B: u += alpha p, r -= alpha q, z = Dinv r, partials of r.z and r.r
//
// MIXED: FP64 flexible CG (Polak-Ribiere beta) whose preconditioner is the
// FP32 two-level V(1,1) cycle of precond.cu.  FP64: K for the outer SpMV, the
// residual recursion r -= alpha K p, the update u += alpha p and every outer
// reduction.  FP32 with FP32 accumulation: the smoother's and the residual's
// SpMV, the block-Jacobi smoother, the restriction and the coarse GEMV.
// Kernels per iteration: A, B (+ pre-smoothing), residual, restriction, GEMV,
// prolongation, post-smoothing (+ the r.z dots).
//
// Three ways to run the iterations: in one resident kernel (resident.cu; PCG64
// and MIXED up to some 10^5 rows), launch per phase with the stored K, and
// launch per phase with the outer products formed from the elements
// (matfree.cu; large models of C3D8 elements).
//
// Scalars (alpha, beta, convergence) are formed redundantly and identically
// by every CTA from the previous kernel's partials, in a fixed order: results
// are bitwise reproducible and no host round trip is needed per iteration.
// Iteration counters and flags live in device memory, so a chunk of
// iterations is captured once as a CUDA graph and replayed; the host polls a
// pinned copy of the flags between chunks.  Convergence is confirmed on a
// freshly computed FP64 residual f - K u before a solve returns.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <functional>

#include "matfree.cuh"
#include "precond.cuh"
#include "resident.cuh"
#include "sell.cuh"
#include "solver_common.cuh"

namespace ofea {

// The BSELL SpMV kernels are latency bound (a gather per block): they are
// compiled for full occupancy (8 CTAs of 256 threads per SM, 32 registers),
// measured on the B200 at 79 % of HBM peak for the FP64 outer SpMV against
// 69 % at the 48 registers the compiler picks on its own.
constexpr int kSpmvCtas = 2048 / kBlock;
// The post-smoothing with its K Z part: 64 registers; the grid is two full waves
// then (6 CTAs per SM: 83 us at 1.56M DOF, 5: 88, 4: 79; without the part 62).
constexpr int kPostModesCtas = 4;

// ---------------------------------------------------------- plain SpMV --

__global__ void __launch_bounds__(kBlock, kSpmvCtas) k_spmv64(int nfree, const int *__restrict__ sl_ptr,
                                                   const int *__restrict__ scols,
                                                   const double *__restrict__ sv64,
                                                   const double *__restrict__ x,
                                                   double *__restrict__ y) {
    for_each_sell_row(nfree, sl_ptr, [&](int r, long S, int t, int W) {
        double v[3];
        sell_row<double, 2>(S, t, W, scols, sv64, [&](int k) { return x[k]; }, v[0], v[1], v[2]);
        for (int i = 0; i < 3; ++i) y[3L * r + i] = v[i];
    });
}

static int sell_grid(const ofea_ctx *c) {
    return grid_for(c, (c->nfree + kSlice - 1) / kSlice, kBlock / kSlice);
}

void spmv64(ofea_ctx *c, const double *d_x, double *d_y) {
    k_spmv64<<<sell_grid(c), kBlock, 0, c->stream>>>(c->nfree, c->sl_ptr.p, c->scols.p, c->sv64.p, d_x, d_y);
    OFEA_CHECK_LAUNCH();
}

// ------------------------------------------------------------ PCG FP64 --

// r = f - K u, z = Dinv r; partials r.z -> rz0, r.r -> rr, f.f -> ff.
__global__ void __launch_bounds__(kBlock, kSpmvCtas) k_residual64(
    int nfree, bool zero_u, const int *__restrict__ sl_ptr, const int *__restrict__ scols,
    const double *__restrict__ sv64, const double *__restrict__ Dinv, const double *__restrict__ f,
    const double *__restrict__ u, double *__restrict__ r, double *__restrict__ z, Parts P) {
    __shared__ double sh[kWarpsPerBlock];
    double prz = 0, prr = 0, pff = 0;
    for_each_sell_row(nfree, sl_ptr, [&](int rw, long S, int t, int W) {
        double y[3] = {0.0, 0.0, 0.0}, rv[3], zz[3];
        if (!zero_u) sell_row<double, 2>(S, t, W, scols, sv64, [&](int k) { return u[k]; }, y[0], y[1], y[2]);
        for (int i = 0; i < 3; ++i) {
            const double fi = f[3L * rw + i];
            rv[i] = fi - y[i];
            r[3L * rw + i] = rv[i];
            prr += rv[i] * rv[i];
            pff += fi * fi;
        }
        block3_apply(Dinv + 9L * rw, rv, zz);
        for (int i = 0; i < 3; ++i) {
            z[3L * rw + i] = zz[i];
            prz += rv[i] * zz[i];
        }
    });
    double a = block_sum(prz, sh);
    double b = block_sum(prr, sh);
    double cf = block_sum(pff, sh);
    if (threadIdx.x == 0) {
        P.rz0[blockIdx.x] = a;
        P.rr[blockIdx.x] = b;
        P.ff[blockIdx.x] = cf;
    }
}

// A row's own entries of p_old, z and q.
struct OwnRow {
    double p[3], z[3], q[3];
};

// Iteration kernel A: p = z + beta p_old, q = K p as K z + beta q_old, partial
// p.q.  tol2 = (target ||r||)^2.
template <class Rows>
__global__ void __launch_bounds__(kBlock, Rows::kCtas) k_pcg64_A(
    int nfree, const Rows K, const double *__restrict__ z, double *__restrict__ pA,
    double *__restrict__ pB, double *__restrict__ q, Parts P, Flags *fl, double tol2) {
    __shared__ double sh[kWarpsPerBlock];
    if (cta_done(fl)) return;
    const int k = fl->itA;
    const double *Pcur = (k & 1) ? P.rz1 : P.rz0;   // rz^(k)
    const double *Pprev = (k & 1) ? P.rz0 : P.rz1;  // rz^(k-1)
    const double rr = sum_partials(P.rr, P.G, sh);
    const double rz = sum_partials(Pcur, P.G, sh);
    const double rzp = k > 0 ? sum_partials(Pprev, P.G, sh) : 1.0;
    if (rr <= tol2) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            fl->done = 1;
            fl->iters = k;
        }
        return;
    }
    const double beta = k > 0 ? rz / rzp : 0.0;
    const double *pold = (k & 1) ? pB : pA;
    double *pnew = (k & 1) ? pA : pB;
    double ppq = 0;
    auto own = [&](int rw) { return OwnRow{{pold[3L * rw], pold[3L * rw + 1], pold[3L * rw + 2]},
                                          {z[3L * rw], z[3L * rw + 1], z[3L * rw + 2]},
                                          {q[3L * rw], q[3L * rw + 1], q[3L * rw + 2]}}; };
    K.rows(nfree, [&](int kk) { return z[kk]; }, own, [&](int rw, const double (&y)[3], const OwnRow &o) {
        for (int i = 0; i < 3; ++i) {
            const long d = 3L * rw + i;
            const double pn = fma(beta, o.p[i], o.z[i]);
            const double qn = fma(beta, o.q[i], y[i]);  // K p = K z + beta K p_old
            pnew[d] = pn;
            q[d] = qn;
            ppq += pn * qn;
        }
    });
    const double s = block_sum(ppq, sh);
    if (threadIdx.x == 0) P.pq[blockIdx.x] = s;
    if (blockIdx.x == 0 && threadIdx.x == 0) fl->itB = k;
}

__global__ void __launch_bounds__(kBlock) k_pcg64_B(
    int nfree, const double *__restrict__ Dinv, const double *__restrict__ pA,
    const double *__restrict__ pB, const double *__restrict__ q, double *__restrict__ u,
    double *__restrict__ r, double *__restrict__ z, Parts P, Flags *fl) {
    __shared__ double sh[kWarpsPerBlock];
    if (cta_done(fl)) return;
    const int k = fl->itB;
    const double *Pcur = (k & 1) ? P.rz1 : P.rz0;
    double *Pnext = (k & 1) ? P.rz0 : P.rz1;
    const double pq = sum_partials(P.pq, P.G, sh);
    const double rz = sum_partials(Pcur, P.G, sh);
    if (!(pq > 0.0) || !isfinite(pq)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            fl->done = 1;
            fl->status = OFEA_ERR_BREAKDOWN;
            fl->iters = k;
        }
        return;
    }
    const double alpha = rz / pq;
    const double *p = (k & 1) ? pA : pB;  // written by A(k)
    double prz = 0, prr = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nfree; i += gridDim.x * blockDim.x) {
        double rv[3], zz[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const long d = 3L * i + c;
            u[d] = fma(alpha, p[d], u[d]);
            rv[c] = fma(-alpha, q[d], r[d]);
            r[d] = rv[c];
        }
        block3_apply(Dinv + 9L * i, rv, zz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            z[3L * i + c] = zz[c];
            prz += rv[c] * zz[c];
            prr += rv[c] * rv[c];
        }
    }
    const double a = block_sum(prz, sh);
    const double b = block_sum(prr, sh);
    if (threadIdx.x == 0) {
        Pnext[blockIdx.x] = a;
        P.rr[blockIdx.x] = b;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        fl->itA = k + 1;
        fl->iters = k + 1;
    }
}

// --------------------------------------------------- MIXED: FP64 FCG --

// Outer A: beta (Polak-Ribiere) from the post-smoothing partials,
// p <- double(z_k) + beta p, q = K64 p as K64 z + beta q (the SpMV gathers z
// alone; drift of q from K p is caught by the FP64 true-residual check),
// partial p.q.
template <class Rows>
__global__ void __launch_bounds__(kBlock, Rows::kCtas) k_fcg_A(
    int nfree, const Rows K, const float *__restrict__ zA, const float *__restrict__ zB,
    double *__restrict__ pA, double *__restrict__ pB, double *__restrict__ q, Parts P, Flags *fl,
    double tol2) {
    __shared__ double sh[kWarpsPerBlock];
    if (cta_done(fl)) return;
    const int k = fl->itA;
    const double rr = sum_partials(P.rr, P.G, sh);
    if (rr <= tol2) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            fl->done = 1;
            fl->iters = k;
        }
        return;
    }
    double beta = 0.0;
    if (k > 0) {
        const double rz = sum_partials((k & 1) ? P.rz1 : P.rz0, P.G, sh);   // r_k . z_k
        const double rzp = sum_partials((k & 1) ? P.rz0 : P.rz1, P.G, sh);  // r_{k-1} . z_{k-1}
        const double rzo = sum_partials(P.rzo, P.G, sh);                    // r_k . z_{k-1}
        beta = (rz - rzo) / rzp;
    }
    const float *z = (k & 1) ? zB : zA;
    const double *pold = (k & 1) ? pB : pA;
    double *pnew = (k & 1) ? pA : pB;
    double ppq = 0;
    auto own = [&](int rw) { return OwnRow{{pold[3L * rw], pold[3L * rw + 1], pold[3L * rw + 2]},
                                          {(double)z[3L * rw], (double)z[3L * rw + 1], (double)z[3L * rw + 2]},
                                          {q[3L * rw], q[3L * rw + 1], q[3L * rw + 2]}}; };
    K.rows(nfree, [&](int kk) { return (double)z[kk]; }, own, [&](int rw, const double (&y)[3], const OwnRow &o) {
        for (int i = 0; i < 3; ++i) {
            const long d = 3L * rw + i;
            const double pn = fma(beta, o.p[i], o.z[i]);
            const double qn = fma(beta, o.q[i], y[i]);  // K p = K z + beta K p_old
            pnew[d] = pn;
            q[d] = qn;
            ppq += pn * qn;
        }
    });
    const double s = block_sum(ppq, sh);
    if (threadIdx.x == 0) P.pq[blockIdx.x] = s;
    if (blockIdx.x == 0 && threadIdx.x == 0) fl->itB = k;
}

// Outer B: u += alpha p, r -= alpha q (FP64), ||r||^2, then the start of the
// preconditioner: b32 = float(r), x32 = w Dinv32 b32 (pre-smoothing).
__global__ void __launch_bounds__(kBlock) k_fcg_B(
    int nfree, const float *__restrict__ Dinv32, float w, const double *__restrict__ pA,
    const double *__restrict__ pB, const double *__restrict__ q, double *__restrict__ u,
    double *__restrict__ r, float *__restrict__ b32, float *__restrict__ x32, Parts P, Flags *fl) {
    __shared__ double sh[kWarpsPerBlock];
    if (cta_done(fl)) return;
    const int k = fl->itB;
    const double pq = sum_partials(P.pq, P.G, sh);
    const double rz = sum_partials((k & 1) ? P.rz1 : P.rz0, P.G, sh);
    if (!(pq > 0.0) || !isfinite(pq)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            fl->done = 1;
            fl->status = OFEA_ERR_BREAKDOWN;
            fl->iters = k;
        }
        return;
    }
    const double alpha = rz / pq;
    const double *p = (k & 1) ? pA : pB;
    double prr = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nfree; i += gridDim.x * blockDim.x) {
        float b[3], x[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const long d = 3L * i + c;
            u[d] = fma(alpha, p[d], u[d]);
            const double rv = fma(-alpha, q[d], r[d]);
            r[d] = rv;
            prr += rv * rv;
            b[c] = (float)rv;
        }
        block3_apply(Dinv32 + 9L * i, b, x);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            b32[3L * i + c] = b[c];
            x32[3L * i + c] = w * x[c];
        }
    }
    const double s = block_sum(prr, sh);
    if (threadIdx.x == 0) P.rr[blockIdx.x] = s;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        fl->itA = k + 1;
        fl->iters = k + 1;
    }
}

// Init for MIXED: r = f - K64 u (FP64), ||r||^2, ||f||^2, b32, x32 pre-smoothing.
__global__ void __launch_bounds__(kBlock, kSpmvCtas) k_fcg_init(
    int nfree, bool zero_u, const int *__restrict__ sl_ptr, const int *__restrict__ scols,
    const double *__restrict__ sv64, const float *__restrict__ Dinv32, float w,
    const double *__restrict__ f, const double *__restrict__ u, double *__restrict__ r,
    float *__restrict__ b32, float *__restrict__ x32, Parts P) {
    __shared__ double sh[kWarpsPerBlock];
    double prr = 0, pff = 0;
    for_each_sell_row(nfree, sl_ptr, [&](int rw, long S, int t, int W) {
        double y[3] = {0.0, 0.0, 0.0};
        float b[3], x[3];
        if (!zero_u) sell_row<double, 2>(S, t, W, scols, sv64, [&](int k) { return u[k]; }, y[0], y[1], y[2]);
        for (int i = 0; i < 3; ++i) {
            const double fi = f[3L * rw + i];
            const double rv = fi - y[i];
            r[3L * rw + i] = rv;
            prr += rv * rv;
            pff += fi * fi;
            b[i] = (float)rv;
        }
        block3_apply(Dinv32 + 9L * rw, b, x);
        for (int i = 0; i < 3; ++i) {
            b32[3L * rw + i] = b[i];
            x32[3L * rw + i] = w * x[i];
        }
    });
    const double b = block_sum(prr, sh);
    const double cf = block_sum(pff, sh);
    if (threadIdx.x == 0) {
        P.rr[blockIdx.x] = b;
        P.ff[blockIdx.x] = cf;
    }
}

// Post-smoothing and the end of the preconditioner:
// z_{k+1} = x + w Dinv32 (b32 - K32 x); partials r.z_{k+1} and r.z_k (FP64).
// k = itB (itB = -1 for the initial application).
// MODES: x is x0 still, and the correction Z e and K Z e are added here:
// z_{k+1} = x0 + Z e + w Dinv32 (b32 - K32 x0 - K Z e).
template <bool MODES>
__global__ void __launch_bounds__(kBlock, MODES ? kPostModesCtas : kSpmvCtas) k_fcg_post(
    int nfree, const int *__restrict__ sl_ptr, const int *__restrict__ scols,
    const int *__restrict__ sl_g, const __nv_bfloat16 *__restrict__ svg, const float *__restrict__ Dinv32, float w,
    const float *__restrict__ b32, const float *__restrict__ x32, const double *__restrict__ r,
    float *__restrict__ zA, float *__restrict__ zB, Parts P, Flags *fl, const RowModes md,
    const float *__restrict__ evec) {
    __shared__ double sh[kWarpsPerBlock];
    if (cta_done(fl)) return;
    const int k = fl->itB;
    float *znew = ((k + 1) & 1) ? zB : zA;
    const float *zold = ((k + 1) & 1) ? zA : zB;
    double *Pnext = ((k + 1) & 1) ? P.rz1 : P.rz0;
    double prz = 0, przo = 0;
    for_each_sell_row(nfree, sl_ptr, [&](int rw, long S, int t, int W) {
        float y[3], d[3], o[3], ze[3] = {0.f, 0.f, 0.f}, kz[3] = {0.f, 0.f, 0.f};
        if constexpr (MODES) md.row(rw, evec, kz);
        sell_row_g4(S, sl_g[rw / kSlice], t, W, scols, svg, [&](int kk) { return x32[kk]; }, y[0], y[1], y[2]);
        for (int i = 0; i < 3; ++i) d[i] = MODES ? (b32[3L * rw + i] - y[i]) - kz[i] : b32[3L * rw + i] - y[i];
        block3_apply(Dinv32 + 9L * rw, d, o);
        if constexpr (MODES) md.modes(rw, evec, ze);
        for (int i = 0; i < 3; ++i) {
            const long dd = 3L * rw + i;
            const float zn = fmaf(w, o[i], MODES ? x32[dd] + ze[i] : x32[dd]);
            const double rv = r[dd];
            prz += rv * (double)zn;
            przo += rv * (double)zold[dd];
            znew[dd] = zn;
        }
    });
    const double a = block_sum(prz, sh);
    const double b = block_sum(przo, sh);
    if (threadIdx.x == 0) {
        Pnext[blockIdx.x] = a;
        P.rzo[blockIdx.x] = b;
    }
}

// Single CTA: final reductions of rr and ff into out[0..1]; the partials of rr
// and rz0 become G entries of the same sum.
__global__ void k_final_norms(Parts P, int G, double *out) {
    __shared__ double sh[kWarpsPerBlock];
    const double rr = sum_partials(P.rr, P.G, sh);
    const double ff = sum_partials(P.ff, P.G, sh);
    const double rz = sum_partials(P.rz0, P.G, sh);
    for (int i = threadIdx.x; i < G; i += blockDim.x) {
        P.rr[i] = i ? 0.0 : rr;
        P.rz0[i] = i ? 0.0 : rz;
    }
    if (threadIdx.x == 0) {
        out[0] = rr;
        out[1] = ff;
    }
}

__global__ void k_set_itB(Flags *fl, int v) { fl->itB = v; }

// ------------------------------------------------------------------- host --

void setup_marks_clear(ofea_ctx *c) {
    for (auto &m : c->setup_marks) cudaEventDestroy(m.second);
    c->setup_marks.clear();
}

void setup_mark(ofea_ctx *c, const char *phase) {
    if (!c->setup_trace) return;
    cudaEvent_t e = nullptr;
    OFEA_CUDA(cudaEventCreate(&e));
    c->setup_marks.emplace_back(phase, e);
    OFEA_CUDA(cudaEventRecord(e, c->stream));
}

namespace {

struct Workspace {
    Parts P;
    Flags *fl;
    double *scal;  // device scalars [4]
};

int solver_grid(const ofea_ctx *c) { return std::min(kMaxGrid, c->num_sms * (2048 / kBlock)); }

constexpr size_t kPartials = 6 * (size_t)kMaxGrid + 8;
void reserve(SolverWork &w) {
    w.partials.ensure(kPartials);
    w.flags.ensure(sizeof(Flags) / sizeof(int));
    w.bar.ensure(2);
}

Workspace setup(ofea_ctx *c, int G) {
    SolverWork &w = c->w;
    reserve(w);
    double *b = w.partials.p;
    Workspace ws;
    ws.P.pq = b;
    ws.P.rz0 = b + kMaxGrid;
    ws.P.rz1 = b + 2 * kMaxGrid;
    ws.P.rzo = b + 3 * kMaxGrid;
    ws.P.rr = b + 4 * kMaxGrid;
    ws.P.ff = b + 5 * kMaxGrid;
    ws.scal = b + 6 * kMaxGrid;
    ws.P.G = G;
    ws.fl = reinterpret_cast<Flags *>(w.flags.p);
    OFEA_CUDA(cudaMemsetAsync(w.partials.p, 0, kPartials * sizeof(double), c->stream));
    OFEA_CUDA(cudaMemsetAsync(w.flags.p, 0, sizeof(Flags), c->stream));
    w.hflags.ensure(2 * sizeof(Flags) / sizeof(int));  // two slots: drive() reads one chunk's flags while the next runs
    w.hscal.ensure(4);
    return ws;
}

double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// Replays `chunk(iters)` (as a captured CUDA graph when requested) until the
// device flags say done, max_iter is reached or the time budget runs out.
// Without per-chunk host work the next chunk is enqueued before the flags of
// the one before it are read, so the GPU does not wait for the host's round
// trip; a chunk that starts after the solve stopped returns at once in every
// kernel (the stop flag), and the flags are read again after the last one.
// There the first chunk is launched directly and the graph is captured and
// instantiated while the GPU runs it.
template <class ChunkFn>
void drive(ofea_ctx *c, const ofea_solve_opts &o, Workspace &ws, int per_chunk, ChunkFn chunk,
           Flags &hf, long long &launches, int kernels_per_iter, bool &timed_out, double t_start,
           const std::function<void()> &after_chunk) {
    cudaStream_t s = c->stream;
    cudaGraphExec_t exec = nullptr;
    cudaGraph_t graph = nullptr;
    auto make_graph = [&]() {
        if (!o.use_graph || exec) return;
        OFEA_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        try {
            chunk(per_chunk);
        } catch (...) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(s, &g);
            if (g) cudaGraphDestroy(g);
            throw;
        }
        cudaError_t e = cudaStreamEndCapture(s, &graph);
        if (e != cudaSuccess) fail_cuda(e, "cudaStreamEndCapture", __FILE__, __LINE__);
        e = cudaGraphInstantiate(&exec, graph, 0);
        if (e != cudaSuccess) fail_cuda(e, "cudaGraphInstantiate", __FILE__, __LINE__);
    };
    int launched = 0;
    Flags *h = reinterpret_cast<Flags *>(c->w.hflags.p);  // two slots
    cudaEvent_t ev[2] = {nullptr, nullptr};
    auto launch_chunk = [&]() {
        if (exec)
            OFEA_CUDA(cudaGraphLaunch(exec, s));
        else
            chunk(per_chunk);
        launched += per_chunk;
        launches += (long long)per_chunk * kernels_per_iter;
    };
    auto over_budget = [&]() { return o.time_budget_s > 0 && now_s() - t_start > o.time_budget_s; };
    try {
        if (!after_chunk) {
            for (auto &e : ev) OFEA_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            int k = 0;
            launch_chunk();
            OFEA_CUDA(cudaMemcpyAsync(&h[0], ws.fl, sizeof(Flags), cudaMemcpyDeviceToHost, s));
            OFEA_CUDA(cudaEventRecord(ev[0], s));
            make_graph();
            while (true) {
                const bool more = launched < o.max_iter;
                if (more) {  // slot k ^ 1 was read two chunks ago
                    launch_chunk();
                    OFEA_CUDA(cudaMemcpyAsync(&h[k ^ 1], ws.fl, sizeof(Flags), cudaMemcpyDeviceToHost, s));
                    OFEA_CUDA(cudaEventRecord(ev[k ^ 1], s));
                }
                OFEA_CUDA(cudaEventSynchronize(ev[k]));
                if (h[k].done || !more) break;
                if (over_budget()) {
                    timed_out = true;
                    break;
                }
                k ^= 1;
            }
            OFEA_CUDA(cudaMemcpyAsync(&h[0], ws.fl, sizeof(Flags), cudaMemcpyDeviceToHost, s));
            OFEA_CUDA(cudaStreamSynchronize(s));
        } else {
            make_graph();
            while (true) {
                launch_chunk();
                OFEA_CUDA(cudaMemcpyAsync(h, ws.fl, sizeof(Flags), cudaMemcpyDeviceToHost, s));
                OFEA_CUDA(cudaStreamSynchronize(s));
                if (h->done || launched >= o.max_iter) break;
                after_chunk();
                if (over_budget()) {
                    timed_out = true;
                    break;
                }
            }
        }
    } catch (...) {
        for (auto &e : ev)
            if (e) cudaEventDestroy(e);
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        throw;
    }
    for (auto &e : ev)
        if (e) cudaEventDestroy(e);
    hf = *h;
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
}

// The iterations by the resident solver (resident.cu): it stops by itself, so
// one launch takes up to kResidentChunk iterations; with a time budget or a
// poll interval of the caller's the launches are as long as those.  The iteration limit is rounded up to whole poll intervals.
constexpr int kResidentChunk = 4096;
void drive_resident(ofea_ctx *c, const ofea_solve_opts &o, Workspace &ws, const ResidentPlan &plan, bool mixed, bool modes,
                    int per_chunk, double *d_u, float wsm, double tol2, Flags &hf, long long &launches,
                    bool &timed_out, double t_start) {
    cudaStream_t s = c->stream;
    Flags *h = reinterpret_cast<Flags *>(c->w.hflags.p);
    const bool polled = o.time_budget_s > 0 || o.check_every > 0;
    const long limit = ((long)o.max_iter + per_chunk - 1) / per_chunk * per_chunk;
    for (long done = 0;;) {
        const int iters = (int)std::min<long>(polled ? per_chunk : kResidentChunk, limit - done);
        resident_iterations(c, plan, mixed, modes, ws.P, ws.fl, d_u, wsm, tol2, iters, mixed && done == 0);
        ++launches;
        done += iters;
        OFEA_CUDA(cudaMemcpyAsync(h, ws.fl, sizeof(Flags), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaStreamSynchronize(s));
        if (h->done || done >= limit) break;
        if (o.time_budget_s > 0 && now_s() - t_start > o.time_budget_s) {
            timed_out = true;
            break;
        }
    }
    hf = *h;
}

// Clears the context's V-cycle stop flag when the solve's iterations end
// (normally or by an exception).
struct StopFlagScope {
    ofea_ctx *c;
    ~StopFlagScope() { c->vc_stop = nullptr; }
};

}  // namespace

// Block rows from which the outer products of a linear C3D8 model are formed
// from its elements (matfree.cu).  Below, K stays in L2 and the resident
// solver's PCG64 iteration is the faster one (139k DOF: 18.4 us there, 27.9
// from the elements; 288k: 48 and 37; 706k: 105 and 68; 1.56M: 221 and 130;
// MIXED, launch per phase, stored K and elements: 706k 215 and 170, 1.56M 398
// and 311).  The smoother's products keep the stored BF16 K: formed from the
// elements in FP32 they took as long (44 + 14 us against 61 at 1.56M DOF).
constexpr int kMatfreeRows = 70000;

// Damping of the block-Jacobi smoother: omega = damping / lmax, lmax the power
// iteration's estimate of lambda_max(D^-1 K).  The V(1,1) cycle stays
// positive definite while omega lmax < 2 (with margin for the estimate,
// which lies below lambda_max).
float smoother_weight(const ofea_ctx *c, double damping) { return (float)(damping / c->coarse.lmax); }

void solve_device(ofea_ctx *c, const double *d_f, double *d_u, const ofea_solve_opts &o,
                  ofea_solve_stats &st, const std::function<void(const double *)> &on_chunk) {
    cudaStream_t s = c->stream;
    const int n = c->n, nf = c->nfree;
    if (n == 0) {
        st.status = OFEA_OK;
        return;
    }
    const double t_start = now_s();
    SolverWork &w = c->w;
    cudaEvent_t e0, e1;
    OFEA_CUDA(cudaEventCreate(&e0));
    OFEA_CUDA(cudaEventCreate(&e1));
    OFEA_CUDA(cudaEventRecord(e0, s));
    // default poll interval: a preconditioned iteration is long and its solves
    // short (a poll every 4 iterations wastes fewer iterations after
    // convergence than it costs in host round trips); plain PCG polls every 16
    const bool precond = o.method == OFEA_SOLVER_MIXED || o.method == OFEA_SOLVER_LEARNED;
    int per_chunk = o.check_every > 0 ? o.check_every : (precond ? 4 : 16);
    per_chunk = std::max(1, std::min(per_chunk, o.max_iter));
    long long launches = 0;
    Flags hf{};
    bool timed_out = false;
    double rel = 0;
    int total_iters = 0, restarts = 0;
    w.r.ensure(n);
    w.q.ensure(n);
    w.p0.ensure(n);
    w.p1.ensure(n);
    const bool learned = o.method == OFEA_SOLVER_LEARNED;
    const bool mixed = o.method == OFEA_SOLVER_MIXED || learned;
    float setup_ms = 0.f;
    bool modes = false;  // the restriction takes K Z instead of the residual
    ResidentPlan plan;
    // A solve that hands its residuals to a callback (the learned stage's
    // training samples) keeps the launch-per-phase kernels on the stored K and
    // their order of sums: training amplifies rounding (samples 1e-13 apart on
    // an unsmoothed density field gave weights 3 % apart), so a model trained
    // before is still the one that training gives.
    const bool sampling = (bool)on_chunk;
    // plain PCG prefers the elements to the resident kernel, MIXED the other way
    // round: the elements' tables are built for the solves that use them
    const bool elements = !sampling && nf >= kMatfreeRows && matfree_possible(c);
    auto from_elements = [&] { return elements && matfree_ready(c); };
    bool matfree = false, resident = false;
    if (mixed) {
        const bool had = c->coarse.K_ok;
        cudaEvent_t es;
        OFEA_CUDA(cudaEventCreate(&es));
        setup_marks_clear(c);
        setup_mark(c, "start");
        if (learned) {
            if (!c->learned.have_weights) fail(OFEA_ERR_STATE, "train or load the learned stage first");
            setup_learned_solver(c);
        } else {
            setup_coarse(c, c->coarse_nodes);
        }
        w.b32.ensure(n);
        w.x32.ensure(n);
        w.t32.ensure(n);
        w.z32a.ensure(n);
        w.z32b.ensure(n);
        resident = !sampling && !learned && resident_plan(c, true, elements, plan);
        if (resident) c->coarse.Einv32.ensure((size_t)c->coarse.m * c->coarse.m);
        // every buffer the solve cannot do without is there, before the tables
        // that are optional (K Z, the elements'): where memory ends, those give way
        reserve(w);
        modes = solver_modes(c, learned ? c->coarse2 : c->coarse);
        OFEA_CUDA(cudaEventRecord(es, s));
        OFEA_CUDA(cudaEventSynchronize(es));
        OFEA_CUDA(cudaEventElapsedTime(&setup_ms, e0, es));
        cudaEventDestroy(es);
        if (!had) launches += 4 + 4 * ((c->coarse.m + 31) / 32) + 14;
        if (resident) coarse_dense_inverse(c);  // after the wait: the GPU forms it while the solve is enqueued
        else matfree = from_elements();
    } else {
        w.z.ensure(n);
        reserve(w);
        matfree = from_elements();
        resident = !sampling && !matfree && resident_plan(c, false, elements, plan);
    }
    const int G = resident ? plan.G : solver_grid(c);
    Workspace ws = setup(c, G);
    const float wsm = mixed ? smoother_weight(c, kSmootherDamping) : 0.f;
    for (int attempt = 0; attempt < 8; ++attempt) {
        // the whole GPU forms the residual, whatever the iterations run on; its
        // partials are then folded into the G the iterations read.  Every solve
        // starts from u = 0: the first residual is f, without the product.
        Parts PI = ws.P;
        PI.G = solver_grid(c);
        if (mixed)
            k_fcg_init<<<PI.G, kBlock, 0, s>>>(nf, attempt == 0, c->sl_ptr.p, c->scols.p, c->sv64.p, c->Dinv32.p, wsm, d_f,
                                               d_u, w.r.p, w.b32.p, w.x32.p, PI);
        else
            k_residual64<<<PI.G, kBlock, 0, s>>>(nf, attempt == 0, c->sl_ptr.p, c->scols.p, c->sv64.p, c->Dinv.p, d_f, d_u,
                                                 w.r.p, w.z.p, PI);
        OFEA_CHECK_LAUNCH();
        k_final_norms<<<1, kBlock, 0, s>>>(PI, G, ws.scal);
        OFEA_CUDA(cudaMemcpyAsync(w.hscal.p, ws.scal, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaStreamSynchronize(s));
        launches += 2;
        const double rr = w.hscal.p[0], ff = w.hscal.p[1];
        if (ff == 0.0) {
            OFEA_CUDA(cudaMemsetAsync(d_u, 0, sizeof(double) * n, s));
            rel = 0;
            break;
        }
        rel = std::sqrt(rr / ff);
        if (!std::isfinite(rel)) {
            hf.status = OFEA_ERR_BREAKDOWN;
            break;
        }
        if (rel <= o.rtol || total_iters >= o.max_iter || timed_out) break;
        if (attempt > 0) ++restarts;
        OFEA_CUDA(cudaMemsetAsync(w.p0.p, 0, sizeof(double) * n, s));
        OFEA_CUDA(cudaMemsetAsync(w.p1.p, 0, sizeof(double) * n, s));
        OFEA_CUDA(cudaMemsetAsync(w.q.p, 0, sizeof(double) * n, s));  // q = K p is kept by recurrence
        OFEA_CUDA(cudaMemsetAsync(ws.fl, 0, sizeof(Flags), s));
        if (mixed) {
            OFEA_CUDA(cudaMemsetAsync(w.z32a.p, 0, sizeof(float) * n, s));
            OFEA_CUDA(cudaMemsetAsync(w.z32b.p, 0, sizeof(float) * n, s));
        }
        // recursive residual target a little below rtol; the true residual is re-checked
        const double tol2 = (0.5 * o.rtol) * (0.5 * o.rtol) * ff;
        ofea_solve_opts oo = o;
        oo.max_iter = o.max_iter - total_iters;
        if (resident) {
            drive_resident(c, oo, ws, plan, mixed, modes, per_chunk, d_u, wsm, tol2, hf, launches, timed_out, t_start);
        } else if (mixed) {
            // the V-cycle kernels of this attempt return at once once the
            // solve has stopped (the flag is cleared at every attempt)
            c->vc_stop = &ws.fl->done;
            const StopFlagScope stop_scope{c};
            // initial preconditioner application z_0 = M(r_0)
            k_set_itB<<<1, 1, 0, s>>>(ws.fl, -1);
            auto precondition = [&] {
                if (modes) {
                    Coarse &C = learned ? c->coarse2 : c->coarse;
                    restrict_modes(c, C, w.b32.p, w.x32.p, C.cvec.p);
                    if (learned) learned_coarse_solve(c);
                    else coarse_gemv(c, C.cvec.p, C.evec.p);
                    k_fcg_post<true><<<G, kBlock, 0, s>>>(nf, c->sl_ptr.p, c->scols.p, c->sl_g.p, c->sv16g.p, c->Dinv32.p,
                                                          wsm, w.b32.p, w.x32.p, w.r.p, w.z32a.p, w.z32b.p, ws.P, ws.fl,
                                                          row_modes(C), learned ? C.cvec.p : C.evec.p);
                } else {
                    vc_resid(c, w.b32.p, w.x32.p, w.t32.p);
                    if (learned) learned_coarse_correct(c, w.t32.p, w.x32.p);
                    else coarse_correct(c, w.t32.p, w.x32.p);
                    k_fcg_post<false><<<G, kBlock, 0, s>>>(nf, c->sl_ptr.p, c->scols.p, c->sl_g.p, c->sv16g.p, c->Dinv32.p,
                                                           wsm, w.b32.p, w.x32.p, w.r.p, w.z32a.p, w.z32b.p, ws.P, ws.fl,
                                                           RowModes{}, nullptr);
                }
                OFEA_CHECK_LAUNCH();
            };
            precondition();
            launches += (learned ? 12 : 6) - (modes ? 2 : 0);
            auto chunk = [&](int iters) {
                for (int it = 0; it < iters; ++it) {
                    auto A = [&](auto K) {
                        k_fcg_A<<<G, kBlock, 0, s>>>(nf, K, w.z32a.p, w.z32b.p, w.p0.p, w.p1.p, w.q.p, ws.P, ws.fl, tol2);
                    };
                    if (matfree) {
                        matfree_forces(c, w.z32a.p, w.z32b.p, ws.fl);
                        A(matfree_rows(c));
                    } else {
                        A(sell_rows(c));
                    }
                    k_fcg_B<<<G, kBlock, 0, s>>>(nf, c->Dinv32.p, wsm, w.p0.p, w.p1.p, w.q.p, d_u, w.r.p,
                                                 w.b32.p, w.x32.p, ws.P, ws.fl);
                    precondition();
                }
                OFEA_CHECK_LAUNCH();
            };
            drive(c, oo, ws, per_chunk, chunk, hf, launches, (learned ? 13 : 7) + (matfree ? 1 : 0) - (modes ? 2 : 0), timed_out, t_start, {});
        } else {
            auto chunk = [&](int iters) {
                for (int it = 0; it < iters; ++it) {
                    auto A = [&](auto K) {
                        k_pcg64_A<<<G, kBlock, 0, s>>>(nf, K, w.z.p, w.p0.p, w.p1.p, w.q.p, ws.P, ws.fl, tol2);
                    };
                    if (matfree) {
                        matfree_forces(c, w.z.p, ws.fl);
                        A(matfree_rows(c));
                    } else {
                        A(sell_rows(c));
                    }
                    k_pcg64_B<<<G, kBlock, 0, s>>>(nf, c->Dinv.p, w.p0.p, w.p1.p, w.q.p, d_u, w.r.p, w.z.p,
                                                   ws.P, ws.fl);
                }
                OFEA_CHECK_LAUNCH();
            };
            std::function<void()> after;
            if (on_chunk) after = [&] { on_chunk(w.r.p); };
            drive(c, oo, ws, per_chunk, chunk, hf, launches, matfree ? 3 : 2, timed_out, t_start, after);
        }
        total_iters += hf.iters;
        if (hf.status == OFEA_ERR_BREAKDOWN) break;
        if (hf.status == OFEA_ERR_TIMEOUT) fail(OFEA_ERR_TIMEOUT, "a wait of the resident solver ran out");
    }
    OFEA_CUDA(cudaEventRecord(e1, s));
    OFEA_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    OFEA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    st.iterations = total_iters;
    st.refinements = restarts;
    st.rel_residual = rel;
    st.seconds = ms * 1e-3;
    st.setup_seconds = setup_ms * 1e-3;
    st.kernel_launches = launches;
    if (hf.status == OFEA_ERR_BREAKDOWN)
        st.status = OFEA_ERR_BREAKDOWN;
    else if (!(rel <= o.rtol))
        st.status = timed_out ? OFEA_ERR_TIMEOUT : OFEA_ERR_NOT_CONVERGED;
    else
        st.status = OFEA_OK;
    if (learned && st.status != OFEA_OK) {
        // The learned stage is judged by the FP64 true residual: it missed the
        // target, so plain FP64 PCG restarts from zero and finishes the solve.
        ofea_solve_opts plain = o;
        plain.method = OFEA_SOLVER_PCG64;
        ofea_solve_stats st2{};
        OFEA_CUDA(cudaMemsetAsync(d_u, 0, sizeof(double) * n, s));
        solve_device(c, d_f, d_u, plain, st2, {});
        st2.iterations += st.iterations;
        st2.seconds += st.seconds;
        st2.setup_seconds += st.setup_seconds;
        st2.kernel_launches += st.kernel_launches;
        st2.rejected_learned = 1;
        st = st2;
    }
}

// Times the per-iteration kernels in isolation on the current state (after a
// solve of the same method): ms[0]/bytes[0] = the FP64 SpMV kernel (A),
// ms[1]/bytes[1] = B for PCG64, the FP32 post-smoothing SpMV for MIXED.
void profile_kernels(ofea_ctx *c, int method, int reps, double *ms, double *bytes) {
    cudaStream_t s = c->stream;
    const int n = c->n, nf = c->nfree;
    const int G = solver_grid(c);
    Workspace ws = setup(c, G);
    SolverWork &w = c->w;
    Flags f0{};
    f0.itA = 1;
    f0.itB = 1;
    OFEA_CUDA(cudaMemcpyAsync(ws.fl, &f0, sizeof(Flags), cudaMemcpyHostToDevice, s));
    std::vector<double> ones(5 * kMaxGrid, 1.0);
    OFEA_CUDA(cudaMemcpyAsync(ws.P.pq, ones.data(), sizeof(double) * 5 * kMaxGrid, cudaMemcpyHostToDevice, s));
    const double nnzv = 9.0 * c->sell_len * kSlice;  // stored values incl. padding
    const double nblk = (double)c->sell_len * kSlice;
    cudaEvent_t e0, e1, e2;
    OFEA_CUDA(cudaEventCreate(&e0));
    OFEA_CUDA(cudaEventCreate(&e1));
    OFEA_CUDA(cudaEventCreate(&e2));
    const double tol2 = -1.0;  // never converged: every launch does the full work
    if (method == OFEA_SOLVER_PCG64) {
        if (!w.z.p || w.z.n < (size_t)n) fail(OFEA_ERR_STATE, "run a GPU_PCG solve first");
        double *u = w.t.p;
        OFEA_CUDA(cudaEventRecord(e0, s));
        for (int i = 0; i < reps; ++i)
            k_pcg64_A<<<G, kBlock, 0, s>>>(nf, sell_rows(c), w.z.p, w.p0.p, w.p1.p, w.q.p, ws.P, ws.fl, tol2);
        OFEA_CUDA(cudaEventRecord(e1, s));
        for (int i = 0; i < reps; ++i)
            k_pcg64_B<<<G, kBlock, 0, s>>>(nf, c->Dinv.p, w.p0.p, w.p1.p, w.q.p, u, w.r.p, w.z.p, ws.P, ws.fl);
        OFEA_CUDA(cudaEventRecord(e2, s));
        // K values + columns + slice pointers, z, p_old and q_old read, p_new and q written
        bytes[0] = 8 * nnzv + 4 * nblk + 4.0 * ((nf + 31) / 32 + 1) + 8.0 * n * 5;
        bytes[1] = 72.0 * nf + 8.0 * n * 7;  // Dinv; u r/w, r r/w, p, q, z
    } else {
        if (!w.z32a.p || w.z32a.n < (size_t)n) fail(OFEA_ERR_STATE, "run a GPU_MIXED solve first");
        const float wsm = smoother_weight(c, kSmootherDamping);
        OFEA_CUDA(cudaEventRecord(e0, s));
        for (int i = 0; i < reps; ++i)
            k_fcg_A<<<G, kBlock, 0, s>>>(nf, sell_rows(c), w.z32a.p, w.z32b.p, w.p0.p, w.p1.p, w.q.p, ws.P, ws.fl, tol2);
        OFEA_CUDA(cudaEventRecord(e1, s));
        for (int i = 0; i < reps; ++i)
            k_fcg_post<false><<<G, kBlock, 0, s>>>(nf, c->sl_ptr.p, c->scols.p, c->sl_g.p, c->sv16g.p, c->Dinv32.p, wsm,
                                                   w.b32.p, w.x32.p, w.r.p, w.z32a.p, w.z32b.p, ws.P, ws.fl, RowModes{},
                                                   nullptr);
        OFEA_CUDA(cudaEventRecord(e2, s));
        // FP64 K + columns + slice pointers, z (FP32), p_old and q_old read, p_new and q written
        bytes[0] = 8 * nnzv + 4 * nblk + 4.0 * ((nf + 31) / 32 + 1) + 4.0 * n + 8.0 * n * 4;
        // BF16 K + columns, x32 and b32 read, Dinv32, r (FP64) and z_old read, z_new written
        bytes[1] = 2 * nnzv + 4 * nblk + 4.0 * n * 2 + 36.0 * nf + 8.0 * n + 4.0 * n * 2;
    }
    OFEA_CHECK_LAUNCH();
    OFEA_CUDA(cudaEventSynchronize(e2));
    float a = 0, b = 0;
    OFEA_CUDA(cudaEventElapsedTime(&a, e0, e1));
    OFEA_CUDA(cudaEventElapsedTime(&b, e1, e2));
    ms[0] = a / reps;
    ms[1] = b / reps;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaEventDestroy(e2);
}

// The kernels that one iteration of a solve launches on the context's K, in
// order (none where the resident kernel runs them all), each timed by itself.
// bytes: what it has to read and write, each array once (0: not counted);
// flops: FP64 operations of the element forces.
std::vector<KernelTime> profile_iteration(ofea_ctx *c, int method, int reps) {
    cudaStream_t s = c->stream;
    const int n = c->n, nf = c->nfree;
    SolverWork &w = c->w;
    const bool learned = method == OFEA_SOLVER_LEARNED, mixed = method == OFEA_SOLVER_MIXED || learned;
    Coarse &C = learned ? c->coarse2 : c->coarse;
    if (mixed ? !c->coarse.K_ok || !C.K_ok || !w.z32a.p || w.z32a.n < (size_t)n : !w.z.p || w.z.n < (size_t)n)
        fail(OFEA_ERR_STATE, "run a solve with this method first");
    const int G = solver_grid(c);
    Workspace ws = setup(c, G);
    ResidentPlan plan;
    const bool elements = nf >= kMatfreeRows && matfree_possible(c);
    bool matfree = !mixed && elements && matfree_ready(c);
    if (!learned && !matfree && resident_plan(c, mixed, elements, plan)) return {};
    const bool modes = mixed && solver_modes(c, C);
    if (mixed) matfree = elements && matfree_ready(c);
    const double nnzv = 9.0 * c->sell_len * kSlice, nblk = (double)c->sell_len * kSlice;  // incl. padding
    const double zb = mixed ? 4.0 : 8.0, vec = 8.0 * n, slices = 4.0 * ((nf + 31) / 32 + 1);
    const float wsm = mixed ? smoother_weight(c, kSmootherDamping) : 0.f;
    double *u = w.t.p;

    struct Step {
        const char *name;
        double bytes, flops;
        std::function<void()> launch;
    };
    std::vector<Step> steps;
    double listed = 0;  // element forces a row reads
    if (matfree) {
        std::vector<int> list((size_t)c->mf_width * nf);
        std::vector<unsigned char> link(c->ne8);
        OFEA_CUDA(cudaMemcpyAsync(list.data(), c->mf_list.p, sizeof(int) * list.size(), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaMemcpyAsync(link.data(), c->mf_link.p, link.size(), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaStreamSynchronize(s));
        for (int p : list) listed += p >= 0;
        double written = 4.0 * c->ne8;
        for (unsigned char l : link) written += l ? 0 : 4;
        // nodes and rows of the elements, moduli, links, coordinates, z; forces
        steps.push_back({"k_hex_forces", 73.0 * c->ne8 + 24.0 * c->nd + zb * n + 24.0 * written, kHexForceOps * c->ne8, [=, &w] {
                             if (mixed) matfree_forces(c, w.z32a.p, w.z32b.p, ws.fl);
                             else matfree_forces(c, w.z.p, ws.fl);
                         }});
    }
    auto A = [=, &w](auto K) {
        if (mixed) k_fcg_A<<<G, kBlock, 0, s>>>(nf, K, w.z32a.p, w.z32b.p, w.p0.p, w.p1.p, w.q.p, ws.P, ws.fl, -1.0);
        else k_pcg64_A<<<G, kBlock, 0, s>>>(nf, K, w.z.p, w.p0.p, w.p1.p, w.q.p, ws.P, ws.fl, -1.0);
    };
    // K (or the list and the forces), z, p and q read, p and q written
    const double kb = matfree ? 4.0 * c->mf_width * nf + 24.0 * listed : 8 * nnzv + 4 * nblk + slices;
    steps.push_back({mixed ? "k_fcg_A" : "k_pcg64_A", kb + zb * n + 4 * vec, 0.0, [=] {
                         if (matfree) A(matfree_rows(c));
                         else A(sell_rows(c));
                     }});
    if (!mixed) {
        steps.push_back({"k_pcg64_B", 72.0 * nf + 7 * vec, 0.0, [=, &w] {
                             k_pcg64_B<<<G, kBlock, 0, s>>>(nf, c->Dinv.p, w.p0.p, w.p1.p, w.q.p, u, w.r.p, w.z.p, ws.P, ws.fl);
                         }});
    } else {
        steps.push_back({"k_fcg_B", 36.0 * nf + 6 * vec + 8.0 * n, 0.0, [=, &w] {
                             k_fcg_B<<<G, kBlock, 0, s>>>(nf, c->Dinv32.p, wsm, w.p0.p, w.p1.p, w.q.p, u, w.r.p, w.b32.p, w.x32.p,
                                                          ws.P, ws.fl);
                         }});
        const double k16 = 2 * nnzv + 4 * nblk + 2 * slices, entries = modes ? 76.0 * C.md_n : 0.0;
        const float *evec = learned ? C.cvec.p : C.evec.p;
        if (modes) {
            steps.push_back({"k_restrict_modes", 16.0 * nf + 8.0 * n + entries, 0.0,
                             [=, &w, &C] { restrict_modes(c, C, w.b32.p, w.x32.p, C.cvec.p); }});
        } else {
            steps.push_back({"k_vc_resid", k16 + 12.0 * n, 0.0, [=, &w] { vc_resid(c, w.b32.p, w.x32.p, w.t32.p); }});
            steps.push_back({"k_restrict", 16.0 * nf + 4.0 * n, 0.0, [=, &w, &C] { restrict_level(c, C, w.t32.p, C.cvec.p); }});
        }
        steps.push_back({learned ? "learned coarse solve" : "coarse solve", 0.0, 0.0, [=, &C] {
                             if (learned) learned_coarse_solve(c);
                             else coarse_gemv(c, C.cvec.p, C.evec.p);
                         }});
        if (!modes)
            steps.push_back({"k_prolong", 16.0 * nf + 8.0 * n, 0.0, [=, &w, &C] { prolong_level(c, C, evec, w.x32.p); }});
        // BF16 K, b, x, Dinv32, r and z_old read, z written; with K Z its entries by row and the rows' offsets
        steps.push_back({"k_fcg_post", k16 + 8.0 * n + 36.0 * nf + vec + 8.0 * n + (modes ? entries + 20.0 * nf : 0.0), 0.0, [=, &w, &C] {
                             if (modes)
                                 k_fcg_post<true><<<G, kBlock, 0, s>>>(nf, c->sl_ptr.p, c->scols.p, c->sl_g.p, c->sv16g.p,
                                                                       c->Dinv32.p, wsm, w.b32.p, w.x32.p, w.r.p, w.z32a.p,
                                                                       w.z32b.p, ws.P, ws.fl, row_modes(C), evec);
                             else
                                 k_fcg_post<false><<<G, kBlock, 0, s>>>(nf, c->sl_ptr.p, c->scols.p, c->sl_g.p, c->sv16g.p,
                                                                        c->Dinv32.p, wsm, w.b32.p, w.x32.p, w.r.p, w.z32a.p,
                                                                        w.z32b.p, ws.P, ws.fl, RowModes{}, nullptr);
                         }});
    }
    Flags f0{};
    f0.itA = f0.itB = 1;
    const std::vector<double> ones(6 * kMaxGrid, 1.0);
    cudaEvent_t e[2];
    for (auto &x : e) OFEA_CUDA(cudaEventCreate(&x));
    std::vector<KernelTime> out;
    for (const Step &k : steps) {
        Flags f{};
        OFEA_CUDA(cudaMemcpyAsync(ws.fl, &f0, sizeof(Flags), cudaMemcpyHostToDevice, s));
        OFEA_CUDA(cudaMemcpyAsync(ws.P.pq, ones.data(), sizeof(double) * ones.size(), cudaMemcpyHostToDevice, s));
        k.launch();
        OFEA_CUDA(cudaEventRecord(e[0], s));
        for (int i = 0; i < reps; ++i) k.launch();
        OFEA_CUDA(cudaEventRecord(e[1], s));
        OFEA_CHECK_LAUNCH();
        OFEA_CUDA(cudaMemcpyAsync(&f, ws.fl, sizeof(Flags), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaStreamSynchronize(s));
        if (f.done) fail(OFEA_ERR_STATE, std::string(k.name) + " stopped while it was timed");
        float t = 0;
        OFEA_CUDA(cudaEventElapsedTime(&t, e[0], e[1]));
        out.push_back({k.name, t / reps, k.bytes, k.flops});
    }
    for (auto &x : e) cudaEventDestroy(x);
    return out;
}

}  // namespace ofea
