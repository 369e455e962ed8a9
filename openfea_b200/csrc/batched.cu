// Batched reanalysis: many design variants (each an assembled context on one
// GPU) times up to kMaxBatchRhs load cases each, solved by ONE persistent
// cooperative kernel launched from a CUDA graph.  The reference solves such
// batches variant by variant with a kept SuperLU factor and dgstrs per load
// case (src/solver/solver_superlu.cpp:31-94, the CA reanalysis of
// src/ca_analysis.cpp:148-248).
//
// Layout in HBM: the variants' DOF are concatenated (variant v starts at
// dof0[v]) and every vector is load-case interleaved, x[(dof0 + d) * NP + j]
// (NP = the NR load cases padded to a power of two >= 4): the load cases of
// one DOF are one contiguous run.  Matrices stay where their contexts keep
// them (BSELL-32, FP64 and BF16 copies); a table of per-variant
// descriptors points at them, one of records at their slices.
//
// Algorithm per (variant, load case): the MIXED method of solve.cu, FP64
// flexible CG with the FP32 two-level V(1,1) preconditioner of precond.cu (with
// K Z where every variant has it, with few entries per row: one product
// instead of two, 8 to 46 % less time at 1 to 32 variants of 7k and 27k nodes
// and 3 to 16 load cases; the phases of a trace stay, the residual's is then a
// barrier alone), or
// PCG64 (FP64 CG, block Jacobi).  The kernel runs every variant in lock step
// through phases separated by grid barriers.  In the matrix phases a CTA owns
// one slice (32 block rows) of some variant at a time: bulk copies bring the
// operand's entries of the slice's distinct columns and stream its slots
// through shared memory (matrix_phase), and its threads take (block row, load
// cases) pairs, so each matrix value is read from HBM once for all load cases
// and each column's entries once per slice.  The restriction takes one
// aggregate per CTA; other phases take (coarse row) or (variant, load case)
// items per warp.
// The outer SpMM multiplies the preconditioned residual z, not p: q = K z +
// beta q_old equals K p (p = z + beta p_old), and gathering z (FP32 for
// MIXED) instead of p_old and z cuts the gathered bytes by 3x (MIXED) or 2x
// (PCG64).  Any drift of q from K p is caught by the true FP64 residual that
// the host checks after the kernel.
// Per-(variant, load case) scalars come from per-slice partial sums reduced
// in a fixed order: results are bitwise reproducible.  Converged load cases
// stop updating; the kernel ends when none is left or at max_iter.
//
// Every wait, at a grid barrier and for a copy into shared memory, is bounded
// (time limit on %globaltimer): on expiry the kernel records an error, reads
// nothing that may not have arrived, and every CTA returns.
#include <cuda/atomic>
#include <sys/stat.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <type_traits>
#include <memory>
#include <mutex>
#include <sstream>
#include <string>
#include <type_traits>
#include <vector>

#include "precond.cuh"
#include "sell.cuh"
#include "solver_common.cuh"

namespace ofea {

constexpr int kMaxBatchRhs = 32;

// Per-variant descriptor (device copy).
struct BVar {
    int nfree, nslice, slice0, na, m, agg0, crow0, n;
    long dof0;  // first DOF of the variant in the batch (its vectors start at dof0 * NR)
    long c0;    // first coarse entry of the variant (times NR)
    const int *sl_ptr, *scols, *sl_g, *su_n;
    const int2 *su_runs;
    const uint16_t *su_idx;
    const double *sv64, *Dinv;
    const __nv_bfloat16 *sv16g;
    const float *Dinv32;
    const int *agg_ptr;
    const float4 *agg_off, *row_off;  // offsets from the centroids (precond.cu)
    const float *Einv32;
    const int *md_ptr, *md_row;  // K Z by aggregate and by row (precond.cu)
    const float *md_val;
    RowModes md;
    float wsm, pad2;
};

// One slice of the batch (device table, in batch order): where its slots
// start, its distinct columns as runs of consecutive ones (first column;
// position << 16 | length) and every slot's position among them (lidx; nu = 0:
// read the columns directly), and what the phases need of its rows.
struct __align__(16) BSlice {
    const double *v64;
    const __nv_bfloat16 *vg;  // grouped BF16 values (sell.cuh)
    const int *cols;
    const int2 *runs;
    const uint16_t *lidx;
    const double *Dinv;
    const float *Dinv32;
    long dof;  // the variant's first DOF in the batch
    int W, nu, nrun, row0, nfree, v;
    float wsm;
    int pad;
};

struct BArgs {
    int V, NR, nslices, naggs, ncrows, max_iter, extra_arrivals;
    int copy_arrivals;  // arrivals a slot copy's barrier waits for (1; more: it never completes)
    unsigned long long limit_ns;
    double rtol;
    const BVar *var;
    const BSlice *slice;
    unsigned *vmask;  // [V]: bit j set while load case j runs
    int modes, parts; // the V-cycle takes K Z (every variant has it); parts per aggregate of its restriction
    int ncoarse;      // values of cvec per load case
    float *cpart;     // cvec's parts
    int cap;          // columns the staged products' buffer holds
    const int *slice_var, *agg_var, *crow_var;
    const double *f;
    double *u, *r, *p0, *p1, *q, *z64;
    float *b32, *x32, *t32, *zA, *zB, *cvec, *evec;
    double *pa, *pb;                                    // partials [slice][NR]
    double *ff, *tol2, *rz, *alpha, *beta;              // [V * NR]
    int *live, *iters, *status, *live_cnt;              // [V * NR], live_cnt[3]
    GridBar *gs;
    unsigned long long *trace;  // NULL, or %globaltimer at the start and after each grid barrier (CTA 0)
    int trace_cap;
};

namespace {

// Entry (node i, component c, load case j) of a variant in a batch vector
// whose load-case stride is NP (NR rounded up; padding entries stay zero).
template <int NP>
__device__ __forceinline__ long vidx(const BVar &B, long i, int c, int j) {
    return (B.dof0 + 3 * i + c) * NP + j;
}

// RL consecutive load cases of one DOF as one vector access (the offset is
// a multiple of RL: aligned).
template <class V, int RL>
__device__ __forceinline__ void ldv(const V *p, V (&o)[RL]) {
    if constexpr (sizeof(V) * RL == 32) {
        using T = typename std::conditional<sizeof(V) == 8, double2, float4>::type;
        const T a = reinterpret_cast<const T *>(p)[0], b = reinterpret_cast<const T *>(p)[1];
        std::memcpy(&o[0], &a, 16);
        std::memcpy(&o[RL / 2], &b, 16);
    } else if constexpr (sizeof(V) * RL == 16) {
        using T = typename std::conditional<sizeof(V) == 8, double2, float4>::type;
        const T a = *reinterpret_cast<const T *>(p);
        std::memcpy(&o[0], &a, 16);
    } else if constexpr (sizeof(V) * RL == 8 && sizeof(V) == 4) {
        const float2 a = *reinterpret_cast<const float2 *>(p);
        o[0] = a.x;
        o[1] = a.y;
    } else {
#pragma unroll
        for (int q = 0; q < RL; ++q) o[q] = p[q];
    }
}
template <class V, int RL>
__device__ __forceinline__ void stv(V *p, const V (&o)[RL]) {
    if constexpr (sizeof(V) * RL == 32) {
        using T = typename std::conditional<sizeof(V) == 8, double2, float4>::type;
        T a, b;
        std::memcpy(&a, &o[0], 16);
        std::memcpy(&b, &o[RL / 2], 16);
        reinterpret_cast<T *>(p)[0] = a;
        reinterpret_cast<T *>(p)[1] = b;
    } else if constexpr (sizeof(V) * RL == 16) {
        using T = typename std::conditional<sizeof(V) == 8, double2, float4>::type;
        T a;
        std::memcpy(&a, &o[0], 16);
        *reinterpret_cast<T *>(p) = a;
    } else if constexpr (sizeof(V) * RL == 8 && sizeof(V) == 4) {
        *reinterpret_cast<float2 *>(p) = make_float2(o[0], o[1]);
    } else {
#pragma unroll
        for (int q = 0; q < RL; ++q) p[q] = o[q];
    }
}

// Thread roles in the CTA that owns one slice: LW = NP / RL lanes per block
// row, each carrying RL consecutive load cases; 32 / LW rows per warp.
template <int NP, int RL>
struct Lanes {
    static constexpr int kLW = NP / RL;
    static constexpr int kRowsPerWarp = 32 / kLW;
    static constexpr int kWarps = kSlice / kRowsPerWarp;
    __device__ static int row() { return (threadIdx.x >> 5) * kRowsPerWarp + (threadIdx.x & 31) / kLW; }
    __device__ static int j0() { return (threadIdx.x & (kLW - 1)) * RL; }
};

// Shared memory of a matrix phase: three buffers of the slice's slots (kKC64
// FP64 slots or kKC16 BF16 ones, then their column positions) and the records
// of this slice and the next ones; partial sums and the distinct columns'
// entries of the operand follow (dynamic).  Filled by bulk copies that complete on the
// mbarriers (bx: the operand, bv: the slot buffers).
constexpr int kKC64 = 4, kKC16 = 16, kStages = 3;
struct __align__(128) Stage {
    unsigned char v[kStages][kKC64 * 9 * kSlice * 8];
    int col[kStages][kKC16 * kSlice];
    BSlice rec[3];
    unsigned long long bx, bv[kStages];
};
static_assert(sizeof(Stage::v) >= 6 * 32 * 32 * sizeof(float), "the restriction's per-warp sums fit in the stage");
static_assert(kKC16 / 4 * 9 * kSlice * 8 <= sizeof(Stage::v[0]), "a BF16 chunk fits a buffer");

// Partial sums of a slice: [sum][warp][load case].
__host__ __device__ constexpr int red_bytes(int np, int rl) { return 2 * (np / rl) * np * 8; }

// The mbarriers' phase parities (the same in every thread): bits 0 .. kStages
// - 1 the slot buffers', kOperand the operand's.  kLost: a wait of this thread
// has run out.
struct Pipe {
    static constexpr unsigned kOperand = kStages, kLost = 1u << 8;
    unsigned par = 0;
    __device__ __forceinline__ bool lost() const { return par & kLost; }
};
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void stage_init(Stage &st, int arrivals, int *s_fail) {
    if (threadIdx.x == 0) {
        *s_fail = 0;
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(&st.bx)) : "memory");
        for (int i = 0; i < kStages; ++i)
            asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_addr(&st.bv[i])), "r"(arrivals) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}
// Waits for the phase of parity `par`; gives up after limit_ns and returns
// false (the caller reads nothing of that copy).
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned par, unsigned long long limit_ns) {
    unsigned long long t0 = 0;
    for (;;) {
        unsigned ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(smem_addr(b)), "r"(par)
                     : "memory");
        if (ok) return true;
        const unsigned long long t = global_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > limit_ns) return false;
    }
}

// Bulk prefetch of [p, p + bytes) from HBM into L2 (no data returned, no
// completion to wait for).  p and bytes are multiples of 16 (the BSELL slot
// blocks and the slices' vector runs are); issued in pieces of at most 32 KB.
__device__ __forceinline__ void l2_prefetch(const void *p, long bytes) {
    const size_t g = __cvta_generic_to_global(p);
    for (long o = 0; o < bytes; o += 32768) {
        const unsigned nb = (unsigned)min(32768L, bytes - o);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g + o), "r"(nb) : "memory");
    }
}

// acc[q] += m * x[q] for RL load cases; pairs in one packed FP32 FMA.
template <int RL>
__device__ __forceinline__ void fma_cases(float (&acc)[RL], float m, const float (&x)[RL]) {
    if constexpr (RL % 2 == 0) {
        unsigned long long mm;
        asm("mov.b64 %0, {%1, %1};" : "=l"(mm) : "f"(m));
#pragma unroll
        for (int q = 0; q < RL; q += 2) {
            unsigned long long av, xv;
            asm("mov.b64 %0, {%1, %2};" : "=l"(av) : "f"(acc[q]), "f"(acc[q + 1]));
            asm("mov.b64 %0, {%1, %2};" : "=l"(xv) : "f"(x[q]), "f"(x[q + 1]));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(av) : "l"(mm), "l"(xv));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[q]), "=f"(acc[q + 1]) : "l"(av));
        }
    } else {
#pragma unroll
        for (int q = 0; q < RL; ++q) acc[q] = fmaf(m, x[q], acc[q]);
    }
}
template <int RL, class X>
__device__ __forceinline__ void fma_cases(double (&acc)[RL], double m, const X (&x)[RL]) {
#pragma unroll
    for (int q = 0; q < RL; ++q) acc[q] = fma(m, (double)x[q], acc[q]);
}

// y[c][q] = (K x)_(row, c) for this thread's RL load cases, for every slice of
// this CTA in turn, then fin(slice record, slice index, live mask, y).
//
// A slice's 32 rows name each of their columns about four times (200 to 400
// distinct columns against 864 slots on a structured C3D8 block), so the
// distinct columns' entries (3 NP values each; consecutive columns are one
// contiguous run) are copied to shared memory once and gathered from there:
// gathered through L2 the products were bound by latency, about 600 cycles
// per slot and warp.  Values stream through three buffers shared by every
// load case (FP64 planes, or the grouped BF16 copy, whose 8-byte words bring
// four slots of a plane at once).  All copies are bulk copies issued by warp 0
// (16-byte cp.async of every thread took 4,700 cycles a slice to issue), and
// the next slice's start as soon as this slice's product is formed, under
// fin; pf(next record) prefetches what fin will read then.  A slice without a
// column list, or with one beyond the buffer (cap), gathers its columns
// directly.  Slices whose load cases have all stopped are skipped.
// A thread whose wait for a copy runs out reads nothing more of the stage;
// the whole CTA then leaves the phase at the end of that slice, without fin,
// and the kernel at the next grid barrier (s_fail, and the batch's error).
// (An iteration takes 0 to 1.3 % longer for it, 2.3 % at 32 load cases, MIXED.)
// Measured on 16 variants of 17.6k nodes on average x 16 load cases (ms per
// phase and iteration, before -> after): FP64 product 0.359 -> 0.304,
// residual 0.254 -> 0.170, post-smoothing 0.309 -> 0.210; iteration 1.207 ->
// 0.940.  What bounds them now: the FP64 product's shared-memory reads (values
// nine per slot and warp) with two CTAs per SM to cover the rest of a slice.
//   T: arithmetic type, X: operand type, BF: values from the BF16 copy.
template <class T, class X, bool BF, int NP, int RL, class Pf, class Fin>
__device__ __forceinline__ void matrix_phase(const BArgs &a, Stage &st, Pipe &pipe, unsigned char *dyn, int cap, int *s_fail,
                                             const X *x, bool all, Pf pf, Fin fin) {
    constexpr int KC = BF ? kKC16 : kKC64;
    constexpr int kColBytes = 3 * NP * (int)sizeof(X);
    constexpr int kPieces = (int)sizeof(BSlice) / 16;
    const int r = Lanes<NP, RL>::row(), j0 = Lanes<NP, RL>::j0();
    const int lane = threadIdx.x & 31;
    const bool warp0 = threadIdx.x < 32;
    X *xs = reinterpret_cast<X *>(dyn + red_bytes(NP, RL));
    int gsl = blockIdx.x;
    if (gsl >= a.nslices) return;
    auto wait = [&](unsigned long long *bar, unsigned bit) {  // the next phase of a barrier
        if (mbar_wait(bar, (pipe.par >> bit) & 1u, a.limit_ns)) pipe.par ^= 1u << bit;
        else pipe.par |= Pipe::kLost;
    };
    auto is_staged = [&](const BSlice &R) { return R.nu > 0 && R.nu <= cap; };
    // values and column positions of chunk ch (one thread)
    auto issue_chunk = [&](const BSlice &R, int ch) {
        const int k0 = ch * KC, kc = min(KC, R.W - k0), b = ch % kStages;
        const unsigned nv = (BF ? (kc + 3) / 4 : kc) * (9 * kSlice * 8);
        const bool sg = is_staged(R);
        const unsigned nc = kc * kSlice * (sg ? 2 : 4);
        mbar_expect(&st.bv[b], nv + nc);
        if (BF) bulk_copy(st.v[b], R.vg + (long)k0 * 9 * kSlice, nv, &st.bv[b]);
        else bulk_copy(st.v[b], R.v64 + (long)k0 * 9 * kSlice, nv, &st.bv[b]);
        if (sg) bulk_copy(st.col[b], R.lidx + k0 * kSlice, nc, &st.bv[b]);
        else bulk_copy(st.col[b], R.cols + k0 * kSlice, nc, &st.bv[b]);
    };
    // the start of a slice (warp 0): its first chunks and its columns' entries;
    // r0, r1: the slice's runs lane and lane + 32
    auto issue = [&](const BSlice &R, int2 r0, int2 r1) {
        if (lane == 0) {
            if (is_staged(R)) mbar_expect(&st.bx, R.nu * kColBytes);
            for (int ch = 0; ch < kStages && ch * KC < R.W; ++ch) issue_chunk(R, ch);
        }
        __syncwarp();
        if (is_staged(R)) {
            const X *xv = x + R.dof * NP;
            for (int i = lane; i < R.nrun; i += 32) {
                const int2 q = i < 32 ? r0 : i < 64 ? r1 : R.runs[i];
                bulk_copy(reinterpret_cast<char *>(xs) + (q.y >> 16) * kColBytes, xv + 3L * q.x * NP, (q.y & 0xffff) * kColBytes,
                          &st.bx);
            }
        }
    };
    auto load_runs = [&](const BSlice &R, int2 &r0, int2 &r1) {
        r0 = r1 = make_int2(0, 0);
        if (is_staged(R)) {
            if (lane < R.nrun) r0 = R.runs[lane];
            if (lane + 32 < R.nrun) r1 = R.runs[lane + 32];
        }
    };
    __syncthreads();  // the phase before is done with the stage
    int2 r0 = make_int2(0, 0), r1 = r0;
    if (warp0) {
        // the bulk copies read what earlier phases stored, and write where they wrote
        asm volatile("fence.proxy.async;" ::: "memory");
        if (lane < kPieces) reinterpret_cast<int4 *>(&st.rec[0])[lane] = reinterpret_cast<const int4 *>(a.slice + gsl)[lane];
        __syncwarp();
        load_runs(st.rec[0], r0, r1);
    }
    __syncthreads();
    unsigned mask = all ? 0xffffffffu : a.vmask[st.rec[0].v], mask_next = 0;
    if (warp0 && mask) issue(st.rec[0], r0, r1);
    for (int cur = 0; gsl < a.nslices; gsl += gridDim.x, cur = cur == 2 ? 0 : cur + 1, mask = mask_next) {
        const BSlice &R = st.rec[cur], &Rn = st.rec[cur == 2 ? 0 : cur + 1];
        const bool more = gsl + (int)gridDim.x < a.nslices;
        int4 piece = make_int4(0, 0, 0, 0);
        if (more && threadIdx.x < kPieces) piece = reinterpret_cast<const int4 *>(a.slice + gsl + gridDim.x)[threadIdx.x];
        const int W = R.W, nch = mask ? (W + KC - 1) / KC : 0;
        const bool staged = is_staged(R);
        const X *xv = x + R.dof * NP;
        T y[3][RL];
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < RL; ++q) y[c][q] = 0;
        if (mask && staged) wait(&st.bx, Pipe::kOperand);
        if (more && warp0) {  // the next slice's record and runs
            if (lane < kPieces) reinterpret_cast<int4 *>(const_cast<BSlice *>(&Rn))[lane] = piece;
            __syncwarp();
            load_runs(Rn, r0, r1);
        }
        for (int ch = 0; ch < nch; ++ch) {
            const int b = ch % kStages;
            if (!pipe.lost()) wait(&st.bv[b], b);
            const int kc = pipe.lost() ? 0 : min(KC, W - ch * KC);
            const double *v64 = reinterpret_cast<const double *>(st.v[b]) + r;
            const uint2 *v16 = reinterpret_cast<const uint2 *>(st.v[b]) + r;
            auto run = [&](auto staged_t) {
                constexpr bool ST = decltype(staged_t)::value;
                auto operand = [&](int k, X (&o)[3][RL]) {
                    const X *p;
                    if constexpr (ST) p = xs + (reinterpret_cast<const uint16_t *>(st.col[b])[k * kSlice + r] * 3) * NP + j0;
                    else p = xv + 3L * st.col[b][k * kSlice + r] * NP + j0;
#pragma unroll
                    for (int c = 0; c < 3; ++c) ldv<X, RL>(p + c * NP, o[c]);
                };
                // four slots from k on (full: without per-slot guards, so their
                // loads are all issued before the first FMA)
                auto four = [&](int k, auto full_t) {
                    constexpr bool FULL = decltype(full_t)::value;
                    constexpr int H = RL == 4 && !BF ? 1 : 2;  // slots in flight
                    [[maybe_unused]] uint2 raw[BF ? 9 : 1];
                    if constexpr (BF) {
#pragma unroll
                        for (int e = 0; e < 9; ++e) raw[e] = v16[((k >> 2) * 9 + e) * kSlice];
                    }
#pragma unroll
                    for (int h = 0; h < 4; h += H) {
                        X o[H][3][RL];
#pragma unroll
                        for (int u = 0; u < H; ++u)
                            if (FULL || k + h + u < kc) operand(k + h + u, o[u]);
#pragma unroll
                        for (int u = 0; u < H; ++u)
                            if (FULL || k + h + u < kc)
#pragma unroll
                                for (int i = 2; i >= 0; --i)
#pragma unroll
                                    for (int c = 0; c < 3; ++c) {
                                        if constexpr (BF) {
                                            const unsigned w = (h + u) < 2 ? raw[3 * c + i].x : raw[3 * c + i].y;
                                            fma_cases<RL>(y[c], __uint_as_float(((h + u) & 1) ? (w & 0xFFFF0000u) : (w << 16)),
                                                          o[u][i]);
                                        } else {
                                            fma_cases<RL>(y[c], v64[((k + h + u) * 9 + 3 * c + i) * kSlice], o[u][i]);
                                        }
                                    }
                    }
                };
                int k = 0;
                if constexpr (ST) {
#pragma unroll 1
                    for (; k + 4 <= kc; k += 4) four(k, std::true_type{});
                }
#pragma unroll 1
                for (; k < kc; k += 4) four(k, std::false_type{});
            };
            if (staged) run(std::true_type{});
            else run(std::false_type{});
            if (ch + kStages < nch) {  // this buffer takes a later chunk
                __syncthreads();
                if (threadIdx.x == 0 && !pipe.lost()) issue_chunk(R, ch + kStages);
            }
        }
        // the product is formed: the stage is free, the next record is in place
        if (__syncthreads_or(pipe.lost())) {
            if (threadIdx.x == 0) {
                *s_fail = 1;
                *(volatile int *)&a.gs->err = 1;
                // one more bounded wait for what may still be on its way into
                // the stage (a buffer holds one copy at most)
                if (pipe.lost()) {
                    wait(&st.bx, Pipe::kOperand);
                    for (int b = 0; b < kStages; ++b) wait(&st.bv[b], b);
                }
            }
            return;
        }
        if (more) {
            mask_next = all ? 0xffffffffu : a.vmask[Rn.v];
            if (mask_next) {
                if (warp0) issue(Rn, r0, r1);
                else if (threadIdx.x == 32) pf(Rn);
            }
        }
        if (mask) fin(R, gsl, mask, y);
    }
}

// Sums of p[q] (and p2[q] unless P2 is null) over the CTA's 32 rows for each
// of this thread's load cases, stored as P[gsl * NR + j] for j < NR (fixed
// order: lanes, then warps).
template <int NP, int RL>
__device__ __forceinline__ void slice_partial(unsigned char *dyn, double (&p)[RL], double *P, double (&p2)[RL], double *P2, int gsl,
                                              int NR) {
    constexpr int LW = Lanes<NP, RL>::kLW;
#pragma unroll
    for (int q = 0; q < RL; ++q)
#pragma unroll
        for (int off = LW; off < 32; off <<= 1) {
            p[q] += __shfl_xor_sync(0xffffffffu, p[q], off);
            if (P2) p2[q] += __shfl_xor_sync(0xffffffffu, p2[q], off);
        }
    constexpr int kW = Lanes<NP, RL>::kWarps;
    double *red = reinterpret_cast<double *>(dyn);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane < LW)
#pragma unroll
        for (int q = 0; q < RL; ++q) {
            red[w * NP + lane * RL + q] = p[q];
            if (P2) red[(kW + w) * NP + lane * RL + q] = p2[q];
        }
    __syncthreads();
    const int h = threadIdx.x / NP, j = threadIdx.x % NP;
    if (h < (P2 ? 2 : 1) && j < NR) {
        double s = 0;
        for (int ww = 0; ww < kW; ++ww) s += red[(h * kW + ww) * NP + j];
        (h ? P2 : P)[(long)gsl * NR + j] = s;
    }
}
template <int NP, int RL>
__device__ __forceinline__ void slice_partial(unsigned char *dyn, double (&p)[RL], double *P, int gsl, int NR) {
    slice_partial<NP, RL>(dyn, p, P, p, nullptr, gsl, NR);
}

// Reduce phase: one warp per (variant, load case); f(v, j, sum_pa, sum_pb).
template <class F>
__device__ __forceinline__ void for_pairs(const BArgs &a, bool two, F f) {
    const int warps = blockDim.x / 32, w = threadIdx.x / 32, lane = threadIdx.x & 31;
    for (int it = blockIdx.x * warps + w; it < a.V * a.NR; it += gridDim.x * warps) {
        const int v = it / a.NR, j = it % a.NR;
        const BVar B = a.var[v];
        double sa = 0, sb = 0;
        for (int s = lane; s < B.nslice; s += 32) {
            sa += a.pa[(long)(B.slice0 + s) * a.NR + j];
            if (two) sb += a.pb[(long)(B.slice0 + s) * a.NR + j];
        }
        sa = warp_sum(sa);
        sb = warp_sum(sb);
        if (lane == 0) f(v, j, sa, sb);
    }
}

}  // namespace

// The persistent batched solver.  MIXED: FP64 FCG + FP32 V-cycle; else PCG64.
// One CTA per slice item (grid-stride); NP / RL lanes per block row, RL load
// cases per lane.  Shared memory lets two CTAs share an SM, so the instances
// of up to 256 threads are compiled for two (128 registers).
constexpr int batch_min_ctas(int threads) { return threads <= 256 ? 2 : 1; }
template <int NP, int RL, bool MIXED>
__global__ void __launch_bounds__(32 * (NP / RL), batch_min_ctas(32 * (NP / RL))) k_batch_solve(BArgs a) {
    __shared__ Stage st;
    __shared__ int s_fail;
    extern __shared__ __align__(16) unsigned char dyn[];
    using LN = Lanes<NP, RL>;
    using ZT = typename std::conditional<MIXED, float, double>::type;  // the outer product's operand
    const unsigned nb = gridDim.x + a.extra_arrivals;
    unsigned target = 0;
    Pipe pipe;
    stage_init(st, a.copy_arrivals, &s_fail);
    const int NR = a.NR;
    const int r = LN::row(), j0 = LN::j0();
    const bool tracer = a.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
    int tn = 0;
    if (tracer && tn < a.trace_cap) a.trace[tn++] = global_ns();
    auto sync = [&]() {
        target += nb;
        const bool ok = grid_barrier(a.gs, target, a.limit_ns, &s_fail);
        if (tracer && tn < a.trace_cap) a.trace[tn++] = global_ns();
        return ok;
    };
    auto X = [&](const BVar &B, int row, int c) { return vidx<NP>(B, row, c, j0); };
    // CTA-level loop over slices: f(B, v, gsl, ls, row, live[RL], any).
    // pf(Bn, lsn), run by thread 0 as each slice starts, prefetches into L2
    // what f will read of the CTA's next slice (its HBM latency then overlaps
    // this slice's work).
    auto for_slices_pf = [&](auto pf, auto f) {
        for (int gsl = blockIdx.x; gsl < a.nslices; gsl += gridDim.x) {
            if (threadIdx.x == 0 && gsl + (int)gridDim.x < a.nslices) {
                const int gn = gsl + (int)gridDim.x;
                const BVar &Bn = a.var[a.slice_var[gn]];
                pf(Bn, gn - Bn.slice0);
            }
            const int v = a.slice_var[gsl];
            const BVar B = a.var[v];
            const int ls = gsl - B.slice0;
            const int row = ls * kSlice + r;
            bool live[RL];
            bool any = false;
#pragma unroll
            for (int q = 0; q < RL; ++q) {
                live[q] = j0 + q < NR && a.live[v * NR + j0 + q] != 0;
                any |= live[q];
            }
            f(B, v, gsl, ls, row, live, any);
        }
    };
    auto stop = [&](int v, int jj) {  // load case jj of variant v stops
        a.live[v * NR + jj] = 0;
        atomicAnd(&a.vmask[v], ~(1u << jj));
    };
    auto for_slices = [&](auto f) { for_slices_pf([](const BVar &, int) {}, f); };
    // Prefetch pieces for a slice lsn of variant Bn: the rows' runs of a batch
    // vector (esize bytes per entry), the rows' inverse diagonal blocks (FP32
    // or FP64; a partial last slice is rounded down to 16 bytes).  Used by
    // the vector phases only: in the matrix phases the prefetch measured
    // slower (thread 0's descriptor loads delay the CTA's staging barrier,
    // and K prefetched ahead competes with the gathered columns in L2).
    auto pf_rows = [&](const BVar &Bn, int lsn, const void *base, int esize) {
        const int row0 = lsn * kSlice, rows = min(kSlice, Bn.nfree - row0);
        if (rows > 0)
            l2_prefetch(static_cast<const char *>(base) + (Bn.dof0 + 3L * row0) * NP * esize,
                        3L * rows * NP * esize);
    };
    auto pf_dinv = [&](const BVar &Bn, int lsn) {
        const int row0 = lsn * kSlice, rows = min(kSlice, Bn.nfree - row0);
        if (MIXED) {
            if (rows > 0) l2_prefetch(Bn.Dinv32 + 9L * row0, (36L * rows) & ~15L);
        } else {
            if (rows > 0) l2_prefetch(Bn.Dinv + 9L * row0, (72L * rows) & ~15L);
        }
    };

    // ---- init: r = f - K u, partials ||r||^2 (pa), ||f||^2 (pb); start of M(r)
    // prefetch into L2 of the next slice's rows of a vector (esize bytes per entry)
    auto pf_vec = [&](const BSlice &R, const void *base, int esize) {
        l2_prefetch(static_cast<const char *>(base) + (R.dof + 3L * R.row0) * NP * esize,
                    3L * min(kSlice, R.nfree - R.row0) * NP * esize);
    };
    auto XR = [&](const BSlice &R, int row, int c) { return (R.dof + 3L * row + c) * NP + j0; };
    // MIXED gathers the FP64 u directly: the stage is sized for the iteration's operand
    matrix_phase<double, double, false, NP, RL>(a, st, pipe, dyn, MIXED ? 0 : a.cap, &s_fail, a.u, true, [](const BSlice &) {},
                                                [&](const BSlice &B, int gsl, unsigned, double (&y)[3][RL]) {
        const int row = B.row0 + r;
        double prr[RL] = {}, pff[RL] = {};
        if (row < B.nfree) {
            double rv[3][RL];
            for (int c = 0; c < 3; ++c) {
                double fv[RL];
                ldv<double, RL>(a.f + XR(B, row, c), fv);
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    rv[c][q] = fv[q] - y[c][q];
                    prr[q] += rv[c][q] * rv[c][q];
                    pff[q] += fv[q] * fv[q];
                }
                stv<double, RL>(a.r + XR(B, row, c), rv[c]);
            }
            if (MIXED) {
                float b[3][RL], x[3][RL];
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    float bb[3], xx[3];
                    for (int c = 0; c < 3; ++c) bb[c] = (float)rv[c][q];
                    block3_apply(B.Dinv32 + 9L * row, bb, xx);
                    for (int c = 0; c < 3; ++c) {
                        b[c][q] = bb[c];
                        x[c][q] = B.wsm * xx[c];
                    }
                }
                for (int c = 0; c < 3; ++c) {
                    stv<float, RL>(a.b32 + XR(B, row, c), b[c]);
                    stv<float, RL>(a.x32 + XR(B, row, c), x[c]);
                }
            } else {
                double z[3][RL];
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    double rr[3], zz[3];
                    for (int c = 0; c < 3; ++c) rr[c] = rv[c][q];
                    block3_apply(B.Dinv + 9L * row, rr, zz);
                    for (int c = 0; c < 3; ++c) z[c][q] = zz[c];
                }
                for (int c = 0; c < 3; ++c) stv<double, RL>(a.z64 + XR(B, row, c), z[c]);
            }
        }
        slice_partial<NP, RL>(dyn, prr, a.pa, pff, a.pb, gsl, NR);
    });
    if (!sync()) return;
    for_pairs(a, true, [&](int v, int jj, double rr, double ff) {
        const int vj = v * NR + jj;
        a.ff[vj] = ff;
        const double t = 0.5 * a.rtol;
        a.tol2[vj] = t * t * ff;
        a.live[vj] = (ff > 0.0 && rr > a.tol2[vj] && isfinite(rr)) ? 1 : 0;
        if (a.live[vj]) atomicOr(&a.vmask[v], 1u << jj);
        a.iters[vj] = 0;
        a.status[vj] = isfinite(rr) ? OFEA_OK : OFEA_ERR_BREAKDOWN;
        a.beta[vj] = 0.0;
    });
    if (!sync()) return;

    // MIXED preconditioner z_new = M(r) from b32 / x32 (pre-smoothed by the
    // phase before); partials r.z_new (pa), r.z_old (pb).  Inlined at both
    // call sites: a call would put every captured local on the stack.
    auto precondition = [&](float *znew, const float *zold) __attribute__((always_inline)) -> bool {
        // t = b - K32 x; not with K Z
        if (!a.modes)
            matrix_phase<float, float, true, NP, RL>(a, st, pipe, dyn, a.cap, &s_fail, a.x32, false,
                                                 [&](const BSlice &Rn) { pf_vec(Rn, a.b32, 4); },
                                                 [&](const BSlice &B, int, unsigned mask, float (&y)[3][RL]) {
            const int row = B.row0 + r;
            if (((mask >> j0) & ((1u << RL) - 1)) && row < B.nfree)
                for (int c = 0; c < 3; ++c) {
                    float bv[RL], t[RL];
                    ldv<float, RL>(a.b32 + XR(B, row, c), bv);
#pragma unroll
                    for (int q = 0; q < RL; ++q) t[q] = bv[q] - y[c][q];
                    stv<float, RL>(a.t32 + XR(B, row, c), t);
                }
        });
        if (!sync()) return false;
        // c = Z^T t, or Z^T b - (K Z)^T x in parts: CTA per aggregate (part), JW lanes of RL load cases per node, G nodes
        // side by side and kU per thread in flight; per-warp sums, then a
        // fixed-order sum over the warps.  RL load cases per lane share the 18
        // values of a K Z entry: one per lane reads them NP times per warp.
        // Parts because aggregates are few (about a thousand nodes each): whole
        // ones leave CTAs idle (5 variants of 7k nodes: 21 us of a 75 us
        // iteration, in parts 7 of 61).
        {
            constexpr int JW = NP / RL, kU = 4 / RL > 1 ? 4 / RL : 2;
            const int G = blockDim.x / JW, sub = threadIdx.x / JW, jj = (threadIdx.x % JW) * RL;
            const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
            float *red = reinterpret_cast<float *>(st.v);  // [warp][6][NP]: 6 * 32 * 32 floats at most
            const float *tv = a.modes ? a.b32 : a.t32;
            const int np = a.modes ? a.parts : 1;
            for (int it = blockIdx.x; it < a.naggs * np; it += gridDim.x) {
                const int ga = it / np, part = it - ga * np, v = a.agg_var[ga];
                auto cut = [&](const int *p, int I, int q) { return p[I] + (int)((long)(p[I + 1] - p[I]) * q / np); };
                const BVar &B = a.var[v];
                const int I = ga - B.agg0;
                bool live = false;
#pragma unroll
                for (int q = 0; q < RL; ++q) live |= jj + q < NR && a.live[v * NR + jj + q] != 0;
                float acc[6][RL] = {};
                if (live) {
                    auto at = [&](const float *p, int node, float (&x)[3][RL]) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) ldv<float, RL>(p + vidx<NP>(B, node, c, jj), x[c]);
                    };
                    auto add = [&](const float4 &o, const float (&t)[3][RL]) {
#pragma unroll
                        for (int q = 0; q < RL; ++q) {
                            acc[0][q] += t[0][q];
                            acc[1][q] += t[1][q];
                            acc[2][q] += t[2][q];
                            acc[3][q] += -o.z * t[1][q] + o.y * t[2][q];
                            acc[4][q] += o.z * t[0][q] - o.x * t[2][q];
                            acc[5][q] += -o.y * t[0][q] + o.x * t[1][q];
                        }
                    };
                    const int e = cut(B.agg_ptr, I, part + 1);
                    int idx = cut(B.agg_ptr, I, part) + sub;
                    for (; idx + (kU - 1) * G < e; idx += kU * G) {
                        float4 o[kU];
                        float t[kU][3][RL];
#pragma unroll
                        for (int u = 0; u < kU; ++u) o[u] = __ldg(B.agg_off + idx + u * G);
#pragma unroll
                        for (int u = 0; u < kU; ++u) at(tv, __float_as_int(o[u].w), t[u]);
#pragma unroll
                        for (int u = 0; u < kU; ++u) add(o[u], t[u]);
                    }
                    for (; idx < e; idx += G) {
                        const float4 o = __ldg(B.agg_off + idx);
                        float t[3][RL];
                        at(tv, __float_as_int(o.w), t);
                        add(o, t);
                    }
                    if (a.modes) {  // less (K Z)^T x0, the next entry's row in flight
                        const int end = cut(B.md_ptr, I, part + 1);
                        int t = cut(B.md_ptr, I, part) + sub;
                        int rr = t < end ? __ldg(B.md_row + t) : 0;
                        while (t < end) {
                            float x[3][RL], W[18];
                            mode_entry(t, B.md.n, B.md_val, W);
                            at(a.x32, rr, x);
                            t += G;
                            if (t < end) rr = __ldg(B.md_row + t);
#pragma unroll
                            for (int c = 0; c < 3; ++c)
#pragma unroll
                                for (int l = 0; l < 6; ++l) fma_cases<RL>(acc[l], -W[6 * c + l], x[c]);
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < 6; ++k)
#pragma unroll
                    for (int q = 0; q < RL; ++q)
#pragma unroll
                        for (int off = JW; off < 32; off <<= 1) acc[k][q] += __shfl_xor_sync(0xffffffffu, acc[k][q], off);
                if (lane < JW)
#pragma unroll
                    for (int k = 0; k < 6; ++k) stv<float, RL>(red + (w * 6 + k) * NP + jj, acc[k]);
                __syncthreads();
                for (int s = threadIdx.x; s < 6 * NP; s += blockDim.x) {
                    const int k = s / NP, j = s % NP;
                    float sum = 0.f;
                    for (int ww = 0; ww < nw; ++ww) sum += red[(ww * 6 + k) * NP + j];
                    const long o = B.c0 + 6L * I + k;
                    if (j < NR && a.live[v * NR + j] != 0) (a.modes ? a.cpart[(o * np + part) * NP + j] : a.cvec[o * NP + j]) = sum;
                }
                __syncthreads();
            }
        }
        if (!sync()) return false;
        // Two phases: e = E^-1 c and x += Z e, or with K Z the sum of c's parts
        // and e = E^-1 c (z's Z e is added where z is formed).
#pragma unroll 1
        for (int ph = 0; ph < 2; ++ph) {
            if (a.modes == ph) {
                // e = E^-1 c: warp per coarse row, NP lanes per load case group,
                // kE entries per lane in flight (a row is one serial sum, and only 4
                // to 16 warps share an SM: 20 load cases, 4,536 unknowns 294 us,
                // one after another 443; 16 cases, 2,880 138 and 141)
                constexpr int JW = NP, RPW = 32 / NP, kE = 8;
                const int warps = blockDim.x / 32, w = threadIdx.x / 32, lane = threadIdx.x & 31;
                const int sub = lane / JW, jj = lane % JW;
                for (int gr = blockIdx.x * warps + w; gr < a.ncrows; gr += gridDim.x * warps) {
                    const int v = a.crow_var[gr];
                    const BVar B = a.var[v];
                    const bool live = jj < NR && a.live[v * NR + jj] != 0;
                    const int i = gr - B.crow0, m = B.m;
                    const float *row = B.Einv32 + (long)i * m;
                    float acc = 0.f;
                    if (live) {
                        const float *cv = a.cvec + B.c0 * NP + jj;
                        int k = sub;
                        for (; k + (kE - 1) * RPW < m; k += kE * RPW) {
                            float e[kE], x[kE];
#pragma unroll
                            for (int u = 0; u < kE; ++u) {
                                e[u] = __ldg(row + k + u * RPW);
                                x[u] = cv[(long)(k + u * RPW) * NP];
                            }
#pragma unroll
                            for (int u = 0; u < kE; ++u) acc = fmaf(e[u], x[u], acc);
                        }
                        for (; k < m; k += RPW) acc = fmaf(__ldg(row + k), cv[(long)k * NP], acc);
                    }
#pragma unroll
                    for (int off = JW; off < 32; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
                    if (sub == 0 && live) a.evec[(B.c0 + i) * NP + jj] = acc;
                }
            } else if (a.modes) {
                for (long o = (long)blockIdx.x * blockDim.x + threadIdx.x; o < (long)a.ncoarse * NP;
                     o += (long)gridDim.x * blockDim.x) {
                    const float *p = a.cpart + (o / NP) * a.parts * NP + o % NP;
                    float sum = 0.f;
#pragma unroll 4
                    for (int q = 0; q < a.parts; ++q) sum += p[(long)q * NP];
                    a.cvec[o] = sum;
                }
            } else {
                // x += Z e
                for_slices_pf(
                    [&](const BVar &Bn, int lsn) {
                        pf_rows(Bn, lsn, a.x32, 4);
                    },
                    [&](const BVar &B, int v, int gsl, int ls, int row, const bool (&live)[RL], bool any) {
                    if (!any || row >= B.nfree) return;
                    const float4 o = __ldg(B.row_off + row);
                    const int I = __float_as_int(o.w);
                    const float dx = o.x, dy = o.y, dz = o.z;
                    float e[6][RL], x[3][RL];
                    for (int k = 0; k < 6; ++k) ldv<float, RL>(a.evec + (B.c0 + 6L * I + k) * NP + j0, e[k]);
                    for (int c = 0; c < 3; ++c) ldv<float, RL>(a.x32 + X(B, row, c), x[c]);
#pragma unroll
                    for (int q = 0; q < RL; ++q) {
                        x[0][q] += e[0][q] + dz * e[4][q] - dy * e[5][q];
                        x[1][q] += e[1][q] - dz * e[3][q] + dx * e[5][q];
                        x[2][q] += e[2][q] + dy * e[3][q] - dx * e[4][q];
                    }
                    for (int c = 0; c < 3; ++c) stv<float, RL>(a.x32 + X(B, row, c), x[c]);
                });
            }
            if (!sync()) return false;
        }
        // post-smoothing: z_new = x + w Dinv32 (b - K32 x); partials r.z_new, r.z_old
        matrix_phase<float, float, true, NP, RL>(a, st, pipe, dyn, a.cap, &s_fail, a.x32, false,
                                                 [&](const BSlice &Rn) {
                                                     pf_vec(Rn, a.b32, 4);
                                                     pf_vec(Rn, a.r, 8);
                                                     if (zold) pf_vec(Rn, zold, 4);
                                                 },
                                                 [&](const BSlice &B, int gsl, unsigned mask, float (&y)[3][RL]) {
            const int row = B.row0 + r;
            bool live[RL], any = false;
#pragma unroll
            for (int q = 0; q < RL; ++q) any |= live[q] = (mask >> (j0 + q)) & 1u;
            double pn[RL] = {}, po[RL] = {};
            if (a.modes && any && row < B.nfree) {  // y: K x0 + K Z e
                const BVar &V = a.var[B.v];
                for (int t = __ldg(V.md.rptr + row); t < __ldg(V.md.rptr + row + 1); ++t) {
                    const float *ev = a.evec + (V.c0 + 6L * __ldg(V.md.agg + t)) * NP + j0;
                    float W[18];
                    mode_entry(t, V.md.n, V.md.val, W);
#pragma unroll
                    for (int l = 0; l < 6; ++l) {
                        float e[RL];
                        ldv<float, RL>(ev + l * NP, e);
#pragma unroll
                        for (int c = 0; c < 3; ++c) fma_cases<RL>(y[c], W[6 * c + l], e);
                    }
                }
            }
            if (any && row < B.nfree) {
                float res[3][RL], xv[3][RL], zn[3][RL], zo[3][RL];
                double rv[3][RL];
                for (int c = 0; c < 3; ++c) {
                    float bv[RL];
                    ldv<float, RL>(a.b32 + XR(B, row, c), bv);
                    ldv<float, RL>(a.x32 + XR(B, row, c), xv[c]);
                    ldv<double, RL>(a.r + XR(B, row, c), rv[c]);
                    if (zold) ldv<float, RL>(zold + XR(B, row, c), zo[c]);
#pragma unroll
                    for (int q = 0; q < RL; ++q) res[c][q] = bv[q] - y[c][q];
                }
                if (a.modes) {  // x0 + Z e
                    const BVar &V = a.var[B.v];
                    const float4 o = __ldg(V.row_off + row);
                    const float *ev = a.evec + (V.c0 + 6L * __float_as_int(o.w)) * NP + j0;
                    float e[6][RL];
#pragma unroll
                    for (int l = 0; l < 6; ++l) ldv<float, RL>(ev + l * NP, e[l]);
#pragma unroll
                    for (int q = 0; q < RL; ++q) {
                        xv[0][q] += e[0][q] + o.z * e[4][q] - o.y * e[5][q];
                        xv[1][q] += e[1][q] - o.z * e[3][q] + o.x * e[5][q];
                        xv[2][q] += e[2][q] + o.y * e[3][q] - o.x * e[4][q];
                    }
                }
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    float rr[3], cor[3];
                    for (int c = 0; c < 3; ++c) rr[c] = res[c][q];
                    block3_apply(B.Dinv32 + 9L * row, rr, cor);
                    for (int c = 0; c < 3; ++c) {
                        zn[c][q] = xv[c][q] + B.wsm * cor[c];
                        if (live[q]) {
                            pn[q] += rv[c][q] * (double)zn[c][q];
                            if (zold) po[q] += rv[c][q] * (double)zo[c][q];
                        }
                    }
                }
                for (int c = 0; c < 3; ++c) stv<float, RL>(znew + XR(B, row, c), zn[c]);
            }
            slice_partial<NP, RL>(dyn, pn, a.pa, po, a.pb, gsl, NR);
        });
        return sync();
    };

    float *zcur = a.zA, *znext = a.zB;
    if (MIXED) {
        if (!precondition(zcur, nullptr)) return;
    } else {
        // PCG64: partials r.z with z64 = Dinv r
        for_slices([&](const BVar &B, int v, int gsl, int ls, int row, const bool (&)[RL], bool) {
            double p[RL] = {};
            if (row < B.nfree)
                for (int c = 0; c < 3; ++c) {
                    double rv[RL], zv[RL];
                    ldv<double, RL>(a.r + X(B, row, c), rv);
                    ldv<double, RL>(a.z64 + X(B, row, c), zv);
#pragma unroll
                    for (int q = 0; q < RL; ++q) p[q] += rv[q] * zv[q];
                }
            slice_partial<NP, RL>(dyn, p, a.pa, gsl, NR);
        });
        if (!sync()) return;
    }
    for_pairs(a, false, [&](int v, int jj, double rz, double) { a.rz[v * NR + jj] = rz; });
    if (!sync()) return;

    for (int k = 0; k < a.max_iter; ++k) {
        double *pnew = (k & 1) ? a.p1 : a.p0;
        const double *pold = (k & 1) ? a.p0 : a.p1;
        // live_cnt[k % 3] counts the load cases still running after iteration k;
        // slot (k + 1) % 3 was last read two barriers ago at least
        if (blockIdx.x == 0 && threadIdx.x == 0) a.live_cnt[(k + 1) % 3] = 0;
        // A: p = z + beta p_old, q = K64 z + beta q_old (= K64 p), partial p.q
        auto zval = [&](long d, double (&o)[RL]) {
            if (MIXED) {
                float zf[RL];
                ldv<float, RL>(zcur + d, zf);
#pragma unroll
                for (int q = 0; q < RL; ++q) o[q] = (double)zf[q];
            } else {
                ldv<double, RL>(a.z64 + d, o);
            }
        };
        const ZT *zop;
        if constexpr (MIXED) zop = zcur;
        else zop = a.z64;
        matrix_phase<double, ZT, false, NP, RL>(a, st, pipe, dyn, a.cap, &s_fail, zop, false,
                                                [&](const BSlice &Rn) {
                                                    pf_vec(Rn, pold, 8);
                                                    pf_vec(Rn, a.q, 8);
                                                },
                                                [&](const BSlice &B, int gsl, unsigned mask, double (&y)[3][RL]) {
            const int v = B.v, row = B.row0 + r;
            bool live[RL], any = false;
#pragma unroll
            for (int q = 0; q < RL; ++q) any |= live[q] = (mask >> (j0 + q)) & 1u;
            double bt[RL];
#pragma unroll
            for (int q = 0; q < RL; ++q) bt[q] = live[q] ? a.beta[v * NR + j0 + q] : 0.0;
            double ppq[RL] = {};
            if (any && row < B.nfree)
                for (int c = 0; c < 3; ++c) {
                    const long d = XR(B, row, c);
                    double zn[RL], po[RL], qo[RL], pn[RL], qn[RL];
                    zval(d, zn);
                    ldv<double, RL>(pold + d, po);
                    ldv<double, RL>(a.q + d, qo);
#pragma unroll
                    for (int q = 0; q < RL; ++q) {
                        pn[q] = fma(bt[q], po[q], zn[q]);
                        qn[q] = bt[q] != 0.0 ? fma(bt[q], qo[q], y[c][q]) : y[c][q];
                        if (live[q]) ppq[q] += pn[q] * qn[q];
                    }
                    stv<double, RL>(pnew + d, pn);
                    stv<double, RL>(a.q + d, qn);
                }
            slice_partial<NP, RL>(dyn, ppq, a.pa, gsl, NR);
        });
        if (!sync()) return;
        for_pairs(a, false, [&](int v, int jj, double pq, double) {
            const int vj = v * NR + jj;
            if (!a.live[vj]) return;
            if (!(pq > 0.0) || !isfinite(pq)) {
                stop(v, jj);
                a.status[vj] = OFEA_ERR_BREAKDOWN;
                a.iters[vj] = k;
                return;
            }
            a.alpha[vj] = a.rz[vj] / pq;
        });
        if (!sync()) return;
        // B: u += alpha p, r -= alpha q, partial ||r||^2; start of M(r)
        for_slices_pf(
            [&](const BVar &Bn, int lsn) {
                pf_rows(Bn, lsn, a.u, 8);
                pf_rows(Bn, lsn, pnew, 8);
                pf_rows(Bn, lsn, a.q, 8);
                pf_rows(Bn, lsn, a.r, 8);
                pf_dinv(Bn, lsn);
            },
            [&](const BVar &B, int v, int gsl, int ls, int row, const bool (&live)[RL], bool any) {
            double prr[RL] = {}, prz[RL] = {};
            if (any && row < B.nfree) {
                double al[RL];
#pragma unroll
                for (int q = 0; q < RL; ++q) al[q] = live[q] ? a.alpha[v * NR + j0 + q] : 0.0;
                double rv[3][RL];
                for (int c = 0; c < 3; ++c) {
                    const long d = X(B, row, c);
                    double uu[RL], pp[RL], qq[RL];
                    ldv<double, RL>(a.u + d, uu);
                    ldv<double, RL>(pnew + d, pp);
                    ldv<double, RL>(a.q + d, qq);
                    ldv<double, RL>(a.r + d, rv[c]);
#pragma unroll
                    for (int q = 0; q < RL; ++q)
                        if (live[q]) {
                            uu[q] = fma(al[q], pp[q], uu[q]);
                            rv[c][q] = fma(-al[q], qq[q], rv[c][q]);
                            prr[q] += rv[c][q] * rv[c][q];
                        }
                    stv<double, RL>(a.u + d, uu);
                    stv<double, RL>(a.r + d, rv[c]);
                }
                if (MIXED) {
                    float b[3][RL], x[3][RL];
#pragma unroll
                    for (int q = 0; q < RL; ++q) {
                        float bb[3], xx[3];
                        for (int c = 0; c < 3; ++c) bb[c] = (float)rv[c][q];
                        block3_apply(B.Dinv32 + 9L * row, bb, xx);
                        for (int c = 0; c < 3; ++c) {
                            b[c][q] = bb[c];
                            x[c][q] = B.wsm * xx[c];
                        }
                    }
                    for (int c = 0; c < 3; ++c) {
                        stv<float, RL>(a.b32 + X(B, row, c), b[c]);
                        stv<float, RL>(a.x32 + X(B, row, c), x[c]);
                    }
                } else {
                    double z[3][RL];
#pragma unroll
                    for (int q = 0; q < RL; ++q) {
                        double rr[3], zz[3];
                        for (int c = 0; c < 3; ++c) rr[c] = rv[c][q];
                        block3_apply(B.Dinv + 9L * row, rr, zz);
                        for (int c = 0; c < 3; ++c) {
                            z[c][q] = zz[c];
                            if (live[q]) prz[q] += rr[c] * zz[c];
                        }
                    }
                    for (int c = 0; c < 3; ++c) stv<double, RL>(a.z64 + X(B, row, c), z[c]);
                }
            }
            slice_partial<NP, RL>(dyn, prr, a.pa, prz, MIXED ? nullptr : a.pb, gsl, NR);
        });
        if (!sync()) return;
        for_pairs(a, !MIXED, [&](int v, int jj, double rr, double rz) {
            const int vj = v * NR + jj;
            if (!a.live[vj]) return;
            a.iters[vj] = k + 1;
            if (!isfinite(rr)) {
                stop(v, jj);
                a.status[vj] = OFEA_ERR_BREAKDOWN;
                return;
            }
            if (rr <= a.tol2[vj]) {
                stop(v, jj);
                return;
            }
            if (k + 1 >= a.max_iter) {
                stop(v, jj);
                a.status[vj] = OFEA_ERR_NOT_CONVERGED;
                return;
            }
            if (!MIXED) {
                a.beta[vj] = rz / a.rz[vj];
                a.rz[vj] = rz;
            }
            atomicAdd(&a.live_cnt[k % 3], 1);
        });
        if (!sync()) return;
        if (*(volatile int *)&a.live_cnt[k % 3] == 0) break;
        if (MIXED) {
            if (!precondition(znext, zcur)) return;
            for_pairs(a, true, [&](int v, int jj, double rzn, double rzo) {
                const int vj = v * NR + jj;
                if (!a.live[vj]) return;
                a.beta[vj] = (rzn - rzo) / a.rz[vj];
                a.rz[vj] = rzn;
            });
            if (!sync()) return;
            float *tz = zcur;
            zcur = znext;
            znext = tz;
        }
    }
}

// Host order (load case j at j * n, DOF d) to the batch's interleaved order
// (d * NP + j) for one variant (and back); padding load cases stay zero.
__global__ void k_interleave(long n, int nrhs, int NP, const double *__restrict__ src, double *__restrict__ dst) {
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < n * nrhs; g += (long)gridDim.x * blockDim.x) {
        const long j = g / n, d = g % n;
        dst[d * NP + j] = src[g];
    }
}
__global__ void k_deinterleave(long n, int nrhs, int NP, const double *__restrict__ src, double *__restrict__ dst) {
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < n * nrhs; g += (long)gridDim.x * blockDim.x) {
        const long j = g / n, d = g % n;
        dst[g] = src[d * NP + j];
    }
}

// True FP64 residual partials per (slice, load case): ||f - K u||^2 (pa), ||f||^2 (pb).
template <int NP, int RL>
__global__ void __launch_bounds__(32 * (NP / RL)) k_batch_residual(BArgs a) {
    __shared__ Stage st;
    using LN = Lanes<NP, RL>;
    __shared__ int s_fail;
    extern __shared__ __align__(16) unsigned char dyn[];
    const int NR = a.NR, j0 = LN::j0(), r = LN::row();
    Pipe pipe;
    stage_init(st, a.copy_arrivals, &s_fail);
    // u gathered directly: once per solve
    matrix_phase<double, double, false, NP, RL>(a, st, pipe, dyn, 0, &s_fail, a.u, true, [](const BSlice &) {},
                                                [&](const BSlice &B, int gsl, unsigned, double (&y)[3][RL]) {
        const int row = B.row0 + r;
        double prr[RL] = {}, pff[RL] = {};
        if (row < B.nfree)
            for (int c = 0; c < 3; ++c) {
                double fv[RL];
                ldv<double, RL>(a.f + (B.dof + 3L * row + c) * NP + j0, fv);
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    const double rv = fv[q] - y[c][q];
                    prr[q] += rv * rv;
                    pff[q] += fv[q] * fv[q];
                }
            }
        slice_partial<NP, RL>(dyn, prr, a.pa, pff, a.pb, gsl, NR);
    });
}

// The slices' records from the variants' descriptors.
__global__ void k_batch_slices(int nslices, const BVar *__restrict__ var, const int *__restrict__ slice_var,
                               BSlice *__restrict__ out) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < nslices; g += gridDim.x * blockDim.x) {
        const int v = slice_var[g];
        const BVar &B = var[v];
        const int ls = g - B.slice0;
        const long S = B.sl_ptr[ls];
        BSlice R;
        R.v64 = B.sv64 + S * 9 * kSlice;
        R.vg = B.sv16g + (long)B.sl_g[ls] * 9 * kSlice * 4;
        R.cols = B.scols + S * kSlice;
        R.runs = B.su_runs + S * kSlice;
        R.lidx = B.su_idx + S * kSlice;
        R.Dinv = B.Dinv;
        R.Dinv32 = B.Dinv32;
        R.dof = B.dof0;
        R.W = B.sl_ptr[ls + 1] - (int)S;
        R.nu = B.su_n[2 * ls];
        R.nrun = B.su_n[2 * ls + 1];
        R.row0 = ls * kSlice;
        R.nfree = B.nfree;
        R.v = v;
        R.wsm = B.wsm;
        R.pad = 0;
        out[g] = R;
    }
}

// Per (variant, load case): rel = sqrt(rr / ff).
__global__ void k_batch_rel(BArgs a, double *rel) {
    for_pairs(a, true, [&](int v, int j, double rr, double ff) {
        rel[v * a.NR + j] = ff > 0.0 ? sqrt(rr / ff) : 0.0;
    });
}

// A bounded wait that nothing releases: one extra arrival is expected at
// the first barrier, so every CTA's wait runs out after limit_ns and the
// kernel reports the failure (used to test the failure path).
__global__ void k_barrier_probe(GridBar *gs, unsigned extra, unsigned long long limit_ns, int *out) {
    __shared__ int s_fail;
    if (threadIdx.x == 0) s_fail = 0;
    const bool ok = grid_barrier(gs, gridDim.x + extra, limit_ns, &s_fail);
    if (blockIdx.x == 0 && threadIdx.x == 0) *out = ok ? 1 : 0;
}

// ------------------------------------------------------------------ host --

namespace {

struct TuneCfg {
    int rl = 2, ctas_per_sm = 1;
    double ms_per_iter = 0.0;
};

// Load-case stride of the batch vectors: NR rounded up to a power of two >= 4.
int np_for(int NR) { return NR <= 4 ? 4 : NR <= 8 ? 8 : NR <= 16 ? 16 : 32; }
int threads_for(int np, int rl) { return 32 * (np / rl); }

template <int NP, int RL>
const void *solve_inst(bool mixed) {
    return mixed ? (const void *)k_batch_solve<NP, RL, true> : (const void *)k_batch_solve<NP, RL, false>;
}
template <int NP>
const void *solve_np(int rl, bool mixed) {
    switch (rl) {
        case 1: return solve_inst<NP, 1>(mixed);
        case 2: return solve_inst<NP, 2>(mixed);
        case 4: return solve_inst<NP, 4>(mixed);
    }
    fail(OFEA_ERR_INVALID_ARG, "unsupported load cases per lane");
}
const void *solve_kernel_raw(int np, int rl, bool mixed) {
    switch (np) {
        case 4: return solve_np<4>(rl, mixed);
        case 8: return solve_np<8>(rl, mixed);
        case 16: return solve_np<16>(rl, mixed);
        case 32: return solve_np<32>(rl, mixed);
    }
    fail(OFEA_ERR_INVALID_ARG, "unsupported load-case stride");
}
// Dynamic shared memory of the staged products: the distinct columns' entries
// of the operand (FP32 for MIXED, FP64 for PCG64).
// At most what lets two CTAs share an SM (228 KB, 1 KB reserved per CTA).
constexpr int kStageLimit = 112 * 1024 - (int)sizeof(Stage) - 256;  // partial sums included
int col_bytes(int np, bool mixed) { return 3 * np * (mixed ? 4 : 8); }
int stage_cap(int su_max, int np, int rl, bool mixed) {
    return std::min(su_max, (kStageLimit - red_bytes(np, rl)) / col_bytes(np, mixed));
}
int stage_bytes(int su_max, int np, int rl, bool mixed) {
    return red_bytes(np, rl) + stage_cap(su_max, np, rl, mixed) * col_bytes(np, mixed);
}
// Kernel instance for (NP, RL, mixed), with the shared-memory carveout at its
// maximum so that several CTAs' slot stages fit on an SM.
const void *solve_kernel(int np, int rl, bool mixed) {
    const void *fn = solve_kernel_raw(np, rl, mixed);
    OFEA_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   (int)cudaSharedmemCarveoutMaxShared));
    OFEA_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kStageLimit));
    return fn;
}
template <int NP>
const void *residual_np(int rl) {
    switch (rl) {
        case 1: return (const void *)k_batch_residual<NP, 1>;
        case 2: return (const void *)k_batch_residual<NP, 2>;
        case 4: return (const void *)k_batch_residual<NP, 4>;
    }
    fail(OFEA_ERR_INVALID_ARG, "unsupported load cases per lane");
}
const void *residual_kernel(int np, int rl) {
    switch (np) {
        case 4: return residual_np<4>(rl);
        case 8: return residual_np<8>(rl);
        case 16: return residual_np<16>(rl);
        case 32: return residual_np<32>(rl);
    }
    fail(OFEA_ERR_INVALID_ARG, "unsupported load-case stride");
}

// ---- the on-disk tuning cache: one JSON object per line inside "entries"
std::mutex g_tune_mu;

std::string tune_path() {
    if (const char *p = std::getenv("OFEA_TUNE_FILE")) return p;
    const char *home = std::getenv("HOME");
    return std::string(home ? home : ".") + "/.cache/openfea_b200_tune.json";
}

std::map<std::string, TuneCfg> tune_load(const std::string &path) {
    std::map<std::string, TuneCfg> out;
    std::ifstream in(path);
    std::string line;
    auto num = [](const std::string &l, const char *k, double dflt) {
        const std::string key = std::string("\"") + k + "\": ";
        const size_t p = l.find(key);
        return p == std::string::npos ? dflt : std::strtod(l.c_str() + p + key.size(), nullptr);
    };
    while (std::getline(in, line)) {
        const size_t p = line.find("\"key\": \"");
        if (p == std::string::npos) continue;
        const size_t b = p + 8, e = line.find('"', b);
        if (e == std::string::npos) continue;
        TuneCfg t;
        t.rl = (int)num(line, "rl", 2);
        t.ctas_per_sm = (int)num(line, "ctas_per_sm", 1);
        t.ms_per_iter = num(line, "ms_per_iter", 0);
        out[line.substr(b, e - b)] = t;
    }
    return out;
}

void tune_store(const std::string &path, const std::string &key, const TuneCfg &t) {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto all = tune_load(path);
    all[key] = t;
    const size_t slash = path.rfind('/');
    if (slash != std::string::npos && slash > 0) mkdir(path.substr(0, slash).c_str(), 0755);  // one level (~/.cache)
    std::ofstream o(path);
    if (!o) return;  // the cache is an optimisation: an unwritable path is not an error
    o << "{\n  \"entries\": [\n";
    size_t i = 0;
    for (const auto &kv : all) {
        char buf[512];
        std::snprintf(buf, sizeof(buf),
                      "    {\"key\": \"%s\", \"rl\": %d, \"ctas_per_sm\": %d, \"ms_per_iter\": %.6f}%s\n",
                      kv.first.c_str(), kv.second.rl, kv.second.ctas_per_sm,
                      kv.second.ms_per_iter, ++i < all.size() ? "," : "");
        o << buf;
    }
    o << "  ]\n}\n";
}

}  // namespace

// ---- the batch plan

}  // namespace ofea

struct ofea_batch {
    int device = 0, V = 0, NR = 0, NP = 4, num_sms = 148;
    cudaStream_t stream = nullptr;
    std::vector<ofea_ctx *> ctx;
    std::vector<long> dof0, c0;
    long ndof = 0, ncoarse = 0;
    int nslices = 0, naggs = 0, ncrows = 0, su_max = 0;
    bool mixed_ready = false, have_rhs = false, modes = false;
    int parts = 1;
    ofea::DevBuf<ofea::BVar> var;
    ofea::DevBuf<ofea::BSlice> slice;
    ofea::DevBuf<unsigned> vmask;
    ofea::DevBuf<int> slice_var, agg_var, crow_var;
    ofea::DevBuf<double> f, u, r, p0, p1, q, z64, pa, pb, ff, tol2, rz, alpha, beta, rel, stage;
    ofea::DevBuf<float> b32, x32, t32, zA, zB, cvec, evec, cpart;
    ofea::DevBuf<int> live, iters, status, live_cnt;
    ofea::DevBuf<ofea::GridBar> gs;
    ofea::DevBuf<unsigned long long> trace;  // per-phase timestamps when tracing (trace_cap > 0)
    ofea::HostBuf<double> bounce[2];          // page-locked blocks between the callers' arrays and the device
    int trace_cap = 0;
    std::map<int, ofea::TuneCfg> tuned;  // by method
    // the captured graph of one launch and what it was captured for
    cudaGraphExec_t exec = nullptr;
    std::string exec_key;
    ~ofea_batch() {
        if (exec) cudaGraphExecDestroy(exec);
    }
};

namespace ofea {

namespace {

// The device's name, asked for once per device: the query takes 3.3 ms, and a
// solve with several load cases makes its batch anew.
std::string device_name(int dev) {
    static std::mutex mu;
    static std::map<int, std::string> names;
    std::lock_guard<std::mutex> lock(mu);
    auto it = names.find(dev);
    if (it == names.end()) {
        cudaDeviceProp p{};
        if (cudaGetDeviceProperties(&p, dev) != cudaSuccess) {
            cudaGetLastError();
            return "gpu";
        }
        it = names.emplace(dev, p.name).first;
    }
    return it->second;
}

// Descriptor table; with `mixed` also the coarse levels' pointers and offsets.
void build_desc(ofea_batch *b, bool mixed) {
    std::vector<BVar> d(b->V);
    std::vector<int> sv, av, cv;
    long c0 = 0;
    int slice0 = 0, agg0 = 0, crow0 = 0;
    b->c0.assign(b->V, 0);
    for (int v = 0; v < b->V; ++v) {
        ofea_ctx *c = b->ctx[v];
        BVar &B = d[v];
        std::memset(&B, 0, sizeof(B));
        B.nfree = c->nfree;
        B.n = c->n;
        B.nslice = (c->nfree + kSlice - 1) / kSlice;
        B.slice0 = slice0;
        B.dof0 = b->dof0[v];
        B.sl_ptr = c->sl_ptr.p;
        B.scols = c->scols.p;
        B.sv64 = c->sv64.p;
        B.Dinv = c->Dinv.p;
        B.sl_g = c->sl_g.p;
        B.su_runs = reinterpret_cast<const int2 *>(c->su_runs.p);
        B.su_n = c->su_n.p;
        B.su_idx = c->su_idx.p;
        B.sv16g = c->sv16g.p;
        b->su_max = std::max(b->su_max, c->su_max);
        B.Dinv32 = c->Dinv32.p;
        for (int s = 0; s < B.nslice; ++s) sv.push_back(v);
        slice0 += B.nslice;
        if (mixed) {
            const Coarse &C = c->coarse;
            B.na = C.na;
            B.m = C.m;
            B.agg0 = agg0;
            B.crow0 = crow0;
            B.c0 = c0;
            b->c0[v] = c0;
            B.agg_ptr = C.agg_ptr.p;
            B.agg_off = reinterpret_cast<const float4 *>(C.agg_off.p);
            B.row_off = reinterpret_cast<const float4 *>(C.row_off.p);
            B.Einv32 = C.Einv32.p;
            if (b->modes) {
                B.md_ptr = C.md_ptr.p;
                B.md_row = C.md_row.p;
                B.md_val = C.md_val.p;
                B.md = row_modes(C);
            }
            B.wsm = smoother_weight(c, kBatchSmootherDamping);
            for (int a = 0; a < C.na; ++a) av.push_back(v);
            for (int i = 0; i < C.m; ++i) cv.push_back(v);
            agg0 += C.na;
            crow0 += C.m;
            c0 += C.m;
        }
    }
    b->nslices = slice0;
    b->naggs = agg0;
    b->ncrows = crow0;
    b->ncoarse = c0;
    cudaStream_t s = b->stream;
    b->var.upload(d.data(), d.size(), s);
    b->slice_var.upload(sv.data(), sv.size(), s);
    b->slice.ensure(std::max<size_t>(1, sv.size()));
    b->vmask.ensure(b->V);
    k_batch_slices<<<std::max(1, std::min(kMaxGrid, (slice0 + 255) / 256)), 256, 0, s>>>(slice0, b->var.p, b->slice_var.p,
                                                                                       b->slice.p);
    OFEA_CHECK_LAUNCH();
    if (mixed) {
        b->agg_var.upload(av.data(), av.size(), s);
        b->crow_var.upload(cv.data(), cv.size(), s);
    }
    const size_t NR = b->NR;
    b->pa.ensure(std::max<size_t>(1, (size_t)b->nslices * NR));
    b->pb.ensure(std::max<size_t>(1, (size_t)b->nslices * NR));
    OFEA_CUDA(cudaStreamSynchronize(s));
}

// K Z in a batch up to so many entries per row (about 1,000 nodes per
// aggregate give 0.3 to 1): a product serves all load cases with one read of a
// matrix value, K Z's sums gather six coarse values per entry and load case.
// MIXED solve with K Z / without, ms, 1 variant: 16 load cases, 17.6k nodes C3D8,
// 0.7 entries per row 4.84 / 5.94, 1.3 4.41 / 4.50, 1.8 4.53 / 4.26, 2.6 5.68 /
// 5.14; 32, 4.8k nodes C3D4, 0.4 5.16 / 6.67, 1.4 3.29 / 3.20, 2.2 3.05 / 2.56;
// 16, 46k nodes C3D8, 0.8 12.2 / 13.7, 1.4 10.7 / 11.3, 2.0 11.8 / 11.6.
constexpr double kBatchModes = 1.5;

void prepare(ofea_batch *b, bool mixed) {
    if (mixed && !b->mixed_ready) {
        for (ofea_ctx *c : b->ctx) {
            setup_coarse(c, c->coarse_nodes);
            coarse_dense_inverse(c);
            OFEA_CUDA(cudaStreamSynchronize(c->stream));
        }
        const size_t n = (size_t)b->ndof * b->NP;
        for (auto *buf : {&b->b32, &b->x32, &b->t32, &b->zA, &b->zB}) buf->ensure(n);
        size_t naggs = 0, ncrows = 0;
        for (ofea_ctx *c : b->ctx) {
            naggs += c->coarse.na;
            ncrows += c->coarse.m;
        }
        const size_t nc = std::max<size_t>(1, ncrows * b->NP);
        b->agg_var.ensure(naggs);
        b->crow_var.ensure(ncrows);
        b->cvec.ensure(nc);
        b->evec.ensure(nc);
        // K Z after all that the solve cannot do without: where memory ends, it
        // gives way
        long entries = 0, rows = 0;
        b->modes = true;
        for (ofea_ctx *c : b->ctx) {
            const long e = b->modes ? count_modes(c, c->coarse) : -1;
            b->modes = e >= 0;
            entries += e;
            rows += c->nfree;
        }
        b->modes = b->modes && entries <= kBatchModes * rows;
        for (ofea_ctx *c : b->ctx) {
            if (b->modes) b->modes = ensure_modes(c, c->coarse);
            else c->coarse.md_slots.release();
            OFEA_CUDA(cudaStreamSynchronize(c->stream));
        }
        if (b->modes) {  // about eight parts per SM
            b->parts = std::min(16, 8 * b->num_sms / (int)std::max<size_t>(1, naggs) + 1);
            try {
                b->cpart.ensure(nc * b->parts);
                OFEA_CUDA(cudaMemsetAsync(b->cpart.p, 0, sizeof(float) * nc * b->parts, b->stream));
            } catch (const Failure &f) {
                if (f.code != OFEA_ERR_OOM) throw;
                b->modes = false;
            }
        }
        build_desc(b, true);
        for (auto *buf : {&b->b32, &b->x32, &b->t32, &b->zA, &b->zB})
            OFEA_CUDA(cudaMemsetAsync(buf->p, 0, sizeof(float) * n, b->stream));
        OFEA_CUDA(cudaMemsetAsync(b->cvec.p, 0, sizeof(float) * nc, b->stream));
        OFEA_CUDA(cudaMemsetAsync(b->evec.p, 0, sizeof(float) * nc, b->stream));
        b->mixed_ready = true;
    }
    if (!mixed && !b->z64.p) {
        b->z64.ensure((size_t)b->ndof * b->NP);
        OFEA_CUDA(cudaMemsetAsync(b->z64.p, 0, sizeof(double) * b->ndof * b->NP, b->stream));
    }
}

BArgs make_args(ofea_batch *b, bool mixed, const TuneCfg &t, int max_iter, double rtol) {
    BArgs a{};
    a.V = b->V;
    a.NR = b->NR;
    a.nslices = b->nslices;
    a.naggs = mixed ? b->naggs : 0;
    a.ncrows = mixed ? b->ncrows : 0;
    a.max_iter = max_iter;
    a.extra_arrivals = 0;
    a.copy_arrivals = 1;
    a.limit_ns = 5000000000ull;  // 5 s: far above any phase
    a.rtol = rtol;
    a.var = b->var.p;
    a.slice = b->slice.p;
    a.vmask = b->vmask.p;
    a.modes = mixed && b->modes;
    a.parts = b->parts;
    a.ncoarse = b->ncoarse;
    a.cpart = b->cpart.p;
    a.cap = stage_cap(b->su_max, b->NP, t.rl, mixed);
    a.slice_var = b->slice_var.p;
    a.agg_var = b->agg_var.p;
    a.crow_var = b->crow_var.p;
    a.f = b->f.p;
    a.u = b->u.p;
    a.r = b->r.p;
    a.p0 = b->p0.p;
    a.p1 = b->p1.p;
    a.q = b->q.p;
    a.z64 = b->z64.p;
    a.b32 = b->b32.p;
    a.x32 = b->x32.p;
    a.t32 = b->t32.p;
    a.zA = b->zA.p;
    a.zB = b->zB.p;
    a.cvec = b->cvec.p;
    a.evec = b->evec.p;
    a.pa = b->pa.p;
    a.pb = b->pb.p;
    a.ff = b->ff.p;
    a.tol2 = b->tol2.p;
    a.rz = b->rz.p;
    a.alpha = b->alpha.p;
    a.beta = b->beta.p;
    a.live = b->live.p;
    a.iters = b->iters.p;
    a.status = b->status.p;
    a.live_cnt = b->live_cnt.p;
    a.gs = b->gs.p;
    a.trace = b->trace_cap > 0 ? b->trace.p : nullptr;
    a.trace_cap = b->trace_cap;
    return a;
}

int grid_of(ofea_batch *b, const void *fn, const TuneCfg &t, int smem) {
    int occ = 0;
    OFEA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads_for(b->NP, t.rl), smem));
    if (occ < 1) fail(OFEA_ERR_CAPACITY, "batched solver kernel does not fit on an SM");
    return b->num_sms * std::min(occ, t.ctas_per_sm);
}

// Enqueue one launch: reset of the per-launch state + the cooperative kernel.
void enqueue(ofea_batch *b, const BArgs &a, const TuneCfg &t, bool mixed) {
    cudaStream_t s = b->stream;
    const size_t n = (size_t)b->ndof * b->NP;
    OFEA_CUDA(cudaMemsetAsync(b->p0.p, 0, sizeof(double) * n, s));
    OFEA_CUDA(cudaMemsetAsync(b->p1.p, 0, sizeof(double) * n, s));
    OFEA_CUDA(cudaMemsetAsync(b->gs.p, 0, sizeof(GridBar), s));
    OFEA_CUDA(cudaMemsetAsync(b->live_cnt.p, 0, sizeof(int) * 3, s));
    OFEA_CUDA(cudaMemsetAsync(b->vmask.p, 0, sizeof(unsigned) * b->V, s));
    if (a.trace) OFEA_CUDA(cudaMemsetAsync(a.trace, 0, sizeof(unsigned long long) * a.trace_cap, s));
    const void *fn = solve_kernel(b->NP, t.rl, mixed);
    cudaLaunchConfig_t cfg{};
    const int smem = stage_bytes(b->su_max, b->NP, t.rl, mixed);
    cfg.gridDim = dim3(grid_of(b, fn, t, smem));
    cfg.blockDim = dim3(threads_for(b->NP, t.rl));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {(void *)&a};
    OFEA_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
}

// True FP64 residuals per (variant, load case) into b->rel.
void residuals(ofea_batch *b, BArgs a, const TuneCfg &t) {
    cudaStream_t s = b->stream;
    const void *fn = residual_kernel(b->NP, t.rl);
    const int G = std::min(kMaxGrid, b->num_sms * 4), smem = red_bytes(b->NP, t.rl);
    // with the slot stage above 48 KB at 32 cases, one per lane
    OFEA_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    void *args[] = {(void *)&a};
    OFEA_CUDA(cudaLaunchKernel(fn, dim3(G), dim3(threads_for(b->NP, t.rl)), args, (size_t)smem, s));
    k_batch_rel<<<std::max(1, std::min(kMaxGrid, (b->V * b->NR + 7) / 8)), 256, 0, s>>>(a, b->rel.p);
    OFEA_CHECK_LAUNCH();
}

constexpr int kTuneVersion = 2;  // raised when the kernels' best shapes may have moved

std::string tune_key(ofea_batch *b, bool mixed) {
    // problem class: device, method, load cases, rows rounded to 2 significant
    // digits, variants; what else decides the best shape: the kernels' version,
    // K Z, the most columns of a slice (whether they fit the stage) and the coarse
    // unknowns (both rounded too).
    // With the choices of the kernels before these, 4 variants x 32 load cases
    // took 1,285 us per iteration instead of 551, 1 x 16 54.5 instead of 47.0.
    auto round2 = [](long x) {
        long scale = 1;
        while (x / scale >= 100) scale *= 10;
        return x / scale * scale;
    };
    std::ostringstream k;
    k << device_name(b->device) << "|" << (mixed ? "mixed" : "pcg64") << "|nrhs=" << b->NR
      << "|rows~" << round2((long)b->nslices * kSlice) << "|variants=" << b->V << "|kernels=" << kTuneVersion
      << "|kz=" << (mixed && b->modes ? 1 : 0) << "|columns~" << round2(b->su_max) << "|coarse~"
      << round2(mixed ? b->ncrows : 0);
    return k.str();
}

// Times a few iterations of every candidate and keeps the fastest; the
// result is cached in the batch and on disk (OFEA_TUNE_FILE or
// ~/.cache/openfea_b200_tune.json), keyed by device and problem class.
TuneCfg autotune(ofea_batch *b, bool mixed, double rtol) {
    const std::string key = tune_key(b, mixed);
    const std::string path = tune_path();
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        auto all = tune_load(path);
        auto it = all.find(key);
        if (it != all.end()) {
            TuneCfg t = it->second;
            if ((t.rl == 1 || t.rl == 2 || t.rl == 4) && t.rl <= b->NP && t.ctas_per_sm >= 1 && t.ctas_per_sm <= 32)
                return t;
        }
    }
    std::vector<TuneCfg> cand;
    for (int rl : {1, 2, 4}) {
        int occ = 0;
        OFEA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, solve_kernel(b->NP, rl, mixed),
                                                                threads_for(b->NP, rl),
                                                                stage_bytes(b->su_max, b->NP, rl, mixed)));
        std::vector<int> cps{1, 2, 4, occ};
        std::sort(cps.begin(), cps.end());
        cps.erase(std::unique(cps.begin(), cps.end()), cps.end());
        for (int c : cps)
            if (c >= 1 && c <= occ) cand.push_back(TuneCfg{rl, c, 0.0});
    }
    // per-iteration time = (t(long) - t(short)) / (long - short): the init
    // phases and the launch cancel out
    const int it_short = 4, it_long = 20;
    cudaEvent_t e0, e1;
    OFEA_CUDA(cudaEventCreate(&e0));
    OFEA_CUDA(cudaEventCreate(&e1));
    TuneCfg best;
    double best_ms = 1e300;
    cudaStream_t s = b->stream;
    auto time_launch = [&](const TuneCfg &t, int iters) {
        double ms_min = 1e300;
        for (int rep = 0; rep < 3; ++rep) {
            OFEA_CUDA(cudaMemsetAsync(b->u.p, 0, sizeof(double) * b->ndof * b->NP, s));
            BArgs a = make_args(b, mixed, t, iters, rtol);
            OFEA_CUDA(cudaEventRecord(e0, s));
            enqueue(b, a, t, mixed);
            OFEA_CUDA(cudaEventRecord(e1, s));
            OFEA_CUDA(cudaEventSynchronize(e1));
            float ms = 0;
            OFEA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            GridBar g{};
            OFEA_CUDA(cudaMemcpy(&g, b->gs.p, sizeof(g), cudaMemcpyDeviceToHost));
            if (g.err) fail(OFEA_ERR_TIMEOUT, "batched solver: a grid-barrier wait ran out while tuning");
            ms_min = std::min(ms_min, (double)ms);
        }
        return ms_min;
    };
    const bool verbose = std::getenv("OFEA_TUNE_VERBOSE") != nullptr;
    for (TuneCfg &t : cand) {
        t.ms_per_iter = std::max(0.0, time_launch(t, it_long) - time_launch(t, it_short)) / (it_long - it_short);
        if (verbose)
            std::fprintf(stderr, "ofea tune %s: rl %d ctas/SM %d -> %.4f ms per iteration\n", key.c_str(), t.rl,
                         t.ctas_per_sm, t.ms_per_iter);
        if (t.ms_per_iter < best_ms) {
            best_ms = t.ms_per_iter;
            best = t;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    tune_store(path, key, best);
    return best;
}

}  // namespace

ofea_batch *batch_create(ofea_ctx *const *ctxs, int nv, int nrhs) {
    if (!ctxs || nv < 1) fail(OFEA_ERR_INVALID_ARG, "batch: no variants");
    if (nrhs < 1 || nrhs > kMaxBatchRhs)
        fail(OFEA_ERR_CAPACITY, "batch: 1 to " + std::to_string(kMaxBatchRhs) + " load cases per variant");
    auto b = std::make_unique<ofea_batch>();
    b->V = nv;
    b->NR = nrhs;
    b->NP = np_for(nrhs);
    for (int v = 0; v < nv; ++v) {
        ofea_ctx *c = ctxs[v];
        if (!c) fail(OFEA_ERR_INVALID_ARG, "batch: NULL context");
        if (!c->K_ok || !c->sell_ok) fail(OFEA_ERR_STATE, "batch: variant " + std::to_string(v) + " not assembled");
        OFEA_CUDA(cudaSetDevice(c->device));
        ensure_slice_columns(c);  // once per pattern
        OFEA_CUDA(cudaStreamSynchronize(c->stream));
        if (c->device != ctxs[0]->device) fail(OFEA_ERR_INVALID_ARG, "batch: variants on different GPUs");
        b->ctx.push_back(c);
    }
    b->device = ctxs[0]->device;
    b->num_sms = ctxs[0]->num_sms;
    b->stream = ctxs[0]->stream;
    OFEA_CUDA(cudaSetDevice(b->device));
    int coop = 0;
    OFEA_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, b->device));
    if (!coop) fail(OFEA_ERR_NO_DEVICE, "batch: the GPU does not support cooperative launches");
    long d0 = 0;
    for (ofea_ctx *c : b->ctx) {
        b->dof0.push_back(d0);
        d0 += c->n;
    }
    b->ndof = d0;
    const size_t n = std::max<size_t>(1, (size_t)b->ndof * b->NP), vj = (size_t)nv * nrhs;
    for (auto *buf : {&b->f, &b->u, &b->r, &b->p0, &b->p1, &b->q}) buf->ensure(n);
    for (auto *buf : {&b->ff, &b->tol2, &b->rz, &b->alpha, &b->beta, &b->rel}) buf->ensure(vj);
    for (auto *buf : {&b->live, &b->iters, &b->status}) buf->ensure(vj);
    b->live_cnt.ensure(3);
    b->gs.ensure(1);
    OFEA_CUDA(cudaMemsetAsync(b->f.p, 0, sizeof(double) * n, b->stream));
    OFEA_CUDA(cudaMemsetAsync(b->u.p, 0, sizeof(double) * n, b->stream));
    build_desc(b.get(), false);
    return b.release();
}

void batch_destroy(ofea_batch *b) {
    if (!b) return;
    cudaSetDevice(b->device);
    delete b;
}

namespace {

// dst <- src (host memory, bytes), split over the host pool's chunks when large.
void host_copy(void *dst, const void *src, size_t bytes) {
    if (bytes < (size_t(4) << 20)) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const long units = (long)(bytes / 64);
    host_for_chunks([&](int k) {
        const size_t a = (size_t)chunk_begin(units, k) * 64;
        const size_t e = k + 1 == kHostChunks ? bytes : (size_t)chunk_begin(units, k + 1) * 64;
        std::memcpy(static_cast<char *>(dst) + a, static_cast<const char *>(src) + a, e - a);
    });
}

// Two events for the bounce blocks, destroyed on every exit.
struct EventPair {
    cudaEvent_t e[2] = {nullptr, nullptr};
    EventPair() {
        for (auto &x : e) OFEA_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
    }
    ~EventPair() {
        for (auto &x : e)
            if (x) cudaEventDestroy(x);
    }
};

}  // namespace

// The callers' arrays are pageable: each variant goes through one of two
// page-locked bounce blocks, the host copy of one variant (over the host
// pool's chunks) overlapping the DMA of the other.
void batch_set_rhs(ofea_batch *b, const double *const *f) {
    OFEA_CUDA(cudaSetDevice(b->device));
    cudaStream_t s = b->stream;
    size_t maxn = 1;
    for (int v = 0; v < b->V; ++v) {
        if (!f[v]) fail(OFEA_ERR_INVALID_ARG, "batch: NULL load array");
        maxn = std::max(maxn, (size_t)b->ctx[v]->n * b->NR);
    }
    b->stage.ensure((size_t)b->ndof * b->NR);
    for (auto &h : b->bounce) h.ensure(maxn);
    EventPair ev;
    for (int v = 0; v < b->V; ++v) {
        const long n = b->ctx[v]->n;
        const int k = v & 1;
        double *dst = b->stage.p + b->dof0[v] * b->NR;
        if (v >= 2) OFEA_CUDA(cudaEventSynchronize(ev.e[k]));  // the DMA out of this block (variant v - 2) is done
        host_copy(b->bounce[k].p, f[v], sizeof(double) * n * b->NR);
        OFEA_CUDA(cudaMemcpyAsync(dst, b->bounce[k].p, sizeof(double) * n * b->NR, cudaMemcpyHostToDevice, s));
        OFEA_CUDA(cudaEventRecord(ev.e[k], s));
        k_interleave<<<std::max(1, std::min(kMaxGrid, (int)((n * b->NR + 255) / 256))), 256, 0, s>>>(
            n, b->NR, b->NP, dst, b->f.p + b->dof0[v] * b->NP);
        OFEA_CHECK_LAUNCH();
    }
    OFEA_CUDA(cudaStreamSynchronize(s));
    b->have_rhs = true;
}

void batch_get_solution(ofea_batch *b, double *const *u) {
    OFEA_CUDA(cudaSetDevice(b->device));
    cudaStream_t s = b->stream;
    size_t maxn = 1;
    for (int v = 0; v < b->V; ++v) {
        if (!u[v]) fail(OFEA_ERR_INVALID_ARG, "batch: NULL solution array");
        maxn = std::max(maxn, (size_t)b->ctx[v]->n * b->NR);
    }
    b->stage.ensure((size_t)b->ndof * b->NR);
    for (auto &h : b->bounce) h.ensure(maxn);
    for (int v = 0; v < b->V; ++v) {
        const long n = b->ctx[v]->n;
        k_deinterleave<<<std::max(1, std::min(kMaxGrid, (int)((n * b->NR + 255) / 256))), 256, 0, s>>>(
            n, b->NR, b->NP, b->u.p + b->dof0[v] * b->NP, b->stage.p + b->dof0[v] * b->NR);
        OFEA_CHECK_LAUNCH();
    }
    EventPair ev;
    for (int v = 0; v <= b->V; ++v) {
        if (v < b->V) {  // block v & 1 was last read by the host copy of variant v - 2, already done
            const long n = b->ctx[v]->n;
            OFEA_CUDA(cudaMemcpyAsync(b->bounce[v & 1].p, b->stage.p + b->dof0[v] * b->NR, sizeof(double) * n * b->NR,
                                      cudaMemcpyDeviceToHost, s));
            OFEA_CUDA(cudaEventRecord(ev.e[v & 1], s));
        }
        if (v > 0) {
            const int w = v - 1;
            OFEA_CUDA(cudaEventSynchronize(ev.e[w & 1]));
            host_copy(u[w], b->bounce[w & 1].p, sizeof(double) * b->ctx[w]->n * b->NR);
        }
    }
}

void batch_tuning(ofea_batch *b, int method, int *rl, int *threads, int *ctas_per_sm, double *ms_per_iter) {
    const bool mixed = method == OFEA_SOLVER_MIXED;
    OFEA_CUDA(cudaSetDevice(b->device));
    prepare(b, mixed);
    auto it = b->tuned.find(method);
    if (it == b->tuned.end()) it = b->tuned.emplace(method, autotune(b, mixed, 1e-8)).first;
    const TuneCfg &t = it->second;
    if (rl) *rl = t.rl;
    if (threads) *threads = threads_for(b->NP, t.rl);
    if (ctas_per_sm) *ctas_per_sm = t.ctas_per_sm;
    if (ms_per_iter) *ms_per_iter = t.ms_per_iter;
}

// Solves all (variant, load case) pairs on the resident right-hand sides.
// One graph launch per attempt; a pair whose true FP64 residual misses rtol
// after the kernel (recurrence drift) is resumed from its u by the next
// attempt.  stats: one per variant (worst load case).
void batch_solve(ofea_batch *b, const ofea_solve_opts &o, ofea_solve_stats *stats, ofea_solve_stats *case_stats) {
    if (o.method != OFEA_SOLVER_MIXED && o.method != OFEA_SOLVER_PCG64)
        fail(OFEA_ERR_UNKNOWN_SOLVER, "batch: method must be OFEA_SOLVER_PCG64 or OFEA_SOLVER_MIXED");
    if (!b->have_rhs) fail(OFEA_ERR_STATE, "batch: no load cases set");
    if (!(o.rtol > 0) || o.max_iter < 1) fail(OFEA_ERR_INVALID_ARG, "batch: bad rtol / max_iter");
    const bool mixed = o.method == OFEA_SOLVER_MIXED;
    OFEA_CUDA(cudaSetDevice(b->device));
    prepare(b, mixed);
    batch_tuning(b, o.method, nullptr, nullptr, nullptr, nullptr);
    const TuneCfg t = b->tuned[o.method];
    cudaStream_t s = b->stream;
    const int VJ = b->V * b->NR;
    std::vector<int> iters_tot(VJ, 0), hit(VJ), hst(VJ);
    std::vector<double> hrel(VJ);
    cudaEvent_t e0, e1;
    OFEA_CUDA(cudaEventCreate(&e0));
    OFEA_CUDA(cudaEventCreate(&e1));
    OFEA_CUDA(cudaMemsetAsync(b->u.p, 0, sizeof(double) * b->ndof * b->NP, s));
    OFEA_CUDA(cudaEventRecord(e0, s));
    int attempts = 0, launches = 0, remaining = o.max_iter;
    bool failed_barrier = false;
    for (; attempts < 4 && remaining > 0; ++attempts) {
        BArgs a = make_args(b, mixed, t, remaining, o.rtol);
        std::ostringstream k;
        k << o.method << "/" << t.rl << "/" << t.ctas_per_sm << "/" << remaining << "/"
          << o.rtol << "/" << b->trace_cap;
        if (o.use_graph) {
            if (!b->exec || b->exec_key != k.str()) {
                if (b->exec) {
                    cudaGraphExecDestroy(b->exec);
                    b->exec = nullptr;
                }
                cudaGraph_t g = nullptr;
                OFEA_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
                try {
                    enqueue(b, a, t, mixed);
                } catch (...) {
                    cudaStreamEndCapture(s, &g);
                    if (g) cudaGraphDestroy(g);
                    throw;
                }
                OFEA_CUDA(cudaStreamEndCapture(s, &g));
                cudaError_t e = cudaGraphInstantiate(&b->exec, g, 0);
                cudaGraphDestroy(g);
                if (e != cudaSuccess) fail_cuda(e, "cudaGraphInstantiate(batched solve)", __FILE__, __LINE__);
                b->exec_key = k.str();
            }
            OFEA_CUDA(cudaGraphLaunch(b->exec, s));
        } else {
            enqueue(b, a, t, mixed);
        }
        ++launches;
        residuals(b, make_args(b, false, t, 0, 0.0), t);
        launches += 2;
        GridBar g{};
        OFEA_CUDA(cudaMemcpyAsync(&g, b->gs.p, sizeof(g), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaMemcpyAsync(hit.data(), b->iters.p, sizeof(int) * VJ, cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaMemcpyAsync(hst.data(), b->status.p, sizeof(int) * VJ, cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaMemcpyAsync(hrel.data(), b->rel.p, sizeof(double) * VJ, cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaStreamSynchronize(s));
        if (g.err) {
            failed_barrier = true;
            break;
        }
        int most = 0;
        bool again = false;
        for (int i = 0; i < VJ; ++i) {
            iters_tot[i] += hit[i];
            most = std::max(most, hit[i]);
            if (hst[i] == OFEA_OK && !(hrel[i] <= o.rtol)) again = true;
        }
        remaining -= std::max(most, 1);
        if (!again) break;
    }
    OFEA_CUDA(cudaEventRecord(e1, s));
    OFEA_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    OFEA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (failed_barrier) fail(OFEA_ERR_TIMEOUT, "batched solver: a grid-barrier wait ran out");
    if (stats) {
        for (int v = 0; v < b->V; ++v) {
            ofea_solve_stats &st = stats[v];
            st = ofea_solve_stats{};
            int worst = OFEA_OK;
            for (int j = 0; j < b->NR; ++j) {
                const int i = v * b->NR + j;
                st.iterations = std::max(st.iterations, iters_tot[i]);
                st.rel_residual = std::max(st.rel_residual, hrel[i]);
                int sj = hst[i];
                if (sj == OFEA_OK && !(hrel[i] <= o.rtol)) sj = OFEA_ERR_NOT_CONVERGED;
                if (sj != OFEA_OK) worst = sj;
            }
            st.status = worst;
            st.refinements = attempts;
            st.seconds = ms * 1e-3;
            st.kernel_launches = launches;
        }
    }
    if (case_stats)  // one entry per (variant, load case), load cases of a variant adjacent
        for (int i = 0; i < VJ; ++i) {
            ofea_solve_stats &st = case_stats[i];
            st = ofea_solve_stats{};
            st.status = hst[i];
            if (st.status == OFEA_OK && !(hrel[i] <= o.rtol)) st.status = OFEA_ERR_NOT_CONVERGED;
            st.iterations = iters_tot[i];
            st.rel_residual = hrel[i];
            st.refinements = attempts;
            st.seconds = ms * 1e-3;
            st.kernel_launches = launches;
        }
}

// A cooperative launch whose barrier expects one CTA more than it has: every
// wait runs out after limit_ms and the kernel reports it (*released = 0).
// Phase trace of the solver kernel: with max_phases > 0 every later launch
// records %globaltimer at its start and after each grid barrier (CTA 0,
// thread 0; at most max_phases barriers); 0 turns it off.
void batch_set_trace(ofea_batch *b, int max_phases) {
    if (max_phases < 0 || max_phases > (1 << 20)) fail(OFEA_ERR_INVALID_ARG, "batch: max_phases must be 0..2^20");
    OFEA_CUDA(cudaSetDevice(b->device));
    if (max_phases > 0) {
        b->trace.ensure((size_t)max_phases + 1);
        OFEA_CUDA(cudaMemsetAsync(b->trace.p, 0, sizeof(unsigned long long) * (max_phases + 1), b->stream));
    }
    b->trace_cap = max_phases > 0 ? max_phases + 1 : 0;
}

// Durations (ms) between consecutive records of the last traced launch, in
// barrier order; *count = how many there are (up to cap are written).
void batch_phase_times(ofea_batch *b, double *ms, int cap, int *count) {
    *count = 0;
    if (b->trace_cap == 0) fail(OFEA_ERR_STATE, "batch: tracing is off (ofea_batch_set_trace)");
    OFEA_CUDA(cudaSetDevice(b->device));
    std::vector<unsigned long long> t(b->trace_cap);
    OFEA_CUDA(cudaMemcpyAsync(t.data(), b->trace.p, sizeof(unsigned long long) * t.size(), cudaMemcpyDeviceToHost,
                              b->stream));
    OFEA_CUDA(cudaStreamSynchronize(b->stream));
    int n = 0;
    while (n + 1 < (int)t.size() && t[n] != 0 && t[n + 1] != 0) {
        if (ms && n < cap) ms[n] = (double)(t[n + 1] - t[n]) * 1e-6;
        ++n;
    }
    *count = n;
}

// One launch of the solver and one of the residual kernel whose slot copies'
// barriers expect an arrival more than they get: every wait for a copy runs
// out, nothing of the stage is read, and the kernels report it (*released = 0;
// 1: a kernel ended without the error).
void copy_probe(ofea_batch *b, int method, int limit_ms, int *released) {
    const bool mixed = method == OFEA_SOLVER_MIXED;
    batch_tuning(b, method, nullptr, nullptr, nullptr, nullptr);
    const TuneCfg t = b->tuned[method];
    cudaStream_t s = b->stream;
    *released = 0;
    for (int residual = 0; residual < 2; ++residual) {
        BArgs a = make_args(b, mixed && !residual, t, 2, 1e-8);
        a.copy_arrivals = 2;
        a.limit_ns = (unsigned long long)limit_ms * 1000000ull;
        OFEA_CUDA(cudaMemsetAsync(b->u.p, 0, sizeof(double) * b->ndof * b->NP, s));
        OFEA_CUDA(cudaMemsetAsync(b->gs.p, 0, sizeof(GridBar), s));
        if (residual) residuals(b, a, t);
        else enqueue(b, a, t, mixed);
        GridBar g{};
        OFEA_CUDA(cudaMemcpyAsync(&g, b->gs.p, sizeof(g), cudaMemcpyDeviceToHost, s));
        OFEA_CUDA(cudaStreamSynchronize(s));
        if (!g.err) *released = 1;
    }
}

void barrier_probe(ofea_ctx *c, int limit_ms, int *released) {
    DevBuf<GridBar> gs;
    DevBuf<int> out;
    gs.ensure(1);
    out.ensure(1);
    cudaStream_t s = c->stream;
    OFEA_CUDA(cudaMemsetAsync(gs.p, 0, sizeof(GridBar), s));
    OFEA_CUDA(cudaMemsetAsync(out.p, 0xff, sizeof(int), s));
    unsigned extra = 1;
    unsigned long long lim = (unsigned long long)limit_ms * 1000000ull;
    void *args[] = {(void *)&gs.p, (void *)&extra, (void *)&lim, (void *)&out.p};
    OFEA_CUDA(cudaLaunchCooperativeKernel((const void *)k_barrier_probe, dim3(c->num_sms), dim3(64), args, 0, s));
    int h = -1;
    OFEA_CUDA(cudaMemcpyAsync(&h, out.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    OFEA_CUDA(cudaStreamSynchronize(s));
    *released = h;
}

}  // namespace ofea
