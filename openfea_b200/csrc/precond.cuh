// Coarse space and V-cycle of the two-level preconditioner (precond.cu).
#pragma once
#include "ofea_internal.cuh"

namespace ofea {

// A V-cycle kernel launched among a solve's iterations returns at once when
// the solve has stopped (the iterations a chunk runs past convergence cost
// only their launches).  stop is null outside a solve.  Read once per CTA and
// broadcast: every thread takes the same path before any barrier.
__device__ __forceinline__ bool vc_stopped(const int *stop) {
    if (stop == nullptr) return false;
    __shared__ int s_stop;
    if (threadIdx.x == 0) s_stop = *(volatile const int *)stop;
    __syncthreads();
    return s_stop != 0;
}

// Z_I^T v over the rows [idx, end) of an aggregate in steps, added to a: off
// gives each row's offset from the centroid and the row.
__device__ __forceinline__ void modes_sum(int idx, int end, int step, const float4 *__restrict__ off, const float *v,
                                          float (&a)[6]) {
    for (; idx < end; idx += step) {
        const float4 o = __ldg(off + idx);
        const int r = __float_as_int(o.w);
        const float dx = o.x, dy = o.y, dz = o.z;
        const float tx = v[3L * r], ty = v[3L * r + 1], tz = v[3L * r + 2];
        a[0] += tx;
        a[1] += ty;
        a[2] += tz;
        a[3] += -dz * ty + dy * tz;  // (e_x x d) . t
        a[4] += dz * tx - dx * tz;   // (e_y x d) . t
        a[5] += -dy * tx + dx * ty;  // (e_z x d) . t
    }
}
// Entry e of K Z, W[6 c + l], in 18 planes.
__device__ __forceinline__ void mode_entry(long e, long n, const float *__restrict__ val, float (&W)[18]) {
#pragma unroll
    for (int q = 0; q < 18; ++q) W[q] = __ldg(val + q * n + e);
}
// K Z as the row kernels read it: entries in row order.
struct RowModes {
    const float4 *off;  // a row's offset from its aggregate's centroid, the aggregate
    const int *rptr, *agg;
    const float *val;
    long n;
    // (Z e)_r for e of six values per aggregate
    __device__ __forceinline__ void modes(int r, const float *e, float (&z)[3]) const {
        const float4 o = __ldg(off + r);
        const float *q = e + 6 * __float_as_int(o.w);
        z[0] = q[0] + o.z * q[4] - o.y * q[5];
        z[1] = q[1] - o.z * q[3] + o.x * q[5];
        z[2] = q[2] + o.y * q[3] - o.x * q[4];
    }
    // entry t's part of K Z e
    __device__ __forceinline__ void entry(int t, const float *e, float (&kz)[3]) const {
        const float *v = e + 6 * __ldg(agg + t);
        float W[18];
        mode_entry(t, n, val, W);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            kz[c] = W[6 * c] * v[0];
#pragma unroll
            for (int l = 1; l < 6; ++l) kz[c] = fmaf(W[6 * c + l], v[l], kz[c]);
        }
    }
    // (K Z e)_r
    __device__ __forceinline__ void row(int r, const float *e, float (&kz)[3]) const {
        kz[0] = kz[1] = kz[2] = 0.f;
        for (int t = __ldg(rptr + r); t < __ldg(rptr + r + 1); ++t) {
            float k[3];
            entry(t, e, k);
#pragma unroll
            for (int c = 0; c < 3; ++c) kz[c] += k[c];
        }
    }
};
inline RowModes row_modes(const Coarse &C) {
    return {reinterpret_cast<const float4 *>(C.row_off.p), C.md_rptr.p, C.md_ragg.p, C.md_rval.p, C.md_n};
}
// One entry of K Z: a -= W^T x.
__device__ __forceinline__ void entry_sub(long e, long n, const float *__restrict__ val, float x, float y, float z, float (&a)[6]) {
    float W[18];
    mode_entry(e, n, val, W);
#pragma unroll
    for (int l = 0; l < 6; ++l) a[l] -= fmaf(W[l], x, fmaf(W[6 + l], y, W[12 + l] * z));
}
__device__ __forceinline__ void entries_sum(int e, int end, int step, const int *__restrict__ row, const float *__restrict__ val,
                                            long n, const float *x, float (&a)[6]) {
    for (; e < end; e += step) {
        const long r = 3L * __ldg(row + e);
        entry_sub(e, n, val, x[r], x[r + 1], x[r + 2], a);
    }
}

void build_aggregation(ofea_ctx *c, int target_nodes);
void build_aggregation_fine(ofea_ctx *c);
// Aggregation (once per mesh), E = Z^T K Z, its inverse and lambda_max(D^-1 K)
// (once per K).
void setup_coarse(ofea_ctx *c, int target_nodes);
// The same in parts: the aggregation only; a zeroed dense E to fill (returns
// it); inversion, FP32 copy and lambda_max of a filled E.
void setup_coarse_geometry(ofea_ctx *c, int target_nodes);
double *coarse_begin_E(ofea_ctx *c);
void coarse_finish(ofea_ctx *c);
// Damping weight of the block-Jacobi smoother (needs setup_coarse's lmax).
float smoother_weight(const ofea_ctx *c, double damping);
// omega lmax of the single-matrix solves and of the batched solver, each the
// value that took the fewest outer iterations on its workload: the 1.56M-DOF
// cantilever, LEARNED / MIXED, 1.3: 51 / 69, 1.4: 51 / 67, 1.5: 51 / 65,
// 1.6: 52 / 64, 1.76: 56 / 71, 1.9: MIXED does not converge; the 64 SIMP
// variants of the batched reanalysis, 1.4: 86, 1.5: 83, 1.6: 81, 1.76: 78.
constexpr double kSmootherDamping = 1.5;
constexpr double kBatchSmootherDamping = 1.76;
// x += Z E^-1 Z^T t  (FP32 vectors of n entries)
// evec = E^-1 cvec (FP32 GEMV with the coarse level's inverse)
void coarse_gemv(ofea_ctx *c, const float *cvec, float *evec);
// Einv32 = the dense FP32 inverse of E (formed from the factor when the
// coarse solve is factored); for the batched solver, which applies it densely.
void coarse_dense_inverse(ofea_ctx *c);
void coarse_correct(ofea_ctx *c, const float *t, float *x);
// t = b - K32 x
void vc_resid(ofea_ctx *c, const float *b, const float *x, float *t);
// K Z of a level, current for K: the restriction c = Z^T b - (K Z)^T x
// (restrict_modes) and the post-smoothing's K Z e take the place of a product
// with K.  False where the residual is formed instead (K not the linear
// stiffness of a mesh, or no memory for it).  solver_modes: the same for a single
// solve, only where it is the faster of the two; count_modes: the level's
// entries (-1: none), before anything else of it is built.
bool ensure_modes(ofea_ctx *c, Coarse &C);
bool solver_modes(ofea_ctx *c, Coarse &C);
long count_modes(ofea_ctx *c, Coarse &C);
void restrict_modes(ofea_ctx *c, const Coarse &C, const float *b, const float *x, float *cvec);
// Level-generic pieces (also used by the learned level):
// cvec = Z^T t, x += Z g, and the Galerkin blocks of Z^T K Z into C.part
// ([aggregate][chunk][27 neighbour slots][6 x 6], chunks summed by the caller).
void restrict_level(ofea_ctx *c, const Coarse &C, const float *t, float *cvec);
void prolong_level(ofea_ctx *c, const Coarse &C, const float *g, float *x);
int galerkin_chunks(const ofea_ctx *c, const Coarse &C);
void coarse_E_partials(ofea_ctx *c, Coarse &C, int nchunk);

}  // namespace ofea
