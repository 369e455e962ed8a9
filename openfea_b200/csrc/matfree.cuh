// K x of a linear C3D8 mesh from its elements (matfree.cu).
#pragma once
#include "ofea_internal.cuh"
#include "solver_common.cuh"

namespace ofea {

constexpr double kHexForceOps = 1250;  // FP64 operations of one element's forces

// Whether K is the linear stiffness of a mesh of C3D8 elements alone, so that
// its products can be formed from the elements.
bool matfree_possible(const ofea_ctx *c);
// The same, and the mesh's tables are there: builds them on first use.
bool matfree_ready(ofea_ctx *c);

// Element forces of the free-DOF vector x, FP64: xA or xB by the parity of
// fl->itA (or x); the launch returns at once when the solve has stopped.
void matfree_forces(ofea_ctx *c, const float *xA, const float *xB, const Flags *fl);
void matfree_forces(ofea_ctx *c, const double *x, const Flags *fl);

// A row's sum of the element forces: entries [k * nfree + r] of the gather
// list name a local node and an element (-1: none).
struct MatfreeRows {
    static constexpr int kCtas = 4;  // 64 registers: a row's loads in flight together
    int nfree, width;
    long ne;
    const int *list;
    const double *fe;
    // f(r, y, pre(r)) for each of this thread's rows r; pre's loads are issued
    // with the list's
    template <class XF, class Pre, class F>
    __device__ __forceinline__ void rows(int, XF, Pre pre, F f) const {
        for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nfree; r += gridDim.x * blockDim.x) {
            const auto own = pre(r);
            double y[3] = {0.0, 0.0, 0.0};
            for (int k0 = 0; k0 < width; k0 += 4) {
                int p[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) p[u] = k0 + u < width ? __ldg(list + (long)(k0 + u) * nfree + r) : -1;
                double v[4][3];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[u][c] = p[u] >= 0 ? fe[(3L * (p[u] & 7) + c) * ne + (p[u] >> 3)] : 0.0;
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int c = 0; c < 3; ++c) y[c] += v[u][c];
                if (p[3] < 0) break;  // the entries come first
            }
            f(r, y, own);
        }
    }
};
MatfreeRows matfree_rows(const ofea_ctx *c);

}  // namespace ofea
