// K x of a linear C3D8 mesh without K: the element forces of x, formed from
// the node coordinates and moduli, then summed per row.
//
// The assembled product streams 76/9 bytes per stored value (27 blocks, 2 KB,
// per row) and is bound by HBM; the elements themselves are 24 bytes per node
// and 40 per element.  One thread forms one element's 24 forces with about
// 1,250 FP64 operations: the trilinear fields' 7 difference coefficients per
// component (a Hadamard transform of the nodal values), their gradients at
// the 8 Gauss points from those by fused multiply-adds, at each point the
// stress of the displacement gradient and its product with the inverse
// Jacobian's rows (one reciprocal per point), and the transposed transforms
// back to the nodes.  It is the same 2x2x2 integration as the assembly's
// (src/Elements/C3D8_Gauss.cpp:19-107), in another order of operations.
//
// Forces are written by planes (component of a local node) x element, so a
// warp's stores are contiguous.  Elements that stand on one another (an
// element's nodes 5-8 are the next one's 1-4, the usual numbering along a
// line) first pass their top forces to the next lane, which halves what is
// written and read back: a warp takes 31 elements and forms the one before
// them again in its first lane, so that no chain breaks between warps and an
// inner row reads four entries.  A row sums its entries of the gather list in
// a fixed order: no atomics, bitwise reproducible.
//
// On 500,000 elements (1.56M DOF): forces 64 us, row sums with the vector
// update 37 us, against 170-200 us of the stored product (1.07 GB).  The
// forces are bound by the FP64 pipe (38 us at its measured 58 operations per
// clock and SM) and, with 8 warps per SM, by the latency of their gathers.
#include <algorithm>

#include "matfree.cuh"

namespace ofea {

namespace {

constexpr int kMfBlock = 128;

__device__ __forceinline__ void load8(const int *__restrict__ p, long e, int (&n)[8]) {
    const int4 lo = __ldg(reinterpret_cast<const int4 *>(p) + 2 * e), hi = __ldg(reinterpret_cast<const int4 *>(p) + 2 * e + 1);
    n[0] = lo.x;
    n[1] = lo.y;
    n[2] = lo.z;
    n[3] = lo.w;
    n[4] = hi.x;
    n[5] = hi.y;
    n[6] = hi.z;
    n[7] = hi.w;
}

// Coefficients of the trilinear field with nodal values v: 8 d/dr etc. of its
// monomials r, s, t, rs, rt, st, rst (node order src/Elements/C3D8_Gauss.cpp:27-52).
struct Field {
    double r, s, t, rs, rt, st, rst;
};
__device__ __forceinline__ Field to_field(const double (&v)[8]) {
    double p[4], d[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        p[a] = v[a + 4] + v[a];
        d[a] = v[a + 4] - v[a];
    }
    const double pa = p[2] - p[0], pb = p[1] - p[3], da = d[2] - d[0], db = d[1] - d[3], de = d[0] + d[2], df = d[1] + d[3];
    return {pa + pb, pa - pb, de + df, (p[0] + p[2]) - (p[1] + p[3]), da + db, da - db, de - df};
}
// The transposed map: nodal sums from the coefficients' sums.
__device__ __forceinline__ void to_nodes(const Field &f, double (&v)[8]) {
    const double m = f.r + f.s, l = f.r - f.s, u = f.t + f.rst, w = f.t - f.rst, x = f.rt + f.st, y = f.rt - f.st;
    const double p[4] = {f.rs - m, l - f.rs, f.rs + m, -(l + f.rs)}, q[4] = {u - x, w + y, u + x, w - y};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        v[a] = p[a] - q[a];
        v[a + 4] = p[a] + q[a];
    }
}

__device__ __forceinline__ void cross(const double (&a)[3], const double (&b)[3], double (&o)[3]) {
    o[0] = a[1] * b[2] - a[2] * b[1];
    o[1] = a[2] * b[0] - a[0] * b[2];
    o[2] = a[0] * b[1] - a[1] * b[0];
}

// Forces of one element: lam and mu already divided by 512 (the coefficients
// are 8 times the derivatives).
__device__ __forceinline__ void element_forces(const Field (&X)[3], const Field (&U)[3], double lam, double mu, Field (&F)[3]) {
    const double g = 0.57735026918962576451;  // 1 / sqrt(3)
#pragma unroll
    for (int i = 0; i < 3; ++i) F[i] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int it = 0; it < 2; ++it) {
        const double gt = it ? g : -g;
        double br[2][3], bs[2][3], sl[2][3];  // base of d/dr, d/ds and their common slope, of X and U
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            br[0][i] = fma(gt, X[i].rt, X[i].r);
            bs[0][i] = fma(gt, X[i].st, X[i].s);
            sl[0][i] = fma(gt, X[i].rst, X[i].rs);
            br[1][i] = fma(gt, U[i].rt, U[i].r);
            bs[1][i] = fma(gt, U[i].st, U[i].s);
            sl[1][i] = fma(gt, U[i].rst, U[i].rs);
        }
        double Sr[2][3] = {}, Ss[3] = {}, Ds[3] = {};
#pragma unroll
        for (int ir = 0; ir < 2; ++ir) {
            const double gr = ir ? g : -g;
            double Ta[3] = {}, Tb[3] = {}, Sk[3] = {};
#pragma unroll
            for (int is = 0; is < 2; ++is) {
                const double gs = is ? g : -g;
                double Xr[3], Xs[3], Xt[3], Ur[3], Us[3], Ut[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    Xr[i] = fma(gs, sl[0][i], br[0][i]);
                    Xs[i] = fma(gr, sl[0][i], bs[0][i]);
                    Xt[i] = fma(gs, fma(gr, X[i].rst, X[i].st), fma(gr, X[i].rt, X[i].t));
                    Ur[i] = fma(gs, sl[1][i], br[1][i]);
                    Us[i] = fma(gr, sl[1][i], bs[1][i]);
                    Ut[i] = fma(gs, fma(gr, U[i].rst, U[i].st), fma(gr, U[i].rt, U[i].t));
                }
                double cr[3], cs[3], ct[3];
                cross(Xs, Xt, cr);
                cross(Xt, Xr, cs);
                cross(Xr, Xs, ct);
                const double id = 1.0 / (Xr[0] * cr[0] + Xr[1] * cr[1] + Xr[2] * cr[2]);
                double G[3][3];  // det x displacement gradient
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int k = 0; k < 3; ++k) G[i][k] = fma(Ur[i], cr[k], fma(Us[i], cs[k], Ut[i] * ct[k]));
                const double l = lam * id, m = mu * id, m2 = m + m;
                const double lt = l * (G[0][0] + G[1][1] + G[2][2]);
                double s[3][3];
                s[0][0] = fma(m2, G[0][0], lt);
                s[1][1] = fma(m2, G[1][1], lt);
                s[2][2] = fma(m2, G[2][2], lt);
                s[0][1] = s[1][0] = m * (G[0][1] + G[1][0]);
                s[1][2] = s[2][1] = m * (G[1][2] + G[2][1]);
                s[0][2] = s[2][0] = m * (G[0][2] + G[2][0]);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const double pr = fma(s[i][0], cr[0], fma(s[i][1], cr[1], s[i][2] * cr[2]));
                    const double ps = fma(s[i][0], cs[0], fma(s[i][1], cs[1], s[i][2] * cs[2]));
                    const double pt = fma(s[i][0], ct[0], fma(s[i][1], ct[1], s[i][2] * ct[2]));
                    Sr[is][i] += pr;
                    Sk[i] += ps;
                    Ta[i] += pt;
                    Tb[i] = is ? Tb[i] + pt : Tb[i] - pt;
                }
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                F[i].t += Ta[i];
                F[i].rt = fma(gr, Ta[i], F[i].rt);
                const double gb = g * Tb[i];
                F[i].st += gb;
                F[i].rst = fma(gr, gb, F[i].rst);
                Ss[i] += Sk[i];
                Ds[i] = ir ? Ds[i] + Sk[i] : Ds[i] - Sk[i];
            }
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double sr = Sr[0][i] + Sr[1][i], d = g * ((Sr[1][i] - Sr[0][i]) + Ds[i]);
            F[i].r += sr;
            F[i].rt = fma(gt, sr, F[i].rt);
            F[i].s += Ss[i];
            F[i].st = fma(gt, Ss[i], F[i].st);
            F[i].rs += d;
            F[i].rst = fma(gt, d, F[i].rst);
        }
    }
}

// 255 registers and 8 warps per SM: held to fewer registers it spills (12
// warps 79 us, 16 warps 118 us against 62 us on 500,000 elements).
template <class XV>
__global__ void __launch_bounds__(kMfBlock, 2) k_hex_forces(int ne8, const int *__restrict__ topo8, const int *__restrict__ rows8,
                                                            const unsigned char *__restrict__ link, const double *__restrict__ xyz,
                                                            const double *__restrict__ E8, double cl, double cm,
                                                            const XV *__restrict__ xA, const XV *__restrict__ xB,
                                                            double *__restrict__ fe, const Flags *fl) {
    if (*(volatile const int *)&fl->done) return;
    const XV *x = (*(volatile const int *)&fl->itA & 1) ? xB : xA;
    const int lane = threadIdx.x & 31;
    const long e = (blockIdx.x * (long)(kMfBlock / 32) + (threadIdx.x >> 5)) * 31 + lane - 1;
    const long ec = max(0L, min(e, (long)ne8 - 1));
    Field X[3], U[3], F[3];
    {
        int n[8], f[8];
        load8(topo8, ec, n);
        load8(rows8, ec, f);
        double u[3][8];
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int i = 0; i < 3; ++i) u[i][a] = f[a] >= 0 ? (double)x[3L * f[a] + i] : 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            double v[8];
#pragma unroll
            for (int a = 0; a < 8; ++a) v[a] = __ldg(xyz + 3L * n[a] + i);
            X[i] = to_field(v);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) U[i] = to_field(u[i]);
    }
    const double E = __ldg(E8 + ec);
    const bool below = lane > 0 && ec > 0 && link[ec - 1], top = !link[ec];
    element_forces(X, U, E * cl, E * cm, F);
    const bool write = lane > 0 && e < ne8;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        double v[8];
        to_nodes(F[i], v);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const double up = __shfl_up_sync(0xffffffffu, v[a + 4], 1);
            if (below) v[a] += up;
        }
        if (write) {
#pragma unroll
            for (int a = 0; a < 4; ++a) fe[(3L * a + i) * ne8 + e] = v[a];
            if (top)
#pragma unroll
                for (int a = 4; a < 8; ++a) fe[(3L * a + i) * ne8 + e] = v[a];
        }
    }
}

// Once per mesh: the free row of every element node (-1: fixed), and whether
// the next element stands on this one.
__global__ void k_mf_elements(int ne8, const int *__restrict__ topo8, const int *__restrict__ free_map, int *__restrict__ rows8,
                              unsigned char *__restrict__ link) {
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < ne8; e += (long)gridDim.x * blockDim.x) {
        bool l = e + 1 < ne8;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            rows8[8 * e + a] = free_map[topo8[8 * e + a]];
            if (a < 4) l = l && topo8[8 * (e + 1) + a] == topo8[8 * e + a + 4];
        }
        link[e] = l;
    }
}

// Gather list: the row's incidences whose forces are written, in ascending
// element order, then -1.  Counts the longest row first (list null).
__global__ void k_mf_list(int nfree, const int *__restrict__ node_of_free, const int *__restrict__ inc_ptr,
                          const int *__restrict__ inc, const unsigned char *__restrict__ link, int width, int *__restrict__ list,
                          int *__restrict__ longest) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nfree; r += gridDim.x * blockDim.x) {
        const int node = node_of_free[r];
        int k = 0;
        for (int t = inc_ptr[node]; t < inc_ptr[node + 1]; ++t) {
            const int p = inc[t];
            if ((p & 7) >= 4 && link[p >> 3]) continue;
            if (list) list[(long)k * nfree + r] = p;
            ++k;
        }
        if (list)
            for (; k < width; ++k) list[(long)k * nfree + r] = -1;
        else
            atomicMax(longest, k);
    }
}

template <class XV>
void forces(ofea_ctx *c, const XV *xA, const XV *xB, const Flags *fl) {
    // lam = E cl, mu = E cm (build_cons_mat, src/Elements/C3D8.cpp:23-27), over 512
    const double nu = c->nu, fac = (1.0 - nu) / ((1.0 + nu) * (1.0 - 2.0 * nu));
    const double cl = fac * nu / (1.0 - nu) / 512.0, cm = fac * (1.0 - 2.0 * nu) / (2.0 * (1.0 - nu)) / 512.0;
    const int per_cta = kMfBlock / 32 * 31;
    k_hex_forces<XV><<<(c->ne8 + per_cta - 1) / per_cta, kMfBlock, 0, c->stream>>>(
        c->ne8, c->topo8.p, c->mf_rows.p, c->mf_link.p, c->xyz.p, c->E8.p, cl, cm, xA, xB, c->mf_fe.p, fl);
    OFEA_CHECK_LAUNCH();
}

}  // namespace

// False when a node lies in too many elements for a gather list of that width
// on every row (a fan; 4 to 8 are usual).
constexpr int kMfMaxWidth = 16;
static bool build_tables(ofea_ctx *c) {
    cudaStream_t s = c->stream;
    c->mf_link.ensure(c->ne8);
    c->mf_rows.ensure(8 * (size_t)c->ne8);
    k_mf_elements<<<grid_for(c, c->ne8, kBlock), kBlock, 0, s>>>(c->ne8, c->topo8.p, c->free_map.p, c->mf_rows.p,
                                                                 c->mf_link.p);
    OFEA_CHECK_LAUNCH();
    OFEA_CUDA(cudaMemsetAsync(c->err_flag.p, 0, sizeof(int), s));
    const int g = grid_for(c, c->nfree, kBlock);
    k_mf_list<<<g, kBlock, 0, s>>>(c->nfree, c->node_of_free.p, c->inc_ptr.p, c->inc.p, c->mf_link.p, 0, nullptr, c->err_flag.p);
    OFEA_CHECK_LAUNCH();
    OFEA_CUDA(cudaMemcpyAsync(c->herr.p, c->err_flag.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    OFEA_CUDA(cudaStreamSynchronize(s));
    c->mf_width = c->herr.p[0];
    if (c->mf_width > kMfMaxWidth) return false;
    c->mf_list.ensure((size_t)std::max(c->mf_width, 1) * c->nfree);
    k_mf_list<<<g, kBlock, 0, s>>>(c->nfree, c->node_of_free.p, c->inc_ptr.p, c->inc.p, c->mf_link.p, c->mf_width,
                                   c->mf_list.p, nullptr);
    OFEA_CHECK_LAUNCH();
    c->mf_fe.ensure(24 * (size_t)c->ne8);
    return true;
}

// mf_state: 0 not built, 1 built, -1 not for this mesh or no memory for it
// (the stored K is used, until the next pattern; nothing of the tables is kept).
bool matfree_possible(const ofea_ctx *c) {
    return !c->matrix_only && c->ne4 == 0 && c->ne8 != 0 && c->K_linear && c->mf_state >= 0;
}
bool matfree_ready(ofea_ctx *c) {
    if (!matfree_possible(c)) return false;
    if (c->mf_state == 0) {
        try {
            c->mf_state = build_tables(c) ? 1 : -1;
        } catch (const Failure &e) {
            if (e.code != OFEA_ERR_OOM) throw;
            c->mf_state = -1;
        }
        if (c->mf_state < 0) {
            c->mf_link.release();
            c->mf_rows.release();
            c->mf_list.release();
            c->mf_fe.release();
        }
    }
    return c->mf_state == 1;
}

void matfree_forces(ofea_ctx *c, const float *xA, const float *xB, const Flags *fl) { forces(c, xA, xB, fl); }
void matfree_forces(ofea_ctx *c, const double *x, const Flags *fl) { forces(c, x, x, fl); }
MatfreeRows matfree_rows(const ofea_ctx *c) {
    return {c->nfree, c->mf_width, (long)c->ne8, c->mf_list.p, c->mf_fe.p};
}

}  // namespace ofea
