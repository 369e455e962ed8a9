// The iterations of a single-matrix solve in ONE resident kernel, for
// matrices whose iteration is bound by latency and not by memory.
//
// A launch-per-phase iteration of a matrix of up to some ten thousand block
// rows spends its time on the chain launch - flag read - partial sums - a
// thread's serial walk over the 27 blocks of its row, 5 to 20 us per kernel
// whatever the size (PCG64 on 500 block rows: A 15.0 us, B 5.5 us, 28 us per
// iteration with the gaps; MIXED 62 us).  Here the
// CTAs stay: phases are separated by a grid barrier (one release-add and an
// acquire spin per CTA), every slice of 32 rows is shared by S warps that
// take its slots round-robin (so the serial walk is W / S slots, all of their
// loads in flight at once) and are summed through shared memory in a fixed
// order, and the coarse level's solve and prolongation are one phase: each
// CTA forms the few aggregates' corrections its own rows need from the dense
// inverse.  Phases per iteration: PCG64 A | B; MIXED A | B | residual |
// restriction | coarse solve + prolongation | post-smoothing.  The arithmetic
// is that of the launch-per-phase kernels of solve.cu and precond.cu; only
// the order of the sums differs.  Every sum has a fixed order: results are
// bitwise reproducible.
//
// CTA b owns the slices [b spc, (b + 1) spc), so a row's vectors are written
// by the CTA that reads them as its own rows; other CTAs' entries (the
// gathered columns, t in the restriction, c in the coarse solve) are read
// after a barrier, through plain loads: the barrier's acquire makes them
// visible, so no mutable vector may be read through the non-coherent path.
//
// Per iteration, launch-per-phase kernels before, this after (B200): PCG64
// 27.9 -> 7.6 us at 1.5k DOF, 28.7 -> 9.3 at 46k, 58.0 -> 18.4 at 139k; MIXED
// 62 -> 19.5, 66 -> 24.9, 111 -> 54 and 132 -> 98 us (288k).  What is left at
// the small end is the barriers: 2,600 to 2,900 cycles each, 2,000 more to
// drain a phase's stores, and 800 for the first load after.  Sums of a phase are
// taken under the next product where nothing needs them earlier, a CTA's own
// rows are loaded under the wait.  Measured and not used: every CTA reading
// every other's tagged partial instead of a counter (30 us against 21 at 139k
// DOF), the next step's columns or the own rows in registers across the
// product (spills: 25 against 18).
//
// Every wait is bounded (%globaltimer): on expiry the kernel sets the error
// status and every CTA returns.
#include "precond.cuh"
#include "resident.cuh"
#include "sell.cuh"

namespace ofea {

namespace {

constexpr int kResWarps = kResThreads / 32;

struct RArgs {
    int nfree, nslice, spc, S64, S16, iters, first, na, m;
    const int *sl_ptr, *scols, *sl_g;
    const double *sv64, *Dinv;
    const __nv_bfloat16 *svg;
    const float *Dinv32, *Einv;
    const int *agg_ptr;
    const float4 *agg_off, *row_off;
    double *u, *r, *q, *p0, *p1, *z;
    float *zA, *zB, *b32, *x32, *t32, *cvec;
    float wsm;
    double tol2;
    Parts P;
    Flags *fl;
    GridBar *bar;
    unsigned long long limit_ns;
};

// A warp's slice of the first round, kept in registers for the launch: where
// it starts, and the columns of its part's first step.
struct Home {
    int S, W, c0, c1;
};
__device__ __forceinline__ Home home(const int *__restrict__ sl_ptr, const int *__restrict__ scols, int slice, int lane, int k0, int k1) {
    Home h;
    h.S = __ldg(sl_ptr + slice);
    h.W = __ldg(sl_ptr + slice + 1) - h.S;
    h.c0 = k0 < h.W ? __ldg(scols + ((long)h.S + k0) * kSlice + lane) : 0;
    h.c1 = k1 < h.W ? __ldg(scols + ((long)h.S + k1) * kSlice + lane) : h.c0;
    return h;
}

// Part `part` of S of a row's product: FP64 slots part, part + S, ..., two in
// flight.
template <class XF>
__device__ __forceinline__ void part64(const Home &h, int t, int part, int S, const int *__restrict__ scols,
                                       const double *__restrict__ sv, XF x, double (&y)[3]) {
    const int *cp = scols + (long)h.S * kSlice + t;
    const double *vp = sv + (long)h.S * 9 * kSlice + t;
    y[0] = y[1] = y[2] = 0.0;
    int c0 = h.c0, c1 = h.c1;
    for (int k = part; k < h.W; k += 2 * S) {
        const bool two = k + S < h.W;
        const int k1 = two ? k + S : k;
        if (k != part) {
            c0 = __ldg(cp + (long)k * kSlice);
            c1 = __ldg(cp + (long)k1 * kSlice);
        }
        double v[2][9];
#pragma unroll
        for (int e = 0; e < 9; ++e) {
            v[0][e] = __ldg(vp + ((long)k * 9 + e) * kSlice);
            v[1][e] = two ? __ldg(vp + ((long)k1 * 9 + e) * kSlice) : 0.0;
        }
        double xv[2][3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            xv[0][i] = x(3 * c0 + i);
            xv[1][i] = x(3 * c1 + i);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 3; ++i)
                y[i] = fma(v[u][3 * i], xv[u][0], fma(v[u][3 * i + 1], xv[u][1], fma(v[u][3 * i + 2], xv[u][2], y[i])));
    }
}

// The same from the grouped BF16 copy (sell.cuh): pairs of slots part,
// part + S, ... (the slot beyond W holds zeros)
__device__ __forceinline__ void part16(const Home &h, long Gb, int t, int part, int S, const int *__restrict__ scols,
                                       const __nv_bfloat16 *__restrict__ svg, const float *x, float (&y)[3]) {
    const int *cp = scols + (long)h.S * kSlice + t;
    const unsigned *vp = reinterpret_cast<const unsigned *>(svg) + (Gb * 9 * kSlice + t) * 2;
    y[0] = y[1] = y[2] = 0.f;
    int c0 = h.c0, c1 = h.c1;
    for (int k = 2 * part; k < h.W; k += 2 * S) {
        const bool two = k + 1 < h.W;
        if (k != 2 * part) {
            c0 = __ldg(cp + (long)k * kSlice);
            c1 = __ldg(cp + (long)(two ? k + 1 : k) * kSlice);
        }
        unsigned raw[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) raw[e] = __ldg(vp + ((long)(k >> 2) * 9 + e) * kSlice * 2 + ((k >> 1) & 1));
        float xv[2][3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            xv[0][i] = x[3 * c0 + i];
            xv[1][i] = x[3 * c1 + i];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            y[i] = fmaf(__uint_as_float(raw[3 * i] << 16), xv[0][0],
                        fmaf(__uint_as_float(raw[3 * i + 1] << 16), xv[0][1],
                             fmaf(__uint_as_float(raw[3 * i + 2] << 16), xv[0][2], y[i])));
            if (two)
                y[i] = fmaf(__uint_as_float(raw[3 * i] & 0xFFFF0000u), xv[1][0],
                            fmaf(__uint_as_float(raw[3 * i + 1] & 0xFFFF0000u), xv[1][1],
                                 fmaf(__uint_as_float(raw[3 * i + 2] & 0xFFFF0000u), xv[1][2], y[i])));
        }
    }
}

// Sum of n partials by one warp (every lane returns it), fixed order.
__device__ __forceinline__ double warp_partials(const double *P, int n) {
    double s = 0.0;
    for (int i = threadIdx.x & 31; i < n; i += 32) s += P[i];
    return warp_sum(s);
}

}  // namespace

template <bool MIXED>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const RArgs a) {
    __shared__ double s_red[kResWarps * 3 * 32];
    __shared__ double s_w[2][kResWarps], s_sum[4];
    __shared__ float s_e[MIXED ? kResMaxM : 1];
    __shared__ unsigned s_touch[MIXED ? kResMaxM / 6 / 32 : 1];
    __shared__ int s_fail, s_k, s_done;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int G = gridDim.x;
    const int sl0 = blockIdx.x * a.spc, sl1 = min(a.nslice, sl0 + a.spc);
    const int row0 = sl0 * kSlice, row1 = min(a.nfree, sl1 * kSlice);
    unsigned target = 0;
    if (tid == 0) {
        s_fail = 0;
        s_done = *(volatile int *)&a.fl->done;
        s_k = *(volatile int *)&a.fl->itA;
    }
    if (MIXED)
        for (int i = tid; i < (a.na + 31) / 32; i += kResThreads) s_touch[i] = 0;
    __syncthreads();
    if (s_done) return;
    int k = s_k;
    if (MIXED) {  // the aggregates of this CTA's rows
        for (int r = row0 + tid; r < row1; r += kResThreads) {
            const int I = __float_as_int(__ldg(&a.row_off[r].w));
            atomicOr(&s_touch[I >> 5], 1u << (I & 31));
        }
    }
    // this warp's slices of the first round
    const int ng64 = kResWarps / a.S64, g64 = w / a.S64, p64 = w - g64 * a.S64;
    Home h64{0, 0, 0, 0}, h16{0, 0, 0, 0};
    long G16 = 0;
    if (g64 < ng64 && sl0 + g64 < sl1) h64 = home(a.sl_ptr, a.scols, sl0 + g64, lane, p64, p64 + a.S64);
    const int ng16 = kResWarps / a.S16, g16 = w / a.S16, p16 = w - g16 * a.S16;
    if (MIXED && g16 < ng16 && sl0 + g16 < sl1) {
        h16 = home(a.sl_ptr, a.scols, sl0 + g16, lane, 2 * p16, 2 * p16 + 1);
        G16 = __ldg(a.sl_g + sl0 + g16);
    }
    // a barrier in two steps: what a CTA needs of its own rows next is loaded
    // between them
    auto arrive = [&]() {
        target += G;
        grid_arrive(a.bar);
    };
    auto wait = [&]() { return grid_wait(a.bar, target, a.limit_ns, &s_fail); };
    auto sync = [&]() {
        arrive();
        return wait();
    };
    // this CTA's partial of one or two sums (threads' values x, y)
    auto put = [&](double x, double *Px, double y, double *Py) {
        x = warp_sum(x);
        if (Py) y = warp_sum(y);
        if (lane == 0) {
            s_w[0][w] = x;
            s_w[1][w] = y;
        }
        __syncthreads();
        if (w == 0) {
            const double sx = warp_sum(s_w[0][lane]);
            const double sy = Py ? warp_sum(s_w[1][lane]) : 0.0;
            if (lane == 0) {
                Px[blockIdx.x] = sx;
                if (Py) Py[blockIdx.x] = sy;
            }
        }
    };
    // s_sum[slot] = the sum of the CTAs' partials, by one warp; read after the
    // next block barrier (the products' own: the sums are under them)
    auto sum = [&](int slot, const double *P) {
        const double v = warp_partials(P, G);
        if (lane == 0) s_sum[slot] = v;
    };
    auto stop = [&](int status, int iters) {
        if (blockIdx.x == 0 && tid == 0) {
            a.fl->done = 1;
            a.fl->status = status;
            a.fl->iters = iters;
        }
    };
    auto timed_out = [&]() {
        if (tid == 0) {
            a.fl->done = 1;
            a.fl->status = OFEA_ERR_TIMEOUT;
        }
    };
    // y = (this CTA's rows of) K x in rounds of kResWarps / S slices; the first
    // warps, one row per lane, load pre(row) and pass it to fin(row, y, own)
    // (nothing when done() after the first block barrier: returns true)
    auto spmm64 = [&](auto x, auto pre, auto done, auto fin) {
        const int S = a.S64, ng = ng64, g = g64;
        for (int b = sl0; b < sl1; b += ng) {
            double y[3] = {0.0, 0.0, 0.0};
            if (g < ng && b + g < sl1) {
                const Home h = b == sl0 ? h64 : home(a.sl_ptr, a.scols, b + g, lane, p64, p64 + S);
                part64(h, lane, p64, S, a.scols, a.sv64, x, y);
#pragma unroll
                for (int i = 0; i < 3; ++i) s_red[(w * 3 + i) * 32 + lane] = y[i];
            }
            const int row = (b + w) * kSlice + lane;
            const bool mine = w < ng && b + w < sl1 && row < a.nfree;
            __syncthreads();
            if (b == sl0 && done()) return true;
            if (mine) {
                const auto own = pre(row);
#pragma unroll
                for (int i = 0; i < 3; ++i) y[i] = 0.0;
                for (int p = 0; p < S; ++p)
#pragma unroll
                    for (int i = 0; i < 3; ++i) y[i] += s_red[((w * S + p) * 3 + i) * 32 + lane];
                fin(row, y, own);
            }
            if (b + ng < sl1) __syncthreads();
        }
        return false;
    };
    auto spmm16 = [&](const float *x, auto pre, auto done, auto fin) {
        float *red = reinterpret_cast<float *>(s_red);
        const int S = a.S16, ng = ng16, g = g16;
        for (int b = sl0; b < sl1; b += ng) {
            float y[3] = {0.f, 0.f, 0.f};
            if (g < ng && b + g < sl1) {
                const Home h = b == sl0 ? h16 : home(a.sl_ptr, a.scols, b + g, lane, 2 * p16, 2 * p16 + 1);
                part16(h, b == sl0 ? G16 : (long)__ldg(a.sl_g + b + g), lane, p16, S, a.scols, a.svg, x, y);
#pragma unroll
                for (int i = 0; i < 3; ++i) red[(w * 3 + i) * 32 + lane] = y[i];
            }
            const int row = (b + w) * kSlice + lane;
            const bool mine = w < ng && b + w < sl1 && row < a.nfree;
            __syncthreads();
            if (b == sl0 && done()) return true;
            if (mine) {
                const auto own = pre(row);
#pragma unroll
                for (int i = 0; i < 3; ++i) y[i] = 0.f;
                for (int p = 0; p < S; ++p)
#pragma unroll
                    for (int i = 0; i < 3; ++i) y[i] += red[((w * S + p) * 3 + i) * 32 + lane];
                fin(row, y, own);
            }
            if (b + ng < sl1) __syncthreads();
        }
        return false;
    };
    struct F3 {
        float v[3];
    };
    auto f3 = [](const float *p, int row) { return F3{{p[3L * row], p[3L * row + 1], p[3L * row + 2]}}; };
    auto never = [] { return false; };
    // z_{kk+1} = M(b32), x32 = the pre-smoothed start; partials r.z_{kk+1} and
    // r.z_kk.  With check the solve stops when ||r||^2 has reached the target.
    // 0, 1: stopped, 2: a wait ran out.
    auto vcycle = [&](int kk, bool check) -> int {
        if (check && w == kResWarps - 1) sum(0, a.P.rr);
        if (spmm16(a.x32, [&](int row) { return f3(a.b32, row); }, [&] { return check && s_sum[0] <= a.tol2; },
                   [&](int row, float (&y)[3], const F3 &b) {
#pragma unroll
                       for (int i = 0; i < 3; ++i) a.t32[3L * row + i] = b.v[i] - y[i];
                   })) {
            stop(OFEA_OK, kk + 1);
            return 1;
        }
        if (!sync()) return 2;
        {  // c = Z^T t, one CTA per aggregate
            float *sh = reinterpret_cast<float *>(s_red);  // [6][warps]
            for (int I = blockIdx.x; I < a.na; I += G) {
                float acc[6] = {0, 0, 0, 0, 0, 0};
                for (int idx = __ldg(a.agg_ptr + I) + tid; idx < __ldg(a.agg_ptr + I + 1); idx += kResThreads) {
                    const float4 o = __ldg(a.agg_off + idx);
                    const int r = __float_as_int(o.w);
                    const float dx = o.x, dy = o.y, dz = o.z;
                    const float tx = a.t32[3L * r], ty = a.t32[3L * r + 1], tz = a.t32[3L * r + 2];
                    acc[0] += tx;
                    acc[1] += ty;
                    acc[2] += tz;
                    acc[3] += -dz * ty + dy * tz;
                    acc[4] += dz * tx - dx * tz;
                    acc[5] += -dy * tx + dx * ty;
                }
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    acc[q] = warp_sum(acc[q]);
                    if (lane == 0) sh[q * kResWarps + w] = acc[q];
                }
                __syncthreads();
                if (w < 6) {
                    const float v = warp_sum(sh[w * kResWarps + lane]);
                    if (lane == 0) a.cvec[6 * I + w] = v;
                }
                __syncthreads();
            }
        }
        if (!sync()) return 2;
        // e = E^-1 c for the aggregates of this CTA's rows, x += Z e
        for (int wd = 0, seen = 0; wd < (a.na + 31) / 32; ++wd) {
            unsigned bits = s_touch[wd];
            while (bits) {
                const int I = wd * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
#pragma unroll 1
                for (int q = 0; q < 6; ++q, ++seen) {
                    if (seen % kResWarps != w) continue;
                    const float *row = a.Einv + (long)(6 * I + q) * a.m;
                    float s = 0.f;
#pragma unroll 4
                    for (int j = lane; j < a.m; j += 32) s = fmaf(__ldg(row + j), a.cvec[j], s);
                    s = warp_sum(s);
                    if (lane == 0) s_e[6 * I + q] = s;
                }
            }
        }
        __syncthreads();
        for (int r = row0 + tid; r < row1; r += kResThreads) {
            const float4 o = __ldg(a.row_off + r);
            const float *e = s_e + 6 * __float_as_int(o.w);
            const float dx = o.x, dy = o.y, dz = o.z;
            a.x32[3L * r] += e[0] + dz * e[4] - dy * e[5];
            a.x32[3L * r + 1] += e[1] - dz * e[3] + dx * e[5];
            a.x32[3L * r + 2] += e[2] + dy * e[3] - dx * e[4];
        }
        if (!sync()) return 2;
        float *znew = ((kk + 1) & 1) ? a.zB : a.zA;
        const float *zold = ((kk + 1) & 1) ? a.zA : a.zB;
        double prz = 0.0, przo = 0.0;
        struct Own {
            F3 b, x, z;
            double r[3];
        };
        spmm16(a.x32,
               [&](int row) {
                   return Own{f3(a.b32, row), f3(a.x32, row), f3(zold, row), {a.r[3L * row], a.r[3L * row + 1], a.r[3L * row + 2]}};
               },
               never,
               [&](int row, float (&y)[3], const Own &n) {
                   float d[3], o[3];
#pragma unroll
                   for (int i = 0; i < 3; ++i) d[i] = n.b.v[i] - y[i];
                   block3_apply(a.Dinv32 + 9L * row, d, o);
#pragma unroll
                   for (int i = 0; i < 3; ++i) {
                       const float zn = fmaf(a.wsm, o[i], n.x.v[i]);
                       prz += n.r[i] * (double)zn;
                       przo += n.r[i] * (double)n.z.v[i];
                       znew[3L * row + i] = zn;
                   }
               });
        put(prz, ((kk + 1) & 1) ? a.P.rz1 : a.P.rz0, przo, a.P.rzo);
        return sync() ? 0 : 2;
    };
    if (MIXED) {
        if (a.first) {
            const int e = vcycle(k - 1, false);
            if (e == 2) timed_out();
            if (e) return;
        }
    }
    for (int it = 0; it < a.iters; ++it, ++k) {
        double *Pcur = (k & 1) ? a.P.rz1 : a.P.rz0, *Pother = (k & 1) ? a.P.rz0 : a.P.rz1;
        // the sums of the phases before, by the last warps
        if (w == kResWarps - 1) sum(0, Pcur);
        else if (w == kResWarps - 2 && k > 0) sum(1, Pother);
        else if (w == kResWarps - 3) sum(2, MIXED ? a.P.rzo : a.P.rr);
        const double *pold = (k & 1) ? a.p1 : a.p0;
        double *pnew = (k & 1) ? a.p0 : a.p1;
        const float *zf = (k & 1) ? a.zB : a.zA;
        const double *zd = a.z;
        double ppq = 0.0, beta = 0.0;
        auto zat = [&](long d) { return MIXED ? (double)zf[d] : zd[d]; };
        struct Own {
            double p[3], z[3], q[3];
        };
        if (spmm64(zat,
                   [&](int row) {
                       Own o;
#pragma unroll
                       for (int i = 0; i < 3; ++i) {
                           o.p[i] = pold[3L * row + i];
                           o.z[i] = zat(3L * row + i);
                           o.q[i] = a.q[3L * row + i];
                       }
                       return o;
                   },
                   [&] {
                       if (k > 0) beta = (MIXED ? s_sum[0] - s_sum[2] : s_sum[0]) / s_sum[1];
                       return !MIXED && s_sum[2] <= a.tol2;
                   },
                   [&](int row, double (&y)[3], const Own &o) {
#pragma unroll
                       for (int i = 0; i < 3; ++i) {
                           const double pn = fma(beta, o.p[i], o.z[i]);
                           const double qn = fma(beta, o.q[i], y[i]);  // K p = K z + beta K p_old
                           pnew[3L * row + i] = pn;
                           a.q[3L * row + i] = qn;
                           ppq += pn * qn;
                       }
                   })) {
            stop(OFEA_OK, k);
            return;
        }
        put(ppq, a.P.pq, 0.0, nullptr);
        arrive();
        // B: alpha, u, r, and the block-Jacobi step.  The rows are this CTA's
        // own: the first one's entries are loaded under the wait.
        struct Row {
            double u[3], r[3], p[3], q[3];
        };
        auto load = [&](int i) {
            Row t;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                t.u[c] = a.u[3L * i + c];
                t.r[c] = a.r[3L * i + c];
                t.p[c] = pnew[3L * i + c];
                t.q[c] = a.q[3L * i + c];
            }
            return t;
        };
        int i = row0 + tid;
        Row cur = load(i < row1 ? i : row0);
        if (!wait()) {
            timed_out();
            return;
        }
        if (w == 0) sum(3, a.P.pq);
        __syncthreads();
        const double pq = s_sum[3], rz = s_sum[0];
        if (!(pq > 0.0) || !isfinite(pq)) {
            stop(OFEA_ERR_BREAKDOWN, k);
            return;
        }
        const double alpha = rz / pq;
        double prr = 0.0, prz = 0.0;
        while (i < row1) {
            double rv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                a.u[3L * i + c] = fma(alpha, cur.p[c], cur.u[c]);
                rv[c] = fma(-alpha, cur.q[c], cur.r[c]);
                a.r[3L * i + c] = rv[c];
                prr += rv[c] * rv[c];
            }
            if (MIXED) {
                float b[3] = {(float)rv[0], (float)rv[1], (float)rv[2]}, x[3];
                block3_apply(a.Dinv32 + 9L * i, b, x);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    a.b32[3L * i + c] = b[c];
                    a.x32[3L * i + c] = a.wsm * x[c];
                }
            } else {
                double zz[3];
                block3_apply(a.Dinv + 9L * i, rv, zz);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    a.z[3L * i + c] = zz[c];
                    prz += rv[c] * zz[c];
                }
            }
            i += kResThreads;
            if (i < row1) cur = load(i);
        }
        if (MIXED) put(prr, a.P.rr, 0.0, nullptr);
        else put(prr, a.P.rr, prz, Pother);
        if (!sync()) {
            timed_out();
            return;
        }
        if (MIXED) {
            const int e = vcycle(k, true);
            if (e == 2) timed_out();
            if (e) return;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.fl->itA = k;
        a.fl->iters = k;
    }
}

// ------------------------------------------------------------------- host --

bool resident_plan(const ofea_ctx *c, bool mixed, ResidentPlan &p) {
    const int nslice = (c->nfree + kSlice - 1) / kSlice;
    // MIXED: up to 3,500 slices (336k DOF), beyond which the launch-per-phase
    // kernels' wider grids win (288k DOF: 98 us per iteration here, 132
    // there; 467k DOF: 191 here, 164 there, the coarse solve of 930 unknowns
    // repeated by every CTA); PCG64 with the stored K is the faster one at
    // every size measured (706k DOF 105 against 122 us).
    if (nslice < 1) return false;
    if (mixed && (nslice > 3500 || c->coarse.m > kResMaxM)) return false;
    p.spc = (nslice + c->num_sms - 1) / c->num_sms;
    p.G = (nslice + p.spc - 1) / p.spc;
    // warps per slice: the fewest serial steps over all rounds, a round's own
    // latency counted as two steps
    const int W = (int)std::max<long long>(1, c->sell_len / nslice);
    auto pick = [&](int units) {
        int best = 1;
        long cost = -1;
        for (int S = 1; S <= 32; ++S) {
            const int ng = kResWarps / S, rounds = (p.spc + ng - 1) / ng;
            const long t = (long)rounds * ((units + S - 1) / S + 2);
            if (cost < 0 || t < cost) {
                cost = t;
                best = S;
            }
        }
        return best;
    };
    p.S64 = pick((W + 1) / 2);  // two slots in flight per step
    p.S16 = pick((W + 1) / 2);
    return true;
}

void resident_iterations(ofea_ctx *c, const ResidentPlan &p, bool mixed, const Parts &P, Flags *fl, double *d_u,
                         float wsm, double tol2, int iters, int first) {
    SolverWork &w = c->w;
    const Coarse &C = c->coarse;
    RArgs a{};
    a.nfree = c->nfree;
    a.nslice = (c->nfree + kSlice - 1) / kSlice;
    a.spc = p.spc;
    a.S64 = p.S64;
    a.S16 = p.S16;
    a.iters = iters;
    a.first = first;
    a.sl_ptr = c->sl_ptr.p;
    a.scols = c->scols.p;
    a.sl_g = c->sl_g.p;
    a.sv64 = c->sv64.p;
    a.svg = c->sv16g.p;
    a.Dinv = c->Dinv.p;
    a.Dinv32 = c->Dinv32.p;
    a.u = d_u;
    a.r = w.r.p;
    a.q = w.q.p;
    a.p0 = w.p0.p;
    a.p1 = w.p1.p;
    a.z = w.z.p;
    if (mixed) {
        a.na = C.na;
        a.m = C.m;
        a.Einv = C.Einv32.p;
        a.agg_ptr = C.agg_ptr.p;
        a.agg_off = reinterpret_cast<const float4 *>(C.agg_off.p);
        a.row_off = reinterpret_cast<const float4 *>(C.row_off.p);
        a.zA = w.z32a.p;
        a.zB = w.z32b.p;
        a.b32 = w.b32.p;
        a.x32 = w.x32.p;
        a.t32 = w.t32.p;
        a.cvec = C.cvec.p;
    }
    a.wsm = wsm;
    a.tol2 = tol2;
    a.P = P;
    a.fl = fl;
    w.bar.ensure(2);
    a.bar = reinterpret_cast<GridBar *>(w.bar.p);
    a.limit_ns = 5000000000ull;  // 5 s: far above any phase
    OFEA_CUDA(cudaMemsetAsync(w.bar.p, 0, sizeof(GridBar), c->stream));
    void *args[] = {(void *)&a};
    const void *fn = mixed ? (const void *)k_resident<true> : (const void *)k_resident<false>;
    OFEA_CUDA(cudaLaunchCooperativeKernel(fn, dim3(p.G), dim3(kResThreads), args, 0, c->stream));
}

}  // namespace ofea
