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
// inverse.  Phases per iteration: PCG64 A | B; MIXED with K Z A | B | product
// K x0 and restriction | coarse solve and z, without it A | B | residual |
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
// 67 -> 17.8 (14.5k), 66 -> 21.6, 111 -> 46.5 and 132 -> 85 us (288k); without
// K Z 22.1, 24.9, 54 and 98.  What is left at
// the small end is the barriers: 2,600 to 2,900 cycles each, 2,000 more to
// drain a phase's stores, and 800 for the first load after.  Sums of a phase are
// taken under the next product where nothing needs them earlier, a CTA's own
// rows are loaded under the wait.  Measured and not used: every CTA reading
// every other's tagged partial instead of a counter (30 us against 21 at 139k
// DOF), the next step's columns or the own rows in registers across the
// product (spills: 25 against 18).
//
// Every wait of this kernel is bounded (%globaltimer): on expiry it sets the
// error status and every CTA returns.  The cluster form below waits at the
// hardware's cluster barrier only: no spin on memory; its CTAs are
// resident together and all pass the same barriers, their exits decided by
// values that every CTA sums alike.
#include <map>
#include <mutex>
#include <type_traits>

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
    const int *md_ptr, *md_row;  // K Z by aggregate (null: the residual is restricted)
    const float *md_val;
    RowModes md;                 // K Z by row
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
    __shared__ uint16_t s_list[MIXED ? kResMaxM / 6 : 1];
    __shared__ int s_ntouch;
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
    if (MIXED) {  // the aggregates of this CTA's rows and of their entries
        for (int r = row0 + tid; r < row1; r += kResThreads) {
            const int I = __float_as_int(__ldg(&a.row_off[r].w));
            atomicOr(&s_touch[I >> 5], 1u << (I & 31));
            if (a.md_ptr)
                for (int t = __ldg(a.md.rptr + r); t < __ldg(a.md.rptr + r + 1); ++t) {
                    const int J = __ldg(a.md.agg + t);
                    atomicOr(&s_touch[J >> 5], 1u << (J & 31));
                }
        }
        __syncthreads();
        if (w == 0) {  // as a list, ascending
            int at = 0;
            for (int i = 0; i < (a.na + 31) / 32; ++i) {
                const unsigned m = s_touch[i];
                if (m >> lane & 1u) s_list[at + __popc(m & ((1u << lane) - 1))] = (uint16_t)(32 * i + lane);
                at += __popc(m);
            }
            if (lane == 0) s_ntouch = at;
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
        // t = b - K x; with K Z, beside the restriction (the post-smoothing's
        // residual), else before it
        if (spmm16(a.x32, [&](int row) { return f3(a.b32, row); }, [&] { return check && s_sum[0] <= a.tol2; },
                   [&](int row, float (&y)[3], const F3 &b) {
#pragma unroll
                       for (int i = 0; i < 3; ++i) a.t32[3L * row + i] = b.v[i] - y[i];
                   })) {
            stop(OFEA_OK, kk + 1);
            return 1;
        }
        if (a.md_ptr) __syncthreads();  // s_red is read
        else if (!sync()) return 2;
        {  // c = Z^T t, or Z^T b - (K Z)^T x, one CTA per aggregate
            float *sh = reinterpret_cast<float *>(s_red);  // [6][warps]
            for (int I = blockIdx.x; I < a.na; I += G) {
                float acc[6] = {0, 0, 0, 0, 0, 0};
                modes_sum(__ldg(a.agg_ptr + I) + tid, __ldg(a.agg_ptr + I + 1), kResThreads, a.agg_off,
                          a.md_ptr ? a.b32 : a.t32, acc);
                if (a.md_ptr)
                    entries_sum(__ldg(a.md_ptr + I) + tid, __ldg(a.md_ptr + I + 1), kResThreads, a.md_row, a.md_val, a.md.n,
                                a.x32, acc);
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
        for (int i0 = w; i0 < 6 * s_ntouch; i0 += 4 * kResWarps) {  // four rows of E^-1 in flight per warp
            int at[4];
            const float *row[4];
            float sm[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = min(i0 + u * kResWarps, 6 * s_ntouch - 1), t = i / 6;
                at[u] = 6 * s_list[t] + (i - 6 * t);
                row[u] = a.Einv + (long)at[u] * a.m;
                sm[u] = 0.f;
            }
#pragma unroll 2
            for (int j = lane; j < a.m; j += 32) {
                const float cj = a.cvec[j];
#pragma unroll
                for (int u = 0; u < 4; ++u) sm[u] = fmaf(__ldg(row[u] + j), cj, sm[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                sm[u] = warp_sum(sm[u]);
                if (lane == 0) s_e[at[u]] = sm[u];
            }
        }
        __syncthreads();
        float *znew = ((kk + 1) & 1) ? a.zB : a.zA;
        const float *zold = ((kk + 1) & 1) ? a.zA : a.zB;
        double prz = 0.0, przo = 0.0;
        if (a.md_ptr) {  // z = x0 + Z e + w Dinv32 (t - K Z e): own rows only
            // the own entries' parts first, a thread per entry
            float *part = reinterpret_cast<float *>(s_red);
            const int e0 = __ldg(a.md.rptr + row0), ne = __ldg(a.md.rptr + row1) - e0;
            const bool staged = 3 * ne <= 2 * (int)(sizeof(s_red) / sizeof(double));
            if (staged)
                for (int t = tid; t < ne; t += kResThreads) {
                    float k[3];
                    a.md.entry(e0 + t, s_e, k);
#pragma unroll
                    for (int c = 0; c < 3; ++c) part[3 * t + c] = k[c];
                }
            __syncthreads();
            for (int r = row0 + tid; r < row1; r += kResThreads) {
                float ze[3], kz[3] = {0.f, 0.f, 0.f}, d[3], o[3];
                a.md.modes(r, s_e, ze);
                if (staged) {
                    for (int t = __ldg(a.md.rptr + r) - e0; t < __ldg(a.md.rptr + r + 1) - e0; ++t)
#pragma unroll
                        for (int c = 0; c < 3; ++c) kz[c] += part[3 * t + c];
                } else {
                    a.md.row(r, s_e, kz);
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) d[i] = a.t32[3L * r + i] - kz[i];
                block3_apply(a.Dinv32 + 9L * r, d, o);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const long dd = 3L * r + i;
                    const float zn = fmaf(a.wsm, o[i], a.x32[dd] + ze[i]);
                    const double rv = a.r[dd];
                    prz += rv * (double)zn;
                    przo += rv * (double)zold[dd];
                    znew[dd] = zn;
                }
            }
            put(prz, ((kk + 1) & 1) ? a.P.rz1 : a.P.rz0, przo, a.P.rzo);
            return sync() ? 0 : 2;
        }
        for (int r = row0 + tid; r < row1; r += kResThreads) {
            const float4 o = __ldg(a.row_off + r);
            const float *e = s_e + 6 * __float_as_int(o.w);
            const float dx = o.x, dy = o.y, dz = o.z;
            a.x32[3L * r] += e[0] + dz * e[4] - dy * e[5];
            a.x32[3L * r + 1] += e[1] - dz * e[3] + dx * e[5];
            a.x32[3L * r + 2] += e[2] + dy * e[3] - dx * e[4];
        }
        if (!sync()) return 2;
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

// --------------------------------------------------- one cluster, small K --
//
// The same iterations for matrices of a few thousand rows in one thread-block
// cluster.  A grid barrier costs 2,000 to 5,000 cycles (arrival after the
// phase's stores have drained to L2, the spin, the first load after it); here
// the gathered vectors (z; the V-cycle's x) are kept whole in every CTA's shared
// memory, the owners of rows write them into all CTAs, partial sums go the
// same way, and a phase ends at the cluster's hardware barrier.  The other
// vectors live in the owner's shared memory.  K and the inverse diagonal blocks
// are read through L1.  The coarse level: every CTA restricts its own rows, the
// partial c of all CTAs are summed by each, and e = E^-1 c and x += Z e are
// formed by every CTA for its whole copy of x, so the coarse correction costs
// one barrier, or none with K Z (c's parts travel with ||r||^2).  Barriers per
// iteration: PCG64 2, MIXED 3 (4 without K Z).
//
// The sums of a phase go to an inbox of their own; an inbox, and a whole
// vector, is written again only after a barrier that follows its last reading.
//
// Per iteration, grid of CTAs before, cluster after: PCG64 7.6 -> 5.3 us at 1.5k
// DOF, 7.9 -> 6.5 at 3.3k; MIXED 19.5 -> 12.5 and 20.4 -> 15.0.  With 32 warps
// per CTA instead of 16 the idle ones' instructions cost more than their help
// (6.3 and 14.2 us).  Bound by the instruction chains of its phases (the
// reductions' shuffles, the product's combine) and 700 cycles per barrier.

namespace {

constexpr int kClMax = 16;       // CTAs of the largest cluster (beyond 8 if the device allows it)
constexpr int kClSpc = 4;        // slices per CTA at most
constexpr int kClRows = kClSpc * kSlice;
constexpr int kClM = 192;        // coarse unknowns at most
constexpr int kClThreads = 512, kClWarps = kClThreads / 32;

struct ClShared {
    double red[kClWarps * 3 * 32];
    double u[3 * kClRows], r[3 * kClRows], p[3 * kClRows], q[3 * kClRows];
    double in[4][2][kClMax];     // inboxes: p.q; ||r||^2 (and r.z); r.z and r.z_old
    float b[3 * kClRows], t[3 * kClRows];
    float cin[kClMax][kClM], c[kClM], e[kClM];
    double w[2][kClWarps];
};

// The cluster's barrier.  Writes into other CTAs are ordered by their writers
// (peer_done after the stores), this CTA's own by the block barrier: a
// releasing arrival of every warp cost a fence in each.
__device__ __forceinline__ void peer_done() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    __syncthreads();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The same shared-memory address in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned peer(const void *p, unsigned rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), o;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(rank));
    return o;
}
__device__ __forceinline__ void peer_st(unsigned a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ void peer_st(unsigned a, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void peer_st(unsigned a, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

}  // namespace

template <bool MIXED>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_solve(const RArgs a) {
    extern __shared__ __align__(16) unsigned char dyn[];
    ClShared &sh = *reinterpret_cast<ClShared *>(dyn);
    using ZT = typename std::conditional<MIXED, float, double>::type;
    const int npad = 3 * kSlice * a.nslice;  // whole vectors, padded to slices
    ZT *zr = reinterpret_cast<ZT *>(dyn + sizeof(ClShared));
    float *xr = reinterpret_cast<float *>(zr + npad);  // MIXED
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int C = gridDim.x;
    const int rank = (int)cluster_rank();
    const int sl0 = min(a.nslice, rank * a.spc), sl1 = min(a.nslice, sl0 + a.spc);
    const int row0 = sl0 * kSlice, row1 = min(a.nfree, sl1 * kSlice), own3 = 3 * (row1 - row0);
    if (*(volatile int *)&a.fl->done) return;  // written by an earlier launch: the same in every CTA
    int k = *(volatile int *)&a.fl->itA;
    // state of the launch before
    {
        const double *pold = (k & 1) ? a.p1 : a.p0;
        for (int i = tid; i < own3; i += kClThreads) {
            const long d = 3L * row0 + i;
            sh.u[i] = a.u[d];
            sh.r[i] = a.r[d];
            sh.p[i] = pold[d];
            sh.q[i] = a.q[d];
            if (MIXED) sh.b[i] = a.b32[d];
        }
        const float *zf = (k & 1) ? a.zB : a.zA;
        for (int i = tid; i < npad; i += kClThreads) {
            if constexpr (MIXED) {
                zr[i] = i < 3 * a.nfree ? zf[i] : 0.f;
                xr[i] = i < 3 * a.nfree ? a.x32[i] : 0.f;
            } else {
                zr[i] = i < 3 * a.nfree ? a.z[i] : 0.0;
            }
        }
    }
    double rz = warp_partials((k & 1) ? a.P.rz1 : a.P.rz0, a.P.G), rzp = warp_partials((k & 1) ? a.P.rz0 : a.P.rz1, a.P.G);
    double rzo = MIXED ? warp_partials(a.P.rzo, a.P.G) : 0.0, rr = warp_partials(a.P.rr, a.P.G);
    const int ng64 = kClWarps / a.S64, g64 = w / a.S64, p64 = w - g64 * a.S64;
    const int ng16 = kClWarps / a.S16, g16 = w / a.S16, p16 = w - g16 * a.S16;
    Home h64{0, 0, 0, 0}, h16{0, 0, 0, 0};
    long G16 = 0;
    if (g64 < ng64 && sl0 + g64 < sl1) h64 = home(a.sl_ptr, a.scols, sl0 + g64, lane, p64, p64 + a.S64);
    if (MIXED && g16 < ng16 && sl0 + g16 < sl1) {
        h16 = home(a.sl_ptr, a.scols, sl0 + g16, lane, 2 * p16, 2 * p16 + 1);
        G16 = __ldg(a.sl_g + sl0 + g16);
    }
    for (int i = tid; i < 4 * 2 * kClMax; i += kClThreads) (&sh.in[0][0][0])[i] = 0.0;
    // every CTA is here before the first write into another's shared memory
    cluster_sync();

    // y = K x for the own rows, fin(own row, y)
    auto spmm = [&](auto half, auto x, auto fin) {
        constexpr bool BF = decltype(half)::value;
        using T = typename std::conditional<BF, float, double>::type;
        T *red = reinterpret_cast<T *>(sh.red);
        const int S = BF ? a.S16 : a.S64, ng = BF ? ng16 : ng64, g = BF ? g16 : g64, part = BF ? p16 : p64;
        for (int b = sl0; b < sl1; b += ng) {
            T y[3] = {0, 0, 0};
            if (g < ng && b + g < sl1) {
                const bool first = b == sl0;
                if constexpr (BF) {
                    const Home h = first ? h16 : home(a.sl_ptr, a.scols, b + g, lane, 2 * part, 2 * part + 1);
                    part16(h, first ? G16 : (long)__ldg(a.sl_g + b + g), lane, part, S, a.scols, a.svg, x, y);
                } else {
                    const Home h = first ? h64 : home(a.sl_ptr, a.scols, b + g, lane, part, part + S);
                    part64(h, lane, part, S, a.scols, a.sv64, x, y);
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) red[(w * 3 + i) * 32 + lane] = y[i];
            }
            __syncthreads();
            const int row = (b + w) * kSlice + lane;
            if (w < ng && b + w < sl1 && row < a.nfree) {
#pragma unroll
                for (int i = 0; i < 3; ++i) y[i] = 0;
                for (int p = 0; p < S; ++p)
#pragma unroll
                    for (int i = 0; i < 3; ++i) y[i] += red[((w * S + p) * 3 + i) * 32 + lane];
                fin(row - row0, y);
            }
            __syncthreads();
        }
    };
    // this CTA's partial sums (of its first nw warps' values) into every CTA's
    // inbox
    auto send = [&](int box, int nw, double x, double y) {
        if (w < nw) {
            x = warp_sum(x);
            y = warp_sum(y);
            if (lane == 0) {
                sh.w[0][w] = x;
                sh.w[1][w] = y;
            }
        }
        __syncthreads();
        if (w < 2) {
            const double s = warp_sum(lane < nw ? sh.w[w][lane] : 0.0);
            if (lane < C) peer_st(peer(&sh.in[box][w][rank], lane), s);
            peer_done();
        }
    };
    auto inbox = [&](int box, int which) {  // unused entries are zero
        const double *v = sh.in[box][which];
        double s[kClMax];
#pragma unroll
        for (int i = 0; i < kClMax; ++i) s[i] = v[i];
#pragma unroll
        for (int d = kClMax / 2; d > 0; d >>= 1)
#pragma unroll
            for (int i = 0; i < d; ++i) s[i] += s[i + d];
        return s[0];
    };
    // the own rows of a whole vector, written here, into the other CTAs
    auto spread = [&](auto *v) {
        using T = typename std::remove_reference<decltype(*v)>::type;
        constexpr int E = 16 / (int)sizeof(T);
        __syncthreads();
        const int n4 = (own3 + E - 1) / E;
        for (int i = tid; i < n4 * (C - 1); i += kClThreads) {
            const int j = i / n4, o = i - j * n4;
            int to = rank + 1 + j;
            if (to >= C) to -= C;
            T *src = v + 3 * row0 + o * E;
            peer_st(peer(src, to), *reinterpret_cast<const float4 *>(src));
        }
        peer_done();
    };
    // everything the next launch, or the caller, reads
    auto leave = [&](int status, int done) {
        double *pk = (k & 1) ? a.p1 : a.p0;
        float *zf = (k & 1) ? a.zB : a.zA;
        for (int i = tid; i < own3; i += kClThreads) {
            const long d = 3L * row0 + i;
            a.u[d] = sh.u[i];
            a.r[d] = sh.r[i];
            pk[d] = sh.p[i];
            a.q[d] = sh.q[i];
            if constexpr (MIXED) {
                a.b32[d] = sh.b[i];
                a.x32[d] = xr[d];
                zf[d] = zr[d];
            } else {
                a.z[d] = zr[d];
            }
        }
        if (rank == 0) {
            double *Pc = (k & 1) ? a.P.rz1 : a.P.rz0, *Po = (k & 1) ? a.P.rz0 : a.P.rz1;
            for (int j = tid; j < a.P.G; j += kClThreads) {
                Pc[j] = j ? 0.0 : rz;
                Po[j] = j ? 0.0 : rzp;
                a.P.rzo[j] = j ? 0.0 : rzo;
                a.P.rr[j] = j ? 0.0 : rr;
            }
            if (tid == 0) {
                a.fl->done = done;
                a.fl->status = status;
                a.fl->itA = k;
                a.fl->iters = k;
            }
        }
        cluster_sync();  // no CTA leaves while another may write into it
    };
    // z = M(b), from the pre-smoothed x in every CTA; sums r.z, r.z_old
    // own rows' part of c = Z^T t, or of Z^T b - (K Z)^T x, a warp per aggregate
    auto restrict_own = [&]() {
        if constexpr (MIXED) {
            const float *v = a.md_ptr ? sh.b : sh.t;
            for (int I = w; I < a.na; I += kClWarps) {
                float acc[6] = {0, 0, 0, 0, 0, 0};
                for (int i = lane; i < row1 - row0; i += 32) {
                    const float4 o = __ldg(a.row_off + row0 + i);
                    if (__float_as_int(o.w) != I) continue;
                    const float tx = v[3 * i], ty = v[3 * i + 1], tz = v[3 * i + 2];
                    acc[0] += tx;
                    acc[1] += ty;
                    acc[2] += tz;
                    acc[3] += -o.z * ty + o.y * tz;
                    acc[4] += o.z * tx - o.x * tz;
                    acc[5] += -o.y * tx + o.x * ty;
                }
                if (a.md_ptr)
                    for (int e = __ldg(a.md_ptr + I) + lane; e < __ldg(a.md_ptr + I + 1); e += 32) {
                        const int r = __ldg(a.md_row + e);
                        if (r >= row0 && r < row1) entry_sub(e, a.md.n, a.md_val, xr[3 * r], xr[3 * r + 1], xr[3 * r + 2], acc);
                    }
#pragma unroll
                for (int q = 0; q < 6; ++q) acc[q] = warp_sum(acc[q]);
                if (lane < C)
#pragma unroll
                    for (int q = 0; q < 6; ++q) peer_st(peer(&sh.cin[rank][6 * I + q], lane), acc[q]);
            }
            peer_done();
        }
    };
    // with K Z, c's parts are already here (restrict_own before the barrier)
    auto vcycle = [&]() {
        if constexpr (MIXED) {
            if (!a.md_ptr) {
                spmm(std::true_type{}, (const float *)xr, [&](int i, float (&y)[3]) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) sh.t[3 * i + c] = sh.b[3 * i + c] - y[c];
                });
                restrict_own();
                cluster_sync();
            }
            for (int i = tid; i < a.m; i += kClThreads) {
                float s = 0.f;
                for (int j = 0; j < C; ++j) s += sh.cin[j][i];
                sh.c[i] = s;
            }
            __syncthreads();
            for (int i = w; i < a.m; i += kClWarps) {
                const float *row = a.Einv + (long)i * a.m;
                float s = 0.f;
                for (int j = lane; j < a.m; j += 32) s = fmaf(__ldg(row + j), sh.c[j], s);
                s = warp_sum(s);
                if (lane == 0) sh.e[i] = s;
            }
            __syncthreads();
            if (!a.md_ptr) {
                for (int r = tid; r < a.nfree; r += kClThreads) {
                    const float4 o = __ldg(a.row_off + r);
                    const float *e = sh.e + 6 * __float_as_int(o.w);
                    xr[3 * r] += e[0] + o.z * e[4] - o.y * e[5];
                    xr[3 * r + 1] += e[1] - o.z * e[3] + o.x * e[5];
                    xr[3 * r + 2] += e[2] + o.y * e[3] - o.x * e[4];
                }
                __syncthreads();
            }
            double prz = 0.0, przo = 0.0;
            spmm(std::true_type{}, (const float *)xr, [&](int i, float (&y)[3]) {
                float d[3], o[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) d[c] = sh.b[3 * i + c] - y[c];
                float ze[3] = {0.f, 0.f, 0.f};
                if (a.md_ptr) {
                    float kz[3];
                    a.md.modes(row0 + i, sh.e, ze);
                    a.md.row(row0 + i, sh.e, kz);
#pragma unroll
                    for (int c = 0; c < 3; ++c) d[c] -= kz[c];
                }
                block3_apply(a.Dinv32 + 9L * (row0 + i), d, o);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const int g = 3 * (row0 + i) + c;
                    const float zn = fmaf(a.wsm, o[c], xr[g] + ze[c]);
                    const double rv = sh.r[3 * i + c];
                    prz += rv * (double)zn;
                    przo += rv * (double)zr[g];
                    zr[g] = zn;
                }
            });
            spread(zr);
            send(2, ng16, prz, przo);
            cluster_sync();
            rz = inbox(2, 0);
            rzo = inbox(2, 1);
        }
    };
    if (MIXED && a.first) {
        if (a.md_ptr) {
            restrict_own();
            cluster_sync();
        }
        vcycle();
    }
    for (int it = 0; it < a.iters; ++it) {
        if (!MIXED && rr <= a.tol2) {
            leave(OFEA_OK, 1);
            return;
        }
        const double beta = k > 0 ? (MIXED ? rz - rzo : rz) / rzp : 0.0;
        double ppq = 0.0;
        spmm(std::false_type{}, [&](int i) { return (double)zr[i]; }, [&](int i, double (&y)[3]) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int d = 3 * i + c;
                const double pn = fma(beta, sh.p[d], (double)zr[3 * row0 + d]);
                const double qn = fma(beta, sh.q[d], y[c]);  // K p = K z + beta K p_old
                sh.p[d] = pn;
                sh.q[d] = qn;
                ppq += pn * qn;
            }
        });
        send(0, ng64, ppq, 0.0);
        cluster_sync();
        const double pq = inbox(0, 0);
        if (!(pq > 0.0) || !isfinite(pq)) {
            leave(OFEA_ERR_BREAKDOWN, 1);
            return;
        }
        const double alpha = rz / pq;
        double prr = 0.0, prz = 0.0;
        for (int i = tid; i < row1 - row0; i += kClThreads) {
            double rv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int d = 3 * i + c;
                sh.u[d] = fma(alpha, sh.p[d], sh.u[d]);
                rv[c] = fma(-alpha, sh.q[d], sh.r[d]);
                sh.r[d] = rv[c];
                prr += rv[c] * rv[c];
            }
            if constexpr (MIXED) {
                float b[3] = {(float)rv[0], (float)rv[1], (float)rv[2]}, x[3];
                block3_apply(a.Dinv32 + 9L * (row0 + i), b, x);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    sh.b[3 * i + c] = b[c];
                    xr[3 * (row0 + i) + c] = a.wsm * x[c];
                }
            } else {
                double zz[3];
                block3_apply(a.Dinv + 9L * (row0 + i), rv, zz);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    zr[3 * (row0 + i) + c] = zz[c];
                    prz += rv[c] * zz[c];
                }
            }
        }
        if constexpr (MIXED) {
            spread(xr);
            if (a.md_ptr) restrict_own();
        } else {
            spread(zr);
        }
        send(1, a.spc, prr, prz);
        cluster_sync();
        rr = inbox(1, 0);
        rzp = rz;
        ++k;
        if constexpr (MIXED) {
            if (rr <= a.tol2) {
                leave(OFEA_OK, 1);
                return;
            }
            vcycle();
        } else {
            rz = inbox(1, 1);
        }
    }
    leave(OFEA_OK, 0);
}

// ------------------------------------------------------------------- host --

namespace {

int cluster_smem(int nslice, bool mixed) {
    const size_t whole = 3 * (size_t)kSlice * nslice;
    return (int)(sizeof(ClShared) + whole * 8);  // z in FP64, or z and x in FP32
}

// The largest cluster of k_cluster_solve the device runs (16, 8 or none), asked
// for once per device.
int cluster_limit(int device) {
    static std::mutex mu;
    static std::map<int, int> known;
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(device);
    if (it != known.end()) return it->second;
    int limit = 0;
    for (int C : {16, 8}) {
        bool ok = true;
        for (const void *fn : {(const void *)k_cluster_solve<true>, (const void *)k_cluster_solve<false>}) {
            const int smem = cluster_smem(C * kClSpc, true);
            if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, cluster_smem(kClMax * kClSpc, true)) != cudaSuccess ||
                (C > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
                ok = false;
                break;
            }
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = C;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(C);
            cfg.blockDim = dim3(kClThreads);
            cfg.dynamicSmemBytes = smem;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess || n < 1) {
                ok = false;
                break;
            }
        }
        if (ok) {
            limit = C;
            break;
        }
        cudaGetLastError();
    }
    known[device] = limit;
    return limit;
}

}  // namespace

// Where the lines lie, solve with its set-up on a new K here / launch per phase
// (ms, at 1e-8; C3D8, smoothed moduli).  MIXED up to 3,500 slices (336k DOF):
// with the elements' outer product there, 328k DOF (702 coarse unknowns) 6.2 /
// 6.7, 402k (864) 7.2 / 7.1, 467k (1152) 9.9 / 8.3; without (a tangent) 6.6 /
// 9.0, 7.3 / 9.5, 10.3 / 10.0.  The coarse level is bounded because its dense
// inverse has to be formed, and every CTA multiplies the rows of it that its
// own rows need: 218k DOF with 936 unknowns 4.7 / 5.1, 1344 5.2 / 5.0, 2850
// 11.4 / 5.8; the same as a tangent, 1536 5.3 / 6.6, 2850 10.7 / 7.1; 106k DOF
// with 1440 4.0 / 4.9, 1728 4.8 / 4.8; C3D4, 142k DOF, 1200 3.9 / 5.0, 1980
// 6.3 / 5.1.  PCG64 with the stored K is the faster one at every size measured
// (us per iteration: 807k DOF tangent 114 / 131, 1.56M 221 / 234, C3D4 of 3.0M
// 266 / 280).
constexpr int kResMixedSlices = 3500;
constexpr int kResElementsM = 1250;  // coarse unknowns, where the other side has the elements' product

bool resident_plan(const ofea_ctx *c, bool mixed, bool elements, ResidentPlan &p) {
    const int nslice = (c->nfree + kSlice - 1) / kSlice;
    if (nslice < 1) return false;
    const int W = (int)std::max<long long>(1, c->sell_len / nslice);
    // warps per slice: the fewest serial steps over all rounds, a round's own
    // latency counted as two steps
    auto pick = [&](int units, int warps) {
        int best = 1;
        long cost = -1;
        for (int S = 1; S <= warps; ++S) {
            const int ng = warps / S, rounds = (p.spc + ng - 1) / ng;
            const long t = (long)rounds * ((units + S - 1) / S + 2);
            if (cost < 0 || t < cost) {
                cost = t;
                best = S;
            }
        }
        return best;
    };
    p.cluster = 0;
    // one cluster up to 64 slices (6.1k DOF), where the two meet (6.1k DOF:
    // PCG64 7.5 us, 7.9 on the grid; 7.9k DOF: 7.7 us on the grid)
    const int limit = cluster_limit(c->device);
    if (limit > 0 && nslice <= limit * kClSpc && (!mixed || c->coarse.m <= kClM)) {
        int C = 1;
        while (C < limit && C < nslice) C *= 2;
        p.cluster = p.G = C;
        p.spc = (nslice + C - 1) / C;
        p.S64 = p.S16 = pick((W + 1) / 2, kClWarps);
        return true;
    }
    if (mixed && (nslice > kResMixedSlices || c->coarse.m > (elements ? kResElementsM : kResMaxM))) return false;
    p.spc = (nslice + c->num_sms - 1) / c->num_sms;
    p.G = (nslice + p.spc - 1) / p.spc;
    p.S64 = p.S16 = pick((W + 1) / 2, kResWarps);  // two slots in flight per step
    return true;
}

void resident_iterations(ofea_ctx *c, const ResidentPlan &p, bool mixed, bool modes, const Parts &P, Flags *fl, double *d_u,
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
        if (modes) {
            a.md_ptr = C.md_ptr.p;
            a.md_row = C.md_row.p;
            a.md_val = C.md_val.p;
            a.md = row_modes(C);
        }
    }
    a.wsm = wsm;
    a.tol2 = tol2;
    a.P = P;
    a.fl = fl;
    if (p.cluster) {
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = p.cluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(p.cluster);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = cluster_smem(a.nslice, mixed);
        cfg.stream = c->stream;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        void *args[] = {(void *)&a};
        OFEA_CUDA(cudaLaunchKernelExC(&cfg, mixed ? (const void *)k_cluster_solve<true> : (const void *)k_cluster_solve<false>, args));
        return;
    }
    a.bar = reinterpret_cast<GridBar *>(w.bar.p);
    a.limit_ns = c->wait_limit_ns;
    OFEA_CUDA(cudaMemsetAsync(w.bar.p, 0, sizeof(GridBar), c->stream));
    if (c->wait_missing) OFEA_CUDA(cudaMemsetAsync(&a.bar->count, 0xff, sizeof(a.bar->count), c->stream));  // -1
    void *args[] = {(void *)&a};
    const void *fn = mixed ? (const void *)k_resident<true> : (const void *)k_resident<false>;
    OFEA_CUDA(cudaLaunchCooperativeKernel(fn, dim3(p.G), dim3(kResThreads), args, 0, c->stream));
}

}  // namespace ofea
