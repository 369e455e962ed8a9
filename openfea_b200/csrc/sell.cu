// Conversion of the assembled block-CSR K into the solver's BSELL-32 layout
// (sell.cuh): FP64 values and a BF16 copy grouped by four slots
// (sell_row_g4), once per assembly; and, once per pattern and on demand, the
// slices' distinct columns.
#include <algorithm>

#include "sell.cuh"

namespace ofea {

__global__ void k_slice_width(int nfree, const int *__restrict__ rowptr, int *__restrict__ width) {
    const int nslice = (nfree + kSlice - 1) / kSlice;
    const int lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) / 32; s < nslice;
         s += gridDim.x * blockDim.x / 32) {
        int r = s * kSlice + lane;
        int d = r < nfree ? rowptr[r + 1] - rowptr[r] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d = max(d, __shfl_xor_sync(0xffffffffu, d, o));
        if (lane == 0) width[s] = d;
    }
}

// Pattern part of the layout: the slots' block columns (padding: the row's
// own column, row 0 past the last row).  Once per pattern.
__global__ void k_fill_scols(int nfree, const int *__restrict__ rowptr, const int *__restrict__ cols,
                             const int *__restrict__ sl_ptr, int *__restrict__ scols) {
    const int nslice = (nfree + kSlice - 1) / kSlice;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < (long)nslice * kSlice;
         g += (long)gridDim.x * blockDim.x) {
        const int s = (int)(g / kSlice), t = (int)(g % kSlice);
        const int r = s * kSlice + t;
        const long S = sl_ptr[s];
        const int W = sl_ptr[s + 1] - (int)S;
        const int rb = r < nfree ? rowptr[r] : 0;
        const int deg = r < nfree ? rowptr[r + 1] - rb : 0;
        for (int k = 0; k < W; ++k) scols[(S + k) * kSlice + t] = k < deg ? cols[rb + k] : (r < nfree ? r : 0);
    }
}

// Values: FP64 planes and the grouped BF16 copy, from block-CSR K.
__global__ void k_fill_sell(int nfree, const int *__restrict__ rowptr, const double *__restrict__ Kb,
                            const int *__restrict__ sl_ptr, double *__restrict__ sv64,
                            const int *__restrict__ sl_g,
                            __nv_bfloat16 *__restrict__ svg) {
    const int nslice = (nfree + kSlice - 1) / kSlice;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < (long)nslice * kSlice;
         g += (long)gridDim.x * blockDim.x) {
        const int s = (int)(g / kSlice), t = (int)(g % kSlice);
        const int r = s * kSlice + t;
        const long S = sl_ptr[s];
        const int W = sl_ptr[s + 1] - (int)S;
        const int rb = r < nfree ? rowptr[r] : 0;
        const int deg = r < nfree ? rowptr[r + 1] - rb : 0;
        const long G = sl_g[s];
        uint2 *svg2 = reinterpret_cast<uint2 *>(svg);
        for (int g = 0; g < (W + 3) / 4; ++g) {
            unsigned h[9][2] = {};  // the group's four BF16 values per plane, two per word
            for (int u = 0; u < 4; ++u) {
                const int k = 4 * g + u;
                const bool real = k < deg;
#pragma unroll
                for (int e = 0; e < 9; ++e) {
                    const double v = real ? Kb[9L * (rb + k) + e] : 0.0;
                    const __nv_bfloat16 bv = __double2bfloat16(v);
                    if (k < W) sv64[((S + k) * 9 + e) * kSlice + t] = v;
                    h[e][u >> 1] |= (unsigned)__bfloat16_as_ushort(bv) << (16 * (u & 1));
                }
            }
#pragma unroll
            for (int e = 0; e < 9; ++e) svg2[((G + g) * 9 + e) * kSlice + t] = make_uint2(h[e][0], h[e][1]);
        }
    }
}

__global__ void k_group_width(int nslice, const int *__restrict__ sl_ptr, int *__restrict__ gw) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nslice; s += gridDim.x * blockDim.x)
        gw[s] = (sl_ptr[s + 1] - sl_ptr[s] + 3) / 4;
}

void build_sell_layout(ofea_ctx *c) {
    cudaStream_t s = c->stream;
    const int nslice = (c->nfree + kSlice - 1) / kSlice;
    c->sl_ptr.ensure((size_t)nslice + 1);
    int tmp_len = nslice / 1024 + 4;
    c->scratch_i.ensure((size_t)nslice + 1 + tmp_len);
    int *width = c->scratch_i.p;
    k_slice_width<<<grid_for(c, (long)nslice * 32, kBlock), kBlock, 0, s>>>(c->nfree, c->rowptr.p, width);
    OFEA_CHECK_LAUNCH();
    long long tot = exclusive_scan(width, c->sl_ptr.p, nslice, s, width + nslice + 1, tmp_len);
    c->sell_len = tot;
    size_t slots = (size_t)std::max<long long>(tot, 1) * kSlice;
    c->scols.ensure(slots);
    c->sv64.ensure(9 * slots);
    // slot groups of four per slice for the grouped BF16 copy
    c->sl_g.ensure((size_t)nslice + 1);
    k_group_width<<<grid_for(c, nslice, kBlock), kBlock, 0, s>>>(nslice, c->sl_ptr.p, width);
    OFEA_CHECK_LAUNCH();
    const long long groups = exclusive_scan(width, c->sl_g.p, nslice, s, width + nslice + 1, tmp_len);
    c->sv16g.ensure((size_t)std::max<long long>(groups, 1) * 9 * kSlice * 4);
    k_fill_scols<<<grid_for(c, (long)nslice * kSlice, kBlock), kBlock, 0, s>>>(c->nfree, c->rowptr.p, c->cols.p,
                                                                              c->sl_ptr.p, c->scols.p);
    OFEA_CHECK_LAUNCH();
    c->sell_layout_ok = true;
    c->su_ok = false;
}

// Distinct columns of a slice, one CTA per slice: its 32 W slots' columns are
// sorted (bitonic, in shared memory), the runs of consecutive distinct ones
// listed (first column; position << 16 | length), and each slot gets its
// column's position.  su_n: distinct columns and runs of each slice; a slice
// of more than kSuMax slots is not listed (0).
constexpr int kSuMax = 4096;
__global__ void __launch_bounds__(kBlock) k_slice_columns(int nslice, const int *__restrict__ sl_ptr,
                                                          const int *__restrict__ scols, int2 *__restrict__ su_runs,
                                                          int *__restrict__ su_n, uint16_t *__restrict__ su_idx,
                                                          int *__restrict__ su_max) {
    __shared__ int key[kSuMax], uniq[kSuMax], wsum[kWarpsPerBlock];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int s = blockIdx.x; s < nslice; s += gridDim.x) {
        const long base = (long)sl_ptr[s] * kSlice;
        const int n = (sl_ptr[s + 1] - sl_ptr[s]) * kSlice;
        if (n > kSuMax || n == 0) {
            if (tid == 0) su_n[2 * s] = su_n[2 * s + 1] = 0;
            continue;
        }
        int n2 = 32;
        while (n2 < n) n2 <<= 1;
        __syncthreads();
        for (int i = tid; i < n2; i += kBlock) key[i] = i < n ? scols[base + i] : 0x7fffffff;
        __syncthreads();
        for (int k = 2; k <= n2; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = tid; i < n2; i += kBlock) {
                    const int l = i ^ j;
                    if (l > i) {
                        const int x = key[i], y = key[l];
                        if ((x > y) == ((i & k) == 0)) {
                            key[i] = y;
                            key[l] = x;
                        }
                    }
                }
                __syncthreads();
            }
        int nu = 0;  // distinct so far (the same in every thread)
        for (int b = 0; b < n; b += kBlock) {
            const int i = b + tid;
            const bool first = i < n && (i == 0 || key[i] != key[i - 1]);
            const unsigned m = __ballot_sync(0xffffffffu, first);
            if (lane == 0) wsum[w] = __popc(m);
            __syncthreads();
            int off = nu, tot = 0;
            for (int q = 0; q < kWarpsPerBlock; ++q) {
                if (q < w) off += wsum[q];
                tot += wsum[q];
            }
            if (first) uniq[off + __popc(m & ((1u << lane) - 1))] = key[i];
            nu += tot;
            __syncthreads();
        }
        int nrun = 0;
        for (int b = 0; b < nu; b += kBlock) {
            const int i = b + tid;
            const bool first = i < nu && (i == 0 || uniq[i] != uniq[i - 1] + 1);
            const unsigned m = __ballot_sync(0xffffffffu, first);
            if (lane == 0) wsum[w] = __popc(m);
            __syncthreads();
            int off = nrun, tot = 0;
            for (int q = 0; q < kWarpsPerBlock; ++q) {
                if (q < w) off += wsum[q];
                tot += wsum[q];
            }
            if (first) {
                int len = 1;
                while (i + len < nu && uniq[i + len] == uniq[i] + len) ++len;
                su_runs[base + off + __popc(m & ((1u << lane) - 1))] = make_int2(uniq[i], i << 16 | len);
            }
            nrun += tot;
            __syncthreads();
        }
        for (int i = tid; i < n; i += kBlock) {
            const int c = scols[base + i];
            int lo = 0, hi = nu - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (uniq[mid] < c) lo = mid + 1;
                else hi = mid;
            }
            su_idx[base + i] = (uint16_t)lo;
        }
        if (tid == 0) {
            su_n[2 * s] = nu;
            su_n[2 * s + 1] = nrun;
            atomicMax(su_max, nu);
        }
    }
}

// Once per pattern, when the batched solver first asks for it.
void ensure_slice_columns(ofea_ctx *c) {
    if (c->su_ok) return;
    const int nslice = (c->nfree + kSlice - 1) / kSlice;
    const size_t slots = (size_t)std::max<long long>(c->sell_len, 1) * kSlice;
    c->su_runs.ensure(2 * slots);
    c->su_idx.ensure(slots);
    c->su_n.ensure(2 * (size_t)std::max(nslice, 1));
    OFEA_CUDA(cudaMemsetAsync(c->err_flag.p, 0, sizeof(int), c->stream));
    k_slice_columns<<<grid_for(c, nslice, 1), kBlock, 0, c->stream>>>(nslice, c->sl_ptr.p, c->scols.p,
                                                                     reinterpret_cast<int2 *>(c->su_runs.p),
                                                                     c->su_n.p, c->su_idx.p, c->err_flag.p);
    OFEA_CHECK_LAUNCH();
    OFEA_CUDA(cudaMemcpyAsync(c->herr.p, c->err_flag.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    OFEA_CUDA(cudaStreamSynchronize(c->stream));
    c->su_max = c->herr.p[0];
    c->su_ok = true;
}

void build_sell(ofea_ctx *c) {
    if (!c->sell_layout_ok) build_sell_layout(c);
    cudaStream_t s = c->stream;
    const int nslice = (c->nfree + kSlice - 1) / kSlice;
    k_fill_sell<<<grid_for(c, (long)nslice * kSlice, kBlock), kBlock, 0, s>>>(
        c->nfree, c->rowptr.p, c->Kb.p, c->sl_ptr.p, c->sv64.p, c->sl_g.p, c->sv16g.p);
    OFEA_CHECK_LAUNCH();
    c->sell_ok = true;
}

}  // namespace ofea
