// Cumulative normalised transition rows and the per-row bracket ("guide") table.
//
// C[y, z] = min(1, (sum_{w<=z} P[y, w]) / (sum_w P[y, w])) with a sequential FP32 running
// sum in z order, one FP32 division per entry and the clamp at 1 -- the arithmetic of
// oplib/opcuda/sck.cu:43-84, so the rows are bit-identical to a sequential CPU loop.
// Negative entries (FP32 rounding residue of a squared kernel) are taken as 0 so the
// rows are non-decreasing and every correct inverse-CDF search returns the same state.
//
// The guide table follows the bracket table the reference builds on the host
// (oplib/opmodel/models/CModel Host Double.cs:434-455): for bucket b of nb (a power of
// two) it stores lb = first z with C[z] > b/nb and ub = first z with C[z] >= (b+1)/nb
// (d-1 for the last bucket or if none), packed lb | ub << 16.  A uniform u with
// floor(u*nb) = b has its answer "smallest z with u < C[z], capped at d-1" in [lb, ub].
#include "common.cuh"
#include "lattice.h"

namespace opb {

// Row-major rows (row y contiguous), four rows a block.  The running sum is a serial chain (its
// order is the definition), so it is what bounds a row: one thread per row walks it out of
// shared memory, 16 bytes at a time, while everything around it -- the loads, the divisions,
// the stores -- is spread over the block.  A row longer than a chunk leaves its running sums
// in C between the chain and the division (every thread reads back what it wrote).
// 512 rows of 512: 110 -> 11 us against one warp per 32 rows, which walked the chain twice and
// did the divisions in the chain's own 16 warps.  Rows of up to 128 entries: k_sck_short.
constexpr int SCK_ROWS = 4, SCK_CHUNK = 1024, SCK_THREADS = 128;

__device__ __forceinline__ float sck_positive(float p) { return p > 0.f ? p : 0.f; }
__device__ __forceinline__ float sck_entry(float acc, float total) {
    const float v = __fdiv_rn(acc, total);
    return v < 1.0f ? v : 1.0f;
}

__global__ void __launch_bounds__(SCK_THREADS) k_sck_rm(int d, int nrows, const float *P, float *C) {
    __shared__ __align__(16) float t[SCK_ROWS][SCK_CHUNK + 4];
    __shared__ float total[SCK_ROWS];
    const int tid = threadIdx.x, r0 = blockIdx.x * SCK_ROWS, nr = min(SCK_ROWS, nrows - r0);
    const long long at = (long long)r0 * d;
    float acc = 0.f;
    for (int c0 = 0; c0 < d; c0 += SCK_CHUNK) {
        const int w = min(SCK_CHUNK, d - c0);
#pragma unroll
        for (int r = 0; r < SCK_ROWS; r++)
            if (r < nr)
                for (int c = tid; c < w; c += SCK_THREADS) t[r][c] = P[at + (long long)r * d + c0 + c];
        __syncthreads();
        if (tid < nr) {
            float *row = t[tid];
            int j = 0;
#pragma unroll 4
            for (; j + 4 <= w; j += 4) {
                float4 q = *reinterpret_cast<float4 *>(row + j);
                q.x = acc = __fadd_rn(acc, sck_positive(q.x));
                q.y = acc = __fadd_rn(acc, sck_positive(q.y));
                q.z = acc = __fadd_rn(acc, sck_positive(q.z));
                q.w = acc = __fadd_rn(acc, sck_positive(q.w));
                *reinterpret_cast<float4 *>(row + j) = q;
            }
            for (; j < w; j++) row[j] = acc = __fadd_rn(acc, sck_positive(row[j]));
            total[tid] = acc;
        }
        __syncthreads();
        if (d > SCK_CHUNK) {
            for (int r = 0; r < nr; r++)
                for (int c = tid; c < w; c += SCK_THREADS) C[at + (long long)r * d + c0 + c] = t[r][c];
            __syncthreads();
        }
    }
    for (int r = 0; r < nr; r++) {
        const float sum = total[r];
        float *out = C + at + (long long)r * d;
        if (d > SCK_CHUNK) {
#pragma unroll 4
            for (int c = tid; c < d; c += SCK_THREADS) out[c] = sck_entry(out[c], sum);
        } else {
#pragma unroll 4
            for (int c = tid; c < d; c += SCK_THREADS) out[c] = sck_entry(t[r][c], sum);
        }
    }
}

// Short rows, 32 a block: one warp walks the chains of all of them, and the block's span of memory is
// contiguous.  With four rows a block the blocks had next to nothing to do: 100,000 rows of 16 took
// 37.5 us (11.4 with a warp per 32 rows; now 7.4), 50,000 of 100 30 us (27; now 13), 20,000 of 128 15 us (17; now 9).
constexpr int SCS_ROWS = 32, SCS_MAX = 128;

__global__ void __launch_bounds__(SCK_THREADS) k_sck_short(int d, int nrows, const float *P, float *C) {
    __shared__ __align__(16) float t[SCS_ROWS][SCS_MAX + 4];
    __shared__ float total[SCS_ROWS];
    const int tid = threadIdx.x, r0 = blockIdx.x * SCS_ROWS, nr = min(SCS_ROWS, nrows - r0), n = nr * d;
    const long long at = (long long)r0 * d;
    const int step_r = SCK_THREADS / d, step_c = SCK_THREADS % d;
    auto each = [&](auto &&f) {  // this thread's entries: index in the span, row, column
        int r = tid / d, c = tid % d;
#pragma unroll 4
        for (int e = tid; e < n; e += SCK_THREADS) {
            f(e, r, c);
            r += step_r;
            c += step_c;
            if (c >= d) {
                c -= d;
                r++;
            }
        }
    };
    each([&](int e, int r, int c) { t[r][c] = P[at + e]; });
    __syncthreads();
    if (tid < nr) {
        float *row = t[tid], acc = 0.f;
        int j = 0;
#pragma unroll 4
        for (; j + 4 <= d; j += 4) {
            float4 q = *reinterpret_cast<float4 *>(row + j);
            q.x = acc = __fadd_rn(acc, sck_positive(q.x));
            q.y = acc = __fadd_rn(acc, sck_positive(q.y));
            q.z = acc = __fadd_rn(acc, sck_positive(q.z));
            q.w = acc = __fadd_rn(acc, sck_positive(q.w));
            *reinterpret_cast<float4 *>(row + j) = q;
        }
        for (; j < d; j++) row[j] = acc = __fadd_rn(acc, sck_positive(row[j]));
        total[tid] = acc;
    }
    __syncthreads();
    each([&](int e, int r, int c) { C[at + e] = sck_entry(t[r][c], total[r]); });
}

// Column-major rows as in the reference: element (y1, y2) at m*d*d + y1 + d*y2, thread
// per (m, y1) -- consecutive threads touch consecutive addresses.
__global__ void k_sck_cm(int d, int nm, const float *__restrict__ P, float *__restrict__ C) {
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)nm * d) return;
    long long m = t / d;
    int y1 = (int)(t - m * d);
    const float *p = P + m * d * (long long)d + y1;
    float *c = C + m * d * (long long)d + y1;
    float acc = 0.f;
    for (int z = 0; z < d; z++) {
        float v = p[(long long)z * d];
        v = v > 0.f ? v : 0.f;
        acc = (z == 0) ? v : __fadd_rn(acc, v);
        c[(long long)z * d] = acc;
    }
    for (int z = 0; z < d; z++) {
        float v = __fdiv_rn(c[(long long)z * d], acc);
        c[(long long)z * d] = v < 1.0f ? v : 1.0f;
    }
}

// 2^shift threads a row, a thread per bucket boundary pair, 256 >> shift rows a block.  The searches
// are chains of dependent loads, so a table of few rows gets a block a row, and the row is
// searched in shared memory as long as it fits (GUIDE_STAGED floats).  512 rows, 1024
// buckets: 37 -> 8 us against one warp per row searching in L1.  Many rows fill the SMs with a warp
// each: 50,000 rows of 64, 64 buckets 52 us with a block a row, 25 with a warp; and rows much longer
// than their buckets are cheaper to probe than to read: 4096 of 4096, 1 bucket 10.9 us staged, 6.7.
constexpr int GUIDE_THREADS = 256, GUIDE_STAGED = 48 * 1024 / 4;

template <bool STAGED>
__global__ void __launch_bounds__(GUIDE_THREADS) k_guide(int d, int nrows, int nb, int shift,
                                                         const float *__restrict__ C, uint32_t *__restrict__ guide) {
    extern __shared__ float staged[];
    const int per_row = 1 << shift, rows = GUIDE_THREADS >> shift, r0 = blockIdx.x * rows;
    const int mine = (int)threadIdx.x >> shift;
    const float *row = C + (long long)(r0 + mine) * d;
    if constexpr (STAGED) {
        const int n = min(rows, nrows - r0) * d;
        for (int c = threadIdx.x; c < n; c += GUIDE_THREADS) staged[c] = C[(long long)r0 * d + c];
        __syncthreads();
        row = staged + mine * d;
    }
    if (r0 + mine >= nrows) return;
    const float inv = 1.0f / (float)nb;  // exact: nb is a power of two
    for (int b = threadIdx.x & (per_row - 1); b < nb; b += per_row) {
        float lo_t = (float)b * inv, hi_t = (float)(b + 1) * inv;
        // first z with C[z] > lo_t (binary search on the non-decreasing row)
        int lo = 0, hi = d;  // answer in [lo, hi], d = none
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (row[mid] > lo_t) hi = mid; else lo = mid + 1;
        }
        int lb = lo < d ? lo : d - 1;
        int ub;
        if (b == nb - 1) {
            ub = d - 1;
        } else {
            lo = 0; hi = d;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (row[mid] >= hi_t) hi = mid; else lo = mid + 1;
            }
            ub = lo < d ? lo : d - 1;
        }
        if (ub < lb) ub = lb;
        guide[(long long)(r0 + mine) * nb + b] = (uint32_t)lb | ((uint32_t)ub << 16);
    }
}

int launch_sck_rm(int d, int nrows, const float *P, float *C, cudaStream_t s) {
    if (d <= SCS_MAX) k_sck_short<<<(nrows + SCS_ROWS - 1) / SCS_ROWS, SCK_THREADS, 0, s>>>(d, nrows, P, C);
    else k_sck_rm<<<(nrows + SCK_ROWS - 1) / SCK_ROWS, SCK_THREADS, 0, s>>>(d, nrows, P, C);
    return (int)cudaGetLastError();
}

int launch_guide(int d, int nrows, int nb, const float *C, uint32_t *guide, cudaStream_t s) {
    // tables of few rows: a block a row.  Else a warp a row, twice that and so on while the threads are
    // fewer than 2^18 and no more than the buckets, or a thread would search 32 buckets or more, or
    // the block's rows would leave it fewer than three neighbours on its SM
    int shift = 8;
    bool staged = d <= GUIDE_STAGED;
    if (nrows >= 2048) {
        staged = staged && d < 32 * nb;
        for (shift = 5; shift < 8; shift++) {
            const long long per_row = 1LL << shift;
            if (!((nb > per_row && nrows * per_row < 1 << 18) || nb >= 32 * per_row || (staged && (d << (8 - shift)) > 4096)))
                break;
        }
    }
    const int rows = GUIDE_THREADS >> shift, grid = (nrows + rows - 1) / rows;
    if (staged) k_guide<true><<<grid, GUIDE_THREADS, rows * d * sizeof(float), s>>>(d, nrows, nb, shift, C, guide);
    else k_guide<false><<<grid, GUIDE_THREADS, 0, s>>>(d, nrows, nb, shift, C, guide);
    return (int)cudaGetLastError();
}

}  // namespace opb

// Reference entry point: nm column-major d x d kernels -> cumulative rows
// (oplib/opcuda/sck.cu:88-93).
OPB_API int opcuda_sck(int d, int nm, uint64_t tpker_yy_m, uint64_t ctpker_yy_m) {
    OPB_REQUIRE(d >= 0 && nm >= 0, OPB_E_ARG);
    if (d == 0 || nm == 0) return opb::set_status(OPB_OK);
    OPB_REQUIRE(tpker_yy_m != 0 && ctpker_yy_m != 0, OPB_E_NULL);
    long long n = (long long)nm * d;
    opb::k_sck_cm<<<(int)((n + 127) / 128), 128, 0, opb::stream()>>>(
        d, nm, reinterpret_cast<const float *>(tpker_yy_m), reinterpret_cast<float *>(ctpker_yy_m));
    return opb::launch_check();
}

// Row-major (source-major) cumulative rows for nrows rows of length d.
OPB_API int opb_sck_rm(int d, int nrows, const float *P, float *C) {
    OPB_REQUIRE(d > 0 && nrows >= 0, OPB_E_ARG);
    if (nrows == 0) return opb::set_status(OPB_OK);
    OPB_REQUIRE(P && C, OPB_E_NULL);
    return opb::set_status(opb::launch_sck_rm(d, nrows, P, C, opb::stream()));
}

OPB_API int opb_guide_table(int d, int nrows, int nb, const float *C, uint32_t *guide) {
    OPB_REQUIRE(d > 0 && d <= 65535 && nrows >= 0, OPB_E_ARG);
    OPB_REQUIRE(nb >= 1 && nb <= 4096 && (nb & (nb - 1)) == 0, OPB_E_ARG);
    if (nrows == 0) return opb::set_status(OPB_OK);
    OPB_REQUIRE(C && guide, OPB_E_NULL);
    return opb::set_status(opb::launch_guide(d, nrows, nb, C, guide, opb::stream()));
}
