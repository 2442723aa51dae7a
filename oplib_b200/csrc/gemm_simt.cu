// Plain FP32 GEMM on the SIMT FMA pipes (no tensor cores, no TF32).
//
// This is the "plain FP32" path behind the drop-in entry points
//   opcuda_sgemm  (oplib/opcuda/sgemm.cu:41-44, column-major, alpha/beta),
//   opcuda_ssqmm  (oplib/opcuda/ssqmm.cu:119-179, batched d x d via device pointer tables),
//   opcuda_sgemm4 (oplib/opcuda/sgemm4.cu:84-154, ragged batch through a per-block task table).
// The reference kernels are 64x16-tile Volkov-style SIMT loops for sm_1x; here large products
// take row-major 128x128 CTA tiles with 8x8 outputs per thread, small ones and the task tables
// tiles of a warp each (below).
// Column-major calls are mapped onto it through C^T = B^T . A^T (a column-major matrix
// is the row-major storage of its transpose), so the kernel never transposes data.
#include <type_traits>

#include "common.cuh"

namespace opb {

constexpr int SG_BM = 128, SG_BN = 128, SG_BK = 8, SG_THREADS = 256;
constexpr int SG_APAD = 4;  // keeps the transposed A tile's stores off one bank

struct SgemmArgs {
    int M, N, K;
    int lda, ldb, ldc;
    float alpha, beta;
    const float *A;
    const float *B;
    float *C;
    // batching: either pointer tables (row-major roles) or strides
    const float *const *A_tab;
    const float *const *B_tab;
    float *const *C_tab;
    long long sA, sB, sC;
};

// Row-major C[M,N] = alpha * op(A)[M,K] . op(B)[K,N] + beta * C; TA: A stored K x M
// (element (m,k) at k*lda + m), TB: B stored N x K (element (k,n) at n*ldb + k).
// grid = (ceil(N/128), ceil(M/128), batch)
template <bool TA, bool TB>
__global__ void __launch_bounds__(SG_THREADS, 2) k_sgemm_rm(SgemmArgs p) {
    __shared__ __align__(16) float As[2][SG_BK][SG_BM + SG_APAD];
    __shared__ __align__(16) float Bs[2][SG_BK][SG_BN];

    const int z = blockIdx.z;
    const float *A = p.A_tab ? p.A_tab[z] : p.A + z * p.sA;
    const float *B = p.B_tab ? p.B_tab[z] : p.B + z * p.sB;
    float *C = p.C_tab ? p.C_tab[z] : p.C + z * p.sC;

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * SG_BM, n0 = blockIdx.x * SG_BN;

    // global -> register staging coordinates
    const int a_row = tid >> 1, a_k = (tid & 1) * 4;   // 128 rows x 8 k
    const int b_k = tid >> 5, b_col = (tid & 31) * 4;  // 8 k x 128 cols

    float ra[4], rb[4];
    auto load_tiles = [&](int k0) {
        int gr = m0 + a_row;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int gk = k0 + a_k + j;
            ra[j] = (gr < p.M && gk < p.K)
                        ? __ldg(TA ? A + (long long)gk * p.lda + gr : A + (long long)gr * p.lda + gk)
                        : 0.f;
        }
        int gk = k0 + b_k;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int gc = n0 + b_col + j;
            rb[j] = (gk < p.K && gc < p.N)
                        ? __ldg(TB ? B + (long long)gc * p.ldb + gk : B + (long long)gk * p.ldb + gc)
                        : 0.f;
        }
    };
    auto store_tiles = [&](int buf) {
#pragma unroll
        for (int j = 0; j < 4; j++) As[buf][a_k + j][a_row] = ra[j];
        *reinterpret_cast<float4 *>(&Bs[buf][b_k][b_col]) = make_float4(rb[0], rb[1], rb[2], rb[3]);
    };

    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;

    const int nk = (p.K + SG_BK - 1) / SG_BK;
    load_tiles(0);
    store_tiles(0);
    __syncthreads();

    for (int t = 0; t < nk; t++) {
        const int buf = t & 1;
        if (t + 1 < nk) load_tiles((t + 1) * SG_BK);
#pragma unroll
        for (int k = 0; k < SG_BK; k++) {
            float a[8], b[8];
            float4 a0 = *reinterpret_cast<const float4 *>(&As[buf][k][ty * 4]);
            float4 a1 = *reinterpret_cast<const float4 *>(&As[buf][k][64 + ty * 4]);
            float4 b0 = *reinterpret_cast<const float4 *>(&Bs[buf][k][tx * 4]);
            float4 b1 = *reinterpret_cast<const float4 *>(&Bs[buf][k][64 + tx * 4]);
            a[0] = a0.x; a[1] = a0.y; a[2] = a0.z; a[3] = a0.w;
            a[4] = a1.x; a[5] = a1.y; a[6] = a1.z; a[7] = a1.w;
            b[0] = b0.x; b[1] = b0.y; b[2] = b0.z; b[3] = b0.w;
            b[4] = b1.x; b[5] = b1.y; b[6] = b1.z; b[7] = b1.w;
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (t + 1 < nk) {
            store_tiles(buf ^ 1);
        }
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 8; i++) {
        int r = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
        if (r >= p.M) continue;
        float *crow = C + (long long)r * p.ldc;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            int c = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + (j - 4));
            if (c >= p.N) continue;
            float v = p.alpha * acc[i][j];
            if (p.beta != 0.f) v = fmaf(p.beta, crow[c], v);
            crow[c] = v;
        }
    }
}

// ---- the pipelined form for whole tiles (row-major A and B, M and N multiples of 128, K of
// 16, 16-byte aligned rows, no pointer tables): K in steps of 16 through a 3-stage
// cp.async ring (A rows padded to 20 floats, so the two row groups of a warp fall on
// different banks), each thread 8 x 8 outputs from 128-bit shared loads of A along k and of
// B along n.  Every output still sums its products in k order, so the results are
// bit-identical to k_sgemm_rm's.
constexpr int SF_BK = 16, SF_STAGES = 3, SF_APITCH = SF_BK + 4;
constexpr int SF_A_FLOATS = SG_BM * SF_APITCH, SF_B_FLOATS = SF_BK * SG_BN;
constexpr int SF_SMEM = SF_STAGES * (SF_A_FLOATS + SF_B_FLOATS) * 4;

__device__ __forceinline__ void sf_cp16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void sf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void sf_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Packed FP32 (sm_100): two independent FMAs per lane and instruction, each rounded as a
// scalar fmaf, so every output still sums its products in k order with the same bits.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__global__ void __launch_bounds__(SG_THREADS, 2) k_sgemm_pipe(SgemmArgs p) {
    extern __shared__ __align__(16) float sm[];
    const int z = blockIdx.z;
    const float *A = p.A + z * p.sA;
    const float *B = p.B + z * p.sB;
    float *C = p.C + z * p.sC;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * SG_BM, n0 = blockIdx.x * SG_BN;
    const float *Ab = A + (long long)m0 * p.lda;
    const float *Bb = B + n0;

    auto issue = [&](int stage, int k0) {
        float *As = sm + stage * (SF_A_FLOATS + SF_B_FLOATS);
        float *Bs = As + SF_A_FLOATS;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int c = tid + SG_THREADS * i;
            const int row = c >> 2, kq = (c & 3) * 4;  // 128 rows x 4 chunks of 4 floats
            sf_cp16(As + row * SF_APITCH + kq, Ab + (long long)row * p.lda + k0 + kq);
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int c = tid + SG_THREADS * i;
            const int kr = c >> 5, col = (c & 31) * 4;  // 16 rows x 32 chunks of 4 floats
            sf_cp16(Bs + kr * SG_BN + col, Bb + (long long)(k0 + kr) * p.ldb + col);
        }
        sf_commit();
    };

    // acc2[i][jp] holds the outputs (row i, columns 2jp and 2jp + 1) of this thread's 8 x 8
    uint64_t acc2[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc2[i][j] = 0ull;

    const int nk = p.K / SF_BK;
#pragma unroll
    for (int st = 0; st < SF_STAGES - 1; st++) {
        if (st < nk) issue(st, st * SF_BK);
        else sf_commit();
    }
    for (int kt = 0; kt < nk; kt++) {
        sf_wait<SF_STAGES - 2>();
        __syncthreads();  // stage kt landed for every thread; stage kt - 1 is free to refill
        const int nt = kt + SF_STAGES - 1;
        if (nt < nk) issue(nt % SF_STAGES, nt * SF_BK);
        else sf_commit();
        const float *As = sm + (kt % SF_STAGES) * (SF_A_FLOATS + SF_B_FLOATS);
        const float *Bs = As + SF_A_FLOATS;
#pragma unroll
        for (int kk = 0; kk < SF_BK; kk += 4) {
            float4 a4[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int row = i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4);
                a4[i] = *reinterpret_cast<const float4 *>(As + row * SF_APITCH + kk);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float4 b0 = *reinterpret_cast<const float4 *>(Bs + (kk + u) * SG_BN + tx * 4);
                const float4 b1 = *reinterpret_cast<const float4 *>(Bs + (kk + u) * SG_BN + 64 + tx * 4);
                const uint64_t b2[4] = {f2_pack(b0.x, b0.y), f2_pack(b0.z, b0.w), f2_pack(b1.x, b1.y),
                                        f2_pack(b1.z, b1.w)};
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float a = u == 0 ? a4[i].x : u == 1 ? a4[i].y : u == 2 ? a4[i].z : a4[i].w;
                    const uint64_t a2 = f2_pack(a, a);
#pragma unroll
                    for (int j = 0; j < 4; j++) acc2[i][j] = f2_fma(a2, b2[j], acc2[i][j]);
                }
            }
        }
    }
    sf_wait<0>();

    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) f2_unpack(acc2[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
        float *crow = C + (long long)r * p.ldc + n0;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float4 *cp = reinterpret_cast<float4 *>(crow + h * 64 + tx * 4);
            float4 v = make_float4(p.alpha * acc[i][4 * h], p.alpha * acc[i][4 * h + 1], p.alpha * acc[i][4 * h + 2],
                                   p.alpha * acc[i][4 * h + 3]);
            if (p.beta != 0.f) {
                const float4 c = *cp;
                v.x = fmaf(p.beta, c.x, v.x);
                v.y = fmaf(p.beta, c.y, v.y);
                v.z = fmaf(p.beta, c.z, v.z);
                v.w = fmaf(p.beta, c.w, v.w);
            }
            *cp = v;
        }
    }
}

// ---- small tiles: a warp computes 8 RPT x 16 outputs (a thread RPT x 4), for products whose
// 128 x 128 tiles leave SMs idle, and for the task tables, whose tiles are 64 x 16.
//
// The tile is written column-major (X contiguous in the left operand and in C, K contiguous in
// the right one), which is what the tables hold; a row-major product is C^T = B^T . A^T.  K runs
// in steps of 16 through a ring of shared stages filled by 16-byte cp.async (4-byte ones where an
// operand's rows are not 16-byte aligned), each operand as it lies in memory: transposing the
// right one with 4-byte copies cost about a cycle an element, 1000 cycles a stage (512^3: 27 us
// whatever the tile).  Four steps of K at a time, a thread issues four to eight 128-bit loads of
// the left tile (its X pairs come packed), four of the right one (along K, each value duplicated
// by a move) and 4 RPT / 2 x 4 packed FMAs, so the FMA pipe is what bounds it.  Every output
// sums its products in k order with fma, as the other kernels here do: the same bits.
constexpr int ST_BK = 16, ST_STAGES = 4;

// 16 bytes of global memory into shared memory, bytes beyond `valid` as zeros (valid 0: all).
__device__ __forceinline__ void st_cp16(float *dst, const float *src, int valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid)
                 : "memory");
}
__device__ __forceinline__ void st_cp4(float *dst, const float *src, int valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid)
                 : "memory");
}

// A stage's left tile: X columns [x0, x0 + TX) of K rows [k0, k0 + 16), element (x, k) at
// A[k * lda + x], into dst[k][x] (pitch floats a row), by `nthr` threads of which this is `tid`.
template <int TX>
__device__ __forceinline__ void st_load_a(float *dst, int pitch, const float *A, long long lda, int X, int K, int x0,
                                          int k0, bool vec, int tid, int nthr) {
    if (vec) {
        for (int e = tid; e < ST_BK * TX / 4; e += nthr) {
            const int k = e / (TX / 4), x = (e % (TX / 4)) * 4;
            const int left = k0 + k < K ? X - (x0 + x) : 0;
            const int valid = left >= 4 ? 16 : left > 0 ? 4 * left : 0;
            st_cp16(dst + k * pitch + x, valid ? A + (long long)(k0 + k) * lda + x0 + x : A, valid);
        }
    } else {
        for (int e = tid; e < ST_BK * TX; e += nthr) {
            const int k = e / TX, x = e % TX;
            const bool in = k0 + k < K && x0 + x < X;
            st_cp4(dst + k * pitch + x, in ? A + (long long)(k0 + k) * lda + x0 + x : A, in ? 4 : 0);
        }
    }
}
// A stage's right tile: Y columns [y0, y0 + TY), element (k, y) at B[y * ldb + k], into
// dst[y * ST_BP + k].
constexpr int ST_BP = ST_BK + 4;  // four neighbouring y fall on different banks
template <int TY>
__device__ __forceinline__ void st_load_b(float *dst, const float *B, long long ldb, int Y, int K, int y0, int k0,
                                          bool vec, int tid, int nthr) {
    if (vec) {
        for (int e = tid; e < ST_BK * TY / 4; e += nthr) {
            const int k = (e % (ST_BK / 4)) * 4, y = e / (ST_BK / 4);
            const int left = y0 + y < Y ? K - (k0 + k) : 0;
            const int valid = left >= 4 ? 16 : left > 0 ? 4 * left : 0;
            st_cp16(dst + y * ST_BP + k, valid ? B + (long long)(y0 + y) * ldb + k0 + k : B, valid);
        }
    } else {
        for (int e = tid; e < ST_BK * TY; e += nthr) {
            const int k = e % ST_BK, y = e / ST_BK;
            const bool in = k0 + k < K && y0 + y < Y;
            st_cp4(dst + y * ST_BP + k, in ? B + (long long)(y0 + y) * ldb + k0 + k : B, in ? 4 : 0);
        }
    }
}

// One step of K: this thread's X values at `as` (and, RPT = 8, 32 further on) times its four Y values.
template <int RPT>
__device__ __forceinline__ void st_step(uint64_t (&acc)[RPT / 2][4], const float *as, float b0, float b1, float b2,
                                        float b3) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2 *>(as);
    ulonglong2 a1 = a0;
    if constexpr (RPT == 8) a1 = *reinterpret_cast<const ulonglong2 *>(as + 32);
    const uint64_t bb[4] = {f2_pack(b0, b0), f2_pack(b1, b1), f2_pack(b2, b2), f2_pack(b3, b3)};
    const uint64_t aa[4] = {a0.x, a0.y, a1.x, a1.y};
#pragma unroll
    for (int i = 0; i < RPT / 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = f2_fma(aa[i], bb[j], acc[i][j]);
}
// A stage of kn (<= 16) steps; the thread's Y columns are 4 apart, from bs on.
template <int RPT>
__device__ __forceinline__ void st_steps(uint64_t (&acc)[RPT / 2][4], const float *as, int ap, const float *bs, int kn) {
    if (kn == ST_BK) {
#pragma unroll
        for (int k = 0; k < ST_BK; k += 4) {
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4 *>(bs + 4 * j * ST_BP + k);
            st_step<RPT>(acc, as + k * ap, b[0].x, b[1].x, b[2].x, b[3].x);
            st_step<RPT>(acc, as + (k + 1) * ap, b[0].y, b[1].y, b[2].y, b[3].y);
            st_step<RPT>(acc, as + (k + 2) * ap, b[0].z, b[1].z, b[2].z, b[3].z);
            st_step<RPT>(acc, as + (k + 3) * ap, b[0].w, b[1].w, b[2].w, b[3].w);
        }
    } else {
        for (int k = 0; k < kn; k++)
            st_step<RPT>(acc, as + k * ap, bs[k], bs[4 * ST_BP + k], bs[8 * ST_BP + k], bs[12 * ST_BP + k]);
    }
}
// Two right tiles against one left tile: its values are read once for both.
template <int RPT>
__device__ __forceinline__ void st_steps2(uint64_t (&acc0)[RPT / 2][4], uint64_t (&acc1)[RPT / 2][4], const float *as,
                                          int ap, const float *bs0, const float *bs1, int kn) {
    if (kn == ST_BK) {
#pragma unroll
        for (int k = 0; k < ST_BK; k += 4) {
            float4 b[4], c[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                b[j] = *reinterpret_cast<const float4 *>(bs0 + 4 * j * ST_BP + k);
                c[j] = *reinterpret_cast<const float4 *>(bs1 + 4 * j * ST_BP + k);
            }
            st_step<RPT>(acc0, as + k * ap, b[0].x, b[1].x, b[2].x, b[3].x);
            st_step<RPT>(acc1, as + k * ap, c[0].x, c[1].x, c[2].x, c[3].x);
            st_step<RPT>(acc0, as + (k + 1) * ap, b[0].y, b[1].y, b[2].y, b[3].y);
            st_step<RPT>(acc1, as + (k + 1) * ap, c[0].y, c[1].y, c[2].y, c[3].y);
            st_step<RPT>(acc0, as + (k + 2) * ap, b[0].z, b[1].z, b[2].z, b[3].z);
            st_step<RPT>(acc1, as + (k + 2) * ap, c[0].z, c[1].z, c[2].z, c[3].z);
            st_step<RPT>(acc0, as + (k + 3) * ap, b[0].w, b[1].w, b[2].w, b[3].w);
            st_step<RPT>(acc1, as + (k + 3) * ap, c[0].w, c[1].w, c[2].w, c[3].w);
        }
    } else {
        st_steps<RPT>(acc0, as, ap, bs0, kn);
        st_steps<RPT>(acc1, as, ap, bs1, kn);
    }
}
// Stores this thread's outputs: rows x.. (and x + 32..), columns y, y + 4, y + 8, y + 12 of
// column-major C.
template <int RPT>
__device__ __forceinline__ void st_store(const uint64_t (&acc)[RPT / 2][4], float *C, long long ldc, int X, int Y, int x,
                                         int y, float alpha, float beta, bool vec) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (y + 4 * j >= Y) continue;
#pragma unroll
        for (int h = 0; h < RPT / 4; h++) {
            float v[4];
            f2_unpack(acc[2 * h][j], v[0], v[1]);
            f2_unpack(acc[2 * h + 1][j], v[2], v[3]);
            float *c = C + (long long)(y + 4 * j) * ldc + x + 32 * h;
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] *= alpha;
            if (vec && x + 32 * h + 4 <= X) {
                if (beta != 0.f) {
                    const float4 o = *reinterpret_cast<const float4 *>(c);
                    v[0] = fmaf(beta, o.x, v[0]); v[1] = fmaf(beta, o.y, v[1]);
                    v[2] = fmaf(beta, o.z, v[2]); v[3] = fmaf(beta, o.w, v[3]);
                }
                *reinterpret_cast<float4 *>(c) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (x + 32 * h + i < X) c[i] = beta != 0.f ? fmaf(beta, c[i], v[i]) : v[i];
            }
        }
    }
}

// Row-major C[M,N] = alpha * A . B + beta * C on tiles of 8 RPT WX columns of N x 16 WY rows of M;
// grid (N tiles, M tiles, batch).
template <int RPT, int WX, int WY>
__global__ void __launch_bounds__(32 * WX * WY) k_sgemm_small(SgemmArgs p) {
    constexpr int TX = 8 * RPT * WX, TY = 16 * WY, AP = TX + 4, NT = 32 * WX * WY;
    __shared__ __align__(16) float As[ST_STAGES][ST_BK * AP], Bs[ST_STAGES][TY * ST_BP];
    const int z = blockIdx.z;
    const float *L = p.B_tab ? p.B_tab[z] : p.B + z * p.sB;  // K x N: X contiguous
    const float *R = p.A_tab ? p.A_tab[z] : p.A + z * p.sA;  // M x K: K contiguous
    float *C = p.C_tab ? p.C_tab[z] : p.C + z * p.sC;
    auto al = [](const void *q, long long ld) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0 && ld % 4 == 0; };
    const bool vl = al(L, p.ldb), vr = al(R, p.lda), vc = al(C, p.ldc);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const int xl = (warp % WX) * 8 * RPT + (lane & 7) * 4, yl = (warp / WX) * 16 + (lane >> 3);
    uint64_t acc[RPT / 2][4];
#pragma unroll
    for (int i = 0; i < RPT / 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0ull;
    const int nk = (p.K + ST_BK - 1) / ST_BK;
    auto load = [&](int t) {
        if (t < nk) {
            st_load_a<TX>(As[t % ST_STAGES], AP, L, p.ldb, p.N, p.K, x0, t * ST_BK, vl, tid, NT);
            st_load_b<TY>(Bs[t % ST_STAGES], R, p.lda, p.M, p.K, y0, t * ST_BK, vr, tid, NT);
        }
        sf_commit();
    };
#pragma unroll
    for (int t = 0; t < ST_STAGES - 1; t++) load(t);
    for (int t = 0; t < nk; t++) {
        sf_wait<ST_STAGES - 2>();
        __syncthreads();  // stage t has landed for every thread; stage t - 1 is free to refill
        load(t + ST_STAGES - 1);
        st_steps<RPT>(acc, As[t % ST_STAGES] + xl, AP, Bs[t % ST_STAGES] + yl * ST_BP, min(ST_BK, p.K - t * ST_BK));
    }
    st_store<RPT>(acc, C, p.ldc, p.N, p.M, x0 + xl, y0 + yl, p.alpha, p.beta, vc);
}

static bool sgemm_pipe_ok(const SgemmArgs &a, int batch) {
    auto al = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    return !a.A_tab && !a.B_tab && !a.C_tab && a.M % SG_BM == 0 && a.N % SG_BN == 0 && a.K % SF_BK == 0 &&
           a.K > 0 && a.lda % 4 == 0 && a.ldb % 4 == 0 && a.ldc % 4 == 0 && al(a.A) && al(a.B) && al(a.C) &&
           (batch == 1 || (a.sA % 4 == 0 && a.sB % 4 == 0 && a.sC % 4 == 0));
}

// Which kernel a plain product runs on, by the measured times (B200, us; small = k_sgemm_small):
//   aligned, whole 128-tiles   512^3: small 22, pipe 58; 1024^3: 79, 112; 1280^3 (100 tiles): 130,
//                              140; 1408^3 (121): 177, 152; 4096^3: 3272, 2712 -> the pipe from 112 tiles on
//   aligned, ragged            577 .. 4100: small at every size (4100^3: 3394 against 3576 of k_sgemm_rm)
//   rows off the 16-byte grid  small_tiles_win (the 4-byte copies)
// and of the small tiles 64 x 64 from 240 of them on (1000^3: 79 against 79), 64 x 32 below.
constexpr int SG_PIPE_TILES = 112, ST_WIDE_TILES = 240;

// k_sgemm_small against k_sgemm_rm where the rows of A or B are off the 16-byte grid, by their leading
// dimension or by their base: the first then copies 4 bytes at a time, the second loads that way at
// any alignment.  Both go by the tiles of the busiest SM, in us per unit of K: 128 x 128 ones in pairs
// (0.235 a pair, 0.14 alone; a fifth more with A off the grid at a multiple of 128 bytes, where every
// row's 64 bytes take a further sector), 64 x 64 ones at 0.0333 each with one operand off the grid,
// 0.038 with both, and 0.02.  Measured, us, small / rm, A off, B off, both:
//   1500^3  223/203 221/205 250/203     2560^3   958/1340  958/933  1087/1339
//   1536^3  227/228 226/217 256/228     3000^3  1512/1328 1509/1325 1714/1328
//   1664^3  300/443 300/407 339/443     4096^3  3777/4275 3773/3577 4293/4275
//   2048^3  502/544 502/512 568/544     64 x 256^3 68/75    68/72     76/75
static bool small_tiles_win(const SgemmArgs &a, int batch) {
    auto off = [&](const float *q, const void *tab, int ld, long long stride) {
        return ld % 4 || (!tab && (reinterpret_cast<uintptr_t>(q) % 16 || (batch > 1 && stride % 4)));
    };
    const bool a4 = off(a.A, a.A_tab, a.lda, a.sA), b4 = off(a.B, a.B_tab, a.ldb, a.sB);
    if (!a4 && !b4) return true;
    auto busiest = [&](int t) {
        const long long n = (long long)((a.M + t - 1) / t) * ((a.N + t - 1) / t) * batch;
        return (n + num_sms() - 1) / num_sms();
    };
    const long long u = busiest(128);
    const double rm = (0.235 * (u / 2) + 0.14 * (u % 2)) * (a4 && a.lda % 32 == 0 ? 1.2 : 1.0);
    return (a4 && b4 ? 0.038 : 0.0333) * busiest(64) + 0.02 < rm;
}

int sgemm_rowmajor(const SgemmArgs &a, int batch, cudaStream_t s, bool ta = false, bool tb = false) {
    if (a.M <= 0 || a.N <= 0 || batch <= 0) return OPB_OK;
    const long long tiles = (long long)((a.M + SG_BM - 1) / SG_BM) * ((a.N + SG_BN - 1) / SG_BN) * batch;
    const bool pipe = !ta && !tb && sgemm_pipe_ok(a, batch) && tiles >= SG_PIPE_TILES;
    if (!ta && !tb && !pipe && small_tiles_win(a, batch) && a.M <= 65535 * 64) {  // (grid rows)
        const dim3 g64((a.N + 63) / 64, (a.M + 63) / 64, batch);
        if ((long long)g64.x * g64.y * g64.z >= ST_WIDE_TILES) k_sgemm_small<8, 1, 4><<<g64, 128, 0, s>>>(a);
        else k_sgemm_small<4, 2, 2><<<dim3(g64.x, (a.M + 31) / 32, batch), 128, 0, s>>>(a);
        return static_cast<int>(cudaGetLastError());
    }
    if (pipe) {
        static bool attr[64] = {false};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev >= 0 && dev < 64 && !attr[dev]) {
            cudaError_t e = cudaFuncSetAttribute(k_sgemm_pipe, cudaFuncAttributeMaxDynamicSharedMemorySize, SF_SMEM);
            if (e != cudaSuccess) return (int)e;
            attr[dev] = true;
        }
        dim3 grid(a.N / SG_BN, a.M / SG_BM, batch);
        k_sgemm_pipe<<<grid, SG_THREADS, SF_SMEM, s>>>(a);
        return static_cast<int>(cudaGetLastError());
    }
    dim3 grid((a.N + SG_BN - 1) / SG_BN, (a.M + SG_BM - 1) / SG_BM, batch);
    if (!ta && !tb) k_sgemm_rm<false, false><<<grid, SG_THREADS, 0, s>>>(a);
    else if (ta && !tb) k_sgemm_rm<true, false><<<grid, SG_THREADS, 0, s>>>(a);
    else if (!ta && tb) k_sgemm_rm<false, true><<<grid, SG_THREADS, 0, s>>>(a);
    else k_sgemm_rm<true, true><<<grid, SG_THREADS, 0, s>>>(a);
    return static_cast<int>(cudaGetLastError());
}

// Row-major with transpose flags (see k_sgemm_rm).
int sgemm_rm_t(bool ta, bool tb, int M, int N, int K, float alpha, const float *A, int lda, const float *B, int ldb,
               float beta, float *C, int ldc, cudaStream_t s) {
    SgemmArgs a{};
    a.M = M; a.N = N; a.K = K; a.lda = lda; a.ldb = ldb; a.ldc = ldc;
    a.alpha = alpha; a.beta = beta; a.A = A; a.B = B; a.C = C;
    return sgemm_rowmajor(a, 1, s, ta, tb);
}

int sgemm_rm_strided(bool ta, bool tb, int M, int N, int K, float alpha, const float *A, int lda, long long sA,
                     const float *B, int ldb, long long sB, float beta, float *C, int ldc, long long sC, int batch,
                     cudaStream_t s) {
    SgemmArgs a{};
    a.M = M; a.N = N; a.K = K; a.lda = lda; a.ldb = ldb; a.ldc = ldc;
    a.alpha = alpha; a.beta = beta; a.A = A; a.B = B; a.C = C; a.sA = sA; a.sB = sB; a.sC = sC;
    return sgemm_rowmajor(a, batch, s, ta, tb);
}

// Convenience: row-major, unbatched.
int sgemm_rm(int M, int N, int K, float alpha, const float *A, int lda, const float *B, int ldb,
             float beta, float *C, int ldc, cudaStream_t s) {
    SgemmArgs a{};
    a.M = M; a.N = N; a.K = K; a.lda = lda; a.ldb = ldb; a.ldc = ldc;
    a.alpha = alpha; a.beta = beta; a.A = A; a.B = B; a.C = C;
    return sgemm_rowmajor(a, 1, s);
}

// ------------------------------------------------------------------ sgemm4 task tables

// One task per block, widened from the reference's 9-word record
// {i, bx, by, m, n, k, A, B, C} (oplib/opcuda/sgemm4.cu:84-102): the block computes the
// column-major C tile rows [bx*64, bx*64+64) x columns [by*16, by*16+16) of
// C = A . B with lda = m, ldb = k, ldc = m.
struct Sgemm4Task {
    int32_t i, bx, by, m, n, k;
    uint64_t A, B, C;
};

// A block takes one, two or four consecutive tasks.  Neighbouring tasks of a table mostly share
// a tile (the same rows of A along by, the same columns of B along bx), so each distinct tile is
// staged once for the warps that read it, and a warp that has two tasks with one left tile reads
// it from shared memory once for both: with one task a warp those reads, not the FMAs, were the
// limit.  Tasks that share nothing stage their own.  What a block computes does not depend on
// which they share.  (One 64 x 16 tile per 256-thread block, every operand of A from L1: 9.2
// TFLOP/s over 40 products of 576^3, 1657 us; a task a warp 466; now 417.)
//
constexpr int S4_TASKS = 4, S4_THREADS = 16 * S4_TASKS, S4_AP = 64 + 4;
// Tasks a block takes: one (half of its rows a warp) in tables of up to three tasks an SM, where a
// task's own chain over K is the time, two (a warp each) up to fifteen, four (two a warp) beyond.
// Measured, us, one tile per 256-thread block / now: 20 tasks of K = 300 29 / 17, 400 33 / 21, one
// product of 576^3 (324 tasks) 58 / 35; at 2 / 4 tasks a block: 800 39 / 60, 1296 78 / 94, 3000
// 97 / 97, 5184 218 / 201, 12960 515 / 417.
constexpr int S4_ONE = 3, S4_PAIR = 15;
constexpr int S4_A = ST_BK * S4_AP, S4_B = 16 * ST_BP;   // floats of a left, a right tile
// Shared memory of a block: three stages of tasks that share their left tile, or of strangers'
// tiles one; six blocks an SM (two stages of strangers, 45 KB, left four: 447 us).
constexpr int S4_POOL = 3 * (S4_A + S4_TASKS * S4_B);
static_assert(4 * S4_POOL <= 48 * 1024 && S4_POOL >= S4_TASKS * (S4_A + S4_B), "default limit; a stage of strangers");

template <int PER>
__global__ void __launch_bounds__(S4_THREADS) k_sgemm4(const uint64_t *argptr_bid, int ntasks) {
    __shared__ Sgemm4Task task[S4_TASKS];
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cnt = min(PER, ntasks - (int)blockIdx.x * PER);
    if (tid < cnt) task[tid] = *reinterpret_cast<const Sgemm4Task *>(argptr_bid[blockIdx.x * PER + tid]);
    __syncthreads();
    // the tiles of each task, as offsets (floats) into a stage: those of the first task that has
    // the same one
    int oa[S4_TASKS], ob[S4_TASKS], stage = 0, kmax = 0;
    uint32_t owner = 0;  // bits i, 4 + i: task i stages its own left, right tile
#pragma unroll
    for (int i = 0; i < S4_TASKS; i++) {
        oa[i] = ob[i] = 0;
        if (i >= cnt) continue;
        const Sgemm4Task &t = task[i];
        kmax = max(kmax, t.k);
        int ja = i, jb = i;
#pragma unroll
        for (int j = i - 1; j >= 0; j--) {
            const Sgemm4Task &u = task[j];
            if (u.A == t.A && u.m == t.m && u.k == t.k && u.bx == t.bx) ja = j;
            if (u.B == t.B && u.n == t.n && u.k == t.k && u.by == t.by) jb = j;
        }
        if (ja == i) {
            owner |= 1u << i;
            oa[i] = stage;
            stage += S4_A;
        }
        if (jb == i) {
            owner |= 16u << i;
            ob[i] = stage;
            stage += S4_B;
        }
#pragma unroll
        for (int j = 0; j < S4_TASKS; j++) {  // (registers: no indexing by ja, jb)
            if (j == ja && j < i) oa[i] = oa[j];
            if (j == jb && j < i) ob[i] = ob[j];
        }
    }
    auto load = [&](int t, int ns) {
        const int k0 = t * ST_BK;
        if (k0 < kmax) {
            float *st = sm + (t % ns) * stage;
#pragma unroll
            for (int i = 0; i < S4_TASKS; i++) {
                if (i >= cnt || k0 >= task[i].k) continue;
                const Sgemm4Task &u = task[i];
                if ((owner >> i) & 1u)
                    st_load_a<64>(st + oa[i], S4_AP, reinterpret_cast<const float *>(u.A), u.m, u.m, u.k, u.bx * 64, k0,
                                  u.m % 4 == 0 && u.A % 16 == 0, tid, S4_THREADS);
                if ((owner >> (4 + i)) & 1u)
                    st_load_b<16>(st + ob[i], reinterpret_cast<const float *>(u.B), u.k, u.n, u.k, u.by * 16, k0,
                                  u.k % 4 == 0 && u.B % 16 == 0, tid, S4_THREADS);
            }
        }
        sf_commit();
    };
    // one task a block: a warp takes half of its rows, else a warp takes a task, or two
    constexpr int RPT = PER == 1 ? 4 : 8;
    uint64_t acc0[RPT / 2][4], acc1[RPT / 2][4];
#pragma unroll
    for (int i = 0; i < RPT / 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc0[i][j] = acc1[i][j] = 0ull;
    const int t0 = PER == 1 ? 0 : PER == 2 ? warp : 2 * warp, t1 = PER == 4 ? 2 * warp + 1 : S4_TASKS;
    const int ka = t0 < cnt ? task[t0].k : 0, kb = t1 < cnt ? task[t1].k : 0;
    const int xl = (lane & 7) * 4 + (PER == 1 ? 32 * warp : 0), yl = lane >> 3;
    int wa0 = 0, wb0 = 0, wa1 = 0, wb1 = 0;
#pragma unroll
    for (int i = 0; i < S4_TASKS; i++) {
        if (i == t0) {
            wa0 = oa[i];
            wb0 = ob[i];
        }
        if (i == t1) {
            wa1 = oa[i];
            wb1 = ob[i];
        }
    }
    const bool both = PER == 4 && ka > 0 && kb > 0 && wa0 == wa1;  // (the same left tile: the same k)
    // as many stages as the block's memory holds of these tiles (one: load, then compute)
    auto run = [&](auto depth) {
        constexpr int NS = decltype(depth)::value;
#pragma unroll
        for (int t = 0; t < NS - 1; t++) load(t, NS);
        for (int t = 0, k0 = 0; k0 < kmax; t++, k0 += ST_BK) {
            if (NS == 1) {
                if (t > 0) __syncthreads();
                load(t, NS);
            }
            sf_wait<NS == 1 ? 0 : NS - 2>();
            __syncthreads();
            if (NS > 1) load(t + NS - 1, NS);
            const float *st = sm + (t % NS) * stage;
            const float *bs0 = st + wb0 + yl * ST_BP, *bs1 = st + wb1 + yl * ST_BP;
            if (both) {
                if (k0 < ka) st_steps2<RPT>(acc0, acc1, st + wa0 + xl, S4_AP, bs0, bs1, min(ST_BK, ka - k0));
            } else {
                if (k0 < ka) st_steps<RPT>(acc0, st + wa0 + xl, S4_AP, bs0, min(ST_BK, ka - k0));
                if (PER == 4 && k0 < kb) st_steps<RPT>(acc1, st + wa1 + xl, S4_AP, bs1, min(ST_BK, kb - k0));
            }
        }
    };
    if (3 * stage <= S4_POOL) run(std::integral_constant<int, 3>{});
    else if (2 * stage <= S4_POOL) run(std::integral_constant<int, 2>{});
    else run(std::integral_constant<int, 1>{});
    auto store = [&](int i, const uint64_t (&acc)[RPT / 2][4]) {
        if (i >= cnt) return;
        const Sgemm4Task &t = task[i];
        st_store<RPT>(acc, reinterpret_cast<float *>(t.C), t.m, t.m, t.n, t.bx * 64 + xl, t.by * 16 + yl, 1.f, 0.f,
                    t.m % 4 == 0 && t.C % 16 == 0);
    };
    store(t0, acc0);
    if (PER == 4) store(t1, acc1);
}

}  // namespace opb

using namespace opb;

// Column-major C(m x n) = alpha * A(m x k) . B(k x n) + beta * C, the semantics of
// cublasSgemm('N','N') that the reference wraps (oplib/opcuda/sgemm.cu:41-44).
OPB_API int opcuda_sgemm(int m, int n, int k, float alpha, uint64_t A, int lda, uint64_t B, int ldb,
                         float beta, uint64_t C, int ldc) {
    OPB_REQUIRE(m >= 0 && n >= 0 && k >= 0, OPB_E_ARG);
    if (m == 0 || n == 0) return set_status(OPB_OK);
    OPB_REQUIRE(C != 0 && (k == 0 || (A != 0 && B != 0)), OPB_E_NULL);
    OPB_REQUIRE(lda >= (m > 1 ? m : 1) && ldb >= (k > 1 ? k : 1) && ldc >= (m > 1 ? m : 1), OPB_E_ARG);
    // column-major C = A.B  <=>  row-major C^T(n x m) = B^T(n x k) . A^T(k x m)
    int st = sgemm_rm(n, m, k, alpha, reinterpret_cast<const float *>(B), ldb,
                      reinterpret_cast<const float *>(A), lda, beta, reinterpret_cast<float *>(C), ldc,
                      stream());
    return set_status(st);
}

// Batched C_i = A_i . B_i for ni column-major d x d matrices given as device arrays of
// 64-bit device pointers (oplib/opcuda/ssqmm.cu:174-179; A_i == B_i squares).
OPB_API int opcuda_ssqmm(int d, int ni, uint64_t A_i, uint64_t B_i, uint64_t C_i) {
    OPB_REQUIRE(d >= 0 && ni >= 0, OPB_E_ARG);
    if (d == 0 || ni == 0) return set_status(OPB_OK);
    OPB_REQUIRE(A_i != 0 && B_i != 0 && C_i != 0, OPB_E_NULL);
    SgemmArgs a{};
    a.M = d; a.N = d; a.K = d; a.lda = d; a.ldb = d; a.ldc = d;
    a.alpha = 1.f; a.beta = 0.f;
    // row-major roles: A' = B_i, B' = A_i
    a.A_tab = reinterpret_cast<const float *const *>(B_i);
    a.B_tab = reinterpret_cast<const float *const *>(A_i);
    a.C_tab = reinterpret_cast<float *const *>(C_i);
    return set_status(sgemm_rowmajor(a, ni, stream()));
}

// Strided-batch variant with typed pointers (new; row-major, ld = d).
OPB_API int opb_sgemm_batched_rm(int M, int N, int K, const float *A, long long sA, const float *B,
                                 long long sB, float *C, long long sC, int batch) {
    OPB_REQUIRE(M >= 0 && N >= 0 && K >= 0 && batch >= 0, OPB_E_ARG);
    if (M == 0 || N == 0 || batch == 0) return set_status(OPB_OK);
    OPB_REQUIRE(A && B && C, OPB_E_NULL);
    SgemmArgs a{};
    a.M = M; a.N = N; a.K = K; a.lda = K; a.ldb = N; a.ldc = N;
    a.alpha = 1.f; a.beta = 0.f; a.A = A; a.B = B; a.C = C; a.sA = sA; a.sB = sB; a.sC = sC;
    return set_status(sgemm_rowmajor(a, batch, stream()));
}

OPB_API int opcuda_sgemm4(int nblocks, uint64_t argptr_bid) {
    OPB_REQUIRE(nblocks >= 0, OPB_E_ARG);
    if (nblocks == 0) return set_status(OPB_OK);
    OPB_REQUIRE(argptr_bid != 0, OPB_E_NULL);
    const uint64_t *tab = reinterpret_cast<const uint64_t *>(argptr_bid);
    cudaStream_t s = stream();
    if (nblocks <= S4_ONE * num_sms()) k_sgemm4<1><<<nblocks, S4_THREADS, 4 * S4_POOL, s>>>(tab, nblocks);
    else if (nblocks <= S4_PAIR * num_sms())
        k_sgemm4<2><<<(nblocks + 1) / 2, S4_THREADS, 4 * S4_POOL, s>>>(tab, nblocks);
    else k_sgemm4<S4_TASKS><<<(nblocks + S4_TASKS - 1) / S4_TASKS, S4_THREADS, 4 * S4_POOL, s>>>(tab, nblocks);
    return launch_check();
}

OPB_API int opb_sgemm4_task_size(void) { return static_cast<int>(sizeof(Sgemm4Task)); }
