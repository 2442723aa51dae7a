// Learned surrogate pricer: an MLP 8 -> 256 -> 256 -> 256 -> 256 -> 1 with GELU, from
// (level, skew, width, kappa, rho, r, log-moneyness, T) to implied volatility, trained on
// quotes that the batched lattice solver produces, with the lattice as fallback and judge.
// The reference has no counterpart (its closest piece is the Black-Scholes pricer of its
// known-answer test, tests/bstest/BSPricer.cs:7-65).
//
// Parameters live in one flat FP32 master vector theta (layer l: W_l [out x in] row-major,
// then b_l [out]); training uses BF16-rounded working weights (kept as FP32 values), FP32
// activations and gradients, and Adam on the FP32 master copy.  All kernels are this
// project's: the hidden layers' products on the tensor cores (gemm_tc.cu, split-BF16 parts
// of the activations and gradients), the first and output layers on SIMT GEMMs
// (gemm_simt.cu, with transpose flags), plus the fused element-wise kernels below.  Batched inference of the trained network runs through
// opb_mlp_infer (BF16 weights and activations, FP32 accumulation).
#include <cuda_bf16.h>

#include <cmath>

#include "common.cuh"
#include "lattice.h"

namespace opb {

constexpr int MLP_IN = 8, MLP_H = 256, MLP_LAYERS = 5;  // 4 hidden + output
constexpr int MLP_NPARAM = MLP_H * MLP_IN + MLP_H + 3 * (MLP_H * MLP_H + MLP_H) + MLP_H + 1;  // 199,937

struct MlpLayout {
    int in[MLP_LAYERS], out[MLP_LAYERS];
    long long w[MLP_LAYERS], b[MLP_LAYERS];
};

__host__ __device__ inline MlpLayout mlp_layout() {
    MlpLayout L{};
    const int ins[MLP_LAYERS] = {MLP_IN, MLP_H, MLP_H, MLP_H, MLP_H};
    const int outs[MLP_LAYERS] = {MLP_H, MLP_H, MLP_H, MLP_H, 1};
    long long o = 0;
    for (int l = 0; l < MLP_LAYERS; l++) {
        L.in[l] = ins[l];
        L.out[l] = outs[l];
        L.w[l] = o;
        o += (long long)ins[l] * outs[l];
        L.b[l] = o;
        o += outs[l];
    }
    return L;
}

__device__ __forceinline__ uint32_t hash32(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdULL;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ULL;
    x ^= x >> 33;
    return (uint32_t)x;
}

// Uniform(-a, a) weights with a = sqrt(6 / fan_in) (He-uniform), zero biases.
__global__ void k_mlp_init(float *__restrict__ theta, uint64_t seed) {
    pdl_begin();
    const MlpLayout L = mlp_layout();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < MLP_NPARAM;
         i += (long long)gridDim.x * blockDim.x) {
        int l = 0;
        while (l + 1 < MLP_LAYERS && i >= L.w[l + 1]) l++;
        if (i >= L.b[l]) {
            theta[i] = 0.f;
        } else {
            const float a = sqrtf(6.f / (float)L.in[l]);
            const float u = (hash32(seed * 0x9E3779B97F4A7C15ULL + (uint64_t)i) >> 8) * (1.0f / 16777216.0f);
            theta[i] = (2.f * u - 1.f) * a;
        }
    }
}

// BF16 working copy of the master weights (as FP32 values) and the BF16 storage used by
// inference (same layout).
__global__ void k_mlp_round(const float *__restrict__ theta, float *__restrict__ theta_bf,
                            __nv_bfloat16 *__restrict__ theta_b16, int n) {
    pdl_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const __nv_bfloat16 b = __float2bfloat16_rn(theta[i]);
        if (theta_bf) theta_bf[i] = __bfloat162float(b);
        if (theta_b16) theta_b16[i] = b;
    }
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// A training step is some twenty dependent launches over 4 MB matrices, so what bounds it is the
// number of launches and the passes between the products: 47 launches took 318 us at B = 4096
// (228 us of kernels).  Each element-wise pass below therefore writes everything the following
// products read (the parts, row-major and transposed) and the column sums it passes over (bias,
// first-layer and output-layer gradients, as partial sums per row block), and one launch at the
// end adds up all partial sums in a fixed order: 20 launches, 317 -> 164 us,
// and 135 with each set up while the one before it runs.

constexpr int MLP_RB = 16;  // rows per block of the backward element-wise pass (two blocks an SM at B = 4096)

// First layer: Z = X W^T + b (8 inputs, summed in order), H = GELU(Z) in FP32 and/or as parts; thread
// per column, MLP_RB rows per block.  Blocks from nrow on write the parts of the working weights of
// the hidden layers (three 256 x 256 matrices from wh, the biases between them) instead.
__global__ void __launch_bounds__(MLP_H) k_mlp_first(int B, const float *__restrict__ X, const float *__restrict__ W,
                                                     const float *__restrict__ b, float *__restrict__ Z,
                                                     float *__restrict__ H, __nv_bfloat16 *__restrict__ Hhi,
                                                     __nv_bfloat16 *__restrict__ Hlo, int nrow,
                                                     const float *__restrict__ wh, __nv_bfloat16 *const Wp0h,
                                                     __nv_bfloat16 *const Wp0l, __nv_bfloat16 *const Wp1h,
                                                     __nv_bfloat16 *const Wp1l, __nv_bfloat16 *const Wp2h,
                                                     __nv_bfloat16 *const Wp2l) {
    pdl_begin();
    const int c = threadIdx.x;
    if ((int)blockIdx.x >= nrow) {  // a row of a weight matrix
        const int i = (int)blockIdx.x - nrow, l = i / MLP_H, o = (i % MLP_H) * MLP_H + c;
        __nv_bfloat16 *hi = l == 0 ? Wp0h : l == 1 ? Wp1h : Wp2h, *lo = l == 0 ? Wp0l : l == 1 ? Wp1l : Wp2l;
        split2(wh[(long long)l * (MLP_H * MLP_H + MLP_H) + o], hi[o], lo[o]);
        return;
    }
    __shared__ float xs[MLP_RB][MLP_IN];
    const int r0 = blockIdx.x * MLP_RB, n = min(MLP_RB, B - r0);
    if (c < n * MLP_IN) xs[c / MLP_IN][c % MLP_IN] = X[(long long)r0 * MLP_IN + c];
    float w[MLP_IN];
#pragma unroll
    for (int k = 0; k < MLP_IN; k++) w[k] = W[c * MLP_IN + k];
    const float bc = b[c];
    __syncthreads();
    for (int r = 0; r < n; r++) {
        float z = 0.f;
#pragma unroll
        for (int k = 0; k < MLP_IN; k++) z = fmaf(xs[r][k], w[k], z);
        z += bc;
        const long long i = (long long)(r0 + r) * MLP_H + c;
        Z[i] = z;
        const float h = gelu(z);
        if (H) H[i] = h;
        if (Hhi) split2(h, Hhi[i], Hlo[i]);
    }
}

// Z += b (per column), H = GELU(Z), four columns a thread.  Z, H: [B x 256] row-major.  H
// (optional) in FP32 and/or its BF16 parts Hhi / Hlo (optional, for the tensor-core products).
// Z and H are the workspace's and 16-byte aligned; b is the caller's, any float address (a network
// is 199,937 floats: in an array of several, every second row starts off the 8-byte grid).
__global__ void k_bias_gelu(long long total4, float *__restrict__ Z, const float *__restrict__ b,
                            float *__restrict__ H, __nv_bfloat16 *__restrict__ Hhi, __nv_bfloat16 *__restrict__ Hlo) {
    pdl_begin();
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= total4) return;
    const float4 zv = reinterpret_cast<const float4 *>(Z)[i];
    const float *bc = b + 4 * (i % (MLP_H / 4));
    const float4 bv = reinterpret_cast<uintptr_t>(b) % 16 == 0 ? *reinterpret_cast<const float4 *>(bc)
                                                               : make_float4(bc[0], bc[1], bc[2], bc[3]);
    const float z[4] = {zv.x + bv.x, zv.y + bv.y, zv.z + bv.z, zv.w + bv.w};
    float h[4];
#pragma unroll
    for (int j = 0; j < 4; j++) h[j] = gelu(z[j]);
    reinterpret_cast<float4 *>(Z)[i] = make_float4(z[0], z[1], z[2], z[3]);
    if (H) reinterpret_cast<float4 *>(H)[i] = make_float4(h[0], h[1], h[2], h[3]);
    if (Hhi) {
        uint2 hi, lo;
        split2x2(h[0], h[1], hi.x, lo.x, 0.f);
        split2x2(h[2], h[3], hi.y, lo.y, 0.f);
        reinterpret_cast<uint2 *>(Hhi)[i] = hi;
        reinterpret_cast<uint2 *>(Hlo)[i] = lo;
    }
}

// Last hidden layer's bias and GELU with the output layer (warp per row, eight rows per block):
// Z += b, y = GELU(Z) . w5 + b5, and with targets dy = 2 (y - t) / B and the block's sums of the
// squared errors and of dy.
__global__ void __launch_bounds__(256) k_mlp_out(int B, float *__restrict__ Z, const float *__restrict__ b,
                                                 const float *__restrict__ w5, const float *__restrict__ b5,
                                                 float *__restrict__ y, const float *__restrict__ t,
                                                 float *__restrict__ dy, double *__restrict__ loss_part,
                                                 float *__restrict__ dy_part) {
    pdl_begin();
    __shared__ double se_s[8];
    __shared__ float dy_s[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long r = blockIdx.x * 8LL + warp;
    double se = 0.0;
    float d = 0.f;
    if (r < B) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < MLP_H / 32; i++) {
            const int c = lane + 32 * i;
            const float z = Z[r * MLP_H + c] + b[c];
            Z[r * MLP_H + c] = z;
            s = fmaf(gelu(z), w5[c], s);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float v = s + b5[0];
        if (lane == 0) y[r] = v;
        if (t) {
            const float e = v - t[r];
            d = 2.f * e / (float)B;
            se = (double)e * (double)e;
            if (lane == 0) dy[r] = d;
        }
    }
    if (!t) return;
    if (lane == 0) {
        se_s[warp] = se;
        dy_s[warp] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0;
        float g = 0.f;
        for (int i = 0; i < 8; i++) {
            a += se_s[i];
            g += dy_s[i];
        }
        loss_part[blockIdx.x] = a;
        dy_part[blockIdx.x] = g;
    }
}

// Backward element-wise pass of one hidden layer, two columns a thread, MLP_RB rows per block:
// dZ = dH * GELU'(Z), with dH = dy (outer) w5 for the last layer (dH null).  Writes dZ in FP32
// (optional), its BF16 parts row-major and transposed ([256 x B]; both or neither, B a multiple of
// MLP_RB then), and the block's column sums: of dZ into bsum[block][256]; of dy H (last layer, H =
// GELU(Z) again) into wsum[block][256]; of dZ X (first layer, X non-null) into wsum[block][8][256].
// Rows past the end read the last one and count as zeros, so that all loads are in flight at once.
template <bool LAST, bool FIRST>
__global__ void __launch_bounds__(MLP_H / 2) k_mlp_dz(int B, const float *__restrict__ Z, const float *__restrict__ dH,
                                                      const float *__restrict__ dy, const float *__restrict__ w5,
                                                      const float *__restrict__ X, float *__restrict__ dZ,
                                                      __nv_bfloat16 *__restrict__ Ghi, __nv_bfloat16 *__restrict__ Glo,
                                                      __nv_bfloat16 *__restrict__ Thi, __nv_bfloat16 *__restrict__ Tlo,
                                                      float *__restrict__ bsum, float *__restrict__ wsum) {
    pdl_begin();
    const int c = 2 * threadIdx.x, r0 = blockIdx.x * MLP_RB, n = min(MLP_RB, B - r0);
    __shared__ float xs[MLP_RB][MLP_IN];
    if (FIRST) {
        if ((int)threadIdx.x < n * MLP_IN) xs[threadIdx.x / MLP_IN][threadIdx.x % MLP_IN] = X[(long long)r0 * MLP_IN + threadIdx.x];
        __syncthreads();
    }
    auto at = [&](int r) { return ((long long)r0 + min(r, n - 1)) * MLP_H + c; };
    float2 g[MLP_RB];
    float2 sb = make_float2(0.f, 0.f), sw[FIRST ? MLP_IN : 1];
#pragma unroll
    for (int k = 0; k < (FIRST ? MLP_IN : 1); k++) sw[k] = make_float2(0.f, 0.f);
#pragma unroll
    for (int r = 0; r < MLP_RB; r++) {
        if (LAST) {
            const float d = dy[r0 + min(r, n - 1)];
            g[r] = make_float2(d * w5[c], d * w5[c + 1]);  // (w5: the caller's, any float address)
        } else {
            g[r] = *reinterpret_cast<const float2 *>(dH + at(r));
        }
    }
    float2 z[MLP_RB];
#pragma unroll
    for (int r = 0; r < MLP_RB; r++) z[r] = *reinterpret_cast<const float2 *>(Z + at(r));
#pragma unroll
    for (int r = 0; r < MLP_RB; r++) {
        const bool in = r < n;
        if (LAST) {
            const float d = in ? dy[r0 + r] : 0.f;
            sw[0].x = fmaf(d, gelu(z[r].x), sw[0].x);
            sw[0].y = fmaf(d, gelu(z[r].y), sw[0].y);
        }
        g[r].x = in ? g[r].x * gelu_grad(z[r].x) : 0.f;
        g[r].y = in ? g[r].y * gelu_grad(z[r].y) : 0.f;
        sb.x += g[r].x;
        sb.y += g[r].y;
        if (FIRST && in) {
#pragma unroll
            for (int k = 0; k < MLP_IN; k++) {
                sw[k].x = fmaf(g[r].x, xs[r][k], sw[k].x);
                sw[k].y = fmaf(g[r].y, xs[r][k], sw[k].y);
            }
        }
        if (dZ && in) *reinterpret_cast<float2 *>(dZ + at(r)) = g[r];
    }
    if (!FIRST && Ghi) {
        uint32_t h[2][MLP_RB / 2], l[2][MLP_RB / 2];  // per column, rows in pairs
#pragma unroll
        for (int r = 0; r < MLP_RB; r += 2) {
            const int q = r / 2;
            split2x2(g[r].x, g[r + 1].x, h[0][q], l[0][q], 0.f);
            split2x2(g[r].y, g[r + 1].y, h[1][q], l[1][q], 0.f);
            *reinterpret_cast<uint32_t *>(Ghi + at(r)) = __byte_perm(h[0][q], h[1][q], 0x5410);
            *reinterpret_cast<uint32_t *>(Glo + at(r)) = __byte_perm(l[0][q], l[1][q], 0x5410);
            *reinterpret_cast<uint32_t *>(Ghi + at(r + 1)) = __byte_perm(h[0][q], h[1][q], 0x7632);
            *reinterpret_cast<uint32_t *>(Glo + at(r + 1)) = __byte_perm(l[0][q], l[1][q], 0x7632);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            uint4 *th = reinterpret_cast<uint4 *>(Thi + (long long)(c + u) * B + r0);
            uint4 *tl = reinterpret_cast<uint4 *>(Tlo + (long long)(c + u) * B + r0);
#pragma unroll
            for (int q = 0; q < MLP_RB / 8; q++) {
                th[q] = make_uint4(h[u][4 * q], h[u][4 * q + 1], h[u][4 * q + 2], h[u][4 * q + 3]);
                tl[q] = make_uint4(l[u][4 * q], l[u][4 * q + 1], l[u][4 * q + 2], l[u][4 * q + 3]);
            }
        }
    }
    *reinterpret_cast<float2 *>(bsum + (long long)blockIdx.x * MLP_H + c) = sb;
    if (LAST) *reinterpret_cast<float2 *>(wsum + (long long)blockIdx.x * MLP_H + c) = sw[0];
    if (FIRST) {
#pragma unroll
        for (int k = 0; k < MLP_IN; k++)
            *reinterpret_cast<float2 *>(wsum + ((long long)blockIdx.x * MLP_IN + k) * MLP_H + c) = sw[k];
    }
}

// All partial sums of a step into the gradient, in a fixed order.  Blocks [0, 3 * 256): the
// hidden layers' weight gradients, a row each, over their np[l] slices (np 0: already there); the
// next ones a row of column sums each, over nb row blocks (four biases, then w5, then the eight
// first-layer inputs) by four groups of 64 columns; the last one b5 and the loss over no blocks.
struct MlpFinish {
    const float *wpart[3];  // [np][256 x 256]
    int np[3];
    float *dW[3];
    const float *bsum[4], *w5sum, *w1sum;  // [nb][256], [nb][256], [nb][8][256]
    float *db[4], *dw5, *dw1, *db5;
    int nb;
    const double *loss_part;
    const float *dy_part;
    double *loss;  // optional
    int no;
};
__global__ void __launch_bounds__(256) k_mlp_finish(MlpFinish f) {
    pdl_begin();
    const int tid = threadIdx.x;
    int blk = blockIdx.x;
    if (blk < 3 * MLP_H) {
        const int l = blk / MLP_H;
        const long long i = (long long)(blk % MLP_H) * MLP_H + tid;
        if (f.np[l] == 0) return;
        float acc = 0.f;
#pragma unroll 8
        for (int p = 0; p < f.np[l]; p++) acc += f.wpart[l][(long long)p * MLP_H * MLP_H + i];
        f.dW[l][i] = acc;
        return;
    }
    blk -= 3 * MLP_H;
    __shared__ float red[4][64];
    if (blk < 13 * 4) {
        const int row = blk / 4, c = (blk % 4) * 64 + (tid & 63), grp = tid >> 6;
        const float *src;
        long long step = MLP_H;
        if (row < 4) src = f.bsum[row];
        else if (row == 4) src = f.w5sum;
        else {
            src = f.w1sum + (long long)(row - 5) * MLP_H;
            step = (long long)MLP_IN * MLP_H;
        }
        // four contiguous quarters of the row blocks, added in order
        const int q = (f.nb + 3) / 4, p0 = grp * q, p1 = min(f.nb, p0 + q);
        float acc = 0.f;
#pragma unroll 8
        for (int p = p0; p < p1; p++) acc += src[p * step + c];
        red[grp][tid & 63] = acc;
        __syncthreads();
        if (grp == 0) {
            const float v = red[0][tid] + red[1][tid] + red[2][tid] + red[3][tid];
            if (row < 4) f.db[row][c] = v;
            else if (row == 4) f.dw5[c] = v;
            else f.dw1[c * MLP_IN + (row - 5)] = v;
        }
        return;
    }
    __shared__ double rl[256];
    __shared__ float rd[256];
    double a = 0.0;
    float g = 0.f;
    for (int p = tid; p < f.no; p += 256) {
        a += f.loss_part[p];
        g += f.dy_part[p];
    }
    rl[tid] = a;
    rd[tid] = g;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (tid < o) {
            rl[tid] += rl[tid + o];
            rd[tid] += rd[tid + o];
        }
        __syncthreads();
    }
    if (tid == 0) {
        *f.db5 = rd[0];
        if (f.loss) *f.loss = rl[0];
    }
}

// Adam on the FP32 master weights; refreshes the BF16 working copy.
__global__ void k_adam(int n, float *__restrict__ theta, float *__restrict__ m, float *__restrict__ v,
                       const float *__restrict__ g, float lr, float b1, float b2, float eps, float c1, float c2,
                       float *__restrict__ theta_bf) {
    pdl_begin();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float th = theta[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        theta[i] = th;
        theta_bf[i] = __bfloat162float(__float2bfloat16_rn(th));
    }
}

// The same step with the step count and learning rate on the device: step s = *step + 1,
// lr = lr_table[s - 1] (a schedule), bias corrections 1 - b^s; a following k_step_inc
// advances *step.  A training loop of these launches can be captured in a CUDA graph once
// and replayed every epoch.
__global__ void k_adam_sched(int n, float *__restrict__ theta, float *__restrict__ m, float *__restrict__ v,
                             const float *__restrict__ g, const float *__restrict__ lr_table,
                             const int *__restrict__ step, float b1, float b2, float eps,
                             float *__restrict__ theta_bf) {
    pdl_begin();
    const int s = *step + 1;
    const float c1 = 1.f - powf(b1, (float)s), c2 = 1.f - powf(b2, (float)s);
    const float lr = lr_table[s - 1];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float th = theta[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        theta[i] = th;
        theta_bf[i] = __bfloat162float(__float2bfloat16_rn(th));
    }
}

__global__ void k_step_inc(int *step) {
    pdl_begin();
    *step += 1;
}

// ---- implied volatility of call prices (FP64 bisection on the Black-Scholes price)
__device__ double bs_call(double s, double k, double r, double sig, double t) {
    const double sq = sig * sqrt(t);
    const double d1 = (log(s / k) + (r + 0.5 * sig * sig) * t) / sq;
    return s * normcdf(d1) - k * exp(-r * t) * normcdf(d1 - sq);
}

__global__ void k_implied_vol(long long n, const double *__restrict__ price, const double *__restrict__ K,
                              const double *__restrict__ T, const double *__restrict__ r,
                              const double *__restrict__ S0, double *__restrict__ iv) {
    pdl_begin();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double p = price[i], k = K[i], t = T[i], rr = r[i], s0 = S0[i];
        const double intrinsic = fmax(s0 - k * exp(-rr * t), 0.0);
        double lo = 1e-4, hi = 4.0;
        if (!(p > intrinsic) || p >= s0) {
            iv[i] = nan("");
            continue;
        }
        for (int it = 0; it < 80; it++) {
            const double mid = 0.5 * (lo + hi);
            if (bs_call(s0, k, rr, mid, t) > p) hi = mid; else lo = mid;
        }
        iv[i] = 0.5 * (lo + hi);
    }
}

}  // namespace opb

using namespace opb;

namespace {

struct MlpWs {  // training workspace carve (floats)
    float *Z[4], *H[4], *dZ, *dH, *y, *dy, *part;
    // partial sums: [nb][256] per layer's bias and for w5, [nb][8][256] for the first layer, [no] per
    // row block of the output layer
    float *bsum[4], *w5sum, *w1sum, *dysum;
    double *lossp;
    // 16-bit parts for the tensor-core products of the hidden layers 1..3 (split2, BF16):
    // Hp[l][0/1] of H[l] (l = 0..2, B x 256 row-major), dZp of dZ (B x 256), dZt of dZ^T
    // (256 x B), Wp[l][0/1] of the working weights W_{l+1} (256 x 256, exact BF16: lo = 0)
    __nv_bfloat16 *Hp[3][2], *dZp[2], *dZt[2], *Wp[3][2];
    size_t floats;
};

// Weight gradients reduce over the batch (K = B): split into at most MLP_KSPLIT chunks whose
// partial products the step's last launch adds in a fixed order, so that the reduction keeps
// every SM busy and stays deterministic.
constexpr int MLP_KSPLIT = 32;

int grid_ew(long long n);

MlpWs carve_mlp(float *ws, int B) {
    MlpWs w{};
    size_t o = 0;
    auto take = [&](size_t n) {  // 256-byte aligned pieces
        o = (o + 63) & ~size_t(63);
        float *q = ws + o;
        o += n;
        return q;
    };
    auto parts = [&](size_t n) { return reinterpret_cast<__nv_bfloat16 *>(take((n + 1) / 2)); };  // n BF16 values
    const size_t bh = (size_t)B * MLP_H, nb = ((size_t)B + MLP_RB - 1) / MLP_RB, no = ((size_t)B + 7) / 8;
    for (int l = 0; l < 4; l++) {
        w.Z[l] = take(bh);
        w.H[l] = take(bh);
    }
    w.dZ = take(bh);
    w.dH = take(bh);
    w.y = take(B);
    w.dy = take(B);
    w.part = take(3 * (size_t)MLP_KSPLIT * MLP_H * MLP_H);
    for (int l = 0; l < 4; l++) w.bsum[l] = take(nb * MLP_H);
    w.w5sum = take(nb * MLP_H);
    w.w1sum = take(nb * MLP_IN * MLP_H);
    w.dysum = take(no);
    w.lossp = reinterpret_cast<double *>(take(2 * no));
    for (int l = 0; l < 3; l++)
        for (int k = 0; k < 2; k++) w.Hp[l][k] = parts(bh);
    for (int k = 0; k < 2; k++) w.dZp[k] = parts(bh);
    for (int k = 0; k < 2; k++) w.dZt[k] = parts(bh);
    for (int l = 0; l < 3; l++)
        for (int k = 0; k < 2; k++) w.Wp[l][k] = parts((size_t)MLP_H * MLP_H);
    w.floats = o;
    return w;
}

// The workspace's carve starts at the next 256-byte boundary.
float *mlp_ws_base(float *ws) {
    return reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(ws) + 255) & ~uintptr_t(255));
}

// The hidden layers' products run on the tensor cores (split-BF16, three products, FP32
// accumulation) when the batch is a multiple of 128 rows; the first layer (8 inputs) and
// the output layer stay on the SIMT kernels.  opb_mlp_set_tensor_cores(0): SIMT throughout.
int g_mlp_tc = 1;
bool mlp_tc(int B) { return g_mlp_tc && B % 128 == 0; }

// C[M x N] = A[M x K] . B^T with A's parts row-major (lda) and B's parts N x K row-major
// (b_kn = 0) or K x N row-major (b_kn = 1); ksplit > 1: K-slices into C + s * M * N.
int mlp_tc_gemm(int M, int N, int K, __nv_bfloat16 *const *A, long long lda, __nv_bfloat16 *const *Bp,
                long long ldb, int b_kn, float *C, int ksplit, cudaStream_t s, int tile_n = 0) {
    TcGemmArgs a{};
    a.M = M; a.N = N; a.K = K; a.Ahi = A[0]; a.Alo = A[1]; a.lda = lda; a.Bhi = Bp[0]; a.Blo = Bp[1]; a.ldb = ldb;
    a.b_kn = b_kn; a.C = C; a.ldc = N; a.alpha = 1.f; a.beta = 0.f; a.tile_n = tile_n;
    if (ksplit > 1) {
        a.ksplit = ksplit;
        a.c_slice = (long long)M * N;
    }
    return launch_tc_gemm(a, s);
}

// Partial products of dW[256 x 256] = dZ[B x 256]^T . in[B x 256], split over the batch, on the
// SIMT kernels; returns through *np how many.
int mlp_weight_grad(int B, const float *dZ, const float *in, float *part, int *np, cudaStream_t s) {
    int nch = (B + 63) / 64;
    if (nch > MLP_KSPLIT) nch = MLP_KSPLIT;
    const int kc = (B + nch - 1) / nch;
    const int full = B / kc, rem = B - full * kc;
    const long long n = (long long)MLP_H * MLP_H;
    if (full > 0) {
        int r = sgemm_rm_strided(true, false, MLP_H, MLP_H, kc, 1.f, dZ, MLP_H, (long long)kc * MLP_H, in, MLP_H,
                                 (long long)kc * MLP_H, 0.f, part, MLP_H, n, full, s);
        if (r) return r;
    }
    if (rem > 0) {
        int r = sgemm_rm_t(true, false, MLP_H, MLP_H, rem, 1.f, dZ + (long long)full * kc * MLP_H, MLP_H,
                           in + (long long)full * kc * MLP_H, MLP_H, 0.f, part + (long long)full * n, MLP_H, s);
        if (r) return r;
    }
    *np = full + (rem > 0 ? 1 : 0);
    return (int)cudaGetLastError();
}

int grid_ew(long long n) {
    long long b = (n + 255) / 256;
    long long cap = 8LL * num_sms();
    return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

#define MT(expr)                          \
    do {                                  \
        int _r = (expr);                  \
        if (_r) return set_status(_r);    \
    } while (0)

// The forward pass up to the last hidden layer's product (its bias, GELU and the output layer
// are k_mlp_out's).
int mlp_forward(const float *thb, const float *X, int B, MlpWs &w, cudaStream_t s) {
    const MlpLayout L = mlp_layout();
    const bool tc = mlp_tc(B);
    const int nrow = (B + MLP_RB - 1) / MLP_RB;
    // with the tensor cores, layers 0..2 store only their activations' parts (the next
    // product's A and the weight gradient's B)
    launch_pdl(k_mlp_first, nrow + (tc ? 3 * MLP_H : 0), MLP_H, 0, s, B, X, thb + L.w[0], thb + L.b[0], w.Z[0],
               tc ? nullptr : w.H[0], tc ? w.Hp[0][0] : nullptr, tc ? w.Hp[0][1] : nullptr, nrow, thb + L.w[1],
               w.Wp[0][0], w.Wp[0][1], w.Wp[1][0], w.Wp[1][1], w.Wp[2][0], w.Wp[2][1]);
    for (int l = 1; l < 4; l++) {
        // Z = in . W^T  (W stored out x in: the TB form)
        if (tc) MT(mlp_tc_gemm(B, MLP_H, MLP_H, w.Hp[l - 1], MLP_H, w.Wp[l - 1], MLP_H, 0, w.Z[l], 1, s));
        else
            MT(sgemm_rm_t(false, true, B, MLP_H, MLP_H, 1.f, w.H[l - 1], MLP_H, thb + L.w[l], MLP_H, 0.f, w.Z[l], MLP_H,
                          s));
        if (l == 3) break;
        const long long t4 = (long long)B * MLP_H / 4;
        launch_pdl(k_bias_gelu, (unsigned)((t4 + 255) / 256), 256, 0, s, t4, w.Z[l], thb + L.b[l],
                   tc ? nullptr : w.H[l], tc ? w.Hp[l][0] : nullptr, tc ? w.Hp[l][1] : nullptr);
    }
    return (int)cudaGetLastError();
}

}  // namespace

OPB_API int opb_mlp_param_count(void) { return MLP_NPARAM; }

// floats of training workspace for batch B
OPB_API long long opb_mlp_workspace_floats(int B) {
    if (B <= 0) return 0;
    return (long long)carve_mlp(nullptr, B).floats + 64;  // (+ the alignment of its base)
}

// 1 (default): the hidden layers' training products on the tensor cores (batches of a
// multiple of 128 rows); 0: SIMT FP32 throughout.
OPB_API int opb_mlp_set_tensor_cores(int on) {
    OPB_REQUIRE(on == 0 || on == 1, OPB_E_ARG);
    g_mlp_tc = on;
    return set_status(OPB_OK);
}

OPB_API int opb_mlp_init(float *theta, unsigned long long seed) {
    OPB_REQUIRE(theta, OPB_E_NULL);
    launch_pdl(k_mlp_init, grid_ew(MLP_NPARAM), 256, 0, stream(), theta, seed);
    return launch_check();
}

// theta_bf: BF16-rounded FP32 working copy (optional); theta_b16: BF16 storage (optional)
OPB_API int opb_mlp_round(const float *theta, float *theta_bf, void *theta_b16) {
    OPB_REQUIRE(theta, OPB_E_NULL);
    launch_pdl(k_mlp_round, grid_ew(MLP_NPARAM), 256, 0, stream(), theta, theta_bf,
               reinterpret_cast<__nv_bfloat16 *>(theta_b16), MLP_NPARAM);
    return launch_check();
}

// Forward pass of B rows of X [B x 8] with the working weights thb; y [B].  The workspace
// keeps the pre-activations.
OPB_API int opb_mlp_forward(const float *thb, const float *X, int B, float *ws, float *y) {
    OPB_REQUIRE(thb && X && ws && y, OPB_E_NULL);
    OPB_REQUIRE(B > 0, OPB_E_ARG);
    MlpWs w = carve_mlp(mlp_ws_base(ws), B);
    cudaStream_t s = stream();
    MT(mlp_forward(thb, X, B, w, s));
    const MlpLayout L = mlp_layout();
    launch_pdl(k_mlp_out, (B + 7) / 8, 256, 0, s, B, w.Z[3], thb + L.b[3], thb + L.w[4], thb + L.b[4], y, nullptr,
               nullptr, nullptr, nullptr);
    return launch_check();
}

// Loss (sum of squared errors against t) and the gradient of the mean squared error with respect
// to the working weights, written into grad [param count].  loss: device, 1 double, optional.
OPB_API int opb_mlp_loss_grad(const float *thb, const float *X, const float *t, int B, float *ws, float *grad,
                              double *loss) {
    OPB_REQUIRE(thb && X && t && ws && grad, OPB_E_NULL);
    OPB_REQUIRE(B > 0, OPB_E_ARG);
    MlpWs w = carve_mlp(mlp_ws_base(ws), B);
    cudaStream_t s = stream();
    const MlpLayout L = mlp_layout();
    MT(mlp_forward(thb, X, B, w, s));
    const int no = (B + 7) / 8, nb = (B + MLP_RB - 1) / MLP_RB;
    launch_pdl(k_mlp_out, no, 256, 0, s, B, w.Z[3], thb + L.b[3], thb + L.w[4], thb + L.b[4], w.y, t, w.dy, w.lossp,
               w.dysum);
    const bool tc = mlp_tc(B);
    // weight-gradient K-slices on the tensor cores: at most 16, dividing B / 64.  Sixteen slices of
    // 128 x 64 tiles are 128 CTAs; with 32 slices of 128 x 256 ones (64 CTAs) the output phase of
    // the wide tile was most of the launch
    int ks = B / 64 < MLP_KSPLIT / 2 ? B / 64 : MLP_KSPLIT / 2;
    while (ks > 1 && (B / 64) % ks) ks--;
    MlpFinish f{};
    for (int l = 3; l >= 1; l--) {
        float *dZ = tc ? nullptr : w.dZ;
        __nv_bfloat16 *gh = tc ? w.dZp[0] : nullptr, *gl = tc ? w.dZp[1] : nullptr;
        if (l == 3) {
            // (with SIMT products the last activations are wanted in FP32 by nobody but this pass)
            launch_pdl(k_mlp_dz<true, false>, nb, MLP_H / 2, 0, s, B, w.Z[3], nullptr, w.dy, thb + L.w[4], nullptr,
                       dZ, gh, gl, w.dZt[0], w.dZt[1], w.bsum[3], w.w5sum);
        } else {
            launch_pdl(k_mlp_dz<false, false>, nb, MLP_H / 2, 0, s, B, w.Z[l], w.dH, nullptr, nullptr, nullptr, dZ,
                       gh, gl, w.dZt[0], w.dZt[1], w.bsum[l], nullptr);
        }
        float *part = w.part + (size_t)(l - 1) * MLP_KSPLIT * MLP_H * MLP_H;
        f.wpart[l - 1] = part;
        f.dW[l - 1] = grad + L.w[l];
        if (tc) {
            // dW = dZ^T . in: A = dZ^T's parts (256 x B), B = in's parts read K x N (B x 256);
            // dH = dZ . W: B = W's parts read K x N (out x in)
            f.np[l - 1] = ks;
            MT(mlp_tc_gemm(MLP_H, MLP_H, B, w.dZt, B, w.Hp[l - 1], MLP_H, 1, part, ks, s, 64));
            MT(mlp_tc_gemm(B, MLP_H, MLP_H, w.dZp, MLP_H, w.Wp[l - 1], MLP_H, 1, w.dH, 1, s));
        } else {
            MT(mlp_weight_grad(B, w.dZ, w.H[l - 1], part, &f.np[l - 1], s));
            MT(sgemm_rm_t(false, false, B, MLP_H, MLP_H, 1.f, w.dZ, MLP_H, thb + L.w[l], MLP_H, 0.f, w.dH, MLP_H, s));
        }
    }
    launch_pdl(k_mlp_dz<false, true>, nb, MLP_H / 2, 0, s, B, w.Z[0], w.dH, nullptr, nullptr, X, nullptr, nullptr,
               nullptr, nullptr, nullptr, w.bsum[0], w.w1sum);
    for (int l = 0; l < 4; l++) {
        f.bsum[l] = w.bsum[l];
        f.db[l] = grad + L.b[l];
    }
    f.w5sum = w.w5sum; f.w1sum = w.w1sum; f.dw5 = grad + L.w[4]; f.dw1 = grad + L.w[0]; f.db5 = grad + L.b[4];
    f.nb = nb; f.loss_part = w.lossp; f.dy_part = w.dysum; f.loss = loss; f.no = no;
    launch_pdl(k_mlp_finish, 3 * MLP_H + 13 * 4 + 1, 256, 0, s, f);
    return launch_check();
}

OPB_API int opb_mlp_adam(float *theta, float *m, float *v, const float *grad, int step, float lr, float b1, float b2,
                         float eps, float *theta_bf) {
    OPB_REQUIRE(theta && m && v && grad && theta_bf, OPB_E_NULL);
    OPB_REQUIRE(step >= 1 && lr > 0.f, OPB_E_ARG);
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    launch_pdl(k_adam, grid_ew(MLP_NPARAM), 256, 0, stream(), MLP_NPARAM, theta, m, v, grad, lr, b1, b2, eps, c1,
               c2, theta_bf);
    return launch_check();
}

// Adam with the step counter (device int, advanced by the call) and the learning-rate
// schedule (device lr_table[step - 1]) in device memory, so that a training loop of
// opb_mlp_loss_grad / opb_mlp_adam_sched calls is the same work every epoch and can be
// captured in a CUDA graph.  Same update as opb_mlp_adam.
OPB_API int opb_mlp_adam_sched(float *theta, float *m, float *v, const float *grad, int *step, const float *lr_table,
                               float b1, float b2, float eps, float *theta_bf) {
    OPB_REQUIRE(theta && m && v && grad && step && lr_table && theta_bf, OPB_E_NULL);
    launch_pdl(k_adam_sched, grid_ew(MLP_NPARAM), 256, 0, stream(), MLP_NPARAM, theta, m, v, grad, lr_table, step,
               b1, b2, eps, theta_bf);
    launch_pdl(k_step_inc, 1, 1, 0, stream(), step);
    return launch_check();
}

// Implied volatilities of n call prices with spots S0[i]; NaN where the price carries no
// time value.
OPB_API int opb_implied_vol(long long n, const double *price, const double *K, const double *T, const double *r,
                            const double *S0, double *iv) {
    OPB_REQUIRE(n >= 0, OPB_E_ARG);
    if (n == 0) return set_status(OPB_OK);
    OPB_REQUIRE(price && K && T && r && S0 && iv, OPB_E_NULL);
    launch_pdl(k_implied_vol, grid_ew(n), 256, 0, stream(), n, price, K, T, r, S0, iv);
    return launch_check();
}

// ---------------------------------------------------------------- tensor-core inference
//
// Packed inference weights of one network (bytes): W1 padded to [256 x 64] BF16 (input
// features 8..63 zero), W2..W4 [256 x 256] BF16, then FP32 b1..b4 [4 x 256], w5 [256], b5.
namespace opb {

constexpr long long MLP_PACK_W1 = 256LL * 64 * 2, MLP_PACK_WH = 256LL * 256 * 2;
constexpr long long MLP_PACK_BYTES = MLP_PACK_W1 + 3 * MLP_PACK_WH + (4 * 256 + 256 + 1) * 4;

__global__ void k_mlp_pack(const float *__restrict__ theta, uint8_t *__restrict__ packed) {
    pdl_begin();
    const MlpLayout L = mlp_layout();
    __nv_bfloat16 *w1 = reinterpret_cast<__nv_bfloat16 *>(packed);
    __nv_bfloat16 *wh = reinterpret_cast<__nv_bfloat16 *>(packed + MLP_PACK_W1);
    float *f = reinterpret_cast<float *>(packed + MLP_PACK_W1 + 3 * MLP_PACK_WH);
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, nth = (long long)gridDim.x * blockDim.x;
    for (long long i = tid; i < 256 * 64; i += nth) {
        const int o = (int)(i / 64), c = (int)(i % 64);
        w1[i] = __float2bfloat16_rn(c < MLP_IN ? theta[L.w[0] + (long long)o * MLP_IN + c] : 0.f);
    }
    for (long long i = tid; i < 3LL * 256 * 256; i += nth) {
        const int l = 1 + (int)(i / (256 * 256));
        wh[i] = __float2bfloat16_rn(theta[L.w[l] + i % (256 * 256)]);
    }
    for (long long i = tid; i < 4 * 256 + 256 + 1; i += nth) {
        float v;
        if (i < 4 * 256) v = __bfloat162float(__float2bfloat16_rn(theta[L.b[i / 256] + i % 256]));
        else if (i < 4 * 256 + 256) v = __bfloat162float(__float2bfloat16_rn(theta[L.w[4] + (i - 1024)]));
        else v = __bfloat162float(__float2bfloat16_rn(theta[L.b[4]]));
        f[i] = v;
    }
}

// X [n x 8] FP32 -> Xp [n x 64] BF16 (zero padded)
__global__ void k_mlp_pad_input(long long n, const float *__restrict__ X, __nv_bfloat16 *__restrict__ Xp) {
    pdl_begin();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n * 64;
         i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / 64;
        const int c = (int)(i % 64);
        Xp[i] = __float2bfloat16_rn(c < MLP_IN ? X[r * MLP_IN + c] : 0.f);
    }
}

// Ensemble mean and spread (max - min): member m's output is its MLP_YPARTS column-group
// partial dots yp[(MLP_YPARTS m + g) * np + r] (from the fused last layer) plus its bias b5
// (the last float of its packed weights).
constexpr int MLP_YPARTS = 256 / TC_LAYER_CPT;
__global__ void k_mlp_ensemble(long long n, long long np, int nmem, const float *__restrict__ yp,
                               const uint8_t *__restrict__ packed, long long stride, long long b5_off,
                               float *__restrict__ mean, float *__restrict__ spread) {
    pdl_begin();
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
        float s = 0.f, lo = 3.4e38f, hi = -3.4e38f;
        for (int m = 0; m < nmem; m++) {
            const float b5 = *reinterpret_cast<const float *>(packed + (long long)m * stride + b5_off);
            float v = 0.f;
            for (int g = 0; g < MLP_YPARTS; g++) v += yp[((long long)MLP_YPARTS * m + g) * np + r];
            v += b5;
            s += v;
            lo = fminf(lo, v);
            hi = fmaxf(hi, v);
        }
        mean[r] = s / (float)nmem;
        if (spread) spread[r] = hi - lo;
    }
}

}  // namespace opb

OPB_API long long opb_mlp_packed_bytes(void) { return MLP_PACK_BYTES; }

OPB_API int opb_mlp_pack(const float *theta, void *packed) {
    OPB_REQUIRE(theta && packed, OPB_E_NULL);
    OPB_REQUIRE(aligned(packed, 16), OPB_E_ALIGN);
    launch_pdl(k_mlp_pack, grid_ew(3LL * 256 * 256), 256, 0, stream(), theta, reinterpret_cast<uint8_t *>(packed));
    return launch_check();
}

// Inference workspace bytes for n rows (n padded to a multiple of 128 internally).
OPB_API long long opb_mlp_infer_workspace_bytes(long long n, int nmem) {
    const long long np = (n + 127) / 128 * 128;
    return np * 64 * 2 + 2 * np * 256 * 2 + (long long)MLP_YPARTS * nmem * np * 4 + 1024;
}

// Inference form: 1 = one fused kernel per member (default), 0 = one launch per layer with
// the activations through HBM.  Both give bit-identical outputs.
static int g_mlp_fused = 1;

// Ensemble inference on the tensor cores: members m = 0..nmem-1 with packed weights at
// packed + m * member_stride bytes; X [n x 8] normalised features (FP32).  mean [n] and
// spread [n] (optional) receive the ensemble mean and max - min of the member outputs.
OPB_API int opb_mlp_infer(const void *packed, int nmem, long long member_stride, const float *X, long long n,
                          void *ws, long long ws_bytes, float *mean, float *spread) {
    OPB_NVTX("opb_mlp_infer");
    OPB_REQUIRE(packed && X && ws && mean, OPB_E_NULL);
    OPB_REQUIRE(nmem >= 1 && n >= 1 && member_stride >= MLP_PACK_BYTES, OPB_E_ARG);
    OPB_REQUIRE(ws_bytes >= opb_mlp_infer_workspace_bytes(n, nmem), OPB_E_ARG);
    OPB_REQUIRE(aligned(packed, 16) && member_stride % 16 == 0 && aligned(ws, 256), OPB_E_ALIGN);
    cudaStream_t s = stream();
    const long long np = (n + 127) / 128 * 128;
    uint8_t *w8 = reinterpret_cast<uint8_t *>(ws);
    __nv_bfloat16 *Xp = reinterpret_cast<__nv_bfloat16 *>(w8);
    __nv_bfloat16 *Ha = reinterpret_cast<__nv_bfloat16 *>(w8 + np * 64 * 2);
    __nv_bfloat16 *Hb = Ha + np * 256;
    float *ym = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(Hb + np * 256));
    MT((int)cudaMemsetAsync(Xp, 0, np * 64 * 2, s));
    launch_pdl(k_mlp_pad_input, grid_ew(n * 64), 256, 0, s, n, X, Xp);
    for (int m = 0; m < nmem; m++) {
        const uint8_t *pk = reinterpret_cast<const uint8_t *>(packed) + (long long)m * member_stride;
        const __nv_bfloat16 *W1 = reinterpret_cast<const __nv_bfloat16 *>(pk);
        const __nv_bfloat16 *WH = reinterpret_cast<const __nv_bfloat16 *>(pk + MLP_PACK_W1);
        const float *f = reinterpret_cast<const float *>(pk + MLP_PACK_W1 + 3 * MLP_PACK_WH);
        if (g_mlp_fused) {  // all layers in one kernel, the activations in shared memory
            MT(launch_mlp_fused(np, Xp, W1, WH, f, ym + (long long)MLP_YPARTS * m * np, s));
            continue;
        }
        MT(launch_tc_layer((int)np, 256, 64, Xp, 64, W1, 64, 1.f, f, Ha, 256, s));
        MT(launch_tc_layer((int)np, 256, 256, Ha, 256, WH, 256, 1.f, f + 256, Hb, 256, s));
        MT(launch_tc_layer((int)np, 256, 256, Hb, 256, WH + 65536, 256, 1.f, f + 512, Ha, 256, s));
        // last hidden layer with the output layer fused into its epilogue
        MT(launch_tc_layer((int)np, 256, 256, Ha, 256, WH + 2 * 65536, 256, 1.f, f + 768, nullptr, 256, s, f + 1024,
                           ym + (long long)MLP_YPARTS * m * np));
    }
    launch_pdl(k_mlp_ensemble, grid_ew(n), 256, 0, s, n, np, nmem, ym, reinterpret_cast<const uint8_t *>(packed),
               member_stride, MLP_PACK_W1 + 3 * MLP_PACK_WH + 1280LL * 4, mean, spread);
    return launch_check();
}

OPB_API int opb_mlp_set_fused_inference(int on) {
    OPB_REQUIRE(on == 0 || on == 1, OPB_E_ARG);
    g_mlp_fused = on;
    return set_status(OPB_OK);
}
