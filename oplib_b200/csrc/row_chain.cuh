// The chained kernels' quoted row: one row of P_m = P_{m-1} . P1, and nothing else of it.
// Part of gemm_tc.cu (it shares that file's tcgen05 / TMA helpers and its error word).
//
// A European solve reads P_m in one row alone, the quoted state's: quotes[m][k] = e^{-rT_m}
// (P_m G)[y0, k].  Row y0 of P_m is a function of row y0 of P_{m-1} and of P1, and in the
// tensor cores every output row is formed by itself, so from the same row of P_{m-1} these kernels
// form the product's row bit for bit as the full product does: the same operand parts, the same MMAs
// (hi.hi, hi.lo, lo.hi per 16 of K) in the same K order into an accumulator that starts from
// zero every 128 of K, the chunks added in order in FP32, then the epilogue's arithmetic.  The row's
// normalisation adds its FP64 sum in another order (256 threads and a shuffle tree, not partials
// per 128 columns), so from the third maturity on a row agrees to that order's 1e-16, or to an
// FP32 rounding that it flips.
// (Callers that ask for the values of every state take the full products.)
//
// What bounds it: one pass over P1's parts per maturity (4 d^2 bytes, 151 MB at d = 6144:
// 23 us of HBM) instead of a d^3 product; at d <= 2048 P1 stays in L2 and the chain of
// dependent launches is what is left.  One item is 64 columns of the row, or 128 in the
// batched form, where the SMs are full anyway; its P1 boxes (64 of K, hi and lo) come through a
// ring of shared-memory stages.
//
// P1's columns are the MMA's M (M-major, as they lie in memory) and the row is its N, so that
// the results are one TMEM column: each epilogue thread owns one column of the row and adds
// its chunks in order.  (With the row as one of M's 128 rows the chunk sums lay across one
// lane and went through shared memory.)  An MMA costs about 40 cycles however few columns it
// has, and the issuing warp's own instructions between them count as much: at d = 6144 a step
// took 60 us with a 64-bit modulo for the ring position, 43 without, 40 without the MMA's
// optional lane mask; the loads alone take 26.
//
// The row's 128 K-values of chunk c sit in row c % 8 of an 8-row swizzle atom (one atom for the
// chunk's first 64 of K, one for the second), so the whole row takes 4 d bytes of shared
// memory, and chunk c's sums are in column c % 8.  N is 16, two atoms; the other rows multiply
// whatever lies in shared memory there (other chunks' values, the ring), as do the 64 M-rows
// past a 64-column item's box: neither rows nor columns mix, and nobody reads those sums.
//
// Measured on B200, whole calls, full chain products -> quoted row: the SV solve (d = 6144, 16
// maturities) 24.65 -> 10.91 ms, its 15 chain products of 873 us becoming 15 row steps of 71 us
// (40 now); 512 nodes, 8 maturities 481 -> 345 us (11.9 + 3.8 us of product and
// renormalisation per maturity -> 9.3 us, and one pricing product for all); 256 lattices of the
// sweep 60.8 -> 38.7 ms.

constexpr int RS_N = 16;        // the MMA's N: two 8-row atoms of the row
constexpr int RS_ACC = 8;       // TMEM accumulators (RS_N columns each)
constexpr int RS_PREP = 256;    // threads that prepare the row; the first W finish the columns
constexpr int RS_THREADS = RS_PREP + 64;
constexpr int RS_MAX_STAGES = 8, RS_MIN_STAGES = 3;
constexpr int RS_MAX_D = 30336;

__host__ __device__ constexpr int row_step_part(int w) { return w * 64 * 2; }  // W columns x 64 of K, one part

struct RowStepParams {
    int m;           // the maturity this launch forms (P_m from P_{m-1}); m >= 2
    int fused;       // 1: P_{m-1}'s normalisation is deferred into this product (ROWSCALE), 0: applied to the row
    int stages;      // ring depth
    int dmax;        // the largest row of the launch (its operand sits in front of the ring)
    float alpha, sscale;
};

__host__ __device__ inline int row_step_atoms(int d) { return (d / 128 + 7) / 8; }
// shared memory: the row's parts (2 parts x 2 halves of a chunk), the ring, and behind it what a
// 64-column item's MMA reads past the last stage's low parts
__host__ inline int row_step_smem(int d, int w, int stages) {
    return row_step_atoms(d) * 4096 + stages * 2 * row_step_part(w) + (w < 128 ? 8192 : 0) + 1024;
}

// The row of P_{m-1} as operand parts: P1's own for m = 2, else from the FP32 row that the
// last product left.  fused: its parts as they stand, inv = 1 / row sum for the products that
// read them; else normalised first (the arithmetic of the renormalisation kernel) and inv = 1.
// put(e, hi, lo) receives eight elements from e on.  Called by RS_PREP threads; returns inv.
template <class Put>
__device__ __forceinline__ double row_parts(const RowChainLat &L, const RowStepParams &p, double *red, Put &&put) {
    const int tid = threadIdx.x, n8 = L.d / 8;
    if (p.m == 2) {
        for (int j = tid; j < n8; j += RS_PREP)
            put(8 * j, reinterpret_cast<const uint4 *>(L.hi)[j], reinterpret_cast<const uint4 *>(L.lo)[j]);
        return 1.0;
    }
    const float4 *c4 = reinterpret_cast<const float4 *>(L.C[(p.m - 1) & 1]);
    double s = 0.0;
    for (int j = tid; j < 2 * n8; j += RS_PREP) {
        const float4 v = c4[j];
        s += (double)v.x + (double)v.y + (double)v.z + (double)v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((tid & 31) == 0) red[tid >> 5] = s;
    asm volatile("bar.sync 1, %0;" ::"n"(RS_PREP) : "memory");
    s = 0.0;
#pragma unroll
    for (int i = 0; i < RS_PREP / 32; i++) s += red[i];
    const double inv = s != 0.0 ? 1.0 / s : 0.0;
    for (int j = tid; j < n8; j += RS_PREP) {
        const float4 a = c4[2 * j], b = c4[2 * j + 1];
        float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (!p.fused) {
#pragma unroll
            for (int u = 0; u < 8; u++) f[u] = (float)((double)f[u] * inv);
        }
        uint4 h, l;
        split2x2(f[0], f[1], h.x, l.x, p.sscale);
        split2x2(f[2], f[3], h.y, l.y, p.sscale);
        split2x2(f[4], f[5], h.z, l.z, p.sscale);
        split2x2(f[6], f[7], h.w, l.w, p.sscale);
        put(8 * j, h, l);
    }
    return p.fused ? inv : 1.0;
}

// Stores eight elements of P_{m-1}'s row into its pricing slot.
__device__ __forceinline__ void row_slot(const RowChainLat &L, int m, int e, const uint4 &h, const uint4 &l) {
    const long long o = (long long)((m - 2) % kRowSlots) * L.d + e;
    *reinterpret_cast<uint4 *>(L.Qhi + o) = h;
    *reinterpret_cast<uint4 *>(L.Qlo + o) = l;
}

// One column of an accumulator, 32 rows a warp.
__device__ __forceinline__ float tmem_ld1(uint32_t taddr) {
    uint32_t v;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(v)::"memory");
    return __uint_as_float(v);
}

template <bool BATCHED, bool F16>
__global__ void __launch_bounds__(RS_THREADS)
    k_row_step(const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo, RowChainLat one,
               RowStepParams p, const RowChainLat *__restrict__ lats, const CUtensorMap *__restrict__ maps,
               const uint32_t *__restrict__ work, int nitems) {
    constexpr int W = BATCHED ? 128 : 64, PART = row_step_part(W), STAGE = 2 * PART;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gbase = smem_raw + (base - raw);
    __shared__ uint64_t bars[2 * RS_MAX_STAGES + 2 * RS_ACC + 2];
    __shared__ double red[RS_PREP / 32];
    __shared__ uint32_t tmem_slot_s;
    __shared__ int abort_s;
    volatile int *abort_flag = &abort_s;
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (RS_MAX_STAGES + s); };
    auto accf_bar = [&](int a) { return bar0 + 8u * (2 * RS_MAX_STAGES + a); };
    auto acce_bar = [&](int a) { return bar0 + 8u * (2 * RS_MAX_STAGES + RS_ACC + a); };
    const uint32_t row_bar = bar0 + 8u * (2 * RS_MAX_STAGES + 2 * RS_ACC);
    const uint32_t drain_bar = row_bar + 8u;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    const int m = p.m;
    const uint32_t ring = base + (uint32_t)row_step_atoms(p.dmax) * 4096u;
    // item t -> lattice, first column
    auto lattice = [&](int t, int &n0) -> int {
        if constexpr (BATCHED) {
            const uint32_t w = work[t];
            n0 = (int)(w & 0xffffu) * W;
            return (int)(w >> 16);
        } else {
            n0 = t * W;
            return 0;
        }
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < RS_ACC; a++) {
            mbar_init(accf_bar(a), 1);
            mbar_init(acce_bar(a), W / 32);
        }
        mbar_init(row_bar, RS_PREP);
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot_s)),
                     "r"(RS_ACC * RS_N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot_s);

    if (warp == RS_PREP / 32) {
        if (lane == 0) {
            // ---------------- TMA producer: P1's parts, 64 rows of K x W columns at a time.  From
            // m = 3 on P1 was there before the step that this launch follows (that step waited
            // for it), so the ring fills without waiting for that step.
            if (BATCHED || m == 2) pdl_wait();
            int s = 0, issued = 0;
            uint32_t ph = 1;  // the parity that a free stage's barrier has passed
            bool ok = true;
            for (int t = blockIdx.x; t < nitems && ok; t += gridDim.x) {
                int n0;
                const int li = lattice(t, n0);
                const CUtensorMap *bh = &mBhi, *bl = &mBlo;
                int d = one.d;
                if constexpr (BATCHED) {
                    bh = maps + 4 * li + 2;
                    bl = maps + 4 * li + 3;
                    d = lats[li].d;
                }
                for (int kb = 0; kb < d / 64; kb++) {
                    if (issued == p.stages && !mbar_wait(empty_bar(s), ph, abort_flag, TC_WAIT_NS)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(full_bar(s), STAGE);
#pragma unroll
                    for (int i = 0; i < W / 64; i++) {
                        const uint32_t at = ring + s * STAGE + i * 8192;
                        tma_load_2d(at, bh, full_bar(s), n0 + 64 * i, kb * 64);
                        tma_load_2d(at + PART, bl, full_bar(s), n0 + 64 * i, kb * 64);
                    }
                    if (issued < p.stages) issued++;
                    if (++s == p.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            if (!ok) {
                atomicExch(&g_tc_error, 21);
                *abort_flag = 1;
                // (bounded) for the copies in flight: the ring's last use of each stage; ph is 1 in
                // the even rounds of the ring
                for (int k = 0; k < issued; k++) {
                    s = s == 0 ? p.stages - 1 : s - 1;
                    if (s == p.stages - 1) ph ^= 1;
                    (void)mbar_wait(full_bar(s), ph ^ 1, abort_flag, 100000000ull);
                }
            }
        }
        __syncwarp();
    } else if (warp == RS_PREP / 32 + 1) {
        // ---------------- MMA issuer: the whole warp walks the loop, one elected lane issues
        if (BATCHED) pdl_wait();
        const uint32_t idesc = umma_idesc_16(RS_N, F16, TC_BM, false, true);
        int s = 0, item = 0;
        uint32_t ph = 0;
        unsigned g = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < nitems && ok; t += gridDim.x, item++) {
            int n0;
            const int li = lattice(t, n0);
            const int d = BATCHED ? lats[li].d : one.d;
            const int natoms = row_step_atoms(d);
            if (!mbar_wait_warp(row_bar, (uint32_t)(item & 1), abort_flag, TC_WAIT_NS)) {
                ok = false;
                break;
            }
            for (int c = 0; c < d / 128 && ok; c++, g++) {
                const int a = (int)(g % RS_ACC);
                if (g >= RS_ACC && !mbar_wait_warp(acce_bar(a), ((g / RS_ACC) + 1) & 1, abort_flag, TC_WAIT_NS)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t dacc = tmem + (uint32_t)(a * RS_N);
                for (int half = 0; half < 2; half++) {
                    if (!mbar_wait_warp(full_bar(s), ph, abort_flag, TC_WAIT_NS)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t brow = base + (uint32_t)(half * natoms + (c >> 3)) * 1024u;
                    const uint64_t dBh = umma_desc_sw<TC_BK>(brow);
                    const uint64_t dBl = umma_desc_sw<TC_BK>(brow + (uint32_t)(2 * natoms) * 1024u);
                    const uint64_t dAh = umma_desc_mn<TC_BK>(ring + s * STAGE);
                    const uint64_t dAl = umma_desc_mn<TC_BK>(ring + s * STAGE + PART);
                    if (elect_one()) {
#pragma unroll
                        for (int k16 = 0; k16 < TC_BK / 16; k16++) {
                            const uint64_t adv = (uint64_t)((k16 * 16 * 128) >> 4), advb = (uint64_t)((k16 * 32) >> 4);
                            umma_bf16(dacc, dAh + adv, dBh + advb, idesc, (half || k16) ? 1u : 0u);
                            umma_bf16(dacc, dAl + adv, dBh + advb, idesc, 1u);
                            umma_bf16(dacc, dAh + adv, dBl + advb, idesc, 1u);
                        }
                        umma_commit(empty_bar(s));
                    }
                    if (++s == p.stages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok && elect_one()) umma_commit(accf_bar(a));
            }
        }
        if (!ok) {
            atomicExch(&g_tc_error, 22);
            *abort_flag = 1;
        }
        if (elect_one()) umma_commit(drain_bar);
        (void)mbar_wait_warp(drain_bar, 0, abort_flag, TC_WAIT_NS);
    } else {
        // ---------------- the row's parts, the chunk sums, the item's columns
        pdl_begin();
        unsigned g = 0;
        int held = -1;  // the lattice whose row is in shared memory
        double inv = 1.0;
        bool ok = true;
        for (int t = blockIdx.x; t < nitems; t += gridDim.x) {
            int n0;
            const int li = lattice(t, n0);
            const RowChainLat &L = BATCHED ? lats[li] : one;
            const int nch = L.d / 128;
            if (li != held) {
                // the previous item's MMAs are done (its sums were read) before its row goes
                const uint32_t natoms = (uint32_t)row_step_atoms(L.d);
                inv = row_parts(L, p, red, [&](int e, const uint4 &h, const uint4 &l) {
                    const int c = e >> 7, half = (e >> 6) & 1, r = c & 7, ch = (e & 63) >> 3;
                    uint8_t *at = gbase + ((uint32_t)half * natoms + (uint32_t)(c >> 3)) * 1024u + r * 128 + ((ch ^ r) << 4);
                    *reinterpret_cast<uint4 *>(at) = h;
                    *reinterpret_cast<uint4 *>(at + 2 * natoms * 1024u) = l;
                    if (n0 == 0) row_slot(L, m, e, h, l);
                });
                if (n0 == 0 && threadIdx.x == 0) L.qinv[(m - 2) % kRowSlots] = inv;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                held = li;
            }
            asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(row_bar) : "memory");
            if (warp < W / 32) {
                float acc = 0.f;
                for (int c = 0; c < nch; c++, g++) {
                    const int a = (int)(g % RS_ACC);
                    if (ok && !mbar_wait_warp(accf_bar(a), (g / RS_ACC) & 1, abort_flag, TC_WAIT_NS)) {
                        atomicExch(&g_tc_error, 23);
                        *abort_flag = 1;
                        ok = false;
                    }
                    if (!ok) break;
                    tc_fence_after();
                    acc = __fadd_rn(acc, tmem_ld1(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(a * RS_N + (c & 7))));
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(acce_bar(a)) : "memory");
                }
                float o = p.alpha * acc;
                if (p.fused && m > 2) o *= (float)inv;
                L.C[m & 1][n0 + threadIdx.x] = o;
            }
            // (after a failed wait the loop runs on without waiting, so that every thread meets
            // the barriers; the error word tells the caller)
            asm volatile("bar.sync 1, %0;" ::"n"(RS_PREP) : "memory");  // the row may go
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(RS_ACC * RS_N) : "memory");
    }
}

// The last maturity's row into its pricing slot (block per lattice); p.m is one past it.
template <bool BATCHED>
__global__ void __launch_bounds__(RS_PREP) k_row_finish(RowChainLat one, RowStepParams p, const RowChainLat *__restrict__ lats) {
    pdl_begin();
    __shared__ double red[RS_PREP / 32];
    const RowChainLat &L = BATCHED ? lats[blockIdx.x] : one;
    const double inv = row_parts(L, p, red, [&](int e, const uint4 &h, const uint4 &l) { row_slot(L, p.m, e, h, l); });
    if (threadIdx.x == 0) L.qinv[(p.m - 2) % kRowSlots] = inv;
}

template <bool BATCHED, bool F16>
static int row_step_attr() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return OPB_E_UNSUPPORTED;
    if (!done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(k_row_step<BATCHED, F16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             227 * 1024 - 1024);
        if (e != cudaSuccess) return (int)e;
        done[dev] = true;
    }
    return OPB_OK;
}

// Ring depth for `items` items of rows of up to d states.  Launches of one item an SM take what
// shared memory holds, up to eight stages (a load takes about 1 us, a stage's MMAs 0.2).  With
// more items two CTAs an SM hide as much and one prepares its row while the other's MMAs run,
// as long as four stages (64 columns; three of 128) allow two.  0: the row does not fit.
static int row_step_stages(int d, int w, int items) {
    const int two = w < 128 ? 4 : RS_MIN_STAGES;
    if (items > num_sms() && row_step_smem(d, w, two) <= 110 * 1024) return two;
    for (int st = RS_MAX_STAGES; st >= RS_MIN_STAGES; st--)
        if (row_step_smem(d, w, st) <= 226 * 1024) return st;
    return 0;
}

bool row_chain_fits(int d) { return d > 0 && d % 128 == 0 && d <= RS_MAX_D && row_step_stages(d, 64, d / 64) > 0; }

int launch_row_step(const RowChainLat &L, const __nv_bfloat16 *Bhi, const __nv_bfloat16 *Blo, int m, int fused, int f16,
                    float alpha, float sscale, cudaStream_t s) {
    if (!row_chain_fits(L.d)) return OPB_E_UNSUPPORTED;
    const int items = L.d / 64;
    const RowStepParams p{m, fused, row_step_stages(L.d, 64, items), L.d, alpha, sscale};
    int r = f16 ? row_step_attr<false, true>() : row_step_attr<false, false>();
    if (r) return r;
    CUtensorMap mh, ml;
    if ((r = make_map_mn(&mh, Bhi, L.d, L.d, L.d, f16)) != OPB_OK) return r;
    if ((r = make_map_mn(&ml, Blo, L.d, L.d, L.d, f16)) != OPB_OK) return r;
    const int smem = row_step_smem(L.d, 64, p.stages);
    const int cap = num_sms() * (smem <= 110 * 1024 ? 2 : 1), grid = items < cap ? items : cap;
    if (f16) launch_pdl(k_row_step<false, true>, grid, RS_THREADS, smem, s, mh, ml, L, p, nullptr, nullptr, nullptr,
                        items);
    else launch_pdl(k_row_step<false, false>, grid, RS_THREADS, smem, s, mh, ml, L, p, nullptr, nullptr, nullptr,
                    items);
    return (int)cudaGetLastError();
}

int launch_row_step_batched(const RowChainLat *lats, const CUtensorMap *maps, const uint32_t *work, int nwork, int dmax,
                            int m, int f16, float alpha, float sscale, cudaStream_t s) {
    if (nwork <= 0) return OPB_OK;
    const RowStepParams p{m, 1, row_step_stages(dmax, 128, nwork), dmax, alpha, sscale};
    if (!row_chain_fits(dmax) || p.stages == 0) return OPB_E_UNSUPPORTED;
    int r = f16 ? row_step_attr<true, true>() : row_step_attr<true, false>();
    if (r) return r;
    const int smem = row_step_smem(dmax, 128, p.stages);
    const int cap = num_sms() * (smem <= 110 * 1024 ? 2 : 1), grid = nwork < cap ? nwork : cap;
    CUtensorMap none;
    std::memset(&none, 0, sizeof(none));
    RowChainLat one{};
    if (f16) k_row_step<true, true><<<grid, RS_THREADS, smem, s>>>(none, none, one, p, lats, maps, work, nwork);
    else k_row_step<true, false><<<grid, RS_THREADS, smem, s>>>(none, none, one, p, lats, maps, work, nwork);
    return (int)cudaGetLastError();
}

int launch_row_finish(const RowChainLat &L, int m, int fused, float sscale, cudaStream_t s) {
    RowStepParams p{m + 1, fused, 0, L.d, 1.f, sscale};
    launch_pdl(k_row_finish<false>, 1, RS_PREP, 0, s, L, p, nullptr);
    return (int)cudaGetLastError();
}

int launch_row_finish_batched(const RowChainLat *lats, int nlat, int m, float sscale, cudaStream_t s) {
    RowStepParams p{m + 1, 1, 0, 0, 1.f, sscale};
    k_row_finish<true><<<nlat, RS_PREP, 0, s>>>(RowChainLat{}, p, lats);
    return (int)cudaGetLastError();
}
