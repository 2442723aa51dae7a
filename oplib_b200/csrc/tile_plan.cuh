// Which K-blocks a squaring issues: the ones whose operand parts are not all zero.
// Part of gemm_tc.cu.
//
// A transition matrix over a short time is nearly banded: the density t away from the
// diagonal falls like a Gaussian, and split2 writes no parts below 2^-40 (FP16 parts underflow
// there), so most of the blocks inside the generator's structural band (which doubles with every
// squaring, while the density spreads with its square root) hold exact zeros.  Of the 256 x 256 x
// 64 blocks that the band leaves, those with both operands non-zero are 3.8 of 9.4 dense
// products over the 14 squarings of the SV lattice (d = 6144), 0.8 of 4.4 on a 2048-node
// local-vol lattice.  A left-out block adds +0 products to an accumulator, so the results are
// the same bits -- as long as the other operand is finite.  Whoever stores a value that is NaN or
// infinite, or at 2 or above, where FP16 parts are, sets TilePlan::wild, and from the next level on
// a solve's squarings take no notice of their plans (0 x NaN makes the row NaN, as it does in the
// full product), and its renormalisations leave out no block.
//
// Whoever writes the parts marks the blocks (32 rows x 64 columns) that hold a non-zero hi part
// (lo parts are zero where hi is); before the next squaring one launch of k_tile_plan turns the
// marks into one bit per K-block for every output tile, leaves out the tiles that are zero and
// stay zero, orders the others by the K-blocks they issue, most first (the persistent CTAs walk
// the tiles round robin, and the counts now differ by an order of magnitude between the diagonal
// and the corners), clears the marks that the squaring is going to write, and forms the row
// fixes of the previous level on the way (it replaces that kernel's launch).  It costs a launch of
// 4-6 us per level, so single lattices below OPB_PLAN_MIN_D states, whose whole product takes about 16
// us, go without.  A dense generator has it too: given densely, a banded one of 2048 states takes
// 720 us with its plans, 1330 before there were any; one that leaves no block zero pays for them up
// to there (1017 -> 1065 us) and not from 3072 states on.

struct TilePlanArgs {
    TilePlan pl;
    const uint32_t *work;  // batched items (problem << 16 | m-tile << 8 | n-tile); null: a single product's tiles
    int n, tm, tn;         // items and their tiles
    int level;
    // single product: size, band, marks of its operand; group_m as the product's
    int d, group_m;
    const int *band;
    const uint8_t *occ;
    const TcProblem *probs;  // batched: the squaring's problems (band, occ_in)
    uint8_t *clear;  // marks to be written next (clear_bytes, a multiple of 16)
    long long clear_bytes;
    // row fixes of the previous level (E-form): one problem, or all lattices that square at this level
    const double *partial;
    int nparts;
    double2 *fix;
    const BatchLattice *lats;
    int nlat, parts_div;
    long long total_rows;
};

constexpr int TP_THREADS = 256, TP_BUCKETS = 128;
constexpr uint16_t kIdle = 0xffff;

// The tile of item t of a single product: the raster of k_tc_gemm's get_item.
__device__ __forceinline__ void raster_tile(int t, int mtiles, int ntiles, int group_m, int &mt, int &nt) {
    const int GM = group_m > 0 ? group_m : 8;
    const int per_group = GM * ntiles;
    const int group = t / per_group, first_m = group * GM;
    const int gm = min(mtiles - first_m, GM);
    const int r = t - group * per_group;
    mt = first_m + r % gm;
    nt = r / gm;
}

__global__ void __launch_bounds__(TP_THREADS) k_tile_plan(TilePlanArgs a) {
    pdl_begin();
    const unsigned wild = *a.pl.wild;
    const long long tid = blockIdx.x * (long long)TP_THREADS + threadIdx.x, nth = (long long)gridDim.x * TP_THREADS;
    for (long long i = tid; i < a.clear_bytes / 16; i += nth) reinterpret_cast<uint4 *>(a.clear)[i] = make_uint4(0, 0, 0, 0);
    // ---- row fixes
    if (a.lats && a.level > 0) {
        for (long long t = tid; t < a.total_rows; t += nth) {
            int lo = 0, hi = a.nlat - 1;
            while (lo < hi) {  // last lattice with row_off <= t
                const int mid = (lo + hi + 1) >> 1;
                if (a.lats[mid].row_off <= t) lo = mid; else hi = mid - 1;
            }
            const BatchLattice &L = a.lats[lo];
            if (L.niter <= a.level) continue;
            const int row = (int)(t - L.row_off);
            L.fix[row] = row_fix(L.partial, L.d, L.d / a.parts_div, row, 1);
        }
    } else if (!a.lats && a.fix) {
        for (long long r = tid; r < a.d; r += nth) a.fix[r] = row_fix(a.partial, a.d, a.nparts, (int)r, 1);
    }
    // ---- K-block masks, a warp per item
    const int lane = threadIdx.x & 31;
    const long long warp = tid >> 5, nwarps = nth >> 5;
    const TilePlan &l = a.pl;
    for (long long t = warp; t < a.n; t += nwarps) {
        int mt, nt, d = a.d, h0;
        const uint8_t *occ = a.occ;
        uint32_t w;
        if (a.work) {
            w = a.work[t];
            const TcProblem &pr = a.probs[w >> 16];
            mt = (int)((w >> 8) & 255u);
            nt = (int)(w & 255u);
            d = pr.M;
            h0 = pr.band;
            occ = pr.occ_in;
        } else {
            raster_tile((int)t, d / a.tm, d / a.tn, a.group_m, mt, nt);
            h0 = a.band ? *a.band : 0;
            w = (uint32_t)mt << 16 | (uint32_t)nt;
        }
        const int m0 = mt * a.tm, n0 = nt * a.tn, ncb = d / 64;
        const int nc = min(a.tn, d - n0) / 64, nr = min(a.tm, d - m0) / 32;  // (the last tiles may overhang)
        int kb0, nkb;
        band_kblocks(h0 > 0 ? level_band(h0, a.level) : -1, m0, a.tm, n0, a.tn, d, 64, 2, kb0, nkb);
        int total = 0;
        if (nkb > 0) {
            for (int w0 = 0; w0 < l.nw; w0++) {
                const int kb = 32 * w0 + lane;
                bool on = false;
                if (kb >= kb0 && kb < kb0 + nkb) {
                    uint32_t ra = 0, rb = 0;
                    for (int u = 0; u < nr; u++) ra |= occ[(long long)(m0 / 32 + u) * ncb + kb] & 1u;
                    if (ra)
                        for (int v = 0; v < 2; v++)
                            for (int c = 0; c < nc; c++) rb |= occ[(long long)(2 * kb + v) * ncb + n0 / 64 + c] & 1u;
                    on = ra && rb;
                }
                const uint32_t bits = __ballot_sync(0xffffffffu, on);
                total += __popc(bits);
                if (lane == 0) l.kmask[t * l.nw + w0] = bits;
            }
        }
        // a tile that is zero and stays zero has nothing to do; its row sums start as zeros (one
        // outside twice the band is so by the band alone, and has no mask)
        bool idle = total == 0;
        if (idle && nkb > 0) {
            bool mine = false;
            for (int i = lane; i < nr * nc; i += 32)
                mine |= occ[(long long)(m0 / 32 + i / nc) * ncb + n0 / 64 + i % nc] != 0;
            idle = !__any_sync(0xffffffffu, mine) && (m0 >= n0 + a.tn || n0 >= m0 + a.tm);
        }
        if (lane == 0) {
            l.count[t] = idle ? kIdle : (uint16_t)total;
            l.tile[t] = w;
        }
    }
    // ---- the last block orders the items: buckets of K-block counts, most first
    __shared__ unsigned last;
    __shared__ int bucket[TP_BUCKETS];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(l.done, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int shift = l.nw > 4 ? 32 - __clz(l.nw * 32 / TP_BUCKETS) : 0;
    for (int pass = 0; pass < 2; pass++) {
        if (pass == 0) {
            for (int i = threadIdx.x; i < TP_BUCKETS; i += TP_THREADS) bucket[i] = 0;
            __syncthreads();
        }
        for (int t0 = 0; t0 < a.n; t0 += TP_THREADS) {
            const int t = t0 + threadIdx.x;
            const int cnt = t < a.n ? (int)__ldcg(&l.count[t]) : kIdle;
            // (idle items and those past the end join no bucket)
            const int key = cnt != kIdle ? TP_BUCKETS - 1 - min(cnt >> shift, TP_BUCKETS - 1) : -1;
            const unsigned same = __match_any_sync(0xffffffffu, key);
            const int leader = __ffs(same) - 1, rank = __popc(same & ((1u << lane) - 1u));
            int at = 0;
            if (key >= 0 && lane == leader) at = atomicAdd(&bucket[key], __popc(same));
            at = __shfl_sync(0xffffffffu, at, leader);
            if (pass == 1 && key >= 0) l.order[at + rank] = make_uint2((uint32_t)t, __ldcg(&l.tile[t]));
        }
        __syncthreads();
        if (pass == 0 && threadIdx.x < 32) {  // exclusive sums of the bucket sizes
            int run = 0;
            for (int b0 = 0; b0 < TP_BUCKETS; b0 += 32) {
                const int v = bucket[b0 + lane];
                int s = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, s, o);
                    if (lane >= o) s += u;
                }
                bucket[b0 + lane] = run + s - v;
                run += __shfl_sync(0xffffffffu, s, 31);
            }
            if (lane == 0) {
                l.nlist[0] = (unsigned)run;
                l.nlist[1] = wild;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *l.done = 0u;
}

static int launch_tile_plan(TilePlanArgs &a, cudaStream_t s) {
    const long long items = a.n, rows = a.lats ? a.total_rows : a.fix ? a.d : 0;
    const long long want = std::max({(items + 7) / 8, (rows + TP_THREADS - 1) / TP_THREADS,
                                     (a.clear_bytes / 16 + TP_THREADS - 1) / TP_THREADS, 1LL});
    const int grid = (int)std::min<long long>(want, 4LL * num_sms());
    launch_pdl(k_tile_plan, grid, TP_THREADS, 0, s, a);
    return (int)cudaGetLastError();
}
