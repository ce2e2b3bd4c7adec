// Expert pass of a handful of routed pairs (a token or a few): both projections cut into work items of which every SM gets one or two.
// Included by moe.cu alone.
//
// What bounds it: latency.  One token of a 512-expert layer has 10 pairs of 1280 + 2560 rows (6.1 MB of codes, 1 us at the copy
// bandwidth), and each row's sum is one chain of additions.  The row-per-lane walk of moe_gate_up_kernel runs those chains over table
// gathers, with three of sixteen warps at work on the 92 rows of an item, and a barrier and a whole slice of table copied between any
// two parts of the walk.  Here the work of a row is split: some warps gather its table entries, 16 groups at a time, into a short ring
// in shared memory, and the row's thread in another warp adds them in order (g ascending, one accumulator: the same bits).  The
// tables of gate/up arrive in blocks through a ring of their own.  Whatever does not depend on the launch before is asked for
// before the wait: the first table blocks of gate/up (built two launches earlier); codes, scales and row pointers of down.
// us per routed layer of 64 experts, row-per-lane kernels / these: 2560 / 640, one pair 35.7 / 31.1, 4 36.2 / 26.6, 10 40.8 / 32.7, 20
// 68 / 49; 2560 / 256, 10 37.1 / 28.0; 1024 / 256, 4 26.7 / 21.2; 4096 / 1024, 4 45.8 / 35.2, 10 64 / 59; 512 experts, 10 41.4 / 33.5.
#pragma once

namespace ojx {

constexpr int kFewThreads = 512;                    // threads that gather and add; gate/up has one more warp that brings the tables
constexpr int kFewMaxRows = 256;                    // rows of an item: up to eight of the sixteen warps add
constexpr int kFewPre = 8;                          // outlier entries a thread holds while the gathers run
constexpr int kFewProd = kFewThreads * kFewPre;     // products of one pass
constexpr int kFewBlock = 16;                       // groups in a block of table and in a slot of values
constexpr int kFewValRow = kFewBlock + 4;           // floats a row of values takes: 128-bit accesses of eight rows do not share banks
constexpr int kFewMaxBlocks = 12;
constexpr int kFewSlots = 4;                        // slots of values
constexpr int kFewBars = 272;                       // bytes of barriers and of the word that a wait sets when it runs out

// Map of the dynamic shared memory (byte offsets).
struct MoeFewPlan {
    int tile, tiles;  // output rows of an item (gate/up: as many gate rows and as many up rows), items a pair
    int blocks;       // table blocks held
    int stride;       // bytes per row of codes: an odd multiple of 8, so that 64-bit reads of 16 rows use all banks
    int tab, val, codes, x, prod, res;
    int bytes;        // 0: does not fit
};

__device__ __forceinline__ void few_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ void few_bar_init(void* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))), "r"(count) : "memory");
}
__device__ __forceinline__ void few_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))) : "memory");
}

// Rows of an item in two runs (gate rows and up rows; down has one): local row lr is row first0 + lr or first1 + lr - n0 of the
// flattened matrix.
struct FewRows {
    size_t first0, first1;
    int n0, n1;
    __device__ __forceinline__ int n() const { return n0 + n1; }
    __device__ __forceinline__ size_t row(int lr) const { return lr < n0 ? first0 + lr : first1 + (lr - n0); }
};

// Code rows of an item on their way to shared memory (8-byte pieces: G is a multiple of 8, the matrix 8-byte aligned).
__device__ __forceinline__ void few_stage_codes(unsigned char* dst, int stride, const uint8_t* codes, const FewRows& R, int G) {
    const int ppr = G >> 3, total = R.n() * ppr;
    for (int i = threadIdx.x; i < total; i += kFewThreads) {
        const int lr = i / ppr, c = i - lr * ppr;
        const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst + (size_t)lr * stride + c * 8));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(codes + R.row(lr) * G + c * 8) : "memory");
    }
    cp_async_commit();
}

// Table entries of eight groups of a row, in group order.
__device__ __forceinline__ void few_gather8(const float* tab, const unsigned char* codes, float* dst) {
    const uint2 w = *reinterpret_cast<const uint2*>(codes);
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = tab[j * 256 + (((j < 4 ? w.x : w.y) >> ((j & 3) * 8)) & 0xffu)];
    reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

// Barriers of an item.  full[i]: block i of the table ring has landed; empty[i]: its pieces have been gathered; vfull[i]: a slot of
// values is written; vempty[i]: it has been added.
struct FewBars {
    unsigned long long *full, *empty, *vfull, *vempty;
    int* gone;
    __device__ __forceinline__ explicit FewBars(unsigned char* smem)
        : full(reinterpret_cast<unsigned long long*>(smem)), empty(full + kFewMaxBlocks), vfull(empty + kFewMaxBlocks), vempty(vfull + kFewSlots),
          gone(reinterpret_cast<int*>(vempty + kFewSlots)) {}
    __device__ __forceinline__ void init(int blocks, int rows) const {   // one thread; a barrier follows
        const int nrb = (rows + 31) >> 5;
        for (int i = 0; i < blocks; ++i) {
            bulk_bar_init(full + i);
            few_bar_init(empty + i, 2 * nrb);
        }
        for (int i = 0; i < kFewSlots; ++i) {
            few_bar_init(vfull + i, 2 * nrb);
            few_bar_init(vempty + i, nrb);
        }
        *gone = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // A wait inside the hand-over.  One that runs out makes all later ones of the CTA give up at once, and the item's sums NaN.
    __device__ __forceinline__ void wait(unsigned long long* bar, unsigned parity) const {
        if (!bar_wait(static_cast<unsigned>(__cvta_generic_to_shared(bar)), parity, static_cast<unsigned>(__cvta_generic_to_shared(gone))))
            atomicExch(&g_bulk_copy_timeout, 1);
    }
    __device__ __forceinline__ bool failed() const { return *const_cast<volatile int*>(gone) != 0; }
};
static_assert((2 * kFewMaxBlocks + 2 * kFewSlots) * 8 + 4 <= kFewBars && kFewBars % 16 == 0, "room for the barriers");

// Warps that gather for nrb warps that add.  A wait for a phase of a barrier cannot tell "two phases behind" from "done", so a warp may
// wait for a slot's phase only when it knows the phase before it to be over.  What a gathering warp knows is its own last wait: all
// blocks up to kFewSlots before its last piece's are added (they are added in order).  Its next piece must therefore lie at most
// kFewSlots blocks further, and a block has 2 * nrb pieces.
__host__ __device__ constexpr int few_gatherers(int nrb) {
    return kFewThreads / 32 - nrb < kFewSlots * 2 * nrb ? kFewThreads / 32 - nrb : kFewSlots * 2 * nrb;
}

// Sum of row threadIdx.x of the item, in the threads of the first ceil(rows / 32) warps; the other warps gather.  RING: the table comes
// through the ring of `blocks` blocks, otherwise it lies there whole.  A piece of work is 8 groups of 32 rows.
// Order of a gathering warp's waits: the slot first.  Block b - kFewSlots is then known to be added and its table to have landed, so
// that a ring of at least kFewSlots blocks is at most one phase behind at the second wait.
template <bool RING>
__device__ __forceinline__ float few_sums(const FewBars& B, const unsigned char* tab, int blocks, const unsigned char* codes, int stride, float* val,
                                          int rows, int G) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nrb = (rows + 31) >> 5, upb = 2 * nrb;
    const int nblk = (G + kFewBlock - 1) / kFewBlock, slot = rows * kFewValRow;
    float acc = 0.0f;
    if (warp < nrb) {
        const int lr = threadIdx.x;
        for (int b = 0; b < nblk; ++b) {
            B.wait(B.vfull + b % kFewSlots, (unsigned)(b / kFewSlots) & 1u);
            if (lr < rows) {
                const float4* v = reinterpret_cast<const float4*>(val + (size_t)(b % kFewSlots) * slot + lr * kFewValRow);
                const float4 v0 = v[0], v1 = v[1];
                float4 v2 = v0, v3 = v0;
                const bool two = G - b * kFewBlock > 8;
                if (two) { v2 = v[2]; v3 = v[3]; }
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v0.x), v0.y), v0.z), v0.w);
                acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v1.x), v1.y), v1.z), v1.w);
                if (two) {
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v2.x), v2.y), v2.z), v2.w);
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v3.x), v3.y), v3.z), v3.w);
                }
            }
            __syncwarp();
            if (lane == 0) few_arrive(B.vempty + b % kFewSlots);
        }
        return acc;
    }
    const int ng = few_gatherers(nrb);
    for (int u = warp - nrb; u < nblk * upb && warp < nrb + ng; u += ng) {
        const int b = u / upb, r = u - b * upb, lr = (r >> 1) * 32 + lane, g = b * kFewBlock + (r & 1) * 8, at = RING ? b % blocks : b;
        if (b >= kFewSlots) B.wait(B.vempty + b % kFewSlots, (unsigned)(b / kFewSlots - 1) & 1u);
        if (RING) B.wait(B.full + at, (unsigned)(b / blocks) & 1u);
        if (lr < rows && g < G)
            few_gather8(reinterpret_cast<const float*>(tab) + (size_t)(at * kFewBlock + (r & 1) * 8) * 256, codes + (size_t)lr * stride + g,
                        val + (size_t)(b % kFewSlots) * slot + lr * kFewValRow + (r & 1) * 8);
        __syncwarp();
        if (lane == 0) {
            if (RING) few_arrive(B.empty + at);
            few_arrive(B.vfull + b % kFewSlots);
        }
    }
    return acc;
}

// Outlier entries of an item's rows.  They count from the first entry of the first run; the second run's follow on.
struct FewCsr {
    int jb0, je0, jb1, je1, total;
    int col[kFewPre];
    float val[kFewPre];
    __device__ __forceinline__ void ask(const CsrView& csr, const FewRows& R) {
        jb0 = je0 = jb1 = je1 = 0;
        if (csr.nnz <= 0) return;
        jb0 = csr.row_ptrs[R.first0];
        je0 = csr.row_ptrs[R.first0 + R.n0];
        if (R.n1 > 0) {
            jb1 = csr.row_ptrs[R.first1];
            je1 = csr.row_ptrs[R.first1 + R.n1];
        }
    }
    // Entries base .. base + kFewProd - 1, kFewPre a thread, on their way to registers.
    __device__ __forceinline__ void load(const CsrView& csr, int base) {
        if (csr.nnz <= 0) return;
        const int len0 = je0 - jb0;
        total = len0 + je1 - jb1;
#pragma unroll
        for (int u = 0; u < kFewPre; ++u) {
            const int i = base + threadIdx.x + u * kFewThreads, j = i < len0 ? jb0 + i : jb1 + (i - len0);
            col[u] = i < total ? csr.cols[j] : 0;
            val[u] = i < total ? csr.vals[j] : 0.0f;
        }
    }
    // Number of the entry that row pointer p of row lr names.
    __device__ __forceinline__ int number(int p, int lr, const FewRows& R) const { return lr < R.n0 ? p - jb0 : je0 - jb0 + p - jb1; }
    // Sum of row threadIdx.x's entries [s, e), in order, from zero (rows of at most kFewMaxRows threads; all threads call it after load(0)).
    __device__ __forceinline__ float sum(const CsrView& csr, const float* xs, float* prod, bool mine, int s, int e) {
        float acc = 0.0f;
        for (int base = 0; base < total; base += kFewProd) {
            if (base > 0) {
                few_sync();   // the products before these are used up
                load(csr, base);
            }
#pragma unroll
            for (int u = 0; u < kFewPre; ++u) {
                const int i = base + threadIdx.x + u * kFewThreads;
                if (i < total) prod[i - base] = __fmul_rn(val[u], xs[col[u]]);
            }
            few_sync();
            if (mine)
                for (int j = max(s, base); j < min(e, base + kFewProd); ++j) acc = __fadd_rn(acc, prod[j - base]);
        }
        return acc;
    }
};

// Gate/up of tile blockIdx.x % tiles of pair blockIdx.x / tiles, from the token's table [G][256] that an earlier launch built.
// early: that launch is not the one right before this one in the stream, and neither are the activations.
__global__ void __launch_bounds__(kFewThreads + 32, 1) moe_gate_up_few_kernel(const __grid_constant__ MoeProblem P, const __grid_constant__ MoeFewPlan F,
                                                                              int early) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int pair = blockIdx.x / F.tiles, i0 = (blockIdx.x - pair * F.tiles) * F.tile, n = min(F.tile, P.I - i0), rows = 2 * n;
    const int token = pair / P.k_active, G = P.G, nblk = (G + kFewBlock - 1) / kFewBlock;
    const FewBars B(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (!early) chain_begin();
    if (threadIdx.x == 0) B.init(F.blocks, rows);
    __syncthreads();
    if (warp == kFewThreads / 32) {   // brings the table, block by block
        const int first = min(F.blocks, nblk);
        auto bring = [&](int b) {
            bulk_copy_issue(B.full + b % F.blocks, smem_raw + F.tab + (size_t)(b % F.blocks) * kFewBlock * 1024,
                            P.lut_in + ((size_t)token * G + (size_t)b * kFewBlock) * 256, (unsigned)min(kFewBlock, G - b * kFewBlock) * 1024u);
        };
        if (lane == 0)
            for (int b = 0; b < first; ++b) bring(b);
        if (early) chain_begin();
        const bool mine = decode_pair(P, pair).expert >= 0;
        if (lane == 0) {
            int b = first;
            for (; mine && b < nblk; ++b) {
                B.wait(B.empty + b % F.blocks, (unsigned)(b / F.blocks - 1) & 1u);
                if (B.failed()) break;
                bring(b);
            }
            for (int c = b - first; c < b; ++c) bulk_copy_wait(B.full + c % F.blocks, (unsigned)(c / F.blocks) & 1u);   // nothing may land after the CTA has left
        }
        return;
    }
    float* xs = reinterpret_cast<float*>(smem_raw + F.x);
    float* res = reinterpret_cast<float*>(smem_raw + F.res);
    const bool has = P.gu_csr.nnz > 0;
    const XLoad xl{static_cast<const char*>(P.x) + (size_t)token * P.H * (P.io_dtype == OJX_BF16 ? 2 : 4), P.H, P.io_dtype};
    if (has)
        for (int k = threadIdx.x; k < P.H; k += kFewThreads) xs[k] = xl(k);
    if (early) chain_begin();
    const MoePair pr = decode_pair(P, pair);
    if (pr.expert < 0) return;   // uniform across the CTA
    const size_t row0 = (size_t)pr.expert * 2 * P.I + i0;
    const FewRows R{row0, row0 + P.I, n, n};
    const bool mine = (int)threadIdx.x < rows;
    const size_t row = R.row(mine ? threadIdx.x : 0);
    few_stage_codes(smem_raw + F.codes, F.stride, P.gu_codes, R, G);
    FewCsr c;
    c.ask(P.gu_csr, R);
    const int p0 = has && mine ? P.gu_csr.row_ptrs[row] : 0, p1 = has && mine ? P.gu_csr.row_ptrs[row + 1] : 0;
    const float scale = P.gu_scales && mine ? P.gu_scales[row] : 1.0f;
    cp_async_wait<0>();
    few_sync();
    c.load(P.gu_csr, 0);
    float sum = few_sums<true>(B, smem_raw + F.tab, F.blocks, smem_raw + F.codes, F.stride, reinterpret_cast<float*>(smem_raw + F.val), rows, G);
    if (P.gu_scales) sum = __fmul_rn(sum, scale);
    if (has)
        sum = __fadd_rn(sum, c.sum(P.gu_csr, xs, reinterpret_cast<float*>(smem_raw + F.prod), mine, c.number(p0, threadIdx.x, R),
                                   c.number(p1, threadIdx.x, R)));
    if (mine) res[threadIdx.x] = sum;
    few_sync();
    if ((int)threadIdx.x < n) {
        float gate = sum, up = res[n + threadIdx.x];
        if (P.gate_limit > 0.0f) {
            gate = fminf(gate, P.gate_limit);
            up = fminf(fmaxf(up, -P.gate_limit), P.gate_limit);
        }
        P.inter[(size_t)pair * P.I + i0 + threadIdx.x] = B.failed() ? NAN : __fmul_rn(silu_ref(gate), up);
    }
}

// Down projection of tile blockIdx.x % tiles of pair blockIdx.x / tiles.  The pair's table is built here from its intermediate vector,
// which the launch before wrote; the routing is older, so what follows from the expert alone is asked for first.  A thread builds
// the entries of two centroids: with one, reading the activations keeps shared memory busier than the arithmetic takes.
template <int D>
__global__ void __launch_bounds__(kFewThreads, 1) moe_down_few_kernel(const __grid_constant__ MoeProblem P, const __grid_constant__ MoeFewPlan F,
                                                                      const __grid_constant__ PeerLink link) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int pair = blockIdx.x / F.tiles, h0 = (blockIdx.x - pair * F.tiles) * F.tile, n = min(F.tile, P.H - h0), G = P.Gi;
    const MoePair pr = decode_pair(P, pair);
    if (pr.expert >= 0) {
        const FewBars B(smem_raw);
        float* tab = reinterpret_cast<float*>(smem_raw + F.tab);
        float* xs = reinterpret_cast<float*>(smem_raw + F.x);
        const bool has = P.dn_csr.nnz > 0, mine = (int)threadIdx.x < n;
        const FewRows R{(size_t)pr.expert * P.H + h0, 0, n, 0};
        const size_t row = R.first0 + (mine ? threadIdx.x : 0);
        few_stage_codes(smem_raw + F.codes, F.stride, P.dn_codes, R, G);
        FewCsr c;
        c.ask(P.dn_csr, R);
        const int p0 = has && mine ? P.dn_csr.row_ptrs[row] : 0, p1 = has && mine ? P.dn_csr.row_ptrs[row + 1] : 0;
        const float scale = P.dn_scales && mine ? P.dn_scales[row] : 1.0f;
        const int kc = threadIdx.x & 127;
        float cb[2][D];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int d = 0; d < D; ++d) cb[q][d] = kc + 128 * q < P.Kcb ? P.cb_down[(kc + 128 * q) * D + d] : 0.0f;
        if (threadIdx.x == 0) B.init(0, n);
        chain_begin();
        for (int k = threadIdx.x; k < P.I; k += kFewThreads) xs[k] = P.inter[(size_t)pair * P.I + k];
        few_sync();
        // (arithmetic of RowWalker::build_slice: d ascending, separate multiply and add)
        constexpr int U = 2;
        for (int gb = threadIdx.x >> 7; gb < G; gb += 4 * U) {
            float dot[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float4* xp = reinterpret_cast<const float4*>(xs + (gb + 4 * u < G ? gb + 4 * u : gb) * D);
#pragma unroll
                for (int d4 = 0; d4 < D / 4; ++d4) {
                    const float4 xx = xp[d4];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if (d4 == 0) dot[u][q] = __fmul_rn(xx.x, cb[q][0]);
                        else dot[u][q] = __fadd_rn(dot[u][q], __fmul_rn(xx.x, cb[q][4 * d4]));
                        dot[u][q] = __fadd_rn(dot[u][q], __fmul_rn(xx.y, cb[q][4 * d4 + 1]));
                        dot[u][q] = __fadd_rn(dot[u][q], __fmul_rn(xx.z, cb[q][4 * d4 + 2]));
                        dot[u][q] = __fadd_rn(dot[u][q], __fmul_rn(xx.w, cb[q][4 * d4 + 3]));
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (gb + 4 * u < G) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) tab[(gb + 4 * u) * 256 + kc + 128 * q] = kc + 128 * q < P.Kcb ? dot[u][q] : 0.0f;
                }
        }
        c.load(P.dn_csr, 0);
        cp_async_wait<0>();
        few_sync();
        float sum = few_sums<false>(B, smem_raw + F.tab, 0, smem_raw + F.codes, F.stride, reinterpret_cast<float*>(smem_raw + F.val), n, G);
        if (P.dn_scales) sum = __fmul_rn(sum, scale);
        if (has)
            sum = __fadd_rn(sum, c.sum(P.dn_csr, xs, reinterpret_cast<float*>(smem_raw + F.prod), mine, c.number(p0, 0, R), c.number(p1, 0, R)));
        else few_sync();
        if (mine) peer_store(link, P.expert_out + (size_t)pair * P.H + h0 + threadIdx.x, B.failed() ? NAN : sum);
    } else {
        chain_begin();
    }
    peer_signal_when_last(link, gridDim.x);
}

// Items of `pairs` pairs with `outputs` rows of K inputs each (G blocks of codes; `mats` matrices side by side): few rounds of
// the SMs, or nothing (bytes = 0) when they do not fit or the row-per-lane kernels are faster.  Those walk any number of rows per CTA at
// little more than the price of few, while every round here waits for table, codes and outliers anew; down, and gate/up of a short table,
// pay up to the third round, a second round of gate/up over 128 groups only with fewer than 160 rows an item.  us, row-per-lane / the
// rounds that this leaves out: 2560 / 640, 48 pairs 77.8 / 95.1, 64 83.9 / 113.5; 1024 / 640, 64 57.3 / 63.9; 4096 / 1024, 24 99 / 115;
// 2048 / 384, 60 66.3 / 72.6.  Kept: 2560 / 640, 32 71.4 / 70.2; 2560 / 256, 64 65.4 / 59.7; 4096 / 512, 24 81 / 67.
static MoeFewPlan moe_few_plan(int pairs, int sms, int outputs, int mats, int G, int K, bool whole_table) {
    MoeFewPlan f{};
    if (G < 8 || (G & 7) != 0) return f;
    const int nblk = (G + kFewBlock - 1) / kFewBlock;
    const int most_waves = whole_table || G <= 64 ? 3 : 2;
    for (int waves = 1; waves <= most_waves; ++waves) {
        const int want = sms * waves / pairs;
        if (want < 1) continue;
        f.tile = (outputs + want - 1) / want;
        f.tiles = (outputs + f.tile - 1) / f.tile;
        const long long rows = (long long)f.tile * mats;
        if (rows > kFewMaxRows || (!whole_table && G > 128 && waves > 1 && rows > 160)) continue;
        f.stride = (G >> 3) & 1 ? G : G + 8;
        auto up16 = [](long long b) { return (b + 15) & ~15LL; };
        const long long val = kFewSlots * rows * kFewValRow * 4, codes = up16(rows * f.stride), x = up16(4LL * K), prod = 4 * kFewProd, res = up16(4 * rows);
        const long long rest = kFewBars + val + codes + x + prod + res, cap = (long long)sizeof(CoreSmem);
        const long long fit = rest < cap ? (cap - rest) / (kFewBlock * 1024) : 0;
        const int most = whole_table ? nblk : (nblk < kFewMaxBlocks ? nblk : kFewMaxBlocks), least = whole_table ? nblk : (nblk < kFewSlots ? nblk : kFewSlots);   // (fewer than kFewSlots: see few_sums)
        if (fit < least) continue;
        f.blocks = fit < most ? (int)fit : most;
        f.tab = kFewBars;
        f.val = f.tab + f.blocks * kFewBlock * 1024;
        f.codes = f.val + (int)val;
        f.x = f.codes + (int)codes;
        f.prod = f.x + (int)x;
        f.res = f.prod + (int)prod;
        f.bytes = f.res + (int)res;
        return f;
    }
    return f;
}

}  // namespace ojx
