// Kernels on the walk of four vectors at a time (lut_quad.cuh): fp32 linears of a batch, and the expert pass of top-k MoE
// layers that route several tokens to an expert.  Same bits as the kernels of one vector (linear.cu, moe.cu), which rebuild or
// copy a table per vector.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "lut_quad.cuh"
#include "handles.h"
#include "launch.h"
#include "peer.cuh"
#include "silu.cuh"

namespace ojx {

// ------------------------------------------------------------------------------------- linears
// Item: four vectors of the batch x a tile of rows.
__global__ void __launch_bounds__(kQuThreads, 1) lut_linear_quad_kernel(const __grid_constant__ LinearProblem P, int items, float neg_zero,
                                                                        const __grid_constant__ PeerLink link) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    chain_begin();
    if (quad_begin(smem_raw, P.codebook, P.Kcb)) {
        int first = 0;
        const size_t esz = P.io_dtype == OJX_BF16 ? 2 : 4;
        const int rows_out = P.row_stop - P.row_start;
        for (int item = blockIdx.x; item < items; item += gridDim.x) {
            const int q = item / P.tiles, t = item - q * P.tiles, b0 = q * kQuVecs;
            const int r0 = P.row_start + t * P.tile_rows, n = min(P.tile_rows, P.row_stop - r0);
            QuadItem it{P.codes + (size_t)r0 * P.G, P.codes + (size_t)r0 * P.G, n, n, P.G, {}, P.K, P.io_dtype};
#pragma unroll
            for (int c = 0; c < kQuVecs; ++c) it.x[c] = static_cast<const char*>(P.x) + (size_t)(b0 + c < P.batch ? b0 + c : b0) * P.K * esz;
            if ((int)threadIdx.x >= kQuWalkers * 32) quad_ask_outliers(P.csr, r0, n);
            quad_run(smem_raw, it, P.Kcb, first, neg_zero);
            const float4* xs = P.csr.nnz > 0 ? quad_stage_x(smem_raw, it) : nullptr;
            const float4* acc = qu_at<float4>(smem_raw, kQuAcc);
            quad_rows(acc, n, P.csr, P.scales, P.bias, xs, [&](int lr) { return r0 + lr; }, [&](int lr, const float (&r)[4]) {
                const int m = r0 + lr;
#pragma unroll
                for (int c = 0; c < kQuVecs; ++c) {
                    if (b0 + c >= P.batch) break;
                    const size_t o = P.y_full ? (size_t)(b0 + c) * P.y_ld + m : (size_t)(b0 + c) * rows_out + (m - P.row_start);
                    if (P.io_dtype == OJX_BF16) peer_store(link, reinterpret_cast<__nv_bfloat16*>(P.y) + o, __float2bfloat16_rn(r[c]));
                    else peer_store(link, reinterpret_cast<float*>(P.y) + o, r[c]);
                }
            });
            __syncthreads();   // the next item builds tables where x is staged
        }
    }
    peer_signal_when_last(link, gridDim.x);
}

// ------------------------------------------------------------------------------------- MoE
// Items: up to four pairs of one expert (moe_item_plan_kernel) x a tile of the intermediate indices (gate and up rows) or of the
// hidden rows, claimed from a counter.  A table is built per item, so tiles are as large as they may be while there is a group
// for every CTA; the groups of the last, incomplete round are cut into as many tiles as CTAs are left for each.
struct QuadMoe {
    MoeProblem P;
    int* plan;           // [0] groups of pairs, [1] claims of gate/up, [2] claims of down; sorted pairs from [4] on; groups
    int rows, most, step;   // intermediate indices or hidden rows: all, of a tile at most, a tile is a multiple of
    float neg_zero;
};
struct QuadGroup {
    int expert, count;
    int pair[kQuVecs];
};
__device__ __forceinline__ QuadGroup quad_group(const QuadMoe& A, int g) {
    const int* groups = A.plan + 4 + A.P.n_tokens * A.P.k_active;
    QuadGroup r;
    r.expert = groups[4 * g];
    r.count = groups[4 * g + 2];
    const int at = groups[4 * g + 1];
#pragma unroll
    for (int c = 0; c < kQuVecs; ++c) r.pair[c] = A.plan[4 + at + (c < r.count ? c : 0)];
    return r;
}
// Size of a tile when `cut` of them are wanted.
__host__ __device__ inline int quad_tile(int rows, int most, int step, int cut) {
    const int t = ((rows + cut - 1) / cut + step - 1) / step * step;
    return t < most ? t : most;
}
// Calls work(group, first row, rows) for the items a CTA claims; between two items all threads meet.
template <class F>
__device__ __forceinline__ void quad_items(const QuadMoe& A, unsigned char* raw, int counter, F work) {
    volatile int* next = qu_at<volatile int>(raw, kQuCtl + 64);
    const int groups = A.plan[0], ctas = gridDim.x, whole = groups / ctas * ctas, rest = groups - whole;
    const int tile0 = quad_tile(A.rows, A.most, A.step, 1), tiles0 = (A.rows + tile0 - 1) / tile0;
    const int tile1 = quad_tile(A.rows, A.most, A.step, rest ? max(1, ctas / rest) : 1), tiles1 = (A.rows + tile1 - 1) / tile1;
    const int items0 = whole * tiles0, items = items0 + rest * tiles1;
    if (threadIdx.x == 0) *next = atomicAdd(A.plan + counter, 1);
    for (;;) {
        __syncthreads();
        const int item = *next;
        __syncthreads();
        if (item >= items) return;
        if (threadIdx.x == 0) *next = atomicAdd(A.plan + counter, 1);
        const bool last = item >= items0;
        const int j = last ? item - items0 : item, tiles = last ? tiles1 : tiles0, tile = last ? tile1 : tile0, at = j % tiles * tile;
        work(quad_group(A, (last ? whole : 0) + j / tiles), at, min(tile, A.rows - at));
    }
}

__global__ void __launch_bounds__(kQuThreads, 1) moe_gate_up_quad_kernel(const __grid_constant__ QuadMoe A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const MoeProblem& P = A.P;
    chain_begin();
    if (!quad_begin(smem_raw, P.cb_in, P.Kcb)) return;
    int first = 0;
    const size_t esz = P.io_dtype == OJX_BF16 ? 2 : 4;
    quad_items(A, smem_raw, 1, [&](const QuadGroup& g, int i0, int n) {
        const int gate0 = g.expert * 2 * P.I + i0, up0 = gate0 + P.I;
        QuadItem it{P.gu_codes + (size_t)gate0 * P.G, P.gu_codes + (size_t)up0 * P.G, n, 2 * n, P.G, {}, P.H, P.io_dtype};
#pragma unroll
        for (int c = 0; c < kQuVecs; ++c) it.x[c] = static_cast<const char*>(P.x) + (size_t)(g.pair[c] / P.k_active) * P.H * esz;
        if ((int)threadIdx.x >= kQuWalkers * 32) {
            quad_ask_outliers(P.gu_csr, gate0, n);
            quad_ask_outliers(P.gu_csr, up0, n);
        }
        quad_run(smem_raw, it, P.Kcb, first, A.neg_zero);
        const float4* xs = P.gu_csr.nnz > 0 ? quad_stage_x(smem_raw, it) : nullptr;
        float4* acc = qu_at<float4>(smem_raw, kQuAcc);
        quad_rows(acc, 2 * n, P.gu_csr, P.gu_scales, nullptr, xs, [&](int lr) { return lr < n ? gate0 + lr : up0 + lr - n; },
                  [&](int lr, const float (&r)[4]) { acc[lr] = make_float4(r[0], r[1], r[2], r[3]); });
        __syncthreads();
        const float* sums = reinterpret_cast<const float*>(acc);
        for (int j = threadIdx.x; j < 4 * n; j += kQuThreads) {
            const int c = j / n, i = j - c * n;
            if (c >= g.count) break;
            float gate = sums[4 * i + c], up = sums[4 * (n + i) + c];
            if (P.gate_limit > 0.0f) {
                gate = fminf(gate, P.gate_limit);
                up = fminf(fmaxf(up, -P.gate_limit), P.gate_limit);
            }
            int pair = g.pair[0];
#pragma unroll
            for (int q = 1; q < kQuVecs; ++q) pair = c == q ? g.pair[q] : pair;
            P.inter[(size_t)pair * P.I + i0 + i] = __fmul_rn(silu_ref(gate), up);
        }
    });
}

__global__ void __launch_bounds__(kQuThreads, 1) moe_down_quad_kernel(const __grid_constant__ QuadMoe A, const __grid_constant__ PeerLink link) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const MoeProblem& P = A.P;
    chain_begin();
    if (quad_begin(smem_raw, P.cb_down, P.Kcb)) {
        int first = 0;
        quad_items(A, smem_raw, 2, [&](const QuadGroup& g, int h0, int n) {
            const int row0 = g.expert * P.H + h0;
            QuadItem it{P.dn_codes + (size_t)row0 * P.Gi, P.dn_codes + (size_t)row0 * P.Gi, n, n, P.Gi, {}, P.I, OJX_F32};
#pragma unroll
            for (int c = 0; c < kQuVecs; ++c) it.x[c] = P.inter + (size_t)g.pair[c] * P.I;
            if ((int)threadIdx.x >= kQuWalkers * 32) quad_ask_outliers(P.dn_csr, row0, n);
            quad_run(smem_raw, it, P.Kcb, first, A.neg_zero);
            const float4* xs = P.dn_csr.nnz > 0 ? quad_stage_x(smem_raw, it) : nullptr;
            const float4* acc = qu_at<float4>(smem_raw, kQuAcc);
            quad_rows(acc, n, P.dn_csr, P.dn_scales, nullptr, xs, [&](int lr) { return row0 + lr; }, [&](int lr, const float (&r)[4]) {
#pragma unroll
                for (int c = 0; c < kQuVecs; ++c)   // expert-parallel: every rank gets the pair's output
                    if (c < g.count) peer_store(link, P.expert_out + (size_t)g.pair[c] * P.H + h0 + lr, r[c]);
            });
        });
    }
    peer_signal_when_last(link, gridDim.x);
}

// ------------------------------------------------------------------------------------- host side
static int quad_configure() {   // the kernels' opt-in to large shared memory, once per device
    static std::atomic<bool> configured[64];
    int dev = 0;
    OJX_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && configured[dev].load(std::memory_order_relaxed)) return OJX_OK;
    OJX_CUDA_TRY(cudaFuncSetAttribute(lut_linear_quad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQuSmemBytes));
    OJX_CUDA_TRY(cudaFuncSetAttribute(moe_gate_up_quad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQuSmemBytes));
    OJX_CUDA_TRY(cudaFuncSetAttribute(moe_down_quad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQuSmemBytes));
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    return OJX_OK;
}

// Clocks of an item of n rows with `entries` outliers each.  A slice takes 5050 where its table is the bound, 6600 with 1280 rows and
// 9200 with 2560; the rest are the first table, the staging of the activations, and the outliers and results, a thread for every
// kQuThreads-th row.
static double quad_item_clocks(int n, int G, double entries) {
    const double slices = (G + kQuSlice - 1) / kQuSlice;
    return slices * std::max(5050.0, 3900.0 + 2.1 * ((n + 255) / 256 * 256)) + 10000.0 +
           0.5 * (n + (n + kQuThreads - 1) / kQuThreads * kQuThreads) * (2.5 + 1.5 * entries);
}

static bool quad_codes_fit(const uint8_t* codes, int G) { return G > 0 && G % 8 == 0 && (reinterpret_cast<uintptr_t>(codes) & 7) == 0; }

static bool quad_linear_fits(const LinearProblem& P) {
    return P.D == 8 && P.Kcb <= 256 && quad_codes_fit(P.codes, P.G) && (P.csr.nnz <= 0 || P.K <= kQuMaxK);
}

// Outlier entries of a row, on average.
static double linear_entries(const LinearProblem& P) { return P.csr.nnz > 0 ? (double)P.csr.nnz / P.rows_all : 0.0; }

// Tile of a linear's rows that makes the last CTA finish first, and that CTA's clocks.
static int quad_linear_tile(const LinearProblem& P, double* clocks) {
    const int rows = P.row_stop - P.row_start, quads = (P.batch + kQuVecs - 1) / kQuVecs, sms = num_sms();
    const double entries = linear_entries(P);
    int best = 0;
    for (int cut = 1; cut <= 64; ++cut) {
        const int tile = quad_tile(rows, kQuRows, 32, cut), items = quads * ((rows + tile - 1) / tile);
        const double t = (double)((items + sms - 1) / sms) * quad_item_clocks(tile, P.G, entries);
        if (best == 0 || t < *clocks) { *clocks = t; best = tile; }
        if (tile <= 256) break;
    }
    return best;
}

// Whether a linear is faster with four vectors at a time.  The persistent kernel's items take the groups times (140 + 0.066 per row)
// clocks, 2 per row where code rows are no multiples of 16 bytes (its walk then loads them byte by byte), and 1 + 0.66 per entry for
// a row with outliers.  us, that kernel / this, at no, 0.38 % and 5 % outliers:
//   2560 -> 4096, batch 64 47 / 58, 54 / 64, 162 / 122; 96 70 / 63, 83 / 69, 296 / 145; 256 138 / 90, 161 / 104, 587 / 314
//   4096 -> 2560, 64 58 / 87, 66 / 93, 207 / 140; 96 81 / 89, 95 / 98, 372 / 189; 128 80 / 93, 94 / 102, 371 / 213
//   1024 -> 16384, 16 20 / 27, 24 / 30, 53 / 56; 32 29 / 32, 38 / 35, 99 / 80; 64 82 / 40, 108 / 45, 307 / 125
//   2560 -> 1024, 128 36 / 56, 40 / 60, 97 / 85; 256 69 / 59, 77 / 65, 190 / 123; 3136 -> 3106, 4 52 / 75, 54 / 80, 57 / 110; 8 98 / 75, 101 / 80, 108 / 110
bool quad_linear_pays(const LinearProblem& P) {
    if (!quad_linear_fits(P)) return false;
    const char* e = std::getenv("OJASX_B200_QUAD_MIN_BATCH");   // vectors from which a linear comes here, instead of the estimate
    if (e) return P.batch >= atoi(e);
    if (P.batch < kQuVecs) return false;
    const int rows = P.row_stop - P.row_start, sms = num_sms(), tile = plan_tile_rows(rows, P.batch), items = P.batch * ((rows + tile - 1) / tile);
    double four = 0.0;
    quad_linear_tile(P, &four);
    const double row = P.csr.nnz > 0 ? 1.0 + 0.66 * linear_entries(P) : 0.0;
    return four < (double)((items + sms - 1) / sms) * (P.G * (140.0 + (P.G % 16 ? 2.0 : 0.066) * tile) + row * tile);
}

int launch_quad_linear(LinearProblem P, cudaStream_t s, const PeerLink& link) {
    int rc = quad_configure();
    if (rc != OJX_OK) return rc;
    double clocks = 0.0;
    P.tile_rows = quad_linear_tile(P, &clocks);
    P.tiles = (P.row_stop - P.row_start + P.tile_rows - 1) / P.tile_rows;
    const int items = (P.batch + kQuVecs - 1) / kQuVecs * P.tiles;
    OJX_CUDA_TRY(launch_chained(lut_linear_quad_kernel, std::min(items, num_sms()), kQuThreads, kQuSmemBytes, s, P, items, -0.0f, link));
    count_launch(1);
    return OJX_OK;
}

// The two passes' rows, most rows of a tile and multiple of a tile: 256 rows are a block for each of the eight walkers.
static void quad_passes(const MoeProblem& P, QuadMoe (&pass)[2]) {
    pass[0] = QuadMoe{P, const_cast<int*>(P.plan), P.I, kQuRows / 2, 128, -0.0f};
    pass[1] = QuadMoe{P, const_cast<int*>(P.plan), P.H, kQuRows, 256, -0.0f};
}

// Routed pairs are taken four of an expert at a time where that is estimated to be faster than the chain walk pair by pair, whose
// gate/up and down rows take the groups times (113 + 0.08 per row) clocks each (0.5 where code rows are no multiples of 16 bytes and
// every lane walks its own row), and 1 + 0.6 per entry for a row with outliers, whose last round is half a gate/up item longer, and
// whose tables take 0.8 per group and token.  us per routed layer at hidden 2560 / inter 640, that / this, at no and at 0.38 % outliers:
//   512 experts, top 10: 64 tokens 293 / 359, 342 / 398; 96 402 / 465, 469 / 510; 128 531 / 505, 622 / 559; 256 997 / 761, 1174 / 838
//   128 experts, top 8: 32 tokens 143 / 144, 165 / 167; 48 196 / 162, 227 / 172; 64 235 / 225, 270 / 250; 256 773 / 492, 907 / 544
//   64 experts, top 8, 2048 / 768: 32 117 / 127, 133 / 142; 48 160 / 128, 183 / 141; top 4, 1024 / 512: 64 68 / 72, 77 / 78; 96 94 / 73, 107 / 79
bool moe_quad_wanted(const MoeProblem& P) {
    if (!P.plan || P.D != 8 || P.Kcb > 256 || P.E > 4096 || !quad_codes_fit(P.gu_codes, P.G) || !quad_codes_fit(P.dn_codes, P.Gi)) return false;
    if ((P.gu_csr.nnz > 0 && P.H > kQuMaxK) || (P.dn_csr.nnz > 0 && P.I > kQuMaxK)) return false;
    if ((long long)P.E * 2 * P.I > INT32_MAX || (long long)P.E * P.H > INT32_MAX) return false;
    const char* off = std::getenv("OJASX_B200_MOE_CHAIN");
    if (off && off[0] == '0') return false;
    const long long all = (long long)P.n_tokens * P.k_active, expect = P.E_total > P.E ? (all * P.E + P.E_total - 1) / P.E_total : all;
    const char* e = std::getenv("OJASX_B200_MOE_QUAD_MIN_PAIRS");   // expected pairs from which the layer comes here, instead of the estimate
    if (e) return expect >= atoll(e);
    const int sms = num_sms();
    // groups of four: pairs spread over the experts at random
    double groups = 0.0, p = std::exp(-(double)expect / P.E), below = p;
    for (int n = 1; n < 4096 && 1.0 - below > 1e-6; ++n) {
        if (n % kQuVecs == 1) groups += (1.0 - below) * P.E;
        p *= (double)expect / P.E / n;
        below += p;
    }
    const double entries[2] = {P.gu_csr.nnz / (2.0 * P.E * P.I), P.dn_csr.nnz / ((double)P.E * P.H)};
    const int n = (int)(groups + 1.0), whole = n / sms, rest = n % sms, Gs[2] = {P.G, P.Gi}, unit[2] = {2, 1};
    QuadMoe pass[2];
    quad_passes(P, pass);
    double four = 0.0;
    for (int i = 0; i < 2; ++i) {
        const QuadMoe& A = pass[i];
        const int tile0 = quad_tile(A.rows, A.most, A.step, 1), tile1 = quad_tile(A.rows, A.most, A.step, rest ? std::max(1, sms / rest) : 1);
        four += whole * ((A.rows + tile0 - 1) / tile0) * quad_item_clocks(unit[i] * tile0, Gs[i], entries[i]);
        if (rest) four += std::max(1.0, (double)rest * ((A.rows + tile1 - 1) / tile1) / sms) * quad_item_clocks(unit[i] * tile1, Gs[i], entries[i]);
    }
    auto rows = [](double n, int G, double e) { return G * (113.0 + (G % 16 ? 0.5 : 0.08) * n) + (e > 0.0 ? n * (1.0 + 0.6 * e) : 0.0); };
    const double up = rows(2.0 * P.I, P.G, entries[0]), pair = up + rows(P.H, P.Gi, entries[1]);
    return four < 0.97 * ((double)expect / sms * pair + 0.5 * up + 0.8 * P.n_tokens * P.G);   // (the estimates are 3 % off)
}

int launch_moe_quad(const MoeProblem& P, cudaStream_t s, const PeerLink& link) {
    int rc = quad_configure();
    if (rc != OJX_OK) return rc;
    QuadMoe pass[2];
    quad_passes(P, pass);
    if ((rc = launch_moe_item_plan(P, pass[0].plan, kQuVecs, s)) != OJX_OK) return rc;
    OJX_CUDA_TRY(launch_chained(moe_gate_up_quad_kernel, num_sms(), kQuThreads, kQuSmemBytes, s, pass[0]));
    OJX_CUDA_TRY(launch_chained(moe_down_quad_kernel, num_sms(), kQuThreads, kQuSmemBytes, s, pass[1], link));
    count_launch(2);
    return OJX_OK;
}

int take_quad_error(int* out) {
    int v = 0, zero = 0;
    OJX_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_quad_error, sizeof(int)));
    if (v) OJX_CUDA_TRY(cudaMemcpyToSymbol(g_quad_error, &zero, sizeof(int)));
    *out = v;
    return OJX_OK;
}

}  // namespace ojx
