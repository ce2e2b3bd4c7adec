// Top-k MoE over VQ-coded experts for bf16 batches that route several tokens to an expert: the experts' weights are
// gathered from the codebooks into mma.sync operands once per sixteen tokens (gather_mma.cuh) instead of once per token
// (split_manifold_lut_experiment/native/src/ojasx_lut_cpu.cpp:213-365, fp32 up to the order of a row's sum, rounded once
// to bf16).  fp32 batches stay on the table kernels: their contract is the reference's order of additions.
//
// The table kernels spend a shared-memory gather per (code, token) and copy a token's 393 KB table for every pair.  Here a
// code costs 32 bytes of shared-memory reads for up to sixteen tokens (eight in the down pass).  256 tokens of 512 experts
// (hidden 2560, inter 640, top-10): expert passes 1.08 -> 0.74 ms; of 64 experts, the whole layer: 1.17 -> 0.54 ms.
// L1 pipe 83 % busy in the gate/up pass, 81 % in the down pass (128 tokens of 64 experts); a quarter of both passes are the
// outliers' reads of single elements.  Codebooks and intermediate vectors have 22 bits here; of the outputs 2.0e-4 to 2.9e-4 are
// not the 64-bit result rounded to bf16, of the table kernels' 2.4e-4 to 4.1e-4 (ten layers of five shapes, fewer in each).
//
//   moe_item_plan_kernel     pairs grouped by expert, cut into items of up to sixteen pairs
//   moe_gather_prep_kernel   vectors as fp16 hi + lo fragments, scaled by a power of two per vector (tokens, then inter)
//   moe_gather_up_kernel     item x part of the intermediate indices: silu(gate) * up
//   moe_gather_down_kernel   item x half of its pairs x part of the hidden rows
// and the ordered combine of moe.cu.
//
// Vectors are columns of the products.  A bf16 token is one exact fp16 column (gate/up: one or two tiles of eight pairs).
// The intermediate vectors are fp32, high and low parts: with up to four pairs in columns 0..3 and 4..7 of one tile, else
// in a tile each, and all four products are formed and added in the same order either way, so that a pair's result does
// not depend on its neighbours.
#include <atomic>
#include <cstdlib>

#include "block_scan.cuh"
#include "gather_mma.cuh"
#include "handles.h"
#include "launch.h"
#include "peer.cuh"
#include "silu.cuh"

namespace ojx {

constexpr int kMgPairs = 16;                 // pairs of an item; the down pass takes them in two halves
// As many warps as 96 registers a thread leave room for: 20 per SM, in one CTA (gate/up: the table and sixteen columns of the
// hidden width fill the SM) or in two (down).  A warp takes units of 16 intermediate indices, or 32 hidden rows, of an item's
// part; a part of fewer units than warps leaves the rest idle (inter 256: 8 of 20 in gate/up).  Two parts per item let SMs
// that finish early share the last items.
constexpr int kMgUpThreads = 640, kMgDownThreads = 320;
constexpr int kMgParts = 2;

struct MgArgs {
    MoeProblem P;
    int* plan;                // [0] items, [1] claims of gate/up, [2] claims of down, [3] pairs; sorted pairs; items
    const uint4* x_frag;      // [tokens][chunks_x][2 parts ...]: hi then lo, 512 bytes per chunk each
    const float* x_inv;
    const uint4* i_frag;      // the same for the pairs' intermediate vectors
    const float* i_inv;
    int chunks_x, chunks_i;
};

struct MgItem { int expert, first, count, pad; };

__device__ __forceinline__ int mg_local_expert(const MoeProblem& P, int pair) {
    const int e = P.topk_idx[pair] - P.expert_offset;
    // ojasx_lut_cpu.cpp:284-286: ids outside the expert table and |w| < 1e-8 are skipped.
    return (e < 0 || e >= P.E || fabsf(P.topk_w[pair]) < 1e-8f) ? -1 : e;
}

__global__ void __launch_bounds__(1024) moe_item_plan_kernel(const __grid_constant__ MoeProblem P, int width, int* __restrict__ plan) {
    extern __shared__ int plan_smem[];
    chain_begin();
    int *cnt = plan_smem, *start = plan_smem + P.E;
    __shared__ int warp_tot[33];
    const int pairs = P.n_tokens * P.k_active;
    int* sorted = plan + 4;
    int* items = plan + 4 + pairs;
    for (int e = threadIdx.x; e < P.E; e += blockDim.x) cnt[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = mg_local_expert(P, p);
        if (e >= 0) atomicAdd(&cnt[e], 1);
    }
    __syncthreads();
    const int per = (P.E + (int)blockDim.x - 1) / (int)blockDim.x;   // every thread owns a run of experts
    const int lo = min(P.E, (int)threadIdx.x * per), hi = min(P.E, lo + per);
    int np = 0, ni = 0, tp, ti;
    for (int e = lo; e < hi; ++e) {
        np += cnt[e];
        ni += (cnt[e] + width - 1) / width;
    }
    int bp = block_exclusive_scan(np, warp_tot, &tp), bi = block_exclusive_scan(ni, warp_tot, &ti);
    for (int e = lo; e < hi; ++e) {
        start[e] = bp;
        for (int c = 0; c < cnt[e]; c += width, ++bi) {
            items[4 * bi] = e;
            items[4 * bi + 1] = bp + c;
            items[4 * bi + 2] = min(width, cnt[e] - c);
        }
        bp += cnt[e];
    }
    if (threadIdx.x == 0) {
        plan[0] = ti;
        plan[1] = plan[2] = 0;
        plan[3] = tp;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < pairs; p += blockDim.x) {
        const int e = mg_local_expert(P, p);
        if (e >= 0) sorted[atomicAdd(&start[e], 1)] = p;
    }
}

// One CTA per vector (list: vector ids at list[0 .. *count), else all); K is a multiple of 8.  A vector with an infinity or
// NaN gets a NaN scale.
__global__ void __launch_bounds__(128) moe_gather_prep_kernel(const void* __restrict__ x, int io_dtype, int K, int chunks, const int* __restrict__ list,
                                                              const int* __restrict__ count, uint4* __restrict__ frag, float* __restrict__ inv_out) {
    __shared__ uint32_t red[4];
    if (list && (int)blockIdx.x >= *count) return;
    const int v = list ? list[blockIdx.x] : blockIdx.x, G = K / 8;
    auto load = [&](int g, float (&f)[8]) {
        if (g >= G) {
#pragma unroll
            for (int d = 0; d < 8; ++d) f[d] = 0.0f;
        } else if (io_dtype == OJX_BF16) {
            const uint32_t* p = reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(x) + (size_t)v * K) + g * 4;
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                f[2 * d] = __uint_as_float(p[d] << 16);
                f[2 * d + 1] = __uint_as_float(p[d] & 0xffff0000u);
            }
        } else {
            const float* p = static_cast<const float*>(x) + (size_t)v * K + g * 8;
#pragma unroll
            for (int d = 0; d < 8; ++d) f[d] = p[d];
        }
    };
    uint32_t m = 0u;
    for (int g = threadIdx.x; g < G; g += 128) {
        float f[8];
        load(g, f);
#pragma unroll
        for (int d = 0; d < 8; ++d) m = max(m, __float_as_uint(f[d]) & 0x7fffffffu);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = max(max(red[0], red[1]), max(red[2], red[3]));
    float scale, inv;
    gm_scale(m, scale, inv);
    if (threadIdx.x == 0) inv_out[v] = m >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : inv;
    uint32_t* out = reinterpret_cast<uint32_t*>(frag + (size_t)v * chunks * 64);
    for (int g = threadIdx.x; g < chunks * kGmChunk; g += 128) {
        float f[8];
        load(g, f);
        const int step = g & 15;
        uint32_t* at = out + (g / kGmChunk) * 128 + (step >> 1) * 16 + (step & 1) * 2 + ((g >> 4) & 1);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float a = f[2 * p] * scale, b = f[2 * p + 1] * scale;
            const __half2 h = __floats2half2_rn(a, b);
            at[p * 4] = *reinterpret_cast<const uint32_t*>(&h);
            at[chunks * 128 + p * 4] = gm_pack(a - __low2float(h), b - __high2float(h));
        }
    }
}

// Row sum in the reference's order, for vectors (or codebooks) with infinities or NaN.
template <class X>
__device__ __noinline__ float mg_row_exact(const uint8_t* codes, int G, const float* cb, int Kcb, X x) {
    float acc = 0.0f;
    for (int g = 0; g < G; ++g) {
        const int c = codes[g];
        float dot = 0.0f;
        if (c < Kcb) {
            dot = __fmul_rn(x(g * 8), cb[c * 8]);
            for (int d = 1; d < 8; ++d) dot = __fadd_rn(dot, __fmul_rn(x(g * 8 + d), cb[c * 8 + d]));
        }
        acc = __fadd_rn(acc, dot);
    }
    return acc;
}

template <class X>
__device__ __noinline__ float mg_outliers_exact(const CsrView& csr, size_t row, int K, X x) {
    float o = 0.0f;
    if (csr.nnz > 0)
        for (int j = csr.row_ptrs[row]; j < csr.row_ptrs[row + 1]; ++j)
            if ((unsigned)csr.cols[j] < (unsigned)K) o = __fadd_rn(o, __fmul_rn(csr.vals[j], x(csr.cols[j])));
    return o;
}

struct MgX {
    const void* p;
    int io_dtype;
    __device__ float operator()(int i) const {
        return io_dtype == OJX_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]) : static_cast<const float*>(p)[i];
    }
};

// What a CTA of either pass keeps in shared memory besides the table: the item's columns, `ld` bytes each.
struct MgItemS {
    float inv[kMgPairs];
    int pair[kMgPairs];
    int expert, count, part;
};

// Claims the next (item, half, part), brings its columns in.  False when the list is empty.  Gate/up (kHalves = 1): high
// parts of the pairs' tokens.  Down (kHalves = 2): high and low parts of the pairs' own vectors, eight pairs.
template <int kHalves>
__device__ __forceinline__ bool mg_next(const MgArgs& A, int* counter, const uint4* frag, const float* inv, int chunks, int ld, unsigned char* cols, MgItemS& S) {
    constexpr int kParts = kHalves;   // parts of a vector that are brought in
    __syncthreads();   // the item before this one has been read
    if (threadIdx.x == 0) {
        S.count = 0;
        for (;;) {
            const int i = atomicAdd(counter, 1);
            if (i >= A.plan[0] * kMgParts * kHalves) break;
            const int* item = A.plan + 4 + A.P.n_tokens * A.P.k_active + 4 * (i / (kMgParts * kHalves));
            const int first = kHalves == 2 ? (i / kMgParts) % 2 * 8 : 0;
            const int n = kHalves == 2 ? min(8, item[2] - first) : item[2];
            if (n <= 0) continue;   // an item of up to eight pairs has no second half
            S.expert = item[0];
            S.count = n;
            S.part = i % kMgParts;
            for (int c = 0; c < n; ++c) S.pair[c] = A.plan[4 + item[1] + first + c];
            break;
        }
    }
    __syncthreads();
    const int count = S.count;
    if (count == 0) return false;
    const int pieces = chunks * 32, lo0 = count <= 4 ? 4 : 8;   // 16-byte pieces of one part of a vector
    for (int i = threadIdx.x; i < count * kParts * pieces; i += blockDim.x) {
        const int c = i / (kParts * pieces), k = i - c * kParts * pieces, part = k >= pieces;
        const int v = kHalves == 1 ? S.pair[c] / A.P.k_active : S.pair[c];
        *reinterpret_cast<uint4*>(cols + (c + part * lo0) * ld + (k - part * pieces) * 16) = __ldg(frag + (size_t)v * 2 * pieces + k);
    }
    if (threadIdx.x < count) S.inv[threadIdx.x] = inv[kHalves == 1 ? S.pair[threadIdx.x] / A.P.k_active : S.pair[threadIdx.x]];
    __syncthreads();
    return true;
}

// Sums of two 16-row tiles (the lane's rows at `rows`) with NT x 8 columns: per row tile and column tile the rows
// (lane >> 2) and + 8 with columns 2 (lane & 3) and + 1.
template <int NT>
__device__ __forceinline__ void mg_tiles(float (&tot)[2][NT][4], const uint8_t* const (&rows)[2], int G, int chunks, const unsigned char* cols, int ld, uint32_t table) {
    const int lane = threadIdx.x & 31;
    const bool wide = (G & 15) == 0;
    uint32_t w[2][4], wn[2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m) gm_load_codes(wn[m], rows[m], 0, lane >> 4, G, wide);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) tot[m][n][e] = 0.0f;
    const unsigned char* mine = cols + (lane >> 2) * ld + (lane & 3) * 16;
    for (int c = 0; c < chunks; ++c) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) w[m][i] = wn[m][i];
        if (c + 1 < chunks) {
#pragma unroll
            for (int m = 0; m < 2; ++m) gm_load_codes(wn[m], rows[m], c + 1, lane >> 4, G, wide);
        }
        const unsigned char* at = mine + c * 512;
        gm_chunk<2, NT, 2>(tot, w, min(16, G - c * kGmChunk), table,
                        [&](int j, int n) { return *reinterpret_cast<const uint4*>(at + n * 8 * ld + j * 64); });
    }
}

// Sums over the outliers of row `row` with pairs 8 n + p0 and + 1, in entry order; lo0 > 0: low parts lo0 columns further.
template <int NP>
__device__ __forceinline__ void mg_outliers(float (&o)[NP][2], const CsrView& csr, int row, int K, const unsigned char* cols, int ld, int lo0, const MgItemS& S, int p0) {
#pragma unroll
    for (int n = 0; n < NP; ++n) o[n][0] = o[n][1] = 0.0f;
    const int js = csr.row_ptrs[row], je = csr.row_ptrs[row + 1];
    for (int j = js; j < je; j += 4) {
        int col[4];
        float val[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int jj = min(j + u, je - 1);
            col[u] = csr.cols[jj];
            val[u] = csr.vals[jj];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j + u < je && (unsigned)col[u] < (unsigned)K) {
                const int g = col[u] >> 3, d = col[u] & 7, step = g & 15;
                const unsigned char* at = cols + (g >> 5) * 512 + (step >> 1) * 64 + (d >> 1) * 16 + ((step & 1) * 2 + ((g >> 4) & 1)) * 4 + (d & 1) * 2;
#pragma unroll
                for (int n = 0; n < NP; ++n)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int p = n * 8 + p0 + q;
                        float xv = __half2float(*reinterpret_cast<const __half*>(at + p * ld));
                        if (lo0 > 0) xv += __half2float(*reinterpret_cast<const __half*>(at + (p + lo0) * ld));
                        o[n][q] = __fadd_rn(o[n][q], __fmul_rn(val[u], xv * S.inv[p]));
                    }
            }
    }
}

template <int NT>
__device__ __forceinline__ void mg_up_unit(const MgArgs& A, const MgItemS& S, const unsigned char* cols, int ld, uint32_t table, float inv_cb, int unit) {
    const MoeProblem& P = A.P;
    const int lane = threadIdx.x & 31, g = lane >> 2, i0 = unit * 16;
    const size_t row0 = (size_t)S.expert * 2 * P.I + i0;
    const uint8_t* rows[2] = {P.gu_codes + (row0 + (lane & 15)) * P.G, P.gu_codes + (row0 + P.I + (lane & 15)) * P.G};
    float v[2][NT][4];
    mg_tiles<NT>(v, rows, P.G, A.chunks_x, cols, ld, table);
    const int p0 = (lane & 3) * 2;
    if (p0 >= S.count) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {   // rows g and g + 8
        float o[2][NT][2] = {};
        const size_t rg = row0 + g + 8 * h, ru = rg + P.I;
        if (P.gu_csr.nnz > 0) {
            mg_outliers<NT>(o[0], P.gu_csr, (int)rg, P.H, cols, ld, 0, S, p0);
            mg_outliers<NT>(o[1], P.gu_csr, (int)ru, P.H, cols, ld, 0, S, p0);
        }
        const float sg = P.gu_scales ? P.gu_scales[rg] : 1.0f, su = P.gu_scales ? P.gu_scales[ru] : 1.0f;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int p = n * 8 + p0 + q;
                if (p >= S.count) continue;
                float gate = v[0][n][2 * h + q] * inv_cb * S.inv[p], up = v[1][n][2 * h + q] * inv_cb * S.inv[p];
                const int pair = S.pair[p];
                if (isnan(gate) || isnan(up)) {
                    const MgX x{static_cast<const __nv_bfloat16*>(P.x) + (size_t)(pair / P.k_active) * P.H, OJX_BF16};
                    gate = mg_row_exact(P.gu_codes + rg * P.G, P.G, P.cb_in, P.Kcb, x);
                    up = mg_row_exact(P.gu_codes + ru * P.G, P.G, P.cb_in, P.Kcb, x);
                    o[0][n][q] = mg_outliers_exact(P.gu_csr, rg, P.H, x);
                    o[1][n][q] = mg_outliers_exact(P.gu_csr, ru, P.H, x);
                }
                gate = __fadd_rn(__fmul_rn(gate, sg), o[0][n][q]);
                up = __fadd_rn(__fmul_rn(up, su), o[1][n][q]);
                if (P.gate_limit > 0.0f) {
                    gate = fminf(gate, P.gate_limit);
                    up = fminf(fmaxf(up, -P.gate_limit), P.gate_limit);
                }
                P.inter[(size_t)pair * P.I + i0 + g + 8 * h] = __fmul_rn(silu_ref(gate), up);
            }
    }
}

// Persistent CTAs claim (item, part); a warp takes 16 intermediate indices (their gate rows and up rows) over the whole
// width, so nothing is reduced across warps and SiLU needs no exchange.  Bound: shared-memory wavefronts, 16 per step and
// warp for the two tiles' hi and lo parts plus 4 for the columns.
__global__ void __launch_bounds__(kMgUpThreads, 1) moe_gather_up_kernel(const __grid_constant__ MgArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t red[kMgUpThreads / 32];
    __shared__ MgItemS S;
    const float inv_cb = gm_build_table(smem_raw, red, A.P.cb_in, A.P.Kcb, threadIdx.x);
    const uint32_t table = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)) + (threadIdx.x & 7) * 16;
    unsigned char* cols = smem_raw + kGmTable;
    const int ld = A.chunks_x * 512 + 64, units = A.P.I / 16, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    while (mg_next<1>(A, A.plan + 1, A.x_frag, A.x_inv, A.chunks_x, ld, cols, S)) {
        const int u1 = units * (S.part + 1) / kMgParts;
        for (int u = units * S.part / kMgParts + warp; u < u1; u += warps) {
            if (S.count <= 8) mg_up_unit<1>(A, S, cols, ld, table, inv_cb, u);
            else mg_up_unit<2>(A, S, cols, ld, table, inv_cb, u);
            __syncwarp();   // lanes without a pair have left the unit early
        }
    }
}

template <int NT>
__device__ __forceinline__ void mg_down_unit(const MgArgs& A, const MgItemS& S, const unsigned char* cols, int ld, uint32_t table, float inv_cb, int unit, const PeerLink& link) {
    const MoeProblem& P = A.P;
    const int lane = threadIdx.x & 31, g = lane >> 2, h0 = unit * 32;
    const size_t row0 = (size_t)S.expert * P.H + h0;
    const uint8_t* rows[2] = {P.dn_codes + (row0 + (lane & 15)) * P.Gi, P.dn_codes + (row0 + 16 + (lane & 15)) * P.Gi};
    float t[2][NT][4], v[2][4];
    mg_tiles<NT>(t, rows, P.Gi, A.chunks_i, cols, ld, table);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {   // high parts' sum, then low parts'
            if constexpr (NT == 2) v[m][e] = t[m][0][e] + t[m][1][e];
            else {
                const float o = __shfl_xor_sync(0xffffffffu, t[m][0][e], 2);
                v[m][e] = (lane & 2) ? o + t[m][0][e] : t[m][0][e] + o;
            }
        }
    const int p0 = NT == 1 ? (lane & 1) * 2 : (lane & 3) * 2;
    if (p0 >= S.count || (NT == 1 && (lane & 2))) return;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int hr = m * 16 + g + 8 * h;
            const size_t r = row0 + hr;
            float o[1][2] = {};
            if (P.dn_csr.nnz > 0) mg_outliers<1>(o, P.dn_csr, (int)r, P.I, cols, ld, NT == 1 ? 4 : 8, S, p0);
            const float scale = P.dn_scales ? P.dn_scales[r] : 1.0f;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (p0 + q >= S.count) break;
                float s = v[m][2 * h + q] * inv_cb * S.inv[p0 + q];
                const int pair = S.pair[p0 + q];
                if (isnan(s)) {
                    const MgX x{P.inter + (size_t)pair * P.I, OJX_F32};
                    s = mg_row_exact(P.dn_codes + r * P.Gi, P.Gi, P.cb_down, P.Kcb, x);
                    o[0][q] = mg_outliers_exact(P.dn_csr, r, P.I, x);
                }
                peer_store(link, P.expert_out + (size_t)pair * P.H + h0 + hr, __fadd_rn(__fmul_rn(s, scale), o[0][q]));
            }
        }
}

__global__ void __launch_bounds__(kMgDownThreads, 2) moe_gather_down_kernel(const __grid_constant__ MgArgs A, const __grid_constant__ PeerLink link) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint32_t red[kMgDownThreads / 32];
    __shared__ MgItemS S;
    const float inv_cb = gm_build_table(smem_raw, red, A.P.cb_down, A.P.Kcb, threadIdx.x);
    const uint32_t table = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)) + (threadIdx.x & 7) * 16;
    unsigned char* cols = smem_raw + kGmTable;
    const int ld = A.chunks_i * 512 + 64, units = A.P.H / 32, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    while (mg_next<2>(A, A.plan + 2, A.i_frag, A.i_inv, A.chunks_i, ld, cols, S)) {
        const int u1 = units * (S.part + 1) / kMgParts;
        for (int u = units * S.part / kMgParts + warp; u < u1; u += warps) {
            if (S.count <= 4) mg_down_unit<1>(A, S, cols, ld, table, inv_cb, u, link);
            else mg_down_unit<2>(A, S, cols, ld, table, inv_cb, u, link);
            __syncwarp();
        }
    }
    peer_signal_when_last(link, gridDim.x);
}

// ------------------------------------------------------------------------------------- host side
static size_t mg_smem(int chunks) { return kGmTable + 16 * ((size_t)chunks * 512 + 64); }

bool moe_gather_wanted(const MoeProblem& P) {
    if (P.io_dtype != OJX_BF16 || !P.even_books || !P.lut_in || !P.plan || P.D != 8 || P.G % 8 != 0 || P.Gi % 8 != 0 || P.H != P.G * 8 || P.I != P.Gi * 8 || P.E > 4096) return false;
    if (reinterpret_cast<uintptr_t>(P.x) & 3) return false;   // pairs of bf16 are read as words
    const size_t cx = (P.G + kGmChunk - 1) / kGmChunk, ci = (P.Gi + kGmChunk - 1) / kGmChunk, pairs = (size_t)P.n_tokens * P.k_active;
    if (mg_smem((int)cx) > 224 * 1024 || mg_smem((int)ci) > 110 * 1024) return false;
    if (P.n_tokens * (cx * 1024 + 16) + pairs * (ci * 1024 + 16) > moe_table_bytes(P.n_tokens, P.G, P.D)) return false;
    // The time goes with the experts that are hit, in the chain walk with the pairs: the gather pays from 3.5 expected pairs
    // per expert on, if there are enough items for the SMs.  us per layer at hidden 2560 / inter 640, chain walk against this:
    // 2560 pairs on 512 experts 1329 / 968, 1920 982 / 890, 1280 677 / 800; 1000 on 256 508 / 476, 640 355 / 459; 640 on 128
    // 350 / 299, 400 252 / 278; 2560 on 64 1174 / 541, 400 243 / 209, 240 174 / 204.  OJASX_B200_MOE_GATHER_MIN_PAIRS replaces
    // both conditions.
    const char* e = getenv("OJASX_B200_MOE_GATHER_MIN_PAIRS");
    const long long expect = P.E_total > P.E ? ((long long)pairs * P.E + P.E_total - 1) / P.E_total : (long long)pairs;
    return e ? expect >= atoll(e) : expect >= 400 && 2 * expect >= 7LL * P.E;
}

int launch_moe_item_plan(const MoeProblem& P, int* plan, int width, cudaStream_t s) {
    OJX_CUDA_TRY(launch_chained(moe_item_plan_kernel, 1, 1024, sizeof(int) * 2 * (size_t)P.E, s, P, width, plan));
    count_launch(1);
    return OJX_OK;
}

int launch_moe_gather(const MoeProblem& P, cudaStream_t s, const PeerLink& link) {
    static std::atomic<bool> configured[64];   // the kernels' opt-in, once per device
    int dev = 0;
    OJX_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
        OJX_CUDA_TRY(cudaFuncSetAttribute(moe_gather_up_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
        OJX_CUDA_TRY(cudaFuncSetAttribute(moe_gather_down_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    }
    const int pairs = P.n_tokens * P.k_active, sms = num_sms();
    MgArgs A{};
    A.P = P;
    A.plan = const_cast<int*>(P.plan);
    A.chunks_x = (P.G + kGmChunk - 1) / kGmChunk;
    A.chunks_i = (P.Gi + kGmChunk - 1) / kGmChunk;
    // the token tables' scratch holds the fragments, then their scales
    uint4* p = reinterpret_cast<uint4*>(const_cast<float*>(P.lut_in));
    A.x_frag = p;
    A.i_frag = p + (size_t)P.n_tokens * A.chunks_x * 64;
    A.x_inv = reinterpret_cast<const float*>(A.i_frag + (size_t)pairs * A.chunks_i * 64);
    A.i_inv = A.x_inv + P.n_tokens;
    const int rc = launch_moe_item_plan(P, A.plan, kMgPairs, s);
    if (rc != OJX_OK) return rc;
    moe_gather_prep_kernel<<<P.n_tokens, 128, 0, s>>>(P.x, P.io_dtype, P.H, A.chunks_x, nullptr, nullptr, const_cast<uint4*>(A.x_frag),
                                                      const_cast<float*>(A.x_inv));
    OJX_CUDA_TRY(cudaGetLastError());
    moe_gather_up_kernel<<<sms, kMgUpThreads, mg_smem(A.chunks_x), s>>>(A);
    OJX_CUDA_TRY(cudaGetLastError());
    moe_gather_prep_kernel<<<pairs, 128, 0, s>>>(P.inter, OJX_F32, P.I, A.chunks_i, A.plan + 4, A.plan + 3, const_cast<uint4*>(A.i_frag),
                                                 const_cast<float*>(A.i_inv));
    OJX_CUDA_TRY(cudaGetLastError());
    moe_gather_down_kernel<<<2 * sms, kMgDownThreads, mg_smem(A.chunks_i), s>>>(A, link);
    OJX_CUDA_TRY(cudaGetLastError());
    count_launch(4);
    return OJX_OK;
}

}  // namespace ojx
