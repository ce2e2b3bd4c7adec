// Codebook-VQ KV cache, a chunk of prompt positions at once: every position's key and value are
// encoded by one launch and every position attends to the tokens up to itself by another.  The
// reference handles a prompt in one model call (ojasx_24x96/engine.py:153-175); its attention over
// a cache is the online softmax of ojasx_24x96/long_context.py:92-176.
//
// Appending and decoding position by position cost two launches per position and layer: a chunk
// of 512 positions took 512 x (14.7 + 5.6) us plus the gaps between launches, 13 ms per layer.
#include <algorithm>
#include <cfloat>

#include "gather_mma.cuh"
#include "handles.h"
#include "launch.h"

namespace ojx {

__device__ __forceinline__ float pf_load(const void* p, size_t i, int dtype) {
    return dtype == OJX_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i])
                             : reinterpret_cast<const float*>(p)[i];
}

// ------------------------------------------------------------------------------------ append
// grid = ceil(positions * B / 128) blocks of rows x 2 * Hkv * G tasks, tasks innermost.  A block encodes one (k|v, head, group) of 128
// rows: thread = row, the 256 centroids and their squared norms broadcast from shared memory.  Same
// distance and the same first-minimum rule as kvq_append_kernel (every dot product a sequential fp32
// sum of rounded products), so the codes are equal.  Bound: fp32 issue, 256 x 19 instructions per
// row and task; a warp per row and task (the one-token kernel) spends as much again on its reduction
// and reads the centroids once per row.
constexpr int kPfAppendThreads = 128;

template <int D>
__global__ void __launch_bounds__(kPfAppendThreads) kvq_append_many_kernel(const __grid_constant__ KvqProblem P) {
    __shared__ __align__(16) float cb_s[256 * D];
    __shared__ float cc_s[256];
    const int G = P.G, tasks = 2 * P.Hkv * G, task = blockIdx.x % tasks;
    const int which = task / (P.Hkv * G), rem = task - which * P.Hkv * G;
    const int h = rem / G, g = rem - h * G;
    const float* cb = (which ? P.v_cb : P.k_cb) + (size_t)h * P.Kcb * D;
    for (int i = threadIdx.x; i < P.Kcb * D; i += kPfAppendThreads) cb_s[i] = cb[i];
    __syncthreads();
    for (int c = threadIdx.x; c < P.Kcb; c += kPfAppendThreads) {
        float cc = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) cc = __fadd_rn(cc, __fmul_rn(cb_s[c * D + d], cb_s[c * D + d]));
        cc_s[c] = cc;
    }
    __syncthreads();
    const int row = (int)(blockIdx.x / tasks) * kPfAppendThreads + threadIdx.x;
    if (row >= P.n_pos * P.B) return;
    const int s = row / P.B, b = row - s * P.B;
    const int T = P.seq_lens[b] + s;
    if (T >= P.max_seq) {   // cache full: the token is dropped, the error flag reports it
        if (task == 0) atomicExch(P.error_flag, 1);
        return;
    }
    const void* src = which ? P.new_v : P.new_k;
    const size_t base = ((size_t)row * P.Hkv + h) * P.head_dim + (size_t)g * D;
    float v[D];
    float vv = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        v[d] = pf_load(src, base + d, P.io_dtype);
        vv = __fadd_rn(vv, __fmul_rn(v[d], v[d]));
    }
    float bd = INFINITY;
    int bi = 0x7fffffff;   // code 255 where no distance is finite (NaN or infinite keys), as kvq_append_kernel writes it
#pragma unroll 4
    for (int c = 0; c < P.Kcb; ++c) {
        const float4* cv = reinterpret_cast<const float4*>(cb_s + c * D);
        float vc = 0.0f;
#pragma unroll
        for (int q = 0; q < D / 4; ++q) {
            const float4 f = cv[q];
            vc = __fadd_rn(vc, __fmul_rn(v[4 * q], f.x));
            vc = __fadd_rn(vc, __fmul_rn(v[4 * q + 1], f.y));
            vc = __fadd_rn(vc, __fmul_rn(v[4 * q + 2], f.z));
            vc = __fadd_rn(vc, __fmul_rn(v[4 * q + 3], f.w));
        }
        const float dist = __fadd_rn(__fsub_rn(vv, __fmul_rn(2.0f, vc)), cc_s[c]);
        if (dist < bd) { bd = dist; bi = c; }
    }
    uint8_t* codes = which ? P.v_codes : P.k_codes;
    codes[(((size_t)b * P.Hkv + h) * P.max_seq + T) * G + g] = (uint8_t)bi;
}

// The sequences' lengths after the chunk (the kernels above and below read the lengths before it).
__global__ void kvq_advance_kernel(int* seq_lens, int B, int n, int max_seq) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < B) seq_lens[b] = min(seq_lens[b] + n, max_seq);
}

// --------------------------------------------------------------------------------- attention
// grid = (tiles of 64 query rows, Hkv, B); a query row is one (position, query head of the KV head).
// Per tile of 64 tokens the codes are expanded into shared memory once and serve all 64 rows; scores
// and values are mma.sync products with an online softmax between them, causal per row.
//
// bf16 queries, keys and values as fp16 products (fp32 ones have a kernel of their own below): every operand is scaled by a power of two (per query row, per codebook, 2^14 for
// probabilities) so that its largest element is in [2^14, 2^15), and split into x = hi + lo with two fp16 numbers: 22 bits of
// mantissa.  hi*hi + hi*lo + lo*hi are accumulated in fp32, in runs short enough that the tensor cores' truncation does not show:
// 8.3e-8 against 64 bits before the output is rounded, 512 positions.  78 us per layer of 512 positions with 32 query heads.
//
// Why mma.sync: three products of at most a few GFLOP per chunk and layer are a few microseconds
// at any tensor rate; what the kernel needs is probabilities that go from the accumulators of the
// first product to the operand registers of the second.  Two CTAs per SM (88 KB each) hide one
// another's expansion of the codes.
constexpr int kPfThreads = 128, kPfRows = 64, kPfTok = 64;

// (a, b) as packed fp16 high parts and the packed fp16 remainders
__device__ __forceinline__ void pf_split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
    const __half la = __float2half_rn(a - __half2float(ha)), lb = __float2half_rn(b - __half2float(hb));
    const __half2 H = __halves2half2(ha, hb), L = __halves2half2(la, lb);
    hi = *reinterpret_cast<const uint32_t*>(&H);
    lo = *reinterpret_cast<const uint32_t*>(&L);
}
// power of two that brings a largest magnitude `m` into [2^14, 2^15) (1 for zeros; tiny values stop at 2^100)
__device__ __forceinline__ float pf_scale(float m) {
    if (!(m > 0.0f) || m > 3e38f) return 1.0f;
    int e;
    frexpf(m, &e);   // m in [2^(e-1), 2^e)
    return ldexpf(1.0f, min(15 - e, 100));
}

template <int HD, int D>
__global__ void __launch_bounds__(kPfThreads) kvq_prefill_kernel(const __grid_constant__ KvqProblem P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LD = HD + 8;                                   // halfs per row: 16 bytes of padding, conflict-free ldmatrix
    constexpr int G = HD / D, KT = HD / 16;
    __half* Kh = reinterpret_cast<__half*>(smem_raw);            // [64][LD]
    __half* Kl = Kh + kPfTok * LD;
    __half* Vh = Kl + kPfTok * LD;
    __half* Vl = Vh + kPfTok * LD;
    __half* cbs = Vl + kPfTok * LD;                              // k hi, k lo, v hi, v lo: [256 * D] each
    __shared__ float red[2][kPfThreads / 32];
    __shared__ float row_scale[kPfRows];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tq = lane & 3;
    const int b = blockIdx.z, h = blockIdx.y, R = P.Hq / P.Hkv;
    const int tile = gridDim.x - 1 - blockIdx.x;                 // the longest contexts start first
    const int T0 = P.seq_lens[b];
    const int pos_per = kPfRows / R, s0 = tile * pos_per;
    const int t_all = min(T0 + min(P.n_pos, s0 + pos_per), P.max_seq);   // tokens the tile's last row sees

    // codebooks of the head, scaled and split
    float inv_kv[2];
    {
        float m[2] = {0.0f, 0.0f};
        const float* src[2] = {P.k_cb + (size_t)h * P.Kcb * D, P.v_cb + (size_t)h * P.Kcb * D};
#pragma unroll
        for (int w = 0; w < 2; ++w)
            for (int i = tid; i < P.Kcb * D; i += kPfThreads) m[w] = fmaxf(m[w], fabsf(src[w][i]));
#pragma unroll
        for (int w = 0; w < 2; ++w) {
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) m[w] = fmaxf(m[w], __shfl_xor_sync(0xffffffffu, m[w], off));
            if (lane == 0) red[w][warp] = m[w];
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const float sc = pf_scale(fmaxf(fmaxf(red[w][0], red[w][1]), fmaxf(red[w][2], red[w][3])));
            inv_kv[w] = 1.0f / sc;
            for (int i = tid; i < 256 * D; i += kPfThreads) {
                const float x = i < P.Kcb * D ? src[w][i] * sc : 0.0f;
                const __half hi = __float2half_rn(x);
                cbs[(2 * w) * 256 * D + i] = hi;
                cbs[(2 * w + 1) * 256 * D + i] = __float2half_rn(x - __half2float(hi));
            }
        }
    }
    // query rows: fp32 into the (still unused) K and V tiles, then into registers
    {
        float* qs = reinterpret_cast<float*>(smem_raw);          // [64][HD + 4]
        for (int i = tid; i < kPfRows * HD; i += kPfThreads) {
            const int row = i / HD, c = i - row * HD, s = s0 + row / R;
            float v = 0.0f;
            if (s < P.n_pos) v = pf_load(P.q, (((size_t)s * P.B + b) * P.Hq + (size_t)h * R + row % R) * HD + c, P.io_dtype);
            qs[row * (HD + 4) + c] = v;
        }
        __syncthreads();
        if (tid < kPfRows) {
            float m = 0.0f;
            for (int c = 0; c < HD; ++c) m = fmaxf(m, fabsf(qs[tid * (HD + 4) + c]));
            row_scale[tid] = pf_scale(m);
        }
        __syncthreads();
    }
    uint32_t qh[KT][4], ql[KT][4];
    float descale[2];
    int limit[2];                                                // last token a row may see
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = warp * 16 + g + 8 * i;
        const float* q = reinterpret_cast<const float*>(smem_raw) + row * (HD + 4);
        const float sc = row_scale[row];
        descale[i] = P.scale * (1.0f / sc) * inv_kv[0] * 1.4426950408889634f;   // scores in units of log 2
        limit[i] = min(T0 + min(s0 + row / R, P.n_pos - 1), P.max_seq - 1);
#pragma unroll
        for (int kk = 0; kk < KT; ++kk)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 v = *reinterpret_cast<const float2*>(q + kk * 16 + j * 8 + 2 * tq);
                pf_split2(v.x * sc, v.y * sc, qh[kk][2 * j + i], ql[kk][2 * j + i]);
            }
    }
    __syncthreads();

    // The running maximum starts at the lowest finite number: scores of -inf (they may overflow) then weigh 0, those of NaN NaN.
    float o[HD / 8][4], m_run[2] = {-FLT_MAX, -FLT_MAX}, l_run[2] = {0.0f, 0.0f}, l_err[2] = {0.0f, 0.0f};
#pragma unroll
    for (int n = 0; n < HD / 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] = 0.0f;

    const uint8_t* kc = P.k_codes + (((size_t)b * P.Hkv + h) * P.max_seq) * G;
    const uint8_t* vc = P.v_codes + (((size_t)b * P.Hkv + h) * P.max_seq) * G;
    // words of four codes (G is a multiple of 4): the next tile's are fetched while this one is computed
    constexpr int W = kPfTok * G / 4, WPT = (W + kPfThreads - 1) / kPfThreads;
    uint32_t kw[WPT], vw[WPT];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int u = 0; u < WPT; ++u) {
            const int i = tid + u * kPfThreads, t = t0 + i / (G / 4);
            kw[u] = vw[u] = 0u;
            if (i < W && t < t_all) {
                kw[u] = *reinterpret_cast<const uint32_t*>(kc + (size_t)t * G + (i % (G / 4)) * 4);
                vw[u] = *reinterpret_cast<const uint32_t*>(vc + (size_t)t * G + (i % (G / 4)) * 4);
            }
        }
    };
    auto expand = [&](uint32_t word, const __half* cb, __half* dst) {   // four centroids, D halfs each
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const __half* c = cb + ((word >> (8 * q)) & 255u) * D;
            if constexpr (D == 4) *reinterpret_cast<uint2*>(dst + q * D) = *reinterpret_cast<const uint2*>(c);
            else {
#pragma unroll
                for (int e = 0; e < D / 8; ++e) reinterpret_cast<uint4*>(dst + q * D)[e] = reinterpret_cast<const uint4*>(c)[e];
            }
        }
    };
    const uint32_t kh_a = static_cast<uint32_t>(__cvta_generic_to_shared(Kh)) + (((lane >> 4) * 8 + (lane & 7)) * LD + ((lane >> 3) & 1) * 8) * 2;
    const uint32_t vt_a = static_cast<uint32_t>(__cvta_generic_to_shared(Vh)) + lane * LD * 2;   // row = token of a 32-token step
    constexpr uint32_t kPart = kPfTok * LD * 2;                  // bytes from a tile's hi part to its lo part

    fetch(0);
    for (int t0 = 0; t0 < t_all; t0 += kPfTok) {
#pragma unroll
        for (int u = 0; u < WPT; ++u) {
            const int i = tid + u * kPfThreads;
            if (i < W) {
                const int off = (i / (G / 4)) * LD + (i % (G / 4)) * 4 * D;
                expand(kw[u], cbs, Kh + off);
                expand(kw[u], cbs + 256 * D, Kl + off);
                expand(vw[u], cbs + 2 * 256 * D, Vh + off);
                expand(vw[u], cbs + 3 * 256 * D, Vl + off);
            }
        }
        __syncthreads();
        if (t0 + kPfTok < t_all) fetch(t0 + kPfTok);
        __syncwarp();   // a lane's fetch depends on its tokens; ldmatrix and mma need the warp converged

        // Chains in the tensor cores stay short (the products of two 16-wide steps here, of one below): they truncate,
        // so that the error of a long chain grows with its length.
        float s[kPfTok / 8][4];
#pragma unroll
        for (int n2 = 0; n2 < kPfTok / 16; ++n2)
#pragma unroll
            for (int k2 = 0; k2 < KT; k2 += 2) {
                float t[2][4];
#pragma unroll
                for (int i = 0; i < 8; ++i) t[i >> 2][i & 3] = 0.0f;
#pragma unroll
                for (int kk = k2; kk < k2 + 2; ++kk) {
                    uint32_t bh[4], bl[4];
                    const uint32_t a = kh_a + (n2 * 16 * LD + kk * 16) * 2;
                    gm_ldsm4(a, bh);
                    gm_ldsm4(a + kPart, bl);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        gm_mma(t[j], qh[kk], bl[2 * j], bl[2 * j + 1]);
                        gm_mma(t[j], ql[kk], bh[2 * j], bh[2 * j + 1]);
                        gm_mma(t[j], qh[kk], bh[2 * j], bh[2 * j + 1]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[2 * n2 + j][i] = k2 == 0 ? t[j][i] : s[2 * n2 + j][i] + t[j][i];
            }
        // scale, mask, online softmax (rows g and g + 8 of the warp's sixteen; a row lives in four lanes)
        float mt[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < kPfTok / 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = t0 + n * 8 + 2 * tq + (i & 1);
                s[n][i] = t <= limit[i >> 1] ? s[n][i] * descale[i >> 1] : -INFINITY;
                mt[i >> 1] = fmaxf(mt[i >> 1], s[n][i]);
            }
        float base[2], l_tile[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mt[i] = fmaxf(mt[i], __shfl_xor_sync(0xffffffffu, mt[i], 1));
            mt[i] = fmaxf(mt[i], __shfl_xor_sync(0xffffffffu, mt[i], 2));
            const float m = fmaxf(m_run[i], mt[i]);
            const float alpha = exp2f(m_run[i] - m);
            m_run[i] = m;
            base[i] = m;
            l_run[i] *= alpha;
            l_err[i] *= alpha;
#pragma unroll
            for (int n = 0; n < HD / 8; ++n) {
                o[n][2 * i] *= alpha;
                o[n][2 * i + 1] *= alpha;
            }
        }
#pragma unroll
        for (int n = 0; n < kPfTok / 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[n][i] = exp2f(s[n][i] - base[i >> 1]);
                l_tile[i >> 1] += s[n][i];
            }
#pragma unroll
        for (int i = 0; i < 2; ++i) {   // compensated: thousands of additions follow on a long context
            const float y = l_tile[i] - l_err[i], t = __fadd_rn(l_run[i], y);
            l_err[i] = __fsub_rn(__fsub_rn(t, l_run[i]), y);
            l_run[i] = t;
        }
        uint32_t ph[kPfTok / 16][4], pl[kPfTok / 16][4];
#pragma unroll
        for (int j = 0; j < kPfTok / 16; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float* c = s[2 * j + (i >> 1)] + (i & 1) * 2;
                pf_split2(c[0] * 16384.0f, c[1] * 16384.0f, ph[j][i], pl[j][i]);
            }
#pragma unroll
        for (int n1 = 0; n1 < HD / 8; ++n1) {   // a tile's products are added to one another, then to the output
            float sum[4];
#pragma unroll
            for (int j2 = 0; j2 < kPfTok / 16; j2 += 2) {
                uint32_t bh[4], bl[4];          // eight dimensions of 32 tokens
                const uint32_t a = vt_a + (j2 * 16 * LD + n1 * 8) * 2;
                gm_ldsm4t(a, bh);
                gm_ldsm4t(a + kPart, bl);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    gm_mma(t, ph[j2 + j], bl[2 * j], bl[2 * j + 1]);
                    gm_mma(t, pl[j2 + j], bh[2 * j], bh[2 * j + 1]);
                    gm_mma(t, ph[j2 + j], bh[2 * j], bh[2 * j + 1]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[i] = j2 + j == 0 ? t[i] : sum[i] + t[i];
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) o[n1][i] += sum[i];
        }
        __syncthreads();   // the tile has been read
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
        const int row = warp * 16 + g + 8 * i, s = s0 + row / R;
        if (s >= P.n_pos) continue;
        const float inv = l_run[i] == 0.0f ? 0.0f : inv_kv[1] * (1.0f / 16384.0f) / l_run[i];
        const size_t base = (((size_t)s * P.B + b) * P.Hq + (size_t)h * R + row % R) * HD;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float v = o[n][2 * i + e] * inv;
                const size_t at = base + n * 8 + 2 * tq + e;
                if (P.io_dtype == OJX_BF16) reinterpret_cast<__nv_bfloat16*>(P.out)[at] = __float2bfloat16_rn(v);
                else reinterpret_cast<float*>(P.out)[at] = v;
            }
    }
}

// fp32 queries, keys and values: the same tiles in fp32.  A pair of fp16 numbers is one bit short of fp32 (fp32 outputs would be off by
// up to 1.5 times as much as position by position), so the products are packed fp32 FMAs here.  128 threads, thread = 8 rows x 4 tokens
// of the scores and 8 rows x HD/16 dimensions of the outputs; keys and values of a tile are expanded one after the other into the same
// place, so that two CTAs (105 KB each) share an SM.  Sums are formed in short runs: a score in runs of 32 dimensions, even and odd ones apart,
// outputs in runs of 16 tokens, of a tile, and of 512 tokens, which are added up in `out`.  Relative error against 64 bits (2-norm), position
// by position through the query tables and here: 64 positions 8.7e-8 / 7.6e-8, 512 1.04e-7 / 8.9e-8, 112 behind 400 1.13e-7 / 9.9e-8 (1.22e-7
// with runs of 16 added to the running outputs; block_dim 4 1.15e-7 / 1.09e-7, eight query heads 1.03e-7 / 9.9e-8), 100 behind 4000
// 1.04e-7 / 7.9e-8.
// Bound: fp32 FMAs (8.2 k clocks per tile of 64 x 64 x 128 with packed pairs) and the latency of shared memory; two CTAs take 21 k for
// two tiles.  us per chunk of 512 positions with its codes, 8 KV heads of 4 query heads, head_dim 128: 768 / 191; behind 2000
// 5375 / 707.  With the rounding errors of the running outputs kept beside them the score loop had no registers left for its loads
// (14 k clocks a tile instead of 8); 256 threads of half the rows read shared memory twice as often (no faster).
constexpr int kPf32Pad = 4, kPf32Dims = 32, kPf32Run = 16, kPf32Tiles = 8;
__device__ __forceinline__ uint64_t pf_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 pf_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t pf_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

template <int HD, int D>
__global__ void __launch_bounds__(kPfThreads, D == 16 && HD == 128 ? 1 : 2) kvq_prefill_f32_kernel(const __grid_constant__ KvqProblem P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LD = HD + kPf32Pad, LP = kPfRows + kPf32Pad, G = HD / D, NC = HD / 64;
    float* Qs = reinterpret_cast<float*>(smem_raw);              // [64][LD]
    float* Ts = Qs + kPfRows * LD;                               // [64][LD] keys, then values of a tile
    float* Ps = Ts + kPfTok * LD;                                // [64 tokens][LP rows] probabilities
    float* cbs = Ps + kPfTok * LP;                               // k, v: [256 * D] each
    uint8_t* codes = reinterpret_cast<uint8_t*>(cbs + 2 * 256 * D);   // [2 tiles][k, v][64 * G]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int b = blockIdx.z, h = blockIdx.y, R = P.Hq / P.Hkv;
    const int tile = gridDim.x - 1 - blockIdx.x;                 // the longest contexts start first
    const int T0 = P.seq_lens[b];
    const int pos_per = kPfRows / R, s0 = tile * pos_per;
    const int t_all = min(T0 + min(P.n_pos, s0 + pos_per), P.max_seq);   // tokens the tile's last row sees

    const uint8_t* kc = P.k_codes + (((size_t)b * P.Hkv + h) * P.max_seq) * G;
    const uint8_t* vc = P.v_codes + (((size_t)b * P.Hkv + h) * P.max_seq) * G;
    constexpr int W = kPfTok * G / 4, WPT = (W + kPfThreads - 1) / kPfThreads;   // words of four codes
    uint32_t kw[WPT], vw[WPT];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int u = 0; u < WPT; ++u) {
            const int i = tid + u * kPfThreads, t = t0 + i / (G / 4);
            kw[u] = vw[u] = 0u;
            if (i < W && t < t_all) {
                kw[u] = *reinterpret_cast<const uint32_t*>(kc + (size_t)t * G + (i % (G / 4)) * 4);
                vw[u] = *reinterpret_cast<const uint32_t*>(vc + (size_t)t * G + (i % (G / 4)) * 4);
            }
        }
    };
    auto keep = [&](int buf) {
#pragma unroll
        for (int u = 0; u < WPT; ++u) {
            const int i = tid + u * kPfThreads;
            if (i >= W) break;
            reinterpret_cast<uint32_t*>(codes + (2 * buf) * kPfTok * G)[i] = kw[u];
            reinterpret_cast<uint32_t*>(codes + (2 * buf + 1) * kPfTok * G)[i] = vw[u];
        }
    };
    // A tile's keys or values: 16-byte pieces, consecutive threads on consecutive pieces of a token.
    auto expand = [&](int buf, int which) {
        const uint8_t* c = codes + (2 * buf + which) * kPfTok * G;
        const float* cb = cbs + which * 256 * D;
#pragma unroll 8
        for (int i = tid; i < kPfTok * HD / 4; i += kPfThreads) {
            const int t = i / (HD / 4), piece = i % (HD / 4);
            *reinterpret_cast<float4*>(Ts + t * LD + piece * 4) =
                *reinterpret_cast<const float4*>(cb + (int)c[t * G + piece / (D / 4)] * D + piece % (D / 4) * 4);
        }
    };

    fetch(0);
    // codebooks and query rows as 16-byte pieces, loads of a batch first
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int i = tid; i < 64 * D; i += kPfThreads) {
        const bool ok = 4 * i < P.Kcb * D;
        const float4 k = ok ? reinterpret_cast<const float4*>(P.k_cb + (size_t)h * P.Kcb * D)[i] : none;
        const float4 v = ok ? reinterpret_cast<const float4*>(P.v_cb + (size_t)h * P.Kcb * D)[i] : none;
        reinterpret_cast<float4*>(cbs)[i] = k;
        reinterpret_cast<float4*>(cbs + 256 * D)[i] = v;
    }
    const bool q16 = (reinterpret_cast<uintptr_t>(P.q) & 15) == 0;
#pragma unroll 8
    for (int i = tid; i < kPfRows * HD / 4; i += kPfThreads) {
        const int row = i / (HD / 4), c = (i - row * (HD / 4)) * 4, s = s0 + row / R;
        const float* src = static_cast<const float*>(P.q) + (((size_t)s * P.B + b) * P.Hq + (size_t)h * R + row % R) * HD + c;
        float4 v = none;
        if (s < P.n_pos) v = q16 ? *reinterpret_cast<const float4*>(src) : make_float4(src[0], src[1], src[2], src[3]);
        *reinterpret_cast<float4*>(Qs + row * LD + c) = v;
    }
    keep(0);

    // The running maximum starts at the lowest finite number: scores of -inf (they may overflow) then weigh 0, those of NaN NaN.
    float m_run[8], l_run[8], l_err[8];
    int limit[8];                                                // last token a row may see
    float m_out[8];                                              // maximum that the sums kept in `out` refer to
    uint64_t o[8][NC][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m_run[i] = m_out[i] = -FLT_MAX;
        l_run[i] = l_err[i] = 0.0f;
        limit[i] = min(T0 + min(s0 + (ty * 8 + i) / R, P.n_pos - 1), P.max_seq - 1);
#pragma unroll
        for (int c = 0; c < NC; ++c) o[i][c][0] = o[i][c][1] = 0ull;
    }
    // The outputs of a run of tiles go to `out`, which keeps the sums of the runs before them until the last one divides by the sum of
    // the probabilities.
    int tiles = 0;
    auto flush = [&](bool last) {
        const bool first = tiles <= kPf32Tiles && !(last && tiles > kPf32Tiles);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float inv = 1.0f;
            if (last) {
                float l = l_run[i];
#pragma unroll
                for (int off = 8; off >= 1; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
                inv = l == 0.0f ? 0.0f : 1.0f / l;
            }
            const int row = ty * 8 + i, s = s0 + row / R;
            if (s < P.n_pos) {
                float* out = static_cast<float*>(P.out) + (((size_t)s * P.B + b) * P.Hq + (size_t)h * R + row % R) * HD;
                const float alpha = first ? 0.0f : expf(m_out[i] - m_run[i]);
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 v = pf_unpack(o[i][c][e >> 1]);
                        const int at = 64 * c + tx * 4 + e;
                        float sum = e & 1 ? v.y : v.x;
                        if (!first) sum += out[at] * alpha;
                        out[at] = last ? sum * inv : sum;
                    }
            }
            m_out[i] = m_run[i];
#pragma unroll
            for (int c = 0; c < NC; ++c) o[i][c][0] = o[i][c][1] = 0ull;
        }
    };
    int buf = 0;
    for (int t0 = 0; t0 < t_all; t0 += kPfTok, buf ^= 1) {
        __syncthreads();   // codes of the tile are there, the tile before has been used
        expand(buf, 0);
        if (t0 + kPfTok < t_all) fetch(t0 + kPfTok);
        __syncthreads();
        float s[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 1
        for (int d0 = 0; d0 < HD; d0 += kPf32Dims) {
            uint64_t a[8][4];                                    // even and odd dimensions apart
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) a[i][j] = 0ull;
#pragma unroll
            for (int d = d0; d < d0 + kPf32Dims; d += 4) {
                ulonglong2 k[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const ulonglong2*>(Ts + (tx + 16 * j) * LD + d);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Qs + (ty * 8 + i) * LD + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) a[i][j] = pf_fma2(q.x, k[j].x, a[i][j]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) a[i][j] = pf_fma2(q.y, k[j].y, a[i][j]);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = pf_unpack(a[i][j]);
                    s[i][j] += f.x + f.y;
                }
        }
        // scale, mask, online softmax (a row lives in sixteen lanes)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float m = m_run[i], l = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = t0 + tx + 16 * j <= limit[i] ? s[i][j] * P.scale : -INFINITY;
                m = fmaxf(m, s[i][j]);
            }
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = expf(s[i][j] - m);
                l += s[i][j];
            }
            if (m != m_run[i]) {
                const float alpha = expf(m_run[i] - m);
                m_run[i] = m;
                l_run[i] *= alpha;
                l_err[i] *= alpha;
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float2 v = pf_unpack(o[i][c][e]);
                        o[i][c][e] = pf_pack(v.x * alpha, v.y * alpha);
                    }
            }
            const float y = l - l_err[i], t = __fadd_rn(l_run[i], y);   // compensated: thousands of additions follow on a long context
            l_err[i] = __fsub_rn(__fsub_rn(t, l_run[i]), y);
            l_run[i] = t;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* p = Ps + (tx + 16 * j) * LP + ty * 8;
            *reinterpret_cast<float4*>(p) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
            *reinterpret_cast<float4*>(p + 4) = make_float4(s[4][j], s[5][j], s[6][j], s[7][j]);
        }
        __syncthreads();   // the keys have been read
        expand(buf, 1);
        if (t0 + kPfTok < t_all) keep(buf ^ 1);
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            uint64_t tsum[8][2];                                 // the tile's sums: one addition a tile to the running outputs
#pragma unroll
            for (int i = 0; i < 8; ++i) tsum[i][0] = tsum[i][1] = 0ull;
#pragma unroll 1
            for (int r0 = 0; r0 < kPfTok && t0 + r0 < t_all; r0 += kPf32Run) {
                uint64_t a[8][2];
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i][0] = a[i][1] = 0ull;
#pragma unroll 8
                for (int t = r0; t < r0 + kPf32Run; ++t) {
                    const float4 p0 = *reinterpret_cast<const float4*>(Ps + t * LP + ty * 8), p1 = *reinterpret_cast<const float4*>(Ps + t * LP + ty * 8 + 4);
                    const float p[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Ts + t * LD + 64 * c + tx * 4);
                    uint64_t pp[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) pp[i] = pf_pack(p[i], p[i]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i][0] = pf_fma2(pp[i], v.x, a[i][0]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) a[i][1] = pf_fma2(pp[i], v.y, a[i][1]);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float2 sum = pf_unpack(tsum[i][e]), f = pf_unpack(a[i][e]);
                        tsum[i][e] = pf_pack(sum.x + f.x, sum.y + f.y);
                    }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float2 sum = pf_unpack(o[i][c][e]), f = pf_unpack(tsum[i][e]);
                    o[i][c][e] = pf_pack(sum.x + f.x, sum.y + f.y);
                }
        }
        if (++tiles % kPf32Tiles == 0 && t0 + kPfTok < t_all) flush(false);
    }
    flush(true);
}

// ------------------------------------------------------------------------------------- host side
template <int HD, int D>
static int launch_prefill_f32_t(const KvqProblem& P, cudaStream_t s) {
    constexpr size_t smem = sizeof(float) * ((size_t)(kPfRows + kPfTok) * (HD + kPf32Pad) + kPfTok * (kPfRows + kPf32Pad) + 2 * 256 * (size_t)D) + 4 * kPfTok * (HD / D);
    OJX_CUDA_TRY(cudaFuncSetAttribute(kvq_prefill_f32_kernel<HD, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int pos_per = kPfRows / (P.Hq / P.Hkv);
    kvq_prefill_f32_kernel<HD, D><<<dim3((P.n_pos + pos_per - 1) / pos_per, P.Hkv, P.B), kPfThreads, smem, s>>>(P);
    OJX_CUDA_TRY(cudaGetLastError());
    count_launch(1);
    return OJX_OK;
}

template <int HD, int D>
static int launch_prefill_t(const KvqProblem& P, cudaStream_t s) {
    if (P.io_dtype == OJX_F32) return launch_prefill_f32_t<HD, D>(P, s);
    constexpr size_t smem = sizeof(__half) * (4 * (size_t)kPfTok * (HD + 8) + 4 * 256 * (size_t)D);
    static_assert(sizeof(float) * kPfRows * (HD + 4) <= smem, "query rows are staged in the tiles");
    OJX_CUDA_TRY(cudaFuncSetAttribute(kvq_prefill_kernel<HD, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int R = P.Hq / P.Hkv, pos_per = kPfRows / R;
    kvq_prefill_kernel<HD, D><<<dim3((P.n_pos + pos_per - 1) / pos_per, P.Hkv, P.B), kPfThreads, smem, s>>>(P);
    OJX_CUDA_TRY(cudaGetLastError());
    count_launch(1);
    return OJX_OK;
}

template <int HD>
static int launch_prefill_d(const KvqProblem& P, cudaStream_t s) {
    switch (P.D) {
        case 4: return launch_prefill_t<HD, 4>(P, s);
        case 8: return launch_prefill_t<HD, 8>(P, s);
        case 16: return launch_prefill_t<HD, 16>(P, s);
        default: return OJX_ERR_UNSUPPORTED;
    }
}

// Codebooks that high and low parts do not hold (infinities, wide ranges) go position by position: an infinite value of a masked
// token would be multiplied by its probability of zero.
bool kvq_prefill_supported(const KvqProblem& P) {
    const int R = P.Hq / P.Hkv;
    return P.even_books && R <= kPfRows && kPfRows % R == 0 && P.G % 4 == 0 && P.B <= 65535 && P.Hkv <= 65535 &&
           (P.head_dim == 64 || P.head_dim == 128) && (P.D == 4 || P.D == 8 || P.D == 16);
}

int launch_kvq_prefill_attention(const KvqProblem& P, cudaStream_t s) {
    if (!kvq_prefill_supported(P)) return OJX_ERR_UNSUPPORTED;
    switch (P.head_dim) {
        case 64: return launch_prefill_d<64>(P, s);
        case 128: return launch_prefill_d<128>(P, s);
        default: return OJX_ERR_UNSUPPORTED;
    }
}

template <int D>
static int launch_append_many_t(const KvqProblem& P, cudaStream_t s) {
    const long long rows = (long long)P.n_pos * P.B;
    const long long blocks = (rows + kPfAppendThreads - 1) / kPfAppendThreads * 2 * P.Hkv * P.G;
    if (rows > 0x7fffffff - kPfAppendThreads || blocks > 0x7fffffff) return OJX_ERR_TOO_LARGE;
    kvq_append_many_kernel<D><<<(unsigned)blocks, kPfAppendThreads, 0, s>>>(P);
    OJX_CUDA_TRY(cudaGetLastError());
    count_launch(1);
    return OJX_OK;
}

int launch_kvq_append_many(const KvqProblem& P, cudaStream_t s) {
    if (!P.new_k || !P.new_v || P.n_pos <= 0) return OJX_ERR_ARG;
    switch (P.D) {
        case 4: return launch_append_many_t<4>(P, s);
        case 8: return launch_append_many_t<8>(P, s);
        case 16: return launch_append_many_t<16>(P, s);
        default: return OJX_ERR_UNSUPPORTED;
    }
}

int launch_kvq_advance(const KvqProblem& P, cudaStream_t s) {
    kvq_advance_kernel<<<(P.B + 127) / 128, 128, 0, s>>>(P.seq_lens, P.B, P.n_pos, P.max_seq);
    OJX_CUDA_TRY(cudaGetLastError());
    count_launch(1);
    return OJX_OK;
}

}  // namespace ojx
