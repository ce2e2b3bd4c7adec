// Decode attention over the codebook-VQ cache on mma.sync, for 8-dimensional blocks (online softmax of
// ojasx_24x96/long_context.py:92-176 over the code stream of
// split_manifold_lut_experiment/native/src/ojasx_lut_kv_cache.cpp:67-132).
//
// Both codebooks of the KV head lie in shared memory as gather_mma.cuh tables, so ldmatrix turns code bytes into
// operands: scores are K (16 tokens x 16 dimensions) times the queries, outputs are V transposed (16 dimensions x 16
// tokens) times the probabilities.  Eight columns hold the query heads of a KV head: four as high and low fp16 parts side
// by side (one product yields x * hi and x * lo), eight as two sets of columns.  Every operand is scaled by a power
// of two and split in two fp16 numbers, 22 bits; sums are fp32.
//
// The chunks of all (KV head, sequence or position) pairs, heads outermost, are shared out evenly over at most one CTA per
// SM; a CTA walks its run of chunks, a whole run of one (sequence, head) at a time.  A warp walks its own 16-token tiles
// with its own running maximum, so the main loop has no barrier; the warps are merged at the end of a run, the runs by the
// last CTA of a (sequence, head).
// Bound: shared-memory wavefronts, 4 per ldmatrix: 64 bytes of K and V centroid parts per code pair, 8 clocks per token at
// 16 groups and 1 for the softmax's shuffles; measured 12 (L1 pipe 75 % busy, tensor pipe 29 % at 16384 tokens x 8).  us per
// decode, query-table kernel and this: 2048 tokens, 8 KV heads of 4 query heads 17.2 / 12.3; 32768 tokens x 16 213 / 180; 8000 x
// 4 with 8 query heads 55.7 / 34.4; 500 x 16 with 8 query heads of 64 17.7 / 11.5; 8000 x 4 with 4 of 64 19.2 / 15.9.  One or two
// query heads per KV head fill a quarter or half of the columns and lose (8000 x 4: 16.4 / 27.4 and 19.7 / 29.3): they keep the
// query-table kernel.
//
// bf16 queries and outputs only.  A pair of fp16 numbers is one bit short of fp32, and that shows: fp32 outputs were off by 1.03e-7
// to 1.28e-7 against 64 bits where the query-table kernel's are by 0.85e-7 to 1.17e-7 (500 to 8000 tokens, head_dim 128).
// Adding every product's high parts in fp32 and reducing the exponents exactly changed nothing.  In bf16 the output's
// own rounding is 1.7e-3 on either kernel.
#include <algorithm>
#include <atomic>

#include "gather_mma.cuh"
#include "handles.h"
#include "launch.h"
#include "peer.cuh"

namespace ojx {

constexpr int kKdThreads = 512, kKdWarps = kKdThreads / 32;

__device__ __forceinline__ uint32_t kd_transpose(uint32_t x) {   // 8x8 matrix of 16-bit elements over the warp
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}

__device__ __forceinline__ void kd_split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = gm_pack(a - __low2float(h), b - __high2float(h));
}

template <int W>
__device__ __forceinline__ void kd_load(uint32_t (&w)[W], const uint8_t* p) {
    if constexpr (W == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        w[0] = v.x;
        w[1] = v.y;
    } else w[0] = *reinterpret_cast<const uint32_t*>(p);
}

template <int R, int G>
__global__ void __launch_bounds__(kKdThreads, 1) kvq_decode_mma_kernel(const __grid_constant__ KvqProblem P, const __grid_constant__ PeerLink link) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kSteps = G / 2, W = G / 8, HD = G * 8, NQ = R == 8 ? 2 : 1;
    __shared__ uint32_t red[2 * kKdWarps];
    __shared__ float m_s[kKdWarps][16], l_s[kKdWarps][R];
    __shared__ int s_last, s_at[3];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3;
    const int Z = P.n_pos > 0 ? P.n_pos * P.B : P.B;
    float* out_s = reinterpret_cast<float*>(smem_raw + 2 * kGmTable);   // [warp][R][HD + 4]
    float inv_kv[2];
    auto build = [&](int h) {   // threads 0..255 build the table of keys, the others that of values
        const int half = tid >> 8;
        gm_build_table(smem_raw + half * kGmTable, red + half * kKdWarps, (half ? P.v_cb : P.k_cb) + (size_t)h * P.Kcb * 8, P.Kcb, tid & 255);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint32_t m = 0u;
            float scale;
#pragma unroll
            for (int w = 0; w < 8; ++w) m = max(m, red[i * kKdWarps + w]);
            gm_scale(m, scale, inv_kv[i]);
        }
    };
    // CTA c starts at chunk c * (Hkv * S) / CTAs of Hkv heads with S chunks each: in head c * Hkv / CTAs whatever S is
    int h = (int)((long long)blockIdx.x * P.Hkv / gridDim.x), built = h;
    build(h);
    cudaGridDependencySynchronize();   // the append before this launch: lengths, codes; the query

    auto length = [&](int z) {
        const int T = P.n_pos > 0 ? min(P.seq_lens[z % P.B] + P.pos0 + z / P.B + 1, P.max_seq) : P.seq_lens[z];
        return min(T, P.n_chunks * P.chunk);   // what the plan and its scratch were made for
    };
    auto chunks = [&](int z) { return (length(z) + P.chunk - 1) / P.chunk; };
    if (warp == 0) {
        int n = 0;
        for (int z = lane; z < Z; z += 32) n += chunks(z);
        const int S = __reduce_add_sync(0xffffffffu, n);
        const long long total = (long long)S * P.Hkv;
        const long long from = total * blockIdx.x / gridDim.x, to = total * (blockIdx.x + 1) / gridDim.x;
        int rest = (int)(from - (long long)h * S);   // chunks of head h before the start
        if (lane == 0) s_at[0] = s_at[1] = 0;
        __syncwarp();
        for (int z0 = 0; to > from && z0 < Z; z0 += 32) {
            const int c = z0 + lane < Z ? chunks(z0 + lane) : 0;
            int sum = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, off);
                if (lane >= off) sum += v;
            }
            const unsigned past = __ballot_sync(0xffffffffu, sum > rest);
            if (past) {
                const int l = __ffs(past) - 1;
                if (lane == l) {
                    s_at[0] = z0 + l;
                    s_at[1] = rest - (sum - c);
                }
                break;
            }
            rest -= __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) s_at[2] = (int)(to - from);
    }
    __syncthreads();
    int z = s_at[0], split = s_at[1], left = s_at[2];
    const int row_heads = P.out_heads > 0 ? P.out_heads : P.Hq;
    while (left > 0 && h < P.Hkv) {
        const int T = length(z), nz = (T + P.chunk - 1) / P.chunk;
        if (split >= nz) {   // the next sequence, after the last one the next head
            split = 0;
            if (++z == Z) {
                z = 0;
                ++h;
            }
            continue;
        }
        const int b = P.n_pos > 0 ? z % P.B : z, n_run = min(nz - split, left);
        const int t_begin = split * P.chunk, t_end = min(T, (split + n_run) * P.chunk);
        float* part = P.partials + ((((size_t)z * P.Hkv + h) * P.n_chunks + split) * R) * (HD + 2);
        if (h != built) {
            __syncthreads();   // the old tables have been read
            build(h);
            built = h;
        }
        const uint8_t* kc = P.k_codes + (((size_t)b * P.Hkv + h) * P.max_seq) * G + (lane >> 4) * (G / 2);
        const uint8_t* vc = P.v_codes + (((size_t)b * P.Hkv + h) * P.max_seq) * G + ((lane >> 3) & 1) * (G / 2);
        const int tk = lane & 15, tv = (lane & 7) + (lane >> 4) * 8;   // the lane's token of a tile: keys, values
        int t0 = t_begin + warp * 16;
        uint32_t kn[W], vn[W];
        if (t0 < t_end) {
            kd_load<W>(kn, kc + (size_t)min(t0 + tk, t_end - 1) * G);
            kd_load<W>(vn, vc + (size_t)min(t0 + tv, t_end - 1) * G);
        }
        // queries as B operands: column g is head g % R, low parts from column R on
        uint32_t q[NQ][kSteps][2];
        float descale[2];
        {
            float x[kSteps][4], top = 0.0f;
            const size_t at = ((size_t)z * P.Hq + (size_t)h * R + g % R) * HD;
#pragma unroll
            for (int i = 0; i < kSteps; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const size_t k = at + ((e >> 1) * kSteps + i) * 8 + 2 * tq + (e & 1);
                    x[i][e] = P.io_dtype == OJX_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(P.q)[k]) : static_cast<const float*>(P.q)[k];
                    top = fmaxf(top, fabsf(x[i][e]));
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            float scale, inv;
            gm_scale(__float_as_uint(top), scale, inv);
#pragma unroll
            for (int i = 0; i < kSteps; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    uint32_t hi, lo;
                    kd_split2(x[i][2 * e] * scale, x[i][2 * e + 1] * scale, hi, lo);
                    if constexpr (NQ == 2) {
                        q[0][i][e] = hi;
                        q[1][i][e] = lo;
                    } else q[0][i][e] = g < R ? hi : lo;
                }
            const float d = P.scale * inv * inv_kv[0] * 1.4426950408889634f;   // scores in units of log 2
            descale[0] = __shfl_sync(0xffffffffu, d, 2 * tq * 4);
            descale[1] = __shfl_sync(0xffffffffu, d, (2 * tq + 1) * 4);
        }
        const uint32_t kt = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)) + (lane & 7) * 16, vt = kt + kGmTable;
        float o[kSteps][4], m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < kSteps; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[i][e] = 0.0f;

        for (; t0 < t_end; t0 += kKdWarps * 16) {
            __syncwarp();   // ldmatrix, mma and movmatrix need the warp converged
            uint32_t kw[W], vw[W];
#pragma unroll
            for (int i = 0; i < W; ++i) {
                kw[i] = kn[i];
                vw[i] = vn[i];
            }
            const int t1 = t0 + kKdWarps * 16;
            if (t1 < t_end) {
                kd_load<W>(kn, kc + (size_t)min(t1 + tk, t_end - 1) * G);
                kd_load<W>(vn, vc + (size_t)min(t1 + tv, t_end - 1) * G);
            }
            auto at = [](uint32_t table, const uint32_t (&w)[W], int i) {   // code i * 128
                return table + (((i & 3) == 0 ? w[i >> 2] << 7 : w[i >> 2] >> (8 * (i & 3) - 7)) & 0x7f80u);
            };
            // Chains in the tensor cores are kept short (four and one products of high parts): they truncate, and a long
            // chain's error grows with its length (5e-6 at 32768 tokens with outputs accumulated there).
            float s[4], sl[4], s2[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] = sl[e] = s2[e] = 0.0f;
            uint32_t hi[2][4], lo[2][4];
            gm_ldsm4(at(kt, kw, 0), hi[0]);
            gm_ldsm4(at(kt, kw, 0) + kGmTable / 2, lo[0]);
#pragma unroll
            for (int i = 0; i < kSteps; ++i) {
                const int c = i & 1;
                if (i + 1 < kSteps) {
                    gm_ldsm4(at(kt, kw, i + 1), hi[c ^ 1]);
                    gm_ldsm4(at(kt, kw, i + 1) + kGmTable / 2, lo[c ^ 1]);
                }
                gm_mma(sl, lo[c], q[0][i][0], q[0][i][1]);
                if (i & 1) gm_mma(s2, hi[c], q[0][i][0], q[0][i][1]);
                else gm_mma(s, hi[c], q[0][i][0], q[0][i][1]);
                if constexpr (NQ == 2) gm_mma(sl, hi[c], q[1][i][0], q[1][i][1]);
            }
            // the first value operands are on their way while the softmax is formed
            gm_ldsm4t(at(vt, vw, 0), hi[0]);
            gm_ldsm4t(at(vt, vw, 0) + kGmTable / 2, lo[0]);
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] = s[e] + s2[e] + sl[e];
        #pragma unroll
            for (int e = 0; e < 4; ++e) {
                if constexpr (R == 4) s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);
                s[e] = t0 + g + (e >> 1) * 8 < t_end ? s[e] * descale[e & 1] : -INFINITY;
                mx[e & 1] = fmaxf(mx[e & 1], s[e]);
            }
#pragma unroll
            for (int off = 4; off <= 16; off <<= 1) {
                mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], off));
                mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], off));
            }
            if (__any_sync(0xffffffffu, mx[0] > m_run[0] || mx[1] > m_run[1])) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float m = fmaxf(m_run[c], mx[c]), alpha = m == -INFINITY ? 1.0f : exp2f(m_run[c] - m);
                    m_run[c] = m;
                    l_run[c] *= alpha;
#pragma unroll
                    for (int i = 0; i < kSteps; ++i) {
                        o[i][c] *= alpha;
                        o[i][2 + c] *= alpha;
                    }
                }
            }
            uint32_t ph[2], pl[2];   // tokens 0..7 and 8..15 of the tile
            // no score above -inf yet: weights 0, or NaN where the scores are (a query with an infinity or NaN), never exp(-inf + inf)
            const float base[2] = {m_run[0] == -INFINITY ? 0.0f : m_run[0], m_run[1] == -INFINITY ? 0.0f : m_run[1]};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float p0 = exp2f(s[2 * e] - base[0]), p1 = exp2f(s[2 * e + 1] - base[1]);
                l_run[0] += p0;
                l_run[1] += p1;
                kd_split2(p0 * 16384.0f, p1 * 16384.0f, ph[e], pl[e]);
                if constexpr (R == 4) ph[e] = tq < 2 ? ph[e] : pl[e];
                ph[e] = kd_transpose(ph[e]);
                if constexpr (NQ == 2) pl[e] = kd_transpose(pl[e]);
            }
#pragma unroll
            for (int i = 0; i < kSteps; ++i) {
                const int c = i & 1;
                if (i + 1 < kSteps) {
                    gm_ldsm4t(at(vt, vw, i + 1), hi[c ^ 1]);
                    gm_ldsm4t(at(vt, vw, i + 1) + kGmTable / 2, lo[c ^ 1]);
                }
                float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                gm_mma(t, lo[c], ph[0], ph[1]);
                if constexpr (NQ == 2) gm_mma(t, hi[c], pl[0], pl[1]);
                gm_mma(t, hi[c], ph[0], ph[1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) o[i][e] += t[e];
            }
        }
        constexpr int kLd = HD + 4;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int off = 4; off <= 16; off <<= 1) l_run[c] += __shfl_xor_sync(0xffffffffu, l_run[c], off);
            const int r = 2 * tq + c;
            const bool mine = r < R;
            if (mine && g == 0) {
                m_s[warp][r] = m_run[c];
                l_s[warp][r] = l_run[c];
            }
#pragma unroll
            for (int i = 0; i < kSteps; ++i)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float v = o[i][2 * e + c];
                    if constexpr (R == 4) v += __shfl_xor_sync(0xffffffffu, v, 2);
                    if (mine) out_s[(warp * R + r) * kLd + (e * kSteps + i) * 8 + g] = v;
                }
        }
        __syncthreads();
        for (int i = tid; i < R * HD; i += kKdThreads) {   // warps in order
            const int r = i / HD, c = i - r * HD;
            float M = -INFINITY, L = 0.0f, acc = 0.0f;
#pragma unroll
            for (int w = 0; w < kKdWarps; ++w) M = fmaxf(M, m_s[w][r]);
#pragma unroll
            for (int w = 0; w < kKdWarps; ++w) {
                const float m = m_s[w][r], f = m == -INFINITY ? (l_s[w][r] == 0.0f ? 0.0f : 1.0f) : exp2f(m - M);
                L = fmaf(l_s[w][r], f, L);
                acc = fmaf(out_s[(w * R + r) * kLd + c], f, acc);
            }
            part[(size_t)r * (HD + 2) + 2 + c] = acc * inv_kv[1] * (1.0f / 16384.0f);
            if (c == 0) {
                part[(size_t)r * (HD + 2)] = M;
                part[(size_t)r * (HD + 2) + 1] = L;
            }
        }
        for (int i = tid; i < (n_run - 1) * R; i += kKdThreads) {   // the run's other chunks are in the first one's sums
            part[(size_t)(R + i) * (HD + 2)] = -INFINITY;
            part[(size_t)(R + i) * (HD + 2) + 1] = -1.0f;   // no sum: a run's own is never negative
        }

        // the CTA that arrives last merges the runs in order; the counter returns to zero
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            int* cnt = P.split_done + (size_t)z * P.Hkv + h;
            s_last = atomicAdd(cnt, n_run) == nz - n_run;
            if (s_last) *cnt = 0;
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            float* wgt = out_s;   // [R][nz] weights of the runs, packed
            int* slot = reinterpret_cast<int*>(m_s);   // their first chunks
            const float* base = P.partials + (((size_t)z * P.Hkv + h) * P.n_chunks) * R * (HD + 2);
            if (warp < R) {
                float M = -INFINITY, L = 0.0f;
                for (int c = lane; c < nz; c += 32) M = fmaxf(M, __ldcg(base + ((size_t)c * R + warp) * (HD + 2)));
#pragma unroll
                for (int off = 16; off >= 1; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
                int n = 0;   // chunks that are in another chunk's sums are left out, for every head the same
                for (int c0 = 0; c0 < nz; c0 += 32) {
                    const int c = c0 + lane;
                    const float* p = base + ((size_t)c * R + warp) * (HD + 2);
                    const float m = c < nz ? __ldcg(p) : -INFINITY, l = c < nz ? __ldcg(p + 1) : -1.0f;
                    const bool own = l != -1.0f;   // NaN is unequal
                    const unsigned run = __ballot_sync(0xffffffffu, own);
                    // a run of NaN weights has a maximum of -inf and keeps its NaN
                    const float f = m == -INFINITY ? (l == 0.0f ? 0.0f : 1.0f) : exp2f(m - M);
                    if (own) {
                        const int at = n + __popc(run & ((1u << lane) - 1u));
                        wgt[warp * nz + at] = f;
                        if (warp == 0) slot[at] = c;
                        L = fmaf(l, f, L);
                    }
                    n += __popc(run);
                }
#pragma unroll
                for (int off = 16; off >= 1; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
                if (lane == 0) {
                    l_s[0][warp] = L;
                    if (warp == 0) s_at[0] = n;
                }
            }
            __syncthreads();
            const int n = s_at[0];
            for (int i = tid; i < R * HD; i += kKdThreads) {
                const int r = i / HD, c = i - r * HD;
                float acc = 0.0f;
#pragma unroll 8
                for (int k = 0; k < n; ++k) {
                    const float v = __ldcg(base + ((size_t)slot[k] * R + r) * (HD + 2) + 2 + c), f = wgt[r * nz + k];
                    acc = f != 0.0f ? fmaf(v, f, acc) : acc;
                }
                const float L = l_s[0][r];
                acc *= L == 0.0f ? 0.0f : 1.0f / L;
                const size_t oi = ((size_t)z * row_heads + P.out_head0 + (size_t)h * R + r) * HD + c;
                if (P.io_dtype == OJX_BF16) peer_store(link, reinterpret_cast<__nv_bfloat16*>(P.out) + oi, __float2bfloat16_rn(acc));
                else peer_store(link, reinterpret_cast<float*>(P.out) + oi, acc);
            }
        }
        __syncthreads();   // the run's shared memory has been read
        left -= n_run;
        split += n_run;
    }
    for (int i = blockIdx.x; i < Z * P.Hkv; i += gridDim.x)   // sequences without tokens
        if (length(i / P.Hkv) <= 0)
            for (int c = tid; c < R * HD; c += kKdThreads) {
                const size_t oi = ((size_t)(i / P.Hkv) * row_heads + P.out_head0 + (size_t)(i % P.Hkv) * R) * HD + c;
                if (P.io_dtype == OJX_BF16) peer_store(link, reinterpret_cast<__nv_bfloat16*>(P.out) + oi, __float2bfloat16_rn(0.0f));
                else peer_store(link, reinterpret_cast<float*>(P.out) + oi, 0.0f);
            }
    peer_signal_when_last(link, gridDim.x);
}

bool kvq_decode_mma_supported(const KvqProblem& P) {
    const int R = P.Hq / P.Hkv;
    return P.io_dtype == OJX_BF16 && P.even_books && P.D == 8 && (P.G == 8 || P.G == 16) && P.head_dim == P.G * 8 && (R == 4 || R == 8);
}

template <int R, int G>
static int launch_kd(const KvqProblem& P, cudaStream_t s, const PeerLink& link) {
    constexpr int smem = 2 * kGmTable + (int)sizeof(float) * kKdWarps * R * (G * 8 + 4);   // tables, the warps' outputs
    static_assert(kKdWarps * (G * 8 + 4) >= kKvMaxSplits && kKdWarps * 16 >= kKvMaxSplits, "the merge's weights and chunks fit");
    static std::atomic<bool> configured[64];   // the kernel's opt-in, once per device
    int dev = 0;
    OJX_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
        OJX_CUDA_TRY(cudaFuncSetAttribute(kvq_decode_mma_kernel<R, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    const long long items = (long long)P.n_chunks * P.Hkv * (P.n_pos > 0 ? P.n_pos * P.B : P.B);
    cfg.gridDim = dim3((unsigned)std::min<long long>(items, num_sms()));
    cfg.blockDim = dim3(kKdThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // the tables are built while an append still runs
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    OJX_CUDA_TRY(cudaLaunchKernelEx(&cfg, kvq_decode_mma_kernel<R, G>, P, link));
    count_launch(1);
    return OJX_OK;
}

int launch_kvq_decode_mma(const KvqProblem& P, cudaStream_t s, const PeerLink& link) {
    switch (P.Hq / P.Hkv * 100 + P.G) {
        case 408: return launch_kd<4, 8>(P, s, link);
        case 416: return launch_kd<4, 16>(P, s, link);
        case 808: return launch_kd<8, 8>(P, s, link);
        case 816: return launch_kd<8, 16>(P, s, link);
        default: return OJX_ERR_UNSUPPORTED;
    }
}

}  // namespace ojx
