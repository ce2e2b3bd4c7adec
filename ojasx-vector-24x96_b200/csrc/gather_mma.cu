// VQ linears on bf16 activations for batches below the tcgen05 path's: one prepared copy of the activations, then
// weight tiles gathered from the codebook straight into mma.sync operands (gather_mma.cuh).  The result is the table
// kernels': the reference's fp32 row sum, rounded once to bf16.  A sum formed in another order differs from the
// reference's by a few 1e-7 and rounds the same unless it lies next to a rounding boundary; those (one in a hundred) are
// listed and evaluated again in the reference's order.  What counts as next to it is kGmTolerance's comment.
//
// The table kernels spend one shared-memory gather and one addition per code and vector.  Here a code costs 32 bytes of
// shared-memory reads whatever the batch.  SwiGLU block of widths 2560 and 6912, us, table kernels and these: batch 1
// 55 / 39, 16 138 / 58.  What is left is latency: launches, building the table, the outliers' gathers and the ordered sums;
// clocks of a CTA at 2560 to 6912 columns and batch 16, with a window that 0.5 % of the sums fell into: 4.4 k before the
// activations are there, 8.2 k for the products (a third of the shared-memory rate), 6.2 k for partial sums and outliers,
// 6.0 k for the sums evaluated again.
#include <algorithm>
#include <atomic>

#include "gather_mma.cuh"
#include "handles.h"
#include "launch.h"
#include "silu.cuh"

namespace ojx {

constexpr int kGmMaxBatch = 32;
constexpr int kGmMaxWarps = 10;     // 320 threads, two CTAs per SM
constexpr int kGmProblems = 2;
// A sum is evaluated again in the reference's order if a bf16 rounding boundary lies within a window around it.  What the two
// may differ by, with v the sum, A the sum of the magnitudes of its pieces (chunks, or what a warp or a CTA of a cluster adds
// up), eps = 2^-24 and G ordered additions:
//   eps G / 2 |v|            sums of one sign (A = |v|): partial sums grow to |v|; fades out as A grows to 2 |v|
//   eps 0.5 sqrt(G) A        sums that cancel: partial sums up to (A + |v|) / 2, independent roundings, four deviations
//   eps (16 |v| + 4 A)       truncation in the tensor cores, 32 products of a chunk: a common shrinking, and what chunks differ by
//   kGmTolerance             operands of 22 bits and roundings inside a chunk: times (codebook maximum) * sqrt(sum over chunks
//                            of squared activation maxima), maxima being powers of two scaled by 2^-14 each
// Not a bound for every input (that takes eps G A, and more than twice as many sums); measured: none of 48 million outputs of
// Gaussian, one-signed, constant, cancelling, tiny, large, spiked and ramped activations at widths 64 to 6912 differs.  With a
// window for Gaussian data alone (1536 and 2 eps |v|) 1 in 10 000 of one-signed and 1 in 400 of cancelling sums did; it
// took 50 us where this takes 58 (SwiGLU block of 2560 and 6912, 16 vectors).
constexpr float kGmTolerance = 1024.0f;
constexpr int kGmEntries = 768;     // outliers of a tile brought in before the activations are ready

struct GmArgs {
    LinearProblem P[kGmProblems];
    int tiles0;                     // row tiles of problem 0
    const uint4* frag;
    const float* inv;               // [chunks][bp] inverse scale: 0 where a vector's chunk is all zeros, NaN where it has an infinity or NaN
    const __nv_bfloat16* xT;        // [chunks * 256][bp]
    int chunks, per_split;
};

// ------------------------------------------------------------------------------------ activations
// grid = chunks; a warp prepares vectors warp, warp + 8, ...  With `up`, the vectors are silu(x) * up rounded to bf16
// (as silu_mul_kernel rounds them) and are also written to `h`.
__global__ void __launch_bounds__(256) gm_prep_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ up,
                                                      __nv_bfloat16* __restrict__ h, int K, int batch, int bp, uint4* __restrict__ frag,
                                                      float* __restrict__ inv_out, __nv_bfloat16* __restrict__ xT) {
    __shared__ __align__(16) __nv_bfloat16 tile[kGmMaxBatch][256 + 8];
    cudaTriggerProgrammaticLaunchCompletion();   // the linear behind this launch builds its tables, which nothing in the stream writes
    cudaGridDependencySynchronize();
    const int c = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k0 = c * 256 + lane * 8;
    for (int t = warp; t < bp; t += 8) {
        uint32_t v[4] = {0u, 0u, 0u, 0u};
        if (t < batch && k0 < K) {
            const uint4 a = *reinterpret_cast<const uint4*>(x + (size_t)t * K + k0);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            if (up) {
                const uint4 u4 = *reinterpret_cast<const uint4*>(up + (size_t)t * K + k0);
                const uint32_t u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float2 g2 = make_float2(__uint_as_float(v[p] << 16), __uint_as_float(v[p] & 0xffff0000u));
                    const float2 u2 = make_float2(__uint_as_float(u[p] << 16), __uint_as_float(u[p] & 0xffff0000u));
                    const __nv_bfloat162 r = __halves2bfloat162(__float2bfloat16_rn(__fmul_rn(silu_ref(g2.x), u2.x)),
                                                                __float2bfloat16_rn(__fmul_rn(silu_ref(g2.y), u2.y)));
                    v[p] = *reinterpret_cast<const uint32_t*>(&r);
                }
                *reinterpret_cast<uint4*>(h + (size_t)t * K + k0) = make_uint4(v[0], v[1], v[2], v[3]);
            }
        }
        uint32_t m = 0u;
#pragma unroll
        for (int p = 0; p < 4; ++p) m = max(m, max((v[p] << 16) & 0x7fffffffu, v[p] & 0x7fff0000u));
        m = __reduce_max_sync(0xffffffffu, m);
        float scale, inv;
        gm_scale(m, scale, inv);
        // 0 for zeros: the chunk adds nothing to a sum, so nothing to the bound on its error either (with gm_scale's 1 a padded
        // vector's sums were all evaluated again: 154 us against 35 with 8 zero vectors of 16, 2560 to 6912 columns)
        if (lane == 0) inv_out[c * bp + t] = m == 0u ? 0.0f : m >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : inv;
        *reinterpret_cast<uint4*>(&tile[t][lane * 8]) = make_uint4(v[0], v[1], v[2], v[3]);
        // lane = group of the chunk: step lane & 15, half lane >> 4
        uint32_t* at = reinterpret_cast<uint32_t*>(frag + ((size_t)(c * 8 + ((lane & 15) >> 1)) * bp + t) * 4) + (lane & 1) * 2 + (lane >> 4);
#pragma unroll
        for (int p = 0; p < 4; ++p)
            at[p * 4] = gm_pack(__uint_as_float(v[p] << 16) * scale, __uint_as_float(v[p] & 0xffff0000u) * scale);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 256 * bp / 4; i += 256) {   // four vectors of one dimension per thread
        const int k = i / (bp / 4), t = (i - k * (bp / 4)) * 4;
        __nv_bfloat16 q[4] = {tile[t][k], tile[t + 1][k], tile[t + 2][k], tile[t + 3][k]};
        *reinterpret_cast<uint2*>(xT + ((size_t)c * 256 + k) * bp + t) = *reinterpret_cast<const uint2*>(q);
    }
}

// ----------------------------------------------------------------------------------------- linear
// Table entry <x_g, codebook[c]> in the reference's order (ojasx_lut_cpu.cpp:93-100); codes from Kcb on are zero rows.
__device__ __forceinline__ float gm_entry(const uint4& x, const float* cb, int c, int Kcb) {
    if (c >= Kcb) return 0.0f;
    const float4 c0 = __ldg(reinterpret_cast<const float4*>(cb) + 2 * c), c1 = __ldg(reinterpret_cast<const float4*>(cb) + 2 * c + 1);
    float dot = __fmul_rn(__uint_as_float(x.x << 16), c0.x);
    dot = __fadd_rn(dot, __fmul_rn(__uint_as_float(x.x & 0xffff0000u), c0.y));
    dot = __fadd_rn(dot, __fmul_rn(__uint_as_float(x.y << 16), c0.z));
    dot = __fadd_rn(dot, __fmul_rn(__uint_as_float(x.y & 0xffff0000u), c0.w));
    dot = __fadd_rn(dot, __fmul_rn(__uint_as_float(x.z << 16), c1.x));
    dot = __fadd_rn(dot, __fmul_rn(__uint_as_float(x.z & 0xffff0000u), c1.y));
    dot = __fadd_rn(dot, __fmul_rn(__uint_as_float(x.w << 16), c1.z));
    return __fadd_rn(dot, __fmul_rn(__uint_as_float(x.w & 0xffff0000u), c1.w));
}

// grid (row tiles of all problems, splits), cluster (1, splits).  A CTA owns MT x 16 rows and its split's chunks of 256
// dimensions; every warp takes a run of them for all rows, so fragments go from L2 to registers and every warp reads whole
// sectors of the code rows (a run and not every warps-th chunk: the magnitude of a run's sum then tells how far the ordered
// partial sums go up, also where the first and the second half of a row cancel).  Partial sums of the warps, then of the cluster's CTAs, are added
// in chunk order in shared memory.  The table is built while the activations are still being prepared.
template <int MT, int NT>
__global__ void __launch_bounds__(kGmMaxWarps * 32, 2) gm_linear_kernel(const __grid_constant__ GmArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kRows = MT * 16, kVecs = NT * 8, kLd = kVecs + 1;
    float* part = reinterpret_cast<float*>(smem_raw + kGmTable);           // [warps][kRows][kLd]
    __shared__ uint32_t scale_red[kGmMaxWarps];
    __shared__ float tol_s[kVecs];
    __shared__ int n_fix, rp_s[kRows + 1];
    const int warps = blockDim.x >> 5, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pi = (int)blockIdx.x >= A.tiles0 ? 1 : 0;
    const LinearProblem& P = A.P[pi];
    const int row0 = P.row_start + ((int)blockIdx.x - (pi ? A.tiles0 : 0)) * kRows;
    const int split = blockIdx.y, splits = gridDim.y;
    const int c_begin = split * A.per_split, c_end = min(A.chunks, c_begin + A.per_split);
    const bool wide = (P.G & 15) == 0 && (reinterpret_cast<uintptr_t>(P.codes) & 15) == 0;

    const uint8_t* rows[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) rows[m] = P.codes + (size_t)min(row0 + m * 16 + (lane & 15), P.row_stop - 1) * P.G;
    uint32_t w[MT][4], wn[MT][4];
    const int run = (c_end - c_begin + warps - 1) / warps, c_first = c_begin + warp * run, c_last = min(c_end, c_first + run);
    if (c_first < c_last) {
#pragma unroll
        for (int m = 0; m < MT; ++m) gm_load_codes(wn[m], rows[m], c_first, lane >> 4, P.G, wide);
    }
    constexpr int kItems = kRows * NT * 2;     // four vectors of one row each
    // the rows this CTA finishes: all of its tile, or its share of the cluster's
    const int r_begin = min(kRows * split / splits, P.row_stop - row0), r_end = min(kRows * (split + 1) / splits, P.row_stop - row0);
    if (P.csr.nnz > 0)
        for (int i = tid; i <= kRows; i += blockDim.x) rp_s[i] = P.csr.row_ptrs[min(row0 + i, P.row_stop)];
    int2* ent = reinterpret_cast<int2*>(part + (size_t)warps * kRows * kLd);   // (column, value) of the tile's first kGmEntries outliers
    int jb = 0, je = 0;
    if (P.csr.nnz > 0 && r_end > r_begin) {
        jb = P.csr.row_ptrs[row0 + r_begin];
        je = P.csr.row_ptrs[row0 + r_end];
        for (int j = tid; j < min(je - jb, kGmEntries); j += blockDim.x)
            ent[j] = make_int2(P.csr.cols[jb + j], __float_as_int(P.csr.vals[jb + j]));
    }
    const float inv_cb = gm_build_table(smem_raw, scale_red, P.codebook, P.Kcb, tid);
    const uint32_t table = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw)) + (lane & 7) * 16;
    int boff[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) boff[n] = (n * 8 + (lane >> 2)) * 4 + (lane & 3);

    // (no trigger here: the next preparation's linear would take shared memory and issue slots from this one, SwiGLU block of 16
    // tokens 53 us without and 62 with)
    cudaGridDependencySynchronize();   // the prepared activations

    if (tid < kVecs) {
        float top = 0.0f, m = 0.0f;   // relative to the largest: squares of tiny or huge scales leave the range of fp32
        for (int c = 0; c < A.chunks; ++c) top = fmaxf(top, A.inv[c * kVecs + tid]);
        const float r = top > 0.0f ? 1.0f / top : 0.0f;
        for (int c = 0; c < A.chunks; ++c) m = fmaf(A.inv[c * kVecs + tid] * r, A.inv[c * kVecs + tid] * r, m);
        const float tol = top * inv_cb * sqrtf(m) * kGmTolerance + (float)P.K * 1.4e-45f;   // products may be subnormal
        tol_s[tid] = tol < 1e28f ? tol : __uint_as_float(0x7fc00000u);                        // ordered partial sums may overflow
        if (tid == 0) n_fix = 0;
    }
    float* mine = part + (size_t)warp * kRows * kLd;
    for (int c = c_first; c < c_last; ++c) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) w[m][i] = wn[m][i];
        if (c + 1 < c_last) {
#pragma unroll
            for (int m = 0; m < MT; ++m) gm_load_codes(wn[m], rows[m], c + 1, lane >> 4, P.G, wide);
        }
        float2 iv[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) iv[n] = *reinterpret_cast<const float2*>(A.inv + c * kVecs + n * 8 + (lane & 3) * 2);
        float acc[MT][NT][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.0f;
        const uint4* frag = A.frag + (size_t)c * 8 * kVecs * 4;
        gm_chunk<MT, NT, 16>(acc, w, min(16, P.G - c * kGmChunk), table, [&](int j, int n) { return __ldg(frag + (size_t)j * kVecs * 4 + boff[n]); });
        const bool first = c == c_first;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float* p = mine + (m * 16 + (lane >> 2) + (i >> 1) * 8) * kLd + n * 8 + (lane & 3) * 2 + (i & 1);
                    const float v = acc[m][n][i] * inv_cb * ((i & 1) ? iv[n].y : iv[n].x);
                    *p = first ? v : *p + v;
                }
        }
    }
    __syncthreads();

    const int live = (c_end - c_begin + run - 1) / run;   // warps that had a run
    const unsigned part_addr = static_cast<unsigned>(__cvta_generic_to_shared(part));
    if (splits > 1) {   // the CTA's sum replaces its first warp's part, the cluster's CTAs read one another's
        for (int i = tid; i < kItems * 4; i += blockDim.x) {
            const int at = (i % kRows) * kLd + i / kRows;
            float s = part[at], a = fabsf(s);
            for (int v = 1; v < live; ++v) {
                const float f = part[(size_t)v * kRows * kLd + at];
                s += f;
                a += fabsf(f);
            }
            part[at] = s;
            part[kRows * kLd + at] = a;   // magnitudes, in the second warp's place (there are at least eight)
        }
        __syncwarp();   // the barrier is an aligned one
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    // Sums too close to a rounding boundary of bf16 to decide: listed in the dead table, evaluated in order below.
    uint2* list = reinterpret_cast<uint2*>(smem_raw);                              // [kItems * 4] (row << 8 | vector, outlier sum)
    float* fix_buf = reinterpret_cast<float*>(smem_raw + kItems * 4 * sizeof(uint2));   // [sums][G + 4] table entries
    const int rows_out = P.row_stop - P.row_start;
    auto affine = [&](float v, int m) {
        if (P.scales) v = __fmul_rn(v, P.scales[m]);
        return P.bias ? __fadd_rn(v, P.bias[m]) : v;
    };
    const float one_sign = ((float)P.G + 64.0f) * 0x1p-25f, cancel = (0.5f * sqrtf((float)P.G) + 4.0f) * 0x1p-24f;
    // Outliers: the tile's entries are contiguous, so all threads multiply (entry, four vectors) pieces into the dead
    // table, then a thread per (row, four vectors) adds its row's products in entry order.
    float4* prod = reinterpret_cast<float4*>(smem_raw);                            // [entries of a pass][NT * 2]
    constexpr int kQuads = NT * 2, kPass = (kGmTable / 16) / kQuads, kPer = (kItems + 255) / 256;
    float o[kPer][4];
#pragma unroll
    for (int i = 0; i < kPer; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    if (P.csr.nnz > 0 && r_end > r_begin) {
        for (int j0 = jb; j0 < je; j0 += kPass) {
            const int jn = min(je, j0 + kPass);
            constexpr int U = 8;
            for (int i0 = tid; i0 < (jn - j0) * kQuads; i0 += U * blockDim.x) {
                float val[U];
                uint2 xv[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * blockDim.x;
                    xv[u] = make_uint2(0u, 0u);
                    if (i < (jn - j0) * kQuads) {
                        const int j = j0 + i / kQuads, at = j - jb;
                        const int2 e = at < kGmEntries ? ent[at] : make_int2(P.csr.cols[j], __float_as_int(P.csr.vals[j]));
                        const int col = e.x;
                        val[u] = __int_as_float(e.y);
                        if ((unsigned)col < (unsigned)P.K) xv[u] = *reinterpret_cast<const uint2*>(A.xT + (size_t)col * kVecs + (i % kQuads) * 4);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * blockDim.x;
                    if (i < (jn - j0) * kQuads)
                        prod[i] = make_float4(__fmul_rn(val[u], __uint_as_float(xv[u].x << 16)), __fmul_rn(val[u], __uint_as_float(xv[u].x & 0xffff0000u)),
                                              __fmul_rn(val[u], __uint_as_float(xv[u].y << 16)), __fmul_rn(val[u], __uint_as_float(xv[u].y & 0xffff0000u)));
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kPer; ++i) {
                const int item = tid + i * blockDim.x, r = item % kRows;
                if (item < kItems && r >= r_begin && r < r_end)
                    for (int j = max(rp_s[r], j0); j < min(rp_s[r + 1], jn); ++j) {
                        const float4 f = prod[(j - j0) * kQuads + item / kRows];
                        o[i][0] = __fadd_rn(o[i][0], f.x);
                        o[i][1] = __fadd_rn(o[i][1], f.y);
                        o[i][2] = __fadd_rn(o[i][2], f.z);
                        o[i][3] = __fadd_rn(o[i][3], f.w);
                    }
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int item = tid + i * blockDim.x, r = item % kRows, t0 = item / kRows * 4, m = row0 + r;
        if (item >= kItems || r < r_begin || r >= r_end) continue;
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f}, mag[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (splits > 1) {
            for (int v = 0; v < splits; ++v) {
                unsigned base;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base) : "r"(part_addr + (unsigned)(r * kLd + t0) * 4), "r"(v));
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float f;
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(base + q * 4) : "memory");
                    s[q] += f;
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(base + (kRows * kLd + q) * 4) : "memory");
                    mag[q] += f;
                }
            }
        } else {
            for (int v = 0; v < live; ++v)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float f = part[(size_t)v * kRows * kLd + r * kLd + t0 + q];
                    s[q] += f;
                    mag[q] += fabsf(f);
                }
        }
        const float scale = P.scales ? fabsf(P.scales[m]) : 1.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int t = t0 + q;
            if (t >= P.batch) break;
            const float sa = fabsf(s[q]), w = affine(s[q], m), v = P.csr.nnz > 0 ? __fadd_rn(w, o[i][q]) : w;
            const float tol = scale * (tol_s[t] + one_sign * fmaxf(2.0f * sa - mag[q], 0.0f) + 0x1p-20f * sa + cancel * mag[q]) + 1.8e-7f * (fabsf(w) + fabsf(v));
            const __nv_bfloat16 a = __float2bfloat16_rn(v - tol), b = __float2bfloat16_rn(v + tol);
            if (a == b) reinterpret_cast<__nv_bfloat16*>(P.y)[(size_t)t * rows_out + (m - P.row_start)] = a;
            else list[atomicAdd(&n_fix, 1)] = make_uint2(r << 8 | t, __float_as_uint(o[i][q]));   // NaN is unequal to itself
        }
    }
    __syncthreads();
    // All threads form the table entries of the listed sums, then a thread per sum adds its G entries in order.
    const int ld = P.G + 4, cap = (kGmTable - kItems * 4 * (int)sizeof(uint2)) / (ld * (int)sizeof(float));
    for (int i0 = 0; i0 < n_fix; i0 += cap) {
        const int n = min(cap, n_fix - i0), total = n * P.G;
        constexpr int U = 8;
        for (int i = tid; i < total; i += U * blockDim.x) {
            int code[U], at[U];
            uint4 xv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = i + u * blockDim.x;
                at[u] = -1;
                if (j < total) {
                    const int e = j / P.G, g = j - e * P.G;
                    const uint2 l = list[i0 + e];
                    at[u] = e * ld + g;
                    code[u] = P.codes[(size_t)(row0 + (int)(l.x >> 8)) * P.G + g];
                    xv[u] = *(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(P.x) + (size_t)(l.x & 255) * P.K) + g);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (at[u] >= 0) fix_buf[at[u]] = gm_entry(xv[u], P.codebook, code[u], P.Kcb);
        }
        __syncthreads();
        for (int e = tid; e < n; e += blockDim.x) {   // narrow layers: a pass holds more sums than the CTA has threads
            const uint2 l = list[i0 + e];
            const float4* v = reinterpret_cast<const float4*>(fix_buf + e * ld);
            float acc = 0.0f;
#pragma unroll 4
            for (int i = 0; i < P.G / 4; ++i) {   // G is a multiple of 8
                const float4 f = v[i];
                acc = __fadd_rn(acc, f.x);
                acc = __fadd_rn(acc, f.y);
                acc = __fadd_rn(acc, f.z);
                acc = __fadd_rn(acc, f.w);
            }
            const int m = row0 + (int)(l.x >> 8), t = l.x & 255;
            acc = affine(acc, m);
            if (P.csr.nnz > 0) acc = __fadd_rn(acc, __uint_as_float(l.y));
            reinterpret_cast<__nv_bfloat16*>(P.y)[(size_t)t * rows_out + (m - P.row_start)] = __float2bfloat16_rn(acc);
        }
        __syncthreads();
    }
    __syncwarp();
    if (splits > 1)   // nobody leaves while its sums may still be read
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ------------------------------------------------------------------------------------- host side
static size_t gm_smem(int MT, int NT, int warps) {
    return kGmTable + sizeof(float) * ((size_t)warps * MT * 16 * (NT * 8 + 1)) + kGmEntries * sizeof(int2);
}

template <int MT, int NT>
static int gm_launch_t(const GmArgs& A, int tiles, int splits, int warps, cudaStream_t s) {
    const size_t smem = gm_smem(MT, NT, warps);
    static std::atomic<bool> configured[64];   // the kernel's opt-in, once per device
    int dev = 0;
    OJX_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
        OJX_CUDA_TRY(cudaFuncSetAttribute(gm_linear_kernel<MT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gm_smem(MT, NT, kGmMaxWarps)));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, splits);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = splits;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    OJX_CUDA_TRY(cudaLaunchKernelEx(&cfg, gm_linear_kernel<MT, NT>, A));
    count_launch(1);
    return OJX_OK;
}

// Rows per CTA and K splits.  Times of a wave of resident CTAs in microseconds, fitted to a sweep of seven shapes and
// five batches: 12 of latencies (launch, table, outliers, ordered sums), then 1.5 + 1.5 per 16-row tile for every chunk
// that a warp takes in turn; a cluster's exchange weighs 2.5.  2560 to 6912 columns, batch 16: (32 rows, no split) 17.6,
// (48, 1) 19.8, (48, 2) 17.5, (16, 1) two waves 23.8; 6912 to 2560: (32, 3) 21.7, (16, 1) 25.2, (48, 2) 26.9.
static void gm_plan(const LinearProblem* P, int count, int chunks, int NT, int* MT, int* splits, int* warps) {
    double best = 1e30;
    for (int mt = 1; mt <= (NT <= 2 ? 3 : 2); ++mt)
        for (int sp = 1; sp <= std::min(4, chunks); ++sp) {
            const int per = (chunks + sp - 1) / sp;
            if ((sp - 1) * per >= chunks) continue;
            long tiles = 0;
            for (int p = 0; p < count; ++p) tiles += (P[p].row_stop - P[p].row_start + mt * 16 - 1) / (mt * 16);
            const int rounds = (per + kGmMaxWarps - 1) / kGmMaxWarps;
            const int w = std::max(8, (per + rounds - 1) / rounds);   // at least eight warps build the table
            const long slots = num_sms() * (2 * (gm_smem(mt, NT, w) + 2048) <= 228 * 1024 ? 2L : 1L);
            const long waves = (tiles * sp + slots - 1) / slots;
            const double cost = waves * (12.0 + rounds * (1.5 + 1.5 * mt)) + (sp > 1 ? 2.5 : 0.0);
            if (cost < best) {
                best = cost;
                *MT = mt;
                *splits = sp;
                *warps = w;
            }
        }
}

bool gather_mma_supported(const LinearProblem& P) {
    return P.io_dtype == OJX_BF16 && P.D == 8 && P.batch >= 1 && P.batch < kGmMaxBatch && P.G > 0 && P.G % 8 == 0 &&
           P.K == P.G * 8 && P.K <= 65536 && (reinterpret_cast<uintptr_t>(P.codes) & 7) == 0 && (reinterpret_cast<uintptr_t>(P.codebook) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(P.x) & 15) == 0 && !P.y_full;
}

// frag, inv, xT of one set of activations
size_t gather_mma_workspace(int K, int batch) {
    const size_t chunks = (K + 255) / 256, bp = round_up(batch, 8);
    return chunks * bp * (8 * 64 + 4 + 256 * 2);
}

static void gm_carve(GmArgs& A, void* ws, int K, int batch) {
    const size_t bp = round_up(batch, 8);
    A.chunks = (K + 255) / 256;
    char* p = static_cast<char*>(ws);
    A.frag = reinterpret_cast<const uint4*>(p);
    p += (size_t)A.chunks * bp * 8 * 64;
    A.xT = reinterpret_cast<const __nv_bfloat16*>(p);
    p += (size_t)A.chunks * bp * 512;
    A.inv = reinterpret_cast<const float*>(p);
}

// `count` problems on the same activations (all supported, same K and batch).  With `up`, the activations are
// silu(x) * up and `h` receives them.
int launch_gather_mma(const LinearProblem* P, int count, const void* x, const void* up, void* h, void* workspace, cudaStream_t s) {
    if (count < 1 || count > kGmProblems || !workspace || (reinterpret_cast<uintptr_t>(workspace) & 15)) return OJX_ERR_ARG;
    for (int p = 0; p < count; ++p)
        if (!gather_mma_supported(P[p]) || P[p].K != P[0].K || P[p].batch != P[0].batch || P[p].row_stop <= P[p].row_start) return OJX_ERR_UNSUPPORTED;
    GmArgs A{};
    for (int p = 0; p < count; ++p) A.P[p] = P[p];
    const int batch = P[0].batch, NT = (batch + 7) / 8;
    gm_carve(A, workspace, P[0].K, batch);
    OJX_CUDA_TRY(launch_chained(gm_prep_kernel, A.chunks, 256, 0, s, static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(up),
                                static_cast<__nv_bfloat16*>(h), P[0].K, batch, NT * 8, const_cast<uint4*>(A.frag), const_cast<float*>(A.inv),
                                const_cast<__nv_bfloat16*>(A.xT)));
    count_launch(1);
    int MT = 1, splits = 1, warps = kGmMaxWarps;
    gm_plan(P, count, A.chunks, NT, &MT, &splits, &warps);
    A.per_split = (A.chunks + splits - 1) / splits;
    A.tiles0 = (P[0].row_stop - P[0].row_start + MT * 16 - 1) / (MT * 16);
    const int tiles = A.tiles0 + (count > 1 ? (P[1].row_stop - P[1].row_start + MT * 16 - 1) / (MT * 16) : 0);
    switch (MT * 10 + NT) {
        case 11: return gm_launch_t<1, 1>(A, tiles, splits, warps, s);
        case 12: return gm_launch_t<1, 2>(A, tiles, splits, warps, s);
        case 13: return gm_launch_t<1, 3>(A, tiles, splits, warps, s);
        case 14: return gm_launch_t<1, 4>(A, tiles, splits, warps, s);
        case 21: return gm_launch_t<2, 1>(A, tiles, splits, warps, s);
        case 22: return gm_launch_t<2, 2>(A, tiles, splits, warps, s);
        case 23: return gm_launch_t<2, 3>(A, tiles, splits, warps, s);
        case 24: return gm_launch_t<2, 4>(A, tiles, splits, warps, s);
        case 31: return gm_launch_t<3, 1>(A, tiles, splits, warps, s);
        case 32: return gm_launch_t<3, 2>(A, tiles, splits, warps, s);
        default: return OJX_ERR_UNSUPPORTED;
    }
}

}  // namespace ojx
