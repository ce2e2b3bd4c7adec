// Products of a VQ-coded weight tile with a few activation vectors on the tensor cores, at 22 bits and fp32 sums.
//
// The 8-dimensional centroids are the rows that ldmatrix reads: an 8x8 matrix of fp16 is eight 16-byte rows at
// any eight addresses, so the lanes hand it the addresses of the centroids that the code bytes name and the A
// operand of mma.sync m16n8k16 (16 weight rows x two groups) comes out of the codebook table without ever being
// written to a tile.  A row keeps its place in the fragment, hence its lane its copy: copy q of the table lies in
// 16-byte bank group q and the eight rows of a matrix read eight different copies, four wavefronts for 32 codes
// whatever the codes are.
//
// 22 bits from fp16 operands: the codebook is scaled by a power of two (largest element in [2^14, 2^15)) and
// split into x = hi + lo, 22 bits of mantissa; activations are scaled the same way per vector and 256 dimensions.
// A bf16 activation is then one exact fp16 number (elements 2^29 below the largest of their 256 lose bits), and
// hi * x + lo * x is accumulated in fp32.
//
// Layout of prepared activations ("fragments"), per chunk of 256 dimensions = 32 groups: step i of 16 multiplies
// groups i (k = 0..7) and 16 + i (k = 8..15); a lane with k pair tq of vector t reads for the steps 2j and 2j + 1
// the 16 bytes at ((chunk * 8 + j) * vectors + t) * 4 + tq: {b0, b1} of the first, {b0, b1} of the second step.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace ojx {

constexpr int kGmChunk = 32;                    // groups of a chunk
constexpr int kGmTable = 2 * 256 * 8 * 16;      // bytes: hi, then lo; [256 codes][8 copies][16 bytes] each

__device__ __forceinline__ void gm_ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void gm_ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void gm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Power of two (and its inverse) that brings a largest magnitude, given as float bits, into [2^14, 2^15); tiny
// magnitudes stop at 2^126; 1 for zero, infinity and NaN.
__device__ __forceinline__ void gm_scale(uint32_t abs_bits, float& scale, float& inv) {
    const int e = (int)(abs_bits >> 23);
    const int s = abs_bits == 0u || e == 255 ? 0 : min(141 - e, 126);
    scale = __uint_as_float((uint32_t)(127 + s) << 23);
    inv = __uint_as_float((uint32_t)(127 - s) << 23);
}

__device__ __forceinline__ uint32_t gm_pack(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The codebook (f32 [Kcb][8]) as the two tables at `table`; all threads of the CTA call it, each with its number c among
// the threads of this table (at least 256; `red` holds one word per warp of them).  Codes from Kcb on are zero rows.
// Returns the inverse of the scale; ends with a barrier.
__device__ __forceinline__ float gm_build_table(unsigned char* table, uint32_t* red, const float* cb, int Kcb, int c) {
    const int lane = c & 31;
    float v[8];
    uint32_t m = 0u;
#pragma unroll
    for (int d = 0; d < 8; ++d) v[d] = 0.0f;
    if (c < Kcb) {
        const float4 a = reinterpret_cast<const float4*>(cb)[2 * c], b = reinterpret_cast<const float4*>(cb)[2 * c + 1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
#pragma unroll
        for (int d = 0; d < 8; ++d) m = max(m, __float_as_uint(v[d]) & 0x7fffffffu);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) red[c >> 5] = m;
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) m = max(m, red[w]);
    float scale, inv;
    gm_scale(m, scale, inv);
    if (c < 256) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const float a = v[2 * p] * scale, b = v[2 * p + 1] * scale;
            const __half2 h = __floats2half2_rn(a, b);
            hi[p] = *reinterpret_cast<const uint32_t*>(&h);
            lo[p] = gm_pack(a - __low2float(h), b - __high2float(h));
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {   // the eight lanes of a wavefront write eight different bank groups
            unsigned char* at = table + c * 128 + ((q + lane) & 7) * 16;
            *reinterpret_cast<uint4*>(at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(at + kGmTable / 2) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
    __syncthreads();
    return inv;
}

// The 16 code bytes of a lane's half of a chunk (groups 32 chunk + 16 half ...) of one weight row of G codes; bytes
// past the row's end repeat codes of the row (their activations are zero).  G is a multiple of 8, of 16 if `wide`.
__device__ __forceinline__ void gm_load_codes(uint32_t (&w)[4], const uint8_t* row, int chunk, int half, int G, bool wide) {
    int off = chunk * kGmChunk + half * 16;
    if (off >= G) off = chunk * kGmChunk;
    if (wide) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(row + off));
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else {
        const uint2 a = __ldg(reinterpret_cast<const uint2*>(row + off));
        const uint2 b = __ldg(reinterpret_cast<const uint2*>(row + (off + 8 < G ? off + 8 : off)));
        w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
    }
}

// acc += (weights of MT x 16 rows, one chunk) x (NT x 8 vectors).  w: the lane's codes (row lane & 15 of each tile,
// half lane >> 4).  load(j, n): the lane's 16 bytes of fragments of tile n for steps 2j and 2j + 1.  table: shared address
// of the lane's copy ((lane & 7) * 16 from the table's start).
// kFlush: steps whose products are accumulated in the tensor cores before they are added to acc in fp32 (the tensor
// cores truncate, so a chain's error grows with its length); 16: all of them.
// The lanes meet first: ldmatrix and mma need all 32 of them converged, and callers come from loops of per-lane length.
template <int MT, int NT, int kFlush, class Load>
__device__ __forceinline__ void gm_chunk(float (&acc)[MT][NT][4], const uint32_t (&w)[MT][4], int steps, uint32_t table, Load load) {
    __syncwarp();
    uint4 b[NT], bn[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) bn[n] = load(0, n);
    // step i of tile m: its two table reads are issued before the products of the (step, tile) ahead of it
    auto read = [&](int i, int m, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
        const uint32_t word = w[m][i >> 2];
        const int q = i & 3;
        const uint32_t at = table + ((q == 0 ? word << 7 : word >> (8 * q - 7)) & 0x7f80);   // code * 128
        gm_ldsm4(at, hi);
        gm_ldsm4(at + kGmTable / 2, lo);
    };
    uint32_t hi[2][4], lo[2][4];
    float part[MT][NT][4];
    read(0, 0, hi[0], lo[0]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (2 * j < steps) {
#pragma unroll
            for (int n = 0; n < NT; ++n) b[n] = bn[n];
            if (2 * j + 2 < steps) {
#pragma unroll
                for (int n = 0; n < NT; ++n) bn[n] = load(j + 1, n);
            }
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int at = (2 * j + s) * MT + m, cur = at & 1, next = at + 1;
                    if (next < 16 * MT) read(next / MT, next % MT, hi[cur ^ 1], lo[cur ^ 1]);
                    if (kFlush < 16 && (2 * j + s) % kFlush == 0) {
#pragma unroll
                        for (int n = 0; n < NT; ++n)
#pragma unroll
                            for (int e = 0; e < 4; ++e) part[m][n][e] = 0.0f;
                    }
                    auto& sum = kFlush < 16 ? part : acc;
#pragma unroll
                    for (int n = 0; n < NT; ++n) gm_mma(sum[m][n], lo[cur], s ? b[n].z : b[n].x, s ? b[n].w : b[n].y);
#pragma unroll
                    for (int n = 0; n < NT; ++n) gm_mma(sum[m][n], hi[cur], s ? b[n].z : b[n].x, s ? b[n].w : b[n].y);
                    if (kFlush < 16 && (2 * j + s) % kFlush == kFlush - 1) {
#pragma unroll
                        for (int n = 0; n < NT; ++n)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[m][n][e] += part[m][n][e];
                    }
                }
        }
    }
}

}  // namespace ojx
