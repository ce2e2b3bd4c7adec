// Row walk for four activation vectors at a time: table entries of the four vectors lie side by side, so one code byte
// fetches four fp32 entries with one 16-byte shared-memory read.  Sums keep the reference's order -- entries in ascending
// group order into one fp32 accumulator per (row, vector), table entries as sequential dot products with separate multiply
// and add (split_manifold_lut_experiment/native/src/ojasx_lut_cpu.cpp:93-100, :161-175) -- so results are bit-identical
// to the walks of one vector.
//
// A lane keeps a row; the lanes of a warp run behind one another by one unit of two groups, lane l by l mod 8 units.  The
// eight lanes of a shared-memory wavefront (16 bytes each) are then at eight different units of the table slice, and as
// unit u lies in bank quad u, no gather conflicts whatever the codes are.  A lane that has finished its row's slice goes on
// with the next block of rows, and after the last block with the next slice, in the following step: nothing fills or
// drains but the ends of a whole work item.
//
// A slice is 16 groups: 256 codes x 16 groups x 4 vectors = 64 KB, kept twice.  Warps 0..7 walk one slice (shared-memory
// pipe) while warps 8..11 build the next (fp32 pipe), handing the buffers over through mbarriers with bounded waits.
//
// Bound: the shared-memory pipe (over whole launches 60 % busy in a linear of 2560 to 4096 at batch 512, 53 % in both passes of a MoE
// layer; issue slots 50 to 57 %), the rest are the ends of the work items: first tables, outliers, results.  A step of a warp (32 rows x 2 groups x 4 vectors) is two gathers of 4 wavefronts each, a
// 2-byte code read and shares of parking and code copies, about 10 wavefronts for 256 entries; the walk with one vector needs
// 8.5 for 128, and fills and drains 31 steps per slice.  The build of a slice takes 16384 x 15 fp32 operations (1920 clocks),
// as packed pairs half as many issue slots: a product is fma(a, b, -0) with the -0 from a kernel argument -- the same bits as a
// multiplication, and ptxas cannot merge it with the addition that follows, as it does with a packed multiplication.
//
// Shared memory, by absolute shared-space address (the dynamic area must start at 1024; checked at run time):
//     1024  mbarriers and control words; 1104 set when a wait ran out; 1120 a sum of zero; 1152 a place for the sums of rows that do not exist
//     1664  activations of a slice, [2][8 units x 272 bytes]: element e of a unit at e*16, its four vectors side by side
//     6144  codebook f32[256][8], every number twice
//    22528  parked sums float4[2688]
//    65536  table 0: entry (code k, group j of unit u) at k*256 + j*128 + u*16; 131072 table 1
//   196608  code rings of the walkers, 4 KB each: eight chunks of 32 rows x 16 bytes
// Chunk m of a warp is (slice m / blocks, block m mod blocks).  Row l of a chunk lies at (l >> 3)*16 + (l & 1)*64 + ((l & 7) >> 1)*128,
// which puts the 32 words that the lanes read in a step into different banks.  Chunks p + 5 and p + 6 are asked for when chunk p begins, p even.
#pragma once
#include "lut_core.cuh"

namespace ojx {

constexpr int kQuWalkers = 8, kQuBuilders = 4, kQuSets = 1, kQuChunks = 8, kQuThreads = 32 * (kQuWalkers + kQuBuilders), kQuVecs = 4;
constexpr int kQuSlice = 16;                                   // groups
constexpr uint32_t kQuCtl = 1024, kQuGone = 1104, kQuZero = 1120, kQuDump = 1152, kQuXs = 1664, kQuBook = 6144, kQuAcc = 22528, kQuTab = 65536, kQuRing = 196608;
constexpr uint32_t kQuXsBytes = 2176, kQuTabBytes = 65536, kQuRingBytes = kQuChunks * 512;
constexpr int kQuRows = (int)(kQuTab - kQuAcc) / 16;           // rows of a work item
constexpr size_t kQuSmemBytes = kQuRing + kQuWalkers * kQuRingBytes - kQuCtl;
constexpr int kQuMaxK = (int)(2 * kQuTabBytes / 16);           // activations staged for the outliers after the walk
static_assert(kQuSmemBytes <= 227 * 1024 && kQuRows == 2688, "shared memory of one SM");

static __device__ int g_quad_error;   // 1: shared memory does not start at 1024, 2: a bounded wait ran out

// A work item: rows [0, n0) at base0, [n0, n) at base1, four vectors (an unused one repeats the first).
struct QuadItem {
    const uint8_t *base0, *base1;
    int n0, n, G;
    const void* x[kQuVecs];
    int K, io_dtype;
};

__device__ __forceinline__ uint64_t qu_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ uint64_t qu_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t qu_mul(uint64_t a, uint64_t b, uint64_t neg_zero) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg_zero));
    return r;
}
struct QuadSum { uint64_t a, b; };   // vectors 0, 1 and 2, 3
template <int I>
struct IntC { static constexpr int value = I; };
template <int OFF>
__device__ __forceinline__ QuadSum qu_lds(uint32_t addr) {
    QuadSum v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2+%3];" : "=l"(v.a), "=l"(v.b) : "r"(addr), "n"(OFF) : "memory");
    return v;
}
__device__ __forceinline__ void qu_sts(uint32_t addr, QuadSum v) {
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(v.a), "l"(v.b) : "memory");
}
template <int OFF>
__device__ __forceinline__ uint32_t qu_lds_u16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1+%2];" : "=h"(v) : "r"(addr), "n"(OFF) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t qu_prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// Barriers: full[2] (a builder warp each arrives), then empty[2] (a walker warp each).
__device__ __forceinline__ uint32_t qu_full(int slice) { return kQuCtl + (slice & 1) * 8; }
__device__ __forceinline__ uint32_t qu_empty(int slice) { return kQuCtl + 16 + (slice & 1) * 8; }
__device__ __forceinline__ void qu_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void qu_wait(uint32_t bar, unsigned parity) {
    if (!bar_wait(bar, parity, kQuGone)) atomicExch(&g_quad_error, 2);
}

template <class T>
__device__ __forceinline__ T* qu_at(unsigned char* raw, uint32_t shared_addr) { return reinterpret_cast<T*>(raw + (shared_addr - kQuCtl)); }

// Once per kernel, all threads; ends with a barrier.  False: the shared memory does not start where it should.
__device__ __forceinline__ bool quad_begin(unsigned char* raw, const float* __restrict__ codebook, int Kcb) {
    if (static_cast<uint32_t>(__cvta_generic_to_shared(raw)) != kQuCtl) {
        if (threadIdx.x == 0) atomicExch(&g_quad_error, 1);
        return false;
    }
    if (threadIdx.x < 4) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(kQuCtl + threadIdx.x * 8), "r"(threadIdx.x < 2 ? kQuBuilders : kQuWalkers) : "memory");
    }
    if (threadIdx.x < 4) *qu_at<float>(raw, kQuZero + threadIdx.x * 4) = 0.0f;
    if (threadIdx.x == 0) *qu_at<int>(raw, kQuGone) = 0;
    float2* book = qu_at<float2>(raw, kQuBook);
    for (int i = threadIdx.x; i < 256 * 8; i += kQuThreads) {
        const float c = i < Kcb * 8 ? codebook[i] : 0.0f;
        book[i] = make_float2(c, c);
    }
    __syncthreads();
    return true;
}

// Warps 8..11: the tables of an item's slices.  `first` is the number of slices this CTA has built before; parities follow from it.
// Lane: unit lane & 7; the four centroids of a warp step in lanes 0..7, 8..15, ...; 272 bytes a unit keep its reads of the
// activations apart.
__device__ __forceinline__ void quad_build(unsigned char* raw, const QuadItem& it, int Kcb, int first, float neg_zero) {
    const int tb = threadIdx.x - kQuWalkers * 32, lane = threadIdx.x & 31, wb = tb >> 5, u = lane & 7;
    const int S = (it.G + kQuSlice - 1) / kQuSlice;
    const uint64_t nz = qu_pack(neg_zero, neg_zero);
    // the first 128 threads bring an element (of 16 * 8) of the four vectors each
    const XLoad x0{it.x[0], it.K, it.io_dtype}, x1{it.x[1], it.K, it.io_dtype}, x2{it.x[2], it.K, it.io_dtype}, x3{it.x[3], it.K, it.io_dtype};
    float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tb < kQuSlice * 8) f = make_float4(x0(tb), x1(tb), x2(tb), x3(tb));
    for (int s = 0; s < S; ++s) {
        const int at = first + s;
        const uint32_t xs = kQuXs + (at & 1) * kQuXsBytes;
        if (tb < kQuSlice * 8) *qu_at<float4>(raw, xs + (tb >> 4) * 272 + (tb & 15) * 16) = f;
        asm volatile("bar.sync 1, %0;" ::"n"(kQuBuilders * 32) : "memory");
        if (s + 1 < S && tb < kQuSlice * 8) {
            const int e = (s + 1) * kQuSlice * 8 + tb;
            f = make_float4(x0(e), x1(e), x2(e), x3(e));
        }
        QuadSum x[2][8];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int d = 0; d < 8; ++d) x[j][d] = qu_lds<0>(xs + u * 272 + (j * 8 + d) * 16);
        const bool mine = s * kQuSlice + 2 * u < it.G;   // units past the last group hold -0, which changes no sum
        const bool whole = Kcb == 256 && (s + 1) * kQuSlice <= it.G;
        if (at >= 2) qu_wait(qu_empty(at), (unsigned)(((at >> 1) - 1) & 1));
        const uint32_t out = kQuTab + (at & 1) * kQuTabBytes + u * 16;
        constexpr int kStep = 4 * kQuBuilders;   // centroids that the builders take at a time
        int k = wb * 4 + (lane >> 3);
        QuadSum c[kQuSets][4];                   // (c0, c0, c1, c1) and so on
        auto fetch = [&](int k0) {
#pragma unroll
            for (int h = 0; h < kQuSets; ++h)
#pragma unroll
                for (int q = 0; q < 4; ++q) c[h][q] = qu_lds<0>(kQuBook + (k0 + h * kStep) * 64 + q * 16);
        };
        fetch(k);
#pragma unroll 1
        for (; k < 256; k += kQuSets * kStep) {
            QuadSum dot[kQuSets][2];
#pragma unroll
            for (int d = 0; d < 8; ++d)
#pragma unroll
                for (int h = 0; h < kQuSets; ++h) {
                    const uint64_t cc = d & 1 ? c[h][d >> 1].b : c[h][d >> 1].a;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint64_t pa = qu_mul(x[j][d].a, cc, nz), pb = qu_mul(x[j][d].b, cc, nz);
                        dot[h][j].a = d ? qu_add(dot[h][j].a, pa) : pa;
                        dot[h][j].b = d ? qu_add(dot[h][j].b, pb) : pb;
                    }
                }
            fetch((k + kQuSets * kStep) & 255);
            if (!whole)
#pragma unroll
                for (int h = 0; h < kQuSets; ++h) {
                    if (k + h * kStep >= Kcb) dot[h][0] = dot[h][1] = QuadSum{0ull, 0ull};
                    if (!mine) dot[h][0] = dot[h][1] = QuadSum{0x8000000080000000ull, 0x8000000080000000ull};
                }
#pragma unroll
            for (int h = 0; h < kQuSets; ++h) {
                qu_sts(out + (k + h * kStep) * 256, dot[h][0]);
                qu_sts(out + (k + h * kStep) * 256 + 128, dot[h][1]);
            }
        }
        __syncwarp();
        if (lane == 0) qu_arrive(qu_full(at));
    }
}

// Warps 0..7: adds all slices to the parked sums, which end up in acc[row] (float4).  WIDE: code rows start on 16-byte boundaries
// (else on 8-byte ones).  A step reads the code pair of four steps ahead, gathers the entries of two steps ahead and adds its own.
template <bool WIDE>
__device__ __forceinline__ void quad_walk(const QuadItem& it, int first) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lam = lane & 7;
    const int S = (it.G + kQuSlice - 1) / kQuSlice, blocks = (it.n + 31) >> 5;
    // Blocks warp, warp + 8, ...; at least two, so that a block's sums of the last slice are parked before they are read again.
    const int nb = max(2, (blocks - warp + kQuWalkers - 1) / kQuWalkers), M = S * nb;
    const uint32_t ring = kQuRing + warp * kQuRingBytes, place = (lane >> 3) * 16 + (lam & 1) * 64 + (lam >> 1) * 128;
    const int row_step = 32 * kQuWalkers, row_first = 32 * warp + lane;

    // the next chunk to ask for: its slot, block, slice, this lane's row and where that row lies
    uint32_t rq_dst = ring + place;
    int rq_b = 0, rq_g = 0, rq_row = row_first;
    const ptrdiff_t gap = it.base1 - it.base0 - (ptrdiff_t)it.n0 * it.G;   // between the two runs of rows
    const uint8_t* const src_first = it.base0 + (ptrdiff_t)row_first * it.G;
    const uint8_t* rq_src = src_first;
    const ptrdiff_t src_step = (ptrdiff_t)row_step * it.G;
    auto request = [&]() {
        const uint8_t* src = rq_row < it.n0 ? rq_src : rq_src + gap;
        const int ok = rq_row < it.n && rq_g < it.G;
        if (WIDE) asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p cp.async.cg.shared.global [%0], [%1], 16;\n}" ::"r"(rq_dst), "l"(src), "r"(ok) : "memory");
        else {
            const int ok2 = ok && rq_g + 8 < it.G;
            asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p cp.async.ca.shared.global [%0], [%1], 8;\n}" ::"r"(rq_dst), "l"(src), "r"(ok) : "memory");
            asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p cp.async.ca.shared.global [%0], [%1], 8;\n}" ::"r"(rq_dst + 8), "l"(src + 8), "r"(ok2) : "memory");
        }
        rq_dst += 512;
        if (rq_dst >= ring + kQuRingBytes) rq_dst -= kQuRingBytes;
        rq_row += row_step;
        rq_src += src_step;
        if (++rq_b == nb) {
            rq_b = 0;
            rq_g += kQuSlice;
            rq_row = row_first;
            rq_src = src_first + rq_g;
        }
    };
    for (int m = 0; m < kQuChunks - 3; ++m) {
        request();
        if ((m & 1) == 0) cp_async_commit();   // chunks 0; 1, 2; 3, 4
    }
    cp_async_wait<(kQuChunks - 4) / 2>();
    __syncwarp();
    qu_wait(qu_full(first), (unsigned)((first >> 1) & 1));

    // Of the period p (eight steps, in step i lane l with l mod 8 = i goes on from chunk p - 1 to chunk p): where the lane's codes
    // and entries are, less what the step adds.  Lanes that still are in chunk p - 1 are one row of codes or table units further.
    const uint32_t codes0 = ring + place - 2 * lam;
    auto table_at = [&](int slice) { return kQuTab + ((first + slice) & 1) * kQuTabBytes + 128 - 16 * lam; };
    uint32_t pr = codes0 + (kQuChunks - 1) * 512 + 16, pr_next = codes0, tb = table_at(0) + 128, tb_next = table_at(0);
    uint32_t cw[4];
    QuadSum e[2][2];
    QuadSum run{0ull, 0ull}, start{0ull, 0ull};
    auto code = [&](auto I) {
        constexpr int i = decltype(I)::value;
        if (lam == i) pr = pr_next;
        return qu_lds_u16<2 * i>(pr);
    };
    auto gather = [&](auto I, uint32_t w, QuadSum (&out)[2]) {
        constexpr int i = decltype(I)::value;
        if (lam == i) tb = tb_next;
        out[0] = qu_lds<16 * i - 128>(qu_prmt(w, tb, 0x7604));
        out[1] = qu_lds<16 * i>(qu_prmt(w, tb, 0x7614));
    };
    cw[0] = code(IntC<0>{}); cw[1] = code(IntC<1>{}); cw[2] = code(IntC<2>{}); cw[3] = code(IntC<3>{});
    gather(IntC<0>{}, cw[0], e[0]);
    gather(IntC<1>{}, cw[1], e[1]);

    int b = 0, s = 0;          // block and slice of chunk p
    uint32_t park = kQuDump + lane * 16;   // where the lane parks chunk p - 1
    QuadSum fin{0ull, 0ull};
    for (int p = 0; p <= M; ++p) {
        if ((p & 1) == 0) {
            __syncwarp();      // chunk p - 2 has been read by all lanes
            request();
            request();
            cp_async_commit();
            cp_async_wait<(kQuChunks - 4) / 2>();
            __syncwarp();      // chunks p + 1 and p + 2 are there for all lanes
        }
        const int b1 = b + 1 == nb ? 0 : b + 1, s1 = b1 == 0 ? s + 1 : s;   // of chunk p + 1
        const uint32_t pr_after = pr_next == codes0 + (kQuChunks - 1) * 512 ? codes0 : pr_next + 512, tb_after = table_at(s1);
        const int row = row_first + b * row_step, row1 = row_first + b1 * row_step;
        auto step = [&](auto I) {
            constexpr int i = decltype(I)::value;
            if (i == 4) { pr += 16; pr_next = pr_after; }     // the code pairs of the steps from here on are the next period's
            const uint32_t w = code(IntC<(i + 4) & 7>{});
            QuadSum n[2];
            if (i == 6) {
                tb += 128;
                tb_next = tb_after;
                if (b1 == 0 && s1 < S) qu_wait(qu_full(first + s1), (unsigned)(((first + s1) >> 1) & 1));
            }
            gather(IntC<(i + 2) & 7>{}, cw[(i + 2) & 3], n);
            if (lam == i) {
                fin = run;
                run = start;
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                run.a = qu_add(run.a, e[i & 1][j].a);
                run.b = qu_add(run.b, e[i & 1][j].b);
            }
            e[i & 1][0] = n[0];
            e[i & 1][1] = n[1];
            cw[i & 3] = w;
        };
        step(IntC<0>{}); step(IntC<1>{}); step(IntC<2>{}); step(IntC<3>{});
        step(IntC<4>{}); step(IntC<5>{}); step(IntC<6>{}); step(IntC<7>{});
        qu_sts(park, fin);     // every lane has gone on from chunk p - 1
        park = row < it.n ? kQuAcc + row * 16 : kQuDump + lane * 16;
        start = qu_lds<0>(s1 > 0 && row1 < it.n ? kQuAcc + row1 * 16 : kQuZero);
        if (b == 0 && s > 0) {   // every lane has left the slice before
            __syncwarp();
            if (lane == 0) qu_arrive(qu_empty(first + s - 1));
        }
        b = b1;
        s = s1;
    }
    cp_async_wait<0>();
}

// All threads: acc[row] (float4 at kQuAcc) = the four vectors' sums of the item's rows; ends with a barrier.  `first`: slices this
// CTA has worked through before.
__device__ __forceinline__ void quad_run(unsigned char* raw, const QuadItem& it, int Kcb, int& first, float neg_zero) {
    if ((int)threadIdx.x >= kQuWalkers * 32) quad_build(raw, it, Kcb, first, neg_zero);
    else if ((it.G & 15) == 0 && ((reinterpret_cast<uintptr_t>(it.base0) | reinterpret_cast<uintptr_t>(it.base1)) & 15) == 0) quad_walk<true>(it, first);
    else quad_walk<false>(it, first);
    first += (it.G + kQuSlice - 1) / kQuSlice;
    __syncthreads();
    if (*qu_at<volatile int>(raw, kQuGone)) {   // a wait ran out: no sum of this item is what it should be
        for (int i = threadIdx.x; i < it.n; i += kQuThreads) qu_at<float4>(raw, kQuAcc)[i] = make_float4(NAN, NAN, NAN, NAN);
        __syncthreads();
    }
}

// The four vectors side by side in the (idle) table area: xs[k] for the outliers of the rows.  Ends with a barrier.
__device__ __forceinline__ const float4* quad_stage_x(unsigned char* raw, const QuadItem& it) {
    float4* xs = qu_at<float4>(raw, kQuTab);
    const XLoad x0{it.x[0], it.K, it.io_dtype}, x1{it.x[1], it.K, it.io_dtype}, x2{it.x[2], it.K, it.io_dtype}, x3{it.x[3], it.K, it.io_dtype};
#pragma unroll 4
    for (int k = threadIdx.x; k < it.K; k += kQuThreads) xs[k] = make_float4(x0(k), x1(k), x2(k), x3(k));
    __syncthreads();
    return xs;
}

// The item's rows: (sum * scale + bias) + outlier row sum, the latter formed on its own from zero in entry order, multiply then
// add (ojasx_lut_cpu.cpp:178-182, :117-127); put(local row, four results).  row_of: local row to row of the matrix.  A thread
// has the entries of its next row and the bounds of the one after that on their way while it works on a row: with a row's loads
// in front of its sums this took 21 k clocks for 1280 rows of ten entries or 2560 of two and a half, 16 k and 11.5 k now.
template <class RowOf, class Put>
__device__ __forceinline__ void quad_rows(const float4* acc, int n, const CsrView& csr, const float* __restrict__ scales,
                                          const float* __restrict__ bias, const float4* xs, RowOf row_of, Put put) {
    constexpr int E = 8;
    const bool has = csr.nnz > 0;
    struct Row { int j, je, col[E]; float val[E], sc, bs; };
    auto bounds = [&](int lr, int& j, int& je) {
        j = je = 0;
        if (has && lr < n) {
            const int m = row_of(lr);
            j = csr.row_ptrs[m];
            je = csr.row_ptrs[m + 1];
        }
    };
    auto load = [&](Row& r, int lr, int j, int je) {
        r.j = j;
        r.je = je;
        r.sc = scales && lr < n ? scales[row_of(lr)] : 1.0f;
        r.bs = bias && lr < n ? bias[row_of(lr)] : 0.0f;
#pragma unroll
        for (int q = 0; q < E; ++q) {
            r.col[q] = j + q < je ? csr.cols[j + q] : 0;
            r.val[q] = j + q < je ? csr.vals[j + q] : 0.0f;
        }
    };
    int lr = threadIdx.x, j0, je0, j1, je1;
    Row row;
    bounds(lr, j0, je0);
    bounds(lr + kQuThreads, j1, je1);
    load(row, lr, j0, je0);
    for (; lr < n; lr += kQuThreads) {
        Row next;
        load(next, lr + kQuThreads, j1, je1);
        bounds(lr + 2 * kQuThreads, j1, je1);
        const float4 v = acc[lr];
        float r[4] = {v.x, v.y, v.z, v.w}, o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        auto add = [&](float val, float4 x) {
            o[0] = __fadd_rn(o[0], __fmul_rn(val, x.x));
            o[1] = __fadd_rn(o[1], __fmul_rn(val, x.y));
            o[2] = __fadd_rn(o[2], __fmul_rn(val, x.z));
            o[3] = __fadd_rn(o[3], __fmul_rn(val, x.w));
        };
        if (has) {
#pragma unroll
            for (int q = 0; q < E; ++q)
                if (row.j + q < row.je) add(row.val[q], xs[row.col[q]]);
            for (int j = row.j + E; j < row.je; j += E) {
                int col[E];
                float val[E];
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    col[q] = j + q < row.je ? csr.cols[j + q] : 0;
                    val[q] = j + q < row.je ? csr.vals[j + q] : 0.0f;
                }
#pragma unroll
                for (int q = 0; q < E; ++q)
                    if (j + q < row.je) add(val[q], xs[col[q]]);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (scales) r[c] = __fmul_rn(r[c], row.sc);
            if (bias) r[c] = __fadd_rn(r[c], row.bs);
            if (has) r[c] = __fadd_rn(r[c], o[c]);
        }
        put(lr, r);
        row = next;
    }
}

// The builders ask L2 for the outliers of rows [row0, row0 + n), before the walk that hides it.
__device__ __forceinline__ void quad_ask_outliers(const CsrView& csr, int row0, int n) {
    if (csr.nnz <= 0) return;
    const int jb = csr.row_ptrs[row0], je = csr.row_ptrs[row0 + n];
    for (int j = (jb & ~31) + (threadIdx.x - kQuWalkers * 32) * 32; j < je; j += kQuBuilders * 32 * 32) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(csr.cols + j));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(csr.vals + j));
    }
}

}  // namespace ojx
