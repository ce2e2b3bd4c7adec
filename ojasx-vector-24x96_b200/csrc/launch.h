// Host-side launch entry points shared by the C ABI translation unit.
#pragma once
#include <atomic>

#include "common.cuh"

namespace ojx {

// Launch of a kernel that begins with chain_begin(): its CTAs may be scheduled while the launch before it in the stream still runs
// (programmatic dependent launch), so that a chain of short kernels does not pay a launch latency between any two of them.  us, plain
// launches and these: routed MoE layer at one token (five kernels) 51.2 / 41.4, 32 append + decode pairs of a cache 620 / 568, SwiGLU
// block of one token (four kernels) 40.2 / 36.1, decode steps of two layers (26 kernels) 238 / 225 each.
template <class... Params, class... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
#ifdef __CUDACC__
// Waits until everything before this launch in the stream is done and visible, then lets the launch behind it be scheduled.  In this
// order, so that a kernel that has been scheduled knows that the launch before the last one is complete.
__device__ __forceinline__ void chain_begin() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}
#endif

// A kernel's opt-in to `bytes` of dynamic shared memory, the most that any of its launches takes, once per device.  The attribute belongs
// to the kernel, not to a thread or a launch: one that follows the size of a launch is lowered by another thread's.
inline cudaError_t opt_in_smem(const void* kernel, size_t bytes, std::atomic<bool> (&done)[64]) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool known = dev >= 0 && dev < 64;
    if (known && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t set = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (set == cudaSuccess && known) done[dev].store(true, std::memory_order_release);
    return set;
}

struct PeerLink;   // peer.cuh: exchange over peer memory fused into a kernel's epilogue (null / n == 0: none)
const PeerLink* peer_link_of(void* peer_link_handle);

// --- linear.cu
int plan_tile_rows(int rows, int parallel_items);
int validate_linear(const LinearProblem& P);
int launch_linear(LinearProblem P, cudaStream_t stream, const PeerLink* link = nullptr);
int launch_linear_group(const LinearProblem* d_probs, int nprobs, int total_items, int D, cudaStream_t stream,
                        const PeerLink* link = nullptr);

// --- linear_cluster.cu: OJX_ERR_UNSUPPORTED means "use the persistent kernel"
int try_launch_linear_cluster(const LinearProblem& P, cudaStream_t stream, const PeerLink* link = nullptr);
// Up to 8 host-side problems with the same K, G, block_dim, batch and io dtype in one cluster launch.
int try_launch_linear_cluster_group(const LinearProblem* probs, int count, cudaStream_t stream, const PeerLink* link = nullptr);
// True when OJASX_B200_LINEAR_KERNEL=persistent asks for the streaming kernel only.
bool linear_cluster_disabled();

// --- rvq_generic.cu
int launch_rvq_generic(const uint8_t* packed, const float* codebooks, const float* row_scales, const float* bias,
                       const float* x, int batch, int stages, int bits, int D, int rows, int columns, int row_start,
                       int row_stop, float* out, cudaStream_t stream);

// --- dequant_gemm.cu (tcgen05 path for bf16 batches)
bool dequant_gemm_supported(const LinearProblem& P, bool csr_sorted);
// scratch / scratch_cap: a grow-only device buffer of the caller (per layer handle) for the split-K partial
// sums and tile counters; null = never split.  Calls that share the buffer must not overlap in time.
// Outliers of a layer listed per (128-row, 64-column) weight tile for the tensor-core path; built on the device the
// first time a layer and row range take that path, kept by the layer's handle.
struct DqLists {
    int* off = nullptr;        // [row_tiles * (K / 64 + 1) + 1] tile offsets, followed by the scatter cursors
    int2* ent = nullptr;       // [nnz] (row in tile << 8 | column in tile, value / row scale)
    size_t off_cap = 0, ent_cap = 0;
    int row_start = -1, row_stop = -1;
    unsigned generation = 0;
    const float* csr_vals = nullptr;
    bool valid = false;
    ~DqLists();
};
int launch_dequant_gemm(const LinearProblem& P, cudaStream_t stream, DqLists* lists = nullptr, unsigned generation = 0);
bool dequant_gemm_pair_pays(const LinearProblem& A, const LinearProblem& B);
int launch_dequant_gemm_pair(const LinearProblem* P, cudaStream_t stream, DqLists* const* lists, const unsigned* generation);
int take_dequant_gemm_error(int* out);

// --- gather_mma.cu: bf16 batches below the tensor-core path, weights gathered into mma.sync operands at fp32 accuracy
bool gather_mma_supported(const LinearProblem& P);
size_t gather_mma_workspace(int K, int batch);   // bytes for the prepared activations of one call
int launch_gather_mma(const LinearProblem* P, int count, const void* x, const void* up, void* h, void* workspace, cudaStream_t s);

// --- moe.cu
// link: expert-parallel ranks gather every pair's expert output over peer memory before the combine (null: one rank)
int launch_moe_experts(MoeProblem P, cudaStream_t stream, const PeerLink* link = nullptr);
int launch_build_lut(const void* x, int io_dtype, int n_vectors, int K, int D, const float* codebook, int Kcb, float* out,
                     cudaStream_t stream);
int launch_silu_mul(const void* gate, const void* up, void* out, size_t n, int io_dtype, cudaStream_t stream);
// codebook .. lut_out: when lut_out is not null the gate/up tables of the tokens ([n_tokens, H/D, 256]) are
// built by the same launch as the logits.
int launch_moe_router(const float* Wr, const void* x, int io_dtype, int n_tokens, int H, int E, int k,
                      float* logits, float* probs, int* idx_out, float* w_out, cudaStream_t stream,
                      const float* codebook = nullptr, int Kcb = 0, int D = 0, float* lut_out = nullptr,
                      int lut_blocks = 0, const PeerLink* link = nullptr, int e_begin = 0, int e_end = 0);

// --- moe_fused.cu: whole-expert work items (gate/up, SiLU gate and down fused) for batches of tokens
bool moe_chain_wanted(const MoeProblem& P);   // gate/up by the chain walk: whole experts per work item and a fitting shape
int moe_table_layout(const MoeProblem& P);    // MoeProblem::lut_blocks this forward wants
size_t moe_table_bytes(int n_tokens, int G, int D);   // table scratch that fits every layout
int launch_moe_chain_images(const void* x, int io_dtype, int n_tokens, int H, int D, const float* cb, int Kcb, float* out, cudaStream_t s);
bool moe_fused_wanted(const MoeProblem& P);   // shape fits and enough routed pairs are expected here
int launch_moe_fused(MoeProblem P, cudaStream_t stream, const PeerLink* link = nullptr);   // work list, token tables (unless lut_ready), experts
int launch_moe_prebuild_blocks(const void* x, int io_dtype, int n_tokens, int H, int D, const float* codebook, int Kcb,
                               float* out, cudaStream_t stream);
// --- moe_gather.cu: experts that several tokens are routed to, on mma.sync operands gathered from the codebooks
bool moe_gather_wanted(const MoeProblem& P);
int launch_moe_gather(const MoeProblem& P, cudaStream_t s, const PeerLink& link);   // all but the combine
// Work list of the two: pairs grouped by expert, cut into items of up to `width` pairs.  plan [4 + 5 * pairs]: [0] items, [1], [2]
// claim counters, [3] pairs, sorted pair ids, then (expert, first, count, -) per item.
int launch_moe_item_plan(const MoeProblem& P, int* plan, int width, cudaStream_t s);
// --- lut_quad.cu: four vectors at a time in the reference's order of additions
bool quad_linear_pays(const LinearProblem& P);
int launch_quad_linear(LinearProblem P, cudaStream_t s, const PeerLink& link);
bool moe_quad_wanted(const MoeProblem& P);
int launch_moe_quad(const MoeProblem& P, cudaStream_t s, const PeerLink& link);   // all but the combine
int take_quad_error(int* out);
int take_moe_fused_error(int* out);
int take_moe_bulk_copy_error(int* out);   // moe.cu: a bounded wait for a bulk table copy ran out

// --- kv.cu
constexpr int kKvMaxSplits = 256;   // context splits of one (sequence, KV head) in kvq decode
size_t kvq_decode_smem(const KvqProblem& P, int R);
// Partial sums that a decode may need per (sequence, KV head): one per 256 tokens, or where there are few heads what shares the
// tokens out over the SMs.  A plan never makes more: its chunks are no shorter than 256 tokens or than an SM's share (64 at
// least).  At 128 heads of 4 query heads, head_dim 128 and 16384 tokens 17 MB (one per 64 tokens took 68, and as many for each of
// 16 positions 1.1 GB).
inline int kvq_scratch_splits(int max_seq, int heads, int sms) {
    const int tokens = (max_seq + 255) / 256, least = (max_seq + 63) / 64, share = (sms + heads - 1) / heads;
    const int few = least < share ? least : share, n = tokens > few ? tokens : few;
    return n < kKvMaxSplits ? n : kKvMaxSplits;
}
// The same for positions of a prompt: enough for two CTAs per SM.
inline int kvq_position_splits(int splits, int heads, int sms) {
    const int fill = (2 * sms + heads - 1) / heads, n = splits > fill ? splits : fill;
    return n < kKvMaxSplits ? n : kKvMaxSplits;
}
// Fills P.chunk (tokens per CTA) and P.n_chunks (<= max_splits, what the scratch holds per position) for a context of T tokens.
void plan_kvq_decode(KvqProblem& P, int T, int sms, int max_splits);
// Positions whose partial sums fit a scratch of max_splits per (sequence, KV head).
int kvq_decode_positions(KvqProblem P, int T, int sms, int max_splits);
int launch_kvq_append(const KvqProblem& P, cudaStream_t stream);
bool kvq_table_decode_fits(const KvqProblem& P);   // what the query-table kernel takes: the shapes of fp32 caches
int launch_kvq_decode(const KvqProblem& P, cudaStream_t stream, const PeerLink* link = nullptr);
// --- kv_decode_mma.cu: decode for block_dim 8 and head_dim 64 or 128 (launch_kvq_decode takes it where it fits)
bool kvq_decode_mma_supported(const KvqProblem& P);
int launch_kvq_decode_mma(const KvqProblem& P, cudaStream_t stream, const PeerLink& link);
// --- kv_prefill.cu: a chunk of P.n_pos prompt positions (lengths are advanced last)
int launch_kvq_append_many(const KvqProblem& P, cudaStream_t stream);
bool kvq_prefill_supported(const KvqProblem& P);
int launch_kvq_prefill_attention(const KvqProblem& P, cudaStream_t stream);
int launch_kvq_advance(const KvqProblem& P, cudaStream_t stream);
int launch_legacy_append(const float* k, const float* v, int head_dim, int block_dim, uint8_t* k_row, uint8_t* v_row,
                         float* k_scale, float* v_scale, cudaStream_t stream);
int launch_legacy_attention(const float* q, int head_dim, int block_dim, int T, const uint8_t* k_codes,
                            const uint8_t* v_codes, const float* k_scales, const float* v_scales, float scale_factor,
                            float* logits, float* out, cudaStream_t stream);

}  // namespace ojx
