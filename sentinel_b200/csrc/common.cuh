// Shared declarations of the attention library's translation units.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "sntl_attn.h"

namespace sntl {

// Launch accounting (attn_api.cu).
void count_launch(int n = 1);

// Element strides of a [B][H][S][D]-indexed tensor; covers both layouts of the C ABI.
struct View4 {
    long long sb, sh, ss, sd;
};
// Element strides of a [B][H][S]-indexed fp32 tensor (LSE, delta).
struct View3 {
    long long sb, sh, ss;
};

struct AttnShape {
    int B, Hq, Hkv, Sq, Skv, D;
    float scale;
    int causal;
    int window;         // sliding window (keys a query sees counting itself); <= 0: unlimited.  Needs causal.
    int global_tokens;  // the first global_tokens keys stay visible to every later query
    int deterministic;  // backward: dQ summed in 64-bit fixed point, so the result does not depend on the order of arrival
    int whole_tiles;    // tensor-core backward: never cut key tiles into pieces
};

// The window part of the reference's CausalSelfAttention::allowsKey (CausalSelfAttention.cpp:95-100); the causal part
// (key <= query) is the caller's.
__host__ __device__ __forceinline__ bool window_allows(const AttnShape& s, int query, int key)
{
    return s.window <= 0 || key < s.global_tokens || key >= query - s.window + 1;
}

// Opt-in to more than 48 KB of dynamic shared memory for `kernel`, once per device: cudaFuncSetAttribute applies to the
// current device only, so a process that drives several GPUs needs it on each.  `done_mask` is the caller's static
// bookkeeping word (one bit per device ordinal below 64; higher ordinals simply set the attribute on every call).
// The first call on a device has to come before any stream capture, like the reference's own lazy configuration
// (CudaFlashAttention.cu:49-66).
template <typename Kernel>
inline cudaError_t ensure_dynamic_smem(Kernel kernel, size_t bytes, std::atomic<unsigned long long>& done_mask)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && ((done_mask.load(std::memory_order_acquire) >> dev) & 1ull)) return cudaSuccess;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done_mask.fetch_or(1ull << dev, std::memory_order_release);
    return cudaSuccess;
}

// Programmatic dependent launch: a kernel's blocks may start as soon as all blocks of the one before it in the stream have
// exited or are running out, before that one has been flushed, so that launch latency, barrier set-up and tensor-memory
// allocation overlap its end (1-3 us a launch).  wait_for_stream() comes before the first access to global memory in every
// block of every kernel launched this way: it returns when all earlier work of the stream has completed and its writes are
// visible, so ordering is what it would be without.  (Triggering the next launch explicitly at the start of a kernel was slower
// everywhere: 126 vs 121 us on the B8 H12 S1024 D64 training step, 242 vs 218 on a ragged head_dim-128 one.)
__device__ __forceinline__ void wait_for_stream() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, unsigned cluster, A&&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster > 1) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = cluster;
        attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
    if (e == cudaSuccess) count_launch();
    return e;
}

// What a kernel accesses `bytes` at a time has to start on such a boundary; a misaligned access would take the context down.
template <typename... P> inline bool aligned(uintptr_t bytes, const P*... p) { return (((uintptr_t)p | ... | (uintptr_t)0) % bytes) == 0; }

// Asynchronous copies of 16 bytes, global -> shared (both on 16-byte boundaries), in groups per thread
__device__ __forceinline__ void copy16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_left() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Two fp32 FMAs in one instruction, each rounded as the scalar one
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
          "l"(reinterpret_cast<unsigned long long&>(c)));
    return d;
}

// SMs of the current device (148 on a B200), read once per device ordinal
inline int sm_count()
{
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int n = cached[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Exact-fp32 SIMT kernels (attn_simt_fwd.cu, attn_simt_bwd.cu).  T = float or __nv_bfloat16 element type.
struct SimtArgs {
    AttnShape s;
    int is_bf16;
    const void *q, *k, *v, *o, *dout;
    void *o_out, *dq, *dk, *dv;
    float* lse_out;
    const float* lse;
    View4 vq, vkv;     // q-like tensors (Q, O, dO, dQ) and kv-like tensors (K, V, dK, dV)
    View3 vlse;
    bool vec_q, vec_kv;   // every row of all q-like / kv-like tensors can be accessed four elements at a time
    // The FMA kernels behind the tensor-core ones compute only what those left (blocks of 128 rows with values that their products do
    // not take): forward, query tiles whose LSE rows hold kOddLse; backward, tiles whose word of odd_marks is not 0 (null: all tiles).
    bool only_odd;
    uint32_t* odd_marks;  // backward: one word per 128 keys of every (batch, KV head), then one per 128 queries of every (batch, head)
};
constexpr uint32_t kOddLse = 0x7fc0dd5au;   // a NaN that no computation returns
cudaError_t simt_forward(const SimtArgs& a, cudaStream_t st);
// few query rows per KV head (decode): simt_forward takes this path by itself where it applies
bool simt_decode_supported(const SimtArgs& a);
cudaError_t simt_decode(const SimtArgs& a, cudaStream_t st);
cudaError_t simt_backward(const SimtArgs& a, cudaStream_t st);  // one launch
// The same results from split products on the tensor cores (attn_f32_fwd_sm100.cu, attn_f32_bwd_sm100.cu): fp32, head_dim up to 64, where
// there is enough work.  They leave odd blocks to simt_forward / simt_backward with the marks.
// Where that pays by the estimates of attn_f32_route.cu, from the tiles that the FMA kernels would take (head_dim up to 64).
struct SimtTiles {
    int rows, split;      // query rows of a tile, CTAs that share its keys
};
SimtTiles simt_forward_tiles(const AttnShape& s);
int simt_backward_rows(const AttnShape& s);
bool f32_tc_forward_pays(const AttnShape& s);
bool f32_tc_backward_pays(const AttnShape& s);
bool f32_tc_forward_supported(const SimtArgs& a);
cudaError_t f32_tc_forward(const SimtArgs& a, cudaStream_t st);
bool f32_tc_backward_supported(const SimtArgs& a, size_t marks_bytes);
cudaError_t f32_tc_backward(const SimtArgs& a, cudaStream_t st);

// Results in the reference's feature-major layout: element (b, h, s, d) at ((h*D + d)*stride + b*S + s), LSE (b, h, s) at
// (h*stride + b*S + s); the pointers include the first column of the window.
struct MatrixOut {
    float *o, *lse, *dq, *dk, *dv;
    long long stride;
};

// Tensor-core kernels (attn_fwd_sm100.cu / attn_bwd_sm100.cu): bf16, BHSD contiguous, D in {64,128}.
struct TcArgs {
    AttnShape s;
    const __nv_bfloat16 *q, *k, *v, *o, *dout;
    __nv_bfloat16 *o_out, *dq, *dk, *dv;
    float* lse_out;
    const float* lse;
    float* delta;      // start of the backward workspace: the per-row records (kBwdRowAuxBytes per padded query row)
    float* dq_accum;   // [B][Hq][Sq_pad][D] fp32
    // Backward in pieces (the ring schedule: one query block meets several key blocks).  phases selects which of the
    // three launches run: kBwdPre (per-row records, dQ accumulator zeroed), kBwdMain (the tensor-core kernel, which
    // ADDS this key block's dQ into the accumulator), kBwdPost (accumulator -> bf16 dQ).  0 = all three.
    // dk_acc / dv_acc non-null: the main kernel adds its dK (times scale) / dV into these fp32 [B][Hkv][Skv][D]
    // tensors instead of writing bf16 dk / dv (each element has one owning CTA per launch, so the read-modify-write
    // needs no atomics and stays deterministic).
    int phases = 0;
    float* dk_acc = nullptr;
    float* dv_acc = nullptr;
    MatrixOut mat{};   // non-null members: results leave as fp32 feature-major matrices instead of bf16 [B][H][S][D]
};
enum : int { kBwdPre = 1, kBwdMain = 2, kBwdPost = 4 };
bool tc_fwd_supported(const AttnShape& s);
bool tc_bwd_supported(const AttnShape& s);
cudaError_t tc_forward(const TcArgs& a, cudaStream_t st);
// New tokens against a KV cache (attn_cache_sm100.cu, forward only): s.Sq new tokens per head at positions Skv-Sq .. Skv-1, K/V
// slabs `capacity` rows apart.  Partial results go through `workspace` (tc_cache_workspace_bytes) and a merge kernel.
size_t tc_cache_workspace_bytes(const AttnShape& s);
bool tc_cache_supported(const AttnShape& s);
cudaError_t tc_cache_forward(const TcArgs& a, int capacity, void* workspace, cudaStream_t st);
cudaError_t tc_backward(const TcArgs& a, cudaStream_t st);
// Deterministic backward: whether dQ comes from a kernel with one owner per element (attn_dq_sm100.cu); else the main kernel reduces 64-bit
// words, whose traffic costs less at head_dim 64 than computing S and dP twice (backward, us, reductions against such a kernel: B4 Hq32
// Hkv8 S4096 1056 against 977 with fewer roundings, B8 H8 S2048 57 against 59, one head of 8192 tokens 88 against 106).
__host__ __device__ constexpr bool bwd_dq_has_kernel(int D) { return D == 128; }
cudaError_t tc_backward_dq(const TcArgs& a, cudaStream_t st);   // dQ alone; a.delta holds the row terms
size_t tc_backward_workspace_bytes(const AttnShape& s);
// Bytes per padded query row at the head of the tensor-core backward workspace: two 16-byte records (the extra
// contraction-step operands that carry -delta and -LSE/scale into the dP^T and S^T products)
constexpr size_t kBwdRowAuxBytes = 2 * 16;

// Layout / dtype staging (layout_convert.cu): SENTINEL fp32 feature-major <-> bf16 BHSD.
// The same relayouts with the rotary embedding applied on the way (cos_t == nullptr: plain relayout).
cudaError_t rope_pack_bf16(const float* src, __nv_bfloat16* dst, int B, int H, int S, int D, int stride_columns,
                           int column_start, const float* cos_t, const float* sin_t, int position_offset, cudaStream_t st);
cudaError_t rope_unpack_f32(const __nv_bfloat16* src, float* dst, int B, int H, int S, int D, int stride_columns,
                            int column_start, const float* cos_t, const float* sin_t, int position_offset, bool inverse,
                            cudaStream_t st);
// Everything a tensor-core call needs from feature-major fp32 matrices, in one launch: up to four of them converted to bf16
// [B][H][S][D], and for the backward (o_mat non-null) the per-query terms from O, dO and LSE, and the dQ accumulator zeroed.
struct MatrixStage {
    const float* src[4];
    __nv_bfloat16* dst[4];
    int heads[4];
    int n;
    const float *o_mat, *do_mat, *lse_mat;
    void* row_terms;          // start of the backward workspace
    float* dq_accum;
    size_t accum_bytes;
};
cudaError_t stage_matrices(const MatrixStage& m, int B, int Hq, int S, int D, int stride_columns, int column_start, float scale, cudaStream_t st);
cudaError_t f32_to_bf16(const float* src, __nv_bfloat16* dst, size_t n, cudaStream_t st);
cudaError_t bf16_to_f32(const __nv_bfloat16* src, float* dst, size_t n, cudaStream_t st);
cudaError_t accumulate_f32(int part_dtype, float* acc, const void* part, size_t n, cudaStream_t st);
cudaError_t merge_partials(int acc_dtype, int part_dtype, long long rows, int D, void* o_acc, float* lse_acc,
                           const void* o_part, const float* lse_part, cudaStream_t st);

// A one-warp kernel whose only wait can never complete, limited to limit_ns (attn_fwd_sm100.cu): exercises the
// give-up path of the bounded waits without hanging or faulting anything.  *gave_up (device memory, optional) <- 1.
cudaError_t launch_wait_selftest(unsigned long long limit_ns, cudaStream_t st);

// Device status words written by bounded waits (one per tensor-core translation unit; the first reports the KV-cache kernel's and the fp32 forward's too, the second the
// fp32 backward's).
cudaError_t read_and_clear_fwd_status(cudaStream_t st, uint32_t* word);
cudaError_t read_and_clear_cache_status(uint32_t* word);   // after a synchronisation of the stream
cudaError_t read_and_clear_f32_fwd_status(uint32_t* word);
cudaError_t read_and_clear_f32_bwd_status(uint32_t* word);
cudaError_t read_and_clear_dq_status(uint32_t* word);
cudaError_t read_and_clear_bwd_status(cudaStream_t st, uint32_t* word);

}  // namespace sntl
