// Shared declarations of the kernel library: error reporting, dtype traits and the small set
// of PTX wrappers (cp.async, ldmatrix, mma.sync, ex2) the attention kernels are written with.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <utility>

#include "../../include/nvk.h"
#include "decode_sizes.h"

namespace nvk {

// ---- host-side error reporting -------------------------------------------------------------
// Stores a printf-formatted message for nvk_last_error() and returns `code`.
int fail(int code, const char* fmt, ...);
// Checks cudaPeekAtLastError() right after a launch (the reference's convention,
// src/kernels/attention.cu:442); returns NVK_OK or NVK_ERR_CUDA.
int check_launch(const char* what);

inline bool aligned_to(const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }
inline size_t dtype_size(int dtype) {
    switch (dtype) {
        case NVK_F16: case NVK_BF16: return 2;
        case NVK_F32: case NVK_I32: return 4;
        case NVK_I64: return 8;
        case NVK_I8: return 1;
        default: return 0;
    }
}

// An index tensor of the boundary (cu_seqlens_*, context_lens, block_tables): int32 or int64 elements, each tensor
// on its own, as the reference's kernels accept them (src/kernels/attention.cu:644-660, :708-735).  The width is a
// launch-uniform flag read where an index is loaded; values are widened to 64 bits.
struct IndexArray {
    const void* ptr = nullptr;
    int wide = 0;   // 1 = int64 elements, 0 = int32
    IndexArray() = default;
    __host__ __device__ IndexArray(const void* p, int w) : ptr(p), wide(w) {}
    __host__ __device__ explicit operator bool() const { return ptr != nullptr; }
    __host__ __device__ bool operator==(std::nullptr_t) const { return ptr == nullptr; }
    __host__ __device__ bool operator!=(std::nullptr_t) const { return ptr != nullptr; }
    __host__ __device__ IndexArray operator+(int64_t n) const {
        return IndexArray(static_cast<const char*>(ptr) + n * (wide ? 8 : 4), wide);
    }
#ifdef __CUDACC__
    __device__ __forceinline__ int64_t operator[](int64_t i) const {
        return wide ? static_cast<const int64_t*>(ptr)[i] : static_cast<int64_t>(static_cast<const int32_t*>(ptr)[i]);
    }
    // An index as loaded, both words; value() widens it later, so that other loads can be issued before this one has come back (operator[] waits
    // for it to extend its sign).
    struct Raw { int lo, hi; };
    __device__ __forceinline__ Raw raw(int64_t i, bool there = true) const {   // (0 without a load where there is none)
        Raw r;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %4, 0;\n\tsetp.ne.and.s32 p, %3, 0, q;\n\tmov.s32 %0, 0;\n\tmov.s32 %1, 0;\n\t"
            "@q ld.global.s32 %0, [%2];\n\t@p ld.global.s32 %1, [%2+4];\n\t}\n"
            : "=r"(r.lo), "=r"(r.hi) : "l"(static_cast<const char*>(ptr) + (i << (2 + wide))), "r"(wide), "r"(static_cast<int>(there)));
        return r;
    }
    __device__ __forceinline__ int64_t value(Raw r) const {
        const int hi = wide ? r.hi : r.lo >> 31;
        return static_cast<int64_t>((static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32) | static_cast<uint32_t>(r.lo));
    }
#endif
};

// Division of 0 <= n < 2^31 by a launch-uniform number: a multiplication and a shift instead of some 25 instructions in a chain (the rounded-up
// reciprocal of Granlund and Montgomery, Division by Invariant Integers using Multiplication, 1994).
struct FastDiv {
    uint32_t d = 1, mul = 1, shift = 0;
    FastDiv() = default;
    explicit FastDiv(uint32_t by) : d(by) {   // 1 <= by < 2^31
        while ((1ull << shift) < by) ++shift;
        mul = static_cast<uint32_t>(((1ull << 32) * ((1ull << shift) - by)) / by + 1);
    }
#ifdef __CUDACC__
    __host__ __device__
#endif
    uint32_t div(uint32_t n) const {   // (mul * n / 2^32 <= n, so that the sum stays below 2^32)
        return (static_cast<uint32_t>((static_cast<uint64_t>(n) * mul) >> 32) + n) >> shift;
    }
};

constexpr int kSmCount = 148;   // of a B200; grids are sized by it

// ---- launchers (one per .cu file) -----------------------------------------------------------
struct DecodeArgs {
    const void* q; const void* k_cache; const void* v_cache;
    IndexArray context_lens; IndexArray block_tables;
    void* out;
    int64_t batch, max_blocks, num_cache_blocks;
    int num_heads, num_kv_heads, head_dim, block_size;
    float scale;
    int dtype;
    void* workspace; size_t workspace_bytes;
    cudaStream_t stream;
    bool beside = false;         // runs beside the kernel launched just before it on the stream, see pdl_wait_beside
};
struct DecodeInt8Args {          // 8-bit caches (int8, or e4m3 when fp8 is set) with one fp16 scale per (cache row, KV head)
    DecodeArgs base;
    const void* k_scale; const void* v_scale;
    bool fp8 = false;
};
struct PrefillArgs {
    const void* q; const void* k; const void* v;          // dense keys (k, v) or paged (caches)
    const void* k_cache; const void* v_cache;
    IndexArray cu_q; IndexArray cu_k; IndexArray block_tables;
    void* out;
    int64_t num_seqs, total_q, total_k, max_blocks, num_cache_blocks;
    int max_seqlen_q, num_heads, num_kv_heads, head_dim, block_size;
    float scale;
    int dtype;
    cudaStream_t stream;
};

int launch_store_kvcache(const void* key, const void* value, void* k_cache, void* v_cache,
                         const void* slot_mapping, bool slot_i64, int64_t num_tokens,
                         int64_t row_bytes, int64_t cache_rows, cudaStream_t stream);
int launch_fused_prologue(const void* qkv, const int32_t* positions, const void* qw, const void* kw,
                          float eps, const float* cos_sin, int64_t max_positions,
                          const int32_t* slot_mapping, void* k_cache, void* v_cache,
                          int64_t cache_rows, int64_t rows, int hq, int hkv, int d, void* q_out,
                          int dtype, cudaStream_t stream);
// General SIMT attention (any dtype of F16/BF16/F32, head_dim <= 256, any block size).
int launch_rowwise_decode(const DecodeArgs& a);
int launch_rowwise_prefill(const PrefillArgs& a);
// fp32-arithmetic decode, head_dim 64 / 128 / 256 (decode_simt.cu).
bool decode_simt_supported(const DecodeArgs& a);
int launch_decode_simt(const DecodeArgs& a);
// Tensor-core paths (F16/BF16, head_dim 128).
bool decode_mma_supported(const DecodeArgs& a);
size_t decode_mma_workspace_bytes(int64_t batch, int num_heads, int num_kv_heads, int head_dim,
                                  int64_t max_blocks, int block_size);
int check_decode_mma(const DecodeArgs& a);
int launch_decode_mma(const DecodeArgs& a);
namespace dec { struct DecodeParams; }
int decode_plan(const DecodeArgs& a, int groups, dec::DecodeParams* out, int* cluster);
int launch_decode_merge(const dec::DecodeParams& p, int dtype, cudaStream_t stream);
// Fused all-reduce launchers (tp_allreduce.cu); `pushed`: the other ranks' slices were already pushed by the GEMM
// that produced the addend (gemm_fused.cu), the kernel starts with the reduction.
void set_multimem_wait_cycles(long long cycles);   // tp_allreduce_mm.cu: the wait limit of the multimem kernels
int launch_allreduce_add_rmsnorm(const void* in, void* out, void* norm, void* const* stage_ptrs, size_t stage_bytes, void* flags,
                                 const void* residual, const void* weight, float eps, int rank, int world, int rows, int cols,
                                 int dtype, bool pushed, cudaStream_t stream);
int launch_allreduce_inprocess(const void* const* in_ptrs, void* const* out_ptrs, void* const* norm_ptrs, void* const* stage_ptrs,
                               size_t stage_bytes, void* const* flag_ptrs, const void* const* residual_ptrs, const void* weight,
                               float eps, int world, int rows, int cols, int dtype, bool pushed, cudaStream_t stream);
// One launch for a step that holds prefill sequences and decode sequences (prefill_attn_tc.cu), then the split merge.
bool mixed_step_supported(const PrefillArgs& p, const DecodeArgs& d);
int launch_mixed_step(const PrefillArgs& p, const DecodeArgs& d, int prefill_blocks);
// int8 KV cache (kv_int8.cu; tensor-core decode in decode_attn.cu)
int launch_store_int8(const void* key, const void* value, void* k_cache, void* v_cache, void* k_scale, void* v_scale,
                      const int32_t* slot_mapping, int64_t num_tokens, int num_kv_heads, int head_dim, int64_t cache_rows,
                      int dtype, cudaStream_t stream);
int launch_rowwise_decode_int8(const DecodeInt8Args& a);
bool decode_int8_mma_supported(const DecodeInt8Args& a);
int launch_decode_int8_mma(const DecodeInt8Args& a);
int launch_store_fp8(const void* key, const void* value, void* k_cache, void* v_cache, void* k_scale, void* v_scale,
                     const int32_t* slot_mapping, int64_t num_tokens, int num_kv_heads, int head_dim, int64_t cache_rows,
                     int dtype, cudaStream_t stream);
bool prefill_mma_supported(const PrefillArgs& a);
int launch_prefill_mma(const PrefillArgs& a);
bool prefill_takes_tiles(const PrefillArgs& a);   // launch_prefill_mma is quicker than launch_prefill_tc, by sizes that the host knows
int prefill_tile_status(cudaStream_t stream, int* status);
// tcgen05 / TMEM / TMA path (F16/BF16, head_dim 128, paged block_size % 128 == 0).
bool prefill_tc_supported(const PrefillArgs& a);
int launch_prefill_tc(const PrefillArgs& a);

// ---- device helpers --------------------------------------------------------------------------
#ifdef __CUDACC__

template <typename T> struct ElemTraits;
template <> struct ElemTraits<__nv_bfloat16> {
    static __device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 from_float(float v) { return __float2bfloat16_rn(v); }
    static __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
        __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&p);
    }
};
template <> struct ElemTraits<__half> {
    static __device__ __forceinline__ float to_float(__half v) { return __half2float(v); }
    static __device__ __forceinline__ __half from_float(float v) { return __float2half_rn(v); }
    static __device__ __forceinline__ uint32_t pack2(float lo, float hi) {
        __half2 p = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&p);
    }
};
template <> struct ElemTraits<float> {
    static __device__ __forceinline__ float to_float(float v) { return v; }
    static __device__ __forceinline__ float from_float(float v) { return v; }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16-byte asynchronous global->shared copy that bypasses L1; src_bytes == 0 zero-fills.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}

// D(16x8, f32) += A(16x16) * B(16x8); A row-major, B column-major fragments.
template <typename T>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                         uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                  uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 2^x, approximate (ex2.approx: 2 ulp, exp2(-inf) = +0).
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

constexpr float kLog2e = 1.4426950408889634f;

// The kernels are launched with the programmatic-stream-serialization attribute: a kernel's blocks may be scheduled while
// its predecessor in the stream still runs, wait here until that predecessor has completed and its writes are visible
// (before anything is read or written), and at once allow their own successor the same head start.  In a step of many short
// kernels this hides launch latency.
__device__ __forceinline__ void pdl_wait_then_release() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

// The same place of shared memory in block `rank` of the cluster.
__device__ __forceinline__ uint32_t in_block(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// `bytes` of this block's shared memory into that of block `rank`, counted on its barrier at `bar`.
__device__ __forceinline__ void push_bulk(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar, uint32_t rank) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(in_block(dst, rank)), "r"(src), "r"(bytes), "r"(in_block(bar, rank)) : "memory");
}

// For a kernel that needs nothing of the one launched just before it, which for its part waited (pdl_wait_then_release) before it let this one start:
// all that came earlier has completed, and the two run side by side.  It waits at its end instead, in every block, so that whatever follows it in the
// stream and waits for it has waited for both.
__device__ __forceinline__ void pdl_start_beside() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_beside() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// <<<grid, block, smem, stream>>> with that attribute.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

#endif  // __CUDACC__

}  // namespace nvk
