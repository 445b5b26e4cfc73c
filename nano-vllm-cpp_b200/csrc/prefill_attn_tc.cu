// Varlen causal prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA),
// F16 / BF16, head_dim 128, dense or paged keys (block_size a multiple of 128).
//
// Replaces the same reference code as prefill_attn.cu (src/kernels/attention.cu:114-302,
// src/kernels/flash_attn.cpp:203-300); prefill_attn.cu (mma.sync) takes small steps and what
// these kernels do not (cache blocks that are no multiple of 128, scales that are not positive).
//
// Two kernels live here, chosen by shape: the single-tile kernel described next (odd GQA group sizes) and the
// persistent head-pair kernel further down (even group sizes: the two query heads of a pair share their K / V tiles).
//
// Single-tile kernel: one thread block = 128 query rows of one (sequence, head); 128 threads, thread t owns row t.
//   * Q (128 x 128), K tile (128 keys x 128) and V tile live in shared memory as two 128-byte-wide
//     panels each, written by TMA with the 128-byte swizzle -- exactly the canonical layout the
//     UMMA shared-memory descriptors expect (Q, K: K-major; V: MN-major, so the row-major V tile
//     is consumed as it lies, no transpose).  Paged keys: one TMA box per tile, row coordinate
//     block_tables[seq][tile] * block_size; block ids outside the cache give an out-of-bounds
//     coordinate, which TMA fills with zeros.
//   * S = Q K^T : 8 x tcgen05.mma (M 128, N 128, K 16) issued by one thread, accumulator in TMEM
//     columns [0,128).  Each thread reads its own row of S with tcgen05.ld (no shuffles for the row
//     max / row sum), applies scale + causal mask, and writes P = exp2(s - m) as packed 16-bit pairs
//     back to TMEM columns [0,64) (aliasing S).
//   * O += P V : 8 x tcgen05.mma with A = P from TMEM and B = V from shared memory, accumulator in
//     TMEM columns [128,256).  O is only rescaled when the running maximum grows by more than 8
//     (log2 domain); otherwise the stale maximum keeps being used, which is exact after the final
//     division by the row sum.
//   * 256 TMEM columns and 96 KiB of shared memory per block: two blocks per SM, so one block's
//     softmax overlaps the other's MMAs.  Every mbarrier wait is bounded; on a time-out the block
//     raises an error word, stops waiting, gives what is under way time to land, frees its TMEM and returns.
//   * No cluster launch and no multicast anywhere.
#include "decode_body.cuh"

#include <cuda.h>

#include <cmath>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <utility>

namespace nvk {
namespace {

constexpr int kHeadDim = 128;
constexpr int kBM = 128, kBN = 128, kThreads = 128;
constexpr int kPanelBytes = 128 * 128;          // 128 rows x 64 elements (128 B)
constexpr int kTileBytes = 2 * kPanelBytes;     // 32 KiB
constexpr int kOffQ = 0, kOffK = kTileBytes, kOffV = 2 * kTileBytes, kOffBar = 3 * kTileBytes;
constexpr int kSmemBytes = kOffBar + 128 + 1024;  // + barriers + slack for 1024-byte alignment
constexpr int kTmemCols = 256;
constexpr float kRescaleThreshold = 8.0f;
constexpr long long kWaitCycles = 4000000000LL;  // ~2 s at 2 GHz

__device__ int g_tc_error = 0;

struct TcParams {
    IndexArray cu_q, cu_k, block_tables;
    void* out;
    int64_t num_seqs, total_q, total_k, max_blocks, key_rows, num_cache_blocks;
    int num_heads, num_kv_heads, block_size;
    float scale_log2;
    uint32_t idesc_s, idesc_pv;
};

// ---- PTX wrappers ---------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// Whether a phase has completed, without waiting for it.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: gives up after kWaitCycles or as soon as another thread of the block gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long start = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - start > kWaitCycles) {
            *abort_flag = 1;
            atomicCAS(&g_tc_error, 0, code);
            return false;
        }
    }
}
// Whole-warp wait: lane 0 polls, the result is broadcast (31 fewer spinning threads per warp).
__device__ __forceinline__ bool warp_mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, abort_flag, code) ? 1 : 0;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
// Whoever gives up a wait stays for 2 ms before it goes to the block's end: copies into shared memory and MMAs that read it may still be under way, and a wait
// for each would end with the same limit at the latest.  (In the roles and not behind them: a branch at the block's end, where tensor memory is
// freed, cost launches of 23 to 32 us 0.15 to 0.25 us, this 0.05 to 0.1.)
__device__ __forceinline__ void settle() {
    const long long start = clock64();
    while (clock64() - start < 4000000) {}
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// D(tmem) (+)= A(smem desc) * B(smem desc)
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
// D(tmem) (+)= A(tmem) * B(smem desc)
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
// For an issuing warp that stays converged: all lanes run through the same instructions, so that the descriptors live in uniform registers, which
// is where the MMA wants them, and one lane (`leader` 1) issues.  A single diverged lane has to move every operand there first: 75 to 100
// clocks an MMA, more than the tensor pipe needs for one.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t leader;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(leader));
    return leader;
}
template <bool ACC>
__device__ __forceinline__ void umma_ss_by(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %0, 0;\n\tsetp.ne.u32 p, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], %2, %3, %4, p;\n\t}\n"
        :: "r"(leader), "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0) : "memory");
}
__device__ __forceinline__ void umma_ts_by(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %0, 0;\n\tsetp.ne.u32 p, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], [%2], %3, %4, p;\n\t}\n"
        :: "r"(leader), "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_commit_by(uint32_t leader, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}\n" :: "r"(leader), "r"(bar) : "memory");
}
constexpr uint64_t kmajor_off16(int step) { return ((step / 4) * kPanelBytes + (step % 4) * 32) / 16; }
// The 8 K-steps of S = Q K^T (both operands K-major: two 64-element panels, 32 bytes per step inside a panel).
__device__ __forceinline__ void umma_scores(uint32_t leader, uint32_t d_tmem, uint64_t q_base, uint64_t k_base, uint32_t idesc) {
    umma_ss_by<false>(leader, d_tmem, q_base, k_base, idesc);
#pragma unroll
    for (int ks = 1; ks < 8; ++ks) umma_ss_by<true>(leader, d_tmem, q_base + kmajor_off16(ks), k_base + kmajor_off16(ks), idesc);
}
// K-steps FIRST .. LAST - 1 of O += P V: P in tensor memory (8 columns per 16 keys), V MN-major (2048 bytes per 16 keys).
template <int FIRST, int LAST>
__device__ __forceinline__ void umma_pv(uint32_t leader, uint32_t d_tmem, uint32_t p_tmem, uint64_t v_base, uint32_t idesc, uint32_t acc_first) {
#pragma unroll
    for (int kk = FIRST; kk < LAST; ++kk)
        umma_ts_by(leader, d_tmem, p_tmem + kk * 8, v_base + kk * 2048 / 16, idesc, kk > FIRST ? 1u : acc_first);
}

// These and the other `.sync.aligned` instructions want the whole warp at one place: what a single lane does before one goes by a predicate
// (mbar_arrive_if, *_by) or is followed by a warp barrier, a shuffle or a vote.  The waits for a whole warp are such: warp_mbar_wait ends with a shuffle,
// wait_bar_warp with a vote.
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n"
        ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
        ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}


// The TMEM loads are asynchronous: this pins the use of their results after the preceding
// tcgen05.wait::ld in program order (the compiler may not move register arithmetic across it).
__device__ __forceinline__ void reg_fence32(uint32_t (&r)[32]) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                      "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
    asm volatile("" : "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                      "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}

// sm_100 packed-pair and three-input float instructions: they halve the instruction count of the softmax
// passes, which with two resident warps per scheduler are bound by dependent-issue latency, not by lanes.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Maximum of 32 raw scores (keys key_base .. key_base + 31); MASK hides keys >= lim.
template <bool MASK>
__device__ __forceinline__ float chunk_max(const uint32_t (&r)[32], int key_base, int lim) {
    float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            v[u] = __uint_as_float(r[i + u]);
            if (MASK && key_base + i + u >= lim) v[u] = -INFINITY;
        }
        m0 = max3(m0, v[0], v[1]); m1 = max3(m1, v[2], v[3]); m2 = max3(m2, v[4], v[5]); m3 = max3(m3, v[6], v[7]);
    }
    return fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
}

// 32 scores -> 16 packed probability pairs exp2(s * scale - m); returns their fp32 sum.
template <typename T, bool MASK>
__device__ __forceinline__ float chunk_probs(const uint32_t (&r)[32], uint32_t (&pk)[16], int key_base, int lim,
                                             float scale_log2, float m_use) {
    const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2), neg_m2 = pack_f32x2(-m_use, -m_use);
    uint64_t acc0 = 0ull, acc1 = 0ull;   // two packed pairs of fp32 partial sums
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
        float s0 = __uint_as_float(r[2 * i]), s1 = __uint_as_float(r[2 * i + 1]);
        float s2 = __uint_as_float(r[2 * i + 2]), s3 = __uint_as_float(r[2 * i + 3]);
        if (MASK) {
            if (key_base + 2 * i >= lim) s0 = -INFINITY;
            if (key_base + 2 * i + 1 >= lim) s1 = -INFINITY;
            if (key_base + 2 * i + 2 >= lim) s2 = -INFINITY;
            if (key_base + 2 * i + 3 >= lim) s3 = -INFINITY;
        }
        float x0, x1, x2, x3;
        unpack_f32x2(fma_f32x2(pack_f32x2(s0, s1), scale2, neg_m2), x0, x1);
        unpack_f32x2(fma_f32x2(pack_f32x2(s2, s3), scale2, neg_m2), x2, x3);
        const float p0 = fast_exp2(x0), p1 = fast_exp2(x1), p2 = fast_exp2(x2), p3 = fast_exp2(x3);
        acc0 = add_f32x2(acc0, pack_f32x2(p0, p1));
        acc1 = add_f32x2(acc1, pack_f32x2(p2, p3));
        pk[i] = ElemTraits<T>::pack2(p0, p1);
        pk[i + 1] = ElemTraits<T>::pack2(p2, p3);
    }
    float a0, a1, a2, a3;
    unpack_f32x2(acc0, a0, a1);
    unpack_f32x2(acc1, a2, a3);
    return (a0 + a1) + (a2 + a3);
}
// The same in three stages over registers in place, for callers that interleave the stages of neighbouring chunks: x = s * scale - m,
// p = exp2(x), then sum and pack.
__device__ __forceinline__ float ex2_ordered(float x) {
    float y;
    asm volatile("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void scale_pair(uint32_t (&r)[32], int i, uint64_t scale2, uint64_t neg_m2) {
    uint64_t d;
    asm volatile("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(pack_f32x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]))), "l"(scale2), "l"(neg_m2));
    float a, b;
    unpack_f32x2(d, a, b);
    r[2 * i] = __float_as_uint(a);
    r[2 * i + 1] = __float_as_uint(b);
}
template <typename T>
__device__ __forceinline__ uint32_t sum_pair(const uint32_t (&r)[32], int i, uint64_t& acc) {
    const float a = __uint_as_float(r[2 * i]), b = __uint_as_float(r[2 * i + 1]);
    acc = add_f32x2(acc, pack_f32x2(a, b));
    return ElemTraits<T>::pack2(a, b);
}
// exp2 of chunk `cur`, between them the scaling of the next chunk and the sums of the previous one.  The exponentials are what a step
// spends most of its time on (two warps of a scheduler need 16 of its clocks per pair of elements), so the other work of a row is
// issued in their shadow instead of before and after them.  Measured, 2 x 8192 tokens: 1086 -> 1150 TFLOP/s; 16 x 2048: 813 -> 890.
// (A polynomial for one element in eight on the FMA pipe instead is slower, 1102: the step is not bound by the exponential unit alone.)
template <typename T, bool NEXT, bool PREV>
__device__ __forceinline__ void exp_stage(uint32_t (&cur)[32], uint32_t (&next)[32], const uint32_t (&prev)[32], uint32_t (&pk)[16], uint64_t scale2, uint64_t neg_m2, uint64_t& acc0, uint64_t& acc1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        cur[2 * i] = __float_as_uint(ex2_ordered(__uint_as_float(cur[2 * i])));
        if (NEXT) scale_pair(next, i, scale2, neg_m2);
        cur[2 * i + 1] = __float_as_uint(ex2_ordered(__uint_as_float(cur[2 * i + 1])));
        if (PREV) pk[i] = sum_pair<T>(prev, i, (i & 1) ? acc1 : acc0);
    }
}
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    const uint32_t lo = ((addr & 0x3FFFFu) >> 4) | ((lbo_bytes >> 4) << 16);
    const uint32_t hi = (sbo_bytes >> 4) | (1u << 14) | (2u << 29);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 2)
prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const TcParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ int s_info[4];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;

    const int tid = threadIdx.x, warp = tid >> 5;
    const int head = blockIdx.x;
    const int kvh = head * p.num_kv_heads / p.num_heads;
    pdl_wait_then_release();

    // (reversed) tile index -> (sequence, first query row): later tiles of a sequence see more keys
    if (tid == 0) {
        const int64_t want = static_cast<int64_t>(gridDim.y) - 1 - blockIdx.y;
        int64_t acc = 0;
        int found = -1, q0 = 0;
        if (p.cu_q == nullptr) {
            if (want * kBM < p.total_q) { found = 0; q0 = static_cast<int>(want * kBM); }
        } else {
            for (int64_t s = 0; s < p.num_seqs; ++s) {
                const int64_t tiles = (static_cast<int64_t>(p.cu_q[s + 1]) - p.cu_q[s] + kBM - 1) / kBM;
                if (want < acc + tiles) { found = static_cast<int>(s); q0 = static_cast<int>((want - acc) * kBM); break; }
                acc += tiles;
            }
        }
        s_info[0] = found; s_info[1] = q0;
        s_abort = 0;
    }
    __syncthreads();
    const int seq = s_info[0];
    if (seq < 0) return;
    const int q0 = s_info[1];
    int64_t qb, kb;
    int q_len, k_len;
    if (p.cu_q == nullptr) { qb = 0; kb = 0; q_len = static_cast<int>(p.total_q); k_len = static_cast<int>(p.total_k); }
    else {
        qb = p.cu_q[seq]; kb = p.cu_k[seq];
        q_len = p.cu_q[seq + 1] - static_cast<int>(qb); k_len = p.cu_k[seq + 1] - static_cast<int>(kb);
    }
    const int rows_here = min(kBM, q_len - q0);
    const int shift = k_len - q_len;
    int k_hi = shift + q0 + rows_here;
    if (k_hi > k_len) k_hi = k_len;
    const int num_kt = k_hi > 0 ? (k_hi + kBN - 1) / kBN : 0;

    T* out_row0 = static_cast<T*>(p.out) + (static_cast<size_t>(qb + q0) * p.num_heads + head) * kHeadDim;
    const size_t out_stride = static_cast<size_t>(p.num_heads) * kHeadDim;

    if (num_kt == 0) {   // no visible key for any row of this tile
        for (int i = tid; i < rows_here * (kHeadDim / 8); i += kThreads) {
            const int r = i / (kHeadDim / 8), c = i % (kHeadDim / 8);
            *reinterpret_cast<uint4*>(out_row0 + r * out_stride + c * 8) = make_uint4(0u, 0u, 0u, 0u);
        }
        return;
    }

    // shared memory carve-up (1024-byte aligned panels)
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t sm_q = smem_base + kOffQ, sm_k = smem_base + kOffK, sm_v = smem_base + kOffV;
    const uint32_t bar_q = smem_base + kOffBar, bar_k = bar_q + 8, bar_v = bar_q + 16, bar_s = bar_q + 24, bar_o = bar_q + 32;
    volatile int* abort_flag = &s_abort;

    if (tid == 0) {
        mbar_init(bar_q, 1); mbar_init(bar_k, 1); mbar_init(bar_v, 1); mbar_init(bar_s, 1); mbar_init(bar_o, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;
    const uint32_t t_s = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);   // this warp's lanes, S / P columns
    const uint32_t t_o = t_s + 128;                                               // O columns

    const IndexArray table = p.block_tables ? p.block_tables + static_cast<int64_t>(seq) * p.max_blocks : IndexArray();
    auto key_row = [&](int key0) -> int {   // row coordinate of a key tile; out-of-range ids -> zero-filled box
        if (table) {
            const int64_t id = table[key0 / p.block_size];
            if (id < 0 || id >= p.num_cache_blocks) return static_cast<int>(p.key_rows);
            return static_cast<int>(id) * p.block_size + key0 % p.block_size;
        }
        return static_cast<int>(kb) + key0;
    };

    if (tid == 0) {
        mbar_expect_tx(bar_q, kTileBytes);
        tma_load_3d(sm_q, &tm_q, 0, head, static_cast<int>(qb) + q0, bar_q);
        tma_load_3d(sm_q + kPanelBytes, &tm_q, 64, head, static_cast<int>(qb) + q0, bar_q);
        const int r0 = key_row(0);
        mbar_expect_tx(bar_k, kTileBytes);
        tma_load_3d(sm_k, &tm_k, 0, kvh, r0, bar_k);
        tma_load_3d(sm_k + kPanelBytes, &tm_k, 64, kvh, r0, bar_k);
        mbar_expect_tx(bar_v, kTileBytes);
        tma_load_3d(sm_v, &tm_v, 0, kvh, r0, bar_v);
        tma_load_3d(sm_v + kPanelBytes, &tm_v, 64, kvh, r0, bar_v);
    }

    const int lim = min(shift + q0 + tid + 1, k_len);   // this row sees keys [0, lim)
    float m_ref = -INFINITY, l_run = 0.0f;
    bool alive = true;

    for (int j = 0; j < num_kt && alive; ++j) {
        const int key0 = j * kBN;
        const uint32_t ph = j & 1;
        // ---- S = Q K^T ------------------------------------------------------------------------------
        if (tid == 0) {
            bool ok = true;
            if (j == 0) ok = mbar_wait(bar_q, 0, abort_flag, 1);
            ok = ok && mbar_wait(bar_k, ph, abort_flag, 2);
            if (ok) {
                tc_fence_after();
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) {
                    const uint32_t off = (ks >> 2) * kPanelBytes + (ks & 3) * 32;
                    umma_ss(tmem_base, make_smem_desc(sm_q + off, 16, 1024), make_smem_desc(sm_k + off, 16, 1024),
                            p.idesc_s, ks > 0 ? 1u : 0u);
                }
                tc_commit(bar_s);
            }
        }
        __syncwarp();
        alive = warp_mbar_wait(bar_s, ph, abort_flag, 3);
        if (!alive) break;
        tc_fence_after();
        // S_j done => PV_{j-1} done (MMAs retire in order): the K and V buffers are free again.
        if (tid == 0) {
            if (j + 1 < num_kt) {
                const int r = key_row(key0 + kBN);
                mbar_expect_tx(bar_k, kTileBytes);
                tma_load_3d(sm_k, &tm_k, 0, kvh, r, bar_k);
                tma_load_3d(sm_k + kPanelBytes, &tm_k, 64, kvh, r, bar_k);
            }
            if (j > 0) {
                const int r = key_row(key0);
                mbar_expect_tx(bar_v, kTileBytes);
                tma_load_3d(sm_v, &tm_v, 0, kvh, r, bar_v);
                tma_load_3d(sm_v + kPanelBytes, &tm_v, 64, kvh, r, bar_v);
            }
        }

        __syncwarp();   // lane 0 re-joins its warp before the warp-collective TMEM loads
        // ---- softmax: pass 1, row maximum (TMEM loads run one chunk ahead of the arithmetic) -----------
        const bool need_mask = key0 + kBN > min(shift + q0 + 1, k_len);   // block-uniform
        uint32_t ra[32], rb[32];
        float mx;
        tmem_ld32(t_s, ra);
        tc_wait_ld(); reg_fence32(ra);
        tmem_ld32(t_s + 32, rb);
        if (need_mask) {
            mx = chunk_max<true>(ra, key0, lim);
            tc_wait_ld(); reg_fence32(rb);
            tmem_ld32(t_s + 64, ra);
            mx = fmaxf(mx, chunk_max<true>(rb, key0 + 32, lim));
            tc_wait_ld(); reg_fence32(ra);
            tmem_ld32(t_s + 96, rb);
            mx = fmaxf(mx, chunk_max<true>(ra, key0 + 64, lim));
            tc_wait_ld(); reg_fence32(rb);
            mx = fmaxf(mx, chunk_max<true>(rb, key0 + 96, lim));
        } else {
            mx = chunk_max<false>(ra, 0, 0);
            tc_wait_ld(); reg_fence32(rb);
            tmem_ld32(t_s + 64, ra);
            mx = fmaxf(mx, chunk_max<false>(rb, 0, 0));
            tc_wait_ld(); reg_fence32(ra);
            tmem_ld32(t_s + 96, rb);
            mx = fmaxf(mx, chunk_max<false>(ra, 0, 0));
            tc_wait_ld(); reg_fence32(rb);
            mx = fmaxf(mx, chunk_max<false>(rb, 0, 0));
        }
        // start re-reading the scores for pass 2 while the maximum is settled
        tmem_ld32(t_s, ra);
        mx *= p.scale_log2;
        if (__any_sync(0xffffffffu, mx > m_ref + kRescaleThreshold)) {
            const float m_new = fmaxf(m_ref, mx);
            const float f = (m_new == -INFINITY) ? 1.0f : fast_exp2(m_ref - m_new);
            if (j > 0) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld32(t_o + c * 32, r);
                    tc_wait_ld(); reg_fence32(r);
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
                    tmem_st32(t_o + c * 32, r);
                }
            }
            l_run *= f;
            m_ref = m_new;
        }
        const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;

        // ---- softmax: pass 2, P = exp2(s * scale - m) as 16-bit pairs written over S -----------------------
        {
            uint32_t pk[16];
            tc_wait_ld(); reg_fence32(ra);
            tmem_ld32(t_s + 32, rb);
            l_run += need_mask ? chunk_probs<T, true>(ra, pk, key0, lim, p.scale_log2, m_use)
                               : chunk_probs<T, false>(ra, pk, 0, 0, p.scale_log2, m_use);
            tc_wait_ld(); reg_fence32(rb);        // chunk 1 is in registers: columns [0,16) may be overwritten
            tmem_st16(t_s, pk);
            tmem_ld32(t_s + 64, ra);
            l_run += need_mask ? chunk_probs<T, true>(rb, pk, key0 + 32, lim, p.scale_log2, m_use)
                               : chunk_probs<T, false>(rb, pk, 0, 0, p.scale_log2, m_use);
            tc_wait_ld(); reg_fence32(ra);
            tmem_st16(t_s + 16, pk);
            tmem_ld32(t_s + 96, rb);
            l_run += need_mask ? chunk_probs<T, true>(ra, pk, key0 + 64, lim, p.scale_log2, m_use)
                               : chunk_probs<T, false>(ra, pk, 0, 0, p.scale_log2, m_use);
            tc_wait_ld(); reg_fence32(rb);
            tmem_st16(t_s + 32, pk);
            l_run += need_mask ? chunk_probs<T, true>(rb, pk, key0 + 96, lim, p.scale_log2, m_use)
                               : chunk_probs<T, false>(rb, pk, 0, 0, p.scale_log2, m_use);
            tmem_st16(t_s + 48, pk);
        }
        tc_wait_st();

        // ---- last tile: rows of V past the sequence may hold anything; zero them (0 * NaN = NaN) ---------
        if (key0 + kBN > k_len) {
            alive = warp_mbar_wait(bar_v, ph, abort_flag, 4);
            if (alive) {
                const int first_bad = k_len - key0;   // in (0, 128)
                for (int i = tid; i < (kBN - first_bad) * 16; i += kThreads) {
                    const int r = first_bad + i / 16, c16 = i % 16;
                    *reinterpret_cast<uint4*>(smem_gen + kOffV + (c16 >> 3) * kPanelBytes + r * 128 + (c16 & 7) * 16) =
                        make_uint4(0u, 0u, 0u, 0u);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            }
        }
        tc_fence_before();
        __syncthreads();

        // ---- O += P V ---------------------------------------------------------------------------------
        if (tid == 0 && !*abort_flag) {
            if (mbar_wait(bar_v, ph, abort_flag, 5)) {
                tc_fence_after();
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    umma_ts(tmem_base + 128, tmem_base + kk * 8, make_smem_desc(sm_v + kk * 2048, kPanelBytes, 1024),
                            p.idesc_pv, (j > 0 || kk > 0) ? 1u : 0u);
                }
                tc_commit(bar_o);
            }
        }
    }

    // ---- epilogue ----------------------------------------------------------------------------------------
    __syncwarp();
    if (alive) alive = warp_mbar_wait(bar_o, (num_kt - 1) & 1, abort_flag, 6);
    tc_fence_after();
    if (alive && !*abort_flag) {
        // every thread owns a full row: the row sum needs no cross-lane reduction
        const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
        unsigned char* stage = smem_gen + kOffQ;   // Q is dead after the last S MMA
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32(t_o + c * 32, r);
            tc_wait_ld(); reg_fence32(r);
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
                uint4 v;
                v.x = ElemTraits<T>::pack2(__uint_as_float(r[q4 * 8 + 0]) * inv, __uint_as_float(r[q4 * 8 + 1]) * inv);
                v.y = ElemTraits<T>::pack2(__uint_as_float(r[q4 * 8 + 2]) * inv, __uint_as_float(r[q4 * 8 + 3]) * inv);
                v.z = ElemTraits<T>::pack2(__uint_as_float(r[q4 * 8 + 4]) * inv, __uint_as_float(r[q4 * 8 + 5]) * inv);
                v.w = ElemTraits<T>::pack2(__uint_as_float(r[q4 * 8 + 6]) * inv, __uint_as_float(r[q4 * 8 + 7]) * inv);
                const int chunk = c * 4 + q4;
                *reinterpret_cast<uint4*>(stage + tid * 256 + ((chunk ^ (tid & 15)) << 4)) = v;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (alive && !*abort_flag) {
        unsigned char* stage = smem_gen + kOffQ;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int idx = i * kThreads + tid;
            const int r = idx >> 4, chunk = idx & 15;
            if (r < rows_here) {
                const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 256 + ((chunk ^ (r & 15)) << 4));
                *reinterpret_cast<uint4*>(out_row0 + r * out_stride + chunk * 8) = v;
            }
        }
    }
    if (!alive) settle();
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

constexpr int kTmemCols2 = 512;   // head-pair kernels: S0 S1 O0 O1

__device__ __forceinline__ void mbar_arrive_if(bool one, uint32_t bar) {   // by a predicate, without a branch
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %1, 0;\n\t@q mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}\n" ::"r"(bar), "r"(static_cast<int>(one)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

// =================================================================================================
// Shared memory of the persistent kernel: two Q tiles, a ring of four 32 KiB stages that K and V tiles go through in the order of
// their use, and 4 KiB for each softmax warp's output.  Tensor memory: S0 S1 O0 O1, 128 columns each; a tile's probabilities lie in the first 64 columns of its scores.
// =================================================================================================
constexpr int kRing5 = 4;
constexpr int kOff4Q = 0, kOff4Ring = 2 * kTileBytes, kOff4Out = (2 + kRing5) * kTileBytes, kOff4Bar = kOff4Out + kTileBytes;
constexpr int kSmemBytes4 = kOff4Bar + 256 + 1024;

// Bounded waits of the persistent kernel, by one thread and by a whole warp (the same answer for all its lanes): they give up after 2 to 4 seconds
// or as soon as another thread of the block gave up.  They are inlined at some twenty places, so that their size counts: the block leaves
// its first error in shared memory and reports it once, at its end.
__device__ __forceinline__ uint32_t clock_hi() {   // in units of 2^32 clocks
    uint32_t c;
    asm volatile("mov.u32 %0, %%clock_hi;" : "=r"(c));
    return c;
}
template <bool WARP>
__device__ __forceinline__ bool wait_bar_as(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    auto all = [](bool v) { return WARP ? __all_sync(0xffffffffu, v) != 0 : v; };
    if (all(mbar_try_wait(bar, parity) != 0)) return true;
    const uint32_t start = clock_hi();
    while (!all(mbar_try_wait(bar, parity) != 0)) {
        if (!all(*abort_flag == 0 && clock_hi() - start <= 1u)) {
            if (*abort_flag == 0) *abort_flag = code;
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    return wait_bar_as<false>(bar, parity, abort_flag, code);
}
__device__ __forceinline__ bool wait_bar_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    return wait_bar_as<true>(bar, parity, abort_flag, code);
}

// Raw scores of keys 32 c .. 32 c + 31 of a tile: those from `seen` (keys of the tile that the row sees) on get no weight.  Chunks that the whole warp
// sees are left alone.
template <int C>
__device__ __forceinline__ void hide_chunk(uint32_t (&r)[32], int seen) {
    if (__all_sync(0xffffffffu, seen >= 32 * C + 32)) return;
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = seen > 32 * C + i ? r[i] : 0xff800000u;   // -infinity (the scale is positive)
}

// One online-softmax step of a row: 128 scores (columns of t_s) -> probabilities (16-bit pairs, the first 64 columns of t_s).  All scores are read
// before the first probability is written.  `seen`: keys of the tile that the row sees; `masked`: some row of the warp does not see
// all; `half`: no row of the item sees more than 64, the second half of the probabilities is not wanted.  `on_half` runs when the first 96 are
// written (64 of a half round): their MMAs run under the last exponentials, and two K-steps are left for the chain.
template <typename T, typename OnHalf>
__device__ __forceinline__ void softmax_row(uint32_t t_s, uint32_t t_o, bool masked, int seen, bool half, float scale_log2, bool first,
                                            float& m_ref, float& l_run, OnHalf on_half) {
    uint32_t r0[32], r1[32], r2[32], r3[32];
    tmem_ld32(t_s, r0);
    tmem_ld32(t_s + 32, r1);
    tmem_ld32(t_s + 64, r2);
    tmem_ld32(t_s + 96, r3);
    tc_wait_ld();
    reg_fence32(r0); reg_fence32(r1); reg_fence32(r2); reg_fence32(r3);
    if (masked) {
        hide_chunk<0>(r0, seen); hide_chunk<1>(r1, seen);
        if (!half) { hide_chunk<2>(r2, seen); hide_chunk<3>(r3, seen); }
    }
    float mx = fmaxf(chunk_max<false>(r0, 0, 0), chunk_max<false>(r1, 0, 0));
    if (!half) mx = fmaxf(mx, fmaxf(chunk_max<false>(r2, 0, 0), chunk_max<false>(r3, 0, 0)));
    mx *= scale_log2;
    if (__any_sync(0xffffffffu, mx > m_ref + kRescaleThreshold)) {
        const float m_new = fmaxf(m_ref, mx);
        const float f = (m_new == -INFINITY) ? 1.0f : fast_exp2(m_ref - m_new);
        if (!first) {
            // (the previous P.V was issued before these scores by the same thread: it is complete)
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                uint32_t r[32];
                tmem_ld32(t_o + c * 32, r);
                tc_wait_ld(); reg_fence32(r);
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
                tmem_st32(t_o + c * 32, r);
            }
        }
        l_run *= f;
        m_ref = m_new;
    }
    const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;
    const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2), neg_m2 = pack_f32x2(-m_use, -m_use);
    uint64_t acc0 = 0ull, acc1 = 0ull;
    uint32_t pk[16], pk2[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) scale_pair(r0, i, scale2, neg_m2);
    exp_stage<T, true, false>(r0, r1, r0, pk, scale2, neg_m2, acc0, acc1);
    exp_stage<T, true, true>(r1, r2, r0, pk, scale2, neg_m2, acc0, acc1);
    tmem_st16(t_s, pk);
    if (half) {
#pragma unroll
        for (int i = 0; i < 16; ++i) pk2[i] = sum_pair<T>(r1, i, (i & 1) ? acc1 : acc0);
        tmem_st16(t_s + 16, pk2);
        on_half();
    } else {
        exp_stage<T, true, true>(r2, r3, r1, pk2, scale2, neg_m2, acc0, acc1);
        tmem_st16(t_s + 16, pk2);
        // the last 32: 96 keys' probabilities are handed over before the last 16 exponentials
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            r3[2 * i] = __float_as_uint(ex2_ordered(__uint_as_float(r3[2 * i])));
            pk[2 * i] = sum_pair<T>(r2, 2 * i, acc0);
            r3[2 * i + 1] = __float_as_uint(ex2_ordered(__uint_as_float(r3[2 * i + 1])));
            pk[2 * i + 1] = sum_pair<T>(r2, 2 * i + 1, acc1);
        }
        tmem_st16(t_s + 32, pk);
        on_half();
#pragma unroll
        for (int i = 8; i < 16; ++i) {
            r3[2 * i] = __float_as_uint(ex2_ordered(__uint_as_float(r3[2 * i])));
            r3[2 * i + 1] = __float_as_uint(ex2_ordered(__uint_as_float(r3[2 * i + 1])));
            pk2[i - 8] = sum_pair<T>(r3, i - 8, (i & 1) ? acc1 : acc0);
        }
#pragma unroll
        for (int i = 8; i < 16; ++i) pk2[i] = sum_pair<T>(r3, i, (i & 1) ? acc1 : acc0);
        tmem_st16(t_s + 48, pk2);
    }
    float a0, a1, a2, a3;
    unpack_f32x2(acc0, a0, a1);
    unpack_f32x2(acc1, a2, a3);
    l_run += (a0 + a1) + (a2 + a3);
}

// =================================================================================================
// The persistent head-pair kernel.  An item is one stretch of query rows x the heads of two tiles, all of one KV head, so that a K / V tile is loaded
// once for both.  One block per SM takes items from a ticket counter and keeps TMEM, barriers and the warp roles alive across items.  Per 128-key
// round and tile: S = Q K^T (SS MMA), softmax by one warpgroup (thread = row), P over the first half of its scores in tensor memory, O += P V (TS MMA).
//
// What bounds it is the chain of a tile's round, S -> softmax -> P.V -> next S, with two tiles taking turns: one tile's softmax runs under the other
// tile's MMAs.  MMAs need 2048 clocks a round and exponentials as many.  What made the chain long was not arithmetic but how fast the code runs
// (clocks a round, one item alone; us for 2 x 8192 / 16 x 2048 / 32 x 512 / 24 x 310 tokens, 32 / 8 heads):
//   3600; 958 / 618 / 160 / 89     P through shared memory, one diverged lane issuing the MMAs of a tile, 126 KB of code
//   4060; 984 / 565 / 114 / 57     P in tensor memory, K and V in a ring of five stages, half of the code (short waits, one mask pass, one copy of
//                                  each role's body): roles that alternate over more code than the instruction caches hold wait for it, a
//                                  masked round took 9000 clocks where a steady one took 2600
//   3043; 832 / 498 / 101 / 50     the issuing warp converged, descriptors in uniform registers (umma_ss_by)
//   3002; 805 / 472 / 94 / 47      outputs in whole lines through 32 KB of shared memory (four stages are enough), masks by one compare a score
//   2990; 805 / 470 / 93 / 46      96 of 128 keys' probabilities handed over early, no spills in the third warpgroup
// Not here: the first 32 keys' maximum as reference with the row sum as check (no maxima at all, but nothing can be handed to the MMAs before the
// end: 3307); maxima in the shadow of the exponentials (3427); tickets taken by a warp of its own two items ahead (uneven ends: one prompt of
// 8192 tokens, 16 / 8 heads, 217 -> 255 us).  Steps of 64 keys would need 2560 clocks of MMAs: at N 64 they are bound by shared memory.
// Tiles of 128 >> head_shift query rows x 1 << head_shift heads instead of 128 rows of one head lose less on ragged ends and on the diagonal, and an item
// whose rows see at most half of their last key tile leaves out that tile's second half.  All barrier phases are counted cumulatively over items.
// =================================================================================================
// Ticket counters.  Launches that run at the same time must not share one: each would leave out items that the other took.  An eager launch takes
// the next of 32768, far more launches than streams hold in their queues; a captured one keeps its counter for all replays of its graph,
// so these have 32768 of their own, which no eager launch meets.
constexpr int kEagerSlots = 32768, kTicketSlots = 2 * kEagerSlots;
constexpr int kThreads5 = 384;      // three warpgroups (register reallocation works on whole warpgroups)
constexpr int kRegsLow5 = 88;       // registers per thread of the third warpgroup after setmaxnreg.dec
constexpr int kRegsHigh5 = 208;     // registers per thread of the two softmax warpgroups after setmaxnreg.inc
// Ticket counters, zero between launches: every block takes tickets up to its first one past the end (items + blocks in all, whether the first ones
// come from the counter or are the blocks' numbers), so the launch's last ticket is known, and who holds it sets the counter back.  (A counter of finished blocks is a trip to memory at the end that everything waits for: 1 us.)
__device__ unsigned int g_prefill_ticket[kTicketSlots];

struct Tc5Params {
    TcParams base;
    int head_shift;       // a tile's 128 rows are 128 >> head_shift query rows x 1 << head_shift heads
    int pairs;            // pairs of tiles that make up all heads
    int tiles;            // upper bound of query tiles over all sequences
    unsigned int total;   // pairs * tiles
    int slot;             // ticket counter of this launch
};

// One (query tile, pair of head sets), with all that the roles need to know of it, so that none of them reads the sequence bounds again.
struct Tc5Item {
    int kind;             // 1 = work, 0 = no more work
    int seq, pair;
    int q_row, rows;      // first query row and the rows there are
    int lim0, k_len;      // query row r sees keys [0, min(lim0 + r, k_len))
    int num_kt, last_partial;
    int half;             // no row sees more than 64 keys of the last tile
    int k_row;            // row of the sequence's first key (keys without a block table)
};

// Row of key `key0` of a sequence in the K / V tensors; key_rows (past the end: the copy fills zeros) for an invalid block.
__device__ __forceinline__ int tc5_key_row(const TcParams& p, int seq, int k_row, int key0) {
    if (!p.block_tables) return k_row + key0;
    const int64_t id = p.block_tables[static_cast<int64_t>(seq) * p.max_blocks + key0 / p.block_size];
    if (id < 0 || id >= p.num_cache_blocks) return static_cast<int>(p.key_rows);
    return static_cast<int>(id) * p.block_size + key0 % p.block_size;
}

// Finds the sequence of a query tile.  One warp holds a window of 32 sequences, one per lane, and moves it as the tiles it is asked
// for descend: a look-up is one ballot, and the bounds are loaded once per window.  (One lane walking the sequences one dependent
// load after the other took 5 to 7 thousand clocks an item with 16 to 32 sequences, more than an item of short sequences lasts:
// 64 x 256 tokens 191 -> 130 us, 32 x 512 182 -> 169, 16 x 2048 620 -> 605.)
struct Tc5Finder {
    int base, before, sum;     // first sequence of the window, tiles before it, tiles in it
    int mine;                  // tiles of the window before this lane's sequence
    int tiles, qb, qe, kb, ke; // of this lane's sequence

    __device__ __forceinline__ void load(const TcParams& p, int head_shift, int lane) {
        qb = 0; qe = 0; kb = 0; ke = 0;
        if (p.cu_q == nullptr) {
            if (lane == 0) { qe = static_cast<int>(p.total_q); ke = static_cast<int>(p.total_k); }
        } else if (base + lane < p.num_seqs) {
            // (the low words: the bounds are below 2^31, and both widths take one load without a branch)
            const int *q = static_cast<const int*>(p.cu_q.ptr) + (static_cast<size_t>(base + lane) << p.cu_q.wide);
            const int *k = static_cast<const int*>(p.cu_k.ptr) + (static_cast<size_t>(base + lane) << p.cu_k.wide);
            qb = q[0]; qe = q[1 << p.cu_q.wide];
            kb = k[0]; ke = k[1 << p.cu_k.wide];
        }
        tiles = max((qe - qb + (kBM >> head_shift) - 1) >> (7 - head_shift), 0);
        int inc = tiles;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int up = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += up;
        }
        mine = inc - tiles;
        sum = __shfl_sync(0xffffffffu, inc, 31);
    }
    // Opens on the last window (the first tile asked for is the last one) and returns the number of tiles of all sequences.
    __device__ __forceinline__ int open(const TcParams& p, int head_shift, int lane) {
        before = 0;
#pragma unroll 1
        for (base = 0;; base += 32, before += sum) {
            load(p, head_shift, lane);
            if (p.cu_q == nullptr || base + 32 >= p.num_seqs) return before + sum;
        }
    }
    // Tile number `want`, in [0, open()): its item, without the pair.
    __device__ __forceinline__ void find(const TcParams& p, int head_shift, int lane, int want, Tc5Item& it) {
#pragma unroll 1
        while (want < before) { base -= 32; load(p, head_shift, lane); before -= sum; }
        const int at = 31 - __clz(__ballot_sync(0xffffffffu, before + mine <= want && tiles > 0));
        const int q0 = (want - before - __shfl_sync(0xffffffffu, mine, at)) << (7 - head_shift);
        const int q_begin = __shfl_sync(0xffffffffu, qb, at), q_len = __shfl_sync(0xffffffffu, qe, at) - q_begin;
        it.seq = base + at;
        it.q_row = q_begin + q0;
        it.rows = min(kBM >> head_shift, q_len - q0);
        it.k_row = __shfl_sync(0xffffffffu, kb, at);
        it.k_len = __shfl_sync(0xffffffffu, ke, at) - it.k_row;
        it.lim0 = it.k_len - q_len + q0 + 1;
        const int k_hi = min(it.lim0 + it.rows - 1, it.k_len);
        it.num_kt = k_hi > 0 ? (k_hi + kBN - 1) / kBN : 0;
        it.last_partial = it.num_kt * kBN > it.k_len ? it.num_kt - 1 : -1;
        it.half = k_hi <= it.num_kt * kBN - kBN / 2 ? 1 : 0;
    }
};


// The decode half of a mixed step (prefill_tc5_kernel<T, true>): the (KV head, split, sequence) items of the decode kernels, taken
// from a second ticket counter by the same persistent blocks.  A block runs the two halves one after the other -- blocks
// [0, prefill_blocks) the prefill items first, the others the decode items first -- so while some SMs are busy on the tensor pipe
// the rest stream the KV cache, and no SM idles between the two parts of the step as it does at the boundary of two launches.  In
// the decode half the eight softmax warps form two groups of four warps, each with its own part of the block's shared memory: what
// two resident blocks of decode_split_kernel have per SM.
struct MixedDecode {
    dec::DecodeParams dp;
    int prefill_blocks;
};
__device__ unsigned int g_decode_ticket[kTicketSlots];

template <typename T, bool MIXED>
__global__ void __launch_bounds__(kThreads5, 1)
prefill_tc5_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const Tc5Params pp, const __grid_constant__ MixedDecode md) {
    using Decode16 = dec::Cache16<T>;
    struct MixedGroup {
        dec::GroupSmem<Decode16> g;
        unsigned int item;
    };
    static_assert(Decode16::kGroups * sizeof(MixedGroup) <= kOff4Bar, "the decode half's shared memory");
    const TcParams& p = pp.base;
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    __shared__ Tc5Item s_ring[4];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // (uniform, also to the compiler)
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    auto decode_half = [&]() {
        if (MIXED && warp < Decode16::kGroups * dec::kGroupWarps) {
            const dec::DecodeParams& dp = md.dp;
            MixedGroup& sm = reinterpret_cast<MixedGroup*>(smem_gen)[warp / dec::kGroupWarps];
            const int gtid = tid % dec::kGroupThreads, bar = 1 + warp / dec::kGroupWarps;
            const unsigned int hkv = static_cast<unsigned int>(dp.num_kv_heads), splits = static_cast<unsigned int>(dp.num_splits);
            while (true) {
                if (gtid == 0) sm.item = atomicAdd(&g_decode_ticket[pp.slot], 1u);
                dec::group_sync(bar, dec::kGroupThreads);
                const unsigned int item = sm.item;
                dec::group_sync(bar, dec::kGroupThreads);   // everyone holds the item before the next ticket overwrites it
                const unsigned int total = hkv * splits * static_cast<unsigned int>(dp.batch);
                if (item >= total) {
                    if (gtid == 0 && item == total + Decode16::kGroups * gridDim.x - 1) g_decode_ticket[pp.slot] = 0u;
                    break;
                }
                dec::run_split<Decode16, T>(dp, static_cast<int>(item / (hkv * splits)), static_cast<int>(item % hkv), static_cast<int>((item / hkv) % splits),
                                            sm.g, gtid, bar);
                dec::group_sync(bar, dec::kGroupThreads);   // the group's shared memory is free for its next item
            }
        }
    };
    const bool decode_first = MIXED && static_cast<int>(blockIdx.x) >= md.prefill_blocks;
    if (MIXED) pdl_wait_then_release();
    if (decode_first) {
        decode_half();
        // the prefill half's bulk copies write the shared memory that the decode half has read and written
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
    }
    const uint32_t sm_q = smem_base + kOff4Q, sm_ring = smem_base + kOff4Ring;
    const uint32_t bars = smem_base + kOff4Bar;
    const uint32_t bar_qfull = bars, bar_qempty = bars + 8;
    auto bar_full = [&](int s) { return bars + 16 + 8 * s; };      // ring stage s has landed
    auto bar_empty = [&](int s) { return bars + 56 + 8 * s; };     // and has been read by both tiles' MMAs
    auto bar_sfull = [&](int t) { return bars + 96 + 8 * t; };     // scores of a tile (and its P.V before that) complete
    auto bar_phalf = [&](int t) { return bars + 112 + 8 * t; };    // first 96 keys' probabilities of a tile in tensor memory (64 in a half round)
    auto bar_pfull = [&](int t) { return bars + 128 + 8 * t; };    // all of them
    auto bar_ofinal = [&](int t) { return bars + 144 + 8 * t; };   // an item's last P.V of a tile complete
    auto bar_item = [&](int s) { return bars + 160 + 8 * s; };     // ring entry s published
    volatile int* abort_flag = &s_abort;

    if (tid == 0) {
        s_abort = 0;
        mbar_init(bar_qfull, 1); mbar_init(bar_qempty, 1);
        for (int i = 0; i < kRing5; ++i) { mbar_init(bar_full(i), 1); mbar_init(bar_empty(i), 1); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_sfull(i), 1); mbar_init(bar_phalf(i), 4); mbar_init(bar_pfull(i), 4); mbar_init(bar_ofinal(i), 1);
        }
        for (int i = 0; i < 4; ++i) mbar_init(bar_item(i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncwarp();
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem_base)), "r"(kTmemCols2) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) { prefetch_map(&tm_q); prefetch_map(&tm_k); prefetch_map(&tm_v); }
    if (!MIXED) pdl_wait_then_release();   // barriers, TMEM and tensor maps are set up under the predecessor's tail
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, s_tmem_base, 0);
    const size_t out_stride = static_cast<size_t>(p.num_heads) * kHeadDim;

    // Three warpgroups: 0 and 1 are the softmax warps of tile 0 and 1, 2 holds the issuer, the producer and two idle
    // warps.  The block starts with 168 registers per thread (the cap of 384 threads); the third warpgroup hands
    // half of its registers back and the softmax warpgroups grow to 208, which holds a whole 128-key score row, its
    // probabilities and the step's state without spilling.  (56 and 224 spill in the producer: 24 x 310 tokens 46.4 us, 46.0.)

    if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kRegsLow5));
    if (warp == 9) {
        // ------------------------------------------------------------------ ticket taker + TMA producer
        const int item_heads = 2 << pp.head_shift;
        // A block's first ticket is its own number (a trip to memory less before its first item: 77 tokens on a prefix of 512 14.2 -> 14.0 us, 3 x 40 on
        // 256 10.7 -> 10.4), the counter's come behind those.  In a mixed step the
        // blocks come to their prefill items one after the other and take all from the counter.
        auto take_ticket = [&]() { return atomicAdd(&g_prefill_ticket[pp.slot], 1u) + (MIXED ? 0u : gridDim.x); };
        unsigned int ticket = blockIdx.x;
        if (MIXED && lane == 0) ticket = take_ticket();   // (under the look at the sequence bounds)
        Tc5Finder find;
        const int tiles = min(find.open(p, pp.head_shift, lane), pp.tiles);
        const unsigned int total = static_cast<unsigned int>(tiles) * static_cast<unsigned int>(pp.pairs);
        int stage = 0, n = -1;   // ring stage of the next K / V tile; the item that is being loaded, -1: none yet
        uint32_t turn = 0;       // parity of that stage's round through the ring
        int row = 0, next_row = 0, kvh = 0;
        bool ok = true;
        auto load = [&](const CUtensorMap* map, int r) {   // lane 0: the next K or V tile
            ok = ok && wait_bar(bar_empty(stage), turn ^ 1u, abort_flag, 11);   // (passes at once the first time round)
            if (!ok) return;
            const uint32_t dst = sm_ring + stage * kTileBytes, bar = bar_full(stage);
            mbar_expect_tx(bar, kTileBytes);
            tma_load_3d(dst, map, 0, kvh, r, bar);
            tma_load_3d(dst + kPanelBytes, map, 64, kvh, r, bar);
            if (++stage == kRing5) { stage = 0; turn ^= 1u; }
        };
        Tc5Item it{};
        // Item n is published, its first tiles are under way: take the next ticket under its rounds, then see to the rest of its tiles.  Where a wait
        // gave up nothing is published any more, but the tickets are still taken to the end.
        while (true) {
            Tc5Item next{};
            while (true) {
                ticket = __shfl_sync(0xffffffffu, ticket, 0);
                if (ticket >= total) {
                    if (lane == 0 && ticket == total + gridDim.x - 1) g_prefill_ticket[pp.slot] = 0u;
                    break;
                }
                const unsigned int tile = ticket / static_cast<unsigned int>(pp.pairs);
                next.pair = static_cast<int>(ticket - tile * static_cast<unsigned int>(pp.pairs));
                find.find(p, pp.head_shift, lane, tiles - 1 - static_cast<int>(tile), next);
                if (next.num_kt > 0) { next.kind = 1; break; }
                // rows that see no key: zeros, and the next ticket
                T* o0 = static_cast<T*>(p.out) + (static_cast<size_t>(next.q_row) * p.num_heads + item_heads * next.pair) * kHeadDim;
#pragma unroll 1
                for (int r = 0; r < next.rows; ++r)
#pragma unroll 1
                    for (int c = lane; c < item_heads * (kHeadDim / 8); c += 32) *reinterpret_cast<uint4*>(o0 + r * out_stride + c * 8) = make_uint4(0u, 0u, 0u, 0u);
                if (lane == 0) ticket = take_ticket();
            }
            int first_row = 0;   // rows of its first two key tiles, both trips at once
            if (next.kind != 0 && lane < 2 && lane < next.num_kt) first_row = tc5_key_row(p, next.seq, next.k_row, lane * kBN);
            if (n >= 0 && lane == 0) {
#pragma unroll 1
                for (int j = 1; j < it.num_kt; ++j) {
                    row = next_row;
                    if (j + 1 < it.num_kt) next_row = tc5_key_row(p, it.seq, it.k_row, (j + 1) * kBN);   // (a block's id is read a round before its copy)
                    load(&tm_k, row);
                    load(&tm_v, row);
                }
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            it = next;
            ++n;
            row = first_row;
            next_row = __shfl_sync(0xffffffffu, first_row, 1);
            if (lane == 0 && ok) {
                s_ring[n & 3] = it;
                mbar_arrive(bar_item(n & 3));   // release: the entry is visible to whoever waits on the barrier
            }
            if (it.kind == 0) {
                if (!ok) settle();
                break;
            }
            if (lane == 0) {
                const int head0 = item_heads * it.pair;
                kvh = head0 * p.num_kv_heads / p.num_heads;
                load(&tm_k, row);
                if (n >= 1) ok = ok && wait_bar(bar_qempty, (n - 1) & 1, abort_flag, 14);   // previous item's score MMAs are done with Q
                if (ok) {
                    mbar_expect_tx(bar_qfull, 2 * kTileBytes);
#pragma unroll 1
                    for (int t = 0; t < 2; ++t) {
                        const int head = head0 + (t << pp.head_shift);
                        tma_load_3d(sm_q + t * kTileBytes, &tm_q, 0, head, it.q_row, bar_qfull);
                        tma_load_3d(sm_q + t * kTileBytes + kPanelBytes, &tm_q, 64, head, it.q_row, bar_qfull);
                    }
                }
                load(&tm_v, row);
                ticket = take_ticket();
            }
        }
    } else if (warp == 8) {
        // ------------------------------------------------------------------ MMA issuer, one for both tiles: P.V of a tile and then
        // its next scores, then the same of the other tile, so that one tile's softmax runs under the other tile's MMAs.
        {
            const uint32_t leader = elect_one();
            const uint64_t dq0 = make_smem_desc(sm_q, 16, 1024);
            const uint64_t dk0 = make_smem_desc(sm_ring, 16, 1024), dv0 = make_smem_desc(sm_ring, kPanelBytes, 1024);
            constexpr uint64_t kTile16 = kTileBytes / 16;   // (only moves the descriptor's start address, never carrying out of it)
            int ks = 0, vs = 1;           // ring stages of the next K and V tile, parities of their rounds through the ring
            uint32_t kturn = 0, vturn = 0;
            auto advance = [](int& s, uint32_t& turn) { s += 2; if (s >= kRing5) { s -= kRing5; turn ^= 1u; } };
            int n = -1, G = 0;            // the item whose P.V is next, and the rounds before this one; -1: only scores
            int j = 0, num_kt = 1, half = 0;   // its round, its rounds, whether the last one has keys in its first half only
            int next_kt = 0, next_half = 0;
            bool ok = true, more = true;
            while (ok && more) {
                const bool last = j + 1 == num_kt;
                int scores = 0;           // tiles whose scores of the following round are issued
                bool there = false;       // that round's operands have landed
                if (n >= 0) ok = wait_bar_warp(bar_full(vs), vturn, abort_flag, 23);
#pragma unroll 1
                for (int t = 0; t < 2 && ok; ++t) {
                    if (n >= 0) {
                        const uint64_t dv = dv0 + vs * kTile16;
                        const uint32_t t_s = tmem_base + t * 128, t_o = tmem_base + 256 + t * 128;
                        // (an item's first round: the probabilities also say that the previous item's output has left tensor memory)
                        ok = wait_bar_warp(bar_phalf(t), G & 1, abort_flag, 25);
                        if (!ok) break;
                        tc_fence_after();
                        umma_pv<0, 4>(leader, t_o, t_s, dv, p.idesc_pv, j > 0 ? 1u : 0u);
                        if (!(last && half)) umma_pv<4, 6>(leader, t_o, t_s, dv, p.idesc_pv, 1u);
                        ok = wait_bar_warp(bar_pfull(t), G & 1, abort_flag, 27);
                        if (!ok) break;
                        if (!(last && half)) {
                            tc_fence_after();
                            umma_pv<6, 8>(leader, t_o, t_s, dv, p.idesc_pv, 1u);
                        }
                        if (t == 1) tc_commit_by(leader, bar_empty(vs));
                        if (last) tc_commit_by(leader, bar_ofinal(t));
                    }
                    if (!there && more) {
                        // The next round's K tile; of the next item also what there is and Q.  Tile 0 does not wait for these: this item's other
                        // tile comes first then.
                        const uint32_t item = bar_item((n + 1) & 3), turn_i = ((n + 1) >> 2) & 1;
                        if (!last) {
                            ok = wait_bar_warp(bar_full(ks), kturn, abort_flag, 26);
                        } else {
                            if (t == 0 && !__all_sync(0xffffffffu, mbar_test(item, turn_i) && mbar_test(bar_qfull, (n + 1) & 1) && mbar_test(bar_full(ks), kturn))) continue;
                            ok = wait_bar_warp(item, turn_i, abort_flag, 29);
                            if (!ok) break;
                            const Tc5Item& it = s_ring[(n + 1) & 3];
                            more = __shfl_sync(0xffffffffu, it.kind, 0) != 0;
                            if (!more) continue;
                            next_kt = __shfl_sync(0xffffffffu, it.num_kt, 0);
                            next_half = __shfl_sync(0xffffffffu, it.half, 0);
                            ok = wait_bar_warp(bar_qfull, (n + 1) & 1, abort_flag, 21) && wait_bar_warp(bar_full(ks), kturn, abort_flag, 22);
                        }
                        if (!ok) break;
                        tc_fence_after();
                        there = true;
                    }
                    if (there) {
#pragma unroll 1
                        for (; scores <= t; ++scores) {
                            umma_scores(leader, tmem_base + scores * 128, dq0 + scores * kTile16, dk0 + ks * kTile16, p.idesc_s);
                            tc_commit_by(leader, bar_sfull(scores));
                        }
                    }
                }
                if (!ok) break;
                if (n >= 0) { advance(vs, vturn); ++G; }
                if (!last) {
                    ++j;
                } else {
                    j = 0; num_kt = next_kt; half = next_half; ++n;
                }
                if (there) {
                    tc_commit_by(leader, bar_empty(ks));
                    if (j + 1 == num_kt) tc_commit_by(leader, bar_qempty);   // every score MMA of the item has been issued
                    advance(ks, kturn);
                }
            }
            if (!ok) settle();
        }
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kRegsHigh5));
        // ------------------------------------------------------------------ softmax warps (thread = row)
        const int t = warp >> 2;
        const int wq = warp & 3;
        const int row = wq * 32 + lane;
        const int tok = row >> pp.head_shift;   // query row of the item
        unsigned char* stage_out = smem_gen + kOff4Out + warp * (kTileBytes / 8);
        const uint32_t t_s = tmem_base + (static_cast<uint32_t>(wq * 32) << 16) + t * 128;
        const uint32_t t_o = tmem_base + (static_cast<uint32_t>(wq * 32) << 16) + 256 + t * 128;
        int n = 0, G = 0;
        bool alive = true;
        auto arrive_p = [&](uint32_t bar) {   // this warp's probabilities so far are in tensor memory
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            mbar_arrive_if(lane == 0, bar);   // (the warp stays converged: more tcgen05.st.sync.aligned follow)
        };
        while (alive) {
            alive = wait_bar_warp(bar_item(n & 3), (n >> 2) & 1, abort_flag, 33);
            if (!alive) break;
            const Tc5Item& it = s_ring[n & 3];
            const int num_kt = it.kind != 0 ? it.num_kt : 0;
            if (num_kt == 0) break;
            const int k_len = it.k_len, lim0 = it.lim0, half = it.half, last_partial = it.last_partial;
            const int rows = it.rows, q_row = it.q_row, head0 = (2 * it.pair + t) << pp.head_shift;
            int seen = min(lim0 + tok, k_len);                                      // keys that the row sees, from the tile's first one on
            int all_seen = min(lim0 + ((wq * 32) >> pp.head_shift), k_len);         // the warp's first row, which sees least
            float m_ref = -INFINITY, l_run = 0.0f;
#pragma unroll 1
            for (int j = 0; j < num_kt; ++j, seen -= kBN, all_seen -= kBN) {
                if (t == 0 && j == last_partial) {
                    // Rows of V past the sequence may hold anything (0 * NaN = NaN): tile 0's softmax warps, whose P.V comes first, zero them.
                    const int c = 2 * G + 1, stage = c % kRing5;
                    alive = wait_bar_warp(bar_full(stage), (c / kRing5) & 1, abort_flag, 13);
                    if (!alive) break;
                    if (row >= k_len - j * kBN) {
                        unsigned char* v_row = smem_gen + kOff4Ring + stage * kTileBytes + row * 128;
#pragma unroll 4
                        for (int i = 0; i < 16; ++i)
                            *reinterpret_cast<uint4*>(v_row + (i >> 3) * kPanelBytes + (((i ^ row) & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
                    }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                }
                alive = wait_bar_warp(bar_sfull(t), G & 1, abort_flag, 31);
                if (!alive) break;
                tc_fence_after();
                softmax_row<T>(t_s, t_o, all_seen < kBN, seen, half != 0 && j + 1 == num_kt, p.scale_log2, j == 0, m_ref, l_run,
                               [&] { arrive_p(bar_phalf(t)); });
                arrive_p(bar_pfull(t));
                ++G;
            }
            if (alive) alive = wait_bar_warp(bar_ofinal(t), n & 1, abort_flag, 32);
            if (!alive) break;
            tc_fence_after();
            {
                // Half a row at a time goes through 4 KiB of this warp (16-byte pieces XOR-swizzled by row) and out in whole 128-byte lines, while the
                // next item's first scores are computed.  (Each thread its own row in 32-byte stores: 32 lines an instruction, 1500 to 1900 clocks an item.)
                const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
                const uint64_t inv2 = pack_f32x2(inv, inv);
                T* dst = static_cast<T*>(p.out) + (static_cast<size_t>(q_row) * p.num_heads + head0) * kHeadDim;   // the tile's first row
                uint32_t o[4][32];   // the whole row at once: one TMEM latency instead of four
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld32(t_o + c * 32, o[c]);
                tc_wait_ld();
                // O has left TMEM: the arrive on p_half in the next item's first round tells the issuer so
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    reg_fence32(o[2 * h]); reg_fence32(o[2 * h + 1]);
                    __syncwarp();   // the other half has been read
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const uint32_t* r = o[2 * h + (c >> 2)] + (c & 3) * 8;
                        uint32_t v[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float a, b;
                            unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), inv2), a, b);
                            v[i] = ElemTraits<T>::pack2(a, b);
                        }
                        *reinterpret_cast<uint4*>(stage_out + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = 4 * i + (lane >> 3), at = wq * 32 + r;   // row of the warp and of the tile
                        const uint4 v = *reinterpret_cast<const uint4*>(stage_out + r * 128 + (((lane ^ r) & 7) << 4));
                        if ((at >> pp.head_shift) < rows)
                            *reinterpret_cast<uint4*>(dst + (at >> pp.head_shift) * static_cast<int>(out_stride) + (at & ((1 << pp.head_shift) - 1)) * kHeadDim + h * 64 + (lane & 7) * 8) = v;
                    }
                }
            }
            ++n;
        }
        if (!alive) settle();
        if (MIXED && !decode_first) {
            // Here, where these warps have their 208 registers: behind the roles the code has to make do with those of the other warpgroup (56 then),
            // and a context of 4096 keys took 170 us instead of 90 (1 prompt of 300 tokens, 64 decode rows, 8 blocks: 186 us a step; 3 of 500 to 2048,
            // 90 rows, 30 blocks: 296).  Both tiles are done with the shared memory when all softmax warps are here.
            __syncwarp();   // (lanes come from the stores of their rows)
            asm volatile("bar.sync 3, %0;\n" ::"n"(2 * kBM) : "memory");
            decode_half();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && s_abort != 0) atomicCAS(&g_tc_error, 0, s_abort);
    if (warp == 8) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols2) : "memory");
    }
}

// ---- host side ------------------------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(ptr);
    });
    return fn;
}

// [rows, heads, 128] 16-bit tensor -> boxes of `box_rows` rows x `box_heads` heads x 64 elements, 128-byte swizzle.
bool make_map(CUtensorMap* map, const void* base, int64_t rows, int heads, bool bf16, int box_rows = 128, int box_heads = 1) {
    EncodeFn fn = encode_fn();
    if (fn == nullptr || rows <= 0) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(kHeadDim), static_cast<cuuint64_t>(heads), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(kHeadDim) * 2, static_cast<cuuint64_t>(heads) * kHeadDim * 2};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_heads), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base),
              dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// kind::f16 instruction descriptor: D = F32, A / B = F16 or BF16, N 128, M 128 (one block) or 256 (a block pair).
uint32_t make_idesc(bool bf16, bool b_mn_major, int m = kBM) {
    const uint32_t fmt = bf16 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | (0u << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           (static_cast<uint32_t>(kBN >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}


std::atomic<unsigned int> g_launch_seq{0}, g_capture_seq{0};
int ticket_slot(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {   // (status is undefined; the launch will say what is wrong)
        status = cudaStreamCaptureStatusNone;
        cudaGetLastError();
    }
    return static_cast<int>(status == cudaStreamCaptureStatusNone ? g_launch_seq.fetch_add(1u) % kEagerSlots
                                                                  : kEagerSlots + g_capture_seq.fetch_add(1u) % (kTicketSlots - kEagerSlots));
}

// Tensor maps and kernel parameters of a prefill call.
struct TcLaunch {
    CUtensorMap tq, tk, tv;
    TcParams p;
    int64_t tiles;
};
int prepare_tc_launch(const PrefillArgs& a, bool bf16, int head_shift, TcLaunch* out) {
    const bool paged = a.block_tables != nullptr;
    const int64_t key_rows = paged ? a.num_cache_blocks * a.block_size : a.total_k;
    if (!make_map(&out->tq, a.q, a.total_q, a.num_heads, bf16, kBM >> head_shift, 1 << head_shift) ||
        !make_map(&out->tk, paged ? a.k_cache : a.k, key_rows, a.num_kv_heads, bf16) ||
        !make_map(&out->tv, paged ? a.v_cache : a.v, key_rows, a.num_kv_heads, bf16))
        return fail(NVK_ERR_CUDA, "prefill attention (tcgen05): cuTensorMapEncodeTiled failed");
    TcParams p{};
    p.cu_q = a.cu_q; p.cu_k = a.cu_k; p.block_tables = a.block_tables; p.out = a.out;
    p.num_seqs = a.cu_q ? a.num_seqs : 1; p.total_q = a.total_q; p.total_k = a.total_k; p.max_blocks = a.max_blocks;
    p.key_rows = key_rows; p.num_cache_blocks = a.num_cache_blocks;
    p.num_heads = a.num_heads; p.num_kv_heads = a.num_kv_heads; p.block_size = paged ? a.block_size : 1;
    p.scale_log2 = a.scale * kLog2e;
    p.idesc_s = make_idesc(bf16, false);
    p.idesc_pv = make_idesc(bf16, true);
    out->p = p;
    out->tiles = (a.total_q + kBM - 1) / kBM + (a.cu_q ? a.num_seqs : 0);
    if (out->tiles > 65535) return fail(NVK_ERR_UNSUPPORTED, "prefill attention (tcgen05): too many query tiles");
    return NVK_OK;
}

// Shared-memory attribute and SM count of the persistent head-pair kernel, once per device.
template <typename T, bool MIXED>
int prepare_tc5(int* sms_out) {
    static std::atomic<int> sm_count[64] = {};   // 0 until the attribute is set
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    if (device < 0 || device >= 64) return fail(NVK_ERR_UNSUPPORTED, "prefill attention: device index %d not supported", device);
    if (sm_count[device] == 0) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_tc5_kernel<T, MIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes4);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill attention (head pairs): cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
            return fail(NVK_ERR_CUDA, "prefill attention (head pairs): cannot read the SM count");
        sm_count[device] = sms;
    }
    *sms_out = sm_count[device];
    return NVK_OK;
}

// Heads of one tile of the persistent kernel, as a power of two.  An item takes both tiles from the heads of one KV head; the more heads share
// the 128 rows of a tile, the fewer query rows it has, and the less is lost on the ragged end of a sequence and beyond the diagonal.
int tile_head_shift(int group) { return group % 8 == 0 ? 2 : group % 4 == 0 ? 1 : 0; }
Tc5Params tc5_params(const PrefillArgs& a, const TcParams& p, int head_shift) {
    Tc5Params pp{};
    pp.base = p;
    pp.head_shift = head_shift;
    pp.pairs = a.num_heads / (2 << head_shift);
    pp.tiles = static_cast<int>((a.total_q + (kBM >> head_shift) - 1) / (kBM >> head_shift) + (a.cu_q ? a.num_seqs : 0));
    pp.total = static_cast<unsigned int>(pp.pairs) * static_cast<unsigned int>(pp.tiles);
    pp.slot = ticket_slot(a.stream);
    return pp;
}

template <typename T>
int launch_typed(const PrefillArgs& a, bool bf16) {
    static std::atomic<bool> attr_done[64] = {};
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 0 && device < 64 && !attr_done[device]) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_tc_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill attention (tcgen05): cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        attr_done[device] = true;
    }
    TcLaunch L;
    const int group = a.num_heads / a.num_kv_heads, head_shift = tile_head_shift(group);
    const int rc = prepare_tc_launch(a, bf16, head_shift, &L);
    if (rc != NVK_OK) return rc;
    const CUtensorMap &tq = L.tq, &tk = L.tk, &tv = L.tv;
    const TcParams& p = L.p;
    const int64_t tiles = L.tiles;
    if (group % 2 == 0) {   // pairs of query heads that share a KV head: persistent blocks, one per SM, items from a ticket counter
        int sms = 0;
        const int rc5 = prepare_tc5<T, false>(&sms);
        if (rc5 != NVK_OK) return rc5;
        const Tc5Params pp = tc5_params(a, p, head_shift);
        const unsigned int blocks = pp.total < static_cast<unsigned int>(sms) ? pp.total : static_cast<unsigned int>(sms);
        const cudaError_t e = launch_pdl(prefill_tc5_kernel<T, false>, dim3(blocks), dim3(kThreads5), kSmemBytes4, a.stream, tq, tk, tv, pp, MixedDecode{});
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill_tc5_kernel launch: %s", cudaGetErrorString(e));
        return check_launch("prefill_tc5_kernel launch");
    }
    // odd group sizes: one block per (query tile, head)
    const dim3 grid(a.num_heads, static_cast<unsigned>(tiles));
    const cudaError_t e = launch_pdl(prefill_tc_kernel<T>, grid, dim3(kThreads), kSmemBytes, a.stream, tq, tk, tv, p);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill_tc_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("prefill_tc_kernel launch");
}

}  // namespace

static bool tc_shape_supported(const PrefillArgs& a) {
    if (a.dtype != NVK_F16 && a.dtype != NVK_BF16) return false;
    if (a.head_dim != kHeadDim) return false;
    if (!aligned_to(a.q, 16) || !aligned_to(a.out, 16)) return false;
    if (a.total_q >= (1LL << 31) || a.num_heads > 65535) return false;
    if (a.block_tables) {
        if (a.block_size % kBN != 0) return false;
        if (!aligned_to(a.k_cache, 16) || !aligned_to(a.v_cache, 16)) return false;
        if (a.num_cache_blocks * a.block_size >= (1LL << 31)) return false;
    } else {
        if (!aligned_to(a.k, 16) || !aligned_to(a.v, 16)) return false;
        if (a.total_k <= 0 || a.total_k >= (1LL << 31)) return false;
    }
    return encode_fn() != nullptr;
}

// (A hidden score is minus infinity before it is scaled, in softmax_row as in the chunk_max and chunk_probs of odd groups.)
bool prefill_tc_supported(const PrefillArgs& a) { return a.scale > 0.0f && tc_shape_supported(a); }

int launch_prefill_tc(const PrefillArgs& a) {
    return a.dtype == NVK_BF16 ? launch_typed<__nv_bfloat16>(a, true) : launch_typed<__half>(a, false);
}

namespace {

template <typename T>
int launch_mixed_typed(const PrefillArgs& a, const DecodeArgs& d, int prefill_blocks, bool bf16) {
    TcLaunch L;
    const int head_shift = tile_head_shift(a.num_heads / a.num_kv_heads);
    int rc = prepare_tc_launch(a, bf16, head_shift, &L);
    if (rc != NVK_OK) return rc;
    int sms = 0;
    rc = prepare_tc5<T, true>(&sms);
    if (rc != NVK_OK) return rc;
    MixedDecode md{};
    int cluster = 0;   // the ranges of the cluster kernel are taken one by one here and merged through the workspace
    rc = decode_plan(d, dec::Cache16<T>::kGroups, &md.dp, &cluster);
    if (rc != NVK_OK) return rc;
    const Tc5Params pp = tc5_params(a, L.p, head_shift);
    if (prefill_blocks <= 0) {
        // No hint: split the SMs by a crude estimate from host-known sizes -- prefill flops as if all sequences were equally
        // long and had no prefix, at 0.6 PFLOP/s; decode bytes as if every block table were half full, at 6.5 TB/s.  Against the best of 17
        // splits for 19 steps (1 to 6 prompts of 64 to 4000 tokens, 8 to 192 decode rows) it costs 3 % on average and 11 % at most (with 0.3 PFLOP/s
        // 3.5 % on average, with 1.0 4.7 %): it matters little, since every block sees to what is left of the other kind.
        const double mean_q = static_cast<double>(a.total_q) / static_cast<double>(a.cu_q ? a.num_seqs : 1);
        const double t_prefill = 4.0 * a.num_heads * kHeadDim * static_cast<double>(a.total_q) * (mean_q + 1.0) / 2.0 / 0.6e15;
        const double t_decode = 0.5 * static_cast<double>(d.batch) * d.max_blocks * d.block_size * d.num_kv_heads * kHeadDim * 4.0 / 6.5e12;
        prefill_blocks = static_cast<int>(sms * t_prefill / (t_prefill + t_decode) + 0.5);
    }
    if (prefill_blocks < 1) prefill_blocks = 1;
    if (prefill_blocks > sms) prefill_blocks = sms;
    md.prefill_blocks = prefill_blocks;
    const cudaError_t e = launch_pdl(prefill_tc5_kernel<T, true>, dim3(static_cast<unsigned int>(sms)), dim3(kThreads5), kSmemBytes4, a.stream, L.tq, L.tk,
                                     L.tv, pp, md);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "mixed prefill + decode kernel launch: %s", cudaGetErrorString(e));
    rc = check_launch("mixed prefill + decode kernel launch");
    if (rc != NVK_OK) return rc;
    return launch_decode_merge(md.dp, d.dtype, d.stream);
}

}  // namespace

// One launch for a step with prefill and decode sequences: the head-pair prefill kernel and the tensor-core decode kernel
// must both take their halves, and the decode half needs its split-K workspace.
bool mixed_step_supported(const PrefillArgs& p, const DecodeArgs& d) {
    if (!tc_shape_supported(p) || (p.num_heads / p.num_kv_heads) % 2 != 0) return false;
    if (!decode_mma_supported(d) || d.workspace == nullptr) return false;
    if (p.dtype != d.dtype || p.num_heads != d.num_heads || p.num_kv_heads != d.num_kv_heads || p.stream != d.stream) return false;
    if (p.total_q <= 0 || d.batch <= 0) return false;
    return true;
}

int launch_mixed_step(const PrefillArgs& p, const DecodeArgs& d, int prefill_blocks) {
    return p.dtype == NVK_BF16 ? launch_mixed_typed<__nv_bfloat16>(p, d, prefill_blocks, true)
                               : launch_mixed_typed<__half>(p, d, prefill_blocks, false);
}

}  // namespace nvk

extern "C" int nvk_prefill_status(void* stream, int* status) {
    using namespace nvk;
    if (!status) return fail(NVK_ERR_INVALID_ARGUMENT, "prefill status: null argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int word = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(&word, g_tc_error, sizeof(int), 0, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && word != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbolAsync(g_tc_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill status: %s", cudaGetErrorString(e));
    *status = word;
    return word != 0 ? NVK_OK : prefill_tile_status(st, status);
}
