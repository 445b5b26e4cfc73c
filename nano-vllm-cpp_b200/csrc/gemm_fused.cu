// The two linears on either side of attention, fused with what follows them (tcgen05 + TMEM + TMA, F16 / BF16):
//
//   * QKV projection + attention prologue.  The reference runs qkv_proj as a cuBLASLt GEMM (src/layers/linear.cpp:348-420),
//     writes the packed [rows, (Hq + 2 Hkv) * D] tensor and reads it back in fused_split_norm_rope_store
//     (src/kernels/split_qkv.cu:62-154, called from src/models/transformer.cpp:132-139).  With head_dim 128 one
//     128-column tile of the GEMM IS one head: the epilogue thread that owns a row of the accumulator holds the whole
//     head vector, so the per-head RMSNorm, the rotation pairs (d, d + 64) and the scatter into the paged cache need no
//     exchange at all.  The packed tensor never exists.
//   * Row-parallel projection + all-reduce.  o_proj / down_proj produce a partial sum that is all-reduced over the
//     tensor-parallel ranks (src/layers/linear.cpp:306-320).  Here the epilogue writes each row of the partial sum
//     straight to the rank that will reduce it: its own rows into its addend buffer, the others as tagged vectors into
//     the owners' staging areas over NVLink -- the first phase of nvk_tp_allreduce_add_rmsnorm (tp_allreduce.cu) done
//     by the GEMM, tile by tile, while the other tiles still compute.  The all-reduce kernel that follows is told to
//     skip its push.
//
// GEMM core: C[M, N] = A[M, K] * B[N, K]^T, both operands K-major as torch linears keep them; TMA (128-byte swizzle) into a ring of
// shared-memory stages, tcgen05.mma into TMEM.  Two kernels, chosen by size (choose_gemm):
//   gemm_split_kernel   few rows.  The GEMM streams the weight once and is HBM-bound, so every SM has to stream: a block takes 128
//                       rows x 128 columns of C over a part of K (or 256 rows over all of it), the blocks of a cluster the parts of one
//                       tile; each pushes its sums to the block that finishes a row, which runs the epilogue on its share of the rows.
//   gemm_pair_kernel    many rows, bound by the tensor pipe.  Persistent pairs of blocks (cta_group::2): 256 x 256 tiles, each block
//                       loads half of A and half of B, so an SM moves half the operand bytes of a 128 x 256 tile of its own.  The
//                       accumulator is double buffered in TMEM: the epilogue of a tile runs under the next tile's MMAs.
// Before, one block per 128 x 128 tile whatever the size (microseconds in a loop over weights larger than L2; K 4096):
//   64 x 6144  22 -> 16      64 x 4096  21 -> 12 (with MMAs from a converged warp 14.5 and 11.1, with pushed sums 13.3 and 10.0)     7440 x 4096  295 -> 175 (1430 TFLOP/s)     7440 x 6144 with QKV epilogue  597 -> 277
// What the fusion removes is the round trip of the result and one or two launches per layer.
// Every mbarrier wait is bounded; a wait that runs out raises an error word (nvk_gemm_status), and the block leaves when what it
// has under way has had time to land.
#include "nvk_internal.cuh"

#include <cuda.h>

#include <atomic>
#include <mutex>

namespace nvk {
namespace {

constexpr int kBM = 128, kBN = 128, kBK = 64;
constexpr int kPanelBytes = kBM * kBK * 2;            // 16 KiB: 128 rows x 128 bytes
constexpr int kRingBytes = 12 * kPanelBytes;          // 192 KiB: 6 stages of 2 panels or 4 of 3
constexpr int kEpilogueBytes = 4096;                  // of a warp that takes whole rows from tensor memory
constexpr int kStageOffset = kRingBytes;              // for the epilogue warps, or what peers push in gemm_split_kernel
constexpr int kBarOffset = kStageOffset + 8 * kEpilogueBytes;
constexpr int kSmemBytes = kBarOffset + 256 + 1024;   // + slack for 1024-byte alignment
constexpr int kThreads = 256;                         // warp 0 TMA, warp 1 MMA + TMEM, warps 2-5 TMEM readers, all for the sums
constexpr int kPairThreads = 320;                     // the same with warps 2-9 for the epilogue
constexpr long long kWaitCycles = 4000000000LL;       // ~2 s
constexpr int kMaxRanks = NVK_TP_MAX_RANKS;

__device__ int g_gemm_error = 0;

enum Epilogue { kPlain = 0, kQkvPrologue = 1, kAllReducePush = 2 };

struct GemmParams {
    void* out;                 // kPlain: C [M, N]
    int64_t m, n, k;
    uint32_t idesc;
    int tiles_m, tiles_n;      // gemm_pair_kernel
    int a_rows;                // gemm_split_kernel: rows of A that a load brings in (a multiple of 8; the tile's other rows stay undefined)
    // kQkvPrologue
    const int32_t* positions; const void* q_weight; const void* k_weight; const float* cos_sin; const int32_t* slot_mapping;
    void* q_out; void* k_cache; void* v_cache;
    int64_t cache_rows;
    int max_positions, hq, hkv;
    int table_vec;             // cos_sin starts on a 16-byte boundary
    float eps;
    // kAllReducePush
    void* addend;              // this rank's addend buffer [M, N]: rows it reduces itself
    uint4* stage[kMaxRanks];   // every rank's staging area (index = rank)
    const uint32_t* flags;     // this rank's flag area: [0] = epoch of the last completed all-reduce
    int rank, world;
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
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long start = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - start > kWaitCycles) {
            *abort_flag = 1;
            atomicCAS(&g_gemm_error, 0, code);
            return false;
        }
    }
}
// The same by a converged warp, with the same answer for all its lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity) != 0)) return true;
    const long long start = clock64();
    while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity) != 0)) {
        if (!__all_sync(0xffffffffu, *abort_flag == 0 && clock64() - start <= kWaitCycles)) {
            if (*abort_flag == 0) atomicCAS(&g_gemm_error, 0, code);
            *abort_flag = 1;
            return false;
        }
    }
    return true;
}
// Where a wait gave up, by the warp that frees the block's tensor memory, before it does (the block is there until all its warps have left): copies into
// shared memory and MMAs that read it may still be under way, and a wait for each would end with the same limit at the latest.  2 ms.
__device__ __forceinline__ void settle() {
    const long long start = clock64();
    while (clock64() - start < 4000000) {}
    __syncwarp();
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// The same from a block of a pair: the barrier may be the other block's (`bar`: a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// `.aligned` instructions (this barrier, tcgen05.ld and its wait, allocation) want the whole warp at one place.  What lanes do on their own before one
// -- a branch on a row's slot or position, a single lane's store -- is followed by a warp barrier, a shuffle or a vote.
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %cluster_ctarank;\n" : "=r"(r));
    return r;
}
// MMAs and commits of gemm_split_kernel come from a converged warp: all lanes run through the same instructions, so that the operands are uniform registers, which is where
// the MMA wants them, and one lane (`leader` 1) issues.  A single diverged lane has to move every operand there first, 75 to 100 clocks an
// MMA; gemm_pair_kernel, whose MMAs take 128, keeps that (its QKV epilogue was 3 % slower beside a whole warp that polls).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t leader;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(leader));
    return leader;
}
__device__ __forceinline__ void tc_commit(uint32_t leader, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}\n" ::"r"(leader), "r"(bar) : "memory");
}
__device__ __forceinline__ void umma_ss(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %0, 0;\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%1], %2, %3, %4, p;\n\t}\n"
        ::"r"(leader), "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {                  // arrives in both blocks of the pair
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                 ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void umma_ss_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
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
// pins the use of asynchronously loaded registers after the preceding tcgen05.wait::ld
__device__ __forceinline__ void reg_fence32(uint32_t (&r)[32]) {
    asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                      "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
    asm volatile("" : "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                      "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}
// K-major, 128-byte swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr) {
    const uint32_t lo = ((addr & 0x3FFFFu) >> 4) | ((16u >> 4) << 16);
    const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    return (static_cast<uint64_t>(hi) << 32) | lo;
}
__device__ __forceinline__ void st_tagged(uint4* slot, const uint4& v, uint32_t ep) {   // the all-reduce's wire format
    // one 32-byte store per payload vector: a warp writes 1 KiB of contiguous, fully covered 128-byte lines (two 16-byte
    // stores per lane left every sector half written per instruction, which costs NVLink packets)
    asm volatile("st.volatile.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
                 ::"l"(slot), "r"(v.x), "r"(ep), "r"(v.y), "r"(ep), "r"(v.z), "r"(ep), "r"(v.w), "r"(ep) : "memory");
}

// 32 accumulator columns of this thread's row, rounded to T (what the unfused GEMM would have written)
template <typename T>
__device__ __forceinline__ void load_rounded(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    __syncwarp();   // (epilogue_row branches on what a row needs, lane by lane)
    tmem_ld32(taddr, r);
    tc_wait_ld();
    reg_fence32(r);
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = ElemTraits<T>::to_float(ElemTraits<T>::from_float(__uint_as_float(r[i])));
}
template <typename T> __device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi) {
    const T* e = reinterpret_cast<const T*>(&w);
    lo = ElemTraits<T>::to_float(e[0]);
    hi = ElemTraits<T>::to_float(e[1]);
}
template <typename T> __device__ __forceinline__ uint4 pack8(const float* v) {
    return make_uint4(ElemTraits<T>::pack2(v[0], v[1]), ElemTraits<T>::pack2(v[2], v[3]), ElemTraits<T>::pack2(v[4], v[5]), ElemTraits<T>::pack2(v[6], v[7]));
}
// Every lane has a row: 32 elements for dst + off0 and 32 for dst + off1 (dst == nullptr: nothing).  Through 4 KiB of shared memory, so
// that four lanes write 64 contiguous bytes of a row where one lane each would write 16-byte pieces of 32 rows: with short K the tile's
// epilogue is the bound (7000 x 4096, K 512: 53 -> 38 us).
template <typename T>
__device__ __forceinline__ void store_rows(T* dst, int off0, int off1, const float (&v0)[32], const float (&v1)[32], unsigned char* stage, int lane) {
    uint4* row = reinterpret_cast<uint4*>(stage + lane * 128);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        row[q ^ (lane & 7)] = pack8<T>(v0 + 8 * q);
        row[(4 + q) ^ (lane & 7)] = pack8<T>(v1 + 8 * q);
    }
    __syncwarp();
    const unsigned long long addr = reinterpret_cast<unsigned long long>(dst);
    const int c = lane & 7, off = (c < 4 ? off0 : off1) + (c & 3) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3);
        T* to = reinterpret_cast<T*>(__shfl_sync(0xffffffffu, addr, r));
        const uint4 w = reinterpret_cast<const uint4*>(stage + r * 128)[c ^ (r & 7)];
        if (to != nullptr) *reinterpret_cast<uint4*>(to + off) = w;
    }
    __syncwarp();
}

// ---- epilogues of one 128-column tile (with head_dim 128: of one head) -------------------------------------------------------
// Four elements of a row of the rotary table, which callers may have at any float's address.
__device__ __forceinline__ float4 ld_table(const GemmParams& p, const float* at) {
    if (p.table_vec) return __ldg(reinterpret_cast<const float4*>(at));
    return make_float4(__ldg(at), __ldg(at + 1), __ldg(at + 2), __ldg(at + 3));
}
// What a row of tile `nt` turns into: where it goes, and for q and k heads how it is normalised and rotated.
template <typename T>
struct QkvRow {
    T* dst;
    const T* weight;      // nullptr: no norm
    const float* table;   // nullptr: no rotation
    bool is_v;
};
struct QkvIndex { int pos, slot; bool live; };
__device__ __forceinline__ QkvIndex qkv_index(const GemmParams& p, int64_t row) {
    const bool live = row < p.m;
    return QkvIndex{live ? __ldg(p.positions + row) : 0, live && p.slot_mapping != nullptr ? __ldg(p.slot_mapping + row) : -1, live};
}
template <typename T>
__device__ __forceinline__ QkvRow<T> qkv_row(const GemmParams& p, int head, int64_t row, const QkvIndex& at) {
    const bool is_q = head < p.hq, is_k = !is_q && head < p.hq + p.hkv;
    const int pos = at.pos;
    const int64_t slot = p.slot_mapping != nullptr ? static_cast<int64_t>(at.slot) : row;
    QkvRow<T> x{nullptr, nullptr, nullptr, !is_q && !is_k};
    if (at.live) {
        if (is_q) x.dst = static_cast<T*>(p.q_out) + (row * p.hq + head) * kBN;
        else if (slot >= 0 && slot < p.cache_rows)
            x.dst = static_cast<T*>(is_k ? p.k_cache : p.v_cache) + (slot * p.hkv + (is_k ? head - p.hq : head - p.hq - p.hkv)) * kBN;
    }
    if (p.q_weight != nullptr) x.weight = static_cast<const T*>(is_q ? p.q_weight : p.k_weight);
    if (pos >= 0 && pos < p.max_positions) x.table = p.cos_sin + static_cast<int64_t>(pos) * kBN;
    return x;
}
// Where a row of a partial sum is reduced: `addend` (this rank) or a tagged slot of the owner's staging area.
template <typename T>
struct PushRow {
    T* addend;
    uint4* slot;
    uint32_t epoch;
};
template <typename T>
__device__ __forceinline__ PushRow<T> push_row(const GemmParams& p, int64_t row, bool live, int n0) {
    const uint32_t last = *reinterpret_cast<const volatile uint32_t*>(p.flags);
    PushRow<T> x{nullptr, nullptr, last + 1u == 0u ? 1u : last + 1u};      // the epoch the all-reduce launch after this GEMM will use
    if (!live || *reinterpret_cast<const volatile uint32_t*>(p.flags + 2) != 0u) return x;
    const int64_t rows_per_rank = p.m / p.world, row_vecs = p.n / 8, chunk_vecs = rows_per_rank * row_vecs;
    const int owner = static_cast<int>(row / rows_per_rank);
    if (owner == p.rank) x.addend = static_cast<T*>(p.addend) + row * p.n + n0;
    else x.slot = p.stage[owner] + 2 * (p.rank * chunk_vecs + (row - owner * rows_per_rank) * row_vecs + n0 / 8);
    return x;
}

// One thread holds the whole row in TMEM columns t_row .. t_row + 127 (warp-collective: every lane runs all of it).  `stage`: 4 KiB of
// shared memory of this warp, 8 with WIDE (gemm_pair_kernel has no room for that beside its ring).  `hidden`: other work takes longer than the
// epilogue, whose instructions cost that work more than its time matters (gemm_pair_kernel, 7440 x 6144, K 4096: 264.5 us, so only behind the last tile 260, one lane a row
// throughout 262).
template <typename T, int EPI, bool WIDE>
__device__ __forceinline__ void epilogue_row(const GemmParams& p, uint32_t t_row, int64_t row, const QkvIndex& at_row, int nt, unsigned char* stage, int lane, bool hidden = false) {
    const bool live = row < p.m;
    const int n0 = nt * kBN;
    if (EPI == kAllReducePush) {
        const PushRow<T> x = push_row<T>(p, row, live, n0);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            float v[32];
            load_rounded<T>(t_row + c * 32, v);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 w = pack8<T>(v + 8 * q);
                if (x.addend != nullptr) reinterpret_cast<uint4*>(x.addend + c * 32)[q] = w;
                else if (x.slot != nullptr) st_tagged(x.slot + 2 * (c * 4 + q), w, x.epoch);
            }
        }
        return;
    }
    QkvRow<T> x{};
    if (EPI == kQkvPrologue) x = qkv_row<T>(p, nt, row, at_row);
    if (EPI == kPlain || x.is_v) {             // the rounded GEMM output as it is
        T* dst = EPI == kQkvPrologue ? x.dst : live ? static_cast<T*>(p.out) + row * p.n + n0 : nullptr;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            float v0[32], v1[32];
            load_rounded<T>(t_row + c * 64, v0);
            load_rounded<T>(t_row + c * 64 + 32, v1);
            store_rows<T>(dst, c * 64, c * 64 + 32, v0, v1, stage, lane);
        }
        return;
    }
    // A q or k head.  The thread that has the row takes its sum of squares and leaves the row in shared memory; norm and rotation are done by eight lanes a
    // row, so that they read table rows and write results in whole 128-byte lines: eight rows a trip, the next trip's table rows under way.  Loads without
    // branches around them: a branch waits for what was loaded before it, which cost more than the loads.  (Each lane its own table row, 32
    // lines an instruction, K 512, 1000 rows x 1536 / 3072 columns: pairs 16.3 / 16.0 us, 13.8 / 14.5 now, one block for 128 rows and all of K 8.4, now 6.7 / 12.9;
    // products alone in pairs 7.9 / 8.7.)
    if constexpr (WIDE) {
        const int sub = lane & 7;                  // elements 8 sub .. + 7 of both halves of the head
        const unsigned long long dst_of = reinterpret_cast<unsigned long long>(x.dst), table_of = reinterpret_cast<unsigned long long>(x.table != nullptr ? x.table : p.cos_sin);
        const unsigned int rotated = __ballot_sync(0xffffffffu, x.table != nullptr);
        struct Trig { float4 cs[2], sn[2]; };
        auto fetch = [&](int at, Trig& g) {        // table row of row `at`
            const float* from = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, table_of, at)) + 8 * sub;   // (row 0 where there is none)
#pragma unroll
            for (int i = 0; i < 2; ++i) { g.cs[i] = ld_table(p, from + 4 * i); g.sn[i] = ld_table(p, from + 64 + 4 * i); }
        };
        Trig now[2], next[2];
        T w[16];
        float ss4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float v[32];
            load_rounded<T>(t_row + c * 32, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) ss4[i & 3] += v[i] * v[i];
#pragma unroll
            for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(stage + lane * 256)[(4 * c + q) ^ (lane & 7)] = pack8<T>(v + 8 * q);
        }
        if (x.weight != nullptr) {
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = x.weight[(i >> 3) * 64 + 8 * sub + (i & 7)];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) fetch(4 * u + (lane >> 3), now[u]);
        const float ss = (ss4[0] + ss4[1]) + (ss4[2] + ss4[3]);
        const float inv_rms = rsqrtf(ss / static_cast<float>(kBN) + p.eps);
        __syncwarp();
        auto trip = [&](int r, Trig (&now)[2]) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int at = r + 4 * u + (lane >> 3);
                const uint4* from = reinterpret_cast<const uint4*>(stage + at * 256);
                const uint4 lo4 = from[sub ^ (at & 7)], hi4 = from[(8 + sub) ^ (at & 7)];
                const uint32_t lo_w[4] = {lo4.x, lo4.y, lo4.z, lo4.w}, hi_w[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
                float lo[8], hi[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    unpack2<T>(lo_w[i], lo[2 * i], lo[2 * i + 1]);
                    unpack2<T>(hi_w[i], hi[2 * i], hi[2 * i + 1]);
                }
                if (x.weight != nullptr) {
                    const float inv = __shfl_sync(0xffffffffu, inv_rms, at);
#pragma unroll
                    for (int i = 0; i < 8; ++i) { lo[i] = lo[i] * inv * ElemTraits<T>::to_float(w[i]); hi[i] = hi[i] * inv * ElemTraits<T>::to_float(w[8 + i]); }
                }
                if ((rotated >> at) & 1u) {        // first half: x cos - partner sin; second half: x cos + partner sin
                    const float4 (&c4)[2] = now[u].cs, (&s4)[2] = now[u].sn;
                    const float cs[8] = {c4[0].x, c4[0].y, c4[0].z, c4[0].w, c4[1].x, c4[1].y, c4[1].z, c4[1].w};
                    const float sn[8] = {s4[0].x, s4[0].y, s4[0].z, s4[0].w, s4[1].x, s4[1].y, s4[1].z, s4[1].w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float a = lo[i], b = hi[i];
                        lo[i] = fmaf(a, cs[i], b * -sn[i]);
                        hi[i] = fmaf(b, cs[i], a * sn[i]);
                    }
                }
                T* dst = reinterpret_cast<T*>(__shfl_sync(0xffffffffu, dst_of, at));
                if (dst != nullptr) {
                    *reinterpret_cast<uint4*>(dst + 8 * sub) = pack8<T>(lo);
                    *reinterpret_cast<uint4*>(dst + 64 + 8 * sub) = pack8<T>(hi);
                }
            }
        };
#pragma unroll 1
        for (int r = 0; r < 32; r += 16) {
#pragma unroll
            for (int u = 0; u < 2; ++u) fetch(r + 8 + 4 * u + (lane >> 3), next[u]);
            trip(r, now);
            if (r < 16) {
#pragma unroll
                for (int u = 0; u < 2; ++u) fetch(r + 16 + 4 * u + (lane >> 3), now[u]);
            }
            trip(r + 8, next);
        }
        __syncwarp();                              // the rows have been read
    } else if (hidden) {
        // Each lane the row that it has: fewest instructions, and slow.
        float inv_rms = 1.0f;
        if (x.weight != nullptr) {                 // pass 1 over the accumulator: the head's sum of squares
            float ss4[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // (the order of the other forms: a row's bits do not depend on its tile's place)
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                float v[32];
                load_rounded<T>(t_row + c * 32, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) ss4[i & 3] += v[i] * v[i];
            }
            inv_rms = rsqrtf(((ss4[0] + ss4[1]) + (ss4[2] + ss4[3])) / static_cast<float>(kBN) + p.eps);
        }
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {              // pass 2: columns [32 c, 32 c + 32) rotate with [64 + 32 c, 64 + 32 c + 32)
            float lo[32], hi[32];
            load_rounded<T>(t_row + c * 32, lo);
            load_rounded<T>(t_row + 64 + c * 32, hi);
            if (x.weight != nullptr) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    lo[i] = lo[i] * inv_rms * ElemTraits<T>::to_float(x.weight[c * 32 + i]);
                    hi[i] = hi[i] * inv_rms * ElemTraits<T>::to_float(x.weight[64 + c * 32 + i]);
                }
            }
            if (x.table != nullptr) {              // first half: x cos - partner sin; second half: x cos + partner sin
                // 16-byte loads: every lane reads its own table row, so an instruction costs 32 cache lines whatever its width
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float4 c4 = ld_table(p, x.table + c * 32 + i), s4 = ld_table(p, x.table + 64 + c * 32 + i);
                    const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float a = lo[i + u], b = hi[i + u];
                        lo[i + u] = fmaf(a, cs[u], b * -sn[u]);
                        hi[i + u] = fmaf(b, cs[u], a * sn[u]);
                    }
                }
            }
            store_rows<T>(x.dst, c * 32, 64 + c * 32, lo, hi, stage, lane);
        }
    } else {
        // With 4 KiB: columns [32 c, 32 c + 32) and their partners [64 + 32 c, ...) at a time, four lanes a row, eight rows a trip.
        const int sub = lane & 3;                  // elements 8 sub .. + 7 of the columns and of their partners
        const unsigned long long dst_of = reinterpret_cast<unsigned long long>(x.dst), table_of = reinterpret_cast<unsigned long long>(x.table != nullptr ? x.table : p.cos_sin);
        const unsigned int rotated = __ballot_sync(0xffffffffu, x.table != nullptr);
        struct Trig { float4 cs[2], sn[2]; } even, odd;
        auto fetch = [&](int trip, Trig& g) {      // of eight: four of each c
            const float* from = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, table_of, (trip & 3) * 8 + (lane >> 2))) + (trip >> 2) * 32 + 8 * sub;
#pragma unroll
            for (int i = 0; i < 2; ++i) { g.cs[i] = ld_table(p, from + 4 * i); g.sn[i] = ld_table(p, from + 64 + 4 * i); }
        };
        float ss4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (x.weight != nullptr) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float v[32];
                load_rounded<T>(t_row + c * 32, v);
#pragma unroll
                for (int i = 0; i < 32; ++i) ss4[i & 3] += v[i] * v[i];
            }
        }
        const float inv_rms = rsqrtf(((ss4[0] + ss4[1]) + (ss4[2] + ss4[3])) / static_cast<float>(kBN) + p.eps);
        fetch(0, even);
        fetch(1, odd);
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            T w[16];
            {
                uint4* row16 = reinterpret_cast<uint4*>(stage + lane * 128);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float v[32];
                    load_rounded<T>(t_row + c * 32 + h * 64, v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) row16[(4 * h + q) ^ (lane & 7)] = pack8<T>(v + 8 * q);
                }
            }
            if (x.weight != nullptr) {
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = x.weight[32 * c + (i >> 3) * 64 + 8 * sub + (i & 7)];
            }
            __syncwarp();
            auto trip = [&](int n, Trig& g) {
                const int at = (n & 3) * 8 + (lane >> 2);
                const uint4* from = reinterpret_cast<const uint4*>(stage + at * 128);
                const uint4 lo4 = from[sub ^ (at & 7)], hi4 = from[(4 + sub) ^ (at & 7)];
                const uint32_t lo_w[4] = {lo4.x, lo4.y, lo4.z, lo4.w}, hi_w[4] = {hi4.x, hi4.y, hi4.z, hi4.w};
                float lo[8], hi[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    unpack2<T>(lo_w[i], lo[2 * i], lo[2 * i + 1]);
                    unpack2<T>(hi_w[i], hi[2 * i], hi[2 * i + 1]);
                }
                if (x.weight != nullptr) {
                    const float inv = __shfl_sync(0xffffffffu, inv_rms, at);
#pragma unroll
                    for (int i = 0; i < 8; ++i) { lo[i] = lo[i] * inv * ElemTraits<T>::to_float(w[i]); hi[i] = hi[i] * inv * ElemTraits<T>::to_float(w[8 + i]); }
                }
                if ((rotated >> at) & 1u) {
                    const float cs[8] = {g.cs[0].x, g.cs[0].y, g.cs[0].z, g.cs[0].w, g.cs[1].x, g.cs[1].y, g.cs[1].z, g.cs[1].w};
                    const float sn[8] = {g.sn[0].x, g.sn[0].y, g.sn[0].z, g.sn[0].w, g.sn[1].x, g.sn[1].y, g.sn[1].z, g.sn[1].w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float a = lo[i], b = hi[i];
                        lo[i] = fmaf(a, cs[i], b * -sn[i]);
                        hi[i] = fmaf(b, cs[i], a * sn[i]);
                    }
                }
                fetch((n + 2) & 7, g);
                T* dst = reinterpret_cast<T*>(__shfl_sync(0xffffffffu, dst_of, at));
                if (dst != nullptr) {
                    *reinterpret_cast<uint4*>(dst + 32 * c + 8 * sub) = pack8<T>(lo);
                    *reinterpret_cast<uint4*>(dst + 64 + 32 * c + 8 * sub) = pack8<T>(hi);
                }
            };
#pragma unroll 1
            for (int n = 4 * c; n < 4 * c + 4; n += 2) {
                trip(n, even);
                trip(n + 1, odd);
            }
            __syncwarp();                          // the columns have been read
        }
    }
}

// Eight lanes hold a row: lane `sub` elements 32 q + 4 sub .. + 3, q = 0 .. 3 (v[q]), so that the eight read 128 contiguous bytes of the
// sums at a time and rotation pairs (d, d + 64) meet in a lane.  octet_row fetches what the epilogue of a row needs besides the sums (with the row's
// position and slot, which come first: two dependent trips to memory), so that this can be under way before the sums are there.
template <typename T>
struct OctetRow {
    T* dst;               // kPlain, kQkvPrologue, kAllReducePush (own rows); nullptr: nothing to write there
    uint4* slot;          // kAllReducePush
    uint32_t epoch;
    bool rotate;
    float4 cs[2], sn[2];
};
template <typename T, int EPI>
__device__ __forceinline__ OctetRow<T> octet_row(const GemmParams& p, int64_t row, const QkvIndex& at, int nt, int sub) {
    const bool live = row < p.m;
    OctetRow<T> x{};
    if (EPI == kPlain) {
        x.dst = live ? static_cast<T*>(p.out) + row * p.n + nt * kBN : nullptr;
    } else if (EPI == kQkvPrologue) {
        const QkvRow<T> q = qkv_row<T>(p, nt, row, at);
        x.dst = q.dst;
        x.rotate = !q.is_v && q.table != nullptr;
        if (!q.is_v) {                             // (the same for the whole block; otherwise no branch that waits for what was loaded before it)
            const float* from = (q.table != nullptr ? q.table : p.cos_sin) + 4 * sub;
#pragma unroll
            for (int i = 0; i < 2; ++i) { x.cs[i] = ld_table(p, from + 32 * i); x.sn[i] = ld_table(p, from + 64 + 32 * i); }
        }
    } else {
        const PushRow<T> q = push_row<T>(p, row, live, nt * kBN);
        x.dst = q.addend; x.slot = q.slot; x.epoch = q.epoch;
    }
    return x;
}
// The norm weights of this lane's elements, the same for all rows of the tile.
template <typename T, int EPI>
__device__ __forceinline__ void octet_weights(const GemmParams& p, int nt, int sub, T (&w)[16]) {
    if (EPI != kQkvPrologue || p.q_weight == nullptr || nt >= p.hq + p.hkv) return;
    const T* weight = static_cast<const T*>(nt < p.hq ? p.q_weight : p.k_weight) + 4 * sub;
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = weight[32 * (i >> 2) + (i & 3)];
}
// Every lane of the warp runs it (shuffles).
template <typename T, int EPI>
__device__ __forceinline__ void epilogue_octet(const GemmParams& p, const OctetRow<T>& x, float4 (&v)[4], const T (&weight)[16], int nt, int sub) {
    float e[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        e[q][0] = v[q].x; e[q][1] = v[q].y; e[q][2] = v[q].z; e[q][3] = v[q].w;
#pragma unroll
        for (int i = 0; i < 4; ++i) e[q][i] = ElemTraits<T>::to_float(ElemTraits<T>::from_float(e[q][i]));
    }
    if (EPI == kQkvPrologue && nt < p.hq + p.hkv) {   // a q or k head (the same for the whole block)
        if (p.q_weight != nullptr) {
            float ss = 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
#pragma unroll
                for (int i = 0; i < 4; ++i) ss += e[q][i] * e[q][i];
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float inv_rms = rsqrtf(ss / static_cast<float>(kBN) + p.eps);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
#pragma unroll
                for (int i = 0; i < 4; ++i) e[q][i] = e[q][i] * inv_rms * ElemTraits<T>::to_float(weight[4 * q + i]);
            }
        }
        if (x.rotate) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float cs[4] = {x.cs[q].x, x.cs[q].y, x.cs[q].z, x.cs[q].w}, sn[4] = {x.sn[q].x, x.sn[q].y, x.sn[q].z, x.sn[q].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float a = e[q][i], b = e[q + 2][i];
                    e[q][i] = fmaf(a, cs[i], b * -sn[i]);
                    e[q + 2][i] = fmaf(b, cs[i], a * sn[i]);
                }
            }
        }
    }
    // neighbours exchange pieces: an even lane ends up with eight elements of quarter 0 (and 2), an odd one with eight of quarter 1 (and 3)
    const bool odd = (sub & 1) != 0;
    const int at = (odd ? 32 : 0) + 4 * (sub & ~1);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint2 a = make_uint2(ElemTraits<T>::pack2(e[2 * half][0], e[2 * half][1]), ElemTraits<T>::pack2(e[2 * half][2], e[2 * half][3]));
        const uint2 b = make_uint2(ElemTraits<T>::pack2(e[2 * half + 1][0], e[2 * half + 1][1]), ElemTraits<T>::pack2(e[2 * half + 1][2], e[2 * half + 1][3]));
        const uint2 give = odd ? a : b;
        uint2 got;
        got.x = __shfl_xor_sync(0xffffffffu, give.x, 1);
        got.y = __shfl_xor_sync(0xffffffffu, give.y, 1);
        const uint4 w = odd ? make_uint4(got.x, got.y, b.x, b.y) : make_uint4(a.x, a.y, got.x, got.y);
        if (x.dst != nullptr) *reinterpret_cast<uint4*>(x.dst + 64 * half + at) = w;
        else if (EPI == kAllReducePush && x.slot != nullptr) st_tagged(x.slot + 2 * (8 * half + at / 8), w, x.epoch);
    }
}

// ---- few rows: blocks of a cluster share K ------------------------------------------------------------------------------------
// blockIdx.x = tile column * splits + part of K (= rank in the cluster), blockIdx.y = tile row of MT * 128 rows.
// DIRECT: a block with all of K has nothing to add up and takes its tile from TMEM straight to the result (us: 4096 columns, K 128, 128 rows
// 5.5 -> 4.0); not up to 32 rows, which would leave three of four epilogue warps idle (8 rows 3.2 -> 3.7).  An instantiation of its own: with both
// ways in one the sums were slower (39 rows through 768 x 4096 and 4096 x 512 in a pass of 25.2 us: 26.4).
// Otherwise (MT 1) the partial sums go to shared memory as fp32 rows, and block r adds up and finishes the r-th of `splits` runs of rows: every
// block pushes each run by one bulk copy into the shared memory of the block that finishes it, where all that follows is local (rows of 512
// bytes, their 16-byte pieces XOR-swizzled by row: no bank conflicts for the writing threads, each of which has a row, nor for the readers, eight
// lanes a row).  What peers push has a place of its own, for more than 64 rows the ring's last stage with it.  When the sums were fetched from
// the peers' shared memory instead, 10 bytes a clock came in: from the last MMA to a block's end 4.0 us for 64 x 6144, K 4096 with the QKV epilogue (15.8
// us in all, 14.0 now), 3.2 for 64 x 4096 (11.1, 10.0), 5.5 for QKV 128 x 6144 (17.6, 15.7).
template <typename T, int EPI, int MT, bool DIRECT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ GemmParams p, int splits) {
    static_assert(MT == 1 || DIRECT, "sums of 256 rows have no room beside what peers push");
    constexpr int kStageBytes = (MT + 1) * kPanelBytes, kStages = kRingBytes / kStageBytes, kTmemCols = MT * kBN;
    constexpr uint32_t kSumBytes = kBN * 4;           // a row of partial sums
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // (uniform, also to the compiler)
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = smem_base + kBarOffset;
    auto bar_full = [&](int s) { return bars + 8 * s; };
    auto bar_empty = [&](int s) { return bars + 64 + 8 * s; };
    const uint32_t bar_acc = bars + 128, bar_recv = bars + 136;
    volatile int* abort_flag = &s_abort;
    const int rank = static_cast<int>(blockIdx.x) % splits, nt = static_cast<int>(blockIdx.x) / splits;
    const int n0 = nt * kBN, m0 = blockIdx.y * (MT * kBM);
    const int rows = static_cast<int>(min(static_cast<int64_t>(MT * kBM), p.m - m0));   // of the tile that are in C
    const int kb_all = static_cast<int>((p.k + kBK - 1) / kBK);
    const int kb0 = kb_all * rank / splits, kb_count = kb_all * (rank + 1) / splits - kb0;
    // Rows of a run, this block's run, where peers' parts of it come in, and the stages that leaves (a run per block: at most 64 or 128 rows in all)
    const int run = (rows + splits - 1) / splits, own_rows = min(run, rows - rank * run);
    const bool narrow = !DIRECT && splits > 1 && rows > kBM / 2;
    const int stages = narrow ? kStages - 1 : kStages;
    const uint32_t recv = smem_base + (narrow ? (kStages - 1) * kStageBytes : kStageOffset);

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < kStages; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        mbar_init(bar_acc, 1);
        mbar_init(bar_recv, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if (!DIRECT && splits > 1 && own_rows > 0) mbar_expect_tx(bar_recv, (splits - 1) * own_rows * kSumBytes);
    }
    __syncwarp();
    if (!DIRECT && splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");   // (waited for before the push: all barriers are set up)
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    pdl_wait_then_release();   // A comes from the kernel before this one; barriers and TMEM were set up under its tail
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, s_tmem_base, 0);

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int s = 0;
            uint32_t turn = 1;
            for (int i = 0; i < kb_count; ++i) {
                if (i >= stages && !mbar_wait(bar_empty(s), turn, abort_flag, 1)) break;
                mbar_expect_tx(bar_full(s), kPanelBytes + (MT == 1 ? p.a_rows * kBK * 2 : 2 * kPanelBytes));
                const uint32_t at = smem_base + s * kStageBytes;
                tma_load_2d(at + MT * kPanelBytes, &tm_b, (kb0 + i) * kBK, n0, bar_full(s));
#pragma unroll
                for (int t = 0; t < MT; ++t) tma_load_2d(at + t * kPanelBytes, &tm_a, (kb0 + i) * kBK, m0 + t * kBM, bar_full(s));
                if (++s == stages) { s = 0; turn ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t leader = elect_one();
        bool ok = true;
        int s = 0;
        uint32_t turn = 0;
#pragma unroll 1
        for (int i = 0; i < kb_count && ok; ++i) {
            ok = mbar_wait_warp(bar_full(s), turn, abort_flag, 2);
            if (!ok) break;
            tc_fence_after();
            const uint32_t at = smem_base + s * kStageBytes;
            const uint64_t db = make_smem_desc(at + MT * kPanelBytes);
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                const uint64_t da = make_smem_desc(at + t * kPanelBytes);
#pragma unroll
                for (int ks = 0; ks < kBK / 16; ++ks)   // 32 bytes further along the 128-byte row per K step: +2 in the address field
                    umma_ss(leader, tmem_base + t * kBN, da + 2 * ks, db + 2 * ks, p.idesc, (i > 0 || ks > 0) ? 1u : 0u);
            }
            tc_commit(leader, bar_empty(s));
            if (++s == stages) { s = 0; turn ^= 1u; }
        }
        if (ok) tc_commit(leader, bar_acc);
    } else if (warp < 6) {
        // ------------------------------------------------------------------ TMEM -> shared memory: thread = row of the tile
        const int wq = warp & 3;                       // TMEM lanes 32 wq .. 32 wq + 31 belong to this warp
        bool ok = true;
        QkvIndex index[MT];
#pragma unroll
        for (int t = 0; t < MT; ++t) index[t] = DIRECT && EPI == kQkvPrologue ? qkv_index(p, m0 + t * kBM + wq * 32 + lane) : QkvIndex{};
        if (lane == 0) ok = mbar_wait(bar_acc, 0, abort_flag, 3);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        tc_fence_after();
        if (DIRECT && ok) {
            unsigned char* stage = smem_raw + (smem_base - smem_u32(smem_raw)) + kStageOffset + (warp - 2) * 2 * kEpilogueBytes;
#pragma unroll 1
            for (int t = 0; t < MT; ++t)
                if (t * kBM + wq * 32 < rows)
                    epilogue_row<T, EPI, true>(p, tmem_base + (static_cast<uint32_t>(wq * 32) << 16) + t * kBN, m0 + t * kBM + wq * 32 + lane, MT == 2 && t == 1 ? index[MT - 1] : index[0], nt, stage, lane);
        } else if (ok) {
#pragma unroll 1
            for (int c = 0; c < MT * 4; ++c) {
                if ((c >> 2) * kBM + wq * 32 >= rows) break;   // (warp-uniform: no row of this warp is in C)
                const int row_in_tile = (c >> 2) * kBM + wq * 32 + lane;
                uint32_t r[32];
                tmem_ld32(tmem_base + (static_cast<uint32_t>(wq * 32) << 16) + c * 32, r);
                tc_wait_ld();
                reg_fence32(r);
                const uint32_t dst = smem_base + row_in_tile * kSumBytes + (c & 3) * 128;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(dst + ((q ^ (row_in_tile & 7)) * 16)), "r"(r[4 * q]), "r"(r[4 * q + 1]), "r"(r[4 * q + 2]), "r"(r[4 * q + 3]) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // (bulk copies read it)
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        if (*abort_flag) settle();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
    if (DIRECT) return;
    // ---------------------------------------------------------------------- sum over the cluster and epilogue
    const int sub = lane & 7;
    const bool summed = *abort_flag == 0;          // (the same for the whole block)
    if (splits > 1) {
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        if (warp == 2 && lane < splits && lane != rank && summed) {
            const int n = min(run, rows - lane * run);
            if (n > 0) push_bulk(recv + rank * run * kSumBytes, smem_base + lane * run * kSumBytes, n * kSumBytes, bar_recv, lane);
        }
        __syncwarp();
    }
    constexpr int kTrip = kThreads / 8;            // four rows per warp and trip
    int l = warp * 4;
    auto row_of = [&](int first) { return first + (lane >> 3) < own_rows ? m0 + rank * run + first + (lane >> 3) : p.m; };
    auto index_of = [&](int first) { return EPI == kQkvPrologue && first < own_rows ? qkv_index(p, row_of(first)) : QkvIndex{}; };
    QkvIndex at = index_of(l), at_next = index_of(l + kTrip);
    T weights[16];
    octet_weights<T, EPI>(p, nt, sub, weights);
    OctetRow<T> x = octet_row<T, EPI>(p, row_of(l), at, nt, sub);
    bool ok = summed;
    if (splits > 1) {
        if (summed && l < own_rows) ok = mbar_wait_warp(bar_recv, 0, abort_flag, 5);
        asm volatile("barrier.cluster.arrive;\n" ::: "memory");   // what peers pushed here has landed: they need their copies no more
    }
#pragma unroll 1
    for (; ok && l < own_rows; l += kTrip) {
        // the next trip's table rows and the positions of the one after it are on their way under this one (128 x 6144, K 4096, QKV: 0.6 us)
        OctetRow<T> next{};
        if (l + kTrip < own_rows) next = octet_row<T, EPI>(p, row_of(l + kTrip), at_next, nt, sub);
        at_next = index_of(l + 2 * kTrip);
        const int r_own = min(l + (lane >> 3), own_rows - 1), row = rank * run + r_own;
        float4 sum[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) sum[q] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
        for (int r = 0; r < splits; ++r) {
            const unsigned char* from = smem_raw + (r == rank ? smem_base + row * kSumBytes : recv + (r * run + r_own) * kSumBytes) - smem_u32(smem_raw);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 v = *reinterpret_cast<const float4*>(from + (8 * q + (sub ^ (row & 7))) * 16);
                sum[q].x += v.x; sum[q].y += v.y; sum[q].z += v.z; sum[q].w += v.w;
            }
        }
        epilogue_octet<T, EPI>(p, x, sum, weights, nt, sub);
        x = next;
    }
    if (splits > 1) {                              // no block leaves while a peer still reads what it pushed, or may still push
        asm volatile("barrier.cluster.wait;\n" ::: "memory");
        if (*abort_flag) settle();
    }
}

// ---- many rows: persistent pairs of blocks ---------------------------------------------------------------------------------------
constexpr int kPairStages = 6;
constexpr int kHidingSteps = 48;                      // steps of 64 along K under which a slow epilogue of the tile before disappears: some 9 us
constexpr int kPairStageBytes = 2 * kPanelBytes;      // this block's halves of A (128 of 256 rows) and B (128 of 256 columns)
constexpr int kPairCols = 256;                        // accumulator columns of a tile; two of them fill TMEM
template <typename T, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ GemmParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bars = smem_base + kBarOffset;
    auto bar_full = [&](int s) { return bars + 8 * s; };         // used in the leader: both blocks' loads of a stage
    auto bar_empty = [&](int s) { return bars + 64 + 8 * s; };   // in each block: the pair's MMAs have read the stage
    auto bar_acc = [&](int b) { return bars + 128 + 8 * b; };    // in each block: accumulator b is complete
    auto bar_free = [&](int b) { return bars + 144 + 8 * b; };   // in the leader: both blocks have read accumulator b
    volatile int* abort_flag = &s_abort;
    const uint32_t rank = cluster_rank();
    const int kb_count = static_cast<int>((p.k + kBK - 1) / kBK);
    const int tiles = p.tiles_m * p.tiles_n, first = blockIdx.x >> 1, step = gridDim.x >> 1;
    // tiles in column-major order: a wave of pairs shares a few column panels of the weight
    auto row0_of = [&](int tile) { return (tile % p.tiles_m) * 256 + static_cast<int>(rank) * kBM; };
    auto col0_of = [&](int tile) { return (tile / p.tiles_m) * 256; };

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < kPairStages; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar_acc(b), 1); mbar_init(bar_free(b), 16); }   // eight reading warps in each block
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem_base)), "r"(2 * kPairCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    pdl_wait_then_release();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the other block's barriers are set up
    tc_fence_after();
    const uint32_t tmem_base = s_tmem_base;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer of this block's halves
        if (lane == 0) {
            bool ok = true;
            int it = 0;
            for (int tile = first; tile < tiles && ok; tile += step) {
                const int m0 = row0_of(tile), n0 = col0_of(tile) + static_cast<int>(rank) * kBN;
                for (int kb = 0; kb < kb_count && ok; ++kb, ++it) {
                    const int s = it % kPairStages;
                    if (it >= kPairStages) ok = mbar_wait(bar_empty(s), ((it / kPairStages) & 1) ^ 1, abort_flag, 1);
                    if (!ok) break;
                    if (rank == 0) mbar_expect_tx(bar_full(s), 2 * kPairStageBytes);
                    const uint32_t at = smem_base + s * kPairStageBytes, full = in_block(bar_full(s), 0);
                    tma_load_2d_pair(at, &tm_a, kb * kBK, m0, full);
                    tma_load_2d_pair(at + kPanelBytes, &tm_b, kb * kBK, n0, full);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer, for both blocks
        if (lane == 0 && rank == 0) {
            bool ok = true;
            int it = 0, n = 0;
            for (int tile = first; tile < tiles && ok; tile += step, ++n) {
                const int b = n & 1;
                if (n >= 2) ok = mbar_wait(bar_free(b), ((n >> 1) & 1) ^ 1, abort_flag, 4);
                if (!ok) break;
                tc_fence_after();
                for (int kb = 0; kb < kb_count; ++kb, ++it) {
                    const int s = it % kPairStages;
                    ok = mbar_wait(bar_full(s), (it / kPairStages) & 1, abort_flag, 2);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t da = make_smem_desc(smem_base + s * kPairStageBytes), db = make_smem_desc(smem_base + s * kPairStageBytes + kPanelBytes);
#pragma unroll
                    for (int ks = 0; ks < kBK / 16; ++ks)
                        umma_ss_pair(tmem_base + b * kPairCols, da + 2 * ks, db + 2 * ks, p.idesc, (kb > 0 || ks > 0) ? 1u : 0u);
                    tc_commit_pair(bar_empty(s));
                }
                if (ok) tc_commit_pair(bar_acc(b));
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue: thread = row, warps 2-5 the first 128 columns of
        // the tile, 6-9 the second (with one tile per pair nothing hides it: 500 rows of QKV took 10 us longer than the plain product)
        const int wq = warp & 3, half = warp >= 6 ? 1 : 0;
        int n = 0;
        for (int tile = first; tile < tiles; tile += step, ++n) {
            const int b = n & 1;
            const int64_t row = row0_of(tile) + wq * 32 + lane;
            const QkvIndex index = EPI == kQkvPrologue ? qkv_index(p, row) : QkvIndex{};   // (a trip to memory before the accumulator is there)
            bool ok = true;
            if (lane == 0) ok = mbar_wait(bar_acc(b), (n >> 1) & 1, abort_flag, 3);
            if (__shfl_sync(0xffffffffu, ok ? 1 : 0, 0) == 0) break;
            tc_fence_after();
            const uint32_t t_row = tmem_base + b * kPairCols + (static_cast<uint32_t>(wq * 32) << 16);
            const int nt = col0_of(tile) / kBN + half;
            unsigned char* stage = smem_raw + (smem_base - smem_u32(smem_raw)) + kStageOffset + (warp - 2) * kEpilogueBytes;
            if (nt * kBN < p.n) epilogue_row<T, EPI, false>(p, t_row + half * kBN, row, index, nt, stage, lane, kb_count >= kHidingSteps && tile + step < tiles);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_block(bar_free(b), 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1 && *abort_flag) settle();
    cluster_sync_all();   // neither block leaves while the other may still signal its barriers or read its operands
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(2 * kPairCols) : "memory");
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
// [rows, k] 16-bit row-major -> boxes of `box_rows` rows x 64 elements, 128-byte swizzle; rows past the end read as zeros
bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t k, bool bf16, int box_rows = kBM) {
    EncodeFn fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {kBK, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims,
              strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
uint32_t make_idesc(bool bf16, int m, int n) {   // kind::f16: D = F32, A / B = F16 or BF16 (both K-major)
    const uint32_t fmt = bf16 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// Kernel and shape for a size, by what the slowest SM does: waves of blocks times (steps of 64 along K and a fixed part).  The microseconds
// are fitted to all ways at 1 to 5000 rows x 768 to 8192 columns, K 512 to 4096, with both epilogues (replayed graphs over weights larger than L2).  A
// step costs 32 or 48 KiB out of L2, the bound here, not the tensor pipe (32 KiB per SM for a pair's 256 x 256 tile).  The fixed part (launch,
// first loads, epilogue; with the sum over the cluster also in proportion to the tile's rows) comes with every wave of blocks, that of a
// pair's tile is hidden but for the epilogue.  One rule for all epilogues, so that they round the same sums: for plain products the choice is 0.7 %
// slower than the fastest way on average and 22 % at most (128 x 1536, K 1024, 7.2 us, one block with all of K 5.9), with the QKV epilogue 1.3 % and
// 41 % (48 x 8192, K 512, 9.0 us, clusters of 2 6.4).  A part of K has two steps at least.  Blocks of 256 rows that share K in clusters were never the
// fastest by more than 2 % once peers' sums were pushed (256 x 4096, K 4096: 17.8 us in clusters of 4, 13.9 as two tiles in clusters of 2).
struct GemmShape { int mt, splits; };   // mt 1 or 2: gemm_split_kernel; 0: gemm_pair_kernel
GemmShape choose_gemm(int64_t m, int64_t n, int64_t k) {
    // clusters: what a B200 holds at once (its GPCs have 16 to 20 SMs); rows: per 128 rows of a tile
    struct { int mt, splits, clusters; double step, fixed, rows; } constexpr kWays[] = {
        {1, 1, 148, 0.207, 3.0, 0.85}, {1, 2, 74, 0.24, 3.3, 2.0}, {1, 4, 33, 0.288, 3.1, 2.3}, {1, 8, 15, 0.333, 3.0, 2.75}, {2, 1, 148, 0.345, 5.3, 0.25}};
    const int64_t kb = (k + kBK - 1) / kBK, tiles_n = n / kBN, pair_tiles = ((m + 255) / 256) * ((n + 255) / 256);
    GemmShape best{0, 1};
    double best_time = m > kBM ? static_cast<double>((pair_tiles + 73) / 74) * (static_cast<double>(kb) * 0.321 + 2.0) + 5.3 : 1e30;
    for (const auto& w : kWays) {
        const int64_t tile_rows = w.mt * kBM, tiles = (m + tile_rows - 1) / tile_rows * tiles_n;
        if ((w.mt == 2 && m <= kBM) || (w.splits > 1 && (kb / w.splits < 2 || tiles > w.clusters))) continue;
        const double rows = static_cast<double>(m < tile_rows ? m : tile_rows) / kBM;
        const double time = static_cast<double>((tiles + w.clusters - 1) / w.clusters) *
                            (static_cast<double>((kb + w.splits - 1) / w.splits) * w.step + w.fixed + w.rows * rows);
        if (time < best_time) { best_time = time; best = GemmShape{w.mt, w.splits}; }
    }
    return best;
}

template <typename... KArgs>
int launch_kernel(void (*kernel)(KArgs...), std::atomic<bool>* attr_done, dim3 grid, int threads, int cluster, cudaStream_t stream, const char* what,
                  KArgs... args) {
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 0 && device < 64 && !attr_done[device]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "%s: cudaFuncSetAttribute: %s", what, cudaGetErrorString(e));
        attr_done[device] = true;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 0 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
    return check_launch(what);
}

template <typename T, int EPI>
int launch(const void* a, const void* b, GemmParams& p, bool bf16, cudaStream_t stream, const char* what) {
    static std::atomic<bool> done[4][64] = {};
    CUtensorMap ta, tb;
    const GemmShape g = choose_gemm(p.m, p.n, p.k);
    p.a_rows = g.mt == 1 && p.m < kBM ? static_cast<int>((p.m + 7) / 8 * 8) : kBM;
    if (!make_map(&ta, a, p.m, p.k, bf16, p.a_rows) || !make_map(&tb, b, p.n, p.k, bf16))
        return fail(NVK_ERR_CUDA, "%s: cuTensorMapEncodeTiled failed", what);
    if (g.mt == 0) {
        p.idesc = make_idesc(bf16, 256, 256);
        p.tiles_m = static_cast<int>((p.m + 255) / 256);
        p.tiles_n = static_cast<int>((p.n + 255) / 256);
        const int64_t pairs = static_cast<int64_t>(p.tiles_m) * p.tiles_n;
        return launch_kernel(gemm_pair_kernel<T, EPI>, done[0], dim3(static_cast<unsigned>(2 * (pairs < kSmCount / 2 ? pairs : kSmCount / 2))), kPairThreads, 0,
                             stream, what, ta, tb, p);
    }
    p.idesc = make_idesc(bf16, kBM, kBN);
    const dim3 grid(static_cast<unsigned>(p.n / kBN * g.splits), static_cast<unsigned>((p.m + g.mt * kBM - 1) / (g.mt * kBM)));
    const bool direct = g.splits == 1 && p.m > 32;
    auto* kernel = g.mt == 2 ? gemm_split_kernel<T, EPI, 2, true> : direct ? gemm_split_kernel<T, EPI, 1, true> : gemm_split_kernel<T, EPI, 1, false>;
    return launch_kernel(kernel, done[g.mt == 2 ? 3 : 1 + direct], grid, kThreads, g.splits, stream, what, ta, tb, p, g.splits);
}

int check_gemm(const char* what, const void* a, const void* b, int64_t m, int64_t n, int64_t k, int dtype) {
    if (!a || !b) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: input and weight must be defined", what);
    if (dtype != NVK_F16 && dtype != NVK_BF16) return fail(NVK_ERR_UNSUPPORTED, "%s: dtype must be F16 or BF16", what);
    if (m <= 0 || n <= 0 || k <= 0) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: sizes must be positive", what);
    if (n % kBN != 0) return fail(NVK_ERR_UNSUPPORTED, "%s: the output width must be a multiple of %d", what, kBN);
    if (k % 8 != 0) return fail(NVK_ERR_UNSUPPORTED, "%s: the inner size must be a multiple of 8 (16-byte rows)", what);
    if (!aligned_to(a, 16) || !aligned_to(b, 16)) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: input and weight must be 16-byte aligned", what);
    if (m >= (1LL << 31) || n >= (1LL << 31) || (m + kBM - 1) / kBM > 65535) return fail(NVK_ERR_UNSUPPORTED, "%s: too large", what);
    if (encode_fn() == nullptr) return fail(NVK_ERR_UNSUPPORTED, "%s: cuTensorMapEncodeTiled is not available", what);
    return NVK_OK;
}

}  // namespace
}  // namespace nvk

using namespace nvk;

extern "C" int nvk_linear(const void* x, const void* weight, void* out, int64_t rows, int64_t out_features, int64_t in_features,
                          int dtype, void* stream) {
    const char* what = "linear";
    const int rc = check_gemm(what, x, weight, rows, out_features, in_features, dtype);
    if (rc != NVK_OK) return rc;
    if (!out || !aligned_to(out, 16)) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: the output must be defined and 16-byte aligned", what);
    GemmParams p{};
    p.out = out; p.m = rows; p.n = out_features; p.k = in_features;
    return dtype == NVK_BF16 ? launch<__nv_bfloat16, kPlain>(x, weight, p, true, static_cast<cudaStream_t>(stream), what)
                             : launch<__half, kPlain>(x, weight, p, false, static_cast<cudaStream_t>(stream), what);
}

extern "C" int nvk_qkv_linear_norm_rope_store(const void* x, const void* qkv_weight, int64_t rows, int64_t in_features,
                                              const int32_t* positions, const void* q_norm_weight, const void* k_norm_weight,
                                              float norm_eps, const float* cos_sin_cache, int64_t max_positions,
                                              const int32_t* slot_mapping, void* k_cache, void* v_cache, int64_t cache_rows,
                                              int num_q_heads, int num_kv_heads, int head_dim, void* q_out, int dtype, void* stream) {
    const char* what = "qkv linear + norm + rope + store";
    if (head_dim != kBN) return fail(NVK_ERR_UNSUPPORTED, "%s: head_dim must be %d (one GEMM tile per head)", what, kBN);
    if (num_q_heads <= 0 || num_kv_heads <= 0 || max_positions <= 0 || cache_rows <= 0)
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: sizes must be positive", what);
    const int64_t n = static_cast<int64_t>(num_q_heads + 2 * num_kv_heads) * head_dim;
    const int rc = check_gemm(what, x, qkv_weight, rows, n, in_features, dtype);
    if (rc != NVK_OK) return rc;
    if (!positions || !cos_sin_cache || !k_cache || !v_cache || !q_out)
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: positions, the rotary table, the caches and q_out must be defined", what);
    if ((q_norm_weight == nullptr) != (k_norm_weight == nullptr))
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: q_norm_weight and k_norm_weight go together", what);
    if (!aligned_to(q_out, 16) || !aligned_to(k_cache, 16) || !aligned_to(v_cache, 16))
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: q_out and the caches must be 16-byte aligned", what);
    GemmParams p{};
    p.m = rows; p.n = n; p.k = in_features;
    p.positions = positions; p.q_weight = q_norm_weight; p.k_weight = k_norm_weight; p.cos_sin = cos_sin_cache; p.table_vec = aligned_to(cos_sin_cache, 16);
    p.slot_mapping = slot_mapping; p.q_out = q_out; p.k_cache = k_cache; p.v_cache = v_cache; p.cache_rows = cache_rows;
    p.max_positions = static_cast<int>(max_positions); p.hq = num_q_heads; p.hkv = num_kv_heads; p.eps = norm_eps;
    return dtype == NVK_BF16 ? launch<__nv_bfloat16, kQkvPrologue>(x, qkv_weight, p, true, static_cast<cudaStream_t>(stream), what)
                             : launch<__half, kQkvPrologue>(x, qkv_weight, p, false, static_cast<cudaStream_t>(stream), what);
}

namespace {
// The GEMM of a row-parallel linear on rank `rank`, its result rows delivered to the ranks that reduce them.
int launch_row_linear_push(const char* what, const void* x, const void* weight, int64_t rows, int64_t out_features, int64_t in_features,
                           void* addend, void* const* stage_ptrs, size_t stage_bytes, const void* flags, int rank, int world, int dtype,
                           cudaStream_t stream) {
    const int rc = check_gemm(what, x, weight, rows, out_features, in_features, dtype);
    if (rc != NVK_OK) return rc;
    if (world < 2 || world > kMaxRanks || rank < 0 || rank >= world)
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: world must be 2..%d and rank inside it", what, kMaxRanks);
    if (rows % world != 0) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: rows must be a multiple of world", what);
    if (!addend || !stage_ptrs || !flags || !aligned_to(addend, 16))
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: the addend buffer, the staging table and the flag area must be defined", what);
    if (stage_bytes < nvk_tp_allreduce_stage_bytes(rows * out_features))
        return fail(NVK_ERR_INVALID_ARGUMENT, "%s: staging areas of %zu bytes given, %zu needed", what, stage_bytes,
                    nvk_tp_allreduce_stage_bytes(rows * out_features));
    GemmParams p{};
    p.m = rows; p.n = out_features; p.k = in_features;
    p.addend = addend; p.flags = static_cast<const uint32_t*>(flags); p.rank = rank; p.world = world;
    for (int r = 0; r < world; ++r) {
        // (tagged vectors are stored 32 bytes at a time)
        if (!stage_ptrs[r] || !aligned_to(stage_ptrs[r], 32))
            return fail(NVK_ERR_INVALID_ARGUMENT, "%s: the staging area of rank %d is missing or not 32-byte aligned", what, r);
        p.stage[r] = static_cast<uint4*>(stage_ptrs[r]);
    }
    return dtype == NVK_BF16 ? launch<__nv_bfloat16, kAllReducePush>(x, weight, p, true, stream, what)
                             : launch<__half, kAllReducePush>(x, weight, p, false, stream, what);
}
}  // namespace

extern "C" int nvk_tp_row_linear_allreduce_add_rmsnorm(const void* x, const void* weight, int64_t rows, int64_t out_features,
                                                       int64_t in_features, void* addend, void* out, void* norm,
                                                       void* const* stage_ptrs, size_t stage_bytes, void* flags, const void* residual,
                                                       const void* norm_weight, float eps, int rank, int world, int dtype, void* stream) {
    const char* what = "row-parallel linear + all-reduce + add + rmsnorm";
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (out_features > 8192) return fail(NVK_ERR_UNSUPPORTED, "%s: at most 8192 output features", what);
    int rc = launch_row_linear_push(what, x, weight, rows, out_features, in_features, addend, stage_ptrs, stage_bytes, flags, rank, world, dtype, st);
    if (rc != NVK_OK) return rc;
    return launch_allreduce_add_rmsnorm(addend, out, norm, stage_ptrs, stage_bytes, flags, residual, norm_weight, eps, rank, world,
                                        static_cast<int>(rows), static_cast<int>(out_features), dtype, /*pushed=*/true, st);
}

extern "C" int nvk_tp_row_linear_allreduce_add_rmsnorm_inprocess(const void* const* x_ptrs, const void* const* weight_ptrs, int64_t rows,
                                                                 int64_t out_features, int64_t in_features, void* const* addend_ptrs,
                                                                 void* const* out_ptrs, void* const* norm_ptrs, void* const* stage_ptrs,
                                                                 size_t stage_bytes, void* const* flag_ptrs,
                                                                 const void* const* residual_ptrs, const void* norm_weight, float eps,
                                                                 int world, int dtype, void* stream) {
    const char* what = "row-parallel linear + all-reduce + add + rmsnorm (in-process)";
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!x_ptrs || !weight_ptrs || !addend_ptrs || !flag_ptrs) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: pointer tables must be defined", what);
    if (world < 2 || world > kMaxRanks) return fail(NVK_ERR_INVALID_ARGUMENT, "%s: world must be 2..%d", what, kMaxRanks);
    if (out_features > 8192) return fail(NVK_ERR_UNSUPPORTED, "%s: at most 8192 output features", what);
    for (int r = 0; r < world; ++r) {   // the ranks' GEMMs wait for nobody: one launch after the other
        const int rc = launch_row_linear_push(what, x_ptrs[r], weight_ptrs[r], rows, out_features, in_features, addend_ptrs[r], stage_ptrs,
                                              stage_bytes, flag_ptrs[r], r, world, dtype, st);
        if (rc != NVK_OK) return rc;
    }
    return launch_allreduce_inprocess(const_cast<const void* const*>(reinterpret_cast<void* const*>(addend_ptrs)), out_ptrs, norm_ptrs,
                                      stage_ptrs, stage_bytes, flag_ptrs, residual_ptrs, norm_weight, eps, world, static_cast<int>(rows),
                                      static_cast<int>(out_features), dtype, /*pushed=*/true, st);
}

extern "C" int nvk_gemm_status(void* stream, int* status) {
    if (!status) return fail(NVK_ERR_INVALID_ARGUMENT, "gemm status: null argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int word = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(&word, g_gemm_error, sizeof(int), 0, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && word != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbolAsync(g_gemm_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "gemm status: %s", cudaGetErrorString(e));
    *status = word;
    return NVK_OK;
}
