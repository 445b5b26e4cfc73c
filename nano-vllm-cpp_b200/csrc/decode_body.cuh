// Device code of paged decode attention on tensor cores (F16 / BF16 queries, head_dim 128; 16-bit, int8 or e4m3 cache), shared
// by the decode kernels (decode_attn.cu) and the mixed prefill + decode kernel (prefill_attn_tc.cu).
//
// The op is HBM-bound: every K and V row of every context is read once.  A group of four warps takes a range of the keys of one
// (sequence, KV head); the G = Hq / Hkv <= 8 query heads of the KV head are the columns of the MMA tile, so a K / V row is read once
// per KV head.  Each warp streams every fourth tile of 16 keys through a private ring of cp.async stages (no barrier in the main
// loop); at the end the four warps merge through shared memory.
//
// Three ways to share a sequence out, by the sizes the host knows:
//   chunks     ranges of `chunk_tokens` keys; where a context is longer than one, the ranges leave partial results (maximum, sum,
//              unnormalised output) in the workspace and a second kernel merges them;
//   per_seq    num_splits equal ranges of every sequence in one thread-block cluster, merged through distributed shared memory in
//              the same launch, without a workspace: for small steps;
//   halves     two chunks, each half of the table's row, in one cluster: a context that ends in the first is one block's alone.
//
// Cutting the whole batch's keys into equal runs that ignore sequence boundaries (each block sums up the contexts, warps or groups
// walk on from one sequence to the next with their rings full, a quarter of the work handed out dynamically) was built and measured:
// the main loop gains 2 to 15 %, but the pass over the contexts, the look-ups and three to eight partial results per sequence
// cost more: 48 us against 37 at 37 sequences of 100 to 2048 keys, 700 against 697 at 256 of 1024 to 8192.
#pragma once

#include "nvk_internal.cuh"

namespace nvk {
namespace dec {

constexpr int kHeadDim = 128;
constexpr int kTileTokens = 16;
constexpr int kMaxGroup = 8;           // query heads per KV head
constexpr int kGroupWarps = 4;
constexpr int kGroupThreads = kGroupWarps * 32;
constexpr int kMergeWarps = 8;         // warps that merge the parts of one (sequence, head) where there are many

struct DecodeParams {
    const void* q; const void* k_cache; const void* v_cache;
    const __half* k_scale; const __half* v_scale;      // 8-bit caches
    IndexArray context_lens; IndexArray block_tables;
    void* out; float* ws_o; float2* ws_ml;             // partial results: [sequence][KV head][split][group][128] and (maximum, sum)
    int64_t max_blocks, num_cache_blocks;
    int batch, num_heads, num_kv_heads, group, block_size;
    int chunk_tokens, num_splits;
    int per_seq;                                       // 1: num_splits equal ranges per sequence instead of chunks
    int longest_first;                                 // blocks take the sequences in order of falling context length
    int chunk_major;                                   // decode_split_kernel's grid: all sequences' first chunks, then all second ones, ...
    int split_shift;                                   // clusters: log2 of num_splits
    int beside;                                        // waits at its end (pdl_wait_beside)
    FastDiv by_block, by_kv_heads;
    float scale_log2;
};

// A context length, limited to what the block table can address (max_blocks * block_size), and not negative.
__device__ __forceinline__ int clamped_context(const DecodeParams& p, IndexArray::Raw raw) {
    const int64_t ctx = p.context_lens.value(raw);
    const int64_t cap = p.max_blocks * p.block_size;
    return static_cast<int>(ctx < 0 ? 0 : ctx < cap ? ctx : cap);
}
__device__ __forceinline__ int clamped_context(const DecodeParams& p, int b) { return clamped_context(p, p.context_lens.raw(b)); }
// Range i of a context has keys [i * len, min(ctx, (i + 1) * len)).
__device__ __forceinline__ int range_len(const DecodeParams& p, int ctx) {
    return p.per_seq ? (((ctx + p.num_splits - 1) >> p.split_shift) + kTileTokens - 1) / kTileTokens * kTileTokens : p.chunk_tokens;
}
// Lane i: entry base + i of a sequence's block table, as loaded.  Entries past the context are loaded and not used.
__device__ __forceinline__ IndexArray::Raw load_ids(const DecodeParams& p, int b, int base, int lane) {
    return p.block_tables.raw(b * p.max_blocks + base + lane, base + lane < p.max_blocks);
}

__device__ __forceinline__ void group_sync(int bar_id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(bar_id), "r"(threads) : "memory"); }

// ---- cache formats: how a tile is fetched and what a warp does with it ---------------------------------------------------
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void lds32x4(uint32_t addr, uint32_t (&w)[4]) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
}

// 8 x 8 matrix of 16-bit elements over a warp (lane (g, t): row g, columns 2t, 2t + 1), transposed.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}

// Online-softmax state of a warp.  Lane (g, t) = (lane / 4, lane % 4) holds heads 2t and 2t + 1: columns of the accumulators, the
// maxima (equal over g) and, over the keys that the lane has seen, the sums.
struct SoftmaxState {
    float o[8][4];
    float m[2], l[2];
    __device__ __forceinline__ void reset() {
#pragma unroll
        for (int i = 0; i < 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f; }
        m[0] = m[1] = -INFINITY; l[0] = l[1] = 0.0f;
    }
    // Scores of a tile: rescale where a maximum moves (a handful of tiles of a sequence; the branch is warp-uniform).  `extra`: further
    // columns that are scaled along.
    __device__ __forceinline__ void raise_max(const float (&sc)[4], float* extra) {
        float top[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])};
        if (__any_sync(0xffffffffu, top[0] > m[0] || top[1] > m[1])) {
            float c[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int x = 4; x < 32; x *= 2) top[h] = fmaxf(top[h], __shfl_xor_sync(0xffffffffu, top[h], x));
                const float m_new = fmaxf(m[h], top[h]);   // finite: the tile's first key is always valid
                c[h] = fast_exp2(m[h] - m_new);
                l[h] *= c[h];
                m[h] = m_new;
            }
#pragma unroll
            for (int mt = 0; mt < 8; ++mt) { o[mt][0] *= c[0]; o[mt][1] *= c[1]; o[mt][2] *= c[0]; o[mt][3] *= c[1]; }
            if (extra != nullptr) { extra[0] *= c[0]; extra[1] *= c[1]; extra[2] *= c[0]; extra[3] *= c[1]; }
        }
    }
};

// Scores of lane (g, t): keys g (sc[0], sc[1]) and g + 8 (sc[2], sc[3]), heads 2t and 2t + 1 of each.  Keys past `valid` of a tile get no
// weight; only a sequence's last tile has any (warp-uniform branch).
__device__ __forceinline__ void mask_scores(float (&sc)[4], int g, int valid) {
    if (valid < kTileTokens) {
        if (g >= valid) sc[0] = sc[1] = -INFINITY;
        if (g + 8 >= valid) sc[2] = sc[3] = -INFINITY;
    }
}

// 16-bit cache.  K and V tiles of 16 x 256 bytes, XOR-swizzled by row; S^T = K Q^T as mma.sync m16n8k16: the 16 keys are the rows,
// the (zero padded) query heads the 8 columns; O^T = V^T P^T with V^T taken straight from the row-major V tile by ldmatrix.trans and
// P^T from S^T by two 8 x 8 transposes.  (Heads as the 16 rows need no transpose but twice the MMAs, half of them on padding, in a
// chain twice as long.)  Even and odd k-steps have accumulators of their own: a step is a serial chain that few warps hide.
// Measured: 37 sequences of up to 2048 keys 34.8 -> 33.7 us; 100 int8 ones of up to 4096, where the step is closer to the bound, 97 -> 89.
// 8 warps per SM x 3 stages of 8 KiB: 128 KiB in flight.
template <typename T>
struct Cache16 {
    static constexpr int kGroups = 2;   // resident per SM
    static constexpr int kRowBytes = kHeadDim * 2;
    static constexpr int kTileBytes = kTileTokens * kRowBytes;
    static constexpr int kStageBytes = 2 * kTileBytes;
    static constexpr int kStages = 3;
    static constexpr int kPartStride = kHeadDim + 8;

    SoftmaxState s;
    uint32_t qa[8][2];   // head g of the 8-column B tile; zero from head G on

    __device__ __forceinline__ void start(const DecodeParams& p, int b, int kvh, int lane) {
        const int g = lane >> 2, t = lane & 3;
        const bool live = g < p.group;
        const uint32_t* row = reinterpret_cast<const uint32_t*>(
            static_cast<const T*>(p.q) + (static_cast<int64_t>(b) * p.num_heads + kvh * p.group + (live ? g : 0)) * kHeadDim);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            qa[ks][0] = live ? row[ks * 8 + t] : 0u;
            qa[ks][1] = live ? row[ks * 8 + 4 + t] : 0u;
        }
        s.reset();
    }
    // Rows row0 .. row0 + valid - 1 of the cache into a stage; the rest of the tile is zero-filled (stale cache contents, even NaN,
    // never reach the arithmetic).
    static __device__ __forceinline__ void issue(const DecodeParams& p, int kvh, int64_t row0, int valid, uint32_t stage, int lane) {
        const size_t stride = static_cast<size_t>(p.num_kv_heads) * kRowBytes;
        const int c = lane & 15, rhalf = lane >> 4;   // 16-byte piece c of rows 2 i + rhalf
        const size_t base = static_cast<size_t>(row0) * stride + static_cast<size_t>(kvh) * kRowBytes + c * 16;
        const unsigned char* kc = static_cast<const unsigned char*>(p.k_cache) + base;
        const unsigned char* vc = static_cast<const unsigned char*>(p.v_cache) + base;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 2 * i + rhalf;
            const int bytes = r < valid ? 16 : 0;
            const size_t src = bytes ? r * stride : 0;
            const uint32_t dst = stage + r * kRowBytes + ((c ^ (r & 7)) << 4);
            cp_async16(dst, kc + src, bytes);
            cp_async16(dst + kTileBytes, vc + src, bytes);
        }
    }
    __device__ __forceinline__ void step(const DecodeParams& p, uint32_t stage, int valid, int /*kvh*/, int lane) {
        // ldmatrix lane addressing.  K: matrices (tok 0-7, d lo), (tok 0-7, d hi), (tok 8-15, d lo), (tok 8-15, d hi) of one
        // 16-wide k-step.  V (transposed): the same of one 16-wide d-tile.
        const int row = ((lane >> 4) << 3) + (lane & 7), sel = (lane >> 3) & 1;
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            uint32_t k0, k1, k2, k3;
            ldmatrix_x4(k0, k1, k2, k3, stage + row * kRowBytes + (((2 * ks + sel) ^ (row & 7)) << 4));
            mma_16816<T>(ks & 1 ? s1 : s0, k0, k2, k1, k3, qa[ks][0], qa[ks][1]);
        }
        float sc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[i] = (s0[i] + s1[i]) * p.scale_log2;
        mask_scores(sc, lane >> 2, valid);
        s.raise_max(sc, nullptr);
        const float p0 = fast_exp2(sc[0] - s.m[0]), p1 = fast_exp2(sc[1] - s.m[1]), p2 = fast_exp2(sc[2] - s.m[0]), p3 = fast_exp2(sc[3] - s.m[1]);
        s.l[0] += p0 + p2;
        s.l[1] += p1 + p3;
        const uint32_t pb0 = transpose_8x8(ElemTraits<T>::pack2(p0, p1)), pb1 = transpose_8x8(ElemTraits<T>::pack2(p2, p3));
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) {
            uint32_t a0, a1, a2, a3;
            ldmatrix_x4_trans(a0, a1, a2, a3, stage + kTileBytes + row * kRowBytes + (((2 * mt + sel) ^ (row & 7)) << 4));
            mma_16816<T>(s.o[mt], a0, a1, a2, a3, pb0, pb1);
        }
    }
    // The warp's unnormalised output of head 2t + h.
    __device__ __forceinline__ void write_part(float* row, int h, int g) const {
#pragma unroll
        for (int i = 0; i < 16; ++i) row[8 * i + g] = s.o[i >> 1][(i & 1) * 2 + h];
    }
};

// Two 8-bit cache elements -> two f16 (MMA operand halves).  int8: the byte glued under the exponent byte of 1024 (the word has
// had its sign bits flipped: value + 1152, taken out algebraically afterwards); e4m3: the hardware conversion, exact.
template <bool FP8> __device__ __forceinline__ uint32_t widen_pair_lo(uint32_t x) {   // bytes 0, 1
    if constexpr (FP8) {
        uint32_t d;
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;\n" : "=r"(d) : "h"(static_cast<unsigned short>(x & 0xffffu)));
        return d;
    } else {
        return __byte_perm(x, 0x64646464u, 0x4140);
    }
}
template <bool FP8> __device__ __forceinline__ uint32_t widen_pair_hi(uint32_t x) {   // bytes 2, 3
    if constexpr (FP8) {
        uint32_t d;
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;\n" : "=r"(d) : "h"(static_cast<unsigned short>(x >> 16)));
        return d;
    } else {
        return __byte_perm(x, 0x64646464u, 0x4342);
    }
}

// 8-bit cache (int8, the reference's format: src/kernels/attention.cu:746-842; or e4m3 of the same layout): per token and KV head
// 128 bytes of K, 128 of V and two fp16 scales.  The MMA fragments are built from the bytes in registers -- no widened copy in
// shared memory, no ldmatrix:
//   * an int8 x becomes the fp16 number 1024 + (x + 128) by gluing the byte (x ^ 0x80) under the exponent byte 0x64 (one PRMT per
//     pair); the constant 1152 is taken out afterwards: q . (k' - 1152) = q . k' - 1152 * sum(q), and P (v' - 1152) = P v' - 1152 *
//     sum(P), where sum(P) comes from one extra MMA per tile against a row of ones, i.e. from exactly the rounded probabilities the
//     other MMAs used;
//   * the MMAs contract over d (scores) and over keys (output); a contraction does not care in which order its index runs, and
//     neither does the output care which accumulator row holds which d, so every lane takes whole 16-byte pieces: for K, piece 4q + t
//     of key row g supplies its k-steps 4q .. 4q + 3 (the query fragment is loaded with the same permutation); for V, piece g of key
//     rows 2t, 2t+1, 2t+8, 2t+9 supplies all eight d-tiles after a byte interleave of row pairs (two PRMTs), and accumulator row g /
//     g + 8 of d-tile 2a + e holds d = 16 g + 4 a + 2 e (+ 1);
//   * pieces are XOR-swizzled in the ring so that those 16-byte reads are conflict free.
// The scales never touch the tiles: k_scale multiplies the score of its key after the first MMA, v_scale the probability of its key
// before the second (the row sum uses the unscaled probability).  MMAs run as f16 whatever the query type: the query is converted
// once, probabilities are <= 1.  12 warps per SM x 4 stages of 4.1 KiB: 148 KiB in flight.
template <typename T, bool FP8>
struct Cache8 {
    static constexpr int kGroups = 3;
    static constexpr int kRowBytes = kHeadDim;
    static constexpr int kTileBytes = kTileTokens * kRowBytes;
    static constexpr int kScaleBytes = 2 * kTileTokens * 4;   // one 32-bit word per (K | V, token): the word that holds its fp16 scale
    static constexpr int kStageBytes = 2 * kTileBytes + kScaleBytes;
    static constexpr int kStages = 4;
    static constexpr int kPartStride = kHeadDim + 4;
    static constexpr float kOffset = FP8 ? 0.0f : 1152.0f;    // 1024 (exponent glue) + 128 (sign flip)
    static constexpr uint32_t kFlip = FP8 ? 0u : 0x80808080u; // int8: sign bits flipped before the glue

    SoftmaxState s;
    float osum[4];       // sum of the (scaled, rounded) probabilities per head, from the ones-row MMA
    float q_off[2];
    uint32_t qa[8][2];   // k-step ks = 4 q + w, positions {2t, 2t+1 | 2t+8, 2t+9} <- d = 64 q + 16 t + 4 w + {0, 1 | 2, 3}

    __device__ __forceinline__ void start(const DecodeParams& p, int b, int kvh, int lane) {
        const int g = lane >> 2, t = lane & 3;
        const bool live = g < p.group;
        const T* row = static_cast<const T*>(p.q) + (static_cast<int64_t>(b) * p.num_heads + kvh * p.group + (live ? g : 0)) * kHeadDim;
        float qsum = 0.0f;   // of the f16-rounded query row g
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const int d0 = 64 * (ks >> 2) + 16 * t + 4 * (ks & 3);
#pragma unroll
            for (int hlf = 0; hlf < 2; ++hlf) {
                const __half2 h2 = __floats2half2_rn(ElemTraits<T>::to_float(row[d0 + 2 * hlf]), ElemTraits<T>::to_float(row[d0 + 2 * hlf + 1]));
                qa[ks][hlf] = live ? *reinterpret_cast<const uint32_t*>(&h2) : 0u;
                if (live) qsum += __low2float(h2) + __high2float(h2);
            }
        }
        qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
        qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
        q_off[0] = kOffset * __shfl_sync(0xffffffffu, qsum, 8 * t);
        q_off[1] = kOffset * __shfl_sync(0xffffffffu, qsum, 8 * t + 4);
        osum[0] = osum[1] = osum[2] = osum[3] = 0.0f;
        s.reset();
    }
    static __device__ __forceinline__ void issue(const DecodeParams& p, int kvh, int64_t row0, int valid, uint32_t stage, int lane) {
        const size_t stride = static_cast<size_t>(p.num_kv_heads) * kRowBytes;
        const int c = lane & 7, rq = lane >> 3;   // 16-byte piece c of rows 4 i + rq; ring swizzles: K piece c ^ ((r & 1) << 2), V piece c ^ (r & 6)
        const size_t base = static_cast<size_t>(row0) * stride + static_cast<size_t>(kvh) * kRowBytes + c * 16;
        const unsigned char* kc = static_cast<const unsigned char*>(p.k_cache) + base;
        const unsigned char* vc = static_cast<const unsigned char*>(p.v_cache) + base;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * i + rq;
            const int bytes = r < valid ? 16 : 0;
            const size_t src = bytes ? r * stride : 0;
            cp_async16(stage + r * kRowBytes + ((c ^ ((r & 1) << 2)) << 4), kc + src, bytes);
            cp_async16(stage + kTileBytes + r * kRowBytes + ((c ^ (r & 6)) << 4), vc + src, bytes);
        }
        // the scale of token (lane & 15): lanes 0-15 K, lanes 16-31 V; copied as the aligned 32-bit word around it
        const int tr = lane & 15;
        const int sbytes = tr < valid ? 4 : 0;
        const size_t sidx = sbytes ? (static_cast<size_t>(row0) + tr) * p.num_kv_heads + kvh : 0;
        cp_async4(stage + 2 * kTileBytes + lane * 4, (lane < 16 ? p.k_scale : p.v_scale) + (sidx & ~static_cast<size_t>(1)), sbytes);
    }
    __device__ __forceinline__ void step(const DecodeParams& p, uint32_t stage, int valid, int kvh, int lane) {
        const int g = lane >> 2, t = lane & 3;
        // Scales of keys g and g + 8.  Which half of a copied word is the scale: cache rows of a tile start at an even row, so the parity of
        // row * Hkv + kvh is that of (token & Hkv & 1) + kvh.
        float2 kscale, vscale;
        {
            uint32_t w[4];
            const uint32_t at = stage + 2 * kTileBytes + g * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(w[i]) : "r"(at + i * 32));
            const uint32_t pick = (((g & p.num_kv_heads) ^ kvh) & 1) != 0 ? 0x7632u : 0x5410u;
            const uint32_t k2 = __byte_perm(w[0], w[1], pick), v2 = __byte_perm(w[2], w[3], pick);
            kscale = __half22float2(*reinterpret_cast<const __half2*>(&k2));
            vscale = __half22float2(*reinterpret_cast<const __half2*>(&v2));
            kscale.x *= p.scale_log2;
            kscale.y *= p.scale_log2;
        }
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            uint32_t w0[4], w1[4];
            lds32x4(stage + g * kRowBytes + (((4 * q + t) ^ ((g & 1) << 2)) << 4), w0);
            lds32x4(stage + (g + 8) * kRowBytes + (((4 * q + t) ^ ((g & 1) << 2)) << 4), w1);
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) {
                const int ks = 4 * q + wi;
                const uint32_t x0 = w0[wi] ^ kFlip, x1 = w1[wi] ^ kFlip;
                mma_16816<__half>(ks & 1 ? s1 : s0, widen_pair_lo<FP8>(x0), widen_pair_lo<FP8>(x1), widen_pair_hi<FP8>(x0), widen_pair_hi<FP8>(x1), qa[ks][0],
                                  qa[ks][1]);
            }
        }
        float sc[4] = {(s0[0] + s1[0] - q_off[0]) * kscale.x, (s0[1] + s1[1] - q_off[1]) * kscale.x, (s0[2] + s1[2] - q_off[0]) * kscale.y,
                       (s0[3] + s1[3] - q_off[1]) * kscale.y};
        mask_scores(sc, g, valid);
        s.raise_max(sc, FP8 ? nullptr : osum);
        const float p0 = fast_exp2(sc[0] - s.m[0]), p1 = fast_exp2(sc[1] - s.m[1]), p2 = fast_exp2(sc[2] - s.m[0]), p3 = fast_exp2(sc[3] - s.m[1]);
        s.l[0] += p0 + p2;
        s.l[1] += p1 + p3;
        const uint32_t pb0 = transpose_8x8(ElemTraits<__half>::pack2(p0 * vscale.x, p1 * vscale.x));
        const uint32_t pb1 = transpose_8x8(ElemTraits<__half>::pack2(p2 * vscale.y, p3 * vscale.y));
        // output: V rows 2t, 2t+1, 2t+8, 2t+9, piece g (d = 16 g .. 16 g + 15)
        uint32_t v0[4], v1[4], v2[4], v3[4];
        const uint32_t vbase = stage + kTileBytes;
        lds32x4(vbase + (2 * t) * kRowBytes + ((g ^ ((2 * t) & 6)) << 4), v0);
        lds32x4(vbase + (2 * t + 1) * kRowBytes + ((g ^ ((2 * t + 1) & 6)) << 4), v1);
        lds32x4(vbase + (2 * t + 8) * kRowBytes + ((g ^ ((2 * t + 8) & 6)) << 4), v2);
        lds32x4(vbase + (2 * t + 9) * kRowBytes + ((g ^ ((2 * t + 9) & 6)) << 4), v3);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const uint32_t x0 = v0[a] ^ kFlip, x1 = v1[a] ^ kFlip, x2 = v2[a] ^ kFlip, x3 = v3[a] ^ kFlip;
            // bytes of one d from two consecutive keys, side by side
            const uint32_t lo01 = __byte_perm(x0, x1, 0x5140), hi01 = __byte_perm(x0, x1, 0x7362);
            const uint32_t lo23 = __byte_perm(x2, x3, 0x5140), hi23 = __byte_perm(x2, x3, 0x7362);
            mma_16816<__half>(s.o[2 * a], widen_pair_lo<FP8>(lo01), widen_pair_hi<FP8>(lo01), widen_pair_lo<FP8>(lo23), widen_pair_hi<FP8>(lo23), pb0, pb1);
            mma_16816<__half>(s.o[2 * a + 1], widen_pair_lo<FP8>(hi01), widen_pair_hi<FP8>(hi01), widen_pair_lo<FP8>(hi23), widen_pair_hi<FP8>(hi23), pb0, pb1);
        }
        constexpr uint32_t kOnes = 0x3C003C00u;   // {1.0, 1.0}
        if (!FP8) mma_16816<__half>(osum, kOnes, kOnes, kOnes, kOnes, pb0, pb1);
    }
    __device__ __forceinline__ void write_part(float* row, int h, int g) const {
        const float off = kOffset * osum[h];
#pragma unroll
        for (int i = 0; i < 8; i += 2)
            *reinterpret_cast<float4*>(row + 16 * g + 2 * i) = make_float4(s.o[i][h] - off, s.o[i][2 + h] - off, s.o[i + 1][h] - off, s.o[i + 1][2 + h] - off);
    }
};

// ---- a group's range of keys ---------------------------------------------------------------------------------------------
template <class F>
struct alignas(128) GroupSmem {
    union Warp {
        unsigned char ring[F::kStages * F::kStageBytes];
        struct {                                       // what the warp leaves for the merge, when its ring is idle
            float o[kMaxGroup * F::kPartStride];       // head 2 t + h in row 4 h + t: the lanes of a store hit different banks
            float2 ml[kMaxGroup];
        } part;
    } warps[kGroupWarps];
};

// Keys [t0, t1) of sequence b (t0 < t1), one KV head.  sink(h, quad, o, m, l) takes elements 4 quad .. 4 quad + 3 of head h: unnormalised
// output, maximum and sum.  `tid`: 0..127 inside the group, `bar_id`: its named barrier; all its threads call it.  `raw_ids`: block
// table entries `id_base` + lane as loaded.  The four warps' parts come together in one trip over all heads, after one barrier (a warp writes
// its part over its own ring; before, two barriers and a loop over the heads, a trip each).
template <class F, class Sink>
__device__ __forceinline__ void attend_range(const DecodeParams& p, int b, int kvh, int t0, int t1, IndexArray::Raw raw_ids, int id_base, GroupSmem<F>& sm,
                                             int tid, int bar_id, Sink sink) {
    const int bs = p.block_size, warp = tid >> 5, lane = tid & 31;
    const uint32_t ring = smem_u32(sm.warps[warp].ring);
    const int num_tiles = (t1 - t0 + kTileTokens - 1) / kTileTokens;
    const int my_tiles = num_tiles > warp ? (num_tiles - warp + kGroupWarps - 1) / kGroupWarps : 0;
    // The issuing end: this warp's next tile begins at row `off` of table entry `blk`.  Lane i holds the cache block of entry
    // id_base + i (-1: outside the cache, reads as zeros).
    int tok = t0 + warp * kTileTokens;
    int blk = static_cast<int>(p.by_block.div(tok)), off = tok - blk * bs, ids;
    auto take_ids = [&](IndexArray::Raw raw) {
        const int64_t id = p.block_tables.value(raw);
        ids = (id >= 0 && id < p.num_cache_blocks) ? static_cast<int>(id) : -1;
    };
    auto move_window = [&]() {
        if (blk - id_base >= 32 && tok < t1) {
            id_base = blk;
            take_ids(load_ids(p, b, id_base, lane));
        }
    };
    take_ids(raw_ids);
    move_window();   // (a warp may begin just past what was loaded)
    uint32_t istage = ring;
    auto issue = [&]() {
        if (tok < t1) {
            const int phys = __shfl_sync(0xffffffffu, ids, blk - id_base);
            F::issue(p, kvh, phys < 0 ? 0 : static_cast<int64_t>(phys) * bs + off, phys < 0 ? 0 : t1 - tok, istage, lane);
            istage = istage == ring + (F::kStages - 1) * F::kStageBytes ? ring : istage + F::kStageBytes;
            tok += kGroupWarps * kTileTokens;
            for (off += kGroupWarps * kTileTokens; off >= bs; off -= bs) ++blk;
            move_window();
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < F::kStages - 1; ++s) issue();

    F st;
    st.start(p, b, kvh, lane);
    uint32_t cstage = ring;
    int left = t1 - t0 - warp * kTileTokens;   // keys from this warp's tile on
    for (int j = 0; j < my_tiles; ++j) {
        issue();
        cp_async_wait<F::kStages - 1>();
        __syncwarp();
        st.step(p, cstage, left, kvh, lane);
        __syncwarp();   // the stage is refilled by other lanes' copies
        cstage = cstage == ring + (F::kStages - 1) * F::kStageBytes ? ring : cstage + F::kStageBytes;
        left -= kGroupWarps * kTileTokens;
    }
    cp_async_wait<0>();
    __syncwarp();                              // this warp's ring is idle from here on
    const int g = lane >> 2, t = lane & 3;
    auto& part = sm.warps[warp].part;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float l = st.s.l[h];
#pragma unroll
        for (int x = 4; x < 32; x *= 2) l += __shfl_xor_sync(0xffffffffu, l, x);
        if (2 * t + h < p.group) {
            if (g == 0) part.ml[2 * t + h] = make_float2(st.s.m[h], l);
            st.write_part(part.o + (4 * h + t) * F::kPartStride, h, g);
        }
    }
    group_sync(bar_id, kGroupThreads);
    for (int h = warp; h < p.group; h += kGroupWarps) {
        float4 o[kGroupWarps];
        float2 ml[kGroupWarps];
#pragma unroll
        for (int w = 0; w < kGroupWarps; ++w) {
            const auto& from = sm.warps[w].part;
            ml[w] = from.ml[h];
            o[w] = *reinterpret_cast<const float4*>(from.o + (4 * (h & 1) + (h >> 1)) * F::kPartStride + 4 * lane);
        }
        float mx = ml[0].x, sum = 0.0f;
        float4 total = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int w = 1; w < kGroupWarps; ++w) mx = fmaxf(mx, ml[w].x);
#pragma unroll
        for (int w = 0; w < kGroupWarps; ++w) {
            const float f = fast_exp2(ml[w].x - mx);   // 0 for a warp without a tile
            total.x = fmaf(f, o[w].x, total.x); total.y = fmaf(f, o[w].y, total.y); total.z = fmaf(f, o[w].z, total.z); total.w = fmaf(f, o[w].w, total.w);
            sum = fmaf(f, ml[w].y, sum);
        }
        sink(h, lane, total, mx, sum);
    }
}

template <typename T> __device__ __forceinline__ void write_quad(T* at, const float4& v) {   // four elements of a result
    *reinterpret_cast<uint2*>(at) = make_uint2(ElemTraits<T>::pack2(v.x, v.y), ElemTraits<T>::pack2(v.z, v.w));
}
__device__ __forceinline__ float4 scaled(const float4& v, float f) { return make_float4(v.x * f, v.y * f, v.z * f, v.w * f); }

// Range `split` of (b, kvh): the result if it is all of the context, else a part in the workspace.
template <class F, typename T>
__device__ __forceinline__ void run_split(const DecodeParams& p, int b, int kvh, int split, GroupSmem<F>& sm, int tid, int bar_id) {
    const int lane = tid & 31;
    const IndexArray::Raw raw_ctx = p.context_lens.raw(b);
    // The first range's block ids on their way with the context: a trip to memory less.  Further chunks look whether they have keys first: with tables
    // much wider than the contexts nearly all blocks are of this kind (256 sequences of 100 to 300 keys, 8 KV heads, 32768-key tables, 32768
    // blocks: 82 us a pass, 106 with ids for all), and they leave before anything else (128 such sequences: 56.7 -> 50.8 us a call).
    const bool early = p.per_seq || split == 0;
    int id_base = 0;
    IndexArray::Raw raw_ids{0, 0};
    if (early) raw_ids = load_ids(p, b, 0, lane);
    const int ctx = clamped_context(p, raw_ctx);
    if (!p.per_seq && split > 0 && static_cast<int64_t>(split) * p.chunk_tokens >= ctx) return;
    const int len = range_len(p, ctx), t0 = split * len, t1 = min(ctx, t0 + len);
    if (!early) {
        id_base = static_cast<int>(p.by_block.div(t0));
        raw_ids = load_ids(p, b, id_base, lane);
    }
    T* out = static_cast<T*>(p.out) + (static_cast<int64_t>(b) * p.num_heads + kvh * p.group) * kHeadDim;
    if (t0 >= t1) {
        if (ctx == 0 && split == 0) {
            for (int i = tid; i < p.group * kHeadDim; i += kGroupThreads) out[i] = ElemTraits<T>::from_float(0.0f);
        }
        return;
    }
    const size_t part = (static_cast<size_t>(b) * p.num_kv_heads + kvh) * p.num_splits + split;
    attend_range<F>(p, b, kvh, t0, t1, raw_ids, id_base, sm, tid, bar_id, [&](int h, int quad, const float4& o, float m, float l) {
        if (ctx <= len) {
            write_quad(out + h * kHeadDim + 4 * quad, scaled(o, 1.0f / l));   // (rounded as write_merged does)
        } else {
            reinterpret_cast<float4*>(p.ws_o + (part * p.group + h) * kHeadDim)[quad] = o;
            if (quad == 0) p.ws_ml[part * p.group + h] = make_float2(m, l);
        }
    });
}

// ---- merging the parts of a sequence -------------------------------------------------------------------------------------
// HG heads of one (sequence, KV head) at a time.  Where there can be few parts one warp takes them in order, otherwise they are
// dealt over kMergeWarps warps.
struct PartRef { const float* o; const float2* ml; };   // head 0 of a part
struct Merged {                                         // elements 4 lane .. 4 lane + 3 of a head's output, maximum and row sum
    float4 o;
    float m, l;
    // Four parts at a time (every merge in the same order, so that who merges makes no difference to a bit); one that is not there: zeros, with a
    // maximum of minus infinity.
    __device__ __forceinline__ void add(const float4 (&v)[4], const float2 (&ml)[4]) {
        const float mx = fmaxf(m, fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x))), f = fast_exp2(m - mx);
        o = scaled(o, f);
        l *= f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float w = fast_exp2(ml[u].x - mx);
            o.x = fmaf(w, v[u].x, o.x); o.y = fmaf(w, v[u].y, o.y); o.z = fmaf(w, v[u].z, o.z); o.w = fmaf(w, v[u].w, o.w);
            l = fmaf(w, ml[u].y, l);
        }
        m = mx;
    }
};
__device__ __forceinline__ Merged nothing_merged() { return Merged{make_float4(0.f, 0.f, 0.f, 0.f), -INFINITY, 0.0f}; }

// Heads h0 .. h0 + HG - 1 (clamped to the group) over parts first, first + stride, ...
template <int HG, class Get>
__device__ __forceinline__ void sum_parts(Get get, int n, int first, int stride, int h0, int group, int lane, Merged (&acc)[HG]) {
    constexpr int U = HG == 4 ? 4 : 8;   // parts in flight
#pragma unroll
    for (int h = 0; h < HG; ++h) acc[h] = nothing_merged();
    for (int i0 = first; i0 < n; i0 += U * stride) {
        float2 ml[U][HG];
        float4 v[U][HG];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const PartRef r = get(min(i0 + u * stride, n - 1));   // (loads without branches, so that all are in flight at once)
#pragma unroll
            for (int h = 0; h < HG; ++h) {
                const int hh = min(h0 + h, group - 1);
                ml[u][h] = r.ml[hh];
                v[u][h] = *reinterpret_cast<const float4*>(r.o + hh * kHeadDim + 4 * lane);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u += 4) {
            if (i0 + u * stride < n) {
#pragma unroll
                for (int h = 0; h < HG; ++h) {
                    float4 four[4];
                    float2 ml4[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const bool there = i0 + (u + k) * stride < n;
                        four[k] = there ? v[u + k][h] : make_float4(0.f, 0.f, 0.f, 0.f);
                        ml4[k] = there ? ml[u + k][h] : make_float2(-INFINITY, 0.0f);
                    }
                    acc[h].add(four, ml4);
                }
            }
        }
    }
}
template <typename T>
__device__ __forceinline__ void write_merged(T* row, const Merged& a, int lane) {
    const float inv = a.l > 0.0f ? 1.0f / a.l : 0.0f;
    write_quad(row + 4 * lane, scaled(a.o, inv));
}
// Heads h0 .. h0 + HG - 1 of the group, rows of `out`, by one warp.
template <typename T, int HG, class Get>
__device__ __forceinline__ void merge_by_warp(Get get, int n, int h0, int group, T* out, int lane) {
    Merged acc[HG];
    sum_parts<HG>(get, n, 0, 1, h0, group, lane, acc);
#pragma unroll
    for (int h = 0; h < HG; ++h)
        if (h0 + h < group) write_merged<T>(out + (h0 + h) * kHeadDim, acc[h], lane);
}
// One head, by the whole block; the first kMergeWarps warps work.
struct MergeScratch { float4 o[kMergeWarps][32]; float2 ml[kMergeWarps]; };
template <typename T, class Get>
__device__ __forceinline__ void merge_by_block(Get get, int n, int head, int group, T* row, MergeScratch& sm, int warp, int lane) {
    if (warp < kMergeWarps) {
        Merged acc[1];
        sum_parts<1>(get, n, warp, kMergeWarps, head, group, lane, acc);
        sm.o[warp][lane] = acc[0].o;
        if (lane == 0) sm.ml[warp] = make_float2(acc[0].m, acc[0].l);
    }
    __syncthreads();
    if (warp == 0) {
        Merged a = nothing_merged();
#pragma unroll
        for (int w = 0; w < kMergeWarps; w += 4)
            a.add({sm.o[w][lane], sm.o[w + 1][lane], sm.o[w + 2][lane], sm.o[w + 3][lane]}, {sm.ml[w], sm.ml[w + 1], sm.ml[w + 2], sm.ml[w + 3]});
        write_merged<T>(row, a, lane);
    }
    __syncthreads();
}

}  // namespace dec
}  // namespace nvk
