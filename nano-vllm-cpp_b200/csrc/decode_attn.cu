// Paged-KV decode attention for sm_100a (F16 / BF16 queries, head_dim 128; 16-bit, int8 and e4m3 caches).
//
// Replaces decode_paged_attention_kernel and decode_paged_attention_int8_kernel (src/kernels/attention.cu:313-405, :746-842 of the
// reference: one warp per (sequence, query head), every KV row re-read by each query head of its group, 8 dependent shuffles per
// key) and the FlashAttention-2 call it can dlopen (src/kernels/flash_attn.cpp:302-431).
//
// The op is HBM-bound; decode_body.cuh has the arithmetic and the ways to share out the keys.  What each kernel here adds:
//   decode_split_kernel    one four-warp block per (KV head, chunk, sequence), two per SM (three for 8-bit caches).  The grid is fixed
//                          from host-known sizes: nothing depends on host knowledge of context_lens (CUDA-graph safe); blocks
//                          whose chunk lies beyond the context exit at once.
//   decode_merge_kernel    merges the chunks of long contexts; launched only where the table can hold more than one.
//   decode_cluster_kernel  small steps: a cluster of blocks per (sequence, KV head) takes equal ranges of the context, beyond them two blocks the halves
//                          of the table's row; merged in the same launch.
// Which one is taken depends on the table's WIDTH, not on the contexts: one short sequence in a wide table takes chunks and a merge.
#include "decode_body.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace nvk {
namespace {

using namespace dec;

constexpr size_t kStaticScratchBytes = 32u << 20;
constexpr int kMaxCluster = 8;          // portable cluster size
// Longest range per block (of a full table row) that goes to the cluster kernel: 8 tiles per warp, some 5 us of keys.  Up to there the
// second launch costs more than chunks of even length give: 1 sequence of 300 keys, 32 / 8 heads, with its prologue, took 6.7 us a
// pass in a replayed graph where split and merge took 9.1 (5.9 now).
constexpr int kClusterTokens = 512;

// Sequence number `rank` in order of falling context length, found by every block for itself.  In index order the last blocks to start
// can be the longest: 100 sequences of 500 to 4096 keys, int8, left half the SMs idle for the last 40 of 106 us; in this order the pass
// took 103 us instead of 115 (92 since the keys are the rows of the score MMAs).  64 sequences of 100 to 2048 keys, 16-bit: 6 us less.  The order is that of 128 classes of length, and of
// the index inside a class: a histogram, one scan and a search through the class.  (Comparing every context with every other one took
// each block 5 us at 254 sequences: with 4 KV heads and contexts of up to 157 keys 39 us a pass.)
constexpr int kMaxSorted = 512;
constexpr int kMinSortedTokens = 1024;   // tables of fewer keys: a block lasts hardly longer than the 1 us that this takes
struct SortScratch { int count[128]; unsigned char cls[kMaxSorted]; };
__device__ __forceinline__ int sequence_of_rank(const DecodeParams& p, int rank, SortScratch& sm) {
    static_assert(kGroupThreads == 128, "one thread per class");
    const int tid = threadIdx.x, lane = tid & 31;
    const int shift = max(0, 25 - __clz(static_cast<int>(p.max_blocks * p.block_size)));   // the longest context there can be is in class 127 at most
    sm.count[tid] = 0;
    __syncthreads();
    for (int i = tid; i < p.batch; i += kGroupThreads) {
        const int c = 127 - (clamped_context(p, i) >> shift);
        sm.cls[i] = static_cast<unsigned char>(c);
        atomicAdd(&sm.count[c], 1);
    }
    __syncthreads();
    // every warp finds the class (four per lane), then the sequence
    const int4 n = reinterpret_cast<const int4*>(sm.count)[lane];
    const int mine = n.x + n.y + n.z + n.w;
    int upto = mine;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const int up = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= d) upto += up;
    }
    const int owner = __ffs(__ballot_sync(0xffffffffu, upto > rank)) - 1;
    int c = 4 * lane, left = rank - (upto - mine);   // (the owner's values are used)
    if (left >= n.x) {
        left -= n.x; ++c;
        if (left >= n.y) {
            left -= n.y; ++c;
            if (left >= n.z) { left -= n.z; ++c; }
        }
    }
    c = __shfl_sync(0xffffffffu, c, owner);
    left = __shfl_sync(0xffffffffu, left, owner);
    for (int i0 = 0;; i0 += 32) {
        const bool in = i0 + lane < p.batch && sm.cls[i0 + lane] == c;
        const unsigned int all = __ballot_sync(0xffffffffu, in);
        const unsigned int hit = __ballot_sync(0xffffffffu, in && __popc(all & ((1u << lane) - 1u)) == left);
        if (hit != 0 || i0 + 32 >= p.batch) return i0 + max(0, __ffs(hit) - 1);
        left -= __popc(all);
    }
}

__device__ __forceinline__ void st_cluster4(uint32_t addr, uint32_t rank, const float4& v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(in_block(addr, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_cluster2(uint32_t addr, uint32_t rank, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(in_block(addr, rank)), "f"(x), "f"(y) : "memory");
}

template <class F, typename T>
__global__ void __launch_bounds__(kGroupThreads, F::kGroups) decode_split_kernel(const __grid_constant__ DecodeParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    if (p.beside) pdl_start_beside();
    else pdl_wait_then_release();
    const int rank = p.chunk_major ? blockIdx.y : blockIdx.z, split = p.chunk_major ? blockIdx.z : blockIdx.y;
    const int b = p.longest_first ? sequence_of_rank(p, rank, *reinterpret_cast<SortScratch*>(smem)) : rank;
    if (p.longest_first) __syncthreads();   // (the ring takes the scratch's place)
    run_split<F, T>(p, b, blockIdx.x, split, *reinterpret_cast<GroupSmem<F>*>(smem), threadIdx.x, 1);
    if (p.beside) pdl_wait_beside();
}

// HG > 0: one warp per (sequence, KV head) and HG of its heads, in blocks of kMergeBlockWarps warps, small enough to be resident
// beside the blocks of decode_split_kernel.  HG == 0: one block per (sequence, head), where there can be more parts than one warp
// should add up: 3 sequences of up to 40000 keys left 12 blocks adding up 20 parts each one after the other, 10 us.  These blocks do not
// fit beside those of decode_split_kernel, so that many of them only queue up behind it.  Between the two, up to 4096 rows that can have more than
// four parts, HG is 1: 49 sequences of up to 31475 keys, 32 / 8 heads, 494 us a pass with four heads a warp, 486 with one; but 256
// sequences (8192 rows) of which few have a second part 189 and 192.  By warps -> by blocks, us a call: 32 rows of 75
// parts 18.3 -> 14.3, 128 rows of 64 157.1 -> 155.4, 256 of 64 160.4 -> 157.1; but 512 rows of which none has a second part 10.5 -> 11.2,
// 4096 such rows 45.0 -> 50.8, 4096 rows of 2 parts in 32768-key tables 230 -> 244.
constexpr int kMergeBlockRows = 2 * kSmCount;
constexpr int kMergeSingleRows = 4096;
constexpr int kMergeBlockWarps = 2;
template <typename T, int HG>
__global__ void __launch_bounds__((HG > 0 ? kMergeBlockWarps : kMergeWarps) * 32) decode_merge_kernel(const __grid_constant__ DecodeParams p) {
    __shared__ MergeScratch scratch;
    pdl_wait_then_release();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto parts_of = [&](int b, int kvh, int& n) {   // n parts of (b, kvh) and where they are
        const int ctx = clamped_context(p, b), len = range_len(p, ctx);
        n = ctx > 0 ? (ctx + len - 1) / len : 0;
        const size_t part = (static_cast<size_t>(b) * p.num_kv_heads + kvh) * p.num_splits;
        const float* o = p.ws_o + part * p.group * kHeadDim;
        const float2* ml = p.ws_ml + part * p.group;
        return [o, ml, group = p.group](int i) { return PartRef{o + static_cast<size_t>(i) * group * kHeadDim, ml + i * group}; };
    };
    T* out = static_cast<T*>(p.out);
    int n;
    if constexpr (HG > 0) {
        const int item = blockIdx.x * kMergeBlockWarps + warp, chunks = (p.group + HG - 1) / HG;
        const int pair = item / chunks;
        if (pair >= p.batch * p.num_kv_heads) return;
        const int b = static_cast<int>(p.by_kv_heads.div(pair));
        const auto get = parts_of(b, pair - b * p.num_kv_heads, n);
        if (n > 1) merge_by_warp<T, HG>(get, n, (item - pair * chunks) * HG, p.group, out + static_cast<int64_t>(pair) * p.group * kHeadDim, lane);
    } else {
        const int row = blockIdx.x, b = row / p.num_heads, head = row - b * p.num_heads, kvh = head / p.group;
        const auto get = parts_of(b, kvh, n);
        if (n > 1) merge_by_block<T>(get, n, head - kvh * p.group, p.group, out + static_cast<int64_t>(row) * kHeadDim, scratch, warp, lane);
    }
}

// A block pushes what it has of the result into the shared memory of the block that finishes it: of 32 quads of a head, block r of n
// takes 32 / n from r * 32 / n on.  After one cluster barrier everything there is local, and no block has to wait for its peers to have
// read.  1 sequence of 300 keys, 32 / 8 heads, with its prologue: 7.2 -> 5.85 us a pass with the block ids fetched along with the context and one
// barrier in a block's merge; from a block's last tile to its end it had been 2.5 us of 4.3.
// Equal ranges (per_seq): all blocks of the cluster have a part, if an empty one.  Halves of a table row: where a context ends in the first, that block
// writes the result and the other leaves.
constexpr int kPartQuads = kMaxGroup * kHeadDim / 4;   // n x 8 heads x 32 / n, for the cluster sizes there are: 1, 2, 4, 8
template <class F, typename T>
__global__ void __launch_bounds__(kGroupThreads, F::kGroups) decode_cluster_kernel(const __grid_constant__ DecodeParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float4 s_o[kPartQuads];                         // [block of the cluster][head][quad of this block]
    __shared__ float2 s_ml[kMaxCluster * kMaxGroup];           // [block of the cluster][head]
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");   // (waited for before the first remote store: every block has started)
    if (p.beside) pdl_start_beside();
    else pdl_wait_then_release();
    const int rank = static_cast<int>(blockIdx.x) & (p.num_splits - 1), pair = static_cast<int>(blockIdx.x) >> p.split_shift;
    const int b = static_cast<int>(p.by_kv_heads.div(pair)), kvh = pair - b * p.num_kv_heads;
    const int tid = threadIdx.x, lane = tid & 31;
    const int id_base = p.per_seq ? 0 : static_cast<int>(p.by_block.div(rank * p.chunk_tokens));
    const IndexArray::Raw raw_ctx = p.context_lens.raw(b);
    IndexArray::Raw raw_ids = load_ids(p, b, id_base, lane);
    const int ctx = clamped_context(p, raw_ctx), len = range_len(p, ctx);
    const int t0 = rank * len, t1 = min(ctx, t0 + len);
    T* out = static_cast<T*>(p.out) + (static_cast<int64_t>(b) * p.num_kv_heads + kvh) * p.group * kHeadDim;
    const int n = p.per_seq ? p.num_splits : ctx > len ? 2 : 1;                // blocks with a part (chunks: two)
    const int quad_shift = n == 1 ? 5 : 5 - p.split_shift, quads = 1 << quad_shift;   // quads of a head that a block finishes
    if (rank < n) {
        bool waited = false;
        auto wait_started = [&]() {
            if (!waited) asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
            waited = true;
        };
        auto push = [&](int h, int quad, const float4& o, float m, float l) {
            if (n == 1) {
                write_quad(out + h * kHeadDim + 4 * quad, scaled(o, 1.0f / l));   // (rounded as write_merged does)
                return;
            }
            wait_started();
            const uint32_t to = static_cast<uint32_t>(quad >> quad_shift);
            const int mine = quad & (quads - 1);
            st_cluster4(smem_u32(s_o + ((rank * p.group + h) << quad_shift) + mine), to, o);
            if (mine == 0) st_cluster2(smem_u32(s_ml + rank * p.group + h), to, m, l);
        };
        if (t0 < t1) {
            attend_range<F>(p, b, kvh, t0, t1, raw_ids, id_base, *reinterpret_cast<GroupSmem<F>*>(smem), tid, 1, push);
        } else {                                                                  // (alone: an empty context, zeros)
            for (int h = tid >> 5; h < p.group; h += kGroupWarps) push(h, lane, make_float4(0.f, 0.f, 0.f, 0.f), -INFINITY, n > 1 ? 0.0f : 1.0f);
        }
        if (n > 1) {
            wait_started();                                                       // (a warp without a head)
            asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
            for (int i = tid; i < p.group << quad_shift; i += kGroupThreads) {
                const int h = i >> quad_shift, quad = (rank << quad_shift) + (i & (quads - 1));
                Merged acc = nothing_merged();
                for (int r0 = 0; r0 < n; r0 += 4) {
                    float4 v[4];
                    float2 ml[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool there = r0 + u < n;
                        const int r = there ? r0 + u : 0;
                        v[u] = s_o[(r * p.group << quad_shift) + i];
                        ml[u] = s_ml[r * p.group + h];
                        if (!there) { v[u] = make_float4(0.f, 0.f, 0.f, 0.f); ml[u] = make_float2(-INFINITY, 0.0f); }
                    }
                    acc.add(v, ml);
                }
                if (ctx == 0) acc = nothing_merged();
                write_merged<T>(out + h * kHeadDim, acc, quad);
            }
        }
    }
    if (p.beside) pdl_wait_beside();
}

// ---- host side -----------------------------------------------------------------------------------------------------------

// Blocks per (sequence, KV head) of the cluster kernel, or 0: chunks.  Only clusters that are all resident at once: a cluster has to fit
// into one GPC, so that these are fewer than the places for single blocks (the driver's occupancy query for these kernels at two and
// three blocks per SM).  With one more a second wave follows: clusters of 4, 1024 keys, 70 -> 72 pairs 11.0 -> 15.6 us a call, clusters of
// 8, 300 keys, 32 -> 34 pairs 5.8 -> 9.4 (in one block each 5.7).  Clusters of 4 gain nothing in tables of up to 512 keys (64 pairs of 300 / 512 keys
// 7.6 / 8.7 us, in one block each 6.4 / 7.8), nor clusters of 2 on equal ranges (their halves of a table's row: see below).  Without a workspace there is nothing else, and any cluster that fits is taken.
struct ClusterWay { int size, resident[2]; };
constexpr ClusterWay kWays[] = {{8, {33, 48}}, {4, {71, 104}}, {2, {148, 222}}};
int cluster_size(int64_t batch, int num_kv_heads, int64_t max_blocks, int block_size, int groups, bool have_workspace) {
    const int64_t pairs = batch * num_kv_heads, max_tokens = max_blocks * block_size;
    for (const auto& w : kWays) {
        if (pairs > w.resident[groups == 3]) continue;
        if (!have_workspace) return w.size;
        return w.size > 2 && max_tokens <= static_cast<int64_t>(kClusterTokens) * w.size && (w.size == 8 || max_tokens > kClusterTokens) ? w.size : 0;
    }
    return have_workspace ? 0 : 1;
}

// A grid just past a full wave of resident groups: its last blocks run almost alone, and nothing balances equal ones.
bool just_past_a_wave(int64_t pairs, int groups) {
    return pairs > kSmCount * groups && (groups == 2 ? 4 * pairs < 5 * kSmCount * groups : 3 * pairs < 4 * kSmCount * groups);
}

// How a step beyond the clusters is shared out.  Contexts are rarely as long as the table: a step has one long one among short ones, or a third of them, or
// an even spread.  Figures are us in a replayed graph with inputs beyond L2, for contexts of which one / a tenth / a third fill the table and the others 1/32
// or 1/16 of it, and for spreads of 0.05 / 0.5 / 1.0 to all of the table.
//
// Halves of a table row, merged in a cluster of two blocks, where both halves of all contexts find a place at once and a half is short enough for one long
// context not to be what a step waits for.  16-bit caches, 110 pairs of 2048 keys 10.4 / 12.3 / 13.8, 14.3 / 16.9 / 21.3, in chunks of 512 10.1 / 11.8 /
// 13.3, 16.1 / 22.4 / 24.9; of 3072 14.0 / 16.4 / 18.6, 19.6 / 23.2 / 30.1, in chunks of 1024 13.3 / 15.9 / 17.8, 20.9 / 26.7 / 38.1.  But 90 pairs of 3072
// 13.8 / 15.7 / 18.2, 18.8 / 20.8 / 26.7, in chunks of 512 8.8 / 10.9 / 13.7, 18.9 / 23.2 / 27.8; and 128 of 4096 17.9 / 20.7 / 23.7, 26.3 / 33.6 / 43.5, in
// chunks of 512 10.8 / 13.2 / 21.0, 29.0 / 37.7 / 47.3.  8-bit ones: 200 of 1536 10.1 / 13.3 / 16.5, 17.8 / 18.5 / 19.0, in chunks of 512 10.8 / 14.1 / 16.2,
// 17.0 / 22.1 / 23.8; but 128 of 2048 11.9 / 15.0 / 18.8, 20.4 / 21.1 / 21.4, in chunks of 512 10.2 / 13.8 / 15.8, 16.5 / 17.9 / 21.6.  Fewer pairs than
// clusters of four hold take those, or more chunks; in tables of up to 512 (8-bit: 768) keys whole contexts are as quick.
bool halves(int64_t pairs, int64_t max_tokens, int groups) {
    if (pairs <= kWays[1].resident[groups == 3] || 2 * pairs > static_cast<int64_t>(kSmCount) * groups) return false;
    return groups == 2 ? max_tokens > 512 && max_tokens <= (pairs < 104 ? 2048 : 3072) : max_tokens > 768 && max_tokens <= 1536;
}

// Chunk length in keys (whole cache blocks), from the number of (sequence, KV head) pairs and the table's width.  Whole contexts (no merge, no second launch)
// where a block reads one in little time, or where the step has more of them than places:
//   * 16-bit: tables of up to 1024 keys, 1536 where the halves above have no room (152 pairs 12.8 / 15.0 / 17.5, 16.9 / 18.9 / 21.8, in chunks of 1024 11.8 /
//     14.7 / 16.8, 17.3 / 20.4 / 25.1).  8-bit: 1024 with few pairs, 768 from 1.5 to an SM on, 1280 from two (320 pairs 13.3 / 18.1 / 23.1, 22.4 / 23.6 /
//     25.6, in chunks of 1024 14.2 / 18.0 / 23.0, 23.8 / 24.8 / 26.8).
//   * Tables of up to 4096 keys with a pair for every resident group, but not just past a wave: 304 / 352 16-bit pairs, all of 4096 keys, 116.8 / 123.7 a
//     call, in chunks of 2048 106.1 / 113.5.
// Chunks of 512 where the table has up to 4096 keys (8-bit: 1536) and single contexts leave places free: 200 16-bit pairs of 4096 keys 13.0 / 17.5 / 29.6,
// 40.3 / 54.2 / 68.0, of 2048 20.9 / 26.7 / 30.9, 41.1 / 58.6 / 70.1, whole 30.7 / 35.9 / 40.9, 42.7 / 53.6 / 68.3; 256 int8 pairs of 1536 10.8 / 15.0 /
// 17.3, 21.2 / 25.1 / 27.4, of 1024 13.8 / 18.2 / 21.1, 23.1 / 24.7 / 29.6, whole 15.2 / 20.4 / 25.6, 24.7 / 26.3 / 28.2.  Chunks of 1024 in tables of up to
// 8192 keys with few pairs: 224 of 6144 17.2 / 25.1 / 45.3, 60.9 / 83.3 / 107.9, of 2048 22.1 / 30.8 / 46.9, 65.7 / 85.0 / 111.9.  Chunks of 2048 otherwise.
// All halved down to 256 while they leave resident groups without a block:
//   * What a table of 2048 keys is cut into is cut no finer than it takes to have 1.5 blocks per SM (8-bit: 2.25 of 512 keys).
//   * Longer ones need every place filled, since contexts are often shorter than the table (64 pairs of 1000 keys, 4096-key tables: 512-key chunks 12.0,
//     1024-key ones 14.9), but 512 keys are not cut for the last few (36 pairs of 4096 keys 19.0, as chunks of 256 21.0).
// (Whole contexts of 8192-key tables, 256 sequences: 694 us a pass, 689 with chunks.)
int chunk_tokens(int64_t batch, int num_kv_heads, int64_t max_blocks, int block_size, int groups) {
    const int64_t max_tokens = max_blocks * block_size, pairs = batch * num_kv_heads, resident = static_cast<int64_t>(kSmCount) * groups;
    const int64_t whole = groups == 2 ? (2 * pairs > resident ? 1536 : 1024) : pairs >= 2 * kSmCount ? 1280 : 2 * pairs <= resident ? 1024 : 768;
    if (max_tokens <= whole || (max_tokens <= 4096 && pairs >= resident && !just_past_a_wave(pairs, groups))) return static_cast<int>(max_tokens);
    int64_t chunk = 2048;
    if (groups == 2 ? max_tokens > 2048 && max_tokens <= 4096 && pairs < resident : max_tokens <= 1536 && pairs < 2 * kSmCount) chunk = 512;
    else if (groups == 2 ? max_tokens > 4096 && max_tokens <= 8192 && pairs < 2 * resident : max_tokens <= 8192 && 5 * pairs < 4 * resident) chunk = 1024;
    for (; chunk > 256; chunk >>= 1) {
        const int64_t parts = (max_tokens + chunk - 1) / chunk;
        const double blocks_per_sm = groups == 2 ? (max_tokens <= 2048 ? 1.5 : chunk <= 512 ? 1.8 : 2.0)
                                                 : (parts == 1 ? 2.5 : max_tokens <= 2048 && chunk <= 512 ? 2.25 : 3.0);
        if (static_cast<double>(pairs * parts) >= blocks_per_sm * kSmCount) break;
    }
    chunk = (chunk + block_size - 1) / block_size * block_size;
    return static_cast<int>(chunk < max_tokens ? chunk : max_tokens);
}

// The most parts that a step of up to so many pairs with tables of up to so many keys is shared out into, beyond one for each 2048 keys of a pair (these
// grow with both): clusters and halves, chunks that were halved to fill the chip, then the lines of chunk_tokens where 16-bit caches begin with 512 and
// 1024 keys (8-bit caches stay below them).
int64_t most_parts(int64_t pairs, int64_t max_tokens) {
    auto up_to = [&](int64_t most_pairs, int64_t most_tokens, int64_t chunk) {
        return (pairs < most_pairs ? pairs : most_pairs) * (((max_tokens < most_tokens ? max_tokens : most_tokens) + chunk - 1) / chunk);
    };
    const int64_t each = (max_tokens + 255) / 256, filling = 2 * 3 * kSmCount;   // (at most 3 blocks per SM before the last halving)
    int64_t parts = pairs * (each > kMaxCluster ? each : kMaxCluster);
    if (parts > filling) parts = filling;
    if (max_tokens > 2048) parts = std::max(parts, up_to(2 * kSmCount - 1, 4096, 512));
    if (max_tokens > 4096) parts = std::max(parts, up_to(4 * kSmCount - 1, 8192, 1024));
    return parts;
}

// Split-K scratch of the chunked split that earlier versions of this library used (chunks of 256 to 2048 keys).  The public
// workspace size never falls below it, because the limit of nvk_decode_attention_paged_static and what counts as a problem that
// needs no scratch at all are stated in terms of it.
size_t chunk_scratch_bytes(int64_t batch, int num_heads, int num_kv_heads, int head_dim, int64_t max_blocks, int block_size) {
    const int64_t max_tokens = max_blocks * block_size;
    int64_t chunk = 2048;
    while (chunk > 256 && batch * num_kv_heads * ((max_tokens + chunk - 1) / chunk) < kSmCount) chunk >>= 1;
    chunk = (chunk + block_size - 1) / block_size * block_size;
    if (chunk > max_tokens) chunk = max_tokens;
    if (chunk > 128LL * block_size) chunk = 128LL * block_size;
    const int64_t splits = (max_tokens + chunk - 1) / chunk;
    if (splits <= 1) return 0;
    const size_t rows = static_cast<size_t>(batch) * num_heads * splits;
    return (rows * sizeof(float) + 15) / 16 * 16 + rows * static_cast<size_t>(head_dim) * sizeof(float);
}

struct Splits { int cluster, chunk, count; };   // cluster size, 0: single blocks; chunk length, 0: equal ranges; ranges of a table row
size_t part_bytes(size_t parts, int group) { return parts * group * (kHeadDim * sizeof(float) + sizeof(float2)); }
size_t part_count(const Splits& s, int64_t batch, int num_kv_heads) {   // (the cluster kernel itself needs none: the mixed step does)
    return s.count > 1 ? static_cast<size_t>(batch) * num_kv_heads * s.count : 0;
}
Splits choose_splits(int64_t batch, int num_heads, int num_kv_heads, int64_t max_blocks, int block_size, int groups, bool have_workspace) {
    Splits s{cluster_size(batch, num_kv_heads, max_blocks, block_size, groups, have_workspace), 0, 0};
    if (s.cluster > 0) { s.count = s.cluster; return s; }
    const int64_t max_tokens = max_blocks * block_size;
    if (max_blocks > 1 && halves(batch * num_kv_heads, max_tokens, groups)) {
        s.chunk = static_cast<int>((max_blocks + 1) / 2 * block_size);
        s.cluster = s.count = 2;
        return s;
    }
    s.chunk = chunk_tokens(batch, num_kv_heads, max_blocks, block_size, groups);
    s.count = static_cast<int>((max_tokens + s.chunk - 1) / s.chunk);
    // A row of partial results takes 520 bytes, 516 in earlier versions: what filled the array of nvk_decode_attention_paged_static almost
    // to the end must still fit (127 sequences of 32 / 8 heads, 32768-key tables), in longer chunks.
    while (part_bytes(part_count(s, batch, num_kv_heads), (num_heads + num_kv_heads - 1) / num_kv_heads) > kStaticScratchBytes &&
           chunk_scratch_bytes(batch, num_heads, num_kv_heads, kHeadDim, max_blocks, block_size) <= kStaticScratchBytes) {
        s.chunk *= 2;
        s.count = static_cast<int>((max_tokens + s.chunk - 1) / s.chunk);
    }
    return s;
}

}  // namespace

// Kernel parameters of a decode call from host-known sizes only, for kernels with `groups` resident groups per SM; returns in
// *cluster the cluster size, 0 = chunks.
int decode_plan(const DecodeArgs& a, int groups, dec::DecodeParams* out, int* cluster) {
    DecodeParams p{};
    p.q = a.q; p.k_cache = a.k_cache; p.v_cache = a.v_cache;
    p.context_lens = a.context_lens; p.block_tables = a.block_tables; p.out = a.out;
    p.max_blocks = a.max_blocks; p.num_cache_blocks = a.num_cache_blocks; p.batch = static_cast<int>(a.batch);
    p.num_heads = a.num_heads; p.num_kv_heads = a.num_kv_heads; p.group = a.num_heads / a.num_kv_heads;
    p.block_size = a.block_size;
    p.scale_log2 = a.scale * kLog2e;
    p.beside = a.beside ? 1 : 0;
    if (a.batch * a.num_heads * kMaxCluster >= (1LL << 31) || a.max_blocks * a.block_size >= (1LL << 31) - kTileTokens * kMaxCluster)
        return fail(NVK_ERR_UNSUPPORTED, "decode attention: batch or block table too large");
    const Splits s = choose_splits(a.batch, a.num_heads, a.num_kv_heads, a.max_blocks, a.block_size, groups, a.workspace != nullptr);
    *cluster = s.cluster;
    p.per_seq = s.chunk == 0 ? 1 : 0;
    while ((1 << p.split_shift) < s.cluster) ++p.split_shift;
    p.by_block = FastDiv(static_cast<uint32_t>(a.block_size));
    p.by_kv_heads = FastDiv(static_cast<uint32_t>(a.num_kv_heads));
    p.chunk_tokens = s.chunk;
    p.num_splits = s.count;
    // More than one wave of blocks: the long contexts first, so that the last blocks to start are short.  Contexts in a few chunks as well:
    // 38 / 44 sequences of 500 / 2000 to 4096 keys, 8 KV heads, 65.4 / 90.1 -> 58.7 / 85.9 us a call (whole 59.8 / 84.7).
    p.longest_first = s.chunk > 0 && (s.count == 1 || a.max_blocks * a.block_size <= 4096) && a.batch * a.num_kv_heads > static_cast<int64_t>(kSmCount) * groups &&
                      a.batch <= kMaxSorted && a.max_blocks * a.block_size >= kMinSortedTokens;
    // Contexts shorter than the table leave chunks without keys, whose blocks exit at once.  With sequence after sequence they lie between
    // the blocks with work, and these pile up on the SMs where the empty ones were quickest gone; chunk after chunk the ones with
    // work come first and spread evenly (us a call: 2 int8 sequences of 3000 keys, 8 KV heads, 32768-key tables, 21.4 -> 14.4; 37 of 1000
    // keys 31.2 -> 23.6; 64 of 9000 keys, 10240-key tables, 200.8 -> 190.2; 24 16-bit ones of 300 keys 15.3 -> 10.4).  From two waves of 16-bit
    // blocks on HBM is the bound and the empty ones cost least among the others (128 of 1000 keys: 82.5, chunk after chunk 92.8).
    p.chunk_major = groups == 3 || a.batch * a.num_kv_heads < 2 * static_cast<int64_t>(kSmCount) * groups;
    if (a.workspace != nullptr) {
        p.ws_o = static_cast<float*>(a.workspace);
        p.ws_ml = reinterpret_cast<float2*>(p.ws_o + part_count(s, a.batch, a.num_kv_heads) * p.group * kHeadDim);
    }
    *out = p;
    return NVK_OK;
}

namespace {

template <typename T>
int launch_merge_typed(const dec::DecodeParams& p, cudaStream_t stream) {
    if (p.num_splits <= 1) return NVK_OK;
    cudaError_t e;
    if (p.num_splits > kMergeWarps && p.batch * p.num_heads <= kMergeBlockRows) {
        e = launch_pdl(decode_merge_kernel<T, 0>, dim3(p.batch * p.num_heads), dim3(kMergeWarps * 32), 0, stream, p);
    } else {
        const int hg = p.group == 1 || (p.num_splits > 4 && p.batch * p.num_heads <= kMergeSingleRows) ? 1 : p.group == 2 ? 2 : 4;
        const dim3 grid((p.batch * p.num_kv_heads * ((p.group + hg - 1) / hg) + kMergeBlockWarps - 1) / kMergeBlockWarps), block(kMergeBlockWarps * 32);
        e = hg == 4 ? launch_pdl(decode_merge_kernel<T, 4>, grid, block, 0, stream, p)
            : hg == 2 ? launch_pdl(decode_merge_kernel<T, 2>, grid, block, 0, stream, p)
                      : launch_pdl(decode_merge_kernel<T, 1>, grid, block, 0, stream, p);
    }
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode_merge_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("decode_merge_kernel launch");
}

int check_grid(const DecodeArgs& a, const dec::DecodeParams& p) {   // of decode_split_kernel
    if (a.batch > 65535 || p.num_splits > 65535) return fail(NVK_ERR_UNSUPPORTED, "decode attention: batch or split count exceeds grid limits");
    return NVK_OK;
}

template <class F, typename T>
int launch_typed(const DecodeArgs& a, const void* k_scale, const void* v_scale) {
    constexpr int kSmem = static_cast<int>(sizeof(GroupSmem<F>));
    static std::atomic<bool> attr_done[64] = {};  // per device; the attribute calls are idempotent
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 0 && device < 64 && !attr_done[device]) {
        cudaError_t e = cudaFuncSetAttribute(decode_split_kernel<F, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_cluster_kernel<F, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        attr_done[device] = true;
    }
    DecodeParams p{};
    int cluster = 0;
    const int rc = decode_plan(a, F::kGroups, &p, &cluster);
    if (rc != NVK_OK) return rc;
    p.k_scale = static_cast<const __half*>(k_scale); p.v_scale = static_cast<const __half*>(v_scale);
    if (cluster > 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>(a.batch * a.num_kv_heads * cluster));
        cfg.blockDim = dim3(kGroupThreads);
        cfg.dynamicSmemBytes = kSmem;
        cfg.stream = a.stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_cluster_kernel<F, T>, p);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode_cluster_kernel launch: %s", cudaGetErrorString(e));
        return check_launch("decode_cluster_kernel launch");
    }
    if (const int rc1 = check_grid(a, p); rc1 != NVK_OK) return rc1;
    const unsigned batch = static_cast<unsigned>(a.batch), splits = static_cast<unsigned>(p.num_splits);
    const dim3 grid = p.chunk_major ? dim3(a.num_kv_heads, batch, splits) : dim3(a.num_kv_heads, splits, batch);
    const cudaError_t e = launch_pdl(decode_split_kernel<F, T>, grid, dim3(kGroupThreads), kSmem, a.stream, p);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode_split_kernel launch: %s", cudaGetErrorString(e));
    const int rc2 = check_launch("decode_split_kernel launch");
    return rc2 != NVK_OK ? rc2 : launch_merge_typed<T>(p, a.stream);
}

bool shape_supported(const DecodeArgs& a) {
    if (a.dtype != NVK_F16 && a.dtype != NVK_BF16) return false;
    if (a.head_dim != kHeadDim) return false;
    if (a.num_kv_heads <= 0 || a.num_heads % a.num_kv_heads != 0) return false;
    if (a.num_heads / a.num_kv_heads > kMaxGroup) return false;
    if (a.block_size < kTileTokens || a.block_size % kTileTokens != 0) return false;
    return aligned_to(a.k_cache, 16) && aligned_to(a.v_cache, 16) && aligned_to(a.out, 8);
}

}  // namespace

// The merge after a mixed step's decode half.
int launch_decode_merge(const dec::DecodeParams& p, int dtype, cudaStream_t stream) {
    return dtype == NVK_BF16 ? launch_merge_typed<__nv_bfloat16>(p, stream) : launch_merge_typed<__half>(p, stream);
}

// Whether launch_decode_mma can run a call of this size, for callers that launch something else before it.
int check_decode_mma(const DecodeArgs& a) {
    dec::DecodeParams p{};
    int cluster = 0;
    const int rc = decode_plan(a, Cache16<__half>::kGroups, &p, &cluster);
    return rc != NVK_OK || cluster > 0 ? rc : check_grid(a, p);
}

bool decode_mma_supported(const DecodeArgs& a) { return shape_supported(a) && aligned_to(a.q, 4); }

size_t decode_mma_workspace_needed(int64_t batch, int num_heads, int num_kv_heads, int head_dim,
                                   int64_t max_blocks, int block_size) {
    if (batch <= 0 || num_heads <= 0 || num_kv_heads <= 0 || max_blocks <= 0 || block_size <= 0) return 0;
    size_t need = chunk_scratch_bytes(batch, num_heads, num_kv_heads, head_dim, max_blocks, block_size);
    for (int groups : {Cache16<__half>::kGroups, Cache8<__half, false>::kGroups}) {
        const Splits s = choose_splits(batch, num_heads, num_kv_heads, max_blocks, block_size, groups, true);
        const size_t n = part_bytes(part_count(s, batch, num_kv_heads), (num_heads + num_kv_heads - 1) / num_kv_heads);
        if (n > need) need = n;
    }
    return need;
}

// The same for every call with no more sequences and no wider tables: a smaller one may be cut into more parts (8 sequences of 1024 keys, 8 KV heads, take
// clusters of four, 32 whole contexts), and callers keep one workspace for all of them.
size_t decode_mma_workspace_bytes(int64_t batch, int num_heads, int num_kv_heads, int head_dim,
                                  int64_t max_blocks, int block_size) {
    const size_t need = decode_mma_workspace_needed(batch, num_heads, num_kv_heads, head_dim, max_blocks, block_size);
    // Whole contexts in narrow tables: none, and a caller without scratch passes none to smaller calls either.  (But with 1.5 to 2.5 pairs to an SM,
    // where 8-bit caches were once cut in two, the one workspace has always been enough for fewer sequences.)
    const int64_t pairs = batch * num_kv_heads;
    if (need == 0 && (2 * pairs <= 3 * kSmCount || 2 * pairs >= 5 * kSmCount)) return 0;
    const int group = (num_heads + num_kv_heads - 1) / num_kv_heads;
    const size_t most = part_bytes(static_cast<size_t>(most_parts(pairs, max_blocks * block_size)), group);
    // What fits the static array never needs more than it holds; what fills it but for the last 4 bytes a row of 520 goes on in longer chunks (above), a
    // slightly smaller one fills it.
    if (need <= kStaticScratchBytes && (most > kStaticScratchBytes || need + need / 128 > kStaticScratchBytes)) return kStaticScratchBytes;
    return most > need ? most : need;
}

bool decode_int8_mma_supported(const DecodeInt8Args& x) {
    const DecodeArgs& a = x.base;
    if (!shape_supported(a) || !aligned_to(a.q, 2)) return false;
    if (!aligned_to(x.k_scale, 4) || !aligned_to(x.v_scale, 4)) return false;   // scales are copied as aligned 32-bit words
    return (a.num_cache_blocks * a.block_size * a.num_kv_heads) % 2 == 0;
}

int launch_decode_int8_mma(const DecodeInt8Args& x) {
    using bf = __nv_bfloat16;
    if (x.fp8)
        return x.base.dtype == NVK_BF16 ? launch_typed<Cache8<bf, true>, bf>(x.base, x.k_scale, x.v_scale)
                                        : launch_typed<Cache8<__half, true>, __half>(x.base, x.k_scale, x.v_scale);
    return x.base.dtype == NVK_BF16 ? launch_typed<Cache8<bf, false>, bf>(x.base, x.k_scale, x.v_scale)
                                    : launch_typed<Cache8<__half, false>, __half>(x.base, x.k_scale, x.v_scale);
}

int launch_decode_mma(const DecodeArgs& a) {
    return a.dtype == NVK_BF16 ? launch_typed<Cache16<__nv_bfloat16>, __nv_bfloat16>(a, nullptr, nullptr)
                               : launch_typed<Cache16<__half>, __half>(a, nullptr, nullptr);
}

}  // namespace nvk

// ---------------------------------------------------------------------------------------------
// Allocation-free variant: split-K scratch in a fixed device array owned by this library.
//
// Some callers of decode attention have no way to hand over a workspace: the reference's own
// launch_decode_attention_paged signature carries no allocator, an engine may already have given
// every free byte of HBM to its KV-cache pool, and code running under a "no device allocation
// after start-up" rule (latency-critical serving loops, plug-ins that are only handed tensors)
// must not call cudaMalloc at all.  For them the split-K partials live in the array below.  It is
// part of the loaded module, so every GPU that uses this library keeps kStaticScratchBytes of HBM
// reserved until the process exits.
// ---------------------------------------------------------------------------------------------
namespace nvk {
namespace {

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
std::atomic<void*> g_scratch_addr[kMaxDevices];   // null until the first call on that device (static storage: zeroed)

// Resolves the device address of g_static_scratch for the current device (once per device).
// In host code the symbol's name is only a handle; the kernels need the address returned here.
int static_scratch_for_current_device(void** out) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode attention (static scratch): cudaGetDevice: %s", cudaGetErrorString(e));
    if (device < 0 || device >= kMaxDevices)
        return fail(NVK_ERR_UNSUPPORTED, "decode attention (static scratch): device index %d not supported", device);
    void* ptr = g_scratch_addr[device].load(std::memory_order_acquire);
    if (ptr == nullptr) {   // two threads racing here both look the same address up; either store is fine
        e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || ptr == nullptr)
            return fail(NVK_ERR_CUDA, "decode attention (static scratch): cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_scratch_addr[device].store(ptr, std::memory_order_release);
    }
    *out = ptr;
    return NVK_OK;
}

}  // namespace
}  // namespace nvk

extern "C" size_t nvk_decode_attention_static_scratch_bytes(void) { return nvk::kStaticScratchBytes; }

extern "C" int nvk_decode_attention_paged_static(const void* query, const void* k_cache, const void* v_cache,
                                                 const void* context_lens, int context_lens_dtype,
                                                 const void* block_tables, int block_tables_dtype,
                                                 int64_t batch, int64_t max_blocks, int64_t num_cache_blocks,
                                                 int num_heads, int num_kv_heads, int head_dim, int block_size,
                                                 float scale, void* output, int dtype, void* stream) {
    using namespace nvk;
    const size_t need = decode_mma_workspace_needed(batch, num_heads, num_kv_heads, head_dim, max_blocks, block_size);
    if (need > kStaticScratchBytes)
        return fail(NVK_ERR_INVALID_ARGUMENT,
                    "decode attention (static scratch): this problem needs %zu bytes of split-K scratch but the built-in "
                    "array holds %zu; use nvk_decode_attention_paged with a caller-provided workspace",
                    need, kStaticScratchBytes);
    void* scratch = nullptr;
    // A problem that is not worth splitting leaves the shared array alone, so that such calls may overlap.
    if (batch > 0 && num_heads > 0 && num_kv_heads > 0 && block_size > 0 && max_blocks > 0 &&
        chunk_scratch_bytes(batch, num_heads, num_kv_heads, head_dim, max_blocks, block_size) > 0) {
        const int rc = static_scratch_for_current_device(&scratch);
        if (rc != NVK_OK) return rc;
    }
    // Every part is fully written before the merge kernel reads it, and only written parts are read, so nothing in the array has
    // to start at zero.
    return nvk_decode_attention_paged(query, k_cache, v_cache, context_lens, context_lens_dtype, block_tables,
                                      block_tables_dtype, batch, max_blocks, num_cache_blocks, num_heads, num_kv_heads, head_dim, block_size, scale, output,
                                      dtype, scratch, scratch != nullptr ? kStaticScratchBytes : 0, stream);
}
