// Varlen causal prefill attention for sm_100a (F16 / BF16, head_dim 128), dense or paged keys, on mma.sync: small steps, and what the tcgen05
// kernels of prefill_attn_tc.cu do not take (cache blocks that are no multiple of 128, scales that are not positive).
//
// Replaces prefill_dense_attention_kernel / prefill_paged_attention_kernel
// (src/kernels/attention.cu:114-302 of the reference: one block per (query row, head), serial
// over keys with a block reduction and two barriers per key) and the FlashAttention-2 varlen call
// (src/kernels/flash_attn.cpp:203-300).  One kernel serves both key layouts: the reference sends
// a batch with any prefix-cache hit through the scalar paged kernel
// (src/layers/attention.cpp:142-157); here cached prefix blocks and freshly stored tokens are
// read through block_tables by the same tiled kernel.
//
// An item is 64 rows of one KV head, 64 >> head_shift query rows x 1 << head_shift heads, so that short and ragged sequences fill their tiles.  The
// blocks of a cluster share an item's key tiles (64 keys), and each pushes its part (unnormalised output, maximum, sum) of every row to the
// block that finishes the row; after one cluster barrier everything is local.  4 warps x 16 rows; keys staged by 16-byte cp.async into XOR-swizzled
// shared memory (two stages); S = Q K^T and O += P V as mma.sync m16n8k16 with fp32 accumulation; online softmax in the exp2 domain; key tiles
// above the bottom-right-aligned diagonal are skipped, the diagonal tile is masked per element.  Two blocks per SM.
#include "nvk_internal.cuh"

#include <atomic>
#include <cmath>

namespace nvk {
namespace {

constexpr int kHeadDim = 128;
constexpr int kBM = 64;                 // rows per item
constexpr int kBN = 64;                 // keys per tile
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kRowBytes = kHeadDim * 2;
constexpr int kQBytes = kBM * kRowBytes;          // 16 KiB
constexpr int kKVTileBytes = kBN * kRowBytes;     // 16 KiB each for K and V
constexpr int kStageBytes = 2 * kKVTileBytes;
constexpr int kStages = 2;
constexpr int kSmemBytes = kQBytes + kStages * kStageBytes;  // 80 KiB
constexpr int kPartRow = kHeadDim * 4 + 8;                   // a row of a part: 128 floats, behind a run of rows their (maximum, sum)
constexpr int kPartBytes = kBM * kPartRow;                   // what a block receives, from all blocks of its cluster: 32.5 KiB
constexpr long long kWaitCycles = 4000000000LL;              // some 2 s
constexpr int kMaxCluster = 8;                               // portable cluster size

struct PrefillParams {
    const void* q; const void* k; const void* v; void* out;
    IndexArray cu_q, cu_k, block_tables;
    int64_t num_seqs, total_q, total_k, max_blocks, num_cache_blocks, key_rows;   // key_rows: rows addressable in k / v
    int num_heads, num_kv_heads, block_size;
    int head_shift;        // an item's rows are 64 >> head_shift query rows x 1 << head_shift heads
    int csize_shift;       // log2 of the cluster size
    unsigned int tiles;    // upper bound of query tiles over all sequences
    FastDiv by_sets;       // sets of 1 << head_shift heads
    FastDiv by_block, by_group;
    float scale_log2;
};

__device__ __forceinline__ uint32_t swz(int row, int chunk) {
    return static_cast<uint32_t>(row * kRowBytes + ((chunk ^ (row & 7)) << 4));
}
__device__ int g_prefill_error = 0;

template <typename T>
__global__ void __launch_bounds__(kThreads, 2) prefill_tile_kernel(const __grid_constant__ PrefillParams p) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t s_bar;  // the cluster's parts have landed
    pdl_wait_then_release();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int csize = 1 << p.csize_shift, rank = static_cast<int>(blockIdx.x) & (csize - 1);
    const unsigned int item = blockIdx.x >> p.csize_shift, tile = p.by_sets.div(item);
    const int head0 = static_cast<int>(item - tile * p.by_sets.d) << p.head_shift;
    const int kvh = static_cast<int>(p.by_group.div(head0));
    const int tok_shift = 6 - p.head_shift;

    const IndexArray::Raw first_ids = p.block_tables ? p.block_tables.raw(lane, p.num_seqs == 1 && lane < p.max_blocks) : IndexArray::Raw{0, 0};
    // Sequence and first query row of the (reversed: heavier tiles first) tile, by every warp for itself: 32 sequences at a time, one per lane.
    int seq = 0, q0, qb, kb, q_len, k_len;
    int want = static_cast<int>(p.tiles - 1 - tile);
    if (p.cu_q == nullptr) {
        qb = 0; kb = 0; q_len = static_cast<int>(p.total_q); k_len = static_cast<int>(p.total_k);
        q0 = want << tok_shift;
        if (q0 >= q_len) return;             // (here and below the whole cluster leaves)
    } else if (p.num_seqs == 1) {            // nothing to look for, and the block ids are on their way with the bounds
        const IndexArray::Raw rq0 = p.cu_q.raw(0), rq1 = p.cu_q.raw(1), rk0 = p.cu_k.raw(0), rk1 = p.cu_k.raw(1);
        qb = static_cast<int>(p.cu_q.value(rq0)); q_len = static_cast<int>(p.cu_q.value(rq1)) - qb;
        kb = static_cast<int>(p.cu_k.value(rk0)); k_len = static_cast<int>(p.cu_k.value(rk1)) - kb;
        q0 = want << tok_shift;
        if (q0 >= q_len) return;
    } else {
        for (int base = 0;; base += 32) {
            const bool in = base + lane < p.num_seqs;
            const IndexArray::Raw rq0 = p.cu_q.raw(base + lane, in), rq1 = p.cu_q.raw(base + lane + 1, in);
            const IndexArray::Raw rk0 = p.cu_k.raw(base + lane, in), rk1 = p.cu_k.raw(base + lane + 1, in);
            const int b0 = static_cast<int>(p.cu_q.value(rq0)), n = static_cast<int>(p.cu_q.value(rq1)) - b0;
            const int k0 = static_cast<int>(p.cu_k.value(rk0)), kn = static_cast<int>(p.cu_k.value(rk1)) - k0;
            const int mine = max((n + (1 << tok_shift) - 1) >> tok_shift, 0);
            int upto = mine;
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const int up = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += up;
            }
            const unsigned int past = __ballot_sync(0xffffffffu, upto > want);
            if (past != 0) {
                const int at = __ffs(past) - 1;
                seq = base + at;
                q0 = (want - __shfl_sync(0xffffffffu, upto - mine, at)) << tok_shift;
                qb = __shfl_sync(0xffffffffu, b0, at); q_len = __shfl_sync(0xffffffffu, n, at);
                kb = __shfl_sync(0xffffffffu, k0, at); k_len = __shfl_sync(0xffffffffu, kn, at);
                break;
            }
            if (base + 32 >= p.num_seqs) return;
            want -= __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    const int own_shift = 6 - p.csize_shift, own = 1 << own_shift;   // rows that a block finishes
    const uint32_t bar = smem_u32(&s_bar);
    if (csize > 1) {
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\nfence.mbarrier_init.release.cluster;\n" ::"r"(bar) : "memory");
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(kPartBytes) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");   // (waited for before the first push: every block's barrier is set up)
    }
    const int rows_here = min(1 << tok_shift, q_len - q0);   // query rows
    const int shift = k_len - q_len;                         // bottom-right alignment
    const int k_hi = min(shift + q0 + rows_here, k_len);     // keys visible to the last row of the tile
    const int all_kt = k_hi > 0 ? (k_hi + kBN - 1) / kBN : 0;
    const int kt0 = all_kt * rank >> p.csize_shift, kt1 = all_kt * (rank + 1) >> p.csize_shift;   // this block's key tiles

    const uint32_t q_u32 = smem_u32(smem);
    const uint32_t kv_u32 = q_u32 + kQBytes;
    const IndexArray table = p.block_tables ? p.block_tables + static_cast<int64_t>(seq) * p.max_blocks : IndexArray();
    const size_t kv_row_stride = static_cast<size_t>(p.num_kv_heads) * kRowBytes;
    const unsigned char* kbase = static_cast<const unsigned char*>(p.k) + static_cast<size_t>(kvh) * kRowBytes;
    const unsigned char* vbase = static_cast<const unsigned char*>(p.v) + static_cast<size_t>(kvh) * kRowBytes;

    const int c = tid & 15;        // 16-byte column handled by this thread
    const int r0 = tid >> 4;       // first row; rows r0 + 8 i

    // Lane i holds the cache block of table entry id_base + i (-1: outside the cache, reads as zeros).
    int id_base = 0, ids = -1;
    auto take_ids = [&](IndexArray::Raw raw) {
        const int64_t id = table.value(raw);
        ids = id >= 0 && id < p.num_cache_blocks ? static_cast<int>(id) : -1;
    };
    auto load_ids = [&](int kt) {
        id_base = static_cast<int>(p.by_block.div(kt * kBN));
        take_ids(table.raw(id_base + lane, id_base + lane < p.max_blocks));
    };
    if (table && kt0 < kt1) {
        if (p.num_seqs == 1) take_ids(first_ids);   // (a range that starts past 32 entries loads its own when it comes to them)
        else load_ids(kt0);
    }

    // Q tile -> shared (rows beyond the sequence are zero filled)
    const size_t row_bytes = static_cast<size_t>(p.num_heads) * kRowBytes;   // of a query row
    if (kt0 < kt1) {
        const unsigned char* qsrc = static_cast<const unsigned char*>(p.q) + static_cast<size_t>(qb + q0) * row_bytes + static_cast<size_t>(head0) * kRowBytes + c * 16;
#pragma unroll
        for (int i = 0; i < kBM / 8; ++i) {
            const int r = r0 + 8 * i, tok = r >> p.head_shift;
            const int bytes = tok < rows_here ? 16 : 0;
            cp_async16(q_u32 + swz(r, c), qsrc + (bytes ? tok * row_bytes + (r & ((1 << p.head_shift) - 1)) * kRowBytes : 0), bytes);
        }
    }
    auto issue_kv = [&](int kt) {
        const int key0 = kt * kBN;
        const uint32_t stage = kv_u32 + (kt % kStages) * kStageBytes;
        int64_t tile_row0 = kb + key0;
        bool tile_ok = true;
        if (table) {   // a 64-key tile never straddles a cache block (block_size % 64 == 0)
            const int blk = static_cast<int>(p.by_block.div(key0));
            if (blk - id_base >= 32) load_ids(kt);
            const int id = __shfl_sync(0xffffffffu, ids, blk - id_base);
            tile_row0 = static_cast<int64_t>(id) * p.block_size + (key0 - blk * p.block_size);
            tile_ok = id >= 0;
        }
#pragma unroll
        for (int i = 0; i < kBN / 8; ++i) {
            const int r = r0 + 8 * i;
            const int64_t src_row = tile_row0 + r;
            const int bytes = (tile_ok && key0 + r < k_len && src_row < p.key_rows) ? 16 : 0;
            const size_t off = (bytes ? static_cast<size_t>(src_row) * kv_row_stride : 0) + c * 16;
            cp_async16(stage + swz(r, c), kbase + off, bytes);
            cp_async16(stage + kKVTileBytes + swz(r, c), vbase + off, bytes);
        }
    };
    if (kt0 < kt1) issue_kv(kt0);
    cp_async_commit();

    float o[16][4];
#pragma unroll
    for (int i = 0; i < 16; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f; }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.0f, 0.0f};
    uint32_t qa[8][4];

    const int row0 = warp * 16 + g;                                                 // and row0 + 8
    const int lim0 = min(shift + q0 + (row0 >> p.head_shift) + 1, k_len);          // keys [0, lim) are visible
    const int lim1 = min(shift + q0 + ((row0 + 8) >> p.head_shift) + 1, k_len);
    const int least = min(shift + q0 + ((warp * 16) >> p.head_shift) + 1, k_len), most = min(shift + q0 + ((warp * 16 + 15) >> p.head_shift) + 1, k_len);

    // ldmatrix lane addressing
    const int a_row = warp * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);
    const int a_sel = lane >> 4;
    const int kb_row = ((lane >> 4) << 3) + (lane & 7);
    const int kb_sel = (lane >> 3) & 1;
    const int vb_row = ((lane >> 3) & 1) * 8 + (lane & 7);
    const int vb_sel = lane >> 4;

#pragma unroll 1
    for (int kt = kt0; kt < kt1; ++kt) {
        if (kt + 1 < kt1) issue_kv(kt + 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        if (kt == kt0) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
                ldmatrix_x4(qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], q_u32 + swz(a_row, 2 * ks + a_sel));
        }
        const uint32_t stage = kv_u32 + (kt % kStages) * kStageBytes;
        const int key0 = kt * kBN;
        // a warp whose rows see none of this tile's keys skips the math (still takes the barriers)
        if (key0 < most) {
            float s[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.0f; }
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
                for (int np = 0; np < 4; ++np) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4(b0, b1, b2, b3, stage + swz(np * 16 + kb_row, 2 * ks + kb_sel));
                    mma_16816<T>(s[2 * np], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
                    mma_16816<T>(s[2 * np + 1], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b2, b3);
                }
            }
            const bool need_mask = key0 + kBN > least;   // warp-uniform
            float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
                for (int e = 0; e < 4; ++e) s[nt][e] *= p.scale_log2;
                if (need_mask) {
                    const int key = key0 + nt * 8 + 2 * t;
                    if (key >= lim0) s[nt][0] = -INFINITY;
                    if (key + 1 >= lim0) s[nt][1] = -INFINITY;
                    if (key >= lim1) s[nt][2] = -INFINITY;
                    if (key + 1 >= lim1) s[nt][3] = -INFINITY;
                }
                mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
                mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
            }
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
            const float mn0 = fmaxf(m_run[0], mx0), mn1 = fmaxf(m_run[1], mx1);
            const float base0 = mn0 == -INFINITY ? 0.0f : mn0;   // fully masked row so far
            const float base1 = mn1 == -INFINITY ? 0.0f : mn1;
            const float corr0 = fast_exp2(m_run[0] - base0), corr1 = fast_exp2(m_run[1] - base1);
            m_run[0] = mn0; m_run[1] = mn1;
            float sum0 = 0.0f, sum1 = 0.0f;
            uint32_t pa[4][4];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float p0 = fast_exp2(s[nt][0] - base0), p1 = fast_exp2(s[nt][1] - base0);
                const float p2 = fast_exp2(s[nt][2] - base1), p3 = fast_exp2(s[nt][3] - base1);
                sum0 += p0 + p1; sum1 += p2 + p3;
                pa[nt >> 1][(nt & 1) * 2] = ElemTraits<T>::pack2(p0, p1);
                pa[nt >> 1][(nt & 1) * 2 + 1] = ElemTraits<T>::pack2(p2, p3);
            }
            l_run[0] = l_run[0] * corr0 + sum0;
            l_run[1] = l_run[1] * corr1 + sum1;
#pragma unroll
            for (int nt = 0; nt < 16; ++nt) { o[nt][0] *= corr0; o[nt][1] *= corr0; o[nt][2] *= corr1; o[nt][3] *= corr1; }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
                for (int dp = 0; dp < 8; ++dp) {
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(b0, b1, b2, b3, stage + kKVTileBytes + swz(kk * 16 + vb_row, 2 * dp + vb_sel));
                    mma_16816<T>(o[2 * dp], pa[kk][0], pa[kk][1], pa[kk][2], pa[kk][3], b0, b1);
                    mma_16816<T>(o[2 * dp + 1], pa[kk][0], pa[kk][1], pa[kk][2], pa[kk][3], b2, b3);
                }
            }
        }
        __syncthreads();
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 1);
        l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], 2);
    }
    T* out = static_cast<T*>(p.out) + (static_cast<size_t>(qb + q0) * p.num_heads + head0) * kHeadDim;
    auto out_row = [&](int row) { return out + static_cast<size_t>(row >> p.head_shift) * p.num_heads * kHeadDim + (row & ((1 << p.head_shift) - 1)) * kHeadDim; };
    if (csize == 1) {
        // normalise, stage the warp's 16 x 128 tile over its own Q rows, 16-byte row stores
        __syncthreads();   // covers a block without tiles: shared memory is idle
        const float inv0 = l_run[0] > 0.0f ? 1.0f / l_run[0] : 0.0f;
        const float inv1 = l_run[1] > 0.0f ? 1.0f / l_run[1] : 0.0f;
        unsigned char* stage_out = smem + warp * 16 * kRowBytes;
#pragma unroll
        for (int nt = 0; nt < 16; ++nt) {   // 8 columns = one 16-byte chunk; lane t writes 4 bytes of it
            *reinterpret_cast<uint32_t*>(stage_out + swz(g, nt) + t * 4) = ElemTraits<T>::pack2(o[nt][0] * inv0, o[nt][1] * inv0);
            *reinterpret_cast<uint32_t*>(stage_out + swz(g + 8, nt) + t * 4) = ElemTraits<T>::pack2(o[nt][2] * inv1, o[nt][3] * inv1);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 2 * i + (lane >> 4), cc = lane & 15, row = warp * 16 + r;
            if ((row >> p.head_shift) < rows_here) reinterpret_cast<uint4*>(out_row(row))[cc] = *reinterpret_cast<const uint4*>(stage_out + swz(r, cc));
        }
        return;
    }
    // Row r is finished by block r / own.  A run of own rows lies together (16-byte pieces XOR-swizzled by row, so that a store's lanes hit different
    // banks; maxima and sums behind them) and goes to its block in one bulk copy: stored one by one from registers they took 5 us.
    __syncthreads();                         // all warps are done with the tiles, whose place the parts take
    const int run_bytes = own * kPartRow;
    {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = row0 + 8 * i, at = row & (own - 1);
            unsigned char* run = smem + (row >> own_shift) * run_bytes;
            if (kt0 < kt1) {
                float* dst = reinterpret_cast<float*>(run + at * kHeadDim * 4) + (t & 1) * 2;
#pragma unroll
                for (int nt = 0; nt < 16; ++nt)
                    *reinterpret_cast<float2*>(dst + ((2 * nt + (t >> 1)) ^ ((at & 15) << 1)) * 4) = make_float2(o[nt][2 * i], o[nt][2 * i + 1]);
            }
            if (t == 0) reinterpret_cast<float2*>(run + own * kHeadDim * 4)[at] = make_float2(m_run[i], l_run[i]);   // (minus infinity where there is nothing to add)
        }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
    if (tid < csize) push_bulk(smem_u32(smem) + kSmemBytes + rank * run_bytes, smem_u32(smem) + tid * run_bytes, run_bytes, bar, tid);
    __syncwarp();
    bool landed = false;
    for (const long long start = clock64(); !landed && clock64() - start < kWaitCycles;) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(ok) : "r"(bar) : "memory");
        landed = ok != 0;
    }
    if (!landed) atomicCAS(&g_prefill_error, 0, 41);
    asm volatile("barrier.cluster.arrive;\n" ::: "memory");           // what was pushed here has landed: its senders may leave
    const unsigned char* parts = smem + kSmemBytes;                    // [block of the cluster]: a run
#pragma unroll 1
    for (int at = warp; landed && at < own; at += kWarps) {            // a warp per row, four elements a lane; loads without branches
        const int row = (rank << own_shift) + at;
        if ((row >> p.head_shift) >= rows_here) break;
        float mx = -INFINITY, sum = 0.0f;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
        for (int r0 = 0; r0 < csize; r0 += 2) {
            float2 ml[2];
            float4 a[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const unsigned char* run = parts + (r0 + u) * run_bytes;
                ml[u] = reinterpret_cast<const float2*>(run + own * kHeadDim * 4)[at];
                a[u] = reinterpret_cast<const float4*>(run + at * kHeadDim * 4)[lane ^ ((at & 15) << 1)];
            }
            const float top = fmaxf(mx, fmaxf(ml[0].x, ml[1].x)), base = top == -INFINITY ? 0.0f : top, f = fast_exp2(mx - base);
            v.x *= f; v.y *= f; v.z *= f; v.w *= f;
            sum *= f;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                // (No maximum and no sum: there may be nothing written.  A part whose scores are all NaN has no maximum either, but a NaN as its sum.)
                const bool seen = ml[u].x != -INFINITY || ml[u].y != 0.0f;
                const float w = fast_exp2(ml[u].x - base);
                v.x = fmaf(w, seen ? a[u].x : 0.0f, v.x); v.y = fmaf(w, seen ? a[u].y : 0.0f, v.y);
                v.z = fmaf(w, seen ? a[u].z : 0.0f, v.z); v.w = fmaf(w, seen ? a[u].w : 0.0f, v.w);
                sum = fmaf(w, ml[u].y, sum);
            }
            mx = top;
        }
        const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
        reinterpret_cast<uint2*>(out_row(row))[lane] = make_uint2(ElemTraits<T>::pack2(v.x * inv, v.y * inv), ElemTraits<T>::pack2(v.z * inv, v.w * inv));
    }
    asm volatile("barrier.cluster.wait;\n" ::: "memory");             // no block leaves while its part is on its way, or others push to it
    if (!landed) {                           // give copies under way time to land (2 ms)
        const long long start = clock64();
        while (clock64() - start < 4000000) {}
    }
}

int tile_head_shift(int group) { return group % 8 == 0 ? 3 : group % 4 == 0 ? 2 : group % 2 == 0 ? 1 : 0; }

// What a step takes, in microseconds, from what the host knows: rows and, where the keys are not paged, keys of all sequences together, the block
// tables' width, maybe the longest sequence's rows.  `count` sequences of q rows that see `keys` keys each.
struct Alike { int64_t count, q, keys; };
int64_t sequences(const PrefillArgs& a) { return a.cu_q ? a.num_seqs : 1; }
int64_t ceil_div(int64_t n, int64_t by) { return (n + by - 1) / by; }
// All sequences equally long and, where block tables are wider than these need, behind a cached prefix of whole blocks.
Alike equal_lengths(const PrefillArgs& a) {
    const int64_t n = sequences(a), q = ceil_div(a.total_q, n);
    int64_t keys = ceil_div(a.total_k, n);
    if (a.block_tables) {
        const int64_t before = (a.max_blocks - 1) * a.block_size;
        keys = q > before ? q : before + (q < a.block_size ? q : a.block_size);
    }
    return {n, q, keys < 1 ? 1 : keys};
}
// The other end: sequences as long as any can be (`max_seqlen_q` where it is given; with paged keys none is longer than its table), and the rows that
// are left on the others.  False: all are of one length.
bool unequal_lengths(const PrefillArgs& a, Alike (&l)[2]) {
    const int64_t n = sequences(a), even = ceil_div(a.total_q, n), width = a.block_tables ? a.max_blocks * a.block_size : a.total_q;
    int64_t q = a.total_q - (n - 1);
    if (a.max_seqlen_q > 0 && a.max_seqlen_q < q) q = a.max_seqlen_q;
    if (width < q) q = width;
    if (n == 1 || q <= even) return false;
    int64_t count = a.block_tables || a.max_seqlen_q > 0 ? (a.total_q - n) / (q - 1) : 1;
    if (count < 1) count = 1;
    if (count > n - 1) count = n - 1;
    const int64_t left = a.total_q - count * q, rest = left > n - count ? ceil_div(left, n - count) : 1;
    if (a.block_tables) {
        const int64_t bs = a.block_size, before = (a.max_blocks - 1) * bs;
        auto keys = [&](int64_t rows) { return q > before ? rows : before + (rows < bs ? rows : bs); };
        l[0] = {count, q, keys(q)};
        l[1] = {n - count, rest, keys(rest)};
    } else {
        const int64_t before = a.total_k > a.total_q ? (a.total_k - a.total_q) / n : 0;
        l[0] = {count, q, before + q};
        l[1] = {n - count, rest, before + rest};
    }
    return true;
}
// Items of `rows` rows and `sets` per row range, the rounds of `step` keys that the longest takes, and all of them together.
struct Load { int64_t items, longest; double rounds; };
Load load_of(const Alike* l, int n, int64_t rows, int64_t sets, int64_t step) {
    Load w{0, 1, 0.0};
    for (int i = 0; i < n; ++i) {
        const int64_t ranges = ceil_div(l[i].q, rows), longest = ceil_div(l[i].keys, step);
        w.items += l[i].count * ranges * sets;
        if (longest > w.longest) w.longest = longest;
        const double keys = static_cast<double>(l[i].keys - l[i].q) + 0.5 * static_cast<double>((ranges + 1) * rows);   // of an item, on average
        w.rounds += static_cast<double>(l[i].count * ranges * sets) * (keys / static_cast<double>(step) + 0.5);
    }
    return w;
}
// Here a block takes 3.4 us and 1.4 for each of its key tiles, 2.1 where two share an SM, 2 more for each further wave of blocks, and 2.9 for the parts
// of a cluster (32 / 8 heads, with a store of 1.3 us: 77 tokens alone 7.4 us in one block each, 9.7 and 10.5 in clusters of 2 and 4; 8 on a prefix
// of 256, 5 tiles, 11.4, 9.6 and 8.3 in clusters of 2, 4 and 8).
double tile_time(const PrefillArgs& a, const Alike* l, int n, int csize_shift) {
    const int head_shift = tile_head_shift(a.num_heads / a.num_kv_heads);
    const Load w = load_of(l, n, kBM >> head_shift, a.num_heads >> head_shift, kBN);
    const int64_t blocks = w.items << csize_shift, waves = ceil_div(blocks, 2 * kSmCount), longest = ceil_div(w.longest, 1LL << csize_shift);
    double rounds = static_cast<double>(n == 1 ? waves * longest : longest);
    if (n > 1 && w.rounds > rounds * (2 * kSmCount)) rounds = w.rounds / (2 * kSmCount);
    return 3.4 + rounds * (blocks <= kSmCount ? 1.4 : 2.1) + 2.0 * static_cast<double>(waves - 1) + (csize_shift > 0 ? 2.9 : 0.0);
}
// log2 of the cluster size that takes least for equal lengths, of those that are resident at once.
int best_cluster(const PrefillArgs& a, const Alike& equal) {
    const int head_shift = tile_head_shift(a.num_heads / a.num_kv_heads);
    const int64_t rows = kBM >> head_shift, grid = (ceil_div(a.total_q, rows) + (a.cu_q ? a.num_seqs : 0)) * (a.num_heads >> head_shift);
    int best = 0;
    for (int s = 1; (1 << s) <= kMaxCluster && (grid << s) <= 2 * kSmCount; ++s)
        if (tile_time(a, &equal, 1, s) < tile_time(a, &equal, 1, best)) best = s;
    return best;
}
// The persistent tcgen05 kernel takes 6.8 us and 1.56 for each round of 128 keys of an item of 256 rows (half a microsecond in doubt).
double tcgen05_time(const PrefillArgs& a, const Alike* l, int n) {
    const int group = a.num_heads / a.num_kv_heads, heads = group % 8 == 0 ? 8 : group % 4 == 0 ? 4 : 2;   // of an item
    const Load w = load_of(l, n, 2 * 128 / heads, a.num_heads / heads, 128);
    const double waves = n == 1 ? static_cast<double>(ceil_div(w.items, kSmCount)) : static_cast<double>(w.items) / kSmCount;
    const double more = waves > 1.0 ? 1.5 * (waves - 1.0) : 0.0, longest = 1.56 * static_cast<double>(w.longest);
    if (n == 1) return 6.3 + waves * longest + more;
    const double all = 1.56 * w.rounds / kSmCount + more;
    return 6.3 + (all > longest ? all : longest);
}

template <typename T>
int launch_typed(const PrefillArgs& a) {
    static std::atomic<bool> attr_done[64] = {};
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 0 && device < 64 && !attr_done[device]) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes + kPartBytes);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        attr_done[device] = true;
    }
    PrefillParams p{};
    p.q = a.q; p.out = a.out; p.cu_q = a.cu_q; p.cu_k = a.cu_k; p.block_tables = a.block_tables;
    p.num_seqs = a.cu_q ? a.num_seqs : 1; p.total_q = a.total_q; p.total_k = a.total_k; p.max_blocks = a.max_blocks;
    p.num_heads = a.num_heads; p.num_kv_heads = a.num_kv_heads; p.block_size = a.block_tables ? a.block_size : 1;
    p.scale_log2 = a.scale * kLog2e;
    if (a.block_tables) { p.k = a.k_cache; p.v = a.v_cache; p.key_rows = a.num_cache_blocks * a.block_size; p.num_cache_blocks = a.num_cache_blocks; }
    else { p.k = a.k; p.v = a.v; p.key_rows = a.total_k; }
    const int group = a.num_heads / a.num_kv_heads;
    p.head_shift = tile_head_shift(group);
    const int64_t rows = kBM >> p.head_shift, sets = a.num_heads >> p.head_shift;
    const int64_t tiles = (a.total_q + rows - 1) / rows + (a.cu_q ? a.num_seqs : 0);
    p.by_sets = FastDiv(static_cast<uint32_t>(sets));
    p.by_block = FastDiv(static_cast<uint32_t>(p.block_size));
    p.by_group = FastDiv(static_cast<uint32_t>(group));
    p.csize_shift = best_cluster(a, equal_lengths(a));
    if (tiles * sets << p.csize_shift > 0x7fffffffLL || tiles > 0x7fffffffLL) return fail(NVK_ERR_UNSUPPORTED, "prefill attention: grid too large");
    p.tiles = static_cast<unsigned int>(tiles);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * sets << p.csize_shift));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes + (p.csize_shift > 0 ? kPartBytes : 0);
    cfg.stream = a.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1u << p.csize_shift; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, prefill_tile_kernel<T>, p);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill_tile_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("prefill_tile_kernel launch");
}

}  // namespace

bool prefill_mma_supported(const PrefillArgs& a) {
    if (a.dtype != NVK_F16 && a.dtype != NVK_BF16) return false;
    if (a.head_dim != kHeadDim) return false;
    if (!aligned_to(a.q, 16) || !aligned_to(a.out, 16)) return false;
    if (a.block_tables) {
        if (a.block_size % kBN != 0) return false;
        if (!aligned_to(a.k_cache, 16) || !aligned_to(a.v_cache, 16)) return false;
    } else {
        if (!aligned_to(a.k, 16) || !aligned_to(a.v, 16)) return false;
    }
    return true;
}

int launch_prefill_mma(const PrefillArgs& a) {
    return a.dtype == NVK_BF16 ? launch_typed<__nv_bfloat16>(a) : launch_typed<__half>(a);
}

// Where few items leave most SMs of the persistent tcgen05 kernel idle, or are nearly empty, the smaller tiles above are quicker, although that does six
// times as much at once (us, 32 / 8 heads but where said, tcgen05 / these: 10 tokens 8.4 / 5.9, 77 9.5 / 7.4, 150 11.0 / 8.9, 8 on 256 12.0 / 8.3, 77 on
// 512 16.0 / 14.3, 4 x 8 to 20 on 1024, 4 / 1 heads, 21.5 / 11.2; but 300 tokens 12.7 / 13.7, 12 x 8 on 512 17.7 / 20.3, 11 x 67 to 256, 8 / 2 heads,
// 12.7 / 13.9).  The host does not know how the rows are shared out, and a block of 64 rows of a long prompt takes as long as the tcgen05 kernel for
// four times the heads and rows: one of 2000 tokens and 63 of 8 54 / 117, one of 2000 and 31 of 40 (4 / 1 heads) 30 / 55, one of 1500 and 15 of 5 (8 / 2)
// 24 / 40.  So the tiles have to win for equal lengths and must not lose more than 5 % for the most unequal ones: over 1800 steps of 1 to 64
// prompts, equal, spread and with one or two long ones, 0.81 of the tcgen05 kernel's time and 1.10 at most (by equal lengths alone 0.80 and 1.98).
bool prefill_takes_tiles(const PrefillArgs& a) {
    if ((a.num_heads / a.num_kv_heads) % 2 != 0 || !prefill_mma_supported(a)) return false;   // (odd groups: another tcgen05 kernel)
    const Alike equal = equal_lengths(a);
    const int csize_shift = best_cluster(a, equal);
    if (tile_time(a, &equal, 1, csize_shift) >= tcgen05_time(a, &equal, 1)) return false;
    Alike unequal[2];
    return !unequal_lengths(a, unequal) || tile_time(a, unequal, 2, csize_shift) <= 1.05 * tcgen05_time(a, unequal, 2);
}

// Error word of the waits above; cleared.
int prefill_tile_status(cudaStream_t stream, int* status) {
    int word = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(&word, g_prefill_error, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess && word != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbolAsync(g_prefill_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    }
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "prefill status: %s", cudaGetErrorString(e));
    *status = word;
    return NVK_OK;
}

}  // namespace nvk
