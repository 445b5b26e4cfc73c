// Paged decode attention in fp32 arithmetic for the inputs the tensor-core kernels do not take: fp32 models (any group size,
// any block size) and 16-bit models with head_dim 64 or 256.
//
// Replaces the same reference kernel as decode_attn.cu (src/kernels/attention.cu:313-405).  The op reads each K / V row once
// and does 4 * G flops per element, so HBM bounds it; what has to be organised is enough bytes in flight from a batch of a
// few sequences, and little before the first and after the last of them:
//   * one thread-block cluster per (sequence, KV head, chunk of up to four query heads), blocks of four or eight warps, sixteen (twelve, eight) warps to an
//     SM: cluster size 1, 2, 4 or 8, so 8 sequences x 8 KV heads already occupy every SM;
//   * steps of 32 / (D / 16) keys (4 at D 128) are dealt round-robin to the cluster's warps; a key is spread over D / 16 lanes, 16 elements
//     each, so a warp reads whole 128-byte lines and a dot product needs log2(D / 16) shuffles.  K and V come through a ring in shared
//     memory by cp.async, 12 KiB a warp: a lane copies what it will read itself, so a step waits for nothing but its own copies;
//   * every lane group keeps its own running maximum and sum per query head; the groups of a block come together through shared
//     memory, their sum is pushed to the block of the cluster that finishes those elements, and after one cluster barrier everything is
//     local -- one launch, no workspace.  The merges run once, and code that runs once is as slow as it is long: with every part unrolled
//     they took 3 us of a block's 8, now 1.6.
// Batch 8, 16 / 8 heads, fp32, context 64 .. 1024, store + decode: 2031 us a pass with one warp per (sequence, head) walking its
// keys in order, 15.2 us with rows in registers (trips of 8 keys in a warp that never overlapped, up to 7.7 us of them, and 3.3 us of merges
// by shuffles and by fetching peers' parts), 12.4 us here; 1 sequence of 100 keys 8.1 -> 4.7, 7 of 64 to 200 (8 / 4 heads) 10.0 -> 6.0, 8 of 4000 to 4096
// (32 / 8 heads) 71.5 -> 64.  Sequences in order of falling context so that long and short blocks share an SM: 13.3 -> 13.7 in an earlier form.
#include "nvk_internal.cuh"

#include <atomic>
#include <cmath>

namespace nvk {
namespace {

constexpr int kMaxCluster = 8;   // portable cluster size

struct SimtParams {
    const void* q; const void* k; const void* v; void* out;
    IndexArray context_lens, block_tables;
    int64_t max_blocks, num_cache_blocks;
    int batch, num_heads, num_kv_heads, group, chunks, block_size, csize_shift;
    FastDiv by_block, by_chunks, by_kv_heads;
    float scale;
};

template <typename T> __device__ __forceinline__ void unpack(const uint4& w, float* f);
template <> __device__ __forceinline__ void unpack<float>(const uint4& w, float* f) {
    f[0] = __uint_as_float(w.x); f[1] = __uint_as_float(w.y); f[2] = __uint_as_float(w.z); f[3] = __uint_as_float(w.w);
}
template <> __device__ __forceinline__ void unpack<__nv_bfloat16>(const uint4& w, float* f) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(u[i] << 16); f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
template <> __device__ __forceinline__ void unpack<__half>(const uint4& w, float* f) {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
        f[2 * i] = p.x; f[2 * i + 1] = p.y;
    }
}

__device__ __forceinline__ uint4 lds16(uint32_t addr) {   // (volatile: stays on its side of the copies that refill the place)
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// HG: query heads of a chunk (rounded up to 1, 2 or 4; rows past the group are computed on zeros and not written).
// W: warps of a block; 4, of which four (HG 4: three) fit on an SM, or 8, of which two (one) do.
template <int HG, int W> constexpr int kBlocksPerSm = W == 4 ? (HG <= 2 ? 4 : 3) : HG <= 2 ? 2 : 1;
template <int HG, int W> constexpr int kWarpRing = W == 8 && HG == 4 ? 24 * 1024 : 12 * 1024;
template <typename T, int D, int HG, int W>
__global__ void __launch_bounds__(W * 32, kBlocksPerSm<HG, W>) decode_simt_kernel(const __grid_constant__ SimtParams p) {
    constexpr int kWarps = W, kThreads = W * 32, RING = kWarpRing<HG, W>;
    // Steps in one trip of the loop: a step is a serial chain (dot product, shuffles, exponential, sum), which two warps per scheduler do not hide.
    constexpr int U = W == 8 && HG == 4 ? 2 : 1;
    constexpr int LANES = D / 16;                         // lanes per key
    constexpr int GROUPS = 32 / LANES;                    // keys of a step
    constexpr int VE = 16 / static_cast<int>(sizeof(T));  // elements per 16-byte vector
    constexpr int NV = 16 / VE;                           // vectors per lane and key
    constexpr int STAGE = 2 * NV * 512;                   // K and V of a step: NV x 16 bytes of each per lane
    constexpr int STAGES = RING / STAGE;
    constexpr int QUADS = HG * D / 4;                     // of the result
    constexpr int TPQ = kThreads / QUADS < 1 ? 1 : kThreads / QUADS < kWarps ? kThreads / QUADS : kWarps;   // threads of a quad in a block's merge
    static_assert(GROUPS * HG * D * 4 <= RING, "a warp's parts take its ring's place");
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) float s_q[HG * D];
    __shared__ float2 s_part[HG][kWarps];                 // (maximum, sum) of every warp
    __shared__ float4 s_o[QUADS];                         // [block of the cluster][quad that this block finishes]
    __shared__ float2 s_ml[kMaxCluster][HG];
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");   // (waited for before the first remote store: every block has started)
    pdl_wait_then_release();
    const int csize = 1 << p.csize_shift, rank = static_cast<int>(blockIdx.x) & (csize - 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sub = lane % LANES, grp = lane / LANES;
    const uint32_t item = blockIdx.x >> p.csize_shift;
    const uint32_t pair = p.by_chunks.div(item);
    const int chunk = static_cast<int>(item - pair * p.chunks);
    const int b = static_cast<int>(p.by_kv_heads.div(pair));
    const int kvh = static_cast<int>(pair) - b * p.num_kv_heads;
    const int64_t cap = p.max_blocks * p.block_size;
    auto clamped = [&](IndexArray::Raw raw) {
        const int64_t n = p.context_lens.value(raw);
        return static_cast<int>(n < 0 ? 0 : n < cap ? n : cap);
    };
    const int head0 = kvh * p.group + chunk * HG, heads = min(HG, p.group - chunk * HG);
    const IndexArray table = p.block_tables + b * p.max_blocks;
    const IndexArray::Raw raw_ctx = p.context_lens.raw(b);
    IndexArray::Raw raw_ids = table.raw(lane, lane < p.max_blocks);
    float q_in[(HG * D + kThreads - 1) / kThreads];
#pragma unroll
    for (int i = 0; i < (HG * D + kThreads - 1) / kThreads; ++i) {
        const int at = i * kThreads + tid;
        q_in[i] = at < heads * D ? ElemTraits<T>::to_float(static_cast<const T*>(p.q)[(static_cast<int64_t>(b) * p.num_heads + head0) * D + at]) * p.scale : 0.0f;
    }
    const int ctx = clamped(raw_ctx);

    // The copying end: this warp's next step begins at key `tok`.  Lane i holds the cache block of table entry id_base + i (-1: outside the cache, reads
    // as zeros).
    const uint32_t ring = smem_u32(smem) + warp * RING + lane * 16;
    const size_t row_bytes = static_cast<size_t>(p.num_kv_heads) * D * sizeof(T);
    const size_t lane_at = (static_cast<size_t>(kvh) * D + sub * VE) * sizeof(T);
    const int first = (rank * kWarps + warp) * GROUPS, stride = kWarps * GROUPS << p.csize_shift;
    int tok = first, id_base = 0, ids;
    auto take_ids = [&](IndexArray::Raw raw) {
        const int64_t id = table.value(raw);
        ids = id >= 0 && id < p.num_cache_blocks ? static_cast<int>(id) : -1;
    };
    take_ids(raw_ids);
    uint32_t fill = ring;
    auto issue = [&]() {
        if (tok < ctx) {
            const int key = min(tok + grp, ctx - 1), blk = static_cast<int>(p.by_block.div(key));
            if (static_cast<int>(p.by_block.div(min(tok + GROUPS - 1, ctx - 1))) - id_base >= 32) {   // (warp-uniform; a step's keys lie in fewer blocks)
                id_base = static_cast<int>(p.by_block.div(tok));
                take_ids(table.raw(id_base + lane, id_base + lane < p.max_blocks));
            }
            const int id = __shfl_sync(0xffffffffu, ids, blk - id_base);
            const bool there = id >= 0 && tok + grp < ctx;
            const size_t at = there ? (static_cast<size_t>(id) * p.block_size + (key - blk * p.block_size)) * row_bytes + lane_at : 0;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                cp_async16(fill + i * 512, static_cast<const char*>(p.k) + at + i * LANES * 16, there ? 16 : 0);
                cp_async16(fill + (NV + i) * 512, static_cast<const char*>(p.v) + at + i * LANES * 16, there ? 16 : 0);
            }
            fill = fill == ring + (STAGES - 1) * STAGE ? ring : fill + STAGE;
            tok += stride;
        }
        cp_async_commit();
    };
#pragma unroll 1   // (code that runs once is as slow as it is long)
    for (int s = 0; s < STAGES - U; ++s) issue();
#pragma unroll
    for (int i = 0; i < (HG * D + kThreads - 1) / kThreads; ++i)
        if (i * kThreads + tid < HG * D) s_q[i * kThreads + tid] = q_in[i];
    __syncthreads();
    constexpr bool kQInRegs = HG <= 2;
    float qr[kQInRegs ? HG : 1][16];
    if (kQInRegs) {
#pragma unroll
        for (int h = 0; h < HG; ++h) {
#pragma unroll
            for (int e = 0; e < 16; ++e) qr[h][e] = s_q[h * D + ((e / VE) * LANES + sub) * VE + e % VE];
        }
    }

    float m[HG], l[HG], acc[HG][16];
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        m[h] = -INFINITY; l[h] = 0.0f;
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[h][e] = 0.0f;
    }
    uint32_t use = ring;
    auto next = [&](uint32_t at) { return at == ring + (STAGES - 1) * STAGE ? ring : at + STAGE; };
#pragma unroll 1
    for (int k0 = first; k0 < ctx; k0 += U * stride) {
#pragma unroll
        for (int u = 0; u < U; ++u) issue();
        cp_async_wait<STAGES - U>();
        float sc[U][HG], fv[16];                 // scores, then weights; V (the first step's on its way under the exponentials)
        bool live[U];
        uint32_t at = use;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float f[16];
            live[u] = k0 + u * stride + grp < ctx;
#pragma unroll
            for (int i = 0; i < NV; ++i) unpack<T>(lds16(at + i * 512), f + i * VE);
#pragma unroll
            for (int h = 0; h < HG; ++h) {
                float s[4];
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    float4 qf;
                    if (kQInRegs) qf = make_float4(qr[h][e], qr[h][e + 1], qr[h][e + 2], qr[h][e + 3]);
                    else qf = *reinterpret_cast<const float4*>(&s_q[h * D + ((e / VE) * LANES + sub) * VE + e % VE]);
                    s[0] = e == 0 ? qf.x * f[e] : fmaf(qf.x, f[e], s[0]);
                    s[1] = e == 0 ? qf.y * f[e + 1] : fmaf(qf.y, f[e + 1], s[1]);
                    s[2] = e == 0 ? qf.z * f[e + 2] : fmaf(qf.z, f[e + 2], s[2]);
                    s[3] = e == 0 ? qf.w * f[e + 3] : fmaf(qf.w, f[e + 3], s[3]);
                }
                sc[u][h] = (s[0] + s[1]) + (s[2] + s[3]);
            }
            at = next(at);
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int h = 0; h < HG; ++h) sc[u][h] += __shfl_xor_sync(0xffffffffu, sc[u][h], o);
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) unpack<T>(lds16(use + (NV + i) * 512), fv + i * VE);
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            float top = m[h];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (live[u] && sc[u][h] > top) top = sc[u][h];
            if (top > m[h]) {   // (same for all lanes of a group)
                const float corr = expf(m[h] - top);
                l[h] *= corr;
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[h][e] *= corr;
                m[h] = top;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                sc[u][h] = !live[u] || sc[u][h] == -INFINITY ? 0.0f : expf(sc[u][h] - m[h]);
                l[h] += sc[u][h];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (u == 0 || k0 + u * stride < ctx) {   // (what was not copied for there is not read: nothing times a weight of 0 but what is finite)
                if (u > 0) {
#pragma unroll
                    for (int i = 0; i < NV; ++i) unpack<T>(lds16(use + (NV + i) * 512), fv + i * VE);
                }
#pragma unroll
                for (int h = 0; h < HG; ++h) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[h][e] = fmaf(sc[u][h], fv[e], acc[h][e]);
                }
            }
            use = next(use);
        }
    }

    // lane groups -> block: under the warp's maximum every group leaves its part over its warp's ring, TPQ threads add up a quad of the result
    cp_async_wait<0>();
    __syncwarp();
    float* part = reinterpret_cast<float*>(smem + warp * RING) + grp * HG * D;
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        float mx = m[h];
#pragma unroll
        for (int o = LANES; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float f = m[h] == -INFINITY ? 0.0f : expf(m[h] - mx);
        float sum = l[h] * f;
#pragma unroll
        for (int o = LANES; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(part + h * D + ((e / VE) * LANES + sub) * VE + e % VE) =
                make_float4(acc[h][e] * f, acc[h][e + 1] * f, acc[h][e + 2] * f, acc[h][e + 3] * f);
        if (lane == 0) s_part[h][warp] = make_float2(mx, sum);
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    const int quads = QUADS >> p.csize_shift;             // that a block finishes
    const int split = lane / (32 / TPQ);
#pragma unroll 1
    for (int e = warp * (32 / TPQ) + lane % (32 / TPQ); e < QUADS; e += kThreads / TPQ) {   // (whole warps)
        const int h = e / (D / 4);
        float mx = s_part[h][0].x, sum = 0.0f;
#pragma unroll
        for (int w = 1; w < kWarps; ++w) mx = fmaxf(mx, s_part[h][w].x);
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kWarps / TPQ; ++i) {
            const int w = i * TPQ + split;
            const float2 ml = s_part[h][w];
            const float f = ml.x == -INFINITY ? 0.0f : expf(ml.x - mx);
            const float4* from = reinterpret_cast<const float4*>(smem + w * RING) + e;
            float4 v = from[0];
#pragma unroll
            for (int g = 1; g < GROUPS; ++g) {
                const float4 u = from[g * QUADS];
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
            t.x = fmaf(f, v.x, t.x); t.y = fmaf(f, v.y, t.y); t.z = fmaf(f, v.z, t.z); t.w = fmaf(f, v.w, t.w);
            sum = fmaf(f, ml.y, sum);
        }
#pragma unroll
        for (int o = 32 / TPQ; o < 32; o <<= 1) {
            t.x += __shfl_xor_sync(0xffffffffu, t.x, o); t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
            t.z += __shfl_xor_sync(0xffffffffu, t.z, o); t.w += __shfl_xor_sync(0xffffffffu, t.w, o);
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        const int to = e / quads, at = e - to * quads;
        if (split == 0) {
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};\n"
                         ::"r"(in_block(smem_u32(s_o + rank * quads + at), to)), "f"(t.x), "f"(t.y), "f"(t.z), "f"(t.w) : "memory");
            if (at == 0 || e == h * (D / 4))   // (a block may finish quads of several heads, a head may be finished by several blocks)
                asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(in_block(smem_u32(&s_ml[rank][h]), to)), "f"(mx), "f"(sum) : "memory");
        }
    }
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
    // blocks -> result
    T* out = static_cast<T*>(p.out) + (static_cast<int64_t>(b) * p.num_heads + head0) * D;
#pragma unroll 1
    for (int i = tid; i < quads; i += kThreads) {
        const int e = rank * quads + i, h = e / (D / 4);
        if (h >= heads) break;
        float mx = -INFINITY, sum = 0.0f;
#pragma unroll 4
        for (int r = 0; r < csize; ++r) mx = fmaxf(mx, s_ml[r][h].x);
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int r = 0; r < csize; ++r) {
            const float2 ml = s_ml[r][h];
            const float4 v = s_o[r * quads + i];
            const float f = ml.x == -INFINITY ? 0.0f : expf(ml.x - mx);
            t.x = fmaf(f, v.x, t.x); t.y = fmaf(f, v.y, t.y); t.z = fmaf(f, v.z, t.z); t.w = fmaf(f, v.w, t.w);
            sum = fmaf(f, ml.y, sum);
        }
        const bool any = sum > 0.0f;
        out[4 * e] = ElemTraits<T>::from_float(any ? t.x / sum : 0.0f);
        out[4 * e + 1] = ElemTraits<T>::from_float(any ? t.y / sum : 0.0f);
        out[4 * e + 2] = ElemTraits<T>::from_float(any ? t.z / sum : 0.0f);
        out[4 * e + 3] = ElemTraits<T>::from_float(any ? t.w / sum : 0.0f);
    }
}

template <typename T, int D, int HG, int W>
int launch_simt_blocks(SimtParams& p, int64_t blocks, cudaStream_t stream) {
    constexpr int kSmemBytes = W * kWarpRing<HG, W>;
    auto* kernel = decode_simt_kernel<T, D, HG, W>;
    static std::atomic<bool> attr_done[64] = {};   // per device; the attribute call is idempotent
    int device = 0;
    cudaGetDevice(&device);
    if (device >= 0 && device < 64 && !attr_done[device]) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode_simt_kernel: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        attr_done[device] = true;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks));
    cfg.blockDim = dim3(W * 32);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1u << p.csize_shift; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode_simt_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("decode_simt_kernel launch");
}

// log2 of the cluster size and warps of a block, for so many items and keys of a table row.  Blocks of four warps: as large a cluster as keeps all blocks
// resident; beyond that a larger one only adds merges.  Blocks of eight where that gives an item more warps (with four heads, whose trips then take two steps: as
// many), because one long context is what a step waits for: with few items, and with so many that each gets one block.  us a call, four / eight warps,
// fp32, head_dim 128, contexts of 2600 keys: 1 sequence of 8 / 1 heads 19.8 / 13.9; 4 of 16 / 8, of which one is that long and the others have 80, 13.3 / 11.8; 8 of 32 / 8, from 130
// keys on, 41.2 / 36.4; 48 of 16 / 8, one long, 73.2 / 45.2, from 130 on 101 / 88, all 165 / 160; 120 of 8 / 1, one long, 124 / 76, all 182 / 140; but 200 of 8 / 1,
// all, 185 / 210 (one long 125 / 70), 24 of 16 / 8 from 130 on 53.8 / 56.7, and 300 of 300 keys, 16 / 8 heads of 64, 67 / 77.  (With blocks of four warps alone 120 sequences of 8 / 1
// heads of 256, 16-bit, one of 2600 keys, took 279 us; in an earlier form of eight warps with rows in registers 151, now 148.)
struct Shape { int csize_shift, warps; };
Shape choose_shape(int64_t items, int64_t tokens, int head_dim, int elem_bytes, int heads) {
    const int64_t resident = static_cast<int64_t>(kSmCount) * (heads <= 2 ? 4 : 3);
    const bool slow = heads == 4 && head_dim == 256 && elem_bytes == 2;   // the longest steps for their bytes
    int four = 0;
    while ((1 << four) < kMaxCluster && (items << (four + 1)) <= resident) ++four;
    if (four == 0) {
        if (tokens <= 512) return {0, items <= (heads <= 2 || head_dim == 256 ? 3 : 2) * kSmCount ? 8 : 4};
        return {0, heads <= 2 || head_dim == 256 || items <= 8 * kSmCount ? 8 : 4};
    }
    if (tokens <= 512 && head_dim < 256) return {four, 4};
    if (heads <= 2) return items <= 33 ? Shape{3, 8} : Shape{four, 4};
    // Eight warps, one block to an SM.  A cluster has to fit into one GPC: 15 of eight blocks, 33 of four, 74 of two are resident at once; three of eight blocks more
    // are quicker than smaller ones where a single context is long.
    if (items <= 15 || (items <= 18 && tokens > 2048 && head_dim > 64)) return {3, 8};
    if (items > 18 && items <= 33) return {2, 8};
    if (items > 55 && items <= 74) return {1, 8};
    if (items > 111 && (items <= kSmCount || slow)) return {0, 8};
    return {four, 4};
}
template <typename T, int D, int HG>
int launch_simt_typed(SimtParams& p, cudaStream_t stream) {
    const int64_t items = static_cast<int64_t>(p.batch) * p.num_kv_heads * p.chunks;
    const Shape shape = choose_shape(items, p.max_blocks * p.block_size, D, sizeof(T), HG);
    p.csize_shift = shape.csize_shift;
    const int64_t blocks = items << p.csize_shift;
    p.by_block = FastDiv(static_cast<uint32_t>(p.block_size));
    p.by_chunks = FastDiv(static_cast<uint32_t>(p.chunks));
    p.by_kv_heads = FastDiv(static_cast<uint32_t>(p.num_kv_heads));
    return shape.warps == 8 ? launch_simt_blocks<T, D, HG, 8>(p, blocks, stream) : launch_simt_blocks<T, D, HG, 4>(p, blocks, stream);
}

template <typename T, int D>
int launch_dim(SimtParams& p, cudaStream_t stream) {
    const int hg = p.group >= 3 ? 4 : p.group;
    p.chunks = (p.group + hg - 1) / hg;
    switch (hg) {
        case 1: return launch_simt_typed<T, D, 1>(p, stream);
        case 2: return launch_simt_typed<T, D, 2>(p, stream);
        default: return launch_simt_typed<T, D, 4>(p, stream);
    }
}

template <typename T>
int launch_typed(SimtParams& p, int head_dim, cudaStream_t stream) {
    switch (head_dim) {
        case 64: return launch_dim<T, 64>(p, stream);
        case 128: return launch_dim<T, 128>(p, stream);
        default: return launch_dim<T, 256>(p, stream);
    }
}

}  // namespace

bool decode_simt_supported(const DecodeArgs& a) {
    if (a.head_dim != 64 && a.head_dim != 128 && a.head_dim != 256) return false;
    if (!aligned_to(a.k_cache, 16) || !aligned_to(a.v_cache, 16)) return false;
    if (a.max_blocks * a.block_size >= (1LL << 31) - 4096 || a.num_cache_blocks >= (1LL << 31)) return false;
    return a.batch * a.num_heads * kMaxCluster < (1LL << 31);
}

int launch_decode_simt(const DecodeArgs& a) {
    SimtParams p{};
    p.q = a.q; p.k = a.k_cache; p.v = a.v_cache; p.out = a.out;
    p.context_lens = a.context_lens; p.block_tables = a.block_tables;
    p.max_blocks = a.max_blocks; p.num_cache_blocks = a.num_cache_blocks;
    p.batch = static_cast<int>(a.batch); p.num_heads = a.num_heads; p.num_kv_heads = a.num_kv_heads; p.group = a.num_heads / a.num_kv_heads;
    p.block_size = a.block_size; p.scale = a.scale;
    switch (a.dtype) {
        case NVK_F32: return launch_typed<float>(p, a.head_dim, a.stream);
        case NVK_F16: return launch_typed<__half>(p, a.head_dim, a.stream);
        default: return launch_typed<__nv_bfloat16>(p, a.head_dim, a.stream);
    }
}

}  // namespace nvk
