// Paged decode attention in fp32 arithmetic for the inputs the tensor-core kernels do not take: fp32 models (any group size,
// any block size) and 16-bit models with head_dim 64 or 256.
//
// Replaces the same reference kernel as decode_attn.cu (src/kernels/attention.cu:313-405).  The op reads each K / V row once
// and does 4 * G flops per element, so HBM bounds it; what has to be organised is enough bytes in flight from a batch of a
// few sequences:
//   * one thread-block cluster per (sequence, KV head, chunk of up to four query heads): cluster size 1, 2, 4 or 8, as large
//     as keeps the grid within two blocks per SM, so 8 sequences x 8 KV heads already occupy every SM;
//   * trips of 8 keys (D 128) are dealt round-robin to the cluster's warps; a key is spread over D / 16 lanes, 16 elements
//     each, so a warp reads whole 128-byte lines and a dot product needs log2(D / 16) shuffles for 32 / (D / 16) keys at
//     once; a warp's K and V loads of a trip (8 KiB in fp32) are all in flight together, and the rows of the next trip are
//     looked up in the block table under the current one;
//   * every lane group keeps its own running maximum and sum per query head; groups merge by shuffles, warps through shared
//     memory, blocks through distributed shared memory -- one launch, no workspace.
// Batch 8, 16 / 8 heads, fp32, context 64 .. 1024, store + decode: 2031 us a pass with one warp per (sequence, head) walking its
// keys in order, 15.7 us here (15.4 to 15.9 over boxes; 16.65 with branches around index and row loads and merges written out part by part), of which up to four trips of load, dot product, exponentials and sum follow one another in a warp.
#include "nvk_internal.cuh"

#include <cooperative_groups.h>

#include <cmath>

namespace nvk {
namespace {

namespace cg = cooperative_groups;

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kUnroll = 2;       // keys per lane group and trip
constexpr int kMaxCluster = 8;   // portable cluster size

struct SimtParams {
    const void* q; const void* k; const void* v; void* out;
    IndexArray context_lens, block_tables;
    int64_t max_blocks, cache_rows;
    int num_heads, num_kv_heads, group, chunks, block_size;
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

// K / V rows are read once; zeros, and no read, where there is no row (by a predicate: branches around the loads of each key doubled the loop's code).
__device__ __forceinline__ uint4 ld_stream16(const void* p, bool there) {
    uint4 v;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
        "@q ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}\n"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "r"(static_cast<int>(there)));
    return v;
}

// A float of this block's shared memory, as block `rank` of the cluster has it.
__device__ __forceinline__ float ld_block(const float* p, uint32_t rank) {
    float v;
    asm volatile(
        "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}\n"
        : "=f"(v) : "r"(smem_u32(p)), "r"(rank) : "memory");
    return v;
}

// HG: query heads of a chunk (rounded up to 1, 2 or 4; rows past the group are computed on zeros and not written).
template <typename T, int D, int HG>
__global__ void __launch_bounds__(kThreads, HG <= 2 ? 2 : 1) decode_simt_kernel(const SimtParams p) {
    constexpr int LANES = D / 16;                         // lanes per key
    constexpr int GROUPS = 32 / LANES;                    // keys a warp scores at once
    constexpr int VE = 16 / static_cast<int>(sizeof(T));  // elements per 16-byte vector
    constexpr int NV = 16 / VE;                           // vectors per lane and key
    constexpr int TRIP = GROUPS * kUnroll;
    __shared__ __align__(16) float s_q[HG][D];
    __shared__ float s_o[kWarps][HG][D];
    __shared__ float s_m[kWarps][HG], s_l[kWarps][HG];
    __shared__ float s_po[HG][D];                         // this block's merged partial result, read by the whole cluster
    __shared__ float s_pm[HG], s_pl[HG];
    pdl_wait_then_release();
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int sub = lane % LANES, grp = lane / LANES;
    const int64_t item = blockIdx.x / csize;
    const int chunk = static_cast<int>(item % p.chunks);
    const int kvh = static_cast<int>((item / p.chunks) % p.num_kv_heads);
    const int64_t b = item / (static_cast<int64_t>(p.chunks) * p.num_kv_heads);
    const int head0 = kvh * p.group + chunk * HG;
    const int heads = min(HG, p.group - chunk * HG);
    const int64_t cap = p.max_blocks * p.block_size;
    int64_t ctx = p.context_lens.load(b);
    if (ctx > cap) ctx = cap;
    if (ctx < 0) ctx = 0;

    for (int i = tid; i < HG * D; i += kThreads) {
        const int h = i / D, d = i % D;
        s_q[h][d] = h < heads ? ElemTraits<T>::to_float(static_cast<const T*>(p.q)[(b * p.num_heads + head0 + h) * D + d]) * p.scale : 0.0f;
    }
    __syncthreads();

    const int64_t row_elems = static_cast<int64_t>(p.num_kv_heads) * D;
    const T* kc = static_cast<const T*>(p.k) + static_cast<int64_t>(kvh) * D + sub * VE;
    const T* vc = static_cast<const T*>(p.v) + static_cast<int64_t>(kvh) * D + sub * VE;
    const IndexArray table = p.block_tables + b * p.max_blocks;
    float m[HG], l[HG], acc[HG][16];
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        m[h] = -INFINITY; l[h] = 0.0f;
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[h][e] = 0.0f;
    }

    // cache row of key k, -1 where the block id lies outside the cache (reads as zeros), -2 past the context
    auto row_of = [&](int64_t k) -> int64_t {
        if (k >= ctx) return -2;
        const int ki = static_cast<int>(k);
        const int blk = ki / p.block_size;
        const int64_t r = table.load(blk) * p.block_size + (ki - blk * p.block_size);
        return r >= 0 && r < p.cache_rows ? r : -1;
    };
    const int64_t step = static_cast<int64_t>(csize) * kWarps * TRIP;
    int64_t row[kUnroll];
    const int64_t first = (static_cast<int64_t>(rank) * kWarps + warp) * TRIP;
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) row[u] = row_of(first + u * GROUPS + grp);
    for (int64_t k0 = first; k0 < ctx; k0 += step) {
        uint4 kv[kUnroll][NV], vv[kUnroll][NV];
        bool live[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            live[u] = row[u] != -2;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                kv[u][i] = ld_stream16(kc + row[u] * row_elems + i * LANES * VE, row[u] >= 0);
                vv[u][i] = ld_stream16(vc + row[u] * row_elems + i * LANES * VE, row[u] >= 0);
            }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) row[u] = row_of(k0 + step + u * GROUPS + grp);
        float s[HG][kUnroll];
#pragma unroll
        for (int h = 0; h < HG; ++h) {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) s[h][u] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            float kf[kUnroll][VE];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) unpack<T>(kv[u][i], kf[u]);
#pragma unroll
            for (int h = 0; h < HG; ++h) {
#pragma unroll
                for (int e = 0; e < VE; e += 4) {
                    const float4 qf = *reinterpret_cast<const float4*>(&s_q[h][(i * LANES + sub) * VE + e]);
#pragma unroll
                    for (int u = 0; u < kUnroll; ++u)
                        s[h][u] = fmaf(qf.w, kf[u][e + 3], fmaf(qf.z, kf[u][e + 2], fmaf(qf.y, kf[u][e + 1], fmaf(qf.x, kf[u][e], s[h][u]))));
                }
            }
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int h = 0; h < HG; ++h) {
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) s[h][u] += __shfl_xor_sync(0xffffffffu, s[h][u], o);
            }
        }
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            float m_new = m[h];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) if (live[u]) m_new = fmaxf(m_new, s[h][u]);
            if (m_new > m[h]) {   // (same for all lanes of a group)
                const float corr = expf(m[h] - m_new);
                l[h] *= corr;
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[h][e] *= corr;
                m[h] = m_new;
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                s[h][u] = live[u] ? expf(s[h][u] - m[h]) : 0.0f;
                l[h] += s[h][u];
            }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                float vf[VE];
                unpack<T>(vv[u][i], vf);
#pragma unroll
                for (int h = 0; h < HG; ++h) {
#pragma unroll
                    for (int e = 0; e < VE; ++e) acc[h][i * VE + e] = fmaf(s[h][u], vf[e], acc[h][i * VE + e]);
                }
            }
        }
    }

    // lane groups -> warp
#pragma unroll
    for (int h = 0; h < HG; ++h) {
        float mx = m[h];
#pragma unroll
        for (int o = LANES; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float f = m[h] == -INFINITY ? 0.0f : expf(m[h] - mx);
        m[h] = mx;
        l[h] *= f;
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[h][e] *= f;
#pragma unroll
        for (int o = LANES; o < 32; o <<= 1) {
            l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[h][e] += __shfl_xor_sync(0xffffffffu, acc[h][e], o);
        }
        if (grp == 0) {
#pragma unroll
            for (int e = 0; e < 16; ++e) s_o[warp][h][((e / VE) * LANES + sub) * VE + e % VE] = acc[h][e];
            if (sub == 0) { s_m[warp][h] = m[h]; s_l[warp][h] = l[h]; }
        }
    }
    __syncthreads();
    // warps -> block
    for (int i = tid; i < HG * D; i += kThreads) {
        const int h = i / D, d = i % D;
        float mx = -INFINITY, lsum = 0.0f, o = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, s_m[w][h]);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float f = s_m[w][h] == -INFINITY ? 0.0f : expf(s_m[w][h] - mx);
            lsum += f * s_l[w][h];
            o += f * s_o[w][h][d];
        }
        s_po[h][d] = o;
        if (d == 0) { s_pm[h] = mx; s_pl[h] = lsum; }
    }
    // blocks -> result: every block of the cluster takes its share of the elements
    cluster.sync();
    T* out = static_cast<T*>(p.out) + (b * p.num_heads + head0) * D;
    for (int i = rank * kThreads + tid; i < heads * D; i += csize * kThreads) {
        const int h = i / D, d = i % D;
        float mx = -INFINITY, lsum = 0.0f, o = 0.0f;
#pragma unroll 1
        for (int r0 = 0; r0 < csize; r0 += 4) {   // (four blocks' loads under way at once)
            float pm[4], pl[4], po[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t from = static_cast<uint32_t>(min(r0 + u, csize - 1));
                pm[u] = ld_block(&s_pm[h], from);
                pl[u] = ld_block(&s_pl[h], from);
                po[u] = ld_block(&s_po[h][d], from);
                // (no weight of 0 takes out what a block that is not there would add: the last block's part, read in its place, may be infinite)
                if (r0 + u >= csize) { pm[u] = -INFINITY; pl[u] = po[u] = 0.0f; }
            }
            const float m_new = fmaxf(fmaxf(fmaxf(pm[0], pm[1]), fmaxf(pm[2], pm[3])), mx);
            const float f = mx == -INFINITY ? 0.0f : expf(mx - m_new);
            lsum *= f;
            o *= f;
            mx = m_new;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float w = pm[u] == -INFINITY ? 0.0f : expf(pm[u] - mx);
                lsum += w * pl[u];
                o += w * po[u];
            }
        }
        out[i] = ElemTraits<T>::from_float(lsum > 0.0f ? o / lsum : 0.0f);
    }
    cluster.sync();   // no block leaves while a peer still reads its shared memory
}

template <typename T, int D, int HG>
int launch_simt_typed(const SimtParams& p, int64_t batch, cudaStream_t stream) {
    const int64_t items = batch * p.num_kv_heads * p.chunks;
    // Two blocks per SM (one where four heads' accumulators leave no room for two): beyond that a larger cluster only adds
    // merges.
    const int64_t resident = static_cast<int64_t>(kSmCount) * (HG <= 2 ? 2 : 1);
    int csize = 1;
    while (csize < kMaxCluster && items * csize * 2 <= resident) csize *= 2;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(items * csize));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = csize; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_simt_kernel<T, D, HG>, p);
    if (e != cudaSuccess) return fail(NVK_ERR_CUDA, "decode_simt_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("decode_simt_kernel launch");
}

template <typename T, int D>
int launch_dim(SimtParams& p, int64_t batch, cudaStream_t stream) {
    const int hg = p.group >= 3 ? 4 : p.group;
    p.chunks = (p.group + hg - 1) / hg;
    switch (hg) {
        case 1: return launch_simt_typed<T, D, 1>(p, batch, stream);
        case 2: return launch_simt_typed<T, D, 2>(p, batch, stream);
        default: return launch_simt_typed<T, D, 4>(p, batch, stream);
    }
}

template <typename T>
int launch_typed(SimtParams& p, int head_dim, int64_t batch, cudaStream_t stream) {
    switch (head_dim) {
        case 64: return launch_dim<T, 64>(p, batch, stream);
        case 128: return launch_dim<T, 128>(p, batch, stream);
        default: return launch_dim<T, 256>(p, batch, stream);
    }
}

}  // namespace

bool decode_simt_supported(const DecodeArgs& a) {
    if (a.head_dim != 64 && a.head_dim != 128 && a.head_dim != 256) return false;
    if (!aligned_to(a.k_cache, 16) || !aligned_to(a.v_cache, 16)) return false;
    if (a.max_blocks * a.block_size >= (1LL << 31)) return false;
    return a.batch * a.num_heads * kMaxCluster < (1LL << 31);
}

int launch_decode_simt(const DecodeArgs& a) {
    SimtParams p{};
    p.q = a.q; p.k = a.k_cache; p.v = a.v_cache; p.out = a.out;
    p.context_lens = a.context_lens; p.block_tables = a.block_tables;
    p.max_blocks = a.max_blocks; p.cache_rows = a.num_cache_blocks * a.block_size;
    p.num_heads = a.num_heads; p.num_kv_heads = a.num_kv_heads; p.group = a.num_heads / a.num_kv_heads;
    p.block_size = a.block_size; p.scale = a.scale;
    switch (a.dtype) {
        case NVK_F32: return launch_typed<float>(p, a.head_dim, a.batch, a.stream);
        case NVK_F16: return launch_typed<__half>(p, a.head_dim, a.batch, a.stream);
        default: return launch_typed<__nv_bfloat16>(p, a.head_dim, a.batch, a.stream);
    }
}

}  // namespace nvk
