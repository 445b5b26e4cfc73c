// Which kernel a call takes, from the sizes that the host knows; no GPU.
#include "../../csrc/nvk_internal.cuh"
#include "check.h"

#include <vector>

using namespace nvk;

namespace {

// A causal prefill of prompts of these lengths; behind a prefix of `prefix` keys each with paged keys (tables of the longest's width).
PrefillArgs prefill(int heads, int kv_heads, const std::vector<int>& lens, bool paged, int prefix = 0, bool longest_known = false) {
    static char buffer[64] __attribute__((aligned(64)));
    PrefillArgs a{};
    a.q = a.k = a.v = a.k_cache = a.v_cache = a.out = buffer;
    a.cu_q = a.cu_k = IndexArray(buffer, 0);
    int longest = 0;
    for (int n : lens) {
        a.total_q += n;
        a.total_k += n + prefix;
        if (n > longest) longest = n;
    }
    a.num_seqs = static_cast<int64_t>(lens.size());
    a.num_heads = heads; a.num_kv_heads = kv_heads; a.head_dim = 128; a.block_size = 256; a.scale = 0.088f; a.dtype = NVK_BF16;
    a.max_seqlen_q = longest_known ? longest : 0;
    if (paged) {
        a.block_tables = IndexArray(buffer, 0);
        a.max_blocks = (longest + prefix + 255) / 256;
        a.num_cache_blocks = 4096;
    }
    return a;
}
std::vector<int> one_and(int longest, int others, int length) {
    std::vector<int> lens(1 + static_cast<size_t>(others), length);
    lens[0] = longest;
    return lens;
}

// Parts of `tokens` keys each of tables of `table` keys, the cache blocks of 256: what the workspace has to hold.
size_t parts(int64_t pairs, int64_t table, int64_t tokens, int group) {
    return static_cast<size_t>(pairs * (table / tokens) * group) * (128 * sizeof(float) + 2 * sizeof(float));
}
size_t workspace(int64_t batch, int kv_heads, int64_t table, int group) {
    return decode_mma_workspace_needed(batch, group * kv_heads, kv_heads, 128, table / 256, 256);
}

}  // namespace

// A long prompt among short ones belongs to the tcgen05 kernel (measured, us: tcgen05 / tiles of 64 rows), whether its length is given or not.
TEST_CASE(prefill_of_one_long_prompt_among_short_ones) {
    for (bool known : {false, true}) {
        CHECK(!prefill_takes_tiles(prefill(32, 8, one_and(2000, 63, 8), false, 0, known)));    // 54 / 117
        CHECK(!prefill_takes_tiles(prefill(4, 1, one_and(2000, 31, 40), false, 0, known)));    // 30 / 55
        CHECK(!prefill_takes_tiles(prefill(8, 2, one_and(1500, 15, 5), false, 0, known)));     // 24 / 40
        CHECK(!prefill_takes_tiles(prefill(8, 4, one_and(1000, 3, 40), false, 0, known)));     // 18 / 23
        CHECK(!prefill_takes_tiles(prefill(16, 8, one_and(600, 31, 8), true, 0, known)));      // 17 / 21
        CHECK(!prefill_takes_tiles(prefill(32, 8, one_and(400, 7, 4), false, 0, known)));      // 12 / 15
        CHECK(!prefill_takes_tiles(prefill(2, 1, one_and(1000, 8, 50), false, 0, known)));     // 18 / 22
    }
}

// Small steps stay with the tiles, one prompt or several that are alike.
TEST_CASE(prefill_of_small_steps) {
    CHECK(prefill_takes_tiles(prefill(32, 8, {10}, true)));              // 6.6 / 3.9
    CHECK(prefill_takes_tiles(prefill(32, 8, {77}, true, 512)));         // 13.8 / 12.1
    CHECK(prefill_takes_tiles(prefill(32, 8, {8}, true, 256)));          // 10.2 / 6.4
    CHECK(prefill_takes_tiles(prefill(4, 1, {670}, true)));              // 15.1 / 11.1
    CHECK(prefill_takes_tiles(prefill(4, 1, {8, 12, 16, 20}, true, 1024)));                     // 19.6 / 9.2
    CHECK(prefill_takes_tiles(prefill(16, 8, std::vector<int>(31, 8), true)));                  // 9.9 / 5.4
    CHECK(prefill_takes_tiles(prefill(32, 8, std::vector<int>(8, 50), false, 0, true)));
    CHECK(!prefill_takes_tiles(prefill(32, 8, {512, 1024, 2048}, true)));
}

// Lengths that do not go together, and the least there can be: the choice is some kernel, not a division by zero.
TEST_CASE(prefill_of_odd_sizes) {
    PrefillArgs a = prefill(8, 2, {1}, false);
    for (int64_t seqs : {1, 2, 3, 1000}) {
        for (int64_t rows : {1, 2, 3, 999, 1000, 1001}) {
            for (int longest : {0, 1, 2, 500, 100000}) {
                a.num_seqs = seqs; a.total_q = rows; a.max_seqlen_q = longest;
                for (int64_t keys : {int64_t{0}, int64_t{1}, rows, 10 * rows}) { a.total_k = keys; prefill_takes_tiles(a); }
            }
        }
    }
    a.cu_q = a.cu_k = IndexArray();
    a.num_seqs = 0; a.total_q = a.total_k = 1;
    CHECK(prefill_takes_tiles(a));
}

// One long context among short ones must not be read by one block or two while others have nothing to do (us for 16-bit caches, one context as long
// as the table and the others 1/32 of it: whole or in halves / in these chunks).
TEST_CASE(decode_contexts_are_cut_where_one_may_be_long) {
    CHECK(workspace(200, 1, 4096, 4) >= parts(200, 4096, 512, 4));      // 30.7 / 13.0
    CHECK(workspace(35, 8, 4096, 4) >= parts(280, 4096, 512, 4));       // 31.4 / 15.6
    CHECK(workspace(20, 8, 3072, 4) >= parts(160, 3072, 512, 4));       // 23.4 / 10.8
    CHECK(workspace(128, 1, 4096, 4) >= parts(128, 4096, 512, 4));      // 17.9 / 10.8
    CHECK(workspace(23, 8, 2048, 4) >= parts(184, 2048, 1024, 4));      // 16.4 / 13.1
    CHECK(workspace(140, 1, 8192, 4) >= parts(140, 8192, 1024, 4));     // 31.6 / 15.1
}

// A workspace sized for the most sequences and the widest table is enough for every call with fewer sequences and narrower tables, if there is any.
TEST_CASE(decode_workspace_of_the_largest_call_is_enough_for_smaller_ones) {
    constexpr size_t kStatic = 32u << 20;
    for (int kv_heads : {1, 3, 8}) {
        for (int group : {1, 4, 8}) {
            for (int block_size : {16, 48, 256}) {
                std::vector<size_t> widest(static_cast<size_t>(900 / kv_heads) + 1, 0);   // the largest need of so many sequences in narrower tables
                for (int64_t tokens : {256, 512, 768, 1000, 1024, 1280, 1536, 2048, 2304, 3072, 4096, 5000, 6144, 8192, 10240, 16384, 30720, 32768, 40960}) {
                    const int64_t blocks = tokens / block_size;
                    size_t least = 0;                                                     // and of fewer sequences
                    int wrong = 0;
                    for (size_t batch = 1; batch < widest.size(); ++batch) {
                        const size_t need = decode_mma_workspace_needed(static_cast<int64_t>(batch), kv_heads * group, kv_heads, 128, blocks, block_size);
                        const size_t given = nvk_decode_attention_workspace_bytes(static_cast<int64_t>(batch), kv_heads * group, kv_heads, 128, blocks, block_size);
                        if (need > widest[batch]) widest[batch] = need;
                        if (widest[batch] > least) least = widest[batch];
                        if (given < need) ++wrong;
                        if (given > 0 && given < least && !(need <= kStatic && least > kStatic)) ++wrong;
                        if (need <= kStatic && given > kStatic) ++wrong;                  // what fits the static array still does
                    }
                    CHECK(wrong == 0);
                }
            }
        }
    }
}

int main() { return check::run_all(); }
