"""Python test/bench driver over the C ABI of ``libnvk.so`` (``include/nvk.h``).

The product is the shared library; this module only passes raw device pointers of torch tensors to it
(torch is plumbing: device memory and streams), through the small native binding ``nvk_torch.so``
(``bindings/nvk_torch.cpp``: argument checks and the call in one step); :func:`lib` gives the library
itself to ``ctypes`` users.  The function
names and argument order mirror the reference's operator API
(include/kernels/kvcache.h:7-12, include/kernels/attention.h:7-41,
include/kernels/split_qkv.h:22-33).  There is no fallback: if the CUDA library is missing or a
call fails, an exception is raised (``ValueError`` for invalid arguments, ``RuntimeError`` for
CUDA errors -- the reference throws std::invalid_argument / std::runtime_error).

The directory name contains a hyphen, so import it with :func:`load_package` from
``__graft_entry__`` (or ``importlib``) rather than with an ``import`` statement.
"""
from __future__ import annotations

import ctypes
import os

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "libnvk.so")
BINDING_PATH = os.path.join(HERE, "nvk_torch.so")

F16, BF16, F32, I32, I64, I8 = 0, 1, 2, 3, 4, 5
OK, ERR_INVALID_ARGUMENT, ERR_CUDA, ERR_UNSUPPORTED = 0, 1, 2, 3

EXPORTED_SYMBOLS = (
    "nvk_abi_version", "nvk_last_error", "nvk_store_kvcache", "nvk_fused_split_norm_rope_store",
    "nvk_decode_attention_workspace_bytes", "nvk_decode_attention_paged",
    "nvk_prefill_attention_varlen", "nvk_decode_attention_paged_static",
    "nvk_store_kvcache_int8", "nvk_decode_attention_paged_int8",
    "nvk_tp_allreduce_flag_bytes", "nvk_tp_allreduce_stage_bytes", "nvk_tp_allreduce_set_wait_limit_ms", "nvk_tp_allreduce",
    "nvk_tp_allreduce_status", "nvk_tp_allreduce_reset", "nvk_tp_allreduce_add_rmsnorm", "nvk_tp_allreduce_inprocess",
    "nvk_prefill_status", "nvk_decode_attention_static_scratch_bytes", "nvk_attention_mixed_step",
    "nvk_linear", "nvk_qkv_linear_norm_rope_store", "nvk_tp_row_linear_allreduce_add_rmsnorm",
    "nvk_tp_row_linear_allreduce_add_rmsnorm_inprocess", "nvk_gemm_status",
    "nvk_tp_allreduce_signal_bytes", "nvk_tp_allreduce_multimem", "nvk_tp_allreduce_add_rmsnorm_multimem",
    "nvk_store_kvcache_fp8", "nvk_decode_attention_paged_fp8",
)

_lib = None
_binding = None
launch_count = 0  # kernels launched through this module (claimed by the benchmark)


class NvkLibraryMissing(RuntimeError):
    pass


def lib() -> ctypes.CDLL:
    """Loads ``libnvk.so``; raises if it has not been built (no CPU or library fallback exists)."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise NvkLibraryMissing(
                f"{LIB_PATH} not found: build it with `python nano-vllm-cpp_b200/build.py` "
                "(or __graft_entry__.build()); there is no fallback path")
        L = ctypes.CDLL(LIB_PATH)
        L.nvk_last_error.restype = ctypes.c_char_p
        L.nvk_abi_version.restype = ctypes.c_int
        L.nvk_decode_attention_workspace_bytes.restype = ctypes.c_size_t
        L.nvk_decode_attention_workspace_bytes.argtypes = [
            ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int64, ctypes.c_int]
        L.nvk_decode_attention_static_scratch_bytes.restype = ctypes.c_size_t
        _lib = L
    return _lib


def _load_binding():
    """The native binding; raises if it has not been built."""
    global _binding
    import importlib.util
    import torch  # noqa: F401  (its libraries have to be in the process before the binding that links against them)
    lib()
    if not os.path.exists(BINDING_PATH):
        raise NvkLibraryMissing(f"{BINDING_PATH} not found: build it with `python nano-vllm-cpp_b200/build.py`")
    spec = importlib.util.spec_from_file_location("nvk_torch", BINDING_PATH)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    _binding = module
    return module


def _check(rc: int) -> None:
    if rc == OK:
        return
    msg = lib().nvk_last_error().decode()
    if rc in (ERR_INVALID_ARGUMENT, ERR_UNSUPPORTED):
        raise ValueError(msg)
    raise RuntimeError(msg)


def _dtype_code(t) -> int:
    import torch
    return {torch.float16: F16, torch.bfloat16: BF16, torch.float32: F32, torch.int32: I32,
            torch.int64: I64, torch.int8: I8}[t.dtype]


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def store_kvcache(key, value, k_cache, v_cache, slot_mapping) -> None:
    """``store_kvcache`` (include/kernels/kvcache.h:7-12): in-place scatter into the paged cache."""
    global launch_count
    launch_count += (_binding or _load_binding()).store_kvcache(key, value, k_cache, v_cache, slot_mapping)


def fused_split_norm_rope_store(qkv, positions, q_norm_weight, k_norm_weight, norm_eps, cos_sin_cache,
                                slot_mapping, k_cache, v_cache, num_q_heads, num_kv_heads, head_dim,
                                q_out) -> None:
    """``fused_split_norm_rope_store`` (include/kernels/split_qkv.h:22-33).  ``slot_mapping=None`` writes k / v of
    row r to row r of ``k_cache`` / ``v_cache`` (plain [rows, Hkv, D] tensors); both norm weights ``None`` skips the
    RMSNorm -- the two forms that serve the reference's unfused route (split_qkv, optional norm, rotary)."""
    global launch_count
    launch_count += (_binding or _load_binding()).fused_split_norm_rope_store(
        qkv, positions, q_norm_weight, k_norm_weight, norm_eps, cos_sin_cache, slot_mapping, k_cache, v_cache, num_q_heads,
        num_kv_heads, head_dim, q_out)


def decode_attention_workspace_bytes(batch, num_heads, num_kv_heads, head_dim, max_blocks, block_size) -> int:
    return int(lib().nvk_decode_attention_workspace_bytes(batch, num_heads, num_kv_heads, head_dim,
                                                          max_blocks, block_size))


def launch_decode_attention_paged(query, k_cache, v_cache, context_lens, block_tables, num_kv_heads,
                                  head_dim, block_size, scale, output, workspace=None) -> None:
    """``launch_decode_attention_paged`` (include/kernels/attention.h:31-41).

    ``workspace`` (a uint8 CUDA tensor of ``decode_attention_workspace_bytes`` bytes) plays the role
    of the allocator argument of ``flash_attn_decode_kvcache`` (include/kernels/flash_attn.h:39-50).
    """
    global launch_count
    launch_count += (_binding or _load_binding()).decode(
        query, k_cache, v_cache, context_lens, block_tables, num_kv_heads, head_dim, block_size, scale, output, workspace)


def launch_decode_attention_paged_static(query, k_cache, v_cache, context_lens, block_tables, num_kv_heads,
                                         head_dim, block_size, scale, output) -> None:
    """Decode attention for callers that may not allocate: split-K scratch comes from a 32 MiB array
    inside the library (``nvk_decode_attention_paged_static``).  Calls on one device must not overlap."""
    global launch_count
    launch_count += (_binding or _load_binding()).decode_static(
        query, k_cache, v_cache, context_lens, block_tables, num_kv_heads, head_dim, block_size, scale, output)


def store_kvcache_int8(key, value, k_cache, v_cache, k_scale, v_scale, slot_mapping) -> None:
    """``store_kvcache_int8`` (include/kernels/kvcache.h:14-24): quantising scatter into int8 caches + fp16 scales."""
    global launch_count
    launch_count += (_binding or _load_binding()).store_int8(key, value, k_cache, v_cache, k_scale, v_scale, slot_mapping)


def launch_decode_attention_paged_int8(query, k_cache, v_cache, k_scale, v_scale, context_lens, block_tables,
                                       num_kv_heads, head_dim, block_size, scale, output, workspace=None) -> None:
    """``launch_decode_attention_paged_int8`` (include/kernels/attention.h:43-56), with the optional split-K workspace
    of :func:`launch_decode_attention_paged`."""
    global launch_count
    launch_count += (_binding or _load_binding()).decode_int8(
        query, k_cache, v_cache, k_scale, v_scale, context_lens, block_tables, num_kv_heads, head_dim, block_size, scale,
        output, workspace)


def store_kvcache_fp8(key, value, k_cache, v_cache, k_scale, v_scale, slot_mapping) -> None:
    """Quantising scatter into e4m3 caches (uint8 or float8_e4m3fn tensors) + fp16 scales (``nvk_store_kvcache_fp8``)."""
    global launch_count
    launch_count += (_binding or _load_binding()).store_fp8(key, value, k_cache, v_cache, k_scale, v_scale, slot_mapping)


def launch_decode_attention_paged_fp8(query, k_cache, v_cache, k_scale, v_scale, context_lens, block_tables,
                                      num_kv_heads, head_dim, block_size, scale, output, workspace=None) -> None:
    """Paged decode attention over an e4m3 cache (``nvk_decode_attention_paged_fp8``)."""
    global launch_count
    launch_count += (_binding or _load_binding()).decode_fp8(
        query, k_cache, v_cache, k_scale, v_scale, context_lens, block_tables, num_kv_heads, head_dim, block_size, scale,
        output, workspace)


def _prefill(query, key, value, k_cache, v_cache, cu_q, cu_k, block_tables, num_kv_heads, head_dim,
             block_size, scale, output, max_seqlen_q=0) -> None:
    global launch_count
    launch_count += (_binding or _load_binding()).prefill(
        query, key, value, k_cache, v_cache, cu_q, cu_k, block_tables, num_kv_heads, head_dim, block_size, scale, output,
        max_seqlen_q)


def launch_prefill_attention_dense(query, cu_seqlens_q, key, value, cu_seqlens_k, num_kv_heads, head_dim,
                                   scale, output) -> None:
    """``launch_prefill_attention_dense`` (include/kernels/attention.h:7-16)."""
    _prefill(query, key, value, None, None, cu_seqlens_q, cu_seqlens_k, None, num_kv_heads, head_dim, 1,
             scale, output)


def launch_prefill_attention_paged(query, cu_seqlens_q, k_cache, v_cache, cu_seqlens_k, block_tables,
                                   num_kv_heads, head_dim, block_size, scale, output) -> None:
    """``launch_prefill_attention_paged`` (include/kernels/attention.h:18-29)."""
    if cu_seqlens_q is None or cu_seqlens_k is None:
        raise ValueError("paged prefill attention requires cu_seqlens_q and cu_seqlens_k")
    _prefill(query, None, None, k_cache, v_cache, cu_seqlens_q, cu_seqlens_k, block_tables, num_kv_heads,
             head_dim, block_size, scale, output)


def prefill_status() -> int:
    """Reads and clears the error word of the tensor-core prefill kernels on the current device (synchronises the
    current stream): 0 = every launch since the last call completed normally."""
    out = ctypes.c_int(0)
    _check(lib().nvk_prefill_status(_stream(), ctypes.byref(out)))
    return int(out.value)


def decode_attention_static_scratch_bytes() -> int:
    return int(lib().nvk_decode_attention_static_scratch_bytes())


def attention_mixed_step(p_query, cu_seqlens_q, p_key, p_value, cu_seqlens_k, p_block_tables, p_output, d_query, context_lens,
                         d_block_tables, d_output, k_cache, v_cache, num_kv_heads, head_dim, block_size, scale, workspace,
                         prefill_blocks=0) -> None:
    """One launch for a step with prefill rows and decode rows (``nvk_attention_mixed_step``).  Dense prefill keys:
    ``p_key`` / ``p_value`` given and ``p_block_tables`` None; paged: the other way round."""
    global launch_count
    launch_count += (_binding or _load_binding()).mixed_step(
        p_query, cu_seqlens_q, p_key, p_value, cu_seqlens_k, p_block_tables, p_output, d_query, context_lens, d_block_tables,
        d_output, k_cache, v_cache, num_kv_heads, head_dim, block_size, scale, workspace, prefill_blocks)


def linear(x, weight, out) -> None:
    """``out = x @ weight.T`` on this library's tcgen05 GEMM (``nvk_linear``); weight [out_features, in_features]."""
    global launch_count
    launch_count += (_binding or _load_binding()).linear(x, weight, out)


def qkv_linear_norm_rope_store(x, qkv_weight, positions, q_norm_weight, k_norm_weight, norm_eps, cos_sin_cache, slot_mapping,
                               k_cache, v_cache, num_q_heads, num_kv_heads, head_dim, q_out) -> None:
    """QKV projection + split + q / k RMSNorm + RoPE + cache store as one launch (``nvk_qkv_linear_norm_rope_store``)."""
    global launch_count
    launch_count += (_binding or _load_binding()).qkv_linear(
        x, qkv_weight, positions, q_norm_weight, k_norm_weight, norm_eps, cos_sin_cache, slot_mapping, k_cache, v_cache,
        num_q_heads, num_kv_heads, head_dim, q_out)


def gemm_status() -> int:
    """Reads and clears the error word of the GEMM kernels on the current device (synchronises the current stream)."""
    out = ctypes.c_int(0)
    _check(lib().nvk_gemm_status(_stream(), ctypes.byref(out)))
    return int(out.value)
