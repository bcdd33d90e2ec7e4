"""ctypes binding of libkvm_b200.so (declarations mirror include/kvm_b200.h).

The library is the only compute path of this package: importing this module without the built
library raises, there is no fallback.
"""

from __future__ import annotations

import ctypes as C
import os

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libkvm_b200.so")

KVM_OK = 0
PREFILL_CHAIN, PREFILL_ATTENTION, PREFILL_LEGACY_ATTENTION, PREFILL_LEGACY_CHAIN = 1, 2, 4, 8
PREFILL_TEST_WITHHOLD_ARRIVAL = 16
PREFILL_KEYS_PREPARED = 32
ERROR_NAMES = {1: "bad argument", 2: "capacity", 3: "device timeout", 4: "CUDA error", 5: "unsupported"}


class KvmLayer(C.Structure):
    _fields_ = [
        ("n_q_heads", C.c_int32), ("n_kv_heads", C.c_int32), ("head_dim", C.c_int32),
        ("chunk_len", C.c_int32), ("n_bswa_chunks", C.c_int32), ("rope_dim", C.c_int32),
        ("sink_len", C.c_int32), ("gate_keys", C.c_int32), ("gate_values", C.c_int32),
        ("gate_appends", C.c_int32), ("gate_initial", C.c_int32), ("ln_eps", C.c_float),
        ("ln_weight_dev", C.c_void_p), ("ln_bias_dev", C.c_void_p),
        ("front_temp_dev", C.c_void_p), ("state_temp_dev", C.c_void_p),
    ]


class KvmTensor4(C.Structure):
    _fields_ = [("ptr", C.c_void_p), ("stride_b", C.c_int64), ("stride_h", C.c_int64), ("stride_t", C.c_int64)]


class KvmMemory(C.Structure):
    _fields_ = [("k_sum", C.c_void_p), ("v_sum", C.c_void_p), ("vlen", C.c_void_p),
                ("k_attn", C.c_void_p), ("v_attn", C.c_void_p), ("capacity", C.c_int32)]


class KvmUpdatePlan(C.Structure):
    _fields_ = [("state_before", C.c_int32), ("n_append", C.c_int32), ("version_row", C.c_int32),
                ("reserved", C.c_int32)]


class KvmPrefillLayout(C.Structure):
    _fields_ = [("status_offset", C.c_size_t), ("pool_k_offset", C.c_size_t), ("pool_v_offset", C.c_size_t),
                ("version_table_offset", C.c_size_t), ("prepared_keys_offset", C.c_size_t),
                ("gated_keys_offset", C.c_size_t), ("pool_rows", C.c_int64), ("total_bytes", C.c_size_t)]


class KvmPrologue(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("q_lin", "k_lin", "v_lin", "gate_lin", "shift_q", "shift_k", "shift_v",
                                          "prev_q", "prev_k", "prev_v", "ln_q_w", "ln_q_b", "ln_k_w", "ln_k_b")] + [
        ("ln_qk_eps", C.c_float), ("cos", C.c_void_p), ("sin", C.c_void_p), ("rope_stride_b", C.c_int64)]


class KvmPrologueExt(C.Structure):
    _anonymous_ = ("base",)
    _fields_ = [
        ("base", KvmPrologue),
        ("q_stride_t", C.c_int64), ("k_stride_t", C.c_int64), ("v_stride_t", C.c_int64), ("gate_stride_t", C.c_int64),
        ("prev_q_stride_b", C.c_int64), ("prev_k_stride_b", C.c_int64), ("prev_v_stride_b", C.c_int64),
        ("v_first", C.c_void_p), ("v_gate", C.c_void_p), ("v_gate0", C.c_void_p), ("v_last", C.c_void_p), ("ln_bf16", C.c_int32)]


class KvmDecodeCache(C.Structure):
    _fields_ = [("memory", KvmMemory), ("ring_k", C.c_void_p), ("ring_v", C.c_void_p),
                ("ring_gate", C.c_void_p), ("total_len", C.c_void_p), ("state_len", C.c_void_p)]


class KvmDecodeCall(C.Structure):
    _fields_ = [("layer", C.c_void_p), ("batch", C.c_int32), ("cache", KvmDecodeCache),
                ("q", KvmTensor4), ("k", KvmTensor4), ("v", KvmTensor4), ("gate", KvmTensor4),
                ("n_append_dev", C.c_void_p), ("n_append_host", C.c_void_p),
                ("total_len_host", C.c_void_p), ("state_len_host", C.c_void_p), ("any_update", C.c_int32), ("max_rows", C.c_int32),
                ("out", C.c_void_p), ("route_dev", C.c_void_p), ("workspace", C.c_void_p), ("workspace_bytes", C.c_size_t)]


class KvmTokenCall(C.Structure):
    _fields_ = [("decode", KvmDecodeCall), ("prologue", KvmPrologueExt), ("x", C.c_void_p), ("x_stride", C.c_int64), ("hidden", C.c_int32),
                ("n_weights", C.c_int32), ("weights", C.c_void_p * 5), ("weight_rows", C.c_int32 * 5), ("gated", C.c_int32),
                ("out_features", C.c_int32), ("v_gate2", C.c_void_p), ("c_proj", C.c_void_p), ("lin", C.c_void_p),
                ("lin_stride", C.c_int64), ("scratch", C.c_void_p), ("scratch_bytes", C.c_size_t), ("y", C.c_void_p)]


class KvmPromptCall(C.Structure):
    _fields_ = [("layer", C.c_void_p), ("batch", C.c_int32), ("n_updates", C.c_int32), ("seq_len", C.c_int64),
                ("total_version_rows", C.c_int64), ("plan_host", C.c_void_p), ("prologue", KvmPrologueExt), ("memory", KvmMemory),
                ("cache", KvmDecodeCache), ("decode_workspace", C.c_void_p), ("out", C.c_void_p), ("workspace", C.c_void_p),
                ("workspace_bytes", C.c_size_t)]


EXPORTS = [
    "kvm_prefill_workspace_bytes", "kvm_prefill_forward", "kvm_decode_workspace_bytes", "kvm_decode_step",
    "kvm_memory_refresh", "kvm_last_error_string", "kvm_abi_version", "kvm_decode_step_static", "kvm_prefill_status", "kvm_decode_run",
    "kvm_decode_status", "kvm_prefill_workspace_layout", "kvm_interleave_shards", "kvm_prologue_forward", "kvm_prologue_forward_ext",
    "kvm_prefill_forward_gathered", "kvm_decode_step_call", "kvm_decode_span",
    "kvm_decode_cache_fill", "kvm_project", "kvm_token_scratch_bytes", "kvm_mixer_token",
    "kvm_prompt_workspace_bytes", "kvm_mixer_prompt",
]
STATIC_SCRATCH_BYTES = 32 << 20
PROJECT_ROWS_MAX = 128  # rows of one kvm_project
SPAN_COLUMNS, SPAN_BATCH_MAX = 32, 1024  # tokens x query heads per kv head, and sequences, of one kvm_decode_span
UPDATE_LIST_MAX = 64  # updating sequences that a decode launch can list by itself

_lib = None


def load():
    """Load the library (once) and declare the signatures.  Raises if it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(LIB_PATH):
        raise RuntimeError(
            f"{LIB_PATH} is missing: build it with `python -m kvm_paper_b200.build` "
            "(this package has no CPU or PyTorch fallback)")
    lib = C.CDLL(LIB_PATH)
    LP = C.POINTER
    lib.kvm_prefill_workspace_bytes.restype = C.c_size_t
    lib.kvm_prefill_workspace_bytes.argtypes = [LP(KvmLayer), C.c_int32, C.c_int64, C.c_int64]
    lib.kvm_prefill_forward.restype = C.c_int
    lib.kvm_prefill_forward.argtypes = [
        LP(KvmLayer), C.c_int32, C.c_int64, KvmTensor4, KvmTensor4, KvmTensor4, KvmTensor4,
        C.c_void_p, LP(KvmUpdatePlan), C.c_int32, C.c_int64, KvmMemory, C.c_void_p, C.c_void_p,
        C.c_void_p, C.c_size_t, C.c_uint32, C.c_void_p]
    lib.kvm_prefill_forward_gathered.restype = C.c_int
    lib.kvm_prefill_forward_gathered.argtypes = [
        LP(KvmLayer), C.c_int32, C.c_int64, KvmTensor4, KvmTensor4, KvmTensor4, KvmTensor4,
        C.c_void_p, LP(KvmUpdatePlan), C.c_int32, C.c_int64, KvmMemory, C.c_int32, C.c_int32, LP(C.c_void_p), C.c_void_p,
        C.c_void_p, C.c_size_t, C.c_uint32, C.c_void_p]
    lib.kvm_prefill_status.restype = C.c_int
    lib.kvm_prefill_status.argtypes = [C.c_void_p, C.c_void_p]
    lib.kvm_prefill_workspace_layout.restype = C.c_int
    lib.kvm_prefill_workspace_layout.argtypes = [LP(KvmLayer), C.c_int32, C.c_int64, C.c_int64, LP(KvmPrefillLayout)]
    lib.kvm_decode_status.restype = C.c_int
    lib.kvm_decode_status.argtypes = [LP(KvmLayer), C.c_int32, C.c_void_p, C.c_void_p]
    lib.kvm_decode_workspace_bytes.restype = C.c_size_t
    lib.kvm_decode_workspace_bytes.argtypes = [LP(KvmLayer), C.c_int32, C.c_int32]
    lib.kvm_decode_step.restype = C.c_int
    lib.kvm_decode_step.argtypes = [
        LP(KvmLayer), C.c_int32, KvmDecodeCache, KvmTensor4, KvmTensor4, KvmTensor4, KvmTensor4,
        C.c_void_p, C.c_int32, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
    lib.kvm_decode_step_call.restype = C.c_int
    lib.kvm_decode_step_call.argtypes = [C.c_void_p, C.c_void_p]  # (a kept kvm_decode_call, by its address)
    lib.kvm_decode_span.restype = C.c_int
    lib.kvm_decode_span.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64, C.c_int64, C.c_int64, C.c_int64, C.c_void_p]
    lib.kvm_decode_cache_fill.restype = C.c_int
    lib.kvm_decode_cache_fill.argtypes = [LP(KvmLayer), C.c_int32, C.c_int64, KvmTensor4, KvmTensor4, KvmTensor4, KvmMemory, C.c_int32,
                                          KvmDecodeCache, C.c_void_p, C.c_void_p]
    lib.kvm_decode_run.restype = C.c_int
    lib.kvm_decode_run.argtypes = [
        LP(KvmLayer), C.c_int32, KvmDecodeCache, C.c_int32, KvmTensor4, KvmTensor4, KvmTensor4, KvmTensor4,
        C.c_int64, C.c_int64, C.c_int64, C.c_void_p, LP(C.c_int32), LP(C.c_int32), C.c_void_p, C.c_void_p,
        C.c_size_t, C.c_void_p]
    # decode step with the scratch inside the library (for callers that cannot allocate device memory)
    lib.kvm_decode_step_static.restype = C.c_int
    lib.kvm_decode_step_static.argtypes = [
        LP(KvmLayer), C.c_int32, KvmDecodeCache, KvmTensor4, KvmTensor4, KvmTensor4, KvmTensor4,
        C.c_void_p, C.c_int32, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.kvm_memory_refresh.restype = C.c_int
    lib.kvm_memory_refresh.argtypes = [LP(KvmLayer), C.c_int32, KvmMemory, C.c_void_p, C.c_void_p]
    for fn, arg in ((lib.kvm_prologue_forward, KvmPrologue), (lib.kvm_prologue_forward_ext, KvmPrologueExt)):
        fn.restype = C.c_int
        fn.argtypes = [LP(KvmLayer), C.c_int32, C.c_int64, LP(arg), C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int64,
                       C.c_void_p, C.c_size_t, C.c_void_p]
    lib.kvm_token_scratch_bytes.restype = C.c_size_t
    lib.kvm_token_scratch_bytes.argtypes = [LP(KvmLayer), C.c_int32]
    lib.kvm_mixer_token.restype = C.c_int
    lib.kvm_mixer_token.argtypes = [C.c_void_p, C.c_void_p]  # (kept calls, by their addresses)
    lib.kvm_prompt_workspace_bytes.restype = C.c_size_t
    lib.kvm_prompt_workspace_bytes.argtypes = [LP(KvmLayer), C.c_int32, C.c_int64, C.c_int32, C.c_int64]
    lib.kvm_mixer_prompt.restype = C.c_int
    lib.kvm_mixer_prompt.argtypes = [C.c_void_p, C.c_void_p]
    lib.kvm_project.restype = C.c_int
    lib.kvm_project.argtypes = [C.c_void_p, C.c_int64, C.c_int32, C.c_int32, LP(C.c_void_p), LP(C.c_int32), C.c_int32, C.c_void_p,
                                C.c_int64, C.c_void_p]
    lib.kvm_interleave_shards.restype = C.c_int
    lib.kvm_interleave_shards.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_int64, C.c_int64, C.c_void_p]
    lib.kvm_last_error_string.restype = C.c_char_p
    lib.kvm_last_error_string.argtypes = []
    lib.kvm_abi_version.restype = C.c_int
    lib.kvm_abi_version.argtypes = []
    _lib = lib
    return lib


class KvmError(RuntimeError):
    """A C-ABI call returned a non-zero status."""

    def __init__(self, code: int, message: str):
        super().__init__(f"kvm_b200 status {code} ({ERROR_NAMES.get(code, '?')}): {message}")
        self.code = code


def check(code: int) -> None:
    """Map a status code to the exception type the reference would raise for the same misuse:
    ValueError for unsupported/bad arguments, RuntimeError otherwise."""
    if code == KVM_OK:
        return
    msg = load().kvm_last_error_string().decode()
    if code in (1, 5):
        raise ValueError(f"kvm_b200 status {code} ({ERROR_NAMES[code]}): {msg}")
    raise KvmError(code, msg)
