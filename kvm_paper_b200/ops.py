"""Host side of the KVM operators: schedule tables, device buffers and the calls into libkvm_b200.

PyTorch is used for device memory and streams only; every kernel runs inside the C-ABI library.
Names follow the reference: "memory" = the compressed key/value means (``kvm_s_k`` / ``kvm_s_v`` /
``kvm_s_vlen``), "window" = the block sliding window (BSWA), "block" = ``chunk_len`` tokens.
"""

from __future__ import annotations

import ctypes as C
import math
import operator
from dataclasses import dataclass
from typing import Any, Callable

import numpy as np
import torch

from . import _lib
from ._lib import KvmDecodeCache as _CCache
from ._lib import KvmLayer, KvmMemory, KvmTensor4, KvmUpdatePlan



def _ptr(t: torch.Tensor | None) -> int | None:
    return None if t is None else t.data_ptr()


# address of a device's current stream: the raw query of the torch build, or the stream object where a build lacks it
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda i: torch.cuda.current_stream(i).cuda_stream)


def _stream_ptr(device) -> int:
    i = device.index
    return _raw_stream(torch.cuda.current_device() if i is None else i)


def _tensor4(t: torch.Tensor, name: str) -> KvmTensor4:
    """[B,H,T,D] view with a contiguous last dimension -> C descriptor (strides in elements)."""
    if t.dim() != 4:
        raise ValueError(f"{name} must be 4-dimensional, got {tuple(t.shape)}")
    if t.dtype != torch.bfloat16:
        raise ValueError(f"{name} must be bfloat16, got {t.dtype}")
    if not t.is_cuda:
        raise RuntimeError(f"{name} must live on a CUDA device")
    if t.size(-1) > 1 and t.stride(-1) != 1:
        t = t.contiguous()
    return KvmTensor4(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2))


def _as_bf16_view(t: torch.Tensor) -> torch.Tensor:
    """Keep strided views as they are; only fix dtype / inner stride."""
    if t.dtype != torch.bfloat16:
        t = t.to(torch.bfloat16)
    if t.size(-1) > 1 and t.stride(-1) != 1:
        t = t.contiguous()
    return t


def _fill_tensor4(dst: KvmTensor4, t: torch.Tensor, name: str) -> torch.Tensor:
    """``_tensor4`` into a kept C descriptor; returns the tensor the descriptor points into."""
    st = t.stride()
    if len(st) != 4:
        raise ValueError(f"{name} must be 4-dimensional, got {tuple(t.shape)}")
    if t.dtype is not torch.bfloat16 or (st[3] != 1 and t.size(3) > 1):
        t = _as_bf16_view(t)
        st = t.stride()
    if not t.is_cuda:
        raise RuntimeError(f"{name} must live on a CUDA device")
    dst.ptr, dst.stride_b, dst.stride_h, dst.stride_t = t.data_ptr(), st[0], st[1], st[2]
    return t


@dataclass
class LayerConfig:
    """Static description of one mixer layer (mirror of ``kvm_layer``)."""

    n_q_heads: int
    n_kv_heads: int
    head_dim: int
    chunk_len: int
    n_bswa_chunks: int
    rope_dim: int
    sink_len: int
    gate_keys: bool = True
    gate_values: bool = True
    gate_appends: bool = False
    gate_initial: bool = False
    ln_eps: float = 1e-5


class LayerParams:
    """Device copies (fp32) of the small parameter vectors the kernels read, plus the C struct."""

    def __init__(self, cfg: LayerConfig, ln_weight: torch.Tensor, ln_bias: torch.Tensor,
                 front_temp: torch.Tensor | None, state_temp: torch.Tensor | None, device):
        self.cfg = cfg
        dev = torch.device(device)
        self.device = dev
        self.ln_w = ln_weight.detach().to(dev, torch.float32).contiguous()
        self.ln_b = ln_bias.detach().to(dev, torch.float32).contiguous()
        ones = torch.ones(cfg.n_q_heads, device=dev, dtype=torch.float32)
        self.front = ones if front_temp is None else front_temp.detach().to(dev, torch.float32).contiguous()
        self.state = ones if state_temp is None else state_temp.detach().to(dev, torch.float32).contiguous()
        self.c = KvmLayer(
            cfg.n_q_heads, cfg.n_kv_heads, cfg.head_dim, cfg.chunk_len, cfg.n_bswa_chunks, cfg.rope_dim,
            cfg.sink_len, int(cfg.gate_keys), int(cfg.gate_values), int(cfg.gate_appends), int(cfg.gate_initial),
            float(cfg.ln_eps), self.ln_w.data_ptr(), self.ln_b.data_ptr(), self.front.data_ptr(), self.state.data_ptr())


# --------------------------------------------------------------------------------------- schedule

def bswa_begin_for_total_len(total_len: int, chunk_len: int, n_bswa_chunks: int) -> int:
    """Start of the block sliding window for a sequence of ``total_len`` tokens
    (reference: model/kvm_mixer.py:167-172)."""
    end = ((max(int(total_len), 0) + chunk_len - 1) // chunk_len) * chunk_len
    return max(0, end - n_bswa_chunks * chunk_len)


@dataclass
class PrefillPlan:
    """Per-update schedule of one prefill (uniform over the batch)."""

    seq_len: int
    state_before: list[int]
    n_append: list[int]
    version_row: list[int]
    total_version_rows: int
    final_state_len: int
    final_coverage: int
    bswa_begin: int

    @property
    def n_updates(self) -> int:
        return len(self.n_append) - 1

    def to_ctypes(self):
        arr = (KvmUpdatePlan * len(self.n_append))()
        for i, (sb, na, vr) in enumerate(zip(self.state_before, self.n_append, self.version_row)):
            arr[i] = KvmUpdatePlan(sb, na, vr, 0)
        return arr

    def to_array(self) -> np.ndarray:
        """The table as the C side reads it (kvm_update_plan)."""
        t = np.zeros((len(self.n_append), 4), dtype=np.int32)
        t[:, 0], t[:, 1], t[:, 2] = self.state_before, self.n_append, self.version_row
        return t

    def to_tensor(self, device) -> torch.Tensor:
        return torch.from_numpy(self.to_array()).to(device, non_blocking=True)


def build_prefill_plan(seq_len: int, chunk_len: int, n_bswa_chunks: int,
                       desired_state_len: Callable[[int, int, int], int], keep_versions: bool = True) -> PrefillPlan:
    """Walk the block loop of the reference prefill (model/kvm_mixer.py:450-488) on integers only.

    ``desired_state_len(ctx_len, available_context, current)`` is the mixer's own schedule method, so an
    overridden schedule flows through unchanged."""
    T, Cn, W = int(seq_len), int(chunk_len), int(n_bswa_chunks)
    n_blocks = (T + Cn - 1) // Cn
    init = min(T, Cn)
    state_before, n_append, version_row = [0], [init], [0]
    S = init
    rows = 0
    n_plan = n_blocks - W if n_blocks > W else 1
    keeps_versions = n_blocks > W
    if keeps_versions:
        rows = _round8(S)
    for u in range(1, n_plan):
        ctx_len = (u + W) * Cn
        available = (u + 1) * Cn
        desired = int(desired_state_len(ctx_len, available, S))
        na = min(max(desired - S, 0), Cn)
        state_before.append(S)
        n_append.append(na)
        S += na
        version_row.append(rows)
        rows += _round8(S)
    if not keeps_versions or not keep_versions:
        # no query block reads a memory version (short prompt), or only the final memory is wanted
        version_row = [-1] * len(n_append)
        rows = 0
    bb = bswa_begin_for_total_len(T, Cn, W)
    return PrefillPlan(T, state_before, n_append, version_row, rows, S, max(init, bb), bb)


def _round8(x: int) -> int:
    return (x + 7) // 8 * 8


# ----------------------------------------------------------------------------------------- memory

def _array(name: str):
    """Attribute ``name`` of an object whose arrays' addresses are kept in an argument block: assigning another array counts
    as a change (``changes``), behind which the block is filled in anew.  (Constructors and code that runs per token use
    ``_name``.)"""
    key = "_" + name

    def put(self, value):
        d = self.__dict__
        if d.get(key) is not value:
            d[key] = value
            d["changes"] = self.changes + 1

    return property(operator.attrgetter(key), put)


class MemoryBuffers:
    """The compressed memory of ``n_rows`` kv rows with ``capacity`` rows each (``zero``: rows past the live ones read as
    zeros; the kernels never look at them)."""

    changes = 0
    k_sum, v_sum, vlen, k_attn, v_attn, capacity = map(_array, ("k_sum", "v_sum", "vlen", "k_attn", "v_attn", "capacity"))

    def __init__(self, n_rows: int, capacity: int, head_dim: int, device, zero: bool = True):
        self.n_rows, self._capacity, self.head_dim = n_rows, int(capacity), head_dim
        make = torch.zeros if zero else torch.empty
        kw = dict(device=device, dtype=torch.bfloat16)
        self._k_sum = make(n_rows, capacity, head_dim, **kw)
        self._v_sum = make(n_rows, capacity, head_dim, **kw)
        self._vlen = make(n_rows, capacity, device=device, dtype=torch.float32)
        self._k_attn = make(n_rows, capacity, head_dim, **kw)
        self._v_attn = make(n_rows, capacity, head_dim, **kw)

    def c(self) -> KvmMemory:
        return KvmMemory(self._k_sum.data_ptr(), self._v_sum.data_ptr(), self._vlen.data_ptr(),
                         self._k_attn.data_ptr(), self._v_attn.data_ptr(), self._capacity)

    def grown(self, new_capacity: int) -> "MemoryBuffers":
        out = MemoryBuffers(self.n_rows, new_capacity, self.head_dim, self.k_sum.device)
        n = self.capacity
        for name in ("k_sum", "v_sum", "vlen", "k_attn", "v_attn"):
            getattr(out, name)[:, :n].copy_(getattr(self, name))
        return out


@dataclass
class PrefillResult:
    out: torch.Tensor                 # [B, T, Hq*D] bf16, the input of c_proj
    memory: MemoryBuffers
    plan: PrefillPlan
    route: torch.Tensor | None        # [B*Hkv, n_updates+1, C] int32 if requested
    runner: Any = None                # the PrefillRunner that produced it (workspace inspection)


class PrologueParams:
    """What the fused prologue reads besides the projections, on the device: token-shift scales (bf16),
    per-head LayerNorm of q and k (a fp32 copy), all optional as in the reference module
    (model/value_residual_mixin.py:60-98).  ``share_ln``: the kernel reads bf16 LayerNorm weights where they are instead
    of a copy; ``shared`` then says whether all of it lives in the parameters themselves, whatever is written to them."""

    def __init__(self, device, *, shift_q=None, shift_k=None, shift_v=None, ln_q=None, ln_k=None, ln_eps: float = 1e-5,
                 share_ln: bool = False):
        dev = torch.device(device)
        given = [shift_q, shift_k, shift_v]
        shifts = [None if t is None else t.detach().to(dev, torch.bfloat16).reshape(-1).contiguous() for t in (shift_q, shift_k, shift_v)]
        if any(t is None for t in shifts) and not all(t is None for t in shifts):
            raise ValueError("token-shift scales must be given for q, k and v or for none")
        self.shift_q, self.shift_k, self.shift_v = shifts
        if (ln_q is None) != (ln_k is None):
            raise ValueError("LayerNorm must be given for q and k or for neither")
        self.ln, self.ln_bf16 = None, 0
        if ln_q is not None:
            ln = (ln_q.weight, ln_q.bias, ln_k.weight, ln_k.bias)
            given += ln
            self.ln_bf16 = int(share_ln and all(t.dtype is torch.bfloat16 and t.device == dev and t.is_contiguous()
                                                and t.data_ptr() % 16 == 0 for t in ln))
            self.ln = tuple(t.detach() if self.ln_bf16 else t.detach().to(dev, torch.float32).contiguous() for t in ln)
        self.shared = share_ln and all(a is None or a.data_ptr() == b.data_ptr() for a, b in zip(given, [*shifts, *(self.ln or ())]))
        self.ln_eps = float(ln_eps)
        self.shift_ptrs = tuple(_ptr(t) for t in (self.shift_q, self.shift_k, self.shift_v))
        self.ln_ptrs = None if self.ln is None else tuple(t.data_ptr() for t in self.ln)


def _token_stride(t: torch.Tensor, B: int, T: int, width: int, name: str) -> int:
    """Elements from token to token of a [B,T,width] bf16 projection output: contiguous, or a column range of wider rows."""
    if t.dtype is not torch.bfloat16 or not t.is_cuda or t.shape != (B, T, width):
        raise ValueError(f"{name} projection must be a bf16 CUDA tensor [B,T,{width}], got {tuple(t.shape)} {t.dtype}")
    st = t.stride()
    step = _row_step(st, B, T, width)
    if step is None:
        raise ValueError(f"{name} projection must be contiguous or a column range of contiguous rows, got strides {st}")
    return step


def _row_step(st, B: int, T: int, width: int) -> int | None:
    """Elements from row to row of a [B,T,width] tensor with these strides, None where its rows do not lie one step apart."""
    step = st[1] if T > 1 else (st[0] if B > 1 else (width + 7) // 8 * 8)
    # (a stride of 0 means "contiguous" to the library: rows that are one and the same row do not pass for that)
    if (st[2] != 1 and width > 1) or step < width or (B > 1 and st[0] != T * step):
        return None
    return step


def rotary_tables_arg(position_embeddings, B: int, T: int, D: int, dev):
    """(cos, sin) as contiguous bf16 tables on the device, and whether every sequence has its own."""
    cs = [t if t.dtype is torch.bfloat16 and t.device == dev and t.is_contiguous() else t.to(dev, torch.bfloat16).contiguous()
          for t in position_embeddings]
    n = cs[0].numel() // (T * D)
    if n not in (1, B) or cs[0].numel() != n * T * D or cs[1].numel() != cs[0].numel():
        raise ValueError(f"rotary tables must be [1 or {B}, {T}, .., {D}], got {tuple(cs[0].shape)} and {tuple(cs[1].shape)}")
    return cs[0], cs[1], n > 1


def _aligned(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and on a 16-byte boundary, by a copy where it is not."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _aligned_rows(t: torch.Tensor) -> torch.Tensor:
    """[B,H,T,D] in bf16 whose rows are contiguous and start on 16-byte boundaries, as a view where that is so already."""
    t = _as_bf16_view(t)
    return t if t.data_ptr() % 16 == 0 and not any(s % 8 for s in t.stride()[:-1]) else _aligned(t)


def _first_values(v_first: torch.Tensor, B: int, T: int, width: int, dev) -> torch.Tensor:
    """The first layer's values [B,T,width] as the value residual's kernels read them: broadcast, bf16, contiguous, aligned."""
    if v_first.device != dev:
        raise RuntimeError(f"v_first must be on {dev}, got {v_first.device}")
    if v_first.shape != (B, T, width):
        v_first = v_first.expand(B, T, width)
    return _aligned(v_first.to(torch.bfloat16))


def _prev_rows(prev, B: int, dev, widths=None) -> list[torch.Tensor]:
    """The cached rows [B,1,width] of the previous token as the prologue kernel reads them."""
    rows = []
    for t, width in zip(prev, widths or [t.size(-1) for t in prev]):
        st = t.stride()
        if not (t.shape == (B, 1, width) and t.dtype is torch.bfloat16 and t.device == dev and st[2] == 1 and st[0] % 8 == 0
                and st[0] >= width and t.data_ptr() % 16 == 0):
            t = _aligned(t.to(dev, torch.bfloat16).reshape(B, 1, -1))
            if t.size(2) != width:
                raise ValueError(f"cached rows must be [{B},1,{width}], got {tuple(t.shape)}")
        rows.append(t)
    return rows


def _prologue_arg(params: LayerParams, pro: PrologueParams, q_lin, k_lin, v_lin, gate_lin, position_embeddings, prev, value_residual,
                  v_last):
    """The C argument block of the prologue and the tensors it points into (see ``prologue_forward``)."""
    cfg = params.cfg
    B, T, _ = q_lin.shape
    D, Hq, Hkv = cfg.head_dim, cfg.n_q_heads, cfg.n_kv_heads
    dev = q_lin.device
    keep = []
    arg = _lib.KvmPrologueExt()
    arg.q_lin, arg.k_lin, arg.v_lin = q_lin.data_ptr(), k_lin.data_ptr(), v_lin.data_ptr()
    arg.q_stride_t, arg.k_stride_t, arg.v_stride_t = (
        _token_stride(t, B, T, h * D, n) for n, t, h in (("q", q_lin, Hq), ("k", k_lin, Hkv), ("v", v_lin, Hkv)))
    if gate_lin is not None:
        fits = gate_lin.dtype is torch.bfloat16 and gate_lin.is_cuda and gate_lin.shape == (B, T, Hkv)
        step = _row_step(gate_lin.stride(), B, T, Hkv) if fits else None
        if step is None:
            gate_lin = gate_lin.to(torch.bfloat16).reshape(B, T, Hkv).contiguous()
            keep.append(gate_lin)
            step = _token_stride(gate_lin, B, T, Hkv, "gate")
        arg.gate_lin, arg.gate_stride_t = gate_lin.data_ptr(), step
    if value_residual is not None:
        v_first = _first_values(value_residual[0], B, T, Hkv * D, dev)
        v_gate, v_gate0 = (_aligned(t.to(dev, torch.bfloat16)) for t in value_residual[1:])
        if v_gate.numel() != B * T * Hkv * D or v_gate0.numel() != Hkv * D:
            raise ValueError(f"value residual: v_gate must have {Hkv * D} values per token, v_gate0 {Hkv * D}")
        keep += [v_first, v_gate, v_gate0]
        arg.v_first, arg.v_gate, arg.v_gate0 = v_first.data_ptr(), v_gate.data_ptr(), v_gate0.data_ptr()
        if v_last is not None:
            arg.v_last = v_last.data_ptr()
    if pro.shift_q is not None:
        arg.shift_q, arg.shift_k, arg.shift_v = pro.shift_ptrs
        if prev is not None and all(t is not None for t in prev):
            pv = _prev_rows(prev, B, dev, (Hq * D, Hkv * D, Hkv * D))
            keep += pv
            arg.prev_q, arg.prev_k, arg.prev_v = (t.data_ptr() for t in pv)
            if B > 1:
                arg.prev_q_stride_b, arg.prev_k_stride_b, arg.prev_v_stride_b = (t.stride(0) for t in pv)
    if pro.ln is not None:
        arg.ln_q_w, arg.ln_q_b, arg.ln_k_w, arg.ln_k_b = pro.ln_ptrs
        arg.ln_qk_eps, arg.ln_bf16 = pro.ln_eps, pro.ln_bf16
    if position_embeddings is not None:
        cos, sin, own = rotary_tables_arg(position_embeddings, B, T, D, dev)
        keep += [cos, sin]
        arg.cos, arg.sin, arg.rope_stride_b = cos.data_ptr(), sin.data_ptr(), T * D if own else 0
    return arg, keep


def prologue_forward(params: LayerParams, pro: PrologueParams, q_lin: torch.Tensor, k_lin: torch.Tensor, v_lin: torch.Tensor,
                     gate_lin: torch.Tensor | None, position_embeddings, *, prev=None, runner: "PrefillRunner | None" = None,
                     out: tuple | None = None, value_residual: tuple | None = None, v_last: torch.Tensor | None = None):
    """Value residual, token shift, q/k LayerNorm, rotary embedding and merge gate in one kernel over the projection
    outputs ([B,T,H*D] bf16, contiguous or column ranges of one wider GEMM output).  Returns q [B,Hq,T,D], k, v
    [B,Hkv,T,D], gate [B,Hkv,T,1] as views of [B,T,H,D] / [B,Hkv,T]
    buffers, the layouts the reference hands its mixer (model/kvm_mixer.py:397-399).  With ``runner`` the prepared
    keys of the tokens that memory updates consume are written into that runner's workspace, and its ``run`` may
    be called with ``keys_prepared=True``.  ``prev`` = (q, k, v) rows [B,1,H*D] of the previous call's last token.
    ``out`` = preallocated (q [B,T,Hq,D], k, v [B,T,Hkv,D], gate [B,Hkv,T]) bf16 buffers to write into.
    ``value_residual`` = (v_first, output of v_gate2, v_gate0) of the "rwkv" value residual; ``v_last`` [B,1,Hkv*D]
    receives the last token's value behind it (what the next call's ``prev`` needs)."""
    cfg = params.cfg
    B, T, _ = q_lin.shape
    D, Hq, Hkv = cfg.head_dim, cfg.n_q_heads, cfg.n_kv_heads
    dev = q_lin.device
    arg, keep = _prologue_arg(params, pro, q_lin, k_lin, v_lin, gate_lin, position_embeddings, prev, value_residual, v_last)
    if out is not None:
        q, k, v, gate = out
        for t, shape in ((q, (B, T, Hq, D)), (k, (B, T, Hkv, D)), (v, (B, T, Hkv, D)), (gate, (B, Hkv, T))):
            if tuple(t.shape) != shape or t.dtype != torch.bfloat16 or not t.is_contiguous() or t.device != dev:
                raise ValueError(f"out buffer must be a contiguous bf16 tensor {shape} on {dev}, got {tuple(t.shape)} {t.dtype}")
    else:
        q = torch.empty(B, T, Hq, D, device=dev, dtype=torch.bfloat16)
        k = torch.empty(B, T, Hkv, D, device=dev, dtype=torch.bfloat16)
        v = torch.empty(B, T, Hkv, D, device=dev, dtype=torch.bfloat16)
        gate = torch.empty(B, Hkv, T, device=dev, dtype=torch.bfloat16)
    ws_ptr, ws_bytes, ver_rows = None, 0, 0
    if runner is not None:
        if runner.batch != B or runner.plan.seq_len != T:
            raise ValueError("runner was built for another batch or sequence length")
        ws_ptr, ws_bytes, ver_rows = runner.ws.data_ptr(), runner.ws_bytes, runner.plan.total_version_rows
    rc = _lib.load().kvm_prologue_forward_ext(C.byref(params.c), B, T, C.byref(arg), q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                          gate.data_ptr(), ver_rows, ws_ptr, ws_bytes, _stream_ptr(dev))
    if rc:
        _lib.check(rc)
    del keep  # (the kernel is enqueued on the current stream: torch's allocator keeps the blocks until it has run)
    return q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), gate.unsqueeze(-1)


def project(x: torch.Tensor, weights: list[torch.Tensor]) -> torch.Tensor:
    """[rows, width] bf16 (at most ``PROJECT_ROWS_MAX`` rows) times the transposed weights, side by side:
    [rows, sum of the weights' rows], in one launch."""
    width = x.size(1)
    for w in weights:
        if w.dim() != 2 or w.size(1) != width or w.dtype is not torch.bfloat16 or not w.is_contiguous() or w.device != x.device:
            raise ValueError(f"weights must be contiguous bf16 [.., {width}] on {x.device}, got {tuple(w.shape)} {w.dtype} on {w.device}")
    if x.dtype is not torch.bfloat16 or not x.is_cuda:
        raise ValueError(f"project expects bf16 rows on a CUDA device, got {x.dtype} on {x.device}")
    return project_checked(x, weights)


def project_checked(x: torch.Tensor, weights: list[torch.Tensor]) -> torch.Tensor:
    """``project`` for a caller that has looked at the weights' types, shapes and devices."""
    rows, width = x.shape
    step, inner = x.stride()
    if inner != 1 or step % 8 or step < width or x.data_ptr() % 16:
        x = x.clone(memory_format=torch.contiguous_format)
        step = x.stride(0)
    n = len(weights)
    sizes = [w.shape[0] for w in weights]
    cols = (sum(sizes) + 7) // 8 * 8  # (16-byte aligned rows)
    out = torch.empty(rows, cols, device=x.device, dtype=torch.bfloat16)
    rc = _lib.load().kvm_project(x.data_ptr(), step, rows, width, (C.c_void_p * n)(*[w.data_ptr() for w in weights]),
                                 (C.c_int32 * n)(*sizes), n, out.data_ptr(), cols, _stream_ptr(x.device))
    if rc:
        _lib.check(rc)
    return out


class PrefillRunner:
    """Preallocated buffers for repeated prefills of one shape (memory, workspace with the row pool and version tables, output).

    ``run`` only enqueues kernels on the current stream; nothing is allocated per call."""

    def __init__(self, params: LayerParams, batch: int, plan: PrefillPlan, *, memory_capacity: int | None = None,
                 want_route: bool = False, zero_memory: bool = True):
        lib = _lib.load()
        cfg = params.cfg
        self.params, self.plan, self.batch = params, plan, int(batch)
        dev = params.device
        cap = max(plan.final_state_len, 1) if memory_capacity is None else int(memory_capacity)
        self.memory = MemoryBuffers(batch * cfg.n_kv_heads, cap, cfg.head_dim, dev, zero_memory)
        self.ws_bytes = lib.kvm_prefill_workspace_bytes(C.byref(params.c), batch, plan.seq_len, plan.total_version_rows)
        self.ws = torch.empty(self.ws_bytes, device=dev, dtype=torch.uint8)
        self.out = torch.empty(batch, plan.seq_len, cfg.n_q_heads * cfg.head_dim, device=dev, dtype=torch.bfloat16)
        self.route = None
        if want_route:
            self.route = torch.zeros(batch * cfg.n_kv_heads, plan.n_updates + 1, cfg.chunk_len, device=dev, dtype=torch.int32)
        self.plan_dev = plan.to_tensor(dev)
        self.plan_host = plan.to_ctypes()

    def run(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, gate: torch.Tensor,
            phases: int = _lib.PREFILL_CHAIN | _lib.PREFILL_ATTENTION, *, keys_prepared: bool = False) -> torch.Tensor:
        """``keys_prepared``: ``prologue_forward(..., runner=self)`` has written the prepared keys of this prompt into
        the workspace; the chain phase skips its own pass over the keys."""
        cfg, plan = self.params.cfg, self.plan
        if keys_prepared:
            phases |= _lib.PREFILL_KEYS_PREPARED
        B, Hq, T, D = q.shape
        if (B, Hq, D) != (self.batch, cfg.n_q_heads, cfg.head_dim) or k.shape != (B, cfg.n_kv_heads, T, D) or v.shape != k.shape:
            raise ValueError(f"shape mismatch: q {tuple(q.shape)}, k {tuple(k.shape)}, v {tuple(v.shape)} for {cfg}")
        if gate.shape != (B, cfg.n_kv_heads, T, 1):
            raise ValueError(f"merge gate must be [B,Hkv,T,1], got {tuple(gate.shape)}")
        if T != plan.seq_len:
            raise ValueError("plan was built for another sequence length")
        q, k, v, gate = (_as_bf16_view(t) for t in (q, k, v, gate))
        rc = _lib.load().kvm_prefill_forward(
            C.byref(self.params.c), B, T, _tensor4(q, "q"), _tensor4(k, "k"), _tensor4(v, "v"), _tensor4(gate, "gate"),
            self.plan_dev.data_ptr(), self.plan_host, plan.n_updates, plan.total_version_rows, self.memory.c(),
            self.out.data_ptr(), _ptr(self.route), self.ws.data_ptr(), self.ws_bytes, phases,
            _stream_ptr(self.params.device))
        _lib.check(rc)
        return self.out

    def run_gathered(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, gate: torch.Tensor, rank: int, out_ptrs: list[int],
                     phases: int = _lib.PREFILL_CHAIN | _lib.PREFILL_ATTENTION, *, keys_prepared: bool = False) -> None:
        """One rank of a head-sharded prefill whose attention kernel writes this rank's heads into every rank's
        [B,T,world*Hq*D] output (``out_ptrs``: addresses of all ranks' buffers as this process sees them, see
        ``sharding.GatheredPrefillOutput``).  Nothing is returned: a buffer is complete once every rank's call has
        finished (the caller synchronises the ranks)."""
        cfg, plan = self.params.cfg, self.plan
        B, Hq, T, D = q.shape
        if (B, Hq, D) != (self.batch, cfg.n_q_heads, cfg.head_dim) or k.shape != (B, cfg.n_kv_heads, T, D) or v.shape != k.shape:
            raise ValueError(f"shape mismatch: q {tuple(q.shape)}, k {tuple(k.shape)}, v {tuple(v.shape)} for {cfg}")
        if gate.shape != (B, cfg.n_kv_heads, T, 1) or T != plan.seq_len:
            raise ValueError("merge gate must be [B,Hkv,T,1] and the plan built for this sequence length")
        if keys_prepared:
            phases |= _lib.PREFILL_KEYS_PREPARED
        q, k, v, gate = (_as_bf16_view(t) for t in (q, k, v, gate))
        bases = (C.c_void_p * len(out_ptrs))(*out_ptrs)
        rc = _lib.load().kvm_prefill_forward_gathered(
            C.byref(self.params.c), B, T, _tensor4(q, "q"), _tensor4(k, "k"), _tensor4(v, "v"), _tensor4(gate, "gate"),
            self.plan_dev.data_ptr(), self.plan_host, plan.n_updates, plan.total_version_rows, self.memory.c(),
            len(out_ptrs), int(rank), bases, _ptr(self.route), self.ws.data_ptr(), self.ws_bytes, phases,
            _stream_ptr(self.params.device))
        _lib.check(rc)

    def check_status(self) -> None:
        """Synchronise and raise if a kernel of the last run reported a device-side timeout."""
        rc = _lib.load().kvm_prefill_status(self.ws.data_ptr(), _stream_ptr(self.params.device))
        _lib.check(rc)

    def workspace_views(self) -> dict[str, torch.Tensor]:
        """Views (no copies) of what the last run left in the workspace, for inspection: the row pool of the
        memory's attention view ``pool_k`` / ``pool_v`` [kv rows, pool_rows, D], the version tables
        ``versions`` [kv rows, total_version_rows] (entry ``plan.version_row[u] + r`` = pool row of memory
        row ``r`` after update ``u``) and the prepared keys ``prepared_keys`` [kv rows, (n_updates+1)*C, D]."""
        cfg, plan = self.params.cfg, self.plan
        lay = _lib.KvmPrefillLayout()
        _lib.check(_lib.load().kvm_prefill_workspace_layout(C.byref(self.params.c), self.batch, plan.seq_len,
                                                            plan.total_version_rows, C.byref(lay)))
        rows, D = self.batch * cfg.n_kv_heads, cfg.head_dim

        def view(offset, shape, dtype):
            n = math.prod(shape) * torch.empty((), dtype=dtype).element_size()
            return self.ws[offset:offset + n].view(dtype).view(shape)

        out = {"pool_k": view(lay.pool_k_offset, (rows, lay.pool_rows, D), torch.bfloat16),
               "pool_v": view(lay.pool_v_offset, (rows, lay.pool_rows, D), torch.bfloat16),
               "versions": view(lay.version_table_offset, (rows, plan.total_version_rows), torch.int32)}
        if plan.n_updates > 0:
            out["prepared_keys"] = view(lay.prepared_keys_offset, (rows, (plan.n_updates + 1) * cfg.chunk_len, D),
                                        torch.bfloat16)
        return out


class HostPrefill:
    """Prefill whose inputs and output live in pinned host memory (a serving front end that receives the
    post-QKV tensors of a request batch on the host): the batch is cut into slices of sequences and slice
    i+1 is copied in while slice i is computed and slice i-1 is copied out, on three streams (copy-in,
    the caller's current stream, copy-out) with two sets of device buffers.

    Host tensors are laid out as the projections produce them: q [B,T,Hq,D], k/v [B,T,Hkv,D],
    gate [B,T,Hkv,1], out [B,T,Hq*D], all bf16 and pinned."""

    def __init__(self, params: LayerParams, batch: int, plan: PrefillPlan, slice_batch: int = 1):
        cfg = params.cfg
        if batch % slice_batch:
            raise ValueError(f"batch {batch} is not a multiple of the slice size {slice_batch}")
        dev = params.device
        self.params, self.plan, self.batch, self.bs = params, plan, int(batch), int(slice_batch)
        T, D = plan.seq_len, cfg.head_dim
        kw = dict(device=dev, dtype=torch.bfloat16)
        self.runners = [PrefillRunner(params, self.bs, plan) for _ in range(2)]
        self.dev_in = [(torch.empty(self.bs, T, cfg.n_q_heads, D, **kw), torch.empty(self.bs, T, cfg.n_kv_heads, D, **kw),
                        torch.empty(self.bs, T, cfg.n_kv_heads, D, **kw), torch.empty(self.bs, T, cfg.n_kv_heads, 1, **kw))
                       for _ in range(2)]
        self.s_in, self.s_out = torch.cuda.Stream(device=dev), torch.cuda.Stream(device=dev)
        self.ev_kv = [torch.cuda.Event() for _ in range(2)]      # keys, values and gates of the slot have arrived
        self.ev_in = [torch.cuda.Event() for _ in range(2)]      # ... and the queries
        self.ev_comp = [torch.cuda.Event() for _ in range(2)]    # the slot's kernels are done (inputs free, output ready)
        self.ev_out = [torch.cuda.Event() for _ in range(2)]     # the slot's output has left the device

    def run(self, hq: torch.Tensor, hk: torch.Tensor, hv: torch.Tensor, hg: torch.Tensor, h_out: torch.Tensor) -> torch.Tensor:
        for name, t in (("q", hq), ("k", hk), ("v", hv), ("gate", hg), ("out", h_out)):
            if t.is_cuda or not t.is_pinned() or t.dtype != torch.bfloat16 or t.size(0) != self.batch:
                raise ValueError(f"{name} must be a pinned bf16 host tensor with batch {self.batch}")
        cur = torch.cuda.current_stream(self.params.device)
        self.s_in.wait_stream(cur)  # whatever produced the host buffers' contents is ordered before the copies
        n = self.batch // self.bs
        for i in range(n):
            slot, lo = i % 2, i * self.bs
            with torch.cuda.stream(self.s_in):
                if i >= 2:
                    self.s_in.wait_event(self.ev_comp[slot])  # slice i-2 no longer reads these device buffers
                # keys, values and gates first: the memory trajectory does not need the queries
                for d, h in zip(self.dev_in[slot][1:], (hk, hv, hg)):
                    d.copy_(h[lo:lo + self.bs], non_blocking=True)
                self.ev_kv[slot].record(self.s_in)
                self.dev_in[slot][0].copy_(hq[lo:lo + self.bs], non_blocking=True)
                self.ev_in[slot].record(self.s_in)
            dq, dk, dv, dg = (t.transpose(1, 2) for t in self.dev_in[slot])
            cur.wait_event(self.ev_kv[slot])
            self.runners[slot].run(dq, dk, dv, dg, phases=_lib.PREFILL_CHAIN)
            cur.wait_event(self.ev_in[slot])
            if i >= 2:
                cur.wait_event(self.ev_out[slot])  # the slot's output buffer has been copied out
            out = self.runners[slot].run(dq, dk, dv, dg, phases=_lib.PREFILL_ATTENTION)
            self.ev_comp[slot].record(cur)
            with torch.cuda.stream(self.s_out):
                self.s_out.wait_event(self.ev_comp[slot])
                h_out[lo:lo + self.bs].copy_(out, non_blocking=True)
                self.ev_out[slot].record(self.s_out)
        for slot in range(min(2, n)):
            cur.wait_event(self.ev_out[slot])  # the call is complete, in stream order, when the output is on the host
        return h_out


def prefill_forward(params: LayerParams, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, gate: torch.Tensor,
                    plan: PrefillPlan, *, memory_capacity: int | None = None, want_route: bool = False,
                    phases: int = _lib.PREFILL_CHAIN | _lib.PREFILL_ATTENTION, check: bool = False,
                    runner: "PrefillRunner | None" = None, keys_prepared: bool = False) -> PrefillResult:
    """Whole-prompt prefill through ``kvm_prefill_forward``.

    q [B,Hq,T,D], k/v [B,Hkv,T,D], gate [B,Hkv,T,1]; strided views are passed as they are."""
    if q.dim() != 4:
        raise ValueError(f"q must be [B,Hq,T,D], got {tuple(q.shape)}")
    if not q.is_cuda:
        raise RuntimeError("kvm_b200 runs on CUDA tensors only (there is no CPU path)")
    if runner is None:  # (a caller that ran the fused prologue brings the runner whose workspace holds the prepared keys)
        runner = PrefillRunner(params, q.size(0), plan, memory_capacity=memory_capacity, want_route=want_route)
    out = runner.run(q, k, v, gate, phases=phases, keys_prepared=keys_prepared)
    if check:
        runner.check_status()
    # buffers are released by the caching allocator in stream order
    return PrefillResult(out, runner.memory, plan, runner.route, runner)


# ------------------------------------------------------------------------------------ decode cache

class KvmDecodeCache:
    """Device-resident decode state of one layer for ``batch`` sequences with ragged lengths.

    Replaces the reference's ``TritonKVMDecodeCache`` (model/kvm_triton_decode.py:34-400): preallocated
    memory rows, a ring of the last ``W*C`` tokens (token t at slot ``t mod W*C``) and per-sequence
    lengths on the device; ``logical_state_dict`` returns the reference's eager cache layout."""

    cache_representation = "preallocated memory rows + W*C-token ring, per-sequence lengths on device"
    changes = 0
    params, memory, ring_k, ring_v, ring_gate, out = map(_array, ("params", "memory", "ring_k", "ring_v", "ring_gate", "out"))
    total_len, state_len, total_len_h, state_len_h = map(_array, ("total_len", "state_len", "total_len_h", "state_len_h"))
    _quiet = 0
    _token = None  # the mixer's kept arguments of kvm_mixer_token for this cache

    def __init__(self, params: LayerParams, batch: int, state_capacity: int,
                 desired_state_len: Callable[[int, int, int], int], owner: Any = None, *, _memory: MemoryBuffers | None = None):
        """``_memory``: buffers to live in instead of new ones; the caller fills the cache before it is used (``_fill``)."""
        cfg = params.cfg
        self._params, self.cfg, self.batch, self.owner = params, cfg, int(batch), owner
        self.desired_state_len = desired_state_len
        dev = params.device
        self.device = dev
        self.kv_rows = batch * cfg.n_kv_heads
        self.ring_capacity = cfg.n_bswa_chunks * cfg.chunk_len
        self._memory = MemoryBuffers(self.kv_rows, max(int(state_capacity), 1), cfg.head_dim, dev) if _memory is None else _memory
        make = torch.zeros if _memory is None else torch.empty
        kw = dict(device=dev, dtype=torch.bfloat16)
        self._ring_k = make(self.kv_rows, self.ring_capacity, cfg.head_dim, **kw)
        self._ring_v = make(self.kv_rows, self.ring_capacity, cfg.head_dim, **kw)
        self._ring_gate = make(self.kv_rows, self.ring_capacity, **kw)
        self._lens = make(2, batch, device=dev, dtype=torch.int32)
        self._total_len, self._state_len = self._lens[0], self._lens[1]
        self._total_len_h = np.zeros(batch, dtype=np.int64)
        self._state_len_h = np.zeros(batch, dtype=np.int64)
        self.update_count = 0
        self._out = torch.empty(batch, 1, cfg.n_q_heads * cfg.head_dim, **kw)
        self.route = None
        self._last_any_update, self._last_n_append = False, None
        self._quiet = 0  # tokens until the next one that may update a memory or grow one directly (see _plan_step)
        self._max_rows = 0
        self._q_shape = (self.batch, cfg.n_q_heads, 1, cfg.head_dim)
        self._kv_shape = (self.batch, cfg.n_kv_heads, 1, cfg.head_dim)
        # Append counts on the device and their host staging, for batches in which more sequences may update at a token
        # than a launch can list: a small ring of pinned buffers, each guarded by an event recorded behind its copy, so
        # that a later step never overwrites a buffer the copy engine still reads
        self._n_append = torch.full((batch,), -1, device=dev, dtype=torch.int32) if _memory is None or batch > _lib.UPDATE_LIST_MAX else None
        self._n_append_pinned = None
        self._n_append_slot = 0
        self._alloc_workspace(clear=_memory is None)

    def _alloc_workspace(self, clear: bool = True):
        lib = _lib.load()
        self._max_rows_bound = self._memory.capacity + self.ring_capacity
        self._ws_bytes = lib.kvm_decode_workspace_bytes(C.byref(self._params.c), self.batch, self._max_rows_bound)
        self._ws = torch.empty(self._ws_bytes, device=self.device, dtype=torch.uint8)
        if clear:  # the counter region at the head of the workspace must start at zero; the kernels leave it zero
            self._ws[:4 * (self.kv_rows + self.batch + 1)].zero_()
        # the kept argument block of kvm_decode_step_call; between tokens only input addresses and launch flags change
        call = self._call = _lib.KvmDecodeCall()
        call.layer, call.batch = C.addressof(self._params.c), self.batch
        call.cache = _CCache(self._memory.c(), self._ring_k.data_ptr(), self._ring_v.data_ptr(), self._ring_gate.data_ptr(),
                             self._total_len.data_ptr(), self._state_len.data_ptr())
        call.n_append_dev = _ptr(self._n_append)
        call.total_len_host, call.state_len_host = self._total_len_h.ctypes.data, self._state_len_h.ctypes.data
        call.out, call.workspace, call.workspace_bytes = self._out.data_ptr(), self._ws.data_ptr(), self._ws_bytes
        self._call_args = (C.addressof(call), call.q, call.k, call.v, call.gate)
        self._known = (self.changes, self._memory.changes)  # what the block was filled in from

    def _renew(self):
        """The argument block anew: an array it names has been replaced since (a batch put in another order, say).  The
        schedule is walked for the next token."""
        self._total_len_h, self._state_len_h = (np.ascontiguousarray(t, dtype=np.int64) for t in (self._total_len_h, self._state_len_h))
        self._alloc_workspace()
        self._quiet = 0

    # -- construction ---------------------------------------------------------------------------
    def load_sequence(self, b: int, *, k_sum, v_sum, vlen, window_k, window_v, window_gate, total_len: int,
                      k_attn=None, v_attn=None):
        """Install the state of sequence ``b``: memory rows [Hkv,S,D] (+vlen [Hkv,S]) and the window
        tokens [Hkv,R,D] which are the last R tokens of a sequence of ``total_len`` tokens."""
        cfg = self.cfg
        Hkv, S = k_sum.shape[0], k_sum.shape[1]
        R = window_k.shape[1]
        if S > self.memory.capacity:
            self._reserve(S)
        rows = slice(b * Hkv, (b + 1) * Hkv)
        self.memory.k_sum[rows, :S].copy_(k_sum)
        self.memory.v_sum[rows, :S].copy_(v_sum)
        self.memory.vlen[rows, :S].copy_(vlen.reshape(Hkv, S).float())
        if k_attn is not None:
            self.memory.k_attn[rows, :S].copy_(k_attn)
            self.memory.v_attn[rows, :S].copy_(v_attn)
        begin = total_len - R
        if begin != bswa_begin_for_total_len(total_len, cfg.chunk_len, cfg.n_bswa_chunks):
            raise AssertionError("window tensors do not match the block sliding window of this length")
        slots = (torch.arange(begin, total_len, device=self.device) % self.ring_capacity)
        self.ring_k[rows].index_copy_(1, slots, window_k.to(self.device, torch.bfloat16))
        self.ring_v[rows].index_copy_(1, slots, window_v.to(self.device, torch.bfloat16))
        self.ring_gate[rows].index_copy_(1, slots, window_gate.reshape(Hkv, R).to(self.device, torch.bfloat16))
        self.total_len_h[b] = total_len
        self.state_len_h[b] = S
        self._quiet = 0

    def commit_lengths(self, refresh_attention_view: bool = False):
        """Upload the host-side lengths after ``load_sequence`` calls; optionally rebuild
        ``k_attn`` / ``v_attn`` from the carried sums (when those were not supplied)."""
        self._quiet = 0
        self.total_len.copy_(torch.from_numpy(self.total_len_h.astype(np.int32)))
        self.state_len.copy_(torch.from_numpy(self.state_len_h.astype(np.int32)))
        if refresh_attention_view:
            rc = _lib.load().kvm_memory_refresh(C.byref(self.params.c), self.batch, self.memory.c(),
                                                self.state_len.data_ptr(), _stream_ptr(self.device))
            _lib.check(rc)

    def _reserve(self, required: int):
        if required <= self.memory.capacity:
            return
        new_cap = max(required, int(self.memory.capacity * 1.5) + self.cfg.chunk_len)
        self.memory = self.memory.grown(new_cap)
        self._alloc_workspace()

    # -- schedule -------------------------------------------------------------------------------
    def _plan_step(self):
        """Host bookkeeping of one token: which sequences run a memory update and how many rows it
        appends (reference: model/kvm_mixer.py:617-669).  Returns (n_append array or None, max_rows).
        Between block boundaries of any sequence nothing but the lengths moves: every sequence has one more token in its
        window.  The walk over the batch is skipped for those tokens (``_quiet`` of them are left)."""
        if self._quiet > 0:
            self._quiet -= 1
            self._total_len_h += 1
            self._max_rows += 1
            return None, self._max_rows
        cfg = self.cfg
        Cn, W = cfg.chunk_len, cfg.n_bswa_chunks
        tl, sl = self._total_len_h, self._state_len_h
        cross = (tl % Cn == 0) & (tl // Cn > W)
        n_app = None
        if cross.any():
            n_app = self._plan_updates(np.nonzero(cross)[0])
        direct = (tl < Cn) & (sl == tl)
        sl[direct] += 1
        tl += 1
        begin = np.maximum(0, ((tl + Cn - 1) // Cn) * Cn - W * Cn)
        rows = np.where(begin > 0, sl, 0) + (tl - begin)
        self._max_rows = int(rows.max())
        self._quiet = 0 if tl.min() < Cn else int((-tl % Cn).min())
        return n_app, self._max_rows

    def _plan_updates(self, seqs):
        """The memory updates of the given sequences, which stand at a block boundary: the rows each appends, [batch]
        int32 with -1 for all others; their host lengths grow."""
        cfg = self.cfg
        Cn, W = cfg.chunk_len, cfg.n_bswa_chunks
        n_app = np.full(self.batch, -1, dtype=np.int32)
        for b in seqs:
            cov = int(self.total_len_h[b]) - W * Cn   # coverage before this step
            cur = int(self.state_len_h[b])
            desired = int(self.desired_state_len(W * Cn + cov, cov + Cn, cur))
            na = min(max(desired - cur, 0), Cn)
            if cur + na <= min(cfg.sink_len, cur + na) and na < Cn:
                raise AssertionError("KVM state update requires at least one non-sink slot before merging.")
            n_app[b] = na
            self.state_len_h[b] = cur + na
        self.update_count += len(seqs)
        return n_app

    # -- one token ------------------------------------------------------------------------------
    def step(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, gate: torch.Tensor, *,
             want_route: bool = False) -> torch.Tensor:
        """One decode token for every sequence: q [B,Hq,1,D], k/v [B,Hkv,1,D], gate [B,Hkv,1,1].
        Returns [B,1,Hq*D] (a buffer owned by the cache, overwritten by the next step)."""
        if q.shape != self._q_shape or k.shape != self._kv_shape:
            raise ValueError(f"decode expects one token per sequence, got q {tuple(q.shape)} k {tuple(k.shape)}")
        n_app = self._begin_step()
        any_update = n_app is not None
        call = self._call
        addr, cq, ck, cv, cg = self._call_args
        q, k = _fill_tensor4(cq, q, "q"), _fill_tensor4(ck, k, "k")
        v, gate = _fill_tensor4(cv, v, "v"), _fill_tensor4(cg, gate, "gate")
        call.max_rows = min(self._max_rows, self._max_rows_bound)
        if any_update:
            call.any_update, call.n_append_host = 1, n_app.ctypes.data
            if want_route:
                self.route = torch.zeros(self.kv_rows, self.cfg.chunk_len, device=self.device, dtype=torch.int32)
                call.route_dev = self.route.data_ptr()
        rc = _lib.load().kvm_decode_step_call(addr, _stream_ptr(self.device))
        if any_update:
            call.any_update, call.n_append_host, call.route_dev = 0, None, None
        if rc:
            _lib.check(rc)
        return self._out

    def _begin_step(self):
        """The host side of a token ahead of its launch: schedule, room for the rows it appends.  Returns the append counts
        (None: no sequence updates its memory)."""
        if self._known != (self.changes, self._memory.changes):
            self._renew()
        n_app, _ = self._plan_step()
        self._last_any_update, self._last_n_append = n_app is not None, n_app
        if n_app is not None or self._quiet == 0:
            need = int(self._state_len_h.max())
            if need > self._memory.capacity:
                self._reserve(need)
            if n_app is not None and int((n_app >= 0).sum()) > _lib.UPDATE_LIST_MAX:
                self._upload_n_append(n_app)
        return n_app

    def _upload_n_append(self, n_app):
        """The step's append counts to the device (for steps at which more sequences update than a launch can list)."""
        if self._n_append_pinned is None:
            self._n_append_pinned = [torch.full((self.batch,), -1, dtype=torch.int32).pin_memory() for _ in range(4)]
            self._n_append_events = [None] * 4
        slot = self._n_append_slot
        self._n_append_slot = (slot + 1) % len(self._n_append_pinned)
        if self._n_append_events[slot] is not None:
            self._n_append_events[slot].synchronize()
        self._n_append_pinned[slot].copy_(torch.from_numpy(n_app))
        self._n_append.copy_(self._n_append_pinned[slot], non_blocking=True)
        ev = self._n_append_events[slot] or torch.cuda.Event()
        ev.record(torch.cuda.current_stream(self.device))
        self._n_append_events[slot] = ev

    def run(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, gate: torch.Tensor) -> torch.Tensor:
        """``n`` consecutive decode tokens with inputs already on the device (teacher-forced / synthetic
        decoding): q [n,B,Hq,1,D], k/v [n,B,Hkv,1,D], gate [n,B,Hkv,1,1], contiguous.  Returns [n,B,Hq*D].
        Tokens of one block see the same memory, so a sequence's keys and values are read once for a span of tokens
        (up to its next block boundary, and as many as a launch has columns for); the sequences advance independently."""
        cfg, B = self.cfg, self.batch
        n = q.size(0)
        if q.shape != (n, *self._q_shape) or k.shape != (n, *self._kv_shape):
            raise ValueError(f"run expects [n,B,H,1,D] inputs, got q {tuple(q.shape)} k {tuple(k.shape)}")
        q, k, v, gate = (t.to(torch.bfloat16).contiguous() for t in (q, k, v, gate))
        out = torch.empty(n, B, cfg.n_q_heads * cfg.head_dim, device=self.device, dtype=torch.bfloat16)
        if B > _lib.SPAN_BATCH_MAX:
            for i in range(n):
                out[i] = self.step(q[i], k[i], v[i], gate[i]).view(B, -1)
            return out
        lib, stream = _lib.load(), _stream_ptr(self.device)
        Cn, WC = cfg.chunk_len, self.ring_capacity
        span = max(1, _lib.SPAN_COLUMNS // (cfg.n_q_heads // cfg.n_kv_heads))  # (more query heads: refused by the library)
        if self._known != (self.changes, self._memory.changes):
            self._renew()
        tl, sl = self._total_len_h, self._state_len_h
        self._quiet = 0
        piece = 128  # (a token's place inside a piece fits a byte)
        for lo in range(0, n, piece):
            m = min(piece, n - lo)
            done = np.zeros(B, dtype=np.int64)
            while True:
                at = tl % Cn
                count = np.minimum(np.minimum(m - done, Cn - at), span)
                if not count.any():
                    break
                cross = np.nonzero((count > 0) & (at == 0) & (tl > WC))[0]
                if cross.size > _lib.UPDATE_LIST_MAX:  # the others wait for the next launch
                    count[cross[_lib.UPDATE_LIST_MAX:]] = 0
                    cross = cross[:_lib.UPDATE_LIST_MAX]
                n_app = self._plan_updates(cross) if cross.size else None
                direct = (tl < Cn) & (sl == tl)
                sl[direct] += count[direct]
                tl += count
                need = int(sl.max())
                if need > self.memory.capacity:
                    self._reserve(need)
                call = self._call
                addr, cq, ck, cv, cg = self._call_args
                for dst, t, name in ((cq, q, "q"), (ck, k, "k"), (cv, v, "v"), (cg, gate, "gate")):
                    _fill_tensor4(dst, t[lo], name)
                call.out = out[lo].data_ptr()
                if n_app is not None:
                    call.any_update, call.n_append_host = 1, n_app.ctypes.data
                first8, count8 = done.astype(np.uint8), count.astype(np.uint8)
                rc = lib.kvm_decode_span(addr, first8.ctypes.data, count8.ctypes.data, q.stride(0), k.stride(0), gate.stride(0),
                                         out.stride(0), stream)
                call.out, call.any_update, call.n_append_host = self.out.data_ptr(), 0, None
                _lib.check(rc)
                done += count
        return out

    def check_status(self) -> None:
        """Synchronise and raise if a decode kernel reported a device-side timeout since the last check."""
        rc = _lib.load().kvm_decode_status(C.byref(self.params.c), self.batch, self._ws.data_ptr(), _stream_ptr(self.device))
        _lib.check(rc)

    # -- inspection -----------------------------------------------------------------------------
    def logical_state_dict(self, b: int | None = None) -> dict[str, Any]:
        """The reference's eager cache entries (model/kvm_mixer.py:501-525).  For a batch with uniform
        lengths ``b`` may be omitted; otherwise the entries of sequence ``b`` are returned with a
        leading batch dimension of 1."""
        cfg = self.cfg
        if b is None:
            if len(set(self.total_len_h.tolist())) != 1 or len(set(self.state_len_h.tolist())) != 1:
                raise ValueError("ragged cache: pass the sequence index")
            seqs = list(range(self.batch))
            b0 = 0
        else:
            seqs = [b]
            b0 = b
        Hkv, D = cfg.n_kv_heads, cfg.head_dim
        total = int(self.total_len_h[b0])
        S = int(self.state_len_h[b0])
        begin = bswa_begin_for_total_len(total, cfg.chunk_len, cfg.n_bswa_chunks)
        coverage = max(min(total, cfg.chunk_len), begin)
        rows = torch.cat([torch.arange(s * Hkv, (s + 1) * Hkv) for s in seqs]).to(self.device)
        slots = torch.arange(begin, total, device=self.device) % self.ring_capacity
        nb = len(seqs)
        return {
            "kvm_s_k": self.memory.k_sum[rows, :S].reshape(nb, Hkv, S, D),
            "kvm_s_v": self.memory.v_sum[rows, :S].reshape(nb, Hkv, S, D),
            "kvm_s_vlen": self.memory.vlen[rows, :S].reshape(nb, Hkv, S, 1),
            "kvm_state_coverage_len": coverage,
            "kvm_bswa_begin": begin,
            "kvm_bswa_k": self.ring_k[rows][:, slots].reshape(nb, Hkv, total - begin, D),
            "kvm_bswa_v": self.ring_v[rows][:, slots].reshape(nb, Hkv, total - begin, D),
            "kvm_bswa_merge_gate": self.ring_gate[rows][:, slots].reshape(nb, Hkv, total - begin, 1),
        }

    def persistent_metadata(self) -> dict[str, Any]:
        return {
            "total_len": self.total_len_h.tolist(),
            "active_state_len": self.state_len_h.tolist(),
            "state_capacity": self.memory.capacity,
            "recent_capacity": self.ring_capacity,
            "update_count": self.update_count,
            "cache_representation": self.cache_representation,
        }


def decode_cache_from_prefill(params: LayerParams, res: PrefillResult, k: torch.Tensor, v: torch.Tensor,
                              gate: torch.Tensor, desired_state_len, owner=None, extra_capacity: int | None = None, *,
                              adopt_memory: bool = False) -> KvmDecodeCache:
    """Build the decode cache of a batch right after its prefill (uniform lengths), with one launch.  ``adopt_memory``: the
    cache goes on in the prefill's own memory buffers instead of a copy (the result's memory then changes with it)."""
    cfg = params.cfg
    B, Hkv, T, D = k.shape
    S = res.plan.final_state_len
    extra = cfg.chunk_len if extra_capacity is None else extra_capacity
    cache = KvmDecodeCache(params, B, S + extra, desired_state_len, owner, _memory=res.memory if adopt_memory else None)
    k, v, gate = _aligned_rows(k), _aligned_rows(v), _as_bf16_view(gate.reshape(B, Hkv, T, 1))
    rc = _lib.load().kvm_decode_cache_fill(C.byref(params.c), B, T, _tensor4(k, "k"), _tensor4(v, "v"), _tensor4(gate, "gate"),
                                           res.memory.c(), S, cache._call.cache, cache._ws.data_ptr(), _stream_ptr(cache.device))
    _lib.check(rc)
    cache.total_len_h[:] = T
    cache.state_len_h[:] = S
    return cache


def prompt_forward(params: LayerParams, pro: PrologueParams, q_lin: torch.Tensor, k_lin: torch.Tensor, v_lin: torch.Tensor,
                   gate_lin: torch.Tensor | None, position_embeddings, plan: PrefillPlan, *, prev=None, value_residual=None, v_last=None,
                   desired_state_len=None, owner=None, want_cache: bool = True) -> tuple[KvmDecodeCache | None, torch.Tensor]:
    """A prompt from the projection outputs to the input of ``c_proj`` in one library call: ``prologue_forward``, prefill and
    the decode cache behind it (which lives in the prefill's memory).  Returns (cache or None, [B,T,Hq*D])."""
    lib = _lib.load()
    cfg = params.cfg
    B, T, _ = q_lin.shape
    dev = q_lin.device
    if plan.seq_len != T:
        raise ValueError("plan was built for another sequence length")
    S = plan.final_state_len
    memory = MemoryBuffers(B * cfg.n_kv_heads, S + cfg.chunk_len, cfg.head_dim, dev, zero=False)
    out = torch.empty(B, T, cfg.n_q_heads * cfg.head_dim, device=dev, dtype=torch.bfloat16)
    call = _lib.KvmPromptCall()
    call.layer, call.batch, call.n_updates, call.seq_len = C.addressof(params.c), B, plan.n_updates, T
    call.total_version_rows = plan.total_version_rows
    call.workspace_bytes = lib.kvm_prompt_workspace_bytes(C.byref(params.c), B, T, plan.n_updates, plan.total_version_rows)
    ws = torch.empty(call.workspace_bytes, device=dev, dtype=torch.uint8)
    table = plan.to_array()
    call.plan_host, call.workspace, call.out, call.memory = table.ctypes.data, ws.data_ptr(), out.data_ptr(), memory.c()
    arg, keep = _prologue_arg(params, pro, q_lin, k_lin, v_lin, gate_lin, position_embeddings, prev, value_residual, v_last)
    call.prologue = arg
    cache = None
    if want_cache:
        cache = KvmDecodeCache(params, B, S + cfg.chunk_len, desired_state_len, owner, _memory=memory)
        call.cache, call.decode_workspace = cache._call.cache, cache._ws.data_ptr()
        cache.total_len_h[:] = T
        cache.state_len_h[:] = S
    rc = lib.kvm_mixer_prompt(C.addressof(call), _stream_ptr(dev))
    if rc:
        _lib.check(rc)
    del keep  # (enqueued on the current stream: torch's allocator keeps the blocks until the kernels have run)
    return cache, out


class TokenCall:
    """The kept argument block of ``kvm_mixer_token`` for one decode cache, which holds it (and is not held by it: a cache that
    is let go gives its memory back at once): between tokens only a few addresses change."""

    def __init__(self, cache: KvmDecodeCache, params: LayerParams, pro: PrologueParams):
        self.params, self.pro, self.decode_src = params, pro, cache._call
        c = self.c = _lib.KvmTokenCall()
        c.decode = cache._call
        c.scratch_bytes = _lib.load().kvm_token_scratch_bytes(C.byref(params.c), cache.batch)
        self._scratch = torch.empty(c.scratch_bytes, device=cache.device, dtype=torch.uint8)
        c.scratch = self._scratch.data_ptr()
        p = c.prologue
        if pro.shift_q is not None:
            p.shift_q, p.shift_k, p.shift_v = pro.shift_ptrs
        if pro.ln is not None:
            p.ln_q_w, p.ln_q_b, p.ln_k_w, p.ln_k_b = pro.ln_ptrs
            p.ln_qk_eps, p.ln_bf16 = pro.ln_eps, pro.ln_bf16
        self._views = (C.addressof(c), c.decode, p, c.weights, c.weight_rows)

    @staticmethod
    def of(cache: KvmDecodeCache, params: LayerParams, pro: PrologueParams) -> "TokenCall":
        t = cache._token
        if t is None or t.params is not params or t.pro is not pro:
            t = cache._token = TokenCall(cache, params, pro)
        return t

    def run(self, cache: KvmDecodeCache, x, weights, v_gate2, c_proj, gated, residual, position_embeddings, prev):
        """One token of ``cache``.  x [B,1,hidden]; returns (y [B,1,out], projections [B,1,..], last values behind the residual
        or None)."""
        cfg = cache.cfg
        addr, decode, p, w, rows = self._views
        c, B, dev = self.c, cache.batch, cache.device
        keep = []
        x = _aligned(x)
        cos = sin = None
        if position_embeddings is not None:
            cos, sin, own = rotary_tables_arg(position_embeddings, B, 1, cfg.head_dim, x.device)
            if (cos.data_ptr() | sin.data_ptr()) % 16:
                raise ValueError("rotary tables must be 16-byte aligned")
            p.cos, p.sin, p.rope_stride_b = cos.data_ptr(), sin.data_ptr(), cfg.head_dim if own else 0
        else:
            p.cos, p.sin = None, None
        v_last = None
        if residual is not None:
            v_first, v_gate0 = residual
            v_first = _first_values(v_first, B, 1, cfg.n_kv_heads * cfg.head_dim, x.device)
            v_gate0 = _aligned(v_gate0.to(x.device))
            keep += [v_first, v_gate0]
            v_last = torch.empty(B, 1, cfg.n_kv_heads * cfg.head_dim, device=x.device, dtype=torch.bfloat16)
            p.v_first, p.v_gate0, p.v_last = v_first.data_ptr(), v_gate0.data_ptr(), v_last.data_ptr()
        if self.pro.shift_q is not None:
            if any(t is None for t in prev):
                p.prev_q, p.prev_k, p.prev_v = None, None, None
            else:
                dk = cfg.n_kv_heads * cfg.head_dim
                pv = _prev_rows(prev, B, x.device, (cfg.n_q_heads * cfg.head_dim, dk, dk))
                keep.append(pv)
                p.prev_q, p.prev_k, p.prev_v = pv[0].data_ptr(), pv[1].data_ptr(), pv[2].data_ptr()
                if B > 1:
                    p.prev_q_stride_b, p.prev_k_stride_b, p.prev_v_stride_b = pv[0].stride(0), pv[1].stride(0), pv[2].stride(0)
        cols = 0
        for i, t in enumerate(weights):
            n = t.shape[0]
            w[i], rows[i] = t.data_ptr(), n
            cols += n
        cols = (cols + 7) // 8 * 8
        lin = torch.empty(B, 1, cols, device=x.device, dtype=torch.bfloat16)
        hidden, out_features = x.shape[2], c_proj.shape[0]
        y = torch.empty(B, 1, out_features, device=x.device, dtype=torch.bfloat16)
        c.x, c.x_stride, c.hidden, c.n_weights, c.gated = x.data_ptr(), hidden, hidden, len(weights), gated
        c.v_gate2 = None if v_gate2 is None else v_gate2.data_ptr()
        c.c_proj, c.out_features = c_proj.data_ptr(), out_features
        c.lin, c.lin_stride, c.y = lin.data_ptr(), cols, y.data_ptr()
        n_app = cache._begin_step()
        if self.decode_src is not cache._call:  # (the memory has been moved to larger arrays)
            c.decode = self.decode_src = cache._call
        decode.max_rows = min(cache._max_rows, cache._max_rows_bound)
        if n_app is not None:
            decode.any_update, decode.n_append_host = 1, n_app.ctypes.data
        rc = _lib.load().kvm_mixer_token(addr, _stream_ptr(dev))
        if n_app is not None:
            decode.any_update, decode.n_append_host = 0, None
        if rc:
            _lib.check(rc)
        return y, lin, v_last
