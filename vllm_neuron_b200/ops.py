"""Tensor-level wrappers over the C ABI: validate, allocate the results, call on the current CUDA stream.

Torch is plumbing here (device memory + streams); every op below runs one of the hand-written
sm_100a kernels in libb200_paged.so.  Nothing in this file computes on the host.
"""
from __future__ import annotations

import os

import torch

from . import _cabi
from ._cabi import (ACT_GELU_TANH, ACT_NONE, ACT_RELU2, ACT_SILU, ACT_SWISH_CLAMPED, BF16, F32, FP8_E4M3, INT8, ROUTE_SIGMOID,
                    ROUTE_SOFTMAX_RENORM, ROUTE_SOFTMAX_TOP, check)

_QDT = {None: BF16, "bf16": BF16, "fp8": FP8_E4M3, "int8": INT8}
_TORCH_Q = {FP8_E4M3: torch.float8_e4m3fn, INT8: torch.int8}
INT8_WO = 4  # GEMM ab_dtype only: bf16 activations x int8 weights
_DTN = {BF16: "bf16", FP8_E4M3: "fp8", INT8: "int8", INT8_WO: "int8wo"}


def _stream():
    # the raw handle of the current stream: torch.cuda.current_stream() builds a Stream object on every launch (3 us of host time)
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


# ------------------------------------------------------------------ per-launch device timing (bench.py roofline leg)
_PROF: list | None = None


class kernel_timer:
    """with ops.kernel_timer() as t: ...eager calls...; t.summary() -> {name: (count, mean_ms)}.
    CUDA events are recorded on the launching stream right around each C-ABI call (not usable under graph capture)."""

    def __enter__(self):
        global _PROF
        self.records = _PROF = []
        return self

    def __exit__(self, *exc):
        global _PROF
        _PROF = None
        return False

    def summary(self):
        torch.cuda.synchronize()
        acc: dict[str, list] = {}
        for name, e0, e1 in self.records:
            acc.setdefault(name, []).append(e0.elapsed_time(e1))
        return {k: (len(v), sum(v) / len(v)) for k, v in acc.items()}


class _Timed:
    __slots__ = ("name", "to", "e0")

    def __init__(self, name, to):
        self.name, self.to = name, to  # the timer may be closed by another thread before the launch is over

    def __enter__(self):
        self.e0 = torch.cuda.Event(enable_timing=True)
        self.e0.record()

    def __exit__(self, *exc):
        e1 = torch.cuda.Event(enable_timing=True)
        e1.record()
        self.to.append((self.name, self.e0, e1))
        return False


class _Untimed:
    def __enter__(self):
        pass

    def __exit__(self, *exc):
        return False


_UNTIMED = _Untimed()


def _k(name, *sizes):
    """Context of one launch: timed under its name (a format of the sizes) while a kernel_timer is open."""
    to = _PROF
    return _UNTIMED if to is None else _Timed(name.format(*sizes), to)


def _lib():
    """The library's functions on tensors and plain numbers (csrc/bind.cpp): the stream may be left out, a CPU tensor raises."""
    return _bind or _load_bind()


_bind = None


def _load_bind():
    global _bind
    _bind = _cabi.native()
    return _bind


def _new(like, dtype, *shape):
    """Uninitialised tensor on like's device; dtype None = like's."""
    return _lib().new(like, dtype, *shape)


def _ptr(t):
    return 0 if t is None else t.data_ptr()


def _cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise _cabi.B200Error("b200 ops need CUDA tensors (no CPU fallback)")


def device_check(device: int = 0):
    check(_cabi.load().b200_device_check(device), "b200_device_check")


def set_pdl(enabled: bool) -> bool:
    """Programmatic dependent launch on/off for every kernel of the library; returns the previous setting."""
    return bool(_cabi.load().b200_set_pdl(1 if enabled else 0))


def launch_count() -> int:
    """Kernel launches issued through libb200_paged.so by this process so far."""
    return int(_cabi.load().b200_launch_count())


# ------------------------------------------------------------------ index construction
def build_decode_meta(block_table, row_ids, num_tokens, slot_mapping, positions, ctx_lens, block_size: int):
    """block_table int32 [rows, max_blocks]; row_ids int32 [B] or None; num_tokens int32 [rows];
    outputs: slot_mapping int64 [B] (or [B, k]: k consecutive slots per row for speculation, RUNNER:825-830),
    positions int64 [B], ctx_lens int32 [B]."""
    assert block_table.dtype == torch.int32 and num_tokens.dtype == torch.int32
    assert slot_mapping.dtype == torch.int64 and positions.dtype == torch.int64 and ctx_lens.dtype == torch.int32
    b = positions.numel()
    num_spec = 1 if slot_mapping.dim() == 1 else slot_mapping.shape[1]
    assert slot_mapping.is_contiguous() and slot_mapping.numel() == b * num_spec
    with _k("build_decode_meta"):
        check(
            _lib().b200_build_decode_meta(
                block_table, block_table.stride(0), row_ids, num_tokens, slot_mapping,
                positions, ctx_lens, b, block_table.shape[1], block_size, num_spec),
            "b200_build_decode_meta",
        )


def build_prefill_meta(block_table_row, prompt_len: int, num_computed: int, slot_mapping, positions, block_size: int):
    assert block_table_row.dtype == torch.int32 and slot_mapping.dtype == torch.int64 and positions.dtype == torch.int64
    check(
        _lib().b200_build_prefill_meta(
            block_table_row, prompt_len, num_computed, slot_mapping, positions,
            slot_mapping.numel(), block_size),
        "b200_build_prefill_meta",
    )


def remask_spec_output(accepted, next_pos, positions):
    """LOADER:308-334: accepted int64 [B, T] 0-padded -> -1 past clamp(next_pos - positions, 0, T) tokens per row."""
    b, t = accepted.shape
    assert accepted.dtype == next_pos.dtype == positions.dtype == torch.int64 and accepted.is_contiguous()
    out = torch.empty_like(accepted)
    check(_lib().b200_remask_spec_output(accepted, next_pos, positions, out, b, t),
          "b200_remask_spec_output")
    return out


def block_table_scatter(block_table, updates):
    """updates int32 [n, 3] = (row, col, block_id) on the device."""
    assert block_table.dtype == torch.int32 and updates.dtype == torch.int32 and updates.is_contiguous()
    n = updates.shape[0]
    check(
        _lib().b200_block_table_scatter(
            block_table, block_table.stride(0), updates, n, block_table.shape[0], block_table.shape[1]),
        "b200_block_table_scatter",
    )


def advance_decode(sampled, tokens_io, num_tokens, row_ids):
    check(
        _lib().b200_advance_decode(
            sampled, tokens_io, num_tokens, row_ids, sampled.numel()),
        "b200_advance_decode",
    )


# ------------------------------------------------------------------ KV cache
def kv_write(k, v, k_pool, v_pool, slot_mapping):
    """k, v [T, Hkv, D] bf16 (last two dims contiguous); pools [num_blocks, Hkv, bs, D]."""
    t, hkv, d = k.shape
    nb, hkv2, bs, d2 = k_pool.shape
    assert (hkv, d) == (hkv2, d2) and k.stride(2) == 1 and k.stride(1) == d and v.stride(1) == d
    assert k_pool.is_contiguous() and v_pool.is_contiguous() and slot_mapping.dtype == torch.int64
    check(
        _lib().b200_kv_write(
            k, v, k.stride(0), v.stride(0), k_pool, v_pool, slot_mapping,
            t, hkv, d, bs, nb),
        "b200_kv_write",
    )


def rope_kv_write(qkv, positions, cos, sin, k_pool, v_pool, slot_mapping, num_q_heads: int):
    """qkv [T, (Hq+2Hkv)*D] bf16 contiguous; q is rotated in place, roped k and v go to the pools."""
    nb, hkv, bs, d = k_pool.shape
    t = qkv.shape[0]
    assert qkv.is_contiguous() and qkv.shape[1] == (num_q_heads + 2 * hkv) * d and qkv.dtype == torch.bfloat16
    assert cos.dtype == torch.float32 and cos.shape[1] == d // 2 and cos.is_contiguous() and sin.is_contiguous()
    assert positions.dtype == torch.int64 and slot_mapping.dtype == torch.int64
    with _k("rope_kv_write"):
        check(
            _lib().b200_rope_kv_write(
                qkv, positions, cos, sin, cos.shape[0], k_pool, v_pool,
                slot_mapping, t, num_q_heads, hkv, d, bs, nb),
            "b200_rope_kv_write",
        )


# ------------------------------------------------------------------ paged attention
def paged_attn_decode_workspace_bytes(b, hq, hkv, d, max_blocks, min_quota=0) -> int:
    return int(_lib().b200_paged_attn_decode_workspace_bytes(b, hq, hkv, d, max_blocks, min_quota))


def paged_attn_decode(q, k_pool, v_pool, block_table, ctx_lens, scale, out=None, workspace=None, row_ids=None,
                      max_blocks=None, min_quota=0, quant=None):
    """q [B, Hq, D] bf16 (token stride arbitrary); block_table int32 [rows, max_blocks]; ctx_lens int32 [B].
    quant None -> bf16 out [B, Hq, D]; "fp8"/"int8" -> (q [B, Hq*D], scale [B]) quantised per token in the merge kernel."""
    b, hq, d = q.shape
    nb, hkv, bs, d2 = k_pool.shape
    assert d == d2 and q.stride(2) == 1 and q.stride(1) == d and q.dtype == torch.bfloat16
    assert block_table.dtype == torch.int32 and ctx_lens.dtype == torch.int32
    mb = block_table.shape[1] if max_blocks is None else min(max_blocks, block_table.shape[1])
    qd = _QDT[quant]
    oq = osc = None
    if qd == BF16:
        if out is None:
            out = _new(q, q.dtype, b, hq, d)
        assert out.is_contiguous()
    else:
        oq = _new(q, _TORCH_Q[qd], b, hq * d)
        osc = _new(q, torch.float32, b)
    if workspace is None:
        workspace = torch.empty(paged_attn_decode_workspace_bytes(b, hq, hkv, d, mb, min_quota), dtype=torch.uint8, device=q.device)
    with _k("paged_attn_decode"):
        check(
            _lib().b200_paged_attn_decode(
                q, q.stride(0), k_pool, v_pool, nb, block_table, block_table.stride(0),
                row_ids, ctx_lens, out, oq, osc, qd, workspace,
                workspace.numel() * workspace.element_size(), b, hq, hkv, d, bs, mb, min_quota, float(scale)),
            "b200_paged_attn_decode",
        )
    return out if qd == BF16 else (oq, osc)


def paged_attn_prefill(q, k_pool, v_pool, block_table_row, computed_len: int, scale, out=None):
    """q [S_new, Hq, D] bf16; one sequence; K/V of all computed_len + S_new tokens already in the pools."""
    s_new, hq, d = q.shape
    nb, hkv, bs, _ = k_pool.shape
    assert q.stride(2) == 1 and q.stride(1) == d and block_table_row.dtype == torch.int32
    if out is None:
        out = _new(q, q.dtype, s_new, hq, d)
    with _k("paged_attn_prefill"):
        check(
            _lib().b200_paged_attn_prefill(
                q, q.stride(0), k_pool, v_pool, nb, block_table_row, out, s_new,
                computed_len, hq, hkv, d, bs, float(scale)),
            "b200_paged_attn_prefill",
        )
    return out


# ------------------------------------------------------------------ GEMM
def _ab_dtype(t):
    if t.dtype == torch.bfloat16:
        return BF16
    if t.dtype == torch.float8_e4m3fn:
        return FP8_E4M3
    if t.dtype == torch.int8:
        return INT8
    raise _cabi.B200Error(f"unsupported GEMM operand dtype {t.dtype}")


def _gemm_dtype(a, w):
    """ab_dtype code of a GEMM: both operands alike, or bf16 activations x int8 weights (weight-only)."""
    if a.dtype == torch.bfloat16 and w.dtype == torch.int8:
        return INT8_WO
    if a.dtype != w.dtype:
        raise _cabi.B200Error(f"GEMM operand dtypes {a.dtype} x {w.dtype} not supported")
    return _ab_dtype(a)


def gemm_decode_plan(m, n, k, ab_dtype, split_k=0, silu_mul=False, has_residual=False) -> dict:
    """The decode schedule the library picks for this shape on the current device (for benches / DESIGN notes)."""
    import ctypes

    out = (ctypes.c_int * 6)()
    check(_cabi.load().b200_gemm_decode_plan(m, n, k, ab_dtype, split_k, int(silu_mul), int(has_residual), out),
          "b200_gemm_decode_plan")
    return dict(zip(("split", "ctas_per_sm", "w_stages", "a_stages", "cap_ctas", "smem"), list(out)))


def gemm_pair_plan(m, n, k, ab_dtype, silu_mul=False, has_residual=False) -> dict:
    """What the CTA pairs take of a GEMM that names no split: tokens of a tile (0: another schedule runs), units of two token tiles, all units."""
    import ctypes

    out = (ctypes.c_int * 4)()
    check(_cabi.load().b200_gemm_pair_plan(m, n, k, ab_dtype, int(silu_mul), int(has_residual), out), "b200_gemm_pair_plan")
    return dict(zip(("tokens", "wide", "units", "stages"), list(out)))


def gemm_workspace_bytes(m, n, k, ab_dtype, split_k=0) -> int:
    return int(_lib().b200_gemm_workspace_bytes(m, n, k, ab_dtype, split_k))


def gemm_workspace(m, n, k, ab_dtype, device, split_k=0):
    """Zero-filled workspace (stream-K fix-up counters at its head must start at zero; every call leaves them zeroed).
    The decode schedule (M <= 128) needs none: returns None."""
    nbytes = gemm_workspace_bytes(m, n, k, ab_dtype, split_k)
    return torch.zeros(nbytes, dtype=torch.uint8, device=device) if nbytes else None


def gemm(a, w, a_scale=None, w_scale=None, bias=None, residual=None, out=None, out_dtype=torch.bfloat16, split_k=0,
         workspace=None):
    """out[M,N] = (a[M,K] @ w[N,K]^T) * a_scale[m] * w_scale[n] + bias[n] + residual[m,n]."""
    m, k = a.shape
    n, k2 = w.shape
    assert k == k2 and a.is_contiguous() and w.is_contiguous()
    dt = _gemm_dtype(a, w)
    if out is None:
        out = _new(a, out_dtype, m, n)
    assert out.is_contiguous() and out.shape == (m, n)
    odt = F32 if out.dtype == torch.float32 else BF16
    if residual is not None:
        assert residual.dtype == torch.bfloat16 and residual.is_contiguous() and residual.shape == (m, n)
    if workspace is None:
        workspace = gemm_workspace(m, n, k, dt, a.device, split_k)
    with _k("gemm_{}[{}x{}x{}]", _DTN[dt], m, n, k):
        check(
            _lib().b200_gemm(
                a, w, out, a_scale, w_scale, bias, residual, m, n, k, dt, odt,
                split_k, workspace, 0 if workspace is None else workspace.numel() * workspace.element_size()),
            "b200_gemm",
        )
    return out


def gemm_rope_kv_write(a, w, positions, cos, sin, k_pool, v_pool, slot_mapping, num_q_heads: int, a_scale=None,
                       w_scale=None, bias=None, split_k=0, workspace=None):
    """qkv[M, (Hq+2Hkv)*D] = gemm(a, w, ...) with rope_kv_write fused into the GEMM epilogue when the decode schedule
    allows (one launch), else GEMM + rope_kv_write inside the library (two launches); identical bits.  Returns qkv."""
    m, k = a.shape
    n, k2 = w.shape
    nb, hkv, bs, d = k_pool.shape
    assert k == k2 and a.is_contiguous() and w.is_contiguous() and n == (num_q_heads + 2 * hkv) * d
    assert cos.dtype == torch.float32 and cos.shape[1] == d // 2 and cos.is_contiguous() and sin.is_contiguous()
    assert positions.dtype == torch.int64 and slot_mapping.dtype == torch.int64
    dt = _gemm_dtype(a, w)
    out = _new(a, torch.bfloat16, m, n)
    if workspace is None:
        workspace = gemm_workspace(m, n, k, dt, a.device, split_k)
    with _k("gemm_rope_kv_{}[{}x{}x{}]", _DTN[dt], m, n, k):
        check(
            _lib().b200_gemm_rope_kv_write(
                a, w, out, a_scale, w_scale, bias, m, n, k, dt, split_k,
                workspace, 0 if workspace is None else workspace.numel() * workspace.element_size(),
                positions, cos, sin, cos.shape[0], k_pool, v_pool, slot_mapping,
                num_q_heads, hkv, d, bs, nb),
            "b200_gemm_rope_kv_write",
        )
    return out


def interleave_gate_up(w_gu, *others):
    """Row permutation expected by gemm_silu_mul: [gate(I); up(I)] -> groups of 32 rows = 16 gate rows followed by the
    16 up rows of the same channels.  Applied (load time) to the weight and to every per-row companion (scale, bias)."""
    i = w_gu.shape[0] // 2
    assert i % 16 == 0, "intermediate size must be a multiple of 16"
    idx = torch.arange(i, device=w_gu.device).view(-1, 16)
    perm = torch.cat([idx, idx + i], dim=1).reshape(-1)
    res = [w_gu[perm].contiguous()] + [None if o is None else o[perm].contiguous() for o in others]
    return res[0] if not others else tuple(res)


def gemm_silu_mul(a, w_gu_interleaved, a_scale=None, w_scale=None, bias=None, split_k=0, workspace=None):
    """act[M, I] = bf16(silu(bf16(gate)) * bf16(up)) with gate/up = the two halves of a @ w_gu^T (rows interleaved by
    interleave_gate_up); also returns group_amax [M, 2I/32] for quantize_per_token."""
    m, k = a.shape
    n2, k2 = w_gu_interleaved.shape
    assert k == k2 and a.is_contiguous() and w_gu_interleaved.is_contiguous()
    dt = _gemm_dtype(a, w_gu_interleaved)
    act = _new(a, torch.bfloat16, m, n2 // 2)
    assert n2 % 32 == 0
    group_amax = _new(a, torch.float32, m, n2 // 32)
    if workspace is None:
        workspace = gemm_workspace(m, n2, k, dt, a.device, split_k)
    with _k("gemm_silu_mul_{}[{}x{}x{}]", _DTN[dt], m, n2, k):
        check(
            _lib().b200_gemm_silu_mul(
                a, w_gu_interleaved, act, a_scale, w_scale, bias, group_amax,
                m, n2, k, dt, split_k, workspace, 0 if workspace is None else workspace.numel() * workspace.element_size()),
            "b200_gemm_silu_mul",
        )
    return act, group_amax


_UNSUPPORTED = -4  # B200_ERR_UNSUPPORTED


def gemm_silu_mul_quant(a, w_gu_interleaved, a_scale, w_scale, bias, state, quant: str):
    """gate/up GEMM + SiLU*mul + per-token quantisation in ONE launch (b200_gemm_silu_mul_quant): returns (q [M, I], scale [M])
    or None when the shape does not run as one resident wave of one CTA per weight tile (the caller then uses gemm_silu_mul
    + quantize_per_token, which produce the same bits).  `state`: 1040-byte uint8 device tensor, zeroed once."""
    m, k = a.shape
    n2, k2 = w_gu_interleaved.shape
    assert k == k2 and a.is_contiguous() and w_gu_interleaved.is_contiguous() and n2 % 32 == 0 and state.numel() >= 1040
    if m > 128:
        return None
    dt = _gemm_dtype(a, w_gu_interleaved)
    qd = _QDT[quant]
    q = _new(a, _TORCH_Q[qd], m, n2 // 2)
    sc = _new(a, torch.float32, m)
    with _k("gemm_silu_mul_quant_{}[{}x{}x{}]", _DTN[dt], m, n2, k):
        rc = _lib().b200_gemm_silu_mul_quant(a, w_gu_interleaved, q, sc, a_scale, w_scale,
                                                   bias, state, m, n2, k, dt)
    if rc == _UNSUPPORTED:
        return None
    check(rc, "b200_gemm_silu_mul_quant")
    return q, sc


# ------------------------------------------------------------------ glue
def rmsnorm(x, w, eps, quant=None, out_bf16=None, want_bf16=None):
    """Returns bf16 y, or (q, scale) for quant in {"fp8","int8"} (plus y when want_bf16)."""
    t, h = x.shape
    assert x.is_contiguous() and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16
    qd = _QDT[quant]
    if qd == BF16:
        y = out_bf16 if out_bf16 is not None else _new(x, None, t, h)
        with _k("rmsnorm"):
            check(_lib().b200_rmsnorm(x, w, y, 0, 0, t, h, float(eps), qd), "b200_rmsnorm")
        return y
    q = _new(x, _TORCH_Q[qd], t, h)
    s = _new(x, torch.float32, t)
    y = (out_bf16 if out_bf16 is not None else torch.empty_like(x)) if want_bf16 else None
    with _k("rmsnorm_quant"):
        check(_lib().b200_rmsnorm(x, w, y, q, s, t, h, float(eps), qd), "b200_rmsnorm")
    return (q, s, y) if want_bf16 else (q, s)


def silu_mul(gate_up, quant=None):
    t, i2 = gate_up.shape
    i = i2 // 2
    assert gate_up.is_contiguous() and gate_up.dtype == torch.bfloat16
    qd = _QDT[quant]
    if qd == BF16:
        y = _new(gate_up, torch.bfloat16, t, i)
        with _k("silu_mul"):
            check(_lib().b200_silu_mul(gate_up, y, 0, 0, t, i, qd), "b200_silu_mul")
        return y
    q = _new(gate_up, _TORCH_Q[qd], t, i)
    s = _new(gate_up, torch.float32, t)
    with _k("silu_mul_quant"):
        check(_lib().b200_silu_mul(gate_up, 0, q, s, t, i, qd), "b200_silu_mul")
    return q, s


def quantize_per_token(x, quant: str, group_amax=None):
    """x [T, K] bf16 -> (q [T, K], scale [T]).  group_amax [T, n_groups] (from gemm_silu_mul) skips the row scan."""
    t, k = x.shape
    assert x.is_contiguous() and x.dtype == torch.bfloat16
    qd = _QDT[quant]
    q = _new(x, _TORCH_Q[qd], t, k)
    s = _new(x, torch.float32, t)
    nt = 0
    if group_amax is not None:
        assert group_amax.dtype == torch.float32 and group_amax.is_contiguous() and group_amax.shape[0] == t
        nt = group_amax.shape[1]
    with _k("quantize_per_token"):
        check(_lib().b200_quantize_per_token(x, q, s, group_amax, nt, t, k, qd),
              "b200_quantize_per_token")
    return q, s


def embedding(tokens, table, out=None):
    v, h = table.shape
    t = tokens.numel()
    assert tokens.dtype == torch.int64 and table.is_contiguous()
    if out is None:
        out = _new(table, table.dtype, t, h)
    with _k("embedding"):
        check(_lib().b200_embedding(tokens, table, out, t, h, v), "b200_embedding")
    return out


def argmax(logits, idx_offset: int = 0, want_val: bool = False, out_val=None, out_idx=None):
    t, v = logits.shape
    assert logits.dtype == torch.float32 and logits.stride(1) == 1
    idx = _new(logits, torch.int64, t) if out_idx is None else out_idx[:t]
    val = (_new(logits, torch.float32, t) if out_val is None else out_val[:t]) if want_val else None
    with _k("argmax"):
        check(_lib().b200_argmax(logits, logits.stride(0), val, idx, t, v, idx_offset), "b200_argmax")
    return (val, idx) if want_val else idx


def tp_argmax_merge(peer_vals, peer_idxs, peer_flags, epoch, rank, world, b):
    """Greedy merge of the per-shard (max, global index) pairs over peer memory (tp_comm.TpComm.merge_argmax)."""
    out = _new(epoch, torch.int64, b)
    with _k("tp_argmax_merge"):
        check(_cabi.load().b200_tp_argmax_merge(peer_vals, peer_idxs, peer_flags, _ptr(epoch), rank, world, _ptr(out), b,
                                                _stream()), "b200_tp_argmax_merge")
    return out


SAMPLE_K = 256  # candidates per (row, vocab shard); the reference's _MAX_NEURON_SAMPLING_TOP_K (RUNNER:74)


def topk_candidates(logits, idx_offset: int = 0):
    """logits fp32 [B, V] -> (cand_val [B,256] fp32, cand_idx [B,256] int64) sorted by (value desc, index asc)."""
    b, v = logits.shape
    assert logits.dtype == torch.float32 and logits.stride(1) == 1
    val = _new(logits, torch.float32, b, SAMPLE_K)
    idx = _new(logits, torch.int64, b, SAMPLE_K)
    with _k("topk_candidates"):
        check(_lib().b200_topk_candidates(logits, logits.stride(0), val, idx, b, v, idx_offset), "b200_topk_candidates")
    return val, idx


def sample_candidates(cand_val, cand_idx, params, u, out=None):
    """cand_* [B,256] or [groups,B,256]; params fp32 [B,3] = (top_k, top_p, temperature); u fp32 [B] in [0,1)."""
    if cand_val.dim() == 2:
        cand_val, cand_idx = cand_val.unsqueeze(0), cand_idx.unsqueeze(0)
    g, b, k = cand_val.shape
    assert k == SAMPLE_K and cand_val.is_contiguous() and cand_idx.is_contiguous() and cand_idx.dtype == torch.int64
    assert params.shape == (b, 3) and params.dtype == torch.float32 and params.is_contiguous()
    assert u.shape == (b,) and u.dtype == torch.float32
    if out is None:
        out = _new(cand_val, torch.int64, b)
    with _k("sample_candidates"):
        check(_lib().b200_sample_candidates(cand_val, cand_idx, g, b, params, u, out), "b200_sample_candidates")
    return out


def row_lse(logits):
    """logits fp32 [B, V] -> (row max [B], sum exp(x - max) [B]) of the local vocab shard."""
    b, v = logits.shape
    assert logits.dtype == torch.float32 and logits.stride(1) == 1
    m = _new(logits, torch.float32, b)
    s = _new(logits, torch.float32, b)
    with _k("row_lse"):
        check(_lib().b200_row_lse(logits, logits.stride(0), m, s, b, v), "b200_row_lse")
    return m, s


def gather_logprobs(cand_val, cand_idx, sampled, row_max, row_sumexp, num_logprobs: int):
    """cand_* [B,256] or [groups,B,256]; row_max / row_sumexp [B] or [groups,B]; sampled int64 [B].
    -> (ids int32 [B, 1+n], logprobs fp32 [B, 1+n], ranks int32 [B]) in vLLM's LogprobsTensors layout."""
    if cand_val.dim() == 2:
        cand_val, cand_idx, row_max, row_sumexp = cand_val.unsqueeze(0), cand_idx.unsqueeze(0), row_max.unsqueeze(0), row_sumexp.unsqueeze(0)
    g, b, k = cand_val.shape
    assert k == SAMPLE_K and cand_val.is_contiguous() and cand_idx.is_contiguous() and row_max.is_contiguous()
    assert row_max.shape == (g, b) and row_sumexp.shape == (g, b) and row_sumexp.is_contiguous() and sampled.dtype == torch.int64
    ids = _new(cand_val, torch.int32, b, 1 + num_logprobs)
    lp = _new(cand_val, torch.float32, b, 1 + num_logprobs)
    rk = _new(cand_val, torch.int32, b)
    with _k("gather_logprobs"):
        check(_lib().b200_gather_logprobs(cand_val, cand_idx, g, b, sampled, row_max,
                                                row_sumexp, num_logprobs, ids, lp, rk),
              "b200_gather_logprobs")
    return ids, lp, rk


def allreduce_rmsnorm(peer_bufs, peer_flags, epoch, rank, world, t, h, norm_w, eps, quant=None, want_bf16=False, mc_buf=0):
    """One-shot all-reduce over NVLink peer memory fused with RMSNorm (+ per-token quantisation).
    peer_bufs / peer_flags: ctypes arrays of `world` device pointers (tp_comm.TpComm).  mc_buf != 0: the multicast address
    of the partial -- the sum is then done inside the NVSwitch (b200_allreduce_rmsnorm_nvls).  Returns (x, h_out, h_scale):
    x = the reduced bf16 residual stream; h_out = normed bf16 (quant None) or quantised tensor; h_scale = scales or None."""
    dev = epoch.device
    x = torch.empty((t, h), dtype=torch.bfloat16, device=dev)
    qd = _QDT[quant]
    lib = _cabi.load()
    if mc_buf:
        fn, first, name = lib.b200_allreduce_rmsnorm_nvls, int(mc_buf), "b200_allreduce_rmsnorm_nvls"
    else:
        fn, first, name = lib.b200_allreduce_rmsnorm, peer_bufs, "b200_allreduce_rmsnorm"
    if norm_w is None:
        with _k("allreduce"):
            check(fn(first, peer_flags, _ptr(epoch), rank, world, _ptr(x), 0, 0, 0, 0, t, h, float(eps), BF16, _stream()), name)
        return x, None, None
    if qd == BF16:
        y = torch.empty_like(x)
        with _k("allreduce_rmsnorm"):
            check(fn(first, peer_flags, _ptr(epoch), rank, world, _ptr(x), _ptr(norm_w), _ptr(y), 0, 0, t, h, float(eps), qd,
                     _stream()), name)
        return x, y, None
    q = torch.empty((t, h), dtype=_TORCH_Q[qd], device=dev)
    s = torch.empty((t,), dtype=torch.float32, device=dev)
    y = torch.empty_like(x) if want_bf16 else None
    with _k("allreduce_rmsnorm_quant"):
        check(fn(first, peer_flags, _ptr(epoch), rank, world, _ptr(x), _ptr(norm_w), _ptr(y), _ptr(q), _ptr(s), t, h,
                 float(eps), qd, _stream()), name)
    return x, q, s


# ------------------------------------------------------------------ hybrid decoders (state-space + windowed attention + MoE)
# The residual stream and every norm / recurrence tensor is fp32; tensors that feed a GEMM or live in a KV pool are bf16
# (bf16 serving) or fp32 (32-bit serving).  `meta` is a StepMeta-like object with the ragged-batch index tensors.
def _edt(t):
    if t is torch.bfloat16 or (hasattr(t, "dtype") and t.dtype == torch.bfloat16):
        return BF16
    if t is torch.float32 or (hasattr(t, "dtype") and t.dtype == torch.float32):
        return F32
    raise _cabi.B200Error(f"element type {t} is neither bfloat16 nor float32")


def _f32(*ts):
    for t in ts:
        if t is not None and (t.dtype != torch.float32 or not t.is_contiguous()):
            raise _cabi.B200Error("expected a contiguous fp32 tensor")


def embed_scale(tokens, table, scale: float):
    """tokens int32 [T] -> fp32 [T, W] = table[token] * scale."""
    assert tokens.dtype == torch.int32 and table.is_contiguous()
    t, (v, w) = tokens.numel(), table.shape
    out = _new(table, torch.float32, t, w)
    with _k("embed_scale"):
        check(_lib().b200_embed_scale(tokens, table, _edt(table), out, t, w, v, float(scale)),
              "b200_embed_scale")
    return out


def dyt_norm(x, w, b, alpha: float, out_dtype):
    _f32(x, w, b)
    t, width = x.shape
    out = _new(x, out_dtype, t, width)
    with _k("dyt_norm"):
        check(_lib().b200_dyt_norm(x, w, b, float(alpha), out, _edt(out), t, width),
              "b200_dyt_norm")
    return out


def dyt_residual(x, y, norm, next_norm=None, out_dtype=torch.bfloat16, y2=None, nsum: int = 1):
    """x += dyt(sum of the nsum consecutive rows of y per token [+ y2]); returns dyt_next(x) in out_dtype (or None).
    norm / next_norm: (w, b, alpha)."""
    _f32(x, y, y2)
    t, width = x.shape
    assert y.shape == (t * nsum, width) and (y2 is None or y2.shape == (t, width))
    out2 = _new(x, out_dtype, t, width) if next_norm is not None else None
    w2, b2, a2 = next_norm if next_norm is not None else (None, None, 0.0)
    with _k("dyt_residual"):
        check(_lib().b200_dyt_residual(x, y, nsum, y2, norm[0], norm[1], float(norm[2]),
                                             w2, b2, float(a2), out2, _edt(out_dtype), t, width),
              "b200_dyt_residual")
    return out2


def gated_group_rmsnorm(y, z_src, w, groups: int, eps: float, out_dtype):
    """y fp32 [T, inner]; z = the first `inner` columns of the fp32 rows z_src (any pitch)."""
    _f32(y, w)
    assert z_src.dtype == torch.float32 and z_src.stride(1) == 1
    t, inner = y.shape
    out = _new(y, out_dtype, t, inner)
    with _k("gated_group_rmsnorm"):
        check(_lib().b200_gated_group_rmsnorm(y, z_src, z_src.stride(0), w, out, _edt(out), t, inner,
                                                    groups, float(eps)), "b200_gated_group_rmsnorm")
    return out


def clamped_glu(gate_up, limit: float, out_dtype):
    _f32(gate_up)
    t, ff2 = gate_up.shape
    out = _new(gate_up, out_dtype, t, ff2 // 2)
    with _k("clamped_glu"):
        check(_lib().b200_clamped_glu(gate_up, out, _edt(out), t, ff2 // 2, float(limit)),
              "b200_clamped_glu")
    return out


def causal_conv_silu(src, col0: int, channels: int, conv_w, conv_b, state, meta, out_dtype, *, in_bias=None, silu: bool = True):
    """Columns [col0, col0 + channels) of the fp32 rows `src` -> SiLU(conv) [T, channels]; `state` [slots, taps-1, channels]
    fp32 is read for continuing sequences and updated for all.  in_bias fp32 [channels]: added to the inputs read from `src`
    (a projection's bias; the state holds biased inputs).  silu False: the convolution alone."""
    _f32(src, conv_w, conv_b, state, in_bias)
    t, taps = src.shape[0], conv_w.shape[1]
    assert conv_w.shape[0] == channels and state.shape[1:] == (max(taps - 1, 1), channels)  # one unused row when taps == 1
    out = _new(src, out_dtype, t, channels)
    assert in_bias is None or in_bias.numel() == channels
    with _k("causal_conv_silu" if silu else "causal_conv"):
        check(_lib().b200_causal_conv(src, src.stride(0), col0, conv_w, conv_b, in_bias, 1 if silu else 0,
                                            state, meta.tok_seq, meta.seq_start, meta.seq_slot,
                                            meta.seq_pos0, out, _edt(out), t, meta.num_seqs, channels, taps),
              "b200_causal_conv")
    return out


SCAN_SEGMENT = 128  # tokens per parallel segment of a long portion in the selective scan


def ssd_scan(xbc, dt_src, dt_col0: int, a_log, dt_bias, d_skip, state, meta, heads: int, vdim: int, nstate: int, groups: int):
    """xbc [T, H*P + 2*G*N] (bf16 | fp32), raw dt = columns [dt_col0, dt_col0 + H) of the fp32 rows dt_src; state fp32
    [slots, H, P, N] updated in place; returns y fp32 [T, H*P].  When the step carries a segment list (meta.scan_segs: some
    portion is long) the segments run in parallel from scratch states that a combine pass chains together."""
    _f32(dt_src, a_log, dt_bias, d_skip, state)
    assert xbc.is_contiguous() and state.shape[1:] == (heads, vdim, nstate)
    t = xbc.shape[0]
    y = _new(xbc, torch.float32, t, heads * vdim)
    if getattr(meta, "max_new", 0) == 1:  # one token of every sequence: the state passes once, nothing is walked
        with _k("ssd_step"):
            check(_lib().b200_ssd_step(xbc, _edt(xbc), xbc.shape[1], dt_src, dt_src.stride(0), dt_col0, a_log,
                                             dt_bias, d_skip, state, meta.seq_start, meta.seq_slot,
                                             meta.seq_pos0, y, meta.num_seqs, heads, vdim, nstate, groups), "b200_ssd_step")
        return y
    segs = getattr(meta, "scan_segs", None)
    nseg = meta.num_segs if segs is not None else 0
    seg_state = seg_dt = None
    if nseg:
        seg_state = _new(xbc, torch.float32, nseg, heads, vdim, nstate)
        seg_dt = _new(xbc, torch.float32, nseg, heads)
    with _k("ssd_scan"):
        check(_lib().b200_ssd_scan_mma(xbc, _edt(xbc), xbc.shape[1], dt_src, dt_src.stride(0), dt_col0, a_log,
                                         dt_bias, d_skip, state, meta.seq_start, meta.seq_slot,
                                         meta.seq_pos0, y, meta.num_seqs, heads, vdim, nstate, groups,
                                         segs if nseg else 0, nseg, meta.scan_seq_seg0 if nseg else 0,
                                         seg_state, seg_dt), "b200_ssd_scan_mma")
    return y


def kv_write_vmix(qkv, k_col0: int, v_col0: int, k_pool, v_pool, slot_mapping, *, v_first=None, lam: float = 0.0, mode: int = 0):
    """Pools [num_blocks, G, block_size, D] / [.., Dv].  mode 0 plain, 1 record v_first, 2 mix with v_first before caching."""
    _f32(qkv, v_first)
    assert slot_mapping.dtype == torch.int64 and k_pool.dtype == v_pool.dtype and k_pool.is_contiguous() and v_pool.is_contiguous()
    _, g, bs, d = k_pool.shape
    dv = v_pool.shape[3]
    with _k("kv_write_vmix"):
        check(_lib().b200_kv_write_vmix(qkv, qkv.stride(0), k_col0, v_col0, v_first, float(lam), mode,
                                              k_pool, v_pool, _edt(k_pool), slot_mapping, qkv.shape[0], g, d, dv,
                                              bs), "b200_kv_write_vmix")


PREFILL_ATTN_MIN_TOKENS = 16  # longest portion of a step from which the tensor-core attention kernel is used
# ... and from which the tcgen05 kernel with its 128-row query tiles is.  With a sink, chained launches, us, mma.sync / tcgen05, 16 heads over 4 of 128, window
# 1024: one portion of 128 tokens 19.1 / 10.9, 256 after 1500 104 / 44, 4096 264 / 76; heads of 64, 128 tokens, window 128 13.9 / 8.3; over 576 steps of
# one to eight portions and 2 to 64 heads 0.17 to 0.83 of the time.
PREFILL_TC_MIN_TOKENS = 128
_SWA_PREFILL_LEGACY = bool(os.environ.get("B200_SWA_PREFILL_LEGACY"))


def _span(max_end: int, window: int, chunk: int, pool: int, keep: int) -> int:
    """Keys that a query sees at most in a step whose sequences reach max_end tokens (the pooled blocks before its window count as keys)."""
    return min(max_end, window, chunk or 1 << 30) + (max(max_end - window, 0) // pool if pool else 0) + keep


def _split_pays(parts, num_heads: int, g: int, d: int, dv: int, latent: bool, tc: bool, spans, pages: bool = True) -> bool:
    """Whether the decoded tokens of a mixed step are worth launches of their own.  spans: per part, the keys its queries see at most; pages:
    the cache's pages are whole tiles of the decode kernel (32 rows).
    In the prompt kernel each of them is a row tile per head (the tcgen05 kernel: per two heads) that walks its keys behind the prompts' own
    tiles; apart they cost a launch behind the prompts' and the decode kernel's time.  The estimate of the first is a list of tiles
    over the chip's slots: `us` per key and 5 per tile, the last tile's walk on top where there are more tiles than slots, a tenth for
    sharing the SMs.  The second, over pages of whole tiles: 4 us a launch and 3, the key and value bytes, 8 us for 1000 keys of one token.
    Measured, apart / together, us, prompts of 1600: 16 heads over 4 of 128, window of 512 with sinks, on tcgen05 29 tokens at 1800 54 / 78, 8 48 / 46,
    64 at 300 67 / 110, 29 at 300 72 / 66; 8 heads over 8 of 64, 64 at 1800 49 / 109; 200 tokens beside 64 at 1800 39 / 70 (mma.sync kernel 49 / 52).
    Over 4032 such steps the rule's choice costs 1.1 % more than the better one on average (mma.sync 0.7), always apart 19 (10), always together 38 (64);
    with the decode kernel's time as it was before its tiles lay on pages 6.0 (4.8).
    Over other pages: 14 us a launch, a fifth, and the decode kernel's time.  Over latents that kernel takes 17 us and more for the width of the rows, and
    the rounds of a cluster's keys; rows of 320, prompt of 600, us apart / together: 2 tokens at 200 58 / 31, 29 at 1800 71 / 182, 64 at 300 63 / 125."""
    us, rows, heads, slots = (0.0195, 128, num_heads, 148 * (2 if dv <= 128 else 1)) if tc and latent else \
        (0.026, 128, g * -(-num_heads // (2 * g)), 148) if tc else (0.045 + 0.00014 * (d + dv), 64, num_heads, 148 * (4 if dv <= 128 else 2))
    n, keys, tiles, work, walk = 0, 0, 0, 0.0, 0.0
    for p, span in zip(parts, spans):
        if p.max_new < PREFILL_ATTN_MIN_TOKENS:
            n, keys = n + p.num_tokens, max(keys, span)
        else:
            t = (-(-p.num_tokens // rows) + p.num_seqs - 1) * heads
            tiles, work, walk = tiles + t, work + t * (5 + us * min(span, p.max_end - p.max_new / 2)), max(walk, 5 + us * span)
    last = 5 + us * keys

    def makespan(tiles, work):
        return max(walk, last, work / slots + last * max(0.0, 1 - slots / tiles))

    alone = max(walk, work / slots + walk * max(0.0, 1 - slots / tiles))
    together = makespan(tiles + n * heads, work + n * heads * last)
    if pages and not latent:
        return 1.1 * together > alone + 4 * (len(parts) - 1) + 3 + keys * (4e-7 * n * g * (d + dv) + 0.008)
    if latent:
        splits = _latent_splits(n, num_heads, keys)
        return together > alone + 8 * (len(parts) - 1) + 0.044 * d + 3 + 9e-5 * d * keys / splits * -(-n * -(-num_heads // 16) * splits // 148)
    return 1.2 * together > alone + 14 * (len(parts) - 1) + keys * (n * g / 4000 + 0.008)


def swa_sink_attn(q_src, num_heads: int, k_pool, v_pool, block_table, meta, sink, scale: float, window: int,
                  latent_values: int = 0, *, chunk: int = 0, softcap: float = 0.0, sigmoid_bias=None, out_f32: bool = False,
                  split_p: bool = False, pooled=None, keep: int = 0):
    """q = the first num_heads * D columns of the fp32 rows q_src -> [T, num_heads * Dv] in the pools' element type.
    sink None: ordinary softmax.  latent_values = C > 0: v_pool is ignored and the values are the first C columns of the key
    rows (attention over cached latents: one pool holds both).
    chunk > 0: a query sees only the keys of its own chunk of that many positions (counted from position 0).  softcap > 0:
    scaled scores pass through softcap * tanh(s / softcap).  sigmoid_bias fp32 [H]: weights sigmoid(s + bias[h]), not normalised
    over keys.  A value pool with fewer heads than the key pool: consecutive key heads share a value head (two score maps over
    the same values).  out_f32: fp32 rows.  split_p: the tensor-core kernel carries the weights as two bf16 terms.
    pooled = (pooled key pool, pooled value pool, P) with a window: every block of P positions that lies wholly before a query's
    window is seen as one key / value, the block's row of the pooled pools (kv_pool_mean), in the same softmax.
    keep > 0 with a window: the sequence's first `keep` tokens stay visible to every later query."""
    assert not (keep and (pooled is not None or latent_values))
    if window >= (1 << 30):
        keep = 0
    _cuda(q_src, k_pool, v_pool, block_table, sink, sigmoid_bias)
    pk, pv, pool = pooled if pooled is not None else (None, None, 0)
    if pool:
        _cuda(pk, pv)
        ppb = -(-k_pool.shape[2] // pool)
        assert not latent_values and window < (1 << 30) and pk.dtype == k_pool.dtype and pv.dtype == k_pool.dtype
        assert pk.is_contiguous() and pv.is_contiguous() and pk.shape == (k_pool.shape[0], k_pool.shape[1], ppb, k_pool.shape[3])
        assert pv.shape == (v_pool.shape[0], v_pool.shape[1], ppb, v_pool.shape[3])
    pool_args = (pk, pv, int(pool), int(keep))
    _f32(q_src, sink, sigmoid_bias)
    assert block_table.dtype == torch.int32 and block_table.stride(1) == 1
    _, g, bs, d = k_pool.shape
    if latent_values:
        v_pool, dv, v_pitch = k_pool, int(latent_values), d
        assert g == 1 and dv <= d
    else:
        dv = v_pitch = v_pool.shape[3]
    v_div = g // v_pool.shape[1]
    assert v_pool.shape[1] * v_div == g and v_pool.shape[2] == bs
    out = _new(q_src, torch.float32 if out_f32 else k_pool.dtype, q_src.shape[0], num_heads * dv)
    # decoded tokens beside prompt portions: each kind on its own kernel where that pays, in one launch of the prompt kernel otherwise
    parts = getattr(meta, "parts", None)
    if parts:
        tc = _latent_tc(q_src, k_pool, meta, d, dv, bs, scale, chunk, softcap, sigmoid_bias, out_f32) if latent_values else \
            _prompt_tc(q_src, k_pool, meta, d, dv, bs, v_div, latent_values, softcap, sigmoid_bias, pool)
        spans = [_span(p.max_end, int(window), int(chunk), pool, int(keep)) for p in parts]
        if not (tc or _prompt_mma(q_src, k_pool, meta, d, dv)) or not _split_pays(parts, num_heads, g, d, dv, bool(latent_values), tc, spans, bs % 32 == 0):
            parts = None
    for part in parts or [meta]:
        _swa_part(q_src, num_heads, k_pool, v_pool, block_table, part, sink, scale, window, latent_values, chunk, softcap, sigmoid_bias,
                  out_f32, split_p, pool, pool_args, keep, out, g, bs, d, dv, v_pitch, v_div)
    return out


def _prompt_tc(q, k_pool, meta, d, dv, bs, v_div, latent_values, softcap, sigmoid_bias, pool) -> bool:
    """Long prompt portions in bf16 serving (with or without a sink; a sliding window only without pooled blocks), head sizes of 64 / 128 with pages of 32 tokens: the
    tcgen05 kernel (128-row query tiles, accumulators in tensor memory); B200_SWA_PREFILL_LEGACY=1 keeps the mma.sync kernel (A/B aid)."""
    return bool(k_pool.dtype == torch.bfloat16 and meta.max_new >= PREFILL_TC_MIN_TOKENS and not pool
                and not latent_values and q.stride(0) % 4 == 0 and q.data_ptr() % 16 == 0 and not _SWA_PREFILL_LEGACY
                and _lib().b200_swa_sink_attn_prefill_tc_supported(d, dv, bs, v_div, 1 if softcap else 0,
                                                                         0 if sigmoid_bias is None else 1))


def _prompt_mma(q, k_pool, meta, d, dv) -> bool:
    """Shorter prompt portions in bf16 serving: the mma.sync kernel."""
    return (k_pool.dtype == torch.bfloat16 and meta.max_new >= PREFILL_ATTN_MIN_TOKENS and d % 16 == 0 and dv % 16 == 0
            and d <= 512 and dv <= 256 and q.stride(0) % 2 == 0)


def _latent_tc(q, k_pool, meta, d, dv, bs, scale, chunk, softcap, sigmoid_bias, out_f32) -> bool:
    """Prompt portions over cached latents, bf16 rows of up to 64 columns beside the 128 or 256 value columns, pages of 32 tokens: the tcgen05
    kernel (positive scales: it scales a row's largest score, not the scores).  From the shortest portion on: us, 16 heads over rows of 320, mma.sync / here: 16 tokens 20 / 14, at 1800 227 / 47, 128 41 / 18, 1000 162 / 39,
    1600 310 / 51, 512 at 4000 549 / 107; rows of 160: 16 16 / 12, 1600 184 / 51."""
    return bool(not (chunk or softcap or out_f32) and scale > 0 and sigmoid_bias is None and k_pool.dtype == torch.bfloat16 and meta.max_new >= PREFILL_ATTN_MIN_TOKENS
                and q.stride(0) % 4 == 0 and q.data_ptr() % 16 == 0 and k_pool.data_ptr() % 16 == 0
                and _lib().b200_latent_attn_prefill_tc_supported(d, dv, bs))


def _latent_splits(tokens: int, heads: int, keys: int) -> int:
    """CTAs that share a token's keys in latent attention: while there are rounds of tiles to share (8 warps of 32 keys) and the clusters of all tokens
    and groups of 16 heads are resident together, a CTA an SM (clusters of 4 and 8 leave some free).  us, 16 heads over rows of 320, one CTA / two / four /
    eight: one token at 2000 84 / 59 / 43 / 35, at 200 33 / 37 / 35 / 35; 16 tokens at 2000 84 / 59 / 43 / 66; 29 at 1800 80 / 59 / 45 / 66; 37 at 1500 70 / 53
    / 72; 64 at 2000 84 / 62 / 84; 100 at 1000 55 / 84."""
    ctas = tokens * -(-heads // 16)
    n = 1
    while n < 8 and 256 * n < keys and 2 * n * ctas <= {1: 136, 2: 120, 4: 72}[n]:
        n *= 2
    return n


def _swa_part(q_src, num_heads, k_pool, v_pool, block_table, meta, sink, scale, window, latent_values, chunk, softcap, sigmoid_bias, out_f32,
              split_p, pool, pool_args, keep, out, g, bs, d, dv, v_pitch, v_div):
    """The sequences of `meta` (a step, or a StepPart of one) through the kernel that suits them.  Prompt kernels index the step's rows
    by seq_start; the decode kernels take the part's rows."""
    q_all, out_all = q_src, out
    if hasattr(meta, "tok0"):
        q_src, out = (x[meta.tok0:meta.tok0 + meta.num_tokens] for x in (q_src, out))
    t = q_src.shape[0]
    variant = (int(chunk), float(softcap), sigmoid_bias, v_div, 1 if out_f32 else 0)
    plain = not chunk and not softcap and sigmoid_bias is None and v_div == 1 and not out_f32
    # the per-launch timer tells the variants apart (their floors differ)
    tag = "[latent]" if plain and latent_values else "" if plain and not pool and not keep else "[" + "+".join(n for n, on in (("chunk", chunk), ("cap", softcap), ("sigmoid", sigmoid_bias is not None),
                                                                       ("maps", v_div > 1), ("pool", pool), ("keep", keep)) if on) + "]"
    if _prompt_tc(q_all, k_pool, meta, d, dv, bs, v_div, latent_values, softcap, sigmoid_bias, pool):
        if sink is not None and window < 1:
            raise _cabi.B200Error(f"swa_sink_attn: a window of {window}")
        with _k("swa_sink_attn_prefill_tc" + tag):
            check(_lib().b200_swa_attn_prefill_tc_sink(q_all, q_all.stride(0), k_pool, v_pool, k_pool.shape[0],
                                                             block_table, block_table.stride(0), meta.seq_start,
                                                             meta.seq_slot, meta.seq_pos0, meta.num_seqs, meta.max_new,
                                                             float(scale), out_all, num_heads, g, d, dv, bs, *variant,
                                                             1 if split_p else 0, int(window) if window < (1 << 30) else 0,
                                                             int(keep), sink),
                  "b200_swa_attn_prefill_tc_sink")
        return
    if latent_values and _latent_tc(q_all, k_pool, meta, d, dv, bs, scale, chunk, softcap, sigmoid_bias, out_f32):
        with _k("swa_sink_attn_prefill_tc" + tag):
            check(_lib().b200_latent_attn_prefill_tc(q_all, q_all.stride(0), k_pool, k_pool.shape[0], block_table, block_table.stride(0),
                                                           meta.seq_start, meta.seq_slot, meta.seq_pos0, meta.num_seqs, meta.max_new, sink,
                                                           float(scale), int(window), out_all, num_heads, d, dv, bs),
                  "b200_latent_attn_prefill_tc")
        return
    if _prompt_mma(q_all, k_pool, meta, d, dv):
        with _k("swa_sink_attn_prefill" + tag):
            check(_lib().b200_swa_sink_attn_prefill(q_all, q_all.stride(0), k_pool, v_pool, block_table,
                                                          block_table.stride(0), meta.seq_start, meta.seq_slot,
                                                          meta.seq_pos0, meta.num_seqs, meta.max_new, sink, float(scale),
                                                          int(window), out_all, num_heads, g, d, dv, v_pitch, bs, *variant,
                                                          1 if split_p else 0, *pool_args),
                  "b200_swa_sink_attn_prefill")
        return
    if (plain and latent_values and k_pool.dtype == torch.bfloat16 and d % 16 == 0 and dv % 16 == 0
            and dv <= 256 and q_src.stride(0) % 2 == 0):
        # attention over cached latents, decode-sized steps: the heads of a token are the rows of a tensor-core tile
        with _k("latent_attn_decode"):
            splits = _latent_splits(t, num_heads, _span(getattr(meta, "max_end", 0) or 0, int(window), 0, 0, 0))
            check(_lib().b200_latent_attn_decode_split(q_src, q_src.stride(0), k_pool, block_table,
                                                             block_table.stride(0), meta.tok_row, meta.tok_pos, sink,
                                                             float(scale), int(window), out, t, num_heads, d, dv, bs, splits),
                  "b200_latent_attn_decode_split")
        return
    # decode-sized steps, fp32 pools and odd head sizes.  Long contexts at small batch: several CTAs share a (token, kv head)'s keys, so that
    # every SM has its CTAs
    span = _span(getattr(meta, "max_end", 0) or 0, int(window), int(chunk), pool, int(keep))
    tc = (k_pool.dtype == torch.bfloat16 and not latent_values and d % 16 == 0 and dv % 16 == 0 and d * v_div <= 512 and dv <= 256
          and q_src.stride(0) % 2 == 0)
    gv = g // v_div
    ctas = t * gv * -(-(num_heads // gv) // 16) if tc else t * g
    splits = max(1, min(8, (148 * (3 if tc else 4)) // max(1, ctas), -(-span // (128 if tc else 512))))
    ws = _new(q_src, torch.float32, t * num_heads * splits * (dv + 2)) if splits > 1 else None
    if tc:  # decode-sized steps on bf16 pools: the query heads of a kv head are the rows of a tensor-core tile
        with _k("swa_sink_attn_decode_tc" + tag):
            check(_lib().b200_swa_sink_attn_decode_tc(q_src, q_src.stride(0), k_pool, v_pool, block_table,
                                                            block_table.stride(0), meta.tok_row, meta.tok_pos, sink,
                                                            float(scale), int(window), out, t, num_heads, g, d, dv, v_pitch, bs,
                                                            *variant, 1 if split_p else 0, splits, ws, *pool_args),
                  "b200_swa_sink_attn_decode_tc")
        return
    with _k("swa_sink_attn" + tag):
        check(_lib().b200_swa_sink_attn(q_src, q_src.stride(0), k_pool, v_pool, _edt(k_pool),
                                              block_table, block_table.stride(0), meta.tok_row, meta.tok_pos,
                                              sink, float(scale), int(window), out, t, num_heads, g, d, dv, v_pitch, bs,
                                              *variant, splits, ws, *pool_args), "b200_swa_sink_attn")


def moe_topk(logits, top: int, bias=None, mode: int = ROUTE_SIGMOID):
    """fp32 router logits [T, E] (+ bias fp32 [E]) -> (expert ids int32 [T, top], routing weights fp32 [T, top]): the sigmoid of
    each chosen logit (ROUTE_SIGMOID), the softmax over the chosen logits (ROUTE_SOFTMAX_TOP), or the softmax over all experts with
    the chosen scores divided by their sum (ROUTE_SOFTMAX_RENORM)."""
    _f32(bias)
    assert logits.dtype == torch.float32 and logits.stride(1) == 1
    t, e = logits.shape
    idx = _new(logits, torch.int32, t, top)
    wt = _new(logits, torch.float32, t, top)
    with _k("moe_topk"):
        check(_lib().b200_moe_topk(logits, logits.stride(0), bias, int(mode), idx, wt, t, e, top), "b200_moe_topk")
    return idx, wt


def moe_topk_grouped(logits, correction, top: int, *, groups: int = 1, keep: int = 1, scale: float = 1.0):
    """fp32 router logits [T, E] -> (expert ids int32 [T, top], routing weights fp32 [T, top]).  Scores = softmax over all experts;
    the `top` largest of score + correction (fp32 [E] or None) are chosen among the experts of the best `keep` of `groups` equal
    runs of neighbours (a run's rank: its largest choice score); weight = score * scale."""
    _f32(correction)
    assert logits.dtype == torch.float32 and logits.stride(1) == 1
    t, e = logits.shape
    assert correction is None or correction.numel() == e
    idx = _new(logits, torch.int32, t, top)
    wt = _new(logits, torch.float32, t, top)
    with _k("moe_topk_grouped"):
        check(_lib().b200_moe_topk_grouped(logits, logits.stride(0), correction, int(groups), int(keep), float(scale),
                                                 idx, wt, t, e, top), "b200_moe_topk_grouped")
    return idx, wt


def moe_tile_rows() -> int:
    return int(_lib().b200_moe_tile_rows())


def moe_align(topk_idx, num_experts: int, tile_rows: int | None = None):
    """-> (sorted pair ids int32 [cap] padded with -1, tile owners int32 [max_tiles], device count of used tiles [1], rows per
    tile).  tile_rows: moe_tile_rows() (default) or four times that for prompt-sized bf16 batches."""
    assert topk_idx.dtype == torch.int32 and topk_idx.is_contiguous()
    n, bm = topk_idx.numel(), tile_rows or moe_tile_rows()
    max_tiles = -(-n // bm) + num_experts
    sorted_ids = _new(topk_idx, None, max_tiles * bm)
    tile_expert = _new(topk_idx, None, max_tiles)
    num_tiles = _new(topk_idx, None, 1)
    with _k("moe_align"):
        check(_lib().b200_moe_align(topk_idx, n, num_experts, sorted_ids, sorted_ids.numel(), tile_expert,
                                          max_tiles, num_tiles, bm), "b200_moe_align")
    return sorted_ids, tile_expert, num_tiles, bm


def moe_wide_tiles(h, w_gate_up, num_pairs: int) -> int | None:
    """Rows per expert tile for this batch: the wide tile once the experts see about 64 rows each on average and the
    operands suit the tensor-core kernel, else None (the default tile)."""
    e, ff2, width = w_gate_up.shape
    if h.dtype == torch.bfloat16 and width % 8 == 0 and (ff2 // 2) % 8 == 0 and h.stride(0) % 8 == 0 and num_pairs >= 64 * e:
        return 4 * moe_tile_rows()
    return None


def linear_simt(a, w):
    """fp32 [M, N] = a [M, K] @ w [N, K]^T with fp32 accumulation on the CUDA cores: fp32 operands, or shapes the tensor-core
    GEMM does not take."""
    assert a.dtype == w.dtype and a.stride(1) == 1 and w.is_contiguous() and a.shape[1] == w.shape[1]
    m, k = a.shape
    n = w.shape[0]
    out = _new(a, torch.float32, m, n)
    with _k("linear_simt[{}x{}x{}]", m, n, k):
        check(_lib().b200_grouped_linear(a, a.stride(0), 0, 0, 0, w, 0, 0, 0, -(-m // moe_tile_rows()), m, n, k,
                                               _edt(a), out, n, 0, 0, 0, 0.0, moe_tile_rows()), "b200_grouped_linear")
    return out


def batched_linear(a, w, out, *, a_batch_stride: int, out_batch_stride: int, gate=None, gate_cols: bool = False):
    """out_b = a_b @ w[b]^T for every b of w [batch, N, K] in one launch: a_b = rows of `a` (pitch a.stride(0)) starting at
    column b * a_batch_stride, out_b likewise in `out` (fp32, or the operand type).  gate: fp32 view [M, >= batch] whose
    sigmoid multiplies out_b's rows -- or, with gate_cols, [M, >= batch * N], a gate per output column (column b * N + n)."""
    assert a.dtype == w.dtype and a.stride(1) == 1 and out.stride(1) == 1 and w.is_contiguous() and w.dim() == 3
    b, n, k = w.shape
    m = a.shape[0]
    typed = out.dtype == a.dtype and out.dtype != torch.float32
    assert typed or out.dtype == torch.float32
    if gate is not None:
        assert gate.dtype == torch.float32 and gate.stride(1) == 1 and gate.shape[0] == m
        assert gate.shape[1] >= (b * n if gate_cols else b)
    with _k("batched_linear[{}x{}x{}x{}]", b, m, n, k):
        check(_lib().b200_batched_linear(a, a.stride(0), a_batch_stride, w, n * k, out, out.stride(0),
                                               out_batch_stride, b, m, n, k, _edt(a), 1 if typed else 0, gate,
                                               gate.stride(0) if gate is not None else 0, 1 if gate_cols and gate is not None else 0),
              "b200_batched_linear")
    return out


def moe_experts(h, topk_weight, align, w_gate_up, w_down, top: int, limit: float = 0.0, act: int = ACT_SWISH_CLAMPED,
                scale_input: bool = True):
    """Routed experts: for every (token, choice) pair  W_down glu(W_gate_up (weight * h)) (scale_input), or the unweighted
    expert output (the caller then weighs the outputs).  h [T, W]; w_gate_up [E, 2 ff, W] (gate rows first), w_down
    [E, W, ff]; returns fp32 [T * top, W] in pair order."""
    sorted_ids, tile_expert, num_tiles, bm = align
    e, ff2, width = w_gate_up.shape
    ff = ff2 // 2
    tiles = tile_expert.numel()
    hid = _new(h, h.dtype, sorted_ids.numel(), ff)
    out = _new(h, torch.float32, h.shape[0] * top, width)
    # prompt-sized batches, and experts of whole pair-kernel tiles at any size: gather and scale the pairs once, then plain rows
    pair_tiles = h.dtype == torch.bfloat16 and width % 256 == 0 and ff % 128 == 0 and tiles <= 1024 and h.stride(0) % 8 == 0 and h.data_ptr() % 16 == 0
    if bm > moe_tile_rows() or pair_tiles:
        rows = _new(h, h.dtype, sorted_ids.numel(), width)
        with _k("moe_gather_scale"):
            check(_lib().b200_moe_gather_scale(h, h.stride(0), sorted_ids, sorted_ids.numel(), top,
                                            topk_weight if scale_input else None,
                                            num_tiles, bm, rows, width), "b200_moe_gather_scale")
        a, lda, gdiv, scale = rows, width, 0, None
    else:
        a, lda, gdiv, scale = h, h.stride(0), top, topk_weight if scale_input else None
    with _k("moe_gate_up_glu"):
        check(_lib().b200_grouped_linear(a, lda, sorted_ids, gdiv, scale, w_gate_up, ff2 * width,
                                      tile_expert, num_tiles, tiles, 0, ff, width, _edt(h), hid, ff, 0, 1,
                                      int(act), float(limit), bm), "b200_grouped_linear")
    with _k("moe_down"):
        check(_lib().b200_grouped_linear(hid, ff, sorted_ids, 0, 0, w_down, width * ff, tile_expert,
                                      num_tiles, tiles, 0, width, ff, _edt(h), out, width, 1, 0, 0, 0.0, bm),
              "b200_grouped_linear")
    return out


# ------------------------------------------------------------------ post-norm hybrid decoders (delta rule + latent attention)
def embed_bigram(tokens, table, scale: float, meta, *, bigram=None, buckets: int = 0, mul_prev: int = 0, mul_cur: int = 0,
                 prev_state=None, want_cast: bool = True):
    """tokens int32 [T] -> (x fp32 [T, W], the same rows in the table's type or None).  x = table[token] * scale + bigram[row]
    with row hashed from (previous token, token); prev_state int32 [slots] carries each sequence's last token across steps."""
    assert tokens.dtype == torch.int32 and table.is_contiguous() and (bigram is None or (bigram.is_contiguous() and bigram.dtype == table.dtype))
    t, (v, w) = tokens.numel(), table.shape
    out = _new(table, torch.float32, t, w)
    cast = _new(table, table.dtype, t, w) if want_cast else None
    with _k("embed_bigram"):
        check(_lib().b200_embed_bigram(tokens, table, bigram, _edt(table), int(buckets), int(mul_prev),
                                             int(mul_cur), prev_state, meta.tok_seq, meta.seq_start,
                                             meta.seq_slot, meta.seq_pos0, out, cast, t, w, v, float(scale)), "b200_embed_bigram")
    return out, cast


def rms_residual(x, y, w, eps: float, *, offset: float = 1.0, nsum: int = 1, y_weight=None, out_dtype=None):
    """x += rmsnorm(sum of the nsum consecutive rows of y per token, weighted by y_weight [T, nsum] when given) * (offset + w);
    returns x in out_dtype (the next GEMM's operand) or None."""
    _f32(x, y, w, y_weight)
    t, width = x.shape
    assert y.shape == (t * nsum, width) and (y_weight is None or y_weight.numel() == t * nsum)
    cast = _new(x, out_dtype, t, width) if out_dtype is not None else None
    with _k("rms_residual"):
        check(_lib().b200_rms_residual(x, y, nsum, y_weight, w, float(offset), float(eps), cast,
                                             _edt(out_dtype) if out_dtype is not None else F32, t, width), "b200_rms_residual")
    return cast


def rmsnorm_cols(src, col0: int, n: int, w, eps: float, out_dtype, *, offset: float = 0.0):
    """RMS norm of columns [col0, col0 + n) of the fp32 rows src, times (offset + w) -> [T, n] in out_dtype."""
    _f32(w)
    assert src.dtype == torch.float32 and src.stride(1) == 1 and w.numel() == n
    t = src.shape[0]
    out = _new(src, out_dtype, t, n)
    with _k("rmsnorm_cols"):
        check(_lib().b200_rmsnorm_cols(src, src.stride(0), col0, n, w, float(offset), float(eps), out,
                                             _edt(out), n, t), "b200_rmsnorm_cols")
    return out


def head_rmsnorm_gate(o, gate_src, gate_col0: int, w, eps: float, heads: int, out_dtype):
    """o fp32 [T, H * P]: per head o / rms(o) * w [P] * silu(gate), gate = columns gate_col0.. of the fp32 rows gate_src
    (gate_src None: the norm alone)."""
    _f32(o, w)
    assert gate_src is None or (gate_src.dtype == torch.float32 and gate_src.stride(1) == 1)
    t, hp = o.shape
    p = hp // heads
    assert w.numel() == p
    out = _new(o, out_dtype, t, hp)
    with _k("head_rmsnorm_gate"):
        check(_lib().b200_head_rmsnorm_gate(o, gate_src, gate_src.stride(0) if gate_src is not None else 0, gate_col0, w, float(eps),
                                                  out, _edt(out), t, heads, p), "b200_head_rmsnorm_gate")
    return out


def glu(gate_up, act: int, out_dtype):
    """fp32 [T, 2 ff] (gate columns first) -> act(gate) * up in out_dtype; act = ACT_SILU | ACT_GELU_TANH."""
    _f32(gate_up)
    t, ff2 = gate_up.shape
    out = _new(gate_up, out_dtype, t, ff2 // 2)
    with _k("glu"):
        check(_lib().b200_glu(gate_up, out, _edt(out), t, ff2 // 2, int(act)), "b200_glu")
    return out


def _delta_rounds(longest: int, tokens: int, heads: int, dim: int, vdim: int) -> bool:
    """Whether a step whose longest portion has 8 tokens or more takes the rounds of eight tokens.  They shorten the chain of a portion; where
    portions of one length already fill the chip, the two-token kernel's smaller CTAs share an SM better.  Two-token / rounds, us, heads of
    64 x 64: 4 portions of 17 x 8 heads 9.0 / 7.1, 20 12.7 / 15.9; 12 of 40 17.6 / 15.0, 24 21.9 / 24.2, 64 44.5 / 53.0; 20 of 300 121.7 / 112.0,
    one of 300 beside 31 tokens 71.6 / 30.3.  Of 128 x 128, 20 of 17 x 8 heads 30.9 / 34.0 (rounds of eight pad 17 to 24), of 8 19.7 / 20.4, of 40
    56.7 / 49.1."""
    together = tokens / longest * heads * (vdim // 16)  # CTAs of 16 columns, were all portions the longest
    if dim == 64:
        return together <= 300 or (together <= 640 and longest >= 32)
    return together <= 640 or not 16 < longest < 24


def delta_rule(qkv, proj, b_col0: int, a_col0: int, a_log, dt_bias, state, meta, heads: int, kv_heads: int, dim: int, vdim: int,
               q_scale: float, unit_eps: float = 1e-6):
    """Gated delta rule over a ragged batch.  qkv fp32 [T, q: G*D | k: G*D | v: H*P] (convolved; q and k are normalised IN
    PLACE); raw beta / decay inputs are columns b_col0.. / a_col0.. of the fp32 rows proj; state fp32 [slots, H, P, D] updated
    in place.  Returns o fp32 [T, H * P]."""
    _f32(qkv, a_log, dt_bias, state)
    assert proj.dtype == torch.float32 and proj.stride(1) == 1 and state.shape[1:] == (heads, vdim, dim)
    assert qkv.shape[1] == 2 * kv_heads * dim + heads * vdim
    t = qkv.shape[0]
    bg = _new(qkv, torch.float32, t, 2 * heads)
    kq = _new(qkv, torch.float32, t, kv_heads)
    out = _new(qkv, torch.float32, t, heads * vdim)
    with _k("delta_prep"):
        check(_lib().b200_delta_prep(qkv, qkv.stride(0), proj, proj.stride(0), b_col0, a_col0, a_log, dt_bias,
                                  bg, kq, t, heads, kv_heads, dim, float(q_scale), float(unit_eps)),
              "b200_delta_prep")
    longest = int(meta.max_new)
    if longest >= 8 and not _delta_rounds(longest, t, heads, dim, vdim):
        longest = 7  # the two-token kernel
    with _k("delta_scan"):
        check(_lib().b200_delta_scan(qkv, qkv.stride(0), bg, kq, state, meta.seq_start,
                                  meta.seq_slot, meta.seq_pos0, out, meta.num_seqs, longest, heads, kv_heads, dim, vdim), "b200_delta_scan")
    return out


def latent_kv_write(src, col0: int, kv_rank: int, rot_dim: int, rot_n: int, norm_w, eps: float, cos, sin, meta, pool):
    """Columns [col0, col0 + kv_rank + rot_dim) of the fp32 rows src -> pool rows [RMS-normed latent | rotated shared key part]
    at the step's slots.  pool [num_blocks, 1, block_size, kv_rank + rot_dim]; cos / sin fp32 [positions, rot_n / 2]."""
    _f32(norm_w, cos, sin)
    assert src.dtype == torch.float32 and src.stride(1) == 1 and pool.is_contiguous() and pool.shape[-1] == kv_rank + rot_dim
    with _k("latent_kv_write"):
        check(_lib().b200_latent_kv_write(src, src.stride(0), col0, kv_rank, rot_dim, rot_n, norm_w, float(eps),
                                                cos, sin, meta.tok_pos, meta.slot_mapping, pool,
                                                _edt(pool), src.shape[0]), "b200_latent_kv_write")


def latent_q_prep(q, heads: int, dim: int, rot_dim: int, rot_n: int, kv_rank: int, cos, sin, meta, nope_dtype):
    """q fp32 [T, H * (dim + rot_dim)] -> (unrotated parts [T, H * dim] in nope_dtype, attention query fp32 [T, H * (kv_rank +
    rot_dim)] whose last rot_dim columns per head hold the rotated part; the first kv_rank are left for the absorbing GEMM)."""
    _f32(q, cos, sin)
    t = q.shape[0]
    nope = _new(q, nope_dtype, t, heads * dim)
    q_att = _new(q, torch.float32, t, heads * (kv_rank + rot_dim))
    with _k("latent_q_prep"):
        check(_lib().b200_latent_q_prep(q, q.stride(0), heads, dim, rot_dim, rot_n, kv_rank, cos, sin,
                                              meta.tok_pos, nope, _edt(nope), q_att, t),
              "b200_latent_q_prep")
    return nope, q_att


# ------------------------------------------------------------------ parallel-branch decoders (grouped norm, rotating attention variants)
def add_group_rmsnorm(x, y1, y2, w, groups: int, eps: float, out_dtype=None):
    """x += y1 + y2 (fp32 rows, any pitch; y2 or both may be None), in place; returns the grouped RMS norm of x times w in
    out_dtype (each of the `groups` equal consecutive parts of a row divided by its own RMS), or None when out_dtype is None."""
    _f32(x, w)
    t, width = x.shape
    for y in (y1, y2):
        assert y is None or (y.dtype == torch.float32 and y.stride(1) == 1 and y.shape == (t, width))
    out = _new(x, out_dtype, t, width) if out_dtype is not None else None
    with _k("add_group_rmsnorm"):
        check(_lib().b200_add_group_rmsnorm(x, y1, y1.stride(0) if y1 is not None else 0, y2,
                                                  y2.stride(0) if y2 is not None else 0, w, int(groups), float(eps), out,
                                                  _edt(out) if out is not None else F32, t, width), "b200_add_group_rmsnorm")
    return out


def poly_norm(src, col0: int, n: int, coef, eps: float, out_dtype):
    """Columns [col0, col0 + n) of the fp32 rows src -> a N(z) + b N(z^2) + c N(z^3) + e [T, n] in out_dtype; coef fp32 [4] =
    (a, b, c, e); N divides a row by its RMS."""
    _f32(coef)
    assert src.dtype == torch.float32 and src.stride(1) == 1 and coef.numel() == 4
    t = src.shape[0]
    out = _new(src, out_dtype, t, n)
    with _k("poly_norm"):
        check(_lib().b200_poly_norm(src, src.stride(0), col0, n, coef, float(eps), out, _edt(out), n, t), "b200_poly_norm")
    return out


def diff_head_norm_gate(a, lam: float, post: float, gate_src, gate_col0: int, eps: float, heads: int, rep: int, out_dtype):
    """a fp32 [T, 2 * heads * P] (per kv group of `rep` heads: the first maps' rows, then the second maps') ->
    [T, heads * P] = unit-RMS(a1 - lam * a2) * post * sigmoid(gate), gate = columns gate_col0.. of the fp32 rows gate_src
    (None: no gate)."""
    _f32(a)
    assert gate_src is None or (gate_src.dtype == torch.float32 and gate_src.stride(1) == 1)
    t = a.shape[0]
    p = a.shape[1] // (2 * heads)
    out = _new(a, out_dtype, t, heads * p)
    with _k("diff_head_norm_gate"):
        check(_lib().b200_diff_head_norm_gate(a, float(lam), float(post), gate_src,
                                                    gate_src.stride(0) if gate_src is not None else 0, gate_col0, float(eps),
                                                    out, _edt(out), t, heads, rep, p), "b200_diff_head_norm_gate")
    return out


def qk_norm_rope_kv_write(src, q_col0: int, k_col0: int, v_col0: int, heads: int, k_pool, v_pool, meta, *, q_norm=None,
                          k_norm=None, eps: float = 0.0, rot_n: int = 0, rot_half: bool = True, cos=None, sin=None, q_head_scale=None,
                          head_norm: bool = False, bias=None):
    """fp32 rows src = [.. q: heads * D .. k: G * D .. v: Gv * Dv ..] -> q fp32 [T, heads * D] (normed over the whole projection
    when q_norm is given, leading rot_n columns of every head rotated by the token's position), and the step's keys (same
    treatment) and values written into the pools [num_blocks, G, block_size, D] / [num_blocks, Gv, block_size, Dv].
    q_head_scale fp32 [heads]: q of head h is multiplied by it (a per-head temperature of the scores).
    head_norm: the norms are per head, q_norm / k_norm fp32 [D] shared by the heads.  v_col0 may equal k_col0: the cached values
    are then the keys as projected, before norm and rotation.  bias fp32 [heads * D + G * D + Gv * Dv]: the projections' biases,
    q | k | v, added ahead of everything else."""
    _f32(q_norm, k_norm, cos, sin, q_head_scale, bias)
    assert q_head_scale is None or q_head_scale.numel() == heads
    assert src.dtype == torch.float32 and src.stride(1) == 1 and k_pool.dtype == v_pool.dtype
    assert k_pool.is_contiguous() and v_pool.is_contiguous()
    _, g, bs, d = k_pool.shape
    _, gv, _, dv = v_pool.shape
    assert rot_n == 0 or (cos.shape[1] == rot_n // 2 and sin.shape == cos.shape)
    assert q_norm is None or q_norm.numel() == (d if head_norm else heads * d)
    assert k_norm is None or k_norm.numel() == (d if head_norm else g * d)
    assert bias is None or bias.numel() == (heads + g) * d + gv * dv
    t = src.shape[0]
    q = _new(src, torch.float32, t, heads * d)
    with _k("qk_norm_rope_kv_write"):
        check(_lib().b200_qk_norm_rope_kv_write(src, src.stride(0), q_col0, k_col0, v_col0, q_norm, k_norm,
                                                      float(eps), int(rot_n), 1 if rot_half else 0, cos, sin,
                                                      meta.tok_pos, meta.slot_mapping, q, k_pool,
                                                      v_pool, _edt(k_pool), t, heads, g, gv, d, dv, bs, q_head_scale,
                                                      1 if head_norm else 0, bias),
              "b200_qk_norm_rope_kv_write")
    return q


# ------------------------------------------------------------------ dual-norm parallel decoders (window + pooled-block attention
# beside a gated linear recurrence)
def embed_rmsnorm(tokens, table, w, eps: float):
    """tokens int32 [T] -> fp32 [T, W] = RMS norm of table[token], times w."""
    _f32(w)
    assert tokens.dtype == torch.int32 and table.is_contiguous()
    t, (v, width) = tokens.numel(), table.shape
    out = _new(table, torch.float32, t, width)
    with _k("embed_rmsnorm"):
        check(_lib().b200_embed_rmsnorm(tokens, table, _edt(table), w, float(eps), out, t, width, v), "b200_embed_rmsnorm")
    return out


def scaled_add_rmsnorm2(x, eps: float, *, y1=None, c1: float = 1.0, y2=None, c2: float = 1.0, y3=None, nsum: int = 1, y3_weight=None,
                        c3: float = 1.0, add_rows=None, add_vec=None, w1=None, w2=None, out_dtype=None):
    """x += c1 y1 + c2 y2 + c3 sum_k y3_weight[t, k] y3[t nsum + k] + add_rows + add_vec, in place (fp32; every term optional);
    returns (RMS norm of x times w1, the same times w2) in out_dtype, None for a weight that is not given."""
    _f32(x, y3, y3_weight, add_rows, add_vec, w1, w2)
    t, width = x.shape
    for y in (y1, y2):
        assert y is None or (y.dtype == torch.float32 and y.stride(1) == 1 and y.shape == (t, width))
    assert y3 is None or (y3.shape == (t * nsum, width) and (y3_weight is None or y3_weight.numel() == t * nsum))
    assert add_rows is None or add_rows.shape == (t, width)
    assert add_vec is None or add_vec.numel() == width
    o1 = _new(x, out_dtype, t, width) if w1 is not None else None
    o2 = _new(x, out_dtype, t, width) if w2 is not None else None
    with _k("scaled_add_rmsnorm2"):
        check(_lib().b200_scaled_add_rmsnorm2(x, y1, y1.stride(0) if y1 is not None else 0, float(c1), y2,
                                                    y2.stride(0) if y2 is not None else 0, float(c2), y3, int(nsum),
                                                    y3_weight, float(c3), add_rows, add_vec, w1, o1,
                                                    w2, o2, float(eps), _edt(out_dtype) if out_dtype is not None else F32,
                                                    t, width), "b200_scaled_add_rmsnorm2")
    return o1, o2


def kv_pool_mean(k_pool, v_pool, pk_pool, pv_pool, block_table, meta, pool: int):
    """For every block of `pool` positions that the step's portions close: the mean of the block's cached key rows and value rows
    -> the pooled pools [num_blocks, G, ceil(block_size / pool), D | Dv] (entry of a block: page of its last position)."""
    _, g, bs, d = k_pool.shape
    _, gv, _, dv = v_pool.shape
    ppb = -(-bs // pool)
    assert pk_pool.shape == (k_pool.shape[0], g, ppb, d) and pv_pool.shape == (v_pool.shape[0], gv, ppb, dv)
    assert pk_pool.dtype == k_pool.dtype == v_pool.dtype == pv_pool.dtype and pk_pool.is_contiguous() and pv_pool.is_contiguous()
    assert block_table.dtype == torch.int32 and block_table.stride(1) == 1
    with _k("kv_pool_mean"):
        check(_lib().b200_kv_pool_mean(k_pool, v_pool, pk_pool, pv_pool, _edt(k_pool), block_table,
                                             block_table.stride(0), meta.seq_start, meta.seq_slot, meta.seq_pos0,
                                             meta.num_seqs, meta.num_tokens, g, gv, d, dv, bs, int(pool)),
              "b200_kv_pool_mean")


_GATED_SEGS = {"0": False, "1": True}.get(os.environ.get("B200_GATED_SEGS", ""))
GATED_SEGS_MAX_CTAS = 600  # whole-portion CTAs (16 value columns x head x sequence; about four per SM) below which long portions run as segments


def gated_scan(proj, q_col0: int, f_col0: int, v_col0: int, f_bias, lower, state, meta, heads: int, dim: int, vdim: int):
    """Gated linear recurrence S <- diag(f) S + (1 - f) v^T, o = S^T q per head over a ragged batch.  Raw q / f / v are the columns
    q_col0 / f_col0 / v_col0 of the fp32 rows proj; q = silu(raw), f = lower + (1 - lower) sigmoid(raw + f_bias) are written back
    IN PLACE.  state fp32 [slots, H, vdim, dim] (transposed) updated in place; returns o fp32 [T, H * vdim].  When the step
    carries a segment list (meta.scan_segs: some portion is long) the segments run in parallel from start states that an
    elementwise pass chains together."""
    _f32(f_bias, lower, state)
    assert proj.dtype == torch.float32 and proj.stride(1) == 1 and state.shape[1:] == (heads, vdim, dim)
    assert f_bias.numel() == heads * dim == lower.numel()
    t = proj.shape[0]
    out = _new(proj, torch.float32, t, heads * vdim)
    with _k("gated_scan_prep"):
        check(_lib().b200_gated_scan_prep(proj, proj.stride(0), q_col0, f_col0, heads * dim, f_bias, lower, t), "b200_gated_scan_prep")
    segs = getattr(meta, "scan_segs", None)
    nseg = meta.num_segs if segs is not None else 0
    if _GATED_SEGS is not None:  # A/B aid: B200_GATED_SEGS=0 never cuts portions, =1 always does when the step has a list
        nseg = nseg if _GATED_SEGS else 0
    elif -(-vdim // 16) * heads * meta.num_seqs >= GATED_SEGS_MAX_CTAS:
        nseg = 0  # whole portions already give every SM its CTAs: the two passes of the segment scheme would only add work
    seg_state = seg_decay = None
    if nseg:
        seg_state = _new(proj, torch.float32, nseg, heads, vdim, dim)
        seg_decay = _new(proj, torch.float32, nseg, heads, dim)
    with _k("gated_scan"):
        check(_lib().b200_gated_scan(proj, proj.stride(0), q_col0, f_col0, v_col0, state, meta.seq_start,
                                  meta.seq_slot, meta.seq_pos0, out, meta.num_seqs, heads, dim, vdim,
                                  segs if nseg else 0, nseg, meta.scan_seq_seg0 if nseg else 0, seg_state,
                                  seg_decay), "b200_gated_scan")
    return out


# ------------------------------------------------------------------ post-layer-norm decoders (selective scan, matrix memory)
SEL_SEGS_MAX_CTAS = 592  # whole-portion CTAs of the selective scan (four per SM) below which long portions run as segments


def selective_scan(x, dt_raw, bc, b_col0: int, c_col0: int, z, a_log2, dt_bias, d_skip, state, meta):
    """Selective scan with a step size per channel: S[c, n] <- exp(dt A[c, n]) S[c, n] + dt x B[n], y = S . C + d_skip x, times
    silu(z) when z is given.  x [T, C] (bf16 | fp32); dt_raw fp32 [T, C] (any pitch), dt = softplus(dt_raw + dt_bias); B / C = columns
    b_col0 / c_col0 ([N] each) of the fp32 rows bc; z fp32 [T, C] view (any pitch) or None; a_log2 fp32 [C, N] = A log2(e);
    state fp32 [slots, C, N] updated in place.  Returns y [T, C] in x's type."""
    _f32(a_log2, dt_bias, d_skip, state)
    t, c = x.shape
    n = a_log2.shape[1]
    assert x.is_contiguous() and state.shape[1:] == (c, n) == a_log2.shape and dt_bias.numel() == c == d_skip.numel()
    for r in (dt_raw, bc, z):
        assert r is None or (r.dtype == torch.float32 and r.stride(1) == 1 and r.shape[0] == t)
    assert dt_raw.shape[1] >= c and bc.shape[1] >= max(b_col0, c_col0) + n and (z is None or z.shape[1] >= c)
    out = torch.empty_like(x)
    segs = getattr(meta, "scan_segs", None)
    nseg = meta.num_segs if segs is not None else 0
    lanes = 4 if n <= 64 else 8 if n <= 128 else 16  # lanes that share a channel (256 threads per CTA)
    if -(-c // (256 // lanes)) * meta.num_seqs >= SEL_SEGS_MAX_CTAS:
        nseg = 0
    seg_state = seg_dt = None
    if nseg:
        seg_state = _new(x, torch.float32, nseg, c, n)
        seg_dt = _new(x, torch.float32, nseg, c)
    with _k("selective_scan"):
        check(_lib().b200_selective_scan(x, _edt(x), dt_raw, dt_raw.stride(0), bc, bc.stride(0), b_col0, c_col0,
                                               z, z.stride(0) if z is not None else 0, a_log2, dt_bias,
                                               d_skip, state, meta.seq_start, meta.seq_slot,
                                               meta.seq_pos0, out, meta.num_seqs, c, n, segs if nseg else 0, nseg,
                                               meta.scan_seq_seg0 if nseg else 0, seg_state, seg_dt, meta.max_new),
              "b200_selective_scan")
    return out


def matrix_memory(proj, q_col0: int, k_col0: int, v_col0: int, i_col0: int, f_col0: int, i_bias, f_bias, cap: float, state, m_state,
                  meta, heads: int, dim: int, vdim: int):
    """Matrix memory with exponential input gates over a ragged batch: q / k / v and the raw gates are columns of the fp32 rows proj.
    state fp32 [slots, H, vdim + 1, dim] (the last column is the normaliser) and m_state fp32 [slots, H] (running maximum) are
    updated in place.  Returns (S^T q [T, H * vdim], n . q [T, H], exp(-m) [T, H]), q unscaled."""
    _f32(i_bias, f_bias, state, m_state)
    assert proj.dtype == torch.float32 and proj.stride(1) == 1 and state.shape[1:] == (heads, vdim + 1, dim)
    assert i_bias.numel() == heads == f_bias.numel() and m_state.shape[1:] == (heads,)
    t = proj.shape[0]
    coef = _new(proj, torch.float32, t, heads, 2)
    floor = _new(proj, torch.float32, t, heads)
    out = _new(proj, torch.float32, t, heads * vdim)
    out_n = _new(proj, torch.float32, t, heads)
    with _k("matrix_memory_gates"):
        check(_lib().b200_matrix_memory_gates(proj, proj.stride(0), i_col0, f_col0, i_bias, f_bias, float(cap),
                                           m_state, meta.seq_start, meta.seq_slot, meta.seq_pos0, coef,
                                           floor, meta.num_seqs, heads), "b200_matrix_memory_gates")
    segs = getattr(meta, "scan_segs", None)
    nseg = meta.num_segs if segs is not None else 0
    if -(-(vdim + 1) // 16) * heads * meta.num_seqs >= GATED_SEGS_MAX_CTAS:
        nseg = 0
    seg_state = seg_decay = None
    if nseg:
        seg_state = _new(proj, torch.float32, nseg, heads, vdim + 1, dim)
        seg_decay = _new(proj, torch.float32, nseg, heads, dim)
    with _k("matrix_memory_scan"):
        check(_lib().b200_matrix_memory_scan(proj, proj.stride(0), q_col0, k_col0, v_col0, coef, state,
                                          meta.seq_start, meta.seq_slot, meta.seq_pos0, out, out_n,
                                          meta.num_seqs, heads, dim, vdim, segs if nseg else 0, nseg,
                                          meta.scan_seq_seg0 if nseg else 0, seg_state, seg_decay),
              "b200_matrix_memory_scan")
    return out, out_n, floor


def matrix_memory_out(o, nq, floor, scale: float, gate_src, gate_col0: int, w, eps: float, heads: int, out_dtype):
    """u = scale o / (max(|scale nq|, floor) + 1e-6) per head, then u / rms(u) * w * sigmoid(gate) -> [T, H * P] in out_dtype."""
    _f32(o, nq, floor, w)
    assert gate_src.dtype == torch.float32 and gate_src.stride(1) == 1
    t, hp = o.shape
    assert w.numel() == hp
    out = _new(o, out_dtype, t, hp)
    with _k("matrix_memory_out"):
        check(_lib().b200_matrix_memory_out(o, nq, floor, float(scale), gate_src, gate_src.stride(0),
                                                  gate_col0, w, float(eps), out, _edt(out), t, heads, hp // heads), "b200_matrix_memory_out")
    return out


def postln_residual(x, alpha: float, w, eps: float, *, y1=None, w1=None, y2=None, w2=None, c: float = 1.0, vec=None, out_dtype=None,
                    store: bool = True):
    """u = alpha x + vec + c (N(y1) w1 + N(y2) w2) with N = division by the row's RMS (y2 None: u = alpha x + vec + c y1, every term
    optional), then a layer norm without bias: (u - mean) / sqrt(var + eps) * w -> x in place (store) and, in out_dtype, the
    returned rows (None without out_dtype)."""
    _f32(x, w, w1, w2, vec)
    t, width = x.shape
    for y in (y1, y2):
        assert y is None or (y.dtype == torch.float32 and y.stride(1) == 1 and y.shape == (t, width))
    assert w.numel() == width and (vec is None or vec.numel() == width)
    out = _new(x, out_dtype, t, width) if out_dtype is not None else None
    with _k("postln_residual[2]" if y2 is not None else "postln_residual"):
        check(_lib().b200_postln_residual(x, float(alpha), y1, y1.stride(0) if y1 is not None else 0, w1,
                                                y2, y2.stride(0) if y2 is not None else 0, w2, float(c), vec,
                                                w, float(eps), 1 if store else 0, out,
                                                _edt(out_dtype) if out_dtype is not None else F32, t, width),
              "b200_postln_residual")
    return out


def bias_act(src, col0: int, n: int, bias, act: int, out_dtype):
    """act(columns [col0, col0 + n) of the fp32 rows src + bias) -> [T, n] in out_dtype; act = ACT_NONE | ACT_RELU2; bias may be None."""
    _f32(bias)
    assert src.dtype == torch.float32 and src.stride(1) == 1 and (bias is None or bias.numel() == n)
    t = src.shape[0]
    out = _new(src, out_dtype, t, n)
    with _k("bias_act[relu2]" if act == ACT_RELU2 else "bias_act"):
        check(_lib().b200_bias_act(src, src.stride(0), col0, n, bias, int(act), out, _edt(out), t),
              "b200_bias_act")
    return out


# ------------------------------------------------------------------ hyper-connected decoders (several copies of the residual stream)
def hyper_embed(tokens, table, streams: int, read, w, eps: float):
    """tokens int32 [T] -> (x fp32 [T, streams, W], every copy = table[token]; the RMS norm of sum_s read[s] x_s times w in the
    table's type: the first sublayer's input)."""
    _f32(read, w)
    assert tokens.dtype == torch.int32 and table.is_contiguous() and read.numel() == streams
    t, (v, width) = tokens.numel(), table.shape
    x = _new(table, torch.float32, t, streams, width)
    out = _new(table, table.dtype, t, width)
    with _k("hyper_embed"):
        check(_lib().b200_hyper_embed(tokens, table, _edt(table), x, streams, read, w, float(eps),
                                            out, t, width, v), "b200_hyper_embed")
    return x, out


def hyper_residual(x, mix, write, read, w, eps: float, *, y1=None, y2=None, nsum: int = 1, y2_weight=None, out_dtype, store: bool = True):
    """One sublayer's output joins the copies x fp32 [T, S, W]: with y = y1 + sum_c y2_weight[t, c] y2[t nsum + c],
    x_d <- sum_s mix[s, d] x_s + write[d] y (in place unless store is False); returns the RMS norm of sum_d read[d] x_d of the new
    copies, times w, in out_dtype (the next sublayer's input)."""
    _f32(x, mix, write, read, w, y2, y2_weight)
    t, s, width = x.shape
    assert mix.shape == (s, s) and write.numel() == s and read.numel() == s and w.numel() == width
    assert y1 is None or (y1.dtype == torch.float32 and y1.stride(1) == 1 and y1.shape == (t, width))
    assert y2 is None or (y2.shape == (t * nsum, width) and (y2_weight is None or y2_weight.numel() == t * nsum))
    out = _new(x, out_dtype, t, width)
    with _k("hyper_residual" + ("" if y2 is None else "[experts]")):
        check(_lib().b200_hyper_residual(x, s, y1, y1.stride(0) if y1 is not None else 0, y2, int(nsum),
                                               y2_weight, mix, write, read, w, float(eps),
                                               1 if store else 0, out, _edt(out), t, width), "b200_hyper_residual")
    return out
