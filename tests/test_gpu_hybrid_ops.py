"""GPU: every mechanism of the hybrid decoder alone, against the plain restatement in oracle/pumopel_ref.py (fp64).
Sizes are deliberately awkward (odd widths, sizes that are not multiples of a warp or a page, top > 1, groups != heads)."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _ops():
    from vllm_neuron_b200 import ops

    return ops


def _meta(entries, blocks, bs=8):
    from vllm_neuron_b200.hybrid import StepMeta

    return StepMeta.build(entries, blocks, bs, DEV)


def _close(got, want, tol):
    got, want = got.double().cpu(), want.double().cpu()
    err = (got - want).abs().max().item() / max(want.abs().max().item(), 1e-30)
    assert err < tol, err


def test_dyt_norm_and_fused_residual():
    ops = _ops()
    g = torch.Generator().manual_seed(0)
    T, W, top = 7, 50, 3
    x, y, y2 = (torch.randn(n, W, generator=g) * 2 for n in (T, T * top, T))
    w1, b1, w2, b2 = (torch.randn(W, generator=g) for _ in range(4))
    a1, a2 = 0.7, 1.3
    for odt, tol in ((torch.float32, 1e-6), (torch.bfloat16, 6e-3)):
        _close(ops.dyt_norm(x.to(DEV), w1.to(DEV), b1.to(DEV), a1, odt), torch.tanh(a1 * x.double()) * w1 + b1, tol)
        xd = x.to(DEV).clone()
        h = ops.dyt_residual(xd, y.to(DEV), (w1.to(DEV), b1.to(DEV), a1), (w2.to(DEV), b2.to(DEV), a2), odt, y2=y2.to(DEV), nsum=top)
        s = y.double().view(T, top, W).sum(1) + y2
        xr = x.double() + torch.tanh(a1 * s) * w1 + b1
        _close(xd, xr, 1e-6)                                  # the residual stream stays fp32 in both modes
        _close(h, torch.tanh(a2 * xr) * w2 + b2, tol)
    xd = x.to(DEV).clone()
    assert ops.dyt_residual(xd, y[:T].contiguous().to(DEV), (w1.to(DEV), b1.to(DEV), a1)) is None
    _close(xd, x.double() + torch.tanh(a1 * y[:T].double()) * w1 + b1, 1e-6)


@pytest.mark.parametrize("groups", [1, 3])
def test_gated_group_rmsnorm_gate_before_norm(groups):
    from oracle.pumopel_ref import rms_unit

    ops = _ops()
    g = torch.Generator().manual_seed(1)
    T, inner, eps = 5, 3 * 22, 1e-3
    y, w = torch.randn(T, inner, generator=g), torch.randn(inner, generator=g)
    zsrc = torch.randn(T, inner + 9, generator=g)            # z = the first `inner` columns of wider rows
    z = zsrc[:, :inner].double()
    want = rms_unit((y.double() * F.silu(z)).view(T, groups, -1), eps).reshape(T, inner) * w
    _close(ops.gated_group_rmsnorm(y.to(DEV), zsrc.to(DEV), w.to(DEV), groups, eps, torch.float32), want, 2e-6)
    wrong = rms_unit(y.double().view(T, groups, -1), eps).reshape(T, inner) * w * F.silu(z)   # gate after the norm
    assert (want - wrong).abs().max() > 0.05


def test_clamped_glu_limits():
    ops = _ops()
    g = torch.Generator().manual_seed(2)
    T, ff, limit = 6, 37, 1.25
    gu = torch.randn(T, 2 * ff, generator=g) * 3               # many values beyond +-limit
    gate, up = gu[:, :ff].double().clamp(max=limit), gu[:, ff:].double().clamp(-limit, limit)
    _close(ops.clamped_glu(gu.to(DEV), limit, torch.float32), gate * torch.sigmoid(1.702 * gate) * (up + 1), 2e-6)


@pytest.mark.parametrize("taps", [1, 2, 4, 5])
def test_causal_conv_ragged_portions_and_slot_reuse(taps):
    """Three sequences advance by portions of 1, 2 and more tokens per step; a slot is then handed to a NEW sequence while it
    still holds the old one's inputs.  Every step's output must equal the whole-sequence convolution."""
    from oracle.pumopel_ref import causal_conv_silu

    ops = _ops()
    g = torch.Generator().manual_seed(3)
    C, col0, ld = 45, 6, 60
    cw, cb = torch.randn(C, taps, generator=g), torch.randn(C, generator=g)
    state = torch.full((4, max(taps - 1, 1), C), 7.0, device=DEV)  # garbage: a fresh sequence must not read it (one unused row when taps == 1)
    seqs = {s: torch.randn(n, ld, generator=g) for s, n in ((0, 11), (1, 4), (2, 9), (3, 6))}
    want = {s: causal_conv_silu(u[:, col0:col0 + C].double(), cw.double(), cb.double()) for s, u in seqs.items()}
    slot = {0: 2, 1: 0, 2: 3, 3: 0}                           # sequence 3 reuses sequence 1's slot
    plan = [[(0, 5), (1, 1), (2, 2)], [(0, 1), (1, 3), (2, 1)], [(0, 2), (2, 6), (3, 1)], [(0, 3), (3, 2)], [(3, 3)]]
    done = {s: 0 for s in seqs}
    for step in plan:
        entries = [(slot[s], done[s], n) for s, n in step]
        src = torch.cat([seqs[s][done[s]:done[s] + n] for s, n in step]).to(DEV)
        out = ops.causal_conv_silu(src, col0, C, cw.to(DEV), cb.to(DEV), state, _meta(entries, {slot[s]: [1] * 16 for s, _ in step}), torch.float32)
        o = 0
        for s, n in step:
            _close(out[o:o + n], want[s][done[s]:done[s] + n], 3e-6)
            o += n
            done[s] += n


SHORT_PLAN = ({0: 19, 1: 3, 2: 8}, [[(0, 7), (1, 1)], [(0, 1), (1, 2), (2, 2)], [(0, 11), (2, 6)]])
# portions of 256 tokens and more are cut into parallel segments of 128: ragged last segments (44, 1 and 15 tokens), a
# segmented portion that continues from a state left by an earlier segmented one, short sequences in the same step
LONG_PLAN = ({0: 700, 1: 3, 2: 300}, [[(0, 300), (1, 1)], [(0, 1), (1, 2), (2, 257)], [(0, 399), (2, 43)]])


@pytest.mark.parametrize("plan", [SHORT_PLAN, LONG_PLAN], ids=["short", "segmented"])
@pytest.mark.parametrize("H,G,P,N", [(4, 2, 5, 12), (3, 3, 40, 40), (2, 1, 33, 70), (2, 2, 100, 64), (1, 1, 70, 130)])
def test_selective_scan_ragged(H, G, P, N, plan):
    from oracle.pumopel_ref import selective_scan

    ops = _ops()
    g = torch.Generator().manual_seed(4)
    C = H * P + 2 * G * N
    a_log, dt_bias, d = torch.randn(H, generator=g) * 0.5, torch.randn(H, generator=g), torch.randn(H, generator=g)
    lens, plan = plan
    xbc = {s: torch.randn(n, C, generator=g) for s, n in lens.items()}
    dts = {s: torch.randn(n, H + 3, generator=g) * 2 for s, n in lens.items()}   # dt = columns 3.. of wider rows
    want = {}
    for s, n in lens.items():
        x = xbc[s][:, :H * P].double().view(n, H, P)
        B = xbc[s][:, H * P:H * P + G * N].double().view(n, G, N).repeat_interleave(H // G, 1)
        Cm = xbc[s][:, H * P + G * N:].double().view(n, G, N).repeat_interleave(H // G, 1)
        want[s] = selective_scan(x, B, Cm, dts[s][:, 3:].double(), dt_bias.double(), a_log.double(), d.double()).reshape(n, H * P)
    state = torch.full((3, H, P, N), 5.0, device=DEV)
    done = {s: 0 for s in lens}
    for step in plan:
        entries = [(s, done[s], n) for s, n in step]
        xs = torch.cat([xbc[s][done[s]:done[s] + n] for s, n in step]).to(DEV)
        ds = torch.cat([dts[s][done[s]:done[s] + n] for s, n in step]).to(DEV)
        meta = _meta(entries, {s: [1] * 128 for s, _ in step})
        assert (meta.scan_segs is not None) == (max(n for _, n in step) >= 2 * ops.SCAN_SEGMENT)
        y = ops.ssd_scan(xs, ds, 3, a_log.to(DEV), dt_bias.to(DEV), d.to(DEV), state, meta, H, P, N, G)
        o = 0
        for s, n in step:
            _close(y[o:o + n], want[s][done[s]:done[s] + n], 2e-5)
            o += n
            done[s] += n


def _attn_case(T, H, G, D, Dv, window, bs, *, spike=None, sink_val=None, seed=5):
    """Random q/k/v of one sequence; `spike` = (i, j, head): key j gets a score that dominates query i of that head."""
    g = torch.Generator().manual_seed(seed)
    q, k, v = torch.randn(T, H, D, generator=g), torch.randn(T, G, D, generator=g), torch.randn(T, G, Dv, generator=g)
    sink = torch.randn(H, generator=g) if sink_val is None else torch.full((H,), float(sink_val))
    if spike:
        i, j, h = spike
        k[j, h // (H // G)] = q[i, h] * 40.0 / q[i, h].norm() ** 2 * math.sqrt(D)   # score = 40 at scale 1/sqrt(D)
    return q, k, v, sink


def _run_attn(q, k, v, sink, window, bs, chunks, dtype=torch.float32):
    ops = _ops()
    T, H, D = q.shape
    G, Dv = k.shape[1], v.shape[2]
    nb = -(-T // bs)
    blocks = list(range(nb + 3, 3, -1))                        # descending, non-contiguous with the table order
    kp = torch.zeros(nb + 5, G, bs, D, dtype=dtype, device=DEV)
    vp = torch.zeros(nb + 5, G, bs, Dv, dtype=dtype, device=DEV)
    bt = torch.zeros(3, nb, dtype=torch.int32, device=DEV)
    bt[1, :nb] = torch.tensor(blocks, dtype=torch.int32)
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], 1).to(DEV)
    outs, pos = [], 0
    for n in chunks:
        m = _meta([(1, pos, n)], {1: blocks}, bs)
        rows = qkv[pos:pos + n].contiguous()
        ops.kv_write_vmix(rows, H * D, H * D + G * D, kp, vp, m.slot_mapping)
        outs.append(ops.swa_sink_attn(rows, H, kp, vp, bt, m, sink.to(DEV), 1 / math.sqrt(D), window))
        pos += n
    return torch.cat(outs)


@pytest.mark.parametrize("chunks", [[70], [64, 1, 1, 1, 1, 1, 1], [2, 31, 30, 7]])
def test_attention_window_edges_sink_and_pages(chunks):
    """Window 17 over pages of 8 tokens: the last query's dominant key sits just INSIDE the window (it must take the output)
    or just OUTSIDE (it must not show at all); the same through decoded tokens and ragged portions."""
    from oracle.pumopel_ref import sink_window_attention

    T, H, G, D, Dv, window, bs = 70, 6, 2, 24, 40, 17, 8
    for j, inside in ((T - window, True), (T - 1 - window, False), (T - 1, True), (0, False)):
        q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs, spike=(T - 1, j, 4))
        want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 1 / math.sqrt(D), window)
        got = _run_attn(q, k, v, sink, window, bs, chunks)
        _close(got, want, 2e-5)
        head = got[T - 1].view(H, Dv)[4].cpu()
        assert ((head - v[j, 4 // (H // G)]).abs().max() < 1e-3) == inside
    # a sink that dominates every score empties the output; a sink far below changes nothing
    q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs, sink_val=60.0)
    assert _run_attn(q, k, v, sink, window, bs, chunks).abs().max() < 1e-6
    q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs, sink_val=-60.0)
    want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 1 / math.sqrt(D), window)
    _close(_run_attn(q, k, v, sink, window, bs, chunks), want, 2e-5)
    # bf16 pools: same mask, looser numbers
    q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs)
    want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 1 / math.sqrt(D), window)
    _close(_run_attn(q, k, v, sink, window, bs, chunks, torch.bfloat16), want, 3e-2)


@pytest.mark.parametrize("H,G,D,Dv", [(8, 2, 24, 40), (4, 2, 32, 16), (6, 2, 20, 70), (16, 4, 64, 136)])
def test_warp_attention_shares_key_rows_between_query_heads(H, G, D, Dv):
    """Steps with many tokens on the CUDA-core kernel (fp32 pools; bf16 pools with head sizes the tensor-core kernel does not
    take): one CTA serves 4 or 2 query heads of a kv head (8/2, 16/4 and 4/2 heads), or 1 (6/2).  A dominant key just inside
    and just outside the window of the last query, per head."""
    from oracle.pumopel_ref import sink_window_attention

    T, window, bs = 420, 50, 8
    for head in (0, H - 1):
        for j, inside in ((T - window, True), (T - 1 - window, False)):
            q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs, spike=(T - 1, j, head))
            want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 1 / math.sqrt(D), window)
            got = _run_attn(q, k, v, sink, window, bs, [400, 20])
            _close(got, want, 2e-5)
            row = got[T - 1].view(H, Dv)[head].cpu()
            assert ((row - v[j, head // (H // G)]).abs().max() < 1e-3) == inside
    if D % 16 or Dv % 16:
        q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs)
        want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 1 / math.sqrt(D), window)
        _close(_run_attn(q, k, v, sink, window, bs, [T], torch.bfloat16), want, 3e-2)


@pytest.mark.parametrize("H,G,D,Dv", [(8, 2, 128, 128), (4, 4, 64, 64), (5, 1, 128, 64)])
@pytest.mark.parametrize("window", [100, 128, 1 << 30])
def test_long_prompts_with_a_sink_on_tcgen05(H, G, D, Dv, window):
    """Portions of 128 tokens and more (one of them the second part, one short) in tiles of 128 rows: the sink joins every row's denominator once,
    whether it lies above or below all scores, and a dominant key counts just inside the window and not just outside."""
    from oracle.pumopel_ref import sink_window_attention

    ops = _ops()
    T, scale = 420, 1 / math.sqrt(D)
    bf = lambda t: t.bfloat16().float()  # noqa: E731
    for sink_val in (None, 4.0, -60.0, 60.0):
        q, k, v, sink = _attn_case(T, H, G, D, Dv, window, 32, sink_val=sink_val)
        with ops.kernel_timer() as kt:
            got = _run_attn(bf(q), bf(k), bf(v), sink, window, 32, [150, 200, 70], torch.bfloat16)
        assert any(n.startswith("swa_sink_attn_prefill_tc") for n in kt.summary())
        if sink_val == 60.0:
            assert got.abs().max() < 1e-6
            continue
        want = sink_window_attention(bf(q).double(), bf(k).double(), bf(v).double(), sink.double(), scale, window)
        _close(got, want, 2.0**-8)  # weights in two bf16 terms: the output's rounding is what is left
    if window < T:
        for j, inside in ((T - window, True), (T - 1 - window, False)):
            q, k, v, sink = _attn_case(T, H, G, D, Dv, window, 32, spike=(T - 1, j, H - 1))
            head = _run_attn(bf(q), bf(k), bf(v), sink, window, 32, [T], torch.bfloat16)[T - 1].view(H, Dv)[H - 1].float().cpu()
            assert ((head - bf(v)[j, (H - 1) // (H // G)]).abs().max() < 1e-2) == inside


@pytest.mark.parametrize("D,window", [(128, 100), (64, 1 << 30)])
def test_sink_on_tcgen05_keeps_the_weights_precision(D, window):
    """fp32 outputs of bf16 operands, against 64 bits: weights in two bf16 terms leave 2^-17 of a weight, exponentials and fp32 sums the rest;
    2^-13 of the largest value, where one term leaves up to 2^-9."""
    from oracle.pumopel_ref import sink_window_attention

    ops = _ops()
    T, H, G, bs = 420, 4, 2, 32
    q, k, v, sink = _attn_case(T, H, G, D, D, window, bs, seed=9)
    q, k, v = (x.bfloat16() for x in (q, k, v))
    nb = -(-T // bs)
    pages = lambda x: torch.cat([x, x.new_zeros(nb * bs - T, G, D)]).view(nb, bs, G, D).transpose(1, 2).contiguous().to(DEV)  # noqa: E731
    meta = _meta([(0, 0, T)], {0: list(range(nb))}, bs)
    table = torch.arange(nb, dtype=torch.int32, device=DEV)[None]
    got = ops.swa_sink_attn(q.float().reshape(T, H * D).to(DEV), H, pages(k), pages(v), table, meta, sink.to(DEV), D**-0.5, window, out_f32=True)
    want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), D**-0.5, window)
    assert (got.double().cpu() - want).abs().max() <= 2.0**-13 * v.double().abs().max()


@pytest.mark.parametrize("chunks", [[150], [16, 64, 3, 67], [33, 1, 1, 17, 98]])
def test_tensor_core_prompt_attention_edges(chunks):
    """bf16 pools, head sizes 32 / 48: portions of 16 tokens or more run on the mma.sync kernel (64-row tiles, 32-key tiles
    over pages of 8), shorter ones on the CUDA-core kernel.  A dominant key just inside / outside the window of a query in
    the middle of a tile and of the last query, against the restatement on the bf16-rounded q / k / v."""
    from oracle.pumopel_ref import sink_window_attention

    T, H, G, D, Dv, window, bs = 150, 4, 2, 32, 48, 37, 8
    for i in (T - 1, 100, 40):
        for j, inside in ((i - window + 1, True), (i - window, False), (i, True)):
            q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs, spike=(i, j, 3), seed=11)
            qb, kb, vb = (x.bfloat16().float() for x in (q, k, v))
            want = sink_window_attention(qb.double(), kb.double(), vb.double(), sink.double(), 1 / math.sqrt(D), window)
            got = _run_attn(qb, kb, vb, sink, window, bs, chunks, torch.bfloat16)
            _close(got, want, 1.5e-2)
            head = got[i].float().view(H, Dv)[3].cpu()
            assert ((head - vb[j, 3 // (H // G)]).abs().max() < 3e-2) == inside, (i, j)


@pytest.mark.parametrize("bs", [32, 64, 8])
@pytest.mark.parametrize("window", [37, 64, 96, 1])
def test_decoded_token_window_over_pages(window, bs):
    """Decoded tokens, window tiles that start on pages (32 and 64 rows) and at the window's first key (8): windows that begin at a page's
    first row, one to either side of it and inside it, a dominant key just inside and just outside.  Weights and outputs are rounded to
    bf16 (2^-9 each) and the weights sum to at most 1: 2^-8 of the largest value."""
    from oracle.pumopel_ref import sink_window_attention

    H, G, D, Dv = 4, 2, 32, 48
    for T in (132, window + 63, window + 64, window + 65):
        i = T - 2
        for j, inside in ((i - window + 1, True), (i - window, False)):
            q, k, v, sink = _attn_case(T, H, G, D, Dv, window, bs, spike=(i, j, 3), seed=T)
            q, k, v = (x.bfloat16().float() for x in (q, k, v))
            want = sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 1 / math.sqrt(D), window)[-4:]
            got = _run_attn(q, k, v, sink, window, bs, [T - 4, 1, 1, 1, 1], torch.bfloat16)[-4:]
            assert (got.double().cpu().view(4, H, Dv) - want.view(4, H, Dv)).abs().max() <= 2.0**-8 * v.abs().max()
            assert ((got[2].float().view(H, Dv)[3].cpu() - v[j, 1]).abs().max() < 3e-2) == inside, (T, j)


def test_far_key_among_hundreds_without_window():
    """No window: key 3 of 400 must still decide the last query (pages of 32)."""
    from oracle.pumopel_ref import sink_window_attention

    T, H, G, D, Dv = 400, 2, 2, 16, 8
    q, k, v, sink = _attn_case(T, H, G, D, Dv, 1 << 30, 32, spike=(T - 1, 3, 1))
    got = _run_attn(q, k, v, sink, 1 << 30, 32, [T - 5, 1, 1, 1, 1, 1])
    _close(got, sink_window_attention(q.double(), k.double(), v.double(), sink.double(), 0.25, T + 1), 2e-5)
    assert (got[T - 1].view(H, Dv)[1].cpu() - v[3, 1]).abs().max() < 1e-3


def test_value_mixing_is_what_gets_cached():
    ops = _ops()
    g = torch.Generator().manual_seed(6)
    T, G, D, Dv, bs, lam = 5, 2, 4, 6, 4, 0.3
    rows = torch.randn(T, 3 + G * D + G * Dv, generator=g).to(DEV)
    rows2 = torch.randn(T, 3 + G * D + G * Dv, generator=g).to(DEV)
    m = _meta([(0, 0, T)], {0: [2, 1]}, bs)
    kp, vp = torch.zeros(3, G, bs, D, device=DEV), torch.zeros(3, G, bs, Dv, device=DEV)
    vf = torch.zeros(T, G * Dv, device=DEV)
    ops.kv_write_vmix(rows, 3, 3 + G * D, kp, vp, m.slot_mapping, v_first=vf, mode=1)
    v1 = rows[:, 3 + G * D:]
    assert torch.equal(vf, v1)
    ops.kv_write_vmix(rows2, 3, 3 + G * D, kp, vp, m.slot_mapping, v_first=vf, lam=lam, mode=2)
    want = ((1 - lam) * rows2[:, 3 + G * D:] + lam * v1).view(T, G, Dv)
    got = torch.stack([vp[[2, 1][t // bs], :, t % bs] for t in range(T)])
    _close(got, want, 1e-6)
    _close(torch.stack([kp[[2, 1][t // bs], :, t % bs] for t in range(T)]), rows2[:, 3:3 + G * D].view(T, G, D), 1e-7)


@pytest.mark.parametrize("E,top,shared", [(5, 2, 0), (16, 1, 24), (7, 3, 10)])
def test_moe_weight_on_the_input(E, top, shared):
    """Router + experts + shared expert against the restatement; the routing weight must scale the expert's INPUT (the
    clamps make that differ from scaling its output)."""
    from oracle.pumopel_ref import moe_ff
    from vllm_neuron_b200.hybrid import HybridConfig, HybridCausalLM, random_weights

    W, ff, limit, T = 40, 12, 0.8, 45
    cfgd = {"architecture": "Pumopel", "vocab": 16, "width": W, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "layers": [{"type": "attention", "mixer": {"heads": 2, "kv_heads": 1, "dim": 8, "vdim": 8, "scale": 0.3, "mask": {"size": 4}},
                        "mlp": {"kind": "moe", "router": {"experts": E, "top": top}, "expert": {"ff": ff, "limit": limit},
                                "shared": {"ff": shared, "limit": 2 * limit} if shared else None}}]}
    cfg = HybridConfig.from_dict(cfgd)
    Wt = random_weights(cfg, seed=7, std=0.4)
    model = HybridCausalLM(cfg, Wt, num_blocks=4, max_num_seqs=1, max_model_len=64, device=DEV, dtype=torch.float32)
    h = torch.randn(T, W, generator=torch.Generator().manual_seed(8))
    pairs, sh = model._moe(model.layers[0], h.to(DEV))
    got = pairs.view(T, top, W).sum(1) + (sh if sh is not None else 0)
    W64 = {k: v.double() for k, v in Wt.items()}
    want = moe_ff(h.double(), W64, "l0.mlp.", cfgd["layers"][0]["mlp"])
    _close(got, want, 2e-5)
    idx, wt = _ops().moe_topk(model._linear(h.to(DEV), model.layers[0]["w_router"]), top)
    ties = torch.tensor([[1.0, 3.0, 3.0, -2.0, 3.0]], device=DEV)            # equal logits: the lower index first
    assert _ops().moe_topk(ties, 2)[0].tolist() == [[1, 2]]
    s = torch.sigmoid(h.double() @ W64["l0.mlp.router"].T)
    val, ref_idx = s.topk(top, dim=-1)
    assert torch.equal(idx.cpu().long(), ref_idx) and (wt.cpu().double() - val).abs().max() < 1e-6


def test_moe_wide_tiles_match_the_default_tiles():
    """Prompt-sized bf16 batch: experts with 128-row tiles (ragged tails, an expert that gets almost nothing) give the same
    pairs as the 32-row tiles, and both follow the restatement evaluated on the bf16-rounded operands."""
    from oracle.pumopel_ref import clamped_glu_expert

    ops = _ops()
    E, top, W, ff, T, limit = 5, 2, 64, 24, 700, 0.9
    g = torch.Generator().manual_seed(21)
    h = torch.randn(T, W, generator=g).bfloat16()
    w_gu = (0.3 * torch.randn(E, 2 * ff, W, generator=g)).bfloat16()
    w_dn = (0.3 * torch.randn(E, W, ff, generator=g)).bfloat16()
    logits = torch.randn(T, E, generator=g)
    logits[:, 3] -= 6.0                                     # expert 3 is chosen a handful of times at most
    idx, wt = ops.moe_topk(logits.to(DEV), top)
    hd, gud, dnd = h.to(DEV), w_gu.to(DEV), w_dn.to(DEV)
    assert ops.moe_wide_tiles(hd, gud, T * top) == 4 * ops.moe_tile_rows()
    assert ops.moe_wide_tiles(hd, gud, 10) is None and ops.moe_wide_tiles(hd.float(), gud.float(), T * top) is None
    wide = ops.moe_experts(hd, wt, ops.moe_align(idx, E, 4 * ops.moe_tile_rows()), gud, dnd, top, limit)
    base = ops.moe_experts(hd, wt, ops.moe_align(idx, E), gud, dnd, top, limit)
    assert torch.equal(wide, base)                          # same K order per row: the tile height changes nothing
    want = torch.zeros(T * top, W, dtype=torch.float64)
    for pair in range(T * top):
        e = int(idx.view(-1)[pair])
        x = (h[pair // top].float() * wt.view(-1)[pair].cpu()).bfloat16().double()   # the weight goes into the operand
        Wd = {"gate": w_gu[e, :ff].double(), "up": w_gu[e, ff:].double(), "down": w_dn[e].double()}
        want[pair] = clamped_glu_expert(x[None], Wd, "", limit)[0]
    _close(wide, want, 1e-2)                                # the activation between the two GEMMs is rounded to bf16


def test_linear_paths_agree_with_matmul():
    ops = _ops()
    g = torch.Generator().manual_seed(9)
    for m, n, k in ((45, 70, 20), (3, 774, 256), (300, 129, 288)):
        a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g)
        _close(ops.linear_simt(a.to(DEV), w.to(DEV)), a.double() @ w.double().T, 2e-6)
        ab, wb = a.bfloat16(), w.bfloat16()
        want = ab.double() @ wb.double().T
        _close(ops.linear_simt(ab.to(DEV), wb.to(DEV)), want, 2e-5)   # K % 8 == 0: tensor cores, fp32 accumulation
        if k % 8 == 0:
            _close(ops.gemm(ab.to(DEV), wb.to(DEV), out_dtype=torch.float32), want, 2e-5)


@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (8, 33, 36), (9, 31, 100), (32, 64, 64), (33, 65, 132), (130, 200, 1024), (5, 7, 30), (70, 66, 33)])
def test_fp32_linear_tiles(m, n, k):
    """fp32 rows at the edges of every tile (8, 32 and 64 rows), fewer k than a slice and ragged k; the last two take the kernel for
    rows that are no 16-byte pieces.  Bound: k roundings of fp32 sums of k products."""
    ops = _ops()
    g = torch.Generator().manual_seed(m * 1000 + n + k)
    a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g)
    got = ops.linear_simt(a.to(DEV), w.to(DEV)).double().cpu()
    assert ((got - a.double() @ w.double().T).abs() <= k * 2.0**-24 * (a.abs().double() @ w.abs().double().T)).all()


@pytest.mark.parametrize("m,n,k", [(97, 7233, 68), (33, 8, 36), (10, 13, 132), (301, 16, 1024), (7, 40, 100), (64, 64, 96)])
def test_fp32_linear_many_tiles_and_narrow_rows(m, n, k):
    """Batches of many tiles (64 x 32), fewer slices than stages, and a few outputs per row (a warp per two rows, an odd row left)."""
    test_fp32_linear_tiles(m, n, k)


@pytest.mark.parametrize("H,P,N,G", [(4, 128, 128, 2), (4, 64, 64, 4), (2, 64, 128, 1), (2, 128, 64, 2)])
@pytest.mark.parametrize("shift", [-2.0, -6.0])
@pytest.mark.parametrize("cut", [128, 150])
def test_ssd_scan_segments_as_matrix_products(H, P, N, G, shift, cut, monkeypatch):
    """Segments on the tensor cores: several, one and partial segments, a reused slot, short sequences (decoded tokens) beside them, fast
    and slow decays; a cut beyond the matrix form's 128 tokens walks token by token.  Bound: 1e-6 of the result's norm, eight fp32 ulps
    (bf16 inputs are exact on both sides)."""
    from oracle.pumopel_ref import selective_scan
    from vllm_neuron_b200.hybrid import StepMeta

    ops = _ops()
    monkeypatch.setattr(ops, "SCAN_SEGMENT", cut)
    g = torch.Generator().manual_seed(H * P + N)
    entries = [(0, 0, 2 * cut + 45), (1, 7, cut), (2, 40, 1), (3, 64, 33), (4, 0, 16), (5, 9, cut + 1)]
    T, slots, C = sum(e[2] for e in entries), len(entries), H * P + 2 * G * N
    xbc = torch.nn.functional.silu(torch.randn(T, C, generator=g)).bfloat16()
    raw = torch.randn(T, H, generator=g)
    a_log, bias, D = torch.log(0.5 + 1.5 * torch.rand(H, generator=g)), shift + 1.5 * torch.rand(H, generator=g), torch.randn(H, generator=g)
    state = 0.3 * torch.randn(slots, H, P, N, generator=g)
    meta = StepMeta.build(entries, {r: list(range(1 + 40 * r, 41 + 40 * r)) for r in range(slots)}, 32, torch.device(DEV))
    got_state = state.to(DEV)
    y = ops.ssd_scan(xbc.to(DEV), raw.to(DEV), 0, a_log.to(DEV), bias.to(DEV), D.to(DEV), got_state, meta, H, P, N, G).cpu()
    d, at = xbc.double(), 0
    for r, pos0, n in entries:
        x = d[at:at + n, :H * P].view(n, H, P)
        B, Cm = (d[at:at + n, o:o + G * N].view(n, G, N).repeat_interleave(H // G, 1) for o in (H * P, H * P + G * N))
        S0 = state[r].double().transpose(1, 2) if pos0 else None
        want = selective_scan(x, B, Cm, raw[at:at + n].double(), bias.double(), a_log.double(), D.double(), S0)
        got = y[at:at + n].double().view(n, H, P)
        assert (got - want).norm() <= 1e-6 * want.norm(), (r, n)
        # the new state, read out with unit vectors: one more token of zero step size
        dt = torch.nn.functional.softplus(raw[at:at + n].double() + bias.double())
        cum = -torch.exp(a_log.double()) * dt.cumsum(0)
        w = torch.exp(cum[-1] - cum) * dt
        S = torch.einsum("th,thp,thn->hpn", w, x, B) + (torch.exp(cum[-1])[:, None, None] * state[r].double() if pos0 else 0.0)
        assert (got_state[r].double().cpu() - S).norm() <= 1e-6 * S.norm(), (r, n)
        at += n


@pytest.mark.parametrize("H,P,N,G", [(2, 128, 128, 1), (2, 64, 64, 2)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_ssd_scan_segments_keep_what_is_not_finite_in_its_place(H, P, N, G, bad):
    """One infinite or NaN x in the middle of a block of tokens: earlier tokens, other columns and other heads are those of the clean run
    (its segment is walked token by token: 1e-6 of the norm), the column from that token on is not finite."""
    from vllm_neuron_b200.hybrid import StepMeta

    ops = _ops()
    g = torch.Generator().manual_seed(P)
    T, at, col, C = 300, 150, P + 3, H * P + 2 * G * N  # token 150: the seventh of a block of 16 in the second segment; head 1
    xbc = torch.nn.functional.silu(torch.randn(T, C, generator=g)).bfloat16()
    raw, a_log, bias, D = (torch.randn(*s, generator=g).to(DEV) for s in ((T, H), (H,), (H,), (H,)))
    meta = StepMeta.build([(0, 0, T)], {0: list(range(1, 11))}, 32, torch.device(DEV))

    def scan(x):
        state = torch.zeros(1, H, P, N, device=DEV)
        return ops.ssd_scan(x.to(DEV), raw, 0, a_log, bias, D, state, meta, H, P, N, G), state

    clean, clean_state = scan(xbc)
    x = xbc.clone()
    x[at, col] = bad
    y, state = scan(x)
    assert not torch.isfinite(y[at:, col]).any() and not torch.isfinite(state[0, 1, 3]).any()
    y[at:, col] = clean[at:, col]
    state[0, 1, 3] = clean_state[0, 1, 3]
    assert (y - clean).norm() <= 1e-6 * clean.norm() and (state - clean_state).norm() <= 1e-6 * clean_state.norm()


@pytest.mark.parametrize("entry", ["b200_ssd_scan", "b200_ssd_scan_mma"])
def test_ssd_scan_keeps_to_its_scratch(entry):
    """Scratch of exactly num_segs entries, as the header asks for, a long portion last: the memory behind it stays as it was, and the
    result is that of the wrapper, bit for bit from the entry that it calls; the other takes the sequential scan, whatever the cuts."""
    from vllm_neuron_b200 import _cabi
    from vllm_neuron_b200.hybrid import StepMeta

    ops = _ops()
    H, P, N, G = 4, 64, 128, 2
    g = torch.Generator().manual_seed(5)
    entries = [(0, 3, 40), (1, 0, 1), (2, 9, 300)]
    T, C = sum(e[2] for e in entries), H * P + 2 * G * N
    xbc = torch.nn.functional.silu(torch.randn(T, C, generator=g)).bfloat16().to(DEV)
    raw, a_log, bias, D = (torch.randn(*s, generator=g).to(DEV) for s in ((T, H), (H,), (H,), (H,)))
    state = 0.3 * torch.randn(3, H, P, N, generator=g).to(DEV)
    meta = StepMeta.build(entries, {r: list(range(1 + 10 * r, 11 + 10 * r)) for r in range(3)}, 32, torch.device(DEV))
    want_state = state.clone()
    want = ops.ssd_scan(xbc, raw, 0, a_log, bias, D, want_state, meta, H, P, N, G)
    v, size = meta.num_segs, H * P * N
    scratch, dts = torch.full(((v + 2) * size,), 7.5, device=DEV), torch.full((v * H + 64,), 7.5, device=DEV)
    y = torch.empty(T, H * P, device=DEV)
    assert getattr(_cabi.load(), entry)(xbc.data_ptr(), ops.BF16, C, raw.data_ptr(), H, 0, a_log.data_ptr(), bias.data_ptr(), D.data_ptr(),
                                        state.data_ptr(), meta.seq_start.data_ptr(), meta.seq_slot.data_ptr(), meta.seq_pos0.data_ptr(),
                                        y.data_ptr(), 3, H, P, N, G, meta.scan_segs.data_ptr(), v, meta.scan_seq_seg0.data_ptr(),
                                        scratch.data_ptr(), dts.data_ptr(), ops._stream()) == 0
    assert (scratch[v * size:] == 7.5).all() and (dts[v * H:] == 7.5).all()
    assert (y - want).norm() <= 1e-6 * want.norm() and (state - want_state).norm() <= 1e-6 * want_state.norm()
    assert torch.equal(y, want) == (entry == "b200_ssd_scan_mma")


def test_ssd_scan_writes_outputs_on_any_boundary():
    """Outputs that start one float after a 16-byte boundary: those of the wrapper's aligned ones, and nothing beside them."""
    from vllm_neuron_b200 import _cabi
    from vllm_neuron_b200.hybrid import StepMeta

    ops = _ops()
    H, P, N, G, T = 2, 64, 64, 1, 300
    g = torch.Generator().manual_seed(6)
    C = H * P + 2 * G * N
    xbc = torch.nn.functional.silu(torch.randn(T, C, generator=g)).bfloat16().to(DEV)
    raw, a_log, bias, D = (torch.randn(*s, generator=g).to(DEV) for s in ((T, H), (H,), (H,), (H,)))
    meta = StepMeta.build([(0, 0, T)], {0: list(range(1, 11))}, 32, torch.device(DEV))
    states = torch.zeros(2, 1, H, P, N, device=DEV)
    want = ops.ssd_scan(xbc, raw, 0, a_log, bias, D, states[0], meta, H, P, N, G)
    scratch, dts, buf = torch.empty(meta.num_segs, H, P, N, device=DEV), torch.empty(meta.num_segs, H, device=DEV), torch.full((T * H * P + 2,), 7.0, device=DEV)
    assert _cabi.load().b200_ssd_scan_mma(xbc.data_ptr(), ops.BF16, C, raw.data_ptr(), H, 0, a_log.data_ptr(), bias.data_ptr(), D.data_ptr(),
                                          states[1].data_ptr(), meta.seq_start.data_ptr(), meta.seq_slot.data_ptr(), meta.seq_pos0.data_ptr(),
                                          buf[1:].data_ptr(), 1, H, P, N, G, meta.scan_segs.data_ptr(), meta.num_segs,
                                          meta.scan_seq_seg0.data_ptr(), scratch.data_ptr(), dts.data_ptr(), ops._stream()) == 0
    y = buf[1:-1].view(T, H * P)
    assert (y - want).norm() <= 1e-6 * want.norm() and (states[1] - states[0]).norm() <= 1e-6 * states[0].norm() and buf[0] == 7 and buf[-1] == 7


@pytest.mark.parametrize("counts", [(300, 0, 129, 128, 1), (3, 40, 0, 32, 33), (0, 0, 0, 0, 7)])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("act", ["clamped", "silu"])
def test_moe_experts_on_pairs(counts, wide, act):
    """Experts with whole pair-kernel tiles (256 outputs, 128 hidden channels): tiles that fill, overflow and merge, experts without
    rows, more output tiles than one wave of pairs.  The hidden activation is rounded to bf16: 2^-9 of it, 1e-2 of the norm at most."""
    ops = _ops()
    E, W, ff = len(counts), 1024, 384
    g = torch.Generator().manual_seed(sum(counts))
    T = sum(counts)
    idx = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(T, generator=g)].to(torch.int32).view(T, 1)
    h, wt = torch.randn(T, W, generator=g).bfloat16(), torch.rand(T, 1, generator=g)
    gu, dn = (torch.randn(E, 2 * ff, W, generator=g) * W**-0.5).bfloat16(), (torch.randn(E, W, ff, generator=g) * ff**-0.5).bfloat16()
    align = ops.moe_align(idx.to(DEV), E, 4 * ops.moe_tile_rows() if wide else None)
    got = ops.moe_experts(h.to(DEV), wt.to(DEV), align, gu.to(DEV), dn.to(DEV), 1, 7.0, act=ops.ACT_SILU if act == "silu" else ops.ACT_SWISH_CLAMPED,
                          scale_input=act == "clamped").cpu().double()
    for e in range(E):
        rows = (idx[:, 0] == e).nonzero()[:, 0]
        x = ((h[rows].float() * wt[rows]).bfloat16() if act == "clamped" else h[rows]).double()
        z = x @ gu[e].double().T
        a, b = z[:, :ff], z[:, ff:]
        if act == "clamped":
            a, b = a.clamp(max=7.0), b.clamp(-7.0, 7.0)
            hid = a * torch.sigmoid(1.702 * a) * (b + 1)
        else:
            hid = torch.nn.functional.silu(a) * b
        want = hid @ dn[e].double().T
        assert (got[rows] - want).norm() <= 1e-2 * want.norm() + 1e-9, e


def test_moe_experts_on_rows_off_a_16_byte_boundary():
    """Token rows whose pitch suits the pair kernel but whose first element does not lie on 16 bytes: the experts of the aligned rows."""
    ops = _ops()
    E, W, ff, T = 4, 512, 256, 40
    g = torch.Generator().manual_seed(9)
    buf = torch.randn(T, W + 8, generator=g).bfloat16().to(DEV)
    h = buf[:, 1:W + 1]
    idx, wt = torch.randint(0, E, (T, 1), generator=g).to(torch.int32).to(DEV), torch.rand(T, 1, generator=g).to(DEV)
    gu, dn = (torch.randn(E, 2 * ff, W, generator=g) * W**-0.5).bfloat16().to(DEV), (torch.randn(E, W, ff, generator=g) * ff**-0.5).bfloat16().to(DEV)
    got, want = (ops.moe_experts(x, wt, ops.moe_align(idx, E), gu, dn, 1, 7.0) for x in (h, h.contiguous()))
    assert (got - want).norm() <= 1e-2 * want.norm()  # the hidden activations' rounding to bf16


@pytest.mark.parametrize("rows,tiles", [(0, 1), (33, 1), (40, 2)])
def test_fp32_linear_writes_the_tiles_it_is_asked_for(rows, tiles):
    """Dense rows of the C entry: row_tiles tiles of 32 rows or all M rows, whichever is less; none is none."""
    from vllm_neuron_b200 import _cabi

    ops = _ops()
    N, K = 40, 64
    g = torch.Generator().manual_seed(rows)
    a, w, out = torch.randn(64, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV), torch.full((64, N), 7.0, device=DEV)
    assert _cabi.load().b200_grouped_linear(a.data_ptr(), K, 0, 0, 0, w.data_ptr(), 0, 0, 0, tiles, rows, N, K, ops.F32, out.data_ptr(), N, 0, 0, 0,
                                            0.0, ops.moe_tile_rows(), ops._stream()) == 0
    n = min(rows, 32 * tiles)
    want = a.double() @ w.double().T
    assert ((out[:n].double() - want[:n]).abs() <= K * 2.0**-24 * (a.abs().double() @ w.abs().double().T)[:n]).all() and (out[n:] == 7).all()


@pytest.mark.parametrize("kind", ["full", "window-sink", "chunk", "softcap", "keep", "pooled", "latent", "maps", "sigmoid", "fp32-out"])
def test_attention_of_mixed_steps_apart_and_together(kind, monkeypatch):
    """Prompt portions (one continued, one after decoded tokens) beside decoded ones, through every attention variant in one launch and in
    one per kind: the prompts' rows bit for bit, the decoded ones up to the two kernels' bf16 roundings (weights and outputs, 2^-8 each)."""
    from vllm_neuron_b200.hybrid import StepMeta

    ops = _ops()
    entries = [(0, 0, 140), (1, 200, 1), (2, 77, 3), (3, 500, 1), (4, 60, 40)]
    H, G, D, Dv, bs, win = 8, 2, 64, 64, 32, 1 << 30
    kw, sink, latent = {}, None, 0
    g = torch.Generator(device=DEV).manual_seed(3)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)  # noqa: E731
    rows = {e[0]: list(range(1 + 20 * e[0], 21 + 20 * e[0])) for e in entries}
    if kind in ("window-sink", "keep", "pooled"):
        win = 96
    if kind == "window-sink":
        sink = r(H)
    if kind == "latent":
        G, D, latent = 1, 192, 128
    k_pool = r(101, G, bs, D).bfloat16()
    v_pool = k_pool if latent else r(101, G // 2 if kind == "maps" else G, bs, Dv).bfloat16()
    if kind == "chunk":
        kw["chunk"] = 128
    elif kind == "softcap":
        kw["softcap"] = 20.0
    elif kind == "keep":
        kw["keep"] = 4
    elif kind == "pooled":
        kw["pooled"] = (r(101, G, 2, D).bfloat16(), r(101, G, 2, Dv).bfloat16(), 16)
    elif kind == "sigmoid":
        kw["sigmoid_bias"] = r(H)
    elif kind == "fp32-out":
        kw["out_f32"] = True
    meta = StepMeta.build(entries, rows, bs, torch.device(DEV))
    assert len(meta.parts) == 3
    table = torch.tensor([rows[i] for i in range(5)], dtype=torch.int32, device=DEV)
    q = r(meta.num_tokens, H * D)
    outs = []
    for apart in (False, True):
        monkeypatch.setattr(ops, "_split_pays", lambda *a, apart=apart: apart)
        outs.append(ops.swa_sink_attn(q, H, k_pool, v_pool, table, meta, sink, D**-0.5, win, latent, **kw).float())
    short = torch.zeros(meta.num_tokens, dtype=torch.bool, device=DEV)
    short[140:145] = True
    assert (outs[0][short] - outs[1][short]).norm() <= 2.0**-7 * outs[0][short].norm()
    # the 40 tokens of the last portion may meet another prompt kernel than the step's longest portion does
    assert torch.equal(outs[0][:140], outs[1][:140]) and (outs[0][145:] - outs[1][145:]).norm() <= 2.0**-7 * outs[0][145:].norm()


def test_dyt_residual_sees_weights_that_the_kernel_ahead_wrote():
    """Weight rows that come straight out of another kernel of the library, whose blocks let the next one start early: the last row that it
    writes is the weight, a new one each time."""
    ops = _ops()
    W = 1024
    g = torch.Generator().manual_seed(2)
    src, one, zero = torch.randn(8, 3000, W, generator=g).to(DEV), torch.ones(W, device=DEV), torch.zeros(W, device=DEV)
    y = torch.randn(4, W, generator=g).to(DEV)
    got = []
    for i in range(8):
        w = ops.dyt_norm(src[i], one, zero, 1.0, torch.float32)[-1]
        x = torch.zeros(4, W, device=DEV)
        w2 = ops.dyt_norm(src[i], one, zero, 0.5, torch.float32)[-1]
        got.append((ops.dyt_residual(x, y, (w, zero, 0.7), (w2, zero, 0.4), torch.float32), x))
    for i, (out, x) in enumerate(got):
        want = torch.tanh(0.7 * y.double()) * torch.tanh(src[i, -1].double())
        assert (x.double() - want).abs().max() <= 2e-6
        assert (out.double() - torch.tanh(0.4 * want) * torch.tanh(0.5 * src[i, -1].double())).abs().max() <= 2e-6


@pytest.mark.parametrize("T,inner,groups", [(1, 1024, 8), (63, 512, 2), (300, 512, 2), (700, 264, 2), (820, 1024, 1), (1640, 1024, 1), (5, 516, 1), (400, 2080, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gated_group_rmsnorm_slices(T, inner, groups, dtype):
    """Slices of a warp's registers and of a CTA, few and many of them, ragged ones: against 64 bits, a few fp32 roundings of the result's size
    plus the rounding to the output type."""
    ops = _ops()
    g = torch.Generator().manual_seed(T + inner)
    y, z, w = (torch.randn(*s, generator=g) for s in ((T, inner), (T, inner + 12), (inner,)))
    got = ops.gated_group_rmsnorm(y.to(DEV), z.to(DEV), w.to(DEV), groups, 1e-6, dtype).double().cpu()
    v = (y.double() * torch.nn.functional.silu(z[:, :inner].double())).view(T, groups, -1)
    want = (v / torch.sqrt(v.pow(2).mean(-1, keepdim=True) + 1e-6)).reshape(T, inner) * w.double()
    assert (got - want).abs().max() <= (2.0**-8 if dtype == torch.bfloat16 else 2e-6) * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("m,n,k,short", [(400, 1024, 64, True), (129, 64, 160, True), (1000, 2048, 128, False), (129, 64, 168, False), (100, 64, 64, False)])
def test_short_prompt_rows_take_the_small_kernel(m, n, k, short):
    """Prompts on short rows: the bits of the mma.sync kernel; longer rows, larger products and decode batches leave it.  bf16 products are
    exact: k roundings of fp32 sums either way (cut short, not rounded, on the tensor cores: 2^-23 each)."""
    from types import SimpleNamespace

    from vllm_neuron_b200.hybrid import HybridCausalLM

    ops = _ops()
    g = torch.Generator().manual_seed(m + k)
    a, w = torch.randn(m, k, generator=g).bfloat16().to(DEV), torch.randn(n, k, generator=g).bfloat16().to(DEV)
    before = ops.launch_count()
    got = HybridCausalLM._linear(SimpleNamespace(et=torch.bfloat16, gemm_ws=None, device=DEV), a, w)
    assert ops.launch_count() == before + 1
    if short:
        assert torch.equal(got, ops.linear_simt(a, w))
    want = a.double() @ w.double().T
    assert ((got.double() - want).abs() <= k * 2.0**-23 * (a.double().abs() @ w.double().abs().T)).all()


@pytest.mark.parametrize("T,W,off", [(1, 4, 0), (5, 1028, 0), (2, 4100, 0), (700, 132, 0), (4, 30, 0), (3, 64, 1), (3, 64, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_embedding_and_tanh_norm_in_vectors(T, W, off, dtype):
    """Rows of whole vectors, rows that are none (30), tables and inputs that start one or two elements behind a boundary; token ids outside the
    vocabulary take its ends.  One rounding of the product; the norm two, of tanh's 2 ulp, plus the rounding to the output type."""
    ops = _ops()
    g = torch.Generator().manual_seed(T * W + off)
    table = torch.randn(11 * W + off, generator=g).to(dtype)[off:].view(11, W)
    tokens = torch.randint(-2, 13, (T,), generator=g, dtype=torch.int32)
    placed = torch.empty(11 * W + off, dtype=dtype, device=DEV)[off:].view(11, W).copy_(table)
    want = table.float()[tokens.long().clamp(0, 10)] * 0.37
    assert torch.equal(ops.embed_scale(tokens.to(DEV), placed, 0.37).cpu(), want)
    x, w, b = torch.randn(T, W, generator=g), torch.randn(W, generator=g), torch.randn(W, generator=g)
    xd = torch.empty(T * W + off, device=DEV)[off:].view(T, W).copy_(x)
    got = ops.dyt_norm(xd, w.to(DEV), b.to(DEV), 1.1, dtype).double().cpu()
    ref = torch.tanh(1.1 * x.double()) * w.double() + b.double()
    assert ((got - ref).abs() <= 2.0**-21 * (w.abs() + b.abs()).double() + (2.0**-8 if dtype == torch.bfloat16 else 0.0) * ref.abs()).all()


@pytest.mark.parametrize("T,W", [(1, 4), (3, 1028), (2, 4096), (5, 4100), (700, 132), (4, 30)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_row_kernels_in_vectors(T, W, dtype):
    """Rows of whole vectors at both ends of the register-row range, beyond it, and rows that are none (30): all against 64 bits.  Bounds:
    a few fp32 roundings of the result's size, plus the rounding to the output type."""
    ops = _ops()
    g = torch.Generator().manual_seed(T * W)
    r = lambda *s: torch.randn(s, generator=g)  # noqa: E731
    x, y, y2, w1, b1, w2, b2, wt = r(T, W), r(2 * T, W), r(T, W), r(W), r(W), r(W), r(W), torch.rand(T, 2, generator=g)
    d = lambda t: t.to(DEV)  # noqa: E731
    tol = 2.0**-8 if dtype == torch.bfloat16 else 2e-6

    def close(got, want, t=tol):
        assert (got.double().cpu() - want).abs().max() <= t * max(1.0, float(want.abs().max()))

    xd = d(x)
    out = ops.dyt_residual(xd, d(y), (d(w1), d(b1), 0.7), (d(w2), d(b2), 0.4), dtype, y2=d(y2), nsum=2)
    want = x.double() + torch.tanh(0.7 * (y.view(T, 2, W).double().sum(1) + y2.double())) * w1.double() + b1.double()
    close(xd, want, 2e-6)
    close(out, torch.tanh(0.4 * want) * w2.double() + b2.double())
    xd = d(x)
    out = ops.rms_residual(xd, d(y), d(w1), 1e-6, nsum=2, y_weight=d(wt), out_dtype=dtype)
    s = (wt.double()[:, :, None] * y.view(T, 2, W).double()).sum(1)
    want = x.double() + s / torch.sqrt(s.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + w1.double())
    close(xd, want, 4e-6)
    close(out, want)
    xd = d(x)
    out = ops.add_group_rmsnorm(xd, d(y[:T]), d(y2), d(w1), 2, 1e-6, dtype)
    s = x.double() + y[:T].double() + y2.double()
    n = s.view(T, 2, W // 2)
    close(xd, s, 2e-6)
    close(out, (n / torch.sqrt(n.pow(2).mean(-1, keepdim=True) + 1e-6)).reshape(T, W) * w1.double())
    if W % 4 == 0:
        z = r(T, W + 12)
        out = ops.gated_group_rmsnorm(d(y2), d(z), d(w1), 2, 1e-6, dtype)
        v = (y2.double() * torch.nn.functional.silu(z[:, :W].double())).view(T, 2, W // 2)
        close(out, (v / torch.sqrt(v.pow(2).mean(-1, keepdim=True) + 1e-6)).reshape(T, W) * w1.double())
    gu = 4 * r(T, 2 * W)
    a, b = gu[:, :W].double().clamp(max=7.0), gu[:, W:].double().clamp(-7.0, 7.0)
    close(ops.clamped_glu(d(gu), 7.0, dtype), a * torch.sigmoid(1.702 * a) * (b + 1))


@pytest.mark.parametrize("H,P,N,G", [(4, 128, 128, 2), (2, 70, 64, 1), (3, 5, 32, 3), (2, 257, 128, 2), (2, 12, 40, 1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_ssd_step_of_one_token_each(H, P, N, G, dtype):
    """Decode steps: value columns that end inside a warp's rows, every state size with a kernel of its own and one without, a sequence at
    position 0 over a used slot.  The state is that of the scan bit for bit; y within N roundings of an fp32 sum of N products (one more for D x)."""
    ops = _ops()
    g = torch.Generator().manual_seed(H * P + N)
    entries = [(3, 5, 1), (0, 0, 1), (2, 90, 1)]
    C, slots = H * P + 2 * G * N, 4
    xbc = torch.randn(3, C, generator=g).to(dtype)
    raw = torch.randn(3, H + 2, generator=g)
    a_log, bias, D = 0.5 * torch.randn(H, generator=g), torch.randn(H, generator=g), torch.randn(H, generator=g)
    state = torch.randn(slots, H, P, N, generator=g)
    meta = _meta(entries, {r: [1] * 40 for r in range(slots)})
    args = [t.to(DEV) for t in (xbc, raw)] + [2] + [t.to(DEV) for t in (a_log, bias, D)]
    got, want = state.to(DEV), state.to(DEV)
    y = ops.ssd_scan(*args, got, meta, H, P, N, G)
    meta.max_new = 2
    ops.ssd_scan(*args, want, meta, H, P, N, G)
    assert torch.equal(got, want) and torch.equal(got[1].cpu(), state[1])
    S = got[torch.tensor([3, 0, 2], device=DEV)].double().cpu()
    Cm = xbc[:, H * P + G * N:].double().view(3, G, N).repeat_interleave(H // G, 1)
    skip = D.double()[:, None] * xbc[:, :H * P].double().view(3, H, P)
    terms = S * Cm[:, :, None, :]
    bound = (N + 1) * 2.0**-24 * (terms.abs().sum(-1) + skip.abs())
    assert ((y.double().cpu().view(3, H, P) - terms.sum(-1) - skip).abs() <= bound).all()


def test_ssd_step_sees_parameters_that_the_kernel_ahead_wrote():
    """Decay, bias and skip rows that come straight out of another kernel of the library, whose blocks let the next one start early: the same
    call on the same rows, once they are there, gives the same bits."""
    ops = _ops()
    H, P, N, G, W = 8, 64, 64, 2, 1024
    g = torch.Generator().manual_seed(4)
    src, one, zero = torch.randn(8, 3000, W, generator=g).to(DEV), torch.ones(W, device=DEV), torch.zeros(W, device=DEV)
    xbc, raw, state = torch.randn(2, H * P + 2 * G * N, generator=g).to(DEV), torch.randn(2, H, generator=g).to(DEV), torch.randn(2, H, P, N, generator=g).to(DEV)
    meta = _meta([(0, 5, 1), (1, 9, 1)], {0: [1] * 40, 1: [2] * 40})
    runs = []
    for i in range(8):
        s = state.clone()
        p = ops.dyt_norm(src[i], one, zero, 1.0, torch.float32)[-1]
        runs.append((p, s, ops.ssd_scan(xbc, raw, 0, p[:H], p[H:2 * H], p[2 * H:3 * H], s, meta, H, P, N, G)))
    torch.cuda.synchronize()
    for p, s, y in runs:
        want = state.clone()
        assert torch.equal(y, ops.ssd_scan(xbc, raw, 0, p[:H], p[H:2 * H], p[2 * H:3 * H], want, meta, H, P, N, G)) and torch.equal(s, want)


def test_allocations_leave_the_interpreter_to_other_threads():
    """A result that has to wait for the device, because cached memory is given back for it, does not hold up other threads' Python."""
    import threading
    import time

    ops = _ops()
    like, held, over = torch.zeros(1, device=DEV), [0.0], threading.Event()

    def work():
        last = time.perf_counter()
        while not over.is_set():
            now = time.perf_counter()
            held[0], last = max(held[0], now - last), now

    thread = threading.Thread(target=work)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cached = torch.empty(1 << 30, dtype=torch.uint8, device=DEV)
    del cached
    room = torch.cuda.memory_reserved() + (64 << 20)
    torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
    try:
        torch.cuda._sleep(1 << 29)  # a quarter of a second or more
        thread.start()
        t0 = time.perf_counter()
        made = ops._new(like, torch.uint8, (1 << 30) + (16 << 20))
        took = time.perf_counter() - t0
    finally:
        over.set()
        thread.join()
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert made.numel() > 1 << 30 and took > 0.1 and held[0] < took / 2


def _one_sequence(T, G, Gv, D, Dv, g):
    """bf16 pools of one sequence on pages in reverse, and the same rows in 64 bits: (meta, table, key pool, value pool, keys, values)."""
    from vllm_neuron_b200.hybrid import StepMeta

    nb = -(-T // 32)
    pages = list(range(nb, 0, -1))
    kp, vp = (torch.randn(nb + 1, n, 32, d, generator=g, device=DEV).bfloat16() for n, d in ((G, D), (Gv, Dv)))
    meta = StepMeta.build([(0, 0, T)], {0: pages}, 32, torch.device(DEV))
    k, v = (p[pages].transpose(1, 2).reshape(nb * 32, -1, p.shape[3])[:T].double() for p in (kp, vp))
    return meta, torch.tensor([pages], dtype=torch.int32, device=DEV), kp, vp, k, v


@pytest.mark.parametrize("kind,D,Dv,G", [("cap", 128, 128, 2), ("cap", 128, 64, 4), ("chunk", 64, 64, 2), ("chunk+cap", 64, 64, 2), ("keep", 128, 128, 2),
                                         ("keep", 128, 64, 2), ("maps", 32, 64, 4), ("maps", 64, 128, 2), ("maps+window", 64, 64, 2), ("none", 64, 64, 2)])
def test_sink_of_prompts_beside_the_other_options(kind, D, Dv, G):
    """A sink with a soft cap (which it does not pass), chunks, kept tokens and two score maps, and sinks of -inf, against 64 bits.  Weights in two
    bf16 terms and fp32 rows: 2^-15 of a row's weighted values, and the query's rounding to bf16, which the reference shares."""
    ops = _ops()
    g = torch.Generator(device=DEV).manual_seed(D + G)
    T, H, maps = 300, 8, kind.startswith("maps")
    meta, table, kp, vp, k, v = _one_sequence(T, G, G // 2 if maps else G, D, Dv, g)
    q = torch.randn(T, H * D, generator=g, device=DEV).bfloat16().float()
    sink = 2 * torch.randn(H, generator=g, device=DEV) + 2
    if kind == "none":
        sink[:] = -math.inf
    kw, window, scale = {}, 1 << 30, 2 * D**-0.5
    if "cap" in kind:
        kw["softcap"] = 2.0
    if "chunk" in kind:
        kw["chunk"] = 130
    if kind == "keep":
        kw["keep"], window = 70, 90
    if "window" in kind:
        window = 100
    with ops.kernel_timer() as kt:
        got = ops.swa_sink_attn(q, H, kp, vp, table, meta, sink, scale, window, out_f32=True, **kw)
    assert any(n.startswith("swa_sink_attn_prefill_tc") for n in kt.summary())
    i = torch.arange(T, device=DEV)
    seen = (i[None] <= i[:, None]) & ((i[None] > i[:, None] - window) | (i[None] < kw.get("keep", 0)))
    if "chunk" in kind:
        seen &= i[None] // 130 == i[:, None] // 130
    of = torch.arange(H, device=DEV) // (H // G)
    s = torch.einsum("thd,lhd->htl", q.double().view(T, H, D), k[:, of]) * scale
    if "cap" in kind:
        s = 2.0 * torch.tanh(s / 2.0)
    s = torch.cat([s.masked_fill(~seen, -math.inf), sink.double()[:, None, None].expand(H, T, 1)], 2)
    p, vh = torch.softmax(s, 2)[..., :T], v[:, of // 2 if maps else of]
    want, size = torch.einsum("htl,lhd->thd", p, vh), torch.einsum("htl,lhd->thd", p, vh.abs())
    # scores in fp32 and exponents by the fast exponential: 2^-17 of a weight each, beside the two terms' 2^-16
    assert ((got.double().view(T, H, Dv) - want).abs() <= 2.0**-13 * size).all()


def test_a_window_of_no_tokens_beside_a_sink_is_refused():
    ops = _ops()
    g = torch.Generator(device=DEV).manual_seed(1)
    for T in (40, 200):
        meta, table, kp, vp, _, _ = _one_sequence(T, 2, 2, 64, 64, g)
        with pytest.raises(RuntimeError):
            ops.swa_sink_attn(torch.randn(T, 4 * 64, generator=g, device=DEV), 4, kp, vp, table, meta, torch.zeros(4, device=DEV), 0.1, 0)


@pytest.mark.parametrize("window", [100, 1 << 30])
def test_decode_attention_over_a_page_that_is_not_there(window):
    """A page number below 0 stands for rows of zeros, inside the window too."""
    from vllm_neuron_b200.hybrid import StepMeta

    ops = _ops()
    g = torch.Generator(device=DEV).manual_seed(3)
    G, D, H = 2, 64, 8
    kp, vp = (torch.randn(10, G, 32, D, generator=g, device=DEV).bfloat16() for _ in range(2))
    kp[9], vp[9] = 0, 0
    meta = StepMeta.build([(0, 200, 1), (1, 130, 1)], {0: list(range(1, 8)), 1: list(range(1, 8))}, 32, torch.device(DEV))
    table = torch.tensor([[1, 2, 3, 4, 5, 9, 7], [2, 9, 1, 9, 3, 4, 5]], dtype=torch.int32, device=DEV)
    q, sink = torch.randn(2, H * D, generator=g, device=DEV), torch.randn(H, generator=g, device=DEV)
    want = ops.swa_sink_attn(q, H, kp, vp, table, meta, sink, 0.1, window)
    assert torch.equal(ops.swa_sink_attn(q, H, kp, vp, torch.where(table == 9, -1, table), meta, sink, 0.1, window), want)


@pytest.mark.parametrize("M,N,K", [(3, 40, 64), (9, 40, 64), (33, 100, 60), (8, 33, 128), (70, 65, 100), (20, 30000, 132), (255, 16, 68), (257, 5, 132), (300, 1, 4),
                                   (6001, 9, 40), (6003, 16, 260), (6003, 8, 128)])
def test_fp32_linear_on_short_rows_and_of_few_outputs(M, N, K):
    """Rows of one to four slices in tiles of 8 and 32 rows, wide weights under 32 rows, 2, 4 and 8 rows a warp where a row has few outputs: against 64
    bits, K roundings of an fp32 sum.  A row's sums do not depend on the batch: its first rows alone give the same bits."""
    ops = _ops()
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    got = ops.linear_simt(a, w)
    assert ((got.double() - a.double() @ w.double().T).abs() <= K * 2.0**-24 * (a.abs().double() @ w.abs().double().T)).all()
    for few in (1, 7, 30):
        if few < M:
            assert torch.equal(ops.linear_simt(a[:few], w), got[:few])
