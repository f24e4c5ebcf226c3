"""GPU parity: per-channel-scaled GEMMs (tcgen05) vs the oracle's quantize/dequantize GEMM.

Stated tolerances (north_star: "quantized GEMMs within stated per-channel FP8/INT8 tolerances"):
  * the quantised operands are produced by the ORACLE's quantiser, so both sides multiply the same codes;
  * INT8 W8A8: products and sums are exact integers -> result must match the oracle to 1 bf16 ulp
    (rel 2^-7 per element; only the final rounding/scale order can differ);
  * FP8 e4m3 W8A8 and bf16: fp32 accumulation in a different order -> |err| <= 1e-2 * rms(ref) + 2^-7 |ref|.
"""
import pytest
import torch

from oracle import quant_ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vllm_neuron_b200 import ops as o

    o.device_check(0)
    return o


def _assert_close(got, want, exact_int=False):
    got, want = got.float().cpu(), want.float()
    assert torch.isfinite(got).all()
    rms = want.pow(2).mean().sqrt().item()
    tol = (0.0 if exact_int else 1e-2 * rms) + want.abs() * 2.0**-7 + 1e-6
    bad = (got - want).abs() > tol
    assert not bad.any(), f"{bad.sum().item()} / {bad.numel()} outside tolerance; max err {(got - want).abs().max().item()} rms {rms}"


# last column = split_k: cluster size along K for the decode schedule (M <= 128; 0 = auto), CTA cap for stream-K (M > 128)
SHAPES = [
    (64, 6144, 4096, 0),     # cfg3 qkv (auto: clusters of 4)
    (64, 4096, 4096, 0),     # o_proj (auto: clusters of 8)
    (64, 4096, 14336, 0),    # down_proj (long K)
    (64, 1024, 512, 1),      # no split: epilogue straight from TMEM
    (64, 1024, 512, 2),      # clusters of 2: 64-row slices
    (64, 1024, 512, 4),      # clusters of 4, one k-block per CTA (fp8)
    (33, 896, 2048, 8),      # clusters of 8; N, M ragged (tokens 33 / 8 per owner)
    (64, 896, 2048, 3),      # clusters of 3: 21/21/22 tokens per owner
    (5, 512, 2048, 7),       # fewer tokens than ranks: some owners finish nothing
    (4, 2048, 2048, 0),      # TinyLlama decode batch
    (1, 256, 128, 0),        # single row, single k-block
    (128, 640, 1152, 0),     # Qwen TP=8 o-proj-like, M=128
    (128, 640, 1152, 4),     # M=128 tile through the cluster reduction
    (100, 16032, 256, 0),    # N not a multiple of 128 (vocab shard), ragged M
    (300, 384, 640, 0),      # M > 128: persistent stream-K, two m-tiles
    (300, 384, 640, 5),      # stream-K over 5 CTAs: spans start and end mid-tile
    (200, 1024, 512, 32),    # stream-K, every tile has several contributors
]


@pytest.mark.parametrize("m,n,k,ctas", SHAPES)
@pytest.mark.parametrize("kind", ["fp8", "int8"])
def test_w8a8_gemm(ops, m, n, k, ctas, kind):
    g = torch.Generator().manual_seed(m * 7 + n + k)
    x = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.02).bfloat16()
    xq, xs = quant_ref.quantize_act_per_token(x, kind)
    wq, ws = quant_ref.quantize_weight_per_channel(w, kind)
    bias = torch.randn(n, generator=g).bfloat16() if n % 256 == 0 else None
    res = torch.randn(m, n, generator=g).bfloat16() if k % 1024 == 0 else None
    want = quant_ref.qgemm_ref(xq, xs, wq, ws, bias, res)
    got = ops.gemm(xq.cuda(), wq.cuda(), xs.cuda(), ws.cuda(), None if bias is None else bias.cuda(),
                   None if res is None else res.cuda(), split_k=ctas)
    torch.cuda.synchronize()
    _assert_close(got, want, exact_int=(kind == "int8"))


@pytest.mark.parametrize("m,n,k,ctas", SHAPES[:5] + SHAPES[6:10] + SHAPES[12:14])
def test_bf16_gemm(ops, m, n, k, ctas):
    g = torch.Generator().manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.02).bfloat16()
    want = quant_ref.gemm_ref(x, w)
    got = ops.gemm(x.cuda(), w.cuda(), split_k=ctas)
    torch.cuda.synchronize()
    _assert_close(got, want)


@pytest.mark.parametrize("m,n,k,ctas", SHAPES[:10] + SHAPES[11:])
def test_int8_weight_only_gemm(ops, m, n, k, ctas):
    """bf16 activations x int8 per-channel weights (cfg4, Qwen2.5-32B INT8 weight-only): the int8 rows are widened to
    bf16 inside the kernel (exact), so the result is the bf16 GEMM on the dequantised codes -> same bar as bf16."""
    g = torch.Generator().manual_seed(m * 3 + n + k)
    x = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(n, k, generator=g) * 0.02).bfloat16()
    wq, ws = quant_ref.quantize_weight_per_channel(w, "int8")
    bias = torch.randn(n, generator=g).bfloat16() if n % 256 == 0 else None
    res = torch.randn(m, n, generator=g).bfloat16() if k % 1024 == 0 else None
    want = quant_ref.wo_gemm_ref(x, wq, ws, bias, res)
    got = ops.gemm(x.cuda(), wq.cuda(), None, ws.cuda(), None if bias is None else bias.cuda(),
                   None if res is None else res.cuda(), split_k=ctas)
    torch.cuda.synchronize()
    _assert_close(got, want)


def test_int8_weight_only_exact_on_integer_activations(ops):
    """Size-independent property: with small-integer bf16 activations every product and partial sum is an exact integer
    below 2^24, so the weight-only GEMM must reproduce the integer GEMM bit for bit (decode and stream-K schedules)."""
    g = torch.Generator().manual_seed(5)
    n, k = 1280, 1152
    w = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8)
    for m in (64, 128, 300):
        a = torch.randint(-8, 9, (m, k), generator=g).to(torch.bfloat16)
        got = ops.gemm(a.cuda(), w.cuda(), out_dtype=torch.float32)
        want = (a.double() @ w.double().t()).float()
        assert torch.equal(got.cpu(), want), m


def test_fp32_out_and_linearity(ops):
    """Size-independent property at a BASELINE-size shape (lm_head shard): GEMM(a1+a2) == GEMM(a1)+GEMM(a2) in fp32 out
    for int8 codes (exact integer arithmetic), and fp32 output equals the oracle."""
    g = torch.Generator().manual_seed(9)
    m, n, k = 64, 16032, 4096
    a1 = torch.randint(-50, 50, (m, k), generator=g, dtype=torch.int8)
    a2 = torch.randint(-50, 50, (m, k), generator=g, dtype=torch.int8)
    w = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8)
    o1 = ops.gemm(a1.cuda(), w.cuda(), out_dtype=torch.float32)
    o2 = ops.gemm(a2.cuda(), w.cuda(), out_dtype=torch.float32)
    o12 = ops.gemm((a1 + a2).cuda(), w.cuda(), out_dtype=torch.float32)
    assert torch.equal(o1 + o2, o12)
    want = (a1[:8].double() @ w.double().t()).float()
    assert torch.equal(o1[:8].cpu(), want)


# CTA-pair schedule (M > 128, no CTA cap): token tiles of every width the rule can pick, ragged tokens and rows (a pair's second CTA
# partly or wholly outside), fewer k-blocks than ring stages, one and several tiles per pair (accumulators reused)
PAIR_SHAPES = [(129, 256, 64), (129, 130, 128), (161, 896, 640), (257, 1000, 192), (300, 16032, 256), (700, 4096, 1024), (2000, 6000, 192),
               (1100, 9600, 320)]


@pytest.mark.parametrize("m,n,k", PAIR_SHAPES)
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_pairs_int8_exact(ops, m, n, k, f32):
    """Integer sums are exact: every element is the product of the oracle's integer sum and the two scales, to one bf16 ulp (fp32
    output: two roundings of the scales, 2^-22)."""
    g = torch.Generator().manual_seed(m + n + k)
    xq = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    wq = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8)
    xs, ws = torch.rand(m, generator=g) + 0.5, torch.rand(n, generator=g) + 0.5
    ref = (xq.cuda().double() @ wq.cuda().double().T).cpu() * xs.double()[:, None] * ws.double()
    got = ops.gemm(xq.cuda(), wq.cuda(), xs.cuda(), ws.cuda(), out_dtype=torch.float32 if f32 else torch.bfloat16).double().cpu()
    assert ((got - ref).abs() <= ref.abs() * (2.0**-22 if f32 else 2.0**-8)).all()


@pytest.mark.parametrize("m,n,k", [(129, 64, 64), (300, 1056, 640), (1100, 9600, 320)])
def test_gemm_pairs_silu_residual_bias(ops, m, n, k):
    """bf16 operands through both epilogues: equal to the stream-K schedule's up to the order of the fp32 sums."""
    g = torch.Generator(device="cuda").manual_seed(m)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w, bias, res = r(m, k), r(n, k) * k**-0.5, r(n), r(m, n)
    _assert_close(ops.gemm(x, w, None, None, bias, res), ops.gemm(x, w, None, None, bias, res, split_k=64).cpu())
    a, ga = ops.gemm_silu_mul(x, w, None, None, bias)
    b, gb = ops.gemm_silu_mul(x, w, None, None, bias, split_k=64)
    _assert_close(a, b.cpu())
    _assert_close(ga, a.float().abs().view(m, -1, 16).amax(-1).cpu())


# More of both: two token tiles a unit (777 x 6144), several tiles a pair, ragged tokens and rows, fewer k-blocks than ring stages and many more
WIDE_SHAPES = [(300, 10000, 192), (300, 10001, 192), (777, 6144, 1040), (700, 12800, 96), (1030, 16128, 4000), (771, 28416, 4096)]


@pytest.mark.parametrize("m,n,k", WIDE_SHAPES)
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_pairs_of_two_token_tiles_int8_exact(ops, m, n, k, f32):
    test_gemm_pairs_int8_exact(ops, m, n, k, f32)


# Units of two token tiles: (m, n, k in int8, waves of them, whether lone tiles follow, whether the token tiles are odd in number, so that a weight tile's last
# unit holds one).  With several waves a pair's next unit starts while the epilogue still reads the accumulator of its second tile.  As many k-blocks as
# ring stages and more; none of these plans has fewer.
WIDE_PLANS = [(258, 12851, 720, 1, False, False), (784, 5588, 672, 1, False, True), (258, 19046, 736, 1, True, False), (770, 9717, 752, 1, True, True), (261, 37770, 1792, 2, False, False),
              (1063, 15187, 3984, 2, True, False), (1541, 9389, 10752, 2, False, True), (1038, 15811, 10608, 2, True, True), (577, 31692, 4752, 3, True, False)]


def _wide_plan(ops, m, n, k, kind):
    plan = ops.gemm_pair_plan(m, n, k, kind)
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    return -(-plan["wide"] // pairs), plan["units"] > plan["wide"], -(-m // plan["tokens"]) % 2 == 1


@pytest.mark.parametrize("m,n,k,waves,lone,odd", WIDE_PLANS)
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_pairs_units_of_two_token_tiles_int8_exact(ops, m, n, k, waves, lone, odd, f32):
    """Bounds as in test_gemm_pairs_int8_exact; the plan is the one that the shape stands for."""
    assert _wide_plan(ops, m, n, k, ops.INT8) == (waves, lone, odd)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    r = lambda *s: torch.randint(-127, 128, s, generator=g, dtype=torch.int8, device="cuda")  # noqa: E731
    x, w, xs, ws = r(m, k), r(n, k), torch.rand(m, generator=g, device="cuda") + 0.5, torch.rand(n, generator=g, device="cuda") + 0.5
    want = x.double() @ w.double().T * xs.double()[:, None] * ws.double()
    got = ops.gemm(x, w, xs, ws, out_dtype=torch.float32 if f32 else torch.bfloat16).double()
    assert ((got - want).abs() <= want.abs() * (2.0**-22 if f32 else 2.0**-8)).all()


@pytest.mark.parametrize("m,n,k,waves,lone,odd", [(770, 9728, 376, 1, True, True), (258, 19072, 368, 1, True, False), (261, 37792, 896, 2, False, False)])
def test_gemm_pairs_units_of_two_token_tiles_silu_residual_bias(ops, m, n, k, waves, lone, odd):
    assert _wide_plan(ops, m, n, k, ops.BF16) == (waves, lone, odd)
    test_gemm_pairs_silu_residual_bias(ops, m, n, k)


@pytest.mark.parametrize("f32", [False, True])
def test_gemm_pairs_units_of_two_token_tiles_rows_of_odd_length(ops, f32):
    assert _wide_plan(ops, 258, 12851, 360, ops.BF16) == (1, False, False)
    test_gemm_pairs_bf16_against_64_bits(ops, 258, 12851, 360, f32)


@pytest.mark.parametrize("m,n,k", [(777, 6144, 520), (700, 12800, 96)])
def test_gemm_pairs_of_two_token_tiles_silu_residual_bias(ops, m, n, k):
    test_gemm_pairs_silu_residual_bias(ops, m, n, k)


@pytest.mark.parametrize("kind", ["bf16", "wo"])
@pytest.mark.parametrize("m,n,k", [(33, 640, 1152), (64, 4096, 2048), (300, 1056, 640)])
def test_gemm_outputs_on_any_boundary(ops, kind, m, n, k):
    """Outputs that start one, two or four elements after a 16-byte boundary: the bits of the aligned call on the schedule that they take
    (decode batches in bf16 and narrow weight-only ones: the one that does not cut K, where vectors of four would not lie on their size), nothing written around them."""
    from vllm_neuron_b200 import _cabi

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((m, k), generator=g, device="cuda").bfloat16()
    w = (torch.randn((n, k), generator=g, device="cuda") * k**-0.5).bfloat16() if kind == "bf16" else torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    ws = None if kind == "bf16" else torch.rand(n, generator=g, device="cuda") * 0.01
    dt = ops.BF16 if kind == "bf16" else ops.INT8_WO
    work = ops.gemm_workspace(m, n, k, dt, x.device)
    nw = 0 if work is None else work.numel()
    single = m <= 128 and (kind == "bf16" or n < 2048)  # decode schedules that write vectors where K is cut
    for odt in (torch.bfloat16, torch.float32):
        for off in (1, 2, 4):
            want = ops.gemm(x, w, None, ws, out_dtype=odt, split_k=1 if single and off < 4 else 0)
            buf = torch.full((m * n + 16,), 7.0, dtype=odt, device="cuda")
            ops.gemm(x, w, None, ws, out=buf[off:off + m * n].view(m, n), workspace=work)
            assert torch.equal(buf[off:off + m * n].view(m, n), want)
            assert (buf[:off] == 7).all() and (buf[off + m * n:] == 7).all()
    for off in (1, 2, 4):
        act, amax = ops.gemm_silu_mul(x, w, None, ws, split_k=1 if single and off < 4 else 0)
        buf, am = torch.full((m * n // 2 + 16,), 7.0, dtype=torch.bfloat16, device="cuda"), torch.empty_like(amax)
        out = buf[off:off + m * n // 2]
        assert _cabi.load().b200_gemm_silu_mul(x.data_ptr(), w.data_ptr(), out.data_ptr(), 0, 0 if ws is None else ws.data_ptr(), 0, am.data_ptr(),
                                               m, n, k, dt, 0, 0 if work is None else work.data_ptr(), nw, ops._stream()) == 0
        assert torch.equal(out.view(m, -1), act) and torch.equal(am, amax)
        assert (buf[:off] == 7).all() and (buf[off + m * n // 2:] == 7).all()


@pytest.mark.parametrize("m,n,k,cut", [(129, 5120, 27648, True), (300, 1024, 28672, True), (640, 2048, 5632, False), (129, 4096, 14336, False)])
def test_gemm_prompt_schedule(ops, m, n, k, cut):
    """Short prompts against a long K go to the schedule that cuts K over all SMs, the others to the pairs, which do not: the same bits as a
    call that asks for every SM, or others."""
    g = torch.Generator(device="cuda").manual_seed(k)
    x, w = torch.randn((m, k), generator=g, device="cuda").bfloat16(), torch.randn((n, k), generator=g, device="cuda").bfloat16()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    got = ops.gemm(x, w, out_dtype=torch.float32)
    assert torch.equal(got, ops.gemm(x, w, out_dtype=torch.float32, split_k=sms)) == cut


@pytest.mark.parametrize("m,n,k", PAIR_SHAPES + [(300, 1056, 640), (2048, 4096, 4096)])
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_pairs_bf16_against_64_bits(ops, m, n, k, f32):
    """bf16 operands, every epilogue operand.  Products are exact; the tensor cores cut the low bits of every sum of 16 of them: 2^-23 of the
    magnitudes summed so far, k / 16 times at most; then the epilogue's roundings and the one to bf16."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w, bias, res = r(m, k), r(n, k), r(n), r(m, n)
    want = x.double() @ w.double().T + bias.double() + res.double()
    size = x.double().abs() @ w.double().abs().T + bias.double().abs() + res.double().abs()
    got = ops.gemm(x, w, None, None, bias, res, out_dtype=torch.float32 if f32 else torch.bfloat16).double()
    assert ((got - want).abs() <= (k / 16 + 3) * 2.0**-23 * size + (0.0 if f32 else 2.0**-8) * want.abs()).all()


@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_gemm_rope_kv_write_of_a_decode_batch_on_pairs(ops, kind):
    test_gemm_rope_kv_write_matches_two_launches(ops, kind, 100, 64, 8, 128, 2048, 0)


@pytest.mark.parametrize("m,n,k", [(17, 10272, 2048), (64, 9473, 520), (65, 10272, 2048), (128, 18944, 1032)])
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_decode_batches_on_pairs(ops, m, n, k, f32):
    """Up to 128 tokens against rows that fill a wave of pairs, or miss it by one, and a K of a part of a block, whichever schedule takes them."""
    test_gemm_pairs_bf16_against_64_bits(ops, m, n, k, f32)


@pytest.mark.parametrize("m,n,k", [(9, 49153, 2048), (16, 55296, 1032), (17, 49152, 2040), (64, 49001, 1032), (65, 10272, 2048), (97, 18945, 520), (128, 18944, 1032)])
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_decode_batches_that_the_pairs_take(ops, m, n, k, f32):
    """9 to 128 tokens, rows of odd length, a last k-block that is not whole; every one of these runs on the pairs."""
    assert ops.gemm_pair_plan(m, n, k, ops.BF16, has_residual=True)["tokens"] > 0
    test_gemm_pairs_bf16_against_64_bits(ops, m, n, k, f32)


def test_gemm_rope_kv_write_of_a_decode_batch_has_its_linear_call_on_pairs(ops):
    for kind in (ops.BF16, ops.FP8_E4M3):
        assert ops.gemm_pair_plan(100, 80 * 128, 2048, kind)["tokens"] > 0


@pytest.mark.parametrize("m,n,k", [(41, 10272, 2048), (64, 12288, 4096), (17, 16032, 4096), (100, 6144, 4096)])
@pytest.mark.parametrize("kind", ["bf16", "fp8"])
def test_gemm_decode_batches_cut_k_as_their_plan_says(ops, kind, m, n, k):
    """The sums of a call that names no split are those of the split that the plan reports: a longer sum would lose more low bits."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    dt = torch.bfloat16 if kind == "bf16" else torch.float8_e4m3fn
    a, w = torch.randn(m, k, generator=g, device="cuda").to(dt), torch.randn(n, k, generator=g, device="cuda").to(dt)
    split = ops.gemm_decode_plan(m, n, k, ops._ab_dtype(a))["split"]
    assert m > 64 or split > 1
    assert torch.equal(ops.gemm(a, w, out_dtype=torch.float32), ops.gemm(a, w, out_dtype=torch.float32, split_k=split))


@pytest.mark.parametrize("m,n,k", [(129, 3584, 18944), (512, 1024, 28672), (256, 8192, 28672)])
def test_gemm_prompts_against_a_long_k_keep_the_cut_sums(ops, m, n, k):
    """Few tiles that walk a long K: the sums are those of stream-K over every SM, not one long sum a tile."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, w = torch.randn(m, k, generator=g, device="cuda").bfloat16(), torch.randn(n, k, generator=g, device="cuda").bfloat16()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert torch.equal(ops.gemm(a, w, out_dtype=torch.float32), ops.gemm(a, w, out_dtype=torch.float32, split_k=sms))


@pytest.mark.parametrize("m,n,k", [(257, 1001, 192), (777, 6144, 520)])
@pytest.mark.parametrize("f32", [False, True])
def test_gemm_pairs_rows_of_odd_length_and_two_token_tiles(ops, m, n, k, f32):
    test_gemm_pairs_bf16_against_64_bits(ops, m, n, k, f32)


@pytest.mark.parametrize("m,n,k", [(1, 1056, 512), (31, 256, 144), (33, 640, 1152), (64, 992, 256), (65, 256, 128), (128, 1000, 144), (100, 640, 1152), (127, 32, 64), (128, 38144, 256), (96, 5120, 2048),
                                   (1, 3104, 512), (31, 3072, 144), (33, 3220, 1152), (64, 4064, 256), (65, 3328, 128), (128, 4072, 144), (127, 3072, 64), (100, 3104, 1152)])
def test_gemm_weight_only_256_rows(ops, m, n, k):
    """Decode-sized weight-only batches: ragged rows, k and tokens, every epilogue operand; narrow weights on the 128-row schedule, from 3072
    rows on the one of 256.  bf16 operands are exact on both sides: fp32 sums in another order, one bf16 rounding."""
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, bias, res, ws = r(m, k), r(n), r(m, n), torch.rand(n, generator=g, device="cuda") * 0.02
    wq = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    plain = (x.double() @ wq.double().T) * ws.double()
    _assert_close(ops.gemm(x, wq, None, ws, bias, res), (plain + bias.double() + res.double()).cpu())
    assert ((ops.gemm(x, wq, None, ws, out_dtype=torch.float32).double() - plain).abs() <= 2e-6 * (x.double().abs() @ wq.double().abs().T) * ws.double()).all()
    if n % 32 == 0:
        a, amax = ops.gemm_silu_mul(x, wq, None, ws, bias)
        z = ops.gemm(x, wq, None, ws, bias).view(m, -1, 2, 16).float()
        want = torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]
        _assert_close(a, want.reshape(m, -1).cpu())
        assert torch.equal(amax, a.float().abs().view(m, -1, 16).amax(-1))


@pytest.mark.parametrize("m,n,k,launches", [(128, 38144, 1024, 2), (100, 38100, 1040, 2), (128, 38144, 256, 1), (64, 7168, 5120, 1)])
def test_gemm_weight_only_whole_waves_and_a_cut_rest(ops, m, n, k, launches):
    """More tiles than whole waves hold, K long enough: uncut tiles in one launch, the rest cut along K over a cluster in a second (a ragged
    last tile in one case).  Both epilogues against 64 bits, fp32 sums up to 2e-6 of the sum of magnitudes."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((m, k), generator=g, device="cuda").bfloat16()
    wq, ws = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8), torch.rand(n, generator=g, device="cuda") * 0.02
    ops.gemm(x, wq, None, ws)
    before = ops.launch_count()
    got = ops.gemm(x, wq, None, ws, out_dtype=torch.float32)
    assert ops.launch_count() - before == launches
    ref = torch.cat([x.double() @ w.double().T for w in wq.split(8192)], 1) * ws.double()
    size = torch.cat([x.double().abs() @ w.double().abs().T for w in wq.split(8192)], 1) * ws.double()
    assert ((got.double() - ref).abs() <= 2e-6 * size).all()
    if n % 32 == 0:
        a, amax = ops.gemm_silu_mul(x, wq, None, ws)
        z = ref.bfloat16().double().view(m, -1, 2, 16)
        want = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(m, -1)
        _assert_close(a, want.cpu())
        assert torch.equal(amax, a.float().abs().view(m, -1, 16).amax(-1))


@pytest.mark.parametrize("n,k,wide", [(1024, 2048, False), (896, 4864, False), (4096, 2048, True), (7168, 5120, True)])
def test_gemm_weight_only_plan_is_the_one_that_runs(ops, n, k, wide):
    """Narrow weights keep the 128-row schedule: a call without K splits gives the bits of the one that names the plan's; wide ones leave it."""
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn((48, k), generator=g, device="cuda").bfloat16()
    wq = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(n, generator=g, device="cuda")
    plan = ops.gemm_decode_plan(48, n, k, ops.INT8_WO)
    got = ops.gemm(x, wq, None, ws, out_dtype=torch.float32)
    if wide:
        assert plan["ctas_per_sm"] == 1 and 1 <= plan["split"] <= 8 and plan["w_stages"] == 4
    else:
        assert torch.equal(got, ops.gemm(x, wq, None, ws, out_dtype=torch.float32, split_k=plan["split"]))


@pytest.mark.parametrize("m,n,k", [(128, 55296, 5120), (100, 5120, 27648), (65, 7168, 5120), (64, 5120, 27648), (17, 5120, 13824)])
def test_gemm_weight_only_rings_turn_many_times(ops, m, n, k):
    """Long K with the automatic split: 5 to 40 stages per CTA, so that every ring turns several times and both widening groups reuse each
    other's stages.  A stage read before its load has landed would be off by some 4e-3 of the bound's sum; fp32 sums are not by 2e-6."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x = torch.randn((m, k), generator=g, device="cuda").bfloat16()
    wq = torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8)
    ws = torch.rand(n, generator=g, device="cuda") * 0.02
    ref, size = [], []
    for w in wq.split(8192):
        ref.append(x.double() @ w.double().T)
        size.append(x.double().abs() @ w.double().abs().T)
    ref, size = torch.cat(ref, 1) * ws.double(), torch.cat(size, 1) * ws.double()
    first = ops.gemm(x, wq, None, ws, out_dtype=torch.float32)
    assert ((first.double() - ref).abs() <= 2e-6 * size).all()
    for _ in range(20):
        assert torch.equal(ops.gemm(x, wq, None, ws, out_dtype=torch.float32), first)


def test_gemm_is_deterministic_and_stream_k_leaves_workspace_clean(ops):
    """Partial sums are added in fixed order (cluster rank / stream-K contributor) -> same bits every launch, with PDL on
    or off; the stream-K counters at the head of a shared workspace are zero again after every call (that is what lets
    one workspace serve a whole step)."""
    g = torch.Generator().manual_seed(2)
    w = torch.randn(4096, 4096, generator=g).bfloat16().cuda()
    for m in (64, 200):
        x = torch.randn(m, 4096, generator=g).bfloat16().cuda()
        ws = ops.gemm_workspace(m, 4096, 4096, 0, x.device)
        assert (ws is None) == (m <= 128)
        a = ops.gemm(x, w, workspace=ws)
        b = ops.gemm(x, w, workspace=ws)
        old = ops.set_pdl(False)
        try:
            c = ops.gemm(x, w, workspace=ws)
        finally:
            ops.set_pdl(old)
        assert torch.equal(a, b) and torch.equal(a, c)
        if ws is not None:
            assert int(ws[:4096].view(torch.int32).abs().sum()) == 0


def test_gemm_rejects_bad_split(ops):
    from vllm_neuron_b200._cabi import B200Error

    x = torch.zeros(64, 256, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(256, 256, dtype=torch.bfloat16, device="cuda")
    for bad in (9, 16, 8, -1):  # above 8 / more CTAs than k-blocks (256 bf16 = 4 k-blocks) / negative
        with pytest.raises(B200Error):
            ops.gemm(x, w, split_k=bad)


@pytest.mark.parametrize("kind", ["bf16", "fp8", "int8", "int8_wo"])
@pytest.mark.parametrize("m,i,k,ctas", [(64, 14336, 4096, 0), (4, 5632, 2048, 0), (64, 5632, 2048, 2), (100, 96, 512, 4), (64, 5632, 2048, 6),
                                         (128, 3584, 1024, 1), (300, 1792, 512, 0), (300, 1792, 512, 3)])
def test_gemm_silu_mul_matches_unfused(ops, kind, m, i, k, ctas):
    """gate/up GEMM with SiLU*mul in the epilogue == b200_gemm (on the same interleaved rows) followed by b200_silu_mul,
    bit for bit (same tiles, same stream-K cuts, fixed fix-up order), and within the GEMM tolerance of the oracle.  The per-group
    maxima it emits are exact and give the per-token scale of the oracle's quantiser."""
    from oracle import kv_ref

    g = torch.Generator().manual_seed(m + i + k)
    x = torch.randn(m, k, generator=g).bfloat16()
    w = (torch.randn(2 * i, k, generator=g) * 0.03).bfloat16()
    if kind == "bf16":
        xq, xs, wq, ws = x, None, w, None
        want_gu = quant_ref.gemm_ref(x, w)
    elif kind == "int8_wo":
        wq, ws = quant_ref.quantize_weight_per_channel(w, "int8")
        xq, xs = x, None
        want_gu = quant_ref.wo_gemm_ref(x, wq, ws)
    else:
        xq, xs = quant_ref.quantize_act_per_token(x, kind)
        wq, ws = quant_ref.quantize_weight_per_channel(w, kind)
        want_gu = quant_ref.qgemm_ref(xq, xs, wq, ws)
    want = kv_ref.silu_mul_ref(want_gu)
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    wi, si = ops.interleave_gate_up(dev(wq), dev(ws))
    # unfused twin on the SAME row order (same tiles, same stream-K cuts), de-interleaved before SiLU*mul
    gu_i = ops.gemm(dev(xq), wi, dev(xs), si, split_k=ctas)
    idx = torch.arange(i).view(-1, 16)
    perm = torch.cat([idx, idx + i], dim=1).reshape(-1).cuda()
    gu = torch.empty_like(gu_i)
    gu[:, perm] = gu_i
    unfused = ops.silu_mul(gu)
    act, group_amax = ops.gemm_silu_mul(dev(xq), wi, dev(xs), si, split_k=ctas)
    torch.cuda.synchronize()
    assert torch.equal(act, unfused)
    got, wantf = act.float().cpu(), want.float()
    rms = wantf.pow(2).mean().sqrt().item()
    assert ((got - wantf).abs() <= 2e-2 * rms + wantf.abs() * 2.0**-6 + 1e-6).all()
    assert group_amax.shape == (m, 2 * i // 32)
    assert torch.equal(group_amax.cpu(), act.float().abs().view(m, -1, 16).max(dim=2).values.cpu())
    for qk in ("fp8", "int8"):
        q1, s1 = ops.quantize_per_token(act, qk, group_amax=group_amax)
        qw, sw = quant_ref.quantize_act_per_token(act.cpu(), qk)
        assert torch.equal(s1.cpu(), sw)
        assert torch.equal(q1.cpu().view(torch.uint8), qw.view(torch.uint8))


@pytest.mark.parametrize("kind", ["bf16", "fp8", "int8_wo"])
@pytest.mark.parametrize("m,hq,hkv,d,k,split", [
    (64, 32, 8, 128, 4096, 0),   # cfg3 qkv: auto split (cluster of 5) -> fused epilogue
    (64, 4, 1, 128, 4096, 0),    # cfg3 TP=8 shard
    (37, 8, 2, 64, 256, 2),      # D=64: two heads per 128-row tile, q/k/v heads mixed inside one warp; ragged M
    (128, 10, 2, 64, 640, 4),    # tiny-qwen traits (GQA 5, bias) at M=128
    (64, 8, 2, 64, 256, 1),      # no split: library falls back to GEMM + rope kernel
    (200, 8, 2, 64, 256, 0),     # prefill-sized (stream-K): fallback
])
def test_gemm_rope_kv_write_matches_two_launches(ops, kind, m, hq, hkv, d, k, split):
    """b200_gemm_rope_kv_write == b200_gemm followed by b200_rope_kv_write, bit for bit: the qkv row (rotated q,
    un-rotated k, v) and both KV pools (slots < 0 skipped, untouched blocks stay zero)."""
    g = torch.Generator().manual_seed(5)
    n, bs, nb, max_pos = (hq + 2 * hkv) * d, 32, 40, 512
    w = torch.randn(n, k, generator=g) * 0.05
    a = torch.randn(m, k, generator=g)
    bias = (torch.randn(n, generator=g) * 0.1).bfloat16().cuda() if hq == 10 else None
    if kind == "bf16":
        aq, a_s, wq, w_s = a.bfloat16().cuda(), None, w.bfloat16().cuda(), None
    elif kind == "fp8":
        wq, w_s = quant_ref.quantize_weight_per_channel(w.bfloat16(), "fp8")
        aq, a_s = quant_ref.quantize_act_per_token(a.bfloat16(), "fp8")
        aq, a_s, wq, w_s = aq.cuda(), a_s.cuda(), wq.cuda(), w_s.cuda()
    else:
        wq, w_s = quant_ref.quantize_weight_per_channel(w.bfloat16(), "int8")
        aq, a_s, wq, w_s = a.bfloat16().cuda(), None, wq.cuda(), w_s.cuda()
    pos = torch.randint(0, max_pos, (m,), generator=g)
    slots = (torch.randperm((nb - 1) * bs, generator=g)[:m] + bs)
    slots[::7] = -1  # padding rows
    pos[3] = max_pos + 5  # clamped
    pos, slots = pos.cuda(), slots.cuda()
    inv = 1.0 / (10000.0 ** (torch.arange(0, d, 2).float() / d))
    ang = torch.arange(max_pos).float()[:, None] * inv[None, :]
    cos, sin = ang.cos().cuda().contiguous(), ang.sin().cuda().contiguous()

    def pools():
        return (torch.zeros((nb, hkv, bs, d), dtype=torch.bfloat16, device="cuda"),
                torch.zeros((nb, hkv, bs, d), dtype=torch.bfloat16, device="cuda"))

    kp1, vp1 = pools()
    ref = ops.gemm(aq, wq, a_s, w_s, bias, split_k=split)
    ops.rope_kv_write(ref, pos, cos, sin, kp1, vp1, slots, hq)
    kp2, vp2 = pools()
    got = ops.gemm_rope_kv_write(aq, wq, pos, cos, sin, kp2, vp2, slots, hq, a_s, w_s, bias, split_k=split)
    torch.cuda.synchronize()
    assert torch.equal(got.view(torch.int16), ref.view(torch.int16))
    assert torch.equal(kp2.view(torch.int16), kp1.view(torch.int16)) and torch.equal(vp2.view(torch.int16), vp1.view(torch.int16))
    assert kp1.abs().sum().item() > 0 and (kp2[0] == 0).all()


@pytest.mark.parametrize("kind", ["fp8", "int8"])
@pytest.mark.parametrize("m,i,k", [(64, 14336, 4096), (1, 512, 256), (33, 1792, 512), (128, 3584, 1024), (17, 7168, 2048)])
def test_gemm_silu_mul_quant_fused_equals_two_calls(ops, kind, m, i, k):
    """b200_gemm_silu_mul_quant (SiLU*mul + per-token quantisation inside the gate/up GEMM, CTAs meeting at a grid barrier)
    == b200_gemm_silu_mul + b200_quantize_per_token, bit for bit, launch after launch on the same state buffer."""
    g = torch.Generator().manual_seed(m * 7 + i)
    x = (torch.randn(m, k, generator=g) * 0.7).bfloat16()
    w = (torch.randn(2 * i, k, generator=g) * 0.05).bfloat16()
    xq, xs = quant_ref.quantize_act_per_token(x, kind)
    wq, ws = quant_ref.quantize_weight_per_channel(w, kind)
    wi, si = ops.interleave_gate_up(wq.cuda(), ws.cuda())
    state = torch.zeros(1040, dtype=torch.uint8, device="cuda")
    act, gam = ops.gemm_silu_mul(xq.cuda(), wi, xs.cuda(), si)
    want_q, want_s = ops.quantize_per_token(act, kind, group_amax=gam)
    for rep in range(3):  # the state carries over: the epoch-tagged maxima of earlier launches must never leak
        xin = xq.cuda() if rep != 1 else torch.zeros_like(xq).cuda()
        got = ops.gemm_silu_mul_quant(xin, wi, xs.cuda(), si, None, state, kind)
        if got is None:
            pytest.skip("shape does not run as one resident wave")
        torch.cuda.synchronize()
        if rep == 1:
            assert torch.all(got[1] == 1.0) and torch.all(got[0].view(torch.uint8).int() % 128 == 0)  # all-zero rows: scale 1
            continue
        assert torch.equal(got[1], want_s)
        assert torch.equal(got[0].view(torch.uint8), want_q.view(torch.uint8))


SMALL_SHAPES = [(1, 16, 16), (8, 24, 48), (3, 40, 528), (7, 2000, 144), (5, 2416, 1040), (2, 4808, 272), (1, 9600, 80), (8, 2048, 5632), (4, 2320, 2048)]


@pytest.mark.parametrize("m,n,k", SMALL_SHAPES)
@pytest.mark.parametrize("kind", ["bf16", "fp8", "int8", "int8_wo", "int8_wo_16"])
def test_gemm_of_a_few_tokens(ops, m, n, k, kind):
    """Rows that end inside a tile of 16 and 32, k inside a piece of 64 bytes, fewer k-blocks than warps, every CTA size, up to 16 tokens where the
    weights are widened; scale, bias and residual, both output types.  Bound: the roundings of fp32 sums of k products (none for integers),
    tensor cores cutting each of them, then one ulp of the output type per epilogue step."""
    g = torch.Generator().manual_seed(m * n + k)
    if kind == "int8_wo_16":
        m += 8
    x = torch.randn(m, k, generator=g)
    w = torch.randn(n, k, generator=g)
    if kind in ("bf16", "int8_wo", "int8_wo_16"):
        x = x.bfloat16()
        xs = None
    else:
        x = x.clamp(-4, 4).to(torch.float8_e4m3fn) if kind == "fp8" else (20 * x).round().clamp(-127, 127).to(torch.int8)
        xs = torch.rand(m, generator=g) + 0.5
    if kind == "bf16":
        w, ws = w.bfloat16(), None
    else:
        w = w.clamp(-4, 4).to(torch.float8_e4m3fn) if kind == "fp8" else (40 * w).round().clamp(-127, 127).to(torch.int8)
        ws = torch.rand(n, generator=g) + 0.5
    bias, res = torch.randn(n, generator=g).bfloat16(), torch.randn(m, n, generator=g).bfloat16()
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    a64, w64 = x.double(), w.double()
    scale = (1 if xs is None else xs.double()[:, None]) * (1 if ws is None else ws.double())
    want = a64 @ w64.T * scale + bias.double() + res.double()
    size = a64.abs() @ w64.abs().T * scale + bias.double().abs() + res.double().abs()
    steps = 4 if kind == "int8" else 2 * k + 4
    for dtype, ulp in ((torch.float32, 2.0**-24), (torch.bfloat16, 2.0**-8)):
        out = ops.gemm(dev(x), dev(w), dev(xs), dev(ws), dev(bias), dev(res), out_dtype=dtype).double().cpu()
        assert ((out - want).abs() <= steps * 2.0**-24 * size + ulp * want.abs() * 1.01).all()
    again = ops.gemm(dev(x), dev(w), dev(xs), dev(ws), dev(bias), dev(res), out_dtype=torch.bfloat16)
    assert torch.equal(again.double().cpu(), out)


def test_gemm_of_a_few_tokens_on_any_boundary(ops):
    """An output that starts on no 4-byte boundary."""
    from vllm_neuron_b200 import _cabi

    x, w = torch.randn(3, 256).bfloat16().cuda(), torch.randn(40, 256).bfloat16().cuda()
    buf = torch.zeros(3 * 40 + 8, dtype=torch.bfloat16, device="cuda")
    assert _cabi.load().b200_gemm(x.data_ptr(), w.data_ptr(), buf.data_ptr() + 2, 0, 0, 0, 0, 3, 40, 256, ops.BF16, ops.BF16, 0, 0, 0, 0) == 0
    assert torch.equal(buf[1:121].view(3, 40), ops.gemm(x, w)) and not buf[121:].any() and not buf[0]


@pytest.mark.parametrize("m,n,k", [(1, 1024, 512), (8, 512, 4096)])
def test_gemm_of_a_few_tokens_sees_scales_and_biases_that_the_kernel_ahead_wrote(ops, m, n, k):
    """Scale and bias rows that come straight out of another kernel of the library, whose blocks let the next one start early: the same call
    on the same rows, once they are there, gives the same bits."""
    g = torch.Generator().manual_seed(m)
    src, one, zero = torch.randn(8, 3000, n, generator=g).cuda(), torch.ones(n).cuda(), torch.zeros(n).cuda()
    x, w = torch.randn(m, k, generator=g).bfloat16().cuda(), torch.randint(-127, 128, (n, k), generator=g).to(torch.int8).cuda()
    runs = []
    for i in range(8):
        scale = ops.dyt_norm(src[i], one, zero, 1.0, torch.float32)[-1]
        first = ops.gemm(x, w, None, scale)
        bias = ops.dyt_norm(src[i], one, zero, 0.5, torch.bfloat16)[-1]
        runs.append((scale, bias, first, ops.gemm(x, w, None, scale, bias)))
    torch.cuda.synchronize()
    for scale, bias, first, both in runs:
        assert torch.equal(first, ops.gemm(x, w, None, scale)) and torch.equal(both, ops.gemm(x, w, None, scale, bias))


@pytest.mark.parametrize("kind,m,i,k", [("bf16", 1, 512, 2048), ("bf16", 7, 512, 4096), ("bf16", 8, 96, 5632), ("fp8", 7, 512, 8192), ("int8", 3, 1024, 4096),
                                        ("int8_wo", 5, 512, 5120), ("int8_wo", 13, 512, 2048), ("int8_wo", 16, 2048, 4608)])
def test_gemm_silu_mul_of_a_few_tokens(ops, kind, m, i, k):
    """Sizes at which the linear call takes 16 or 8 warps a CTA and this one four: a row's sum is the same."""
    test_gemm_silu_mul_matches_unfused(ops, kind, m, i, k, 0)


@pytest.mark.parametrize("kind,m", [("bf16", 1), ("bf16", 3), ("bf16", 8), ("fp8", 1), ("fp8", 7), ("int8", 8), ("int8_wo", 3), ("int8_wo", 9), ("int8_wo", 16)])
@pytest.mark.parametrize("hq,hkv,d,k", [(4, 1, 128, 4096), (8, 2, 64, 272), (3, 1, 96, 2048), (32, 4, 64, 2048), (2, 2, 32, 144)])
def test_rope_epilogue_of_a_few_tokens(ops, kind, m, hq, hkv, d, k):
    """Rotation and scatter in the epilogue: the bits of the GEMM and the rotation kernel, and what 64 bits give.  A position past the table is
    the last one, a slot below 0 is skipped.  Bound: fp32 sums of k products and one bf16 rounding in front of the rotation, one behind it."""
    g = torch.Generator().manual_seed(m * hq + d)
    n, bs, nb, max_pos = (hq + 2 * hkv) * d, 32, 4, 64
    x, w, bias = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g), torch.randn(n, generator=g).bfloat16()
    x = x.bfloat16() if kind in ("bf16", "int8_wo") else x.clamp(-4, 4).to(torch.float8_e4m3fn) if kind == "fp8" else (20 * x).round().clamp(-127, 127).to(torch.int8)
    w = w.bfloat16() if kind == "bf16" else w.clamp(-4, 4).to(torch.float8_e4m3fn) if kind == "fp8" else (40 * w).round().clamp(-127, 127).to(torch.int8)
    xs = torch.rand(m, generator=g) + 0.5 if kind in ("fp8", "int8") else None
    ws = None if kind == "bf16" else torch.rand(n, generator=g) + 0.5
    pos, slots = torch.randint(0, max_pos, (m,), generator=g), torch.randperm((nb - 1) * bs, generator=g)[:m] + bs
    pos[0] = max_pos + 5
    if m > 1:
        slots[1] = -1
    ang = torch.arange(max_pos).float()[:, None] / 10000.0 ** (torch.arange(0, d, 2).float() / d)
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    pools = [torch.zeros(nb, hkv, bs, d, dtype=torch.bfloat16).cuda() for _ in range(4)]
    args = (dev(x), dev(w))
    got = ops.gemm_rope_kv_write(*args, dev(pos), dev(cos), dev(sin), pools[0], pools[1], dev(slots), hq, dev(xs), dev(ws), dev(bias))
    two = ops.gemm(*args, dev(xs), dev(ws), dev(bias))
    ops.rope_kv_write(two, dev(pos), dev(cos), dev(sin), pools[2], pools[3], dev(slots), hq)
    assert torch.equal(got.view(torch.int16), two.view(torch.int16))
    assert all(torch.equal(pools[i].view(torch.int16), pools[i + 2].view(torch.int16)) for i in (0, 1))
    a64, w64 = x.double(), w.double()
    scale = (1 if xs is None else xs.double()[:, None]) * (1 if ws is None else ws.double())
    want = (a64 @ w64.T * scale + bias.double()).view(m, -1, d)
    size = (a64.abs() @ w64.abs().T * scale + bias.double().abs()).view(m, -1, d)
    err = (4 if kind == "int8" else 2 * k + 4) * 2.0**-24 * size + 2.0**-8 * want.abs() * 1.01
    p = pos.clamp(max=max_pos - 1)
    c, s = cos.double()[p][:, None], sin.double()[p][:, None]

    def turn(v, c, s):
        lo, hi = v[..., :d // 2], v[..., d // 2:]
        return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)

    both = lambda v: torch.cat([v[..., d // 2:], v[..., :d // 2]], -1)  # noqa: E731
    turned = turn(want, c, s)
    cc, ss = torch.cat([c, c], -1).abs(), torch.cat([s, s], -1).abs()
    terr = err * cc + both(err) * ss
    terr = terr + (turned.abs() + terr) * 2.0**-8 * 1.01 + 2.0**-22 * (want.abs() + both(want).abs())
    row = got.double().cpu().view(m, -1, d)
    assert ((row[:, :hq] - turned[:, :hq]).abs() <= terr[:, :hq]).all()
    assert ((row[:, hq:] - want[:, hq:]).abs() <= err[:, hq:]).all()
    kp, vp = (t.double().cpu() for t in pools[:2])
    seen = torch.zeros(nb, bs, dtype=torch.bool)
    for t in range(m):
        if slots[t] < 0:
            continue
        b, o = divmod(int(slots[t]), bs)
        seen[b, o] = True
        assert ((kp[b, :, o] - turned[t, hq:hq + hkv]).abs() <= terr[t, hq:hq + hkv]).all()
        assert ((vp[b, :, o] - want[t, hq + hkv:]).abs() <= err[t, hq + hkv:]).all()
    assert not kp.transpose(1, 2)[~seen].any() and not vp.transpose(1, 2)[~seen].any()


@pytest.mark.parametrize("m,i,k", [(1, 14336, 4096), (8, 14336, 4096), (5, 9600, 1040), (8, 18688, 512), (3, 512, 256), (7, 512, 128)])
def test_gemm_silu_mul_quant_of_a_few_tokens(ops, m, i, k):
    """Token counts that other shapes' GEMMs take to a kernel of their own: the two forms have one order of sums."""
    test_gemm_silu_mul_quant_fused_equals_two_calls(ops, "fp8", m, i, k)
    test_gemm_silu_mul_matches_unfused(ops, "fp8", m, i, k, 0)


@pytest.mark.parametrize("m,n,k,kind,epi,per_sm,lines", [(1, 2048, 5632, "BF16", 0, 1, 4), (8, 2048, 2048, "BF16", 0, 2, 4), (1, 4096, 4096, "FP8_E4M3", 0, 1, 2), (4, 6144, 4096, "FP8_E4M3", 0, 2, 2),
                                                         (4, 32000, 2048, "INT8", 0, 4, 2), (2, 6144, 4096, "BF16", 2, 2, 2), (2, 11264, 2048, "BF16", 1, 4, 2),
                                                         (3, 2048, 8192, "INT8_WO", 0, 1, 3), (16, 2048, 8192, "INT8_WO", 0, 1, 2), (9, 32000, 2048, "INT8_WO", 0, 4, 1)])
def test_plan_of_a_few_tokens(ops, m, n, k, kind, epi, per_sm, lines):
    """CTAs an SM holds (16 warps of it) and lines of a warp in flight, by the size of the weights."""
    got = ops.gemm_decode_plan(m, n, k, getattr(ops, kind), silu_mul=epi)
    assert list(got.values()) == [1, per_sm, lines, lines, per_sm * torch.cuda.get_device_properties(0).multi_processor_count, 0]


@pytest.mark.parametrize("m,n,k,kind,epi,on", [(64, 55296, 5120, "BF16", 0, True), (128, 12288, 4096, "FP8_E4M3", 2, True), (100, 28672, 4096, "INT8", 1, True), (64, 4096, 4096, "BF16", 0, False),
                                               (41, 12288, 4096, "FP8_E4M3", 2, False), (64, 128256, 4096, "INT8_WO", 0, False)])
def test_plan_of_decode_batches_on_pairs(ops, m, n, k, kind, epi, on):
    """The plan of a call that the CTA pairs take is theirs: one CTA an SM, no cut of K, a ring of their stages of 128 rows of weights and their tokens."""
    dt = getattr(ops, kind)
    got, pair = ops.gemm_decode_plan(m, n, k, dt, silu_mul=epi), ops.gemm_pair_plan(m, n, k, dt, silu_mul=epi == 1)
    assert (pair["tokens"] > 0) == on
    if on:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert pair["wide"] == 0 and pair["units"] == -(-m // pair["tokens"]) * -(-n // 256)
        assert (got["split"], got["ctas_per_sm"], got["w_stages"], got["a_stages"], got["cap_ctas"]) == (1, 1, pair["stages"], pair["stages"], sms // 2 * 2)
        assert got["smem"] >= pair["stages"] * (128 + pair["tokens"] // 2) * 128
    else:
        assert ops.gemm_decode_plan(m, n, k, dt, split_k=got["split"], silu_mul=epi) == got or kind == "INT8_WO"
