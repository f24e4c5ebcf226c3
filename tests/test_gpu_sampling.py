"""GPU parity: on-device sampler (b200_topk_candidates + b200_sample_candidates) vs oracle/sampling_ref.py.

Bars: candidate lists (values AND indices) bit-exact -- integer/compare work; sampled ids identical for every row whose
draw is further than 1e-5 (relative to Z) from a decision boundary in the oracle (expf on the two sides may differ by
an ulp or two); top_k == 1 rows identical to b200_argmax."""
import numpy as np
import pytest
import torch

from oracle import sampling_ref as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vllm_neuron_b200 import ops as o

    o.device_check(0)
    return o


def _logits(b, v, seed, scale=3.0):
    return (torch.randn(b, v, generator=torch.Generator().manual_seed(seed)) * scale).float()


@pytest.mark.parametrize("b,v,off", [(64, 128256, 0), (4, 32000, 0), (7, 16032, 48096), (3, 100, 5), (1, 256, 0), (2, 257, 0)])
def test_topk_candidates_bit_exact(ops, b, v, off):
    x = _logits(b, v, b + v)
    if v > 1000:
        x[0, 17] = x[0, v - 3] = x[0].max() + 1          # tie at the top
        x[1 % b, ::2] = x[1 % b, 0]                         # > 1024 equal values around the threshold (ordered-scan path)
        kth = x[2 % b].topk(256).values[-1]
        x[2 % b, 5] = x[2 % b, 900] = kth                  # a few ties exactly at the 256th value
    val, idx = ops.topk_candidates(x.cuda(), idx_offset=off)
    wv, wi = S.topk_candidates_ref(x.numpy(), idx_offset=off)
    assert np.array_equal(val.cpu().numpy(), wv)
    assert np.array_equal(idx.cpu().numpy(), wi)


@pytest.mark.parametrize("v", [1, 1023, 1024, 1025, 4097, 63999, 64000, 64003])
def test_topk_candidates_at_the_ends_of_its_paths(ops, v):
    """Rows sorted whole, rows that go through the radix select, rows with a threshold and a list; among these a sorted one, one masked but for
    40 logits, one constant and one with 5000 equal to its largest, which the list gives up."""
    x = _logits(5, v, v)
    x[1] = x[1].sort().values
    x[2, torch.randperm(v, generator=torch.Generator().manual_seed(v))[: max(v - 40, 0)]] = -float("inf")
    x[3] = 0.25
    x[4, ::13] = x[4].max()
    val, idx = ops.topk_candidates(x.cuda())
    wv, wi = S.topk_candidates_ref(x.numpy())
    assert np.array_equal(val.cpu().numpy(), wv) and np.array_equal(idx.cpu().numpy(), wi)


@pytest.mark.parametrize("b,v,pitch", [(5, 16383, 16383), (5, 16384, 16384), (5, 16387, 16387), (3, 40001, 40004), (80, 16390, 16392), (160, 16384, 16384)])
def test_topk_candidates_of_rows_cut_by_clusters(ops, b, v, pitch):
    """Eight, four and two CTAs a row, rows that do not start on 16 bytes; kinds of rows as above, and one whose values differ in their last bits only."""
    x = torch.zeros(b, pitch)
    x[:, :v] = _logits(b, v, v)
    x[1, :v] = x[1, :v].sort().values
    x[2, :v] = x[2, 0] * (1 + torch.arange(v) % 7 * 2.0**-23)
    if b > 4:
        x[3, torch.randperm(v, generator=torch.Generator().manual_seed(v))[40:]] = -float("inf")
        x[4, :v:13] = x[4, :v].max()
    val, idx = ops.topk_candidates(x.cuda()[:, :v])
    wv, wi = S.topk_candidates_ref(x[:, :v].contiguous().numpy())
    assert np.array_equal(val.cpu().numpy(), wv) and np.array_equal(idx.cpu().numpy(), wi)


@pytest.mark.parametrize("v", [16385, 40000, 128256])
def test_topk_candidates_around_a_full_list(ops, v):
    """Rows that put 1023, 1024 (the list's size), 1025 and almost all of their elements at the threshold, masked ones among them."""
    x = _logits(7, v, v)
    order = torch.randperm(v, generator=torch.Generator().manual_seed(v))
    for row, n in enumerate((1023, 1024, 1025)):
        x[row, order[:n]] = 20.0
    for row, (n, low) in enumerate(((40, -float("inf")), (255, -float("inf")), (300, torch.finfo(torch.float32).min), (0, 1.0)), 3):
        x[row, order[n:]] = low
    val, idx = ops.topk_candidates(x.cuda())
    wv, wi = S.topk_candidates_ref(x.numpy())
    assert np.array_equal(val.cpu().numpy(), wv) and np.array_equal(idx.cpu().numpy(), wi)


def test_constant_row_keeps_the_lowest_indices(ops):
    x = torch.zeros(2, 5000)
    val, idx = ops.topk_candidates(x.cuda())
    assert torch.equal(idx.cpu(), torch.arange(256).expand(2, 256))


@pytest.mark.parametrize("groups", [1, 2, 8])
def test_sampled_ids_match_oracle(ops, groups):
    b, v = 64, 16384 * groups
    x = _logits(b, v, 11 + groups, scale=2.0)
    rng = np.random.default_rng(groups)
    params = np.stack([rng.choice([1, 2, 5, 40, 200, 256], b), rng.choice([1.0, 0.95, 0.8, 0.3], b),
                       rng.choice([1.0, 0.7, 1.5, 0.2], b)], axis=1).astype(np.float32)
    u = rng.random(b).astype(np.float32)
    vs = v // groups
    cands = [ops.topk_candidates(x[:, g * vs:(g + 1) * vs].contiguous().cuda(), idx_offset=g * vs) for g in range(groups)]
    cv = torch.stack([c[0] for c in cands]).contiguous()
    ci = torch.stack([c[1] for c in cands]).contiguous()
    got = ops.sample_candidates(cv, ci, torch.from_numpy(params).cuda(), torch.from_numpy(u).cuda()).cpu().numpy()
    want, margin = S.sample_candidates_ref(cv.cpu().numpy(), ci.cpu().numpy(), params, u)
    # sharded == unsharded in the oracle (merge is exact)
    wv, wi = S.topk_candidates_ref(x.numpy())
    want_full, _ = S.sample_candidates_ref(wv, wi, params, u)
    assert np.array_equal(want, want_full)
    safe = margin > 1e-5
    assert safe.sum() >= b - 3
    assert np.array_equal(got[safe], want[safe]), (got, want)
    greedy = params[:, 0] == 1
    assert greedy.any() and np.array_equal(got[greedy], ops.argmax(x.cuda()).cpu().numpy()[greedy])


def test_sampler_statistics_at_vocab_size(ops):
    """Size-independent property at the BASELINE vocab (128256): over stratified uniforms the empirical distribution of the
    device sampler equals the truncated, renormalised softmax."""
    v, n, k, top_p, temp = 128256, 2048, 12, 0.85, 0.9
    x = _logits(1, v, 5).expand(n, v).contiguous()
    u = ((torch.arange(n) + 0.5) / n).float()
    params = torch.tensor([[k, top_p, temp]], dtype=torch.float32).repeat(n, 1)
    cv, ci = ops.topk_candidates(x.cuda())
    ids = ops.sample_candidates(cv, ci, params.cuda(), u.cuda()).cpu()
    top = x[0].topk(k)
    p = torch.softmax(top.values.double() / temp, 0)
    kept = int(torch.searchsorted(p.cumsum(0), torch.tensor(top_p - 1e-9, dtype=torch.float64)) + 1)
    q = p[:kept] / p[:kept].sum()
    counts = torch.tensor([(ids == top.indices[j]).sum().item() for j in range(kept)], dtype=torch.float64) / n
    assert abs(counts.sum().item() - 1.0) < 1e-12 and (counts - q).abs().max() < 2e-3


@pytest.mark.parametrize("groups,n", [(1, 1), (1, 5), (1, 20), (2, 5), (8, 256)])
def test_logprobs_match_oracle(ops, groups, n):
    """b200_row_lse + b200_gather_logprobs vs oracle/sampling_ref.logprobs_ref (pinned to vLLM's Sampler): token ids and
    ranks identical (integer work), log-probabilities within 1e-5 (fp32 log-sum-exp over the vocabulary vs fp64)."""
    b, vs = 33, 16384
    v = vs * groups
    x = _logits(b, v, 31 + groups, scale=2.5)
    x[0, 5] = x[0, v - 9] = x[0].max() + 1.0           # tie at the top (rank counts both)
    want_greedy = x.argmax(dim=1)
    sampled = want_greedy.clone()
    # half of the rows "sampled" a non-greedy candidate: the r-th most likely token
    order = torch.argsort(x, dim=1, descending=True, stable=True)
    for r in range(0, b, 2):
        sampled[r] = order[r, (7 * r) % 200]
    parts = [x[:, g * vs:(g + 1) * vs].contiguous().cuda() for g in range(groups)]
    cands = [ops.topk_candidates(p, idx_offset=g * vs) for g, p in enumerate(parts)]
    lses = [ops.row_lse(p) for p in parts]
    cv = torch.stack([c[0] for c in cands]).contiguous()
    ci = torch.stack([c[1] for c in cands]).contiguous()
    m = torch.stack([l[0] for l in lses]).contiguous()
    s = torch.stack([l[1] for l in lses]).contiguous()
    if groups == 1:
        cv, ci, m, s = cv[0], ci[0], m[0], s[0]
    ids, lp, rk = ops.gather_logprobs(cv, ci, sampled.cuda(), m, s, n)
    wi, wl, wr = S.logprobs_ref(x.numpy(), sampled.numpy(), n)
    assert np.array_equal(ids.cpu().numpy(), wi)
    assert np.array_equal(rk.cpu().numpy(), wr)
    np.testing.assert_allclose(lp.cpu().numpy(), wl, rtol=0, atol=1e-5)
