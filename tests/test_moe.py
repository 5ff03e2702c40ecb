"""Mixture of experts on the GPU: routing against the oracle's rule, the row path and the grouped
tensor-core prompt path against the fp32 oracle."""
import pytest
import torch

from b200serve.models.config import small_moe, tiny_moe
from b200serve.models.oracle import OracleKV, OracleModel, argmax_low_tie, moe_route
from b200serve.models.weights import random_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,e,k", [(5, 8, 2), (300, 256, 8), (64, 16, 4)])
def test_route_matches_oracle_rule(t, e, k):
    from b200serve.ops import moe as M
    torch.manual_seed(e)
    ld = e + 8
    logits = torch.randn(t, ld)
    logits[0, :e] = 0.0                                   # all equal: ties go to the lowest ids
    logits[1, 3] = logits[1, 1] = 5.0                     # a two-way tie at the top
    idx = torch.zeros(t * k, dtype=torch.int32, device="cuda")
    w = torch.zeros(t * k, dtype=torch.float32, device="cuda")
    M.route(logits.cuda(), ld, t, e, k, idx, w)
    torch.cuda.synchronize()
    ref_idx, ref_w = moe_route(logits[:, :e], k)
    got_idx = idx.cpu().reshape(t, k).long()
    assert got_idx[0].tolist() == list(range(k))
    assert got_idx[1, :2].tolist() == [1, 3]
    # rows whose k-th and (k+1)-th probabilities are not within rounding of each other must agree exactly
    p = torch.softmax(logits[:, :e], -1).sort(descending=True).values
    clear = (p[:, k - 1] - p[:, k]) > 1e-6 if e > k else torch.ones(t, dtype=torch.bool)
    assert torch.equal(got_idx[clear].sort(-1).values, ref_idx[clear].sort(-1).values)
    assert torch.equal(got_idx[clear], ref_idx[clear])
    assert (w.cpu().reshape(t, k)[clear] - ref_w[clear]).abs().max() < 1e-5


@pytest.mark.parametrize("e,k,rule", [(8, 2, (0, 1, 1, 1)), (256, 8, (0, 1, 1, 1)), (64, 6, (1, 1, 1, 1)), (40, 4, (1, 1, 1, 0)), (64, 6, (1, 8, 3, 1)),
                                      (33, 3, (0, 1, 1, 0)), (512, 32, (0, 1, 1, 1))])
def test_route_of_rows_that_are_not_numbers(e, k, rule):
    """A row without enough scores that are numbers gets distinct ids of the experts and NaN weights; the rows beside it, and rows with
    a few NaN scores, are routed as if those experts were not there."""
    from b200serve.ops import moe as M
    torch.manual_seed(e + k)
    logits = torch.randn(9, e)
    logits[1] = float("nan")
    logits[2, torch.randperm(e)[: e - k + 1]] = float("nan")      # one number too few
    logits[3] = -float("inf")
    logits[4] = float("inf")
    logits[5, torch.randperm(e)[: e // 8]] = float("nan")
    clean = logits.clone()
    clean[5] = torch.where(clean[5].isnan(), -30.0, clean[5])
    got, ref = [], []
    for t, out in ((logits, got), (clean, ref)):
        idx, w = torch.full((9 * k,), -1, dtype=torch.int32, device="cuda"), torch.zeros(9 * k, device="cuda")
        M.route(t.cuda(), e, 9, e, k, idx, w, rule=rule)
        torch.cuda.synchronize()
        out += [idx.view(9, k).cpu(), w.view(9, k).cpu()]
    assert all(0 <= int(i) < e for i in got[0].flatten()) and all(len(set(r)) == k for r in got[0].tolist())
    assert got[1][1:3].isnan().any(-1).all()
    for r in (0, 6, 7, 8):
        assert torch.equal(got[0][r], ref[0][r]) and torch.equal(got[1][r], ref[1][r]) and got[1][r].isfinite().all()
    if rule[1] == 1:
        assert torch.equal(got[0][5], ref[0][5])
        if rule[0] or rule[3]:          # (a softmax over all scores has no normaliser)
            assert torch.allclose(got[1][5], ref[1][5], rtol=1e-5, atol=0)


def test_grouped_step_with_a_row_that_is_not_a_number():
    """The other rows of a step get the bits they get beside a row of numbers."""
    from b200serve.ops import lib as K
    from b200serve.ops import moe as M
    torch.manual_seed(5)
    m, e, k, h = 12, 16, 4, 256
    w, x = torch.randn(e, h, device="cuda").bfloat16(), torch.randn(m, h, device="cuda").bfloat16()
    out = []
    for bad in (False, True):
        xx = x.clone()
        if bad:
            xx[7] = float("nan")
        logits, idx, wt = torch.zeros(m, e, device="cuda"), torch.full((m * k,), -1, dtype=torch.int32, device="cuda"), torch.zeros(m * k, device="cuda")
        tickets, groups = (torch.zeros(n, dtype=torch.int32, device="cuda") for n in (3, M.group_words(m * k)))
        M.router_rows(w, xx, logits, m, e, h, e, e, k, False, False, idx, wt, tickets, groups=groups)
        torch.cuda.synchronize()
        K.check_status()
        tab = groups[16:].view(-1, 10)[: int(groups[0])].tolist()
        assert all(0 <= g[0] < e and 1 <= g[1] <= 8 for g in tab)
        assert sorted(p for g in tab for p in g[2: 2 + g[1]]) == list(range(m * k))
        out.append((idx.view(m, k).cpu(), wt.view(m, k).cpu()))
    rows = [r for r in range(m) if r != 7]
    assert torch.equal(out[0][0][rows], out[1][0][rows]) and torch.equal(out[0][1][rows], out[1][1][rows]) and out[1][1][7].isnan().all()


def _teacher_forced(oracle, prompt, toks, margin):
    kv = OracleKV(oracle.cfg)
    logits = oracle.forward(prompt, kv, 0)[-1]
    for i, t in enumerate(toks):
        want = int(argmax_low_tie(logits[None])[0])
        if t != want:
            assert float(logits[want] - logits[t]) < margin, (i, t, want)
        logits = oracle.forward(torch.tensor([t]), kv, len(prompt) + i)[0]


def test_tiny_moe_rows_path_matches_oracle():
    from b200serve.ops import lib as K
    from b200serve.runtime.engine import Engine, Row
    cfg = tiny_moe()
    w = random_weights(cfg, seed=1)
    oracle = OracleModel(w)
    g = torch.Generator().manual_seed(2)
    prompt = torch.randint(0, cfg.vocab, (70,), generator=g)
    eng = Engine(random_weights(cfg, device="cuda", seed=1), max_seqs=1, max_len=256, nsplit_attn=4)
    eng.forward_rows([Row(0, i, int(t)) for i, t in enumerate(prompt[:40])])
    got = eng.logits(40).float().cpu()
    ref = oracle.forward(prompt[:40])
    K.check_status()
    # a near-tie between the k-th and (k+1)-th expert may flip under bf16 activations and moves that
    # row's logits by a whole expert: most rows must be tight, none may be far off
    err = (got - ref).abs().amax(dim=1) / ref.abs().max()
    assert (err < 0.04).float().mean() >= 0.85 and err.max() < 0.25, err
    toks = eng.generate(prompt.tolist(), 12)
    K.check_status()
    _teacher_forced(oracle, prompt, toks, 0.03)


@pytest.mark.parametrize("rows", [4, 9, 24])
def test_steps_by_groups_or_by_pairs(rows, monkeypatch):
    """Both forms of a step's experts in the engine, and which one a step takes."""
    from b200serve.models import moe
    from b200serve.ops import lib as K
    from b200serve.ops import moe as M
    from b200serve.runtime.engine import Engine, Row
    cfg = small_moe()
    g = torch.Generator().manual_seed(rows)
    ids = torch.randint(0, cfg.vocab, (rows,), generator=g)
    ref = OracleModel(random_weights(cfg, seed=4)).forward(ids)
    calls = []
    real = M.gemv_groups
    monkeypatch.setattr(M, "gemv_groups", lambda *a, **kw: (calls.append(1), real(*a, **kw)))
    got = []
    for least in (0, moe.GROUP_BYTES, 1 << 60):
        monkeypatch.setattr(moe, "GROUP_BYTES", least)
        calls.clear()
        eng = Engine(random_weights(cfg, device="cuda", seed=4), max_seqs=1, max_len=256, use_graphs=False, nsplit_attn=4)
        eng.forward_rows([Row(0, i, int(t)) for i, t in enumerate(ids)])
        K.check_status()
        got.append(eng.logits(rows).float().cpu().clone())
        # a row's experts are 5 x 209 KB of int4: 24 rows read 25 MB by pair
        assert (len(calls) == 2 * cfg.n_layers) == (least == 0 or (least < 1 << 60 and rows == 24)) and len(calls) in (0, 2 * cfg.n_layers)
        err = (got[-1] - ref).abs().amax(dim=1) / ref.abs().max()       # a near-tie between experts may flip under bf16 activations
        assert (err < 0.04).float().mean() >= 0.7 and err.max() < 0.25, err
    assert torch.equal(got[1], got[0 if rows == 24 else 2])


@pytest.mark.parametrize("backend", ["bf16", "bf16-resident", "w4"])
def test_small_moe_prompt_path_matches_oracle(backend):
    from b200serve.ops import lib as K
    from b200serve.runtime.engine import Engine
    cfg = small_moe()
    w = random_weights(cfg, seed=4)
    oracle = OracleModel(w)
    g = torch.Generator().manual_seed(6)
    prompt = torch.randint(0, cfg.vocab, (400,), generator=g)
    eng = Engine(random_weights(cfg, device="cuda", seed=4), max_seqs=1, max_len=1024, prefill_backend=backend,
                 nsplit_attn=4)
    first = eng.prefill(0, prompt.tolist(), chunk=256)
    K.check_status()
    assert eng._prefill is not None
    ref = oracle.forward(prompt)[-1]
    got = eng.logits(1)[0].float().cpu()
    assert (got - ref).abs().max() < 0.04 * ref.abs().max()
    eng.decode_begin([0], [first])
    toks = [first] + [eng.decode_step()[0] for _ in range(5)]
    K.check_status()
    _teacher_forced(oracle, prompt, toks, 0.04)
