"""Tensor-core prompt pass: flash attention over the page pool and the chunked prefill runner (GPU)."""
import math

import pytest
import torch

from b200serve.models.config import small_dense
from b200serve.models.oracle import OracleModel, OracleKV, argmax_low_tie
from b200serve.models.weights import random_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,pos0,n_q,n_kv,window", [(128, 0, 2, 1, 0), (300, 0, 8, 2, 0), (200, 150, 4, 4, 0),
                                                    (77, 1000, 5, 1, 0), (300, 0, 4, 2, 100), (260, 700, 4, 1, 40),
                                                    (200, 150, 2, 2, 300), (128, 512, 2, 1, 128)])
def test_attn_prefill_matches_softmax(c, pos0, n_q, n_kv, window):
    from b200serve.ops import lib as K
    torch.manual_seed(c + pos0)
    d = 128
    total = pos0 + c
    max_blocks = (total + 15) // 16 + 3
    num_pages = max_blocks + 8
    perm = torch.randperm(num_pages - 1)[:max_blocks] + 1
    table = perm.to(torch.int32).cuda()
    kc = torch.zeros(num_pages, n_kv, 16, d, dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    k = torch.randn(total, n_kv, d).to(torch.bfloat16)
    v = torch.randn(total, n_kv, d).to(torch.bfloat16)
    for p in range(total):
        kc[perm[p // 16], :, p % 16] = k[p].cuda()
        vc[perm[p // 16], :, p % 16] = v[p].cuda()
    q = torch.randn(c, n_q, d).to(torch.bfloat16)
    out = torch.full((c, n_q * d), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.attn_prefill(q.reshape(c, -1).cuda(), kc, vc, table, out, c, pos0, n_q, n_kv, d, num_pages, max_blocks,
                   1.0 / math.sqrt(d), window=window)
    torch.cuda.synchronize()
    K.check_status()
    g = n_q // n_kv
    kk, vv = k.float().repeat_interleave(g, 1), v.float().repeat_interleave(g, 1)
    sc = torch.einsum("rhd,shd->hrs", q.float(), kk) / math.sqrt(d)
    qpos = pos0 + torch.arange(c)
    masked = torch.arange(total)[None, :] > qpos[:, None]
    if window > 0:      # sliding window: keys at or before qpos - window are skipped tile-wise or masked
        masked = masked | (torch.arange(total)[None, :] <= qpos[:, None] - window)
    sc = sc.masked_fill(masked[None], float("-inf"))
    ref = torch.einsum("hrs,shd->rhd", torch.softmax(sc, -1), vv).reshape(c, -1)
    got = out.float().cpu()
    assert torch.isfinite(got).all()
    assert (got - ref).abs().max() < 0.02 * ref.abs().max() + 2e-3


@pytest.mark.parametrize("backend", ["bf16", "bf16-resident", "int8", "w4", "bf16-windowed", "bf16-hybrid", "int8-hybrid", "w4-hybrid"])
def test_prefill_runner_matches_oracle(backend):
    from b200serve.runtime.engine import Engine
    from b200serve.ops import lib as K
    cfg = small_dense()
    if backend == "bf16-windowed":      # layers 0 and 2 attend to the last 48 positions
        from b200serve.models.config import preset
        cfg, backend = preset("small-windowed"), "bf16"
    if backend.endswith("-hybrid"):     # layers 0 and 2 are gated delta-net layers: GEMM projections + sequential scan
        from b200serve.models.config import preset
        cfg, backend = preset("small-hybrid"), backend.split("-")[0]
    w = random_weights(cfg, seed=3)
    oracle = OracleModel(w)
    g = torch.Generator().manual_seed(5)
    prompt = torch.randint(0, cfg.vocab, (333,), generator=g)
    wc = random_weights(cfg, device="cuda", seed=3)
    eng = Engine(wc, max_seqs=2, max_len=1024, prefill_backend=backend, nsplit_attn=4)
    first = eng.prefill(1, prompt.tolist(), chunk=200)          # two chunks: 200 + 133
    K.check_status()
    assert eng._prefill is not None
    ref_logits = oracle.forward(prompt)[-1]
    got = eng.logits(1)[0].float().cpu()
    tol = 0.08 if backend == "int8" else 0.03
    assert (got - ref_logits).abs().max() < tol * ref_logits.abs().max()
    want = int(argmax_low_tie(ref_logits[None])[0])
    if first != want:
        assert float(ref_logits[want] - ref_logits[first]) < (0.1 if backend == "int8" else 0.03)
    # decode continues from the prefilled cache; judged against the teacher-forced oracle with the
    # undetermined-row rule (a near-tie may go either way)
    eng.decode_begin([1], [first])
    toks = [first] + [eng.decode_step()[0] for _ in range(6)]
    K.check_status()
    kv = OracleKV(cfg)
    logits = oracle.forward(prompt, kv, 0)[-1]
    margin = 0.12 if backend == "int8" else 0.04
    for i, t in enumerate(toks):
        want = int(argmax_low_tie(logits[None])[0])
        if t != want:
            assert float(logits[want] - logits[t]) < margin, (i, t, want)
        logits = oracle.forward(torch.tensor([t]), kv, len(prompt) + i)[0]


# chunks at and around the row count up to which the GEMM expands the int4 blocks itself: whole prompts on either side, prompts whose
# last chunk falls to the other side, a chunk of one row; matrices of different sizes in turn through the workspace
@pytest.mark.gpu
@pytest.mark.parametrize("family", ["small-dense", "small-hybrid", "small-moe"])
@pytest.mark.parametrize("n,chunk", [(128, 128), (129, 256), (129, 128), (300, 256), (300, 128)])
def test_int4_prompt_backend_has_the_bits_of_bf16(family, n, chunk):
    from b200serve.models.config import preset
    from b200serve.ops import lib as K
    from b200serve.runtime.engine import Engine
    from b200serve.runtime.prefill import W4_FUSED_ROWS
    assert W4_FUSED_ROWS == 128
    cfg = preset(family)
    prompt = torch.randint(0, cfg.vocab, (n,), generator=torch.Generator().manual_seed(n)).tolist()
    got = []
    for backend in ("bf16", "w4", "w4a16"):
        eng = Engine(random_weights(cfg, device="cuda", seed=3), max_seqs=2, max_len=1024, prefill_backend=backend, nsplit_attn=4)
        first = eng.prefill(1, prompt, chunk=chunk)
        K.check_status()
        assert eng._prefill.backend == ("bf16" if backend == "bf16" else "w4")
        assert (eng._prefill._slab is None) == (backend != "bf16" and min(n, chunk) <= W4_FUSED_ROWS)
        got.append((first, eng.logits(1)[0].clone(), {k: t.clone() for k, t in {**eng.kv.page_tensors(), **eng.kv.states}.items()}))
    for g in got[1:]:
        assert g[0] == got[0][0] and torch.equal(g[1], got[0][1]) and all(torch.equal(t, got[0][2][k]) for k, t in g[2].items())


@pytest.mark.gpu
def test_int8_kv_prompt_pass_layer_major_matches_row_kernels():
    """An int8 KV cache is filled by the layer-major GEMM pass (bf16 scratch per layer, quantised afterwards); the
    row kernels writing int8 directly are the reference.  A second turn exercises the dequantise-first path."""
    from b200serve.models.config import preset
    from b200serve.models.weights import random_weights
    from b200serve.ops import lib as K
    from b200serve.runtime.engine import Engine
    cfg = preset("small-dense")
    w = random_weights(cfg, device="cuda", seed=6)
    g = torch.Generator().manual_seed(2)
    ids = torch.randint(0, cfg.vocab, (300,), generator=g).tolist()
    more = torch.randint(0, cfg.vocab, (150,), generator=g).tolist()
    ref = Engine(w, max_seqs=1, max_len=1024, kv_dtype="int8", use_graphs=False, prefill_backend="rows")
    ref.prefill(0, ids)
    l_ref1 = ref.model.buf.logits[ref.last_prefill_row].clone()
    ref.prefill(0, more)
    l_ref2 = ref.model.buf.logits[ref.last_prefill_row].clone()
    eng = Engine(w, max_seqs=1, max_len=1024, kv_dtype="int8", use_graphs=False)
    eng.prefill(0, ids, chunk=128)
    assert eng._prefill is not None
    l1 = eng.model.buf.logits[0].clone()
    eng.prefill(0, more, chunk=128)
    l2 = eng.model.buf.logits[0].clone()
    K.check_status()
    for a, b in ((l1, l_ref1), (l2, l_ref2)):
        assert float((a - b).abs().max()) < 0.04 * float(b.abs().max())
    # decode continues on the int8 pages the pass wrote
    t_ref = ref.forward_rows([__import__("b200serve.runtime.engine", fromlist=["Row"]).Row(0, ref.seq_len[0], 7)])
    t = eng.forward_rows([__import__("b200serve.runtime.engine", fromlist=["Row"]).Row(0, eng.seq_len[0], 7)])
    assert float((eng.model.buf.logits[0] - ref.model.buf.logits[0]).abs().max()) < 0.04 * float(l_ref2.abs().max())
