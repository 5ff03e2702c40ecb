"""Prompt-pass kernels whose tiles or rows were cut anew, against plain 64-bit forms at the edges of their tiles."""
import pytest
import torch
import torch.nn.functional as F

from b200serve.ops import gemm as G
from b200serve.ops import lib as K
from b200serve.utils import quant as Q

pytestmark = pytest.mark.gpu


# rows: one and two 128-row halves, a pair's second half empty, several pairs; columns that end inside a tile, inside a CTA's half, at
# a W4B block's end; k shorter than the ring and longer
@pytest.mark.parametrize("m,n,k", [(129, 256, 64), (128, 512, 128), (256, 264, 320), (257, 640, 576), (300, 1000, 64), (511, 384, 1088), (40, 256, 128),
                                   (1024, 5120, 512), (2049, 776, 256), (130, 40960, 64)])
@pytest.mark.parametrize("bn", [-256, 0])
def test_two_sm_gemm(m, n, k, bn):
    torch.manual_seed(m + n)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), (torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16()
    ref = a.double() @ b.double().T
    # exact products, fp32 sums: a few 2^-24 of the absolute terms; one rounding to bf16 on the way out
    bound = 16 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T)
    out = torch.full((m + 1, n), float("nan"), device="cuda")
    G.gemm_bf16(a, b, out[:m], epi=G.EPI_F32, bn=bn)
    one = torch.empty(m, n, device="cuda")
    G.gemm_bf16(a, b, one, epi=G.EPI_F32, bn=128)
    torch.cuda.synchronize()
    K.check_status()
    assert ((out[:m].double() - ref).abs() <= bound + 1e-9).all() and torch.isnan(out[m]).all()
    assert torch.equal(out[:m], one)            # the same products in the same order as the one-SM form
    resid = torch.randn(m, n, device="cuda").bfloat16()
    got = resid.clone()
    G.gemm_bf16(a, b, got, epi=G.EPI_RESID_ADD, resid=got, bn=bn)
    assert ((got.double() - resid.double() - ref).abs() <= 2.0 ** -8 * (resid.double() + ref).abs() + bound + 1e-9).all()
    if n % 32 == 0:
        act = torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")
        G.gemm_bf16(a, b, act, epi=G.EPI_SILU_MUL, bn=bn)
        v = ref.view(m, n // 32, 2, 16)
        want = (F.silu(v[:, :, 0]) * v[:, :, 1]).reshape(m, n // 2)
        assert ((act.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("n,k", [(128, 64), (100, 256), (1000, 320), (256, 4096), (5120, 1088)])
def test_expanded_weights(n, k):
    """Four blocks per CTA and what is left of them, rows behind the matrix untouched."""
    w = Q.random_w4b(n, k, "cuda", 3)
    out = torch.full((n + 1, k), float("nan"), dtype=torch.bfloat16, device="cuda")
    G.dequant_w4b(w, n, k, out[:n])
    torch.cuda.synchronize()
    assert torch.equal(out[:n], Q.dequant_w4b(w, n).bfloat16()) and torch.isnan(out[n]).all()


@pytest.mark.parametrize("n,k", [(100, 256), (1000, 320)])
def test_expanded_weights_into_a_view(n, k):
    """An output that starts in the middle of an 8-byte word."""
    w = Q.random_w4b(n, k, "cuda", 3)
    flat = torch.full((n * k + 4,), float("nan"), dtype=torch.bfloat16, device="cuda")
    G.dequant_w4b(w, n, k, flat[2: 2 + n * k].view(n, k))
    torch.cuda.synchronize()
    assert torch.equal(flat[2: 2 + n * k].view(n, k), Q.dequant_w4b(w, n).bfloat16()) and torch.isnan(flat[:2]).all() and torch.isnan(flat[-2:]).all()
    with pytest.raises(RuntimeError):
        G.dequant_w4b(w, n, k, flat[1: 1 + n * k].view(n, k))


@pytest.mark.parametrize("m,h", [(512, 64), (513, 2048), (600, 2056), (1000, 4096), (519, 5120), (700, 5128), (512, 8192), (530, 8200), (511, 5120)])
def test_norm_of_prompt_rows(m, h):
    torch.manual_seed(h)
    r, w = (torch.randn(m + 1, h, device="cuda") * 3).bfloat16(), 1 + 0.1 * torch.randn(h, device="cuda")
    x, keep = torch.full((m + 1, h), float("nan"), dtype=torch.bfloat16, device="cuda"), r.clone()
    K.resid_norm(1, m, h, w, 1e-6, r, x, resid_in=r, splits=0)
    torch.cuda.synchronize()
    want = r[:m].double() * torch.rsqrt((r[:m].double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    # one rounding to bf16; the fp32 sum of h squares moves the factor by less than 2^-24 sqrt(h)
    assert ((x[:m].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-30).all()
    assert torch.equal(r, keep) and torch.isnan(x[m]).all()
    few = torch.empty(100, h, dtype=torch.bfloat16, device="cuda")       # a CTA per row: the same bits
    K.resid_norm(1, 100, h, w, 1e-6, r, few, resid_in=r, splits=0)
    assert torch.equal(x[:100], few)


@pytest.mark.parametrize("m,pos0,nq,nkv,d", [(1, 0, 4, 2, 128), (3, 5, 8, 2, 64), (4, 16, 40, 8, 128), (37, 31, 3, 1, 256), (130, 1000, 16, 4, 128), (18, 7, 5, 5, 192)])
def test_rope_append_of_prompt_rows(m, pos0, nq, nkv, d):
    from b200serve.models.oracle import rope_tables
    torch.manual_seed(m)
    ld, blocks = (nq + 2 * nkv) * d, (pos0 + m + 15) // 16 + 1
    qkv = torch.randn(m, ld, device="cuda")
    cos, sin = (t.cuda().contiguous() for t in rope_tables(d, 1e6, pos0 + m + 4))
    table = torch.randperm(blocks + 3, device="cuda")[:blocks].int().view(1, blocks).repeat(2, 1).contiguous()
    kc, vc = (torch.full((blocks + 3, nkv, 16, d), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    q = torch.zeros(m, nq * d, dtype=torch.bfloat16, device="cuda")
    K.rope_append(qkv, 0, 1, m, None, table, blocks, cos, sin, nq, nkv, d, q, kc, vc, None, None, False, req=1, pos0=pos0)
    torch.cuda.synchronize()
    pos = torch.arange(pos0, pos0 + m, device="cuda")
    c, s = (t[pos].double()[:, None] for t in (cos, sin))

    def turned(x):
        a, b = x[..., : d // 2], x[..., d // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], -1)
    v = qkv.double()
    close = lambda got, want: ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()        # noqa: E731  one rounding
    assert close(q.view(m, nq, d), turned(v[:, : nq * d].view(m, nq, d)))
    at = table[1].long()[pos // 16], pos % 16
    assert close(kc[at[0], :, at[1]], turned(v[:, nq * d: (nq + nkv) * d].view(m, nkv, d)))
    assert torch.equal(vc[at[0], :, at[1]], qkv[:, (nq + nkv) * d:].view(m, nkv, d).bfloat16())
    for t in (kc, vc):
        t[at[0], :, at[1]] = 7.0
        assert (t == 7.0).all()


# k blocks around the depths of the tile ring and of the ring of int4 blocks, both tile widths, one tile per CTA and several
@pytest.mark.parametrize("kb", [1, 3, 5, 7, 8, 10, 11, 29])
@pytest.mark.parametrize("m,n,bn", [(130, 776, 256), (2049, 2560, 256), (130, 328, 128), (1500, 2176, 128)])
def test_int4_block_ring(m, n, bn, kb):
    torch.manual_seed(kb)
    k = 64 * kb
    w, a = Q.random_w4b(n, k, "cuda", 5), torch.randn(m, k, device="cuda").bfloat16()
    wb = G.dequant_w4b(w, n, k)
    out = torch.full((m + 1, n), float("nan"), device="cuda")
    G.gemm_w4(a, w, n, k, out[:m], epi=G.EPI_F32, bn=bn)
    torch.cuda.synchronize()
    K.check_status()
    ref, bound = a.double() @ wb.double().T, 16 * 2.0 ** -24 * (a.double().abs() @ wb.double().abs().T)
    assert ((out[:m].double() - ref).abs() <= bound + 1e-9).all() and torch.isnan(out[m]).all()


@pytest.mark.parametrize("n,k", [(256, 64), (1032, 320), (4096, 128)])
def test_blocks_of_few_rows(n, k):
    """Grouped products of blocks of every size around the copies of 32 rows, from int4 blocks and from bf16: unit rows give the weights'
    bf16 bits, whatever their scales; rows beyond a block's last (not a number) reach nothing."""
    rows = [1, 31, 32, 33, 64, 65, 96, 97, 127, 128]
    e = len(rows)
    w = torch.cat([Q.random_w4b(n, k, "cuda", i) for i in range(e)])
    blocks = w.view(-1, 4352)
    blocks[:, :4096] = torch.randint(0, 256, (len(blocks), 4096), device="cuda", dtype=torch.uint8)
    scales = blocks[:, 4096:].view(torch.float16)
    scales[:] = (torch.randn_like(scales, dtype=torch.float32) * 2.0 ** torch.randint(-24, 14, scales.shape, device="cuda")).half()
    per = w.shape[0] // e
    wb = [Q.dequant_w4b(w[i * per: (i + 1) * per], n).bfloat16() for i in range(e)]
    tab = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")        # noqa: E731
    table = (tab(range(e)), tab([128 * i for i in range(e)]), tab(rows), tab([e]), e + 3)
    a = torch.full((128 * e, k), float("nan"), device="cuda").bfloat16()
    for i, r in enumerate(rows):
        a[128 * i: 128 * i + r] = torch.eye(k, device="cuda").repeat(128 // k + 1, 1)[:r]
    for run in (lambda c: G.gemm_w4(a, w, n, k, c, blocks=table, n_experts=e), lambda c: G.gemm_grouped_bf16(a, torch.stack(wb), c, table)):
        c = torch.full((128 * e, n), 7.0, device="cuda").bfloat16()
        run(c)
        torch.cuda.synchronize()
        K.check_status()
        for i, r in enumerate(rows):
            got = c[128 * i: 128 * (i + 1)]
            assert torch.equal(got[:r], wb[i].T.repeat(128 // k + 1, 1)[:r]) and (got[r:] == 7.0).all()


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("grouped", [False, True])
def test_every_scale_expands(bn, grouped):
    """A row for every fp16 there is as its scale, each nibble four times: the bits of the dequantising pass, infinite and not a number
    where that is."""
    n = 65536
    w = Q.random_w4b(n, 64, "cuda", 1)
    blocks = w.view(-1, 4352)
    blocks[:, :4096] = (torch.arange(4096, device="cuda") % 256).to(torch.uint8)
    blocks[:, 4096:].view(torch.int16)[:] = torch.arange(n, device="cuda").to(torch.int16).view(-1, 128)
    wb = G.dequant_w4b(w, n, 64)
    assert int(wb.isnan().all(1).sum()) == 2046 and int(wb.isinf().any(1).sum()) == 2
    finite = wb.isfinite().all(1)
    tab = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")        # noqa: E731
    out = torch.zeros(64, n, device="cuda").bfloat16()
    G.gemm_w4(torch.eye(64, device="cuda").bfloat16(), w, n, 64, out, bn=bn, blocks=(tab([0]), tab([0]), tab([64]), tab([1]), 1) if grouped else None)
    torch.cuda.synchronize()
    K.check_status()
    assert torch.equal(out[:, finite], wb[finite].T) and out[:, ~finite].isnan().all()      # (the zeros of a unit row times infinity are not numbers)


# blocks around the eight whose tiles run together, experts of one block and of several, the last one short; one column of tiles and several
@pytest.mark.parametrize("blocks", [1, 7, 8, 9, 19])
@pytest.mark.parametrize("n,bn", [(200, 128), (648, 128), (1288, 256)])
def test_blocks_in_runs(blocks, n, bn):
    torch.manual_seed(blocks)
    e, k, rows = (blocks + 2) // 3, 192, [128, 97, 33] * 7
    w = torch.cat([Q.random_w4b(n, k, "cuda", i) for i in range(e)])
    per = w.shape[0] // e
    wb = torch.stack([G.dequant_w4b(w[i * per: (i + 1) * per], n, k) for i in range(e)])
    tab = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")        # noqa: E731
    table = (tab([i // 3 for i in range(blocks)]), tab([128 * i for i in range(blocks)]), tab(rows[:blocks]), tab([blocks]), blocks + 2)
    a = torch.randn(128 * blocks, k, device="cuda").bfloat16()
    ref = torch.stack([a[128 * i: 128 * i + 128].double() @ wb[i // 3].double().T for i in range(blocks)])
    bound = 16 * 2.0 ** -24 * torch.stack([a[128 * i: 128 * i + 128].double().abs() @ wb[i // 3].double().abs().T for i in range(blocks)])
    for run in (lambda c: G.gemm_w4(a, w, n, k, c, epi=G.EPI_F32, blocks=table, n_experts=e, bn=bn), lambda c: G.gemm_grouped_bf16(a, wb, c, table, epi=G.EPI_F32, bn=bn)):
        c = torch.full((128 * blocks, n), 7.0, device="cuda")
        run(c)
        torch.cuda.synchronize()
        K.check_status()
        for i, r in enumerate(rows[:blocks]):
            got = c[128 * i: 128 * (i + 1)]
            assert ((got[:r].double() - ref[i, :r]).abs() <= bound[i, :r] + 1e-9).all() and (got[r:] == 7.0).all()


# one tile; a last wave of one, of a few and of half the pairs behind none, one and three whole ones; ragged rows and columns; parts of unequal length
@pytest.mark.parametrize("m,n,k", [(300, 1000, 1088), (256, 19200, 1024), (900, 5120, 4160), (1000, 9728, 1536), (2048, 5640, 2048), (256, 256, 16384)])
@pytest.mark.parametrize("epi", [G.EPI_BF16, G.EPI_F32, G.EPI_SILU_MUL, G.EPI_RESID_ADD])
def test_last_wave_in_parts(m, n, k, epi):
    if epi == G.EPI_SILU_MUL:
        n = n // 32 * 32
    torch.manual_seed(m + n)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), (torch.randn(n, k, device="cuda") * k ** -0.5).bfloat16()
    shape = (m, n // 2 if epi == G.EPI_SILU_MUL else n)
    dt = torch.float32 if epi == G.EPI_F32 else torch.bfloat16
    resid = torch.randn(shape, device="cuda").bfloat16() if epi == G.EPI_RESID_ADD else None
    parts = G.gemm_parts("cuda")
    parts[0].fill_(float("nan"))
    outs = []
    for ws in (None, parts, parts):
        c = torch.full((m + 1, shape[1]), float("nan"), dtype=dt, device="cuda")
        G.gemm_bf16(a, b, c[:m], epi=epi, resid=resid, bn=-256, parts=ws)
        torch.cuda.synchronize()
        assert torch.isnan(c[m]).all() and int(parts[1].abs().sum()) == 0
        outs.append(c[:m].double())
    K.check_status()
    assert torch.equal(outs[1], outs[2])                       # the same bits whichever part comes last
    # Exact products, k sums in fp32: a few 2^-24 of the sum of the terms' sizes; and the tensor core cuts off what does not fit at each of k / 16 steps,
    # up to 2^-23 of a partial sum of about sqrt(k) terms where all k have k * 0.64: 0.2 sqrt(k) 2^-24 of that
    y, bound = a.double() @ b.double().T, (16 + 0.4 * k ** 0.5) * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T)
    if epi == G.EPI_SILU_MUL:            # and what the product makes of that: silu's slope is at most 1.1
        (g, u), (eg, eu) = (t.view(m, n // 32, 2, 16).unbind(2) for t in (y, bound))
        y = (torch.nn.functional.silu(g) * u).reshape(shape)
        bound = (1.1 * eg * u.abs() + eu * torch.nn.functional.silu(g).abs() + 1.1 * eg * eu).reshape(shape) + 2.0 ** -19 * y.abs()
    y = y + resid.double() if resid is not None else y
    bound = bound + (0 if epi == G.EPI_F32 else 2.0 ** -8) * (y.abs() + bound) + 1e-9        # the result's own rounding
    assert all(((o - y).abs() <= bound).all() for o in outs)


# a last wave that is cut: one tile, and few in eight parts; few behind three whole waves; half the pairs in two parts behind one; some in two behind four.
# Ragged rows and columns, parts of unequal length
@pytest.mark.parametrize("m,n,k", [(130, 200, 4928), (300, 1000, 4096), (900, 15000, 3072), (700, 9464, 4096), (1200, 16480, 5120)])
@pytest.mark.parametrize("epi", [G.EPI_BF16, G.EPI_F32, G.EPI_SILU_MUL, G.EPI_RESID_ADD])
def test_last_wave_that_is_cut(m, n, k, epi, monkeypatch):
    made, make = [], G.gemm_parts
    monkeypatch.setattr(G, "gemm_parts", lambda device: made.append(make(device)) or made[-1])
    test_last_wave_in_parts(m, n, k, epi)
    left = int((~made[0][0].isnan()).sum())          # whole parts of 256 x 256 sums, two and more
    assert left % 65536 == 0 and left >= 2 * 65536


# blocks around the eight whose tiles run together, short blocks among them
@pytest.mark.parametrize("blocks", [1, 8, 9, 17])
@pytest.mark.parametrize("n,bn", [(192, 128), (640, 256)])
def test_blocks_that_arrive_and_return(blocks, n, bn):
    """Blocks whose rows are counted as arrived, and rows that go back to where they came from (two buffers of this GPU): the bits of the plain form."""
    torch.manual_seed(blocks)
    e, k, rows = (blocks + 2) // 3, 192, ([128, 97, 33] * 6)[:blocks]
    tab = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")        # noqa: E731
    table = (tab([i // 3 for i in range(blocks)]), tab([128 * i for i in range(blocks)]), tab(rows), tab([blocks]), blocks + 2)
    a, b = torch.randn(128 * blocks, k, device="cuda").bfloat16(), torch.randn(e, n, k, device="cuda").bfloat16()
    live = torch.cat([128 * i + torch.arange(r) for i, r in enumerate(rows)]).cuda()
    full = lambda m, n: torch.full((m, n), 7.0, device="cuda").bfloat16()        # noqa: E731
    want, got = full(len(a), n // 2), full(len(a), n // 2)
    G.gemm_grouped_bf16(a, b, want, table, epi=G.EPI_SILU_MUL, bn=bn)
    G.gemm_grouped_ep(a, b, got, table, G.EPI_SILU_MUL, blk_wait=tab(rows), bn=bn)
    assert torch.equal(want, got)
    want, home = full(len(a), n), [full(len(live), n) for _ in range(2)]
    G.gemm_grouped_bf16(a, b, want, table, bn=bn)
    src = torch.randperm(2 * len(live), device="cuda")[: len(live)]          # buffer and slot of each row
    meta = torch.zeros(len(a), dtype=torch.int32, device="cuda")
    meta[live] = (src % 2 * (1 << 24) + src // 2).int()
    ptrs = torch.tensor([h.data_ptr() for h in home], dtype=torch.int64, device="cuda")
    G.gemm_grouped_ep(a, b, None, table, G.EPI_EP_RETURN, row_src=meta, ret_table=ptrs, bn=bn)
    torch.cuda.synchronize()
    K.check_status()
    back = torch.stack([full(len(live), n), full(len(live), n)])
    back[src % 2, src // 2] = want[live]
    assert torch.equal(torch.stack(home), back)


# slots around a pass of eight (combine) and of 32 (scatter), rows of pieces for some of a CTA and for several rounds; two columns a piece
@pytest.mark.parametrize("h", [2, 130, 136, 2048, 4104])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 33])
@pytest.mark.parametrize("shared", [None, "plain", "gated"])
def test_scatter_and_combine(h, k, shared):
    from b200serve.ops import moe as M
    torch.manual_seed(h + k)
    t, e = 37, 64
    idx = torch.stack([torch.randperm(e, device="cuda")[:k] for _ in range(t)]).int()
    x, resid, sh = (torch.randn(t, h, device="cuda").bfloat16() for _ in range(3))
    w, gate = torch.rand(t, k, device="cuda"), torch.randn(t, 3, device="cuda")
    row_of, blocks = torch.randperm(t * k + 5, device="cuda")[: t * k].int(), torch.randn(t * k + 5, h, device="cuda").bfloat16()
    if h % 8 == 0:
        base = torch.arange(e, device="cuda").int() * t
        rank = torch.zeros(t * k, dtype=torch.int32, device="cuda")
        for i in range(e):
            rank[(idx.view(-1) == i).nonzero().flatten()] = torch.arange(int((idx == i).sum()), device="cuda").int()
        at, xs = torch.zeros(t * k, dtype=torch.int32, device="cuda"), torch.full((e * t, h), float("nan"), device="cuda").bfloat16()
        M.scatter(idx.view(-1), rank, base, t, k, x, h, at, xs)
        assert torch.equal(at, base[idx.view(-1).long()] + rank) and torch.equal(xs[at.long()], x.repeat_interleave(k, 0))
        assert int(xs.isnan().all(-1).sum()) == e * t - t * k
    out = torch.empty_like(resid)
    M.combine(blocks, row_of, w, t, k, h, sh if shared else None, gate if shared == "gated" else None, 3, resid, out)
    torch.cuda.synchronize()
    want = resid.double() + (blocks.double()[row_of.long()].view(t, k, h) * w.double()[..., None]).sum(1)
    if shared:
        want += sh.double() * (torch.sigmoid(gate[:, :1].double()) if shared == "gated" else 1.0)
    size = resid.double().abs() + (blocks.double().abs()[row_of.long()].view(t, k, h) * w.double()[..., None]).sum(1) + sh.double().abs()
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + (k + 2) * 2.0 ** -22 * size).all()       # rounded once; fp32 sums, the gate by a fast exponential


@pytest.mark.parametrize("m", [80, 128, 129, 256, 257])
@pytest.mark.parametrize("n,k", [(1024, 1024), (5120, 5120), (5120, 17408), (16480, 5120)])
def test_int4_linear_on_either_side_of_its_rule(m, n, k):
    """A linear of backend ``w4`` is the product with the weight's bf16 copy, whichever way the rule sends it."""
    from types import SimpleNamespace as N
    from b200serve.runtime.prefill import PrefillRunner
    torch.manual_seed(m)
    w, a = Q.random_w4b(n, k, "cuda", 2), torch.randn(m, k, device="cuda").bfloat16()
    runner = PrefillRunner.__new__(PrefillRunner)
    runner.backend, runner.dev, runner._slab, runner._parts = "w4", torch.device("cuda"), None, None
    out = torch.empty(m, n, device="cuda")
    runner.linear(N(w4b=w, n=n, k=k, _w_bf16=None), a, out, G.EPI_F32)
    torch.cuda.synchronize()
    K.check_status()
    assert (runner._parts is not None) == (runner._slab is not None and G.gemm_in_parts(m, n, k))
    assert (runner._slab is None) == (m <= 256 and G.w4_from_blocks(m, n, k)) and (m > 128 or n * k >= 1 << 24 or runner._slab is None)
    wb = Q.dequant_w4b(w, n).bfloat16().double()
    # as in the last wave's test: fp32 sums, and what the tensor core cuts off
    assert ((out.double() - a.double() @ wb.T).abs() <= (16 + 0.4 * k ** 0.5) * 2.0 ** -24 * (a.double().abs() @ wb.abs().T) + 1e-9).all()


def test_rule_of_int4_linears_follows_what_was_measured():
    """Shapes whose two forms were measured 4 % and more apart, and those too small for two launches."""
    blocks = [(20, 1024, 1024), (128, 2048, 2048), (100, 9216, 2048), (160, 9216, 2048), (128, 12288, 2048), (160, 12288, 2048), (100, 7168, 5120), (160, 7168, 5120),
              (128, 8192, 5120), (256, 8192, 5120), (20, 16480, 5120), (256, 16480, 5120), (128, 22016, 4096), (160, 22016, 4096), (20, 34816, 5120), (256, 34816, 5120)]
    copies = [(129, 1024, 1024), (20, 3072, 2048), (100, 3072, 2048), (128, 2048, 4096), (256, 2048, 4096), (100, 4096, 4096), (160, 4096, 4096), (20, 2048, 6144), (100, 5120, 5120),
              (256, 5120, 5120), (128, 5120, 6144), (20, 4096, 11008), (256, 4096, 11008), (100, 5120, 17408), (256, 5120, 17408)]
    assert [s for s in blocks if not G.w4_from_blocks(*s)] == [] and [s for s in copies if G.w4_from_blocks(*s)] == []


@pytest.mark.parametrize("over", [-400, 0, 1])
def test_experts_from_int4_or_copies(over, monkeypatch):
    """Prompt chunks on both sides of the rule: expanding a tile's blocks gives the bits of the bf16 copies."""
    from b200serve.models import moe
    from b200serve.models.config import small_moe
    from b200serve.models.weights import random_weights
    from b200serve.runtime.engine import Engine
    cfg = small_moe()
    rows = moe.W4_EXPERT_ROWS * cfg.n_experts // cfg.top_k + over
    prompt = torch.randint(0, cfg.vocab, (rows,), generator=torch.Generator().manual_seed(rows)).tolist()
    got = []
    for limit in (moe.W4_EXPERT_ROWS, 0, 1 << 20):
        monkeypatch.setattr(moe, "W4_EXPERT_ROWS", limit)
        eng = Engine(random_weights(cfg, device="cuda", seed=4), max_seqs=1, max_len=1024, prefill_backend="bf16")
        first = eng.prefill(0, prompt, chunk=1024)
        K.check_status()
        got.append((first, eng.logits(1)[0].clone()))
    assert all(g[0] == got[0][0] and torch.equal(g[1], got[0][1]) for g in got)


@pytest.mark.parametrize("tiles", [0, 1 << 20])
def test_resident_copies_or_int4(tiles, monkeypatch):
    """A resident model's experts from its copies or from the blocks: the bits of the model that makes copies anew."""
    from b200serve.models import moe
    from b200serve.models.config import small_moe
    from b200serve.models.weights import random_weights
    from b200serve.runtime.engine import Engine
    cfg = small_moe()
    monkeypatch.setattr(moe, "W4_EXPERT_TILES", tiles)
    prompt = torch.randint(0, cfg.vocab, (200,), generator=torch.Generator().manual_seed(8)).tolist()
    got = []
    for backend in ("bf16", "bf16-resident"):
        eng = Engine(random_weights(cfg, device="cuda", seed=4), max_seqs=1, max_len=1024, prefill_backend=backend)
        got.append((eng.prefill(0, prompt), eng.logits(1)[0].clone()))
        K.check_status()
    assert (getattr(eng.model.w.layers[0], "_experts_bf16", None) is None) == (tiles == 0)
    assert got[0][0] == got[1][0] and torch.equal(got[0][1], got[1][1])
