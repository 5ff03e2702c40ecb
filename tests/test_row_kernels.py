"""Kernels that spread a step's rows over the CTAs, against plain 64-bit forms at the edges of their tiles."""
import pytest
import torch
import torch.nn.functional as F

from b200serve.ops import lib as K

pytestmark = pytest.mark.gpu


def _ctrl(slots):
    c = torch.zeros(K.CTRL_WORDS, dtype=torch.int32)
    c[K.CTRL_N_ROWS] = len(slots)
    c[K.CTRL_ROW_REQ: K.CTRL_ROW_REQ + len(slots)] = torch.tensor(slots, dtype=torch.int32)
    return c.cuda()


def _conv_reference(proj, conv_w, state, slots):
    cc = conv_w.shape[0]
    out, state = proj.clone(), state.clone()
    for i, s in enumerate(slots):
        hist = torch.cat([state[s], proj[i, :cc, None]], dim=1)
        out[i, :cc] = F.silu((hist * conv_w).sum(1))
        state[s] = hist[:, 1:]
    return out, state


# (rows of one slot's prompt chunk or slots of a step's rows, key heads, value heads, splits): chunks of 16 rows and their halo of
# 3, columns of four and, with an odd number of value heads, the form of one column per thread
@pytest.mark.parametrize("rows,nk,nv,splits", [(r, 2, 4, 1) for r in (1, 2, 3, 4, 15, 16, 17, 19, 33, 160)] + [
    (50, 1, 3, 2), (16, 1, 1, 1), ([2, 0, 2, 2, 1, 0], 2, 4, 3), ([1], 2, 4, 16), (list(range(5)) * 12, 1, 3, 2), (list(range(64)), 2, 2, 5)])
def test_convolution_over_rows(rows, nk, nv, splits):
    torch.manual_seed(3)
    slots = rows if isinstance(rows, list) else [1] * rows
    m, cc = len(slots), (2 * nk + nv) * 128
    n = cc + nv * 128 + 2 * nv
    part, conv_w = torch.randn(splits, m, n), torch.randn(cc, 4) * 0.5
    state = torch.randn(max(slots) + 2, cc, 3)
    ref, ref_state = _conv_reference(part.double().sum(0), conv_w.double(), state.double(), slots)
    act, st = torch.full((m, n), float("nan"), device="cuda"), state.cuda()
    K.gdn_conv(part.cuda(), splits, m, n, cc, _ctrl(slots) if isinstance(rows, list) else None, conv_w.cuda(), st, act, slot=1)
    torch.cuda.synchronize()
    # sums of `splits` and 4 fp32 terms of size <= ~10: 2^-24 per addition; SiLU through __expf (2 ulp of its argument's magnitude)
    assert (act.double().cpu() - ref).abs().max() < 1e-5
    assert (st.double().cpu() - ref_state).abs().max() < 1e-5


@pytest.mark.parametrize("rows", [3, 40, 700, [1, 0, 1, 1, 2]])
def test_convolution_in_place(rows):
    """The activations in the projection's own memory: the values of a buffer of its own."""
    torch.manual_seed(rows if isinstance(rows, int) else 5)
    slots = rows if isinstance(rows, list) else [1] * rows
    m, cc = len(slots), 1024
    n = cc + 520
    part, conv_w, state = torch.randn(m, n, device="cuda"), torch.randn(cc, 4, device="cuda") * 0.5, torch.randn(3, cc, 3, device="cuda")
    ctrl = _ctrl(slots) if isinstance(rows, list) else None
    act, st, here = torch.empty_like(part), state.clone(), part.clone()
    K.gdn_conv(part, 1, m, n, cc, ctrl, conv_w, st, act, slot=1)
    K.gdn_conv(here, 1, m, n, cc, ctrl, conv_w, state, here, slot=1)
    torch.cuda.synchronize()
    # four products and a SiLU of values up to ~10, which one form may contract to fmas where the other does not
    assert (act - here).abs().max() < 1e-5 and torch.equal(st, state)


@pytest.mark.parametrize("slots", [[0], [2, 0, 1], [1, 1, 1, 0, 0, 2], [0, 1, 0, 2, 1, 0], list(range(3)) * 5])
def test_delta_step_per_slot(slots):
    """Slots interleaved in any order: every slot's rows in order, no slot touched that has none."""
    torch.manual_seed(4)
    nk, nv, d, m = 2, 4, 128, len(slots)
    kd, vd = nk * d, nv * d
    n = 2 * kd + 2 * vd + 2 * nv
    act, state = torch.randn(m, n), torch.randn(4, nv, d, d) * 0.1
    a_log, dt, nw = torch.log(torch.rand(nv) * 4 + 0.5), torch.randn(nv) * 0.5, 1 + 0.1 * torch.randn(d)
    S, ref = state.double(), torch.zeros(m, vd, dtype=torch.float64)
    for i, s in enumerate(slots):
        a = act[i].double()
        q, k, v, z = a[:kd].view(nk, d), a[kd: 2 * kd].view(nk, d), a[2 * kd: 2 * kd + vd].view(nv, d), a[2 * kd + vd: 2 * kd + 2 * vd].view(nv, d)
        b, al = a[2 * kd + 2 * vd: 2 * kd + 2 * vd + nv], a[2 * kd + 2 * vd + nv:]
        q = (q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(nv // nk, 0)
        k = (k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(nv // nk, 0)
        T = S[s] * torch.exp(-torch.exp(a_log.double()) * F.softplus(al + dt.double()))[:, None, None]
        T = T + torch.einsum("hi,hj->hij", k, (v - torch.einsum("hij,hi->hj", T, k)) * torch.sigmoid(b)[:, None])
        S[s] = T
        o = torch.einsum("hij,hi->hj", T, q)
        ref[i] = (o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-6) * nw.double() * F.silu(z)).reshape(vd)
    st, out = state.cuda(), torch.zeros(m, vd, dtype=torch.bfloat16, device="cuda")
    K.gdn_step(act.cuda(), m, n, nk, nv, d, _ctrl(slots), a_log.cuda(), dt.cuda(), nw.cuda(), 1e-6, st, out)
    torch.cuda.synchronize()
    assert (st.double().cpu() - S).abs().max() < 1e-4 * S.abs().max()
    assert (out.double().cpu() - ref).abs().max() < 2.0 ** -8 * ref.abs().max() + 1e-4       # one rounding to bf16
    assert torch.equal(st[3].cpu(), state[3])


# rows, slots per row, routed experts, shared slots, hidden, expert width: rows of an expert below, at and beyond a group of eight;
# n-blocks in pairs and a lone one; widths whose last ring stage is short
@pytest.mark.parametrize("m,k,e,shared,h,f", [(8, 2, 4, 0, 256, 128), (1, 1, 3, 1, 64, 192), (9, 4, 16, 1, 512, 256), (64, 8, 256, 1, 2048, 512),
                                              (33, 8, 8, 1, 320, 64), (64, 1, 1, 1, 128, 320), (17, 3, 64, 0, 4096, 448)])
def test_grouped_experts(m, k, e, shared, h, f):
    """Routing in slices, the table of groups, and both matrices of every expert against its rows in fp64."""
    from b200serve.ops import moe as M
    from b200serve.utils import quant as Q
    torch.manual_seed(m + h)
    ks, dev = k + shared, "cuda"
    ids = e + shared
    w_r = torch.randn((e + shared + 7) // 8 * 8, h, device=dev).div_(h ** 0.5).bfloat16()
    x = torch.randn(m, h, device=dev).bfloat16()
    ld = w_r.shape[0]
    logits, idx = torch.zeros(m, ld, device=dev), torch.full((m * ks,), -1, dtype=torch.int32, device=dev)
    wt, tickets = torch.zeros(m * ks, device=dev), torch.zeros((m + 7) // 8 + 1, dtype=torch.int32, device=dev)
    groups = torch.zeros(M.group_words(m * ks), dtype=torch.int32, device=dev)
    for t in (tickets, torch.zeros(1, dtype=torch.int32, device=dev)):          # slices side by side, or one
        groups.zero_()
        M.router_rows(w_r, x, logits, m, e + shared, h, ld, e, k, bool(shared), bool(shared), idx, wt, t, groups=groups)
        torch.cuda.synchronize()
        ref = x.double() @ w_r.double().T
        assert (logits.double() - ref)[:, : e + shared].abs().max() < 1e-4 and int(t.abs().sum()) == 0
        n, tab = int(groups[0]), groups[16:].view(-1, 10).cpu()
        seen = []
        for g in tab[:n].tolist():
            assert 1 <= g[1] <= 8
            seen += g[2: 2 + g[1]]
            assert all(int(idx[p]) == g[0] for p in g[2: 2 + g[1]])
        assert sorted(seen) == list(range(m * ks)) and n <= M.max_groups(m * ks, ids)
    gu, dn = (torch.cat([Q.random_w4b(r, c, dev, s0 + i) for i in range(ids)]) for r, c, s0 in ((2 * f, h, 100), (h, f, 5)))
    per_gu, per_dn = gu.numel() // ids, dn.numel() // ids
    up = torch.full((m * ks, 2 * f), float("nan"), device=dev)
    out = torch.full((m * ks, h), float("nan"), device=dev)
    most = M.max_groups(m * ks, ids)
    alt = dict(alt_w=gu.view(-1)[e * per_gu:].clone(), alt_id=e) if shared else {}
    M.gemv_groups(gu, per_gu, groups, most, x, ks, h * 2, up, 2 * f, h, h, **alt)
    alt = dict(alt_w=dn.view(-1)[e * per_dn:].clone(), alt_id=e) if shared else {}
    M.gemv_groups(dn, per_dn, groups, most, up, 1, 2 * f * 4, out, h, f, 2 * f, x_mode=1, **alt)
    torch.cuda.synchronize()
    K.check_status()
    nb_gu, nb_dn = gu.shape[0] // ids, dn.shape[0] // ids
    for i in sorted(set(idx.tolist())):
        pick = (idx == i).nonzero().flatten()
        wu = Q.dequant_w4b(gu[i * nb_gu: (i + 1) * nb_gu], 2 * f).double()
        y = x[pick // ks].double() @ wu.T
        # activations are 15-bit integers against the largest of 64: 2^-15 of it per product, averaged over the row
        assert (up[pick].double() - y).norm() < 1e-4 * y.norm()
        v = up[pick].double().view(len(pick), f // 16, 2, 16)
        a = (F.silu(v[:, :, 0]) * v[:, :, 1]).reshape(len(pick), f)
        z = a @ Q.dequant_w4b(dn[i * nb_dn: (i + 1) * nb_dn], h).double().T
        # the product is rounded to bf16 on the way in, once per element: 2^-9 each, averaged over the row
        assert (out[pick].double() - z).norm() < 2.0 ** -8 * z.norm()


# rows at the edges of the four instances (16, 32, 48 and 64 token rows); splits with unequal and lone groups; n not a multiple of 128; more items than SMs
@pytest.mark.parametrize("m,n,k,splits", [(1, 128, 64, 1), (9, 256, 128, 2), (16, 300, 320, 1), (17, 128, 704, 3), (31, 1000, 1024, 4), (32, 5120, 640, 4),
                                          (33, 640, 448, 7), (48, 128, 1088, 16), (49, 20480, 256, 2), (64, 384, 5120, 7)])
@pytest.mark.parametrize("fold", [False, True])
def test_linears_on_rows(m, n, k, splits, fold):
    from b200serve.utils import quant as Q
    torch.manual_seed(n + m)
    dev, per = "cuda", (-(-(k // 64) // splits) + 3) // 4 * 4
    splits = -(-(k // 64) // per)
    w = Q.random_w4b(n, k, dev, 7)
    wf = Q.dequant_w4b(w, n).double()
    x = torch.randn(m, k, device=dev).bfloat16()
    xr = torch.zeros(K.rows_pad(m) * k * 2, dtype=torch.uint8, device=dev)
    xr.view(-1)[:] = 0xff          # rows that are not staged are NaN
    part = torch.full((splits, m, n), float("nan"), device=dev)
    K.stage_rows(x, m, k, xr)
    nb = (n + 127) // 128
    tickets, ssq = torch.zeros(nb, dtype=torch.int32, device=dev), torch.zeros(m, nb, device=dev)
    resid = torch.randn(m, n, device=dev).bfloat16()
    r0 = resid.clone()
    args = dict(fold_tickets=tickets, fold_resid=resid, fold_ssq=ssq) if fold else {}
    K.gemm_w4_rows(w, xr, part, m, n, k, splits, **args)
    torch.cuda.synchronize()
    K.check_status()
    ref = x.double() @ wf.T
    # exact products; k sums in fp32 whatever the order: a few 2^-24 of the terms' root sum of squares
    bound = 16 * 2.0 ** -24 * (x.double().abs() @ wf.abs().T)
    assert ((part.double().sum(0) - ref).abs() <= bound + 1e-12).all()
    for s in range(splits):
        lo, hi = s * per * 64, min(k, (s + 1) * per * 64)
        assert (part[s].double() - x[:, lo:hi].double() @ wf[:, lo:hi].T).norm() < 1e-5 * ref.norm()
    if fold:
        want = r0.double() + ref
        assert ((resid.double() - want).abs() <= 2.0 ** -8 * want.abs() + bound + 1e-6).all() and int(tickets.abs().sum()) == 0
        sq = torch.nn.functional.pad(resid.double() ** 2, (0, nb * 128 - n)).view(m, nb, 128).sum(-1)
        assert (ssq.double() - sq).abs().max() < 1e-5 * sq.max()


# n-blocks alone and in pairs, whose last one is alone
@pytest.mark.parametrize("m,n,k,splits", [(16, 9472, 512, 2), (17, 9473, 512, 2), (40, 2048, 2048, 8), (64, 9601, 512, 2)])
@pytest.mark.parametrize("fold", [False, True])
def test_linears_on_rows_in_pairs_and_alone(m, n, k, splits, fold):
    test_linears_on_rows(m, n, k, splits, fold)


# rings of 8, 8, 7 and 6 stages that go round several times, n-blocks alone (21 stages) and in pairs (12 and 9), the last stage with one group and the last
# pair with one block; two items a CTA, the ring's turn in the middle of one
@pytest.mark.parametrize("m", [16, 32, 48, 64])
@pytest.mark.parametrize("n,k,splits", [(300, 2624, 1), (10000, 2624, 2), (37890, 1344, 1)])
def test_linears_on_rows_of_many_stages(m, n, k, splits):
    test_linears_on_rows(m, n, k, splits, n < 20000)


# each instance: copies that end before the ring is full, in its second turn, in a CTA's second item
@pytest.mark.parametrize("m,n,k,splits,stages", [(9, 640, 2560, 1, 1), (24, 300, 2560, 2, 5), (40, 38100, 1280, 1, 11), (64, 2048, 5120, 2, 13)])
def test_linears_on_rows_whose_waits_run_out(m, n, k, splits, stages):
    """Copies that never come: the call ends, says so, counts its tickets, and gives tensor memory back: the next calls have the bits they had before."""
    from b200serve.utils import quant as Q
    torch.manual_seed(m)
    w, x = Q.random_w4b(n, k, "cuda", 7), torch.randn(m, k, device="cuda").bfloat16()
    nb = (n + 127) // 128
    xr, tickets, ssq = torch.zeros(K.rows_pad(m) * k * 2, dtype=torch.uint8, device="cuda"), torch.zeros(nb, dtype=torch.int32, device="cuda"), torch.zeros(m, nb, device="cuda")
    K.stage_rows(x, m, k, xr)

    def sums(**how):
        part, resid = torch.zeros(splits, m, n, device="cuda"), torch.zeros(m, n, device="cuda").bfloat16()
        K.gemm_w4_rows(w, xr, part, m, n, k, splits, fold_tickets=tickets, fold_resid=resid, fold_ssq=ssq, **how)
        torch.cuda.synchronize()
        return part
    want = sums()
    K.check_status()
    sums(stages=stages)
    said = K.status()
    K.status_clear()
    assert set(said) == {"gemmrows"} and int(tickets.abs().sum()) == 0
    for _ in range(3):
        assert torch.equal(sums(), want)
    K.check_status()


@pytest.mark.parametrize("m,n,k", [(16, 38500, 192), (17, 19300, 64), (48, 19100, 320), (64, 38016, 128)])
def test_linears_on_rows_keep_every_weight(m, n, k):
    """Unit rows give the weights themselves, bit by bit: all sixteen nibbles in every place, scales of any size; more pairs of blocks than
    SMs, the last one alone in odd numbers."""
    from b200serve.utils import quant as Q
    w = Q.random_w4b(n, k, "cuda", m)
    blocks = w.view(-1, 4352)
    blocks[:, :4096] = torch.randint(0, 256, (len(blocks), 4096), device="cuda", dtype=torch.uint8)
    scales = blocks[:, 4096:].view(torch.float16)
    scales[:] = (torch.randn_like(scales, dtype=torch.float32) * 2.0 ** torch.randint(-20, 14, scales.shape, device="cuda")).half()
    wf = Q.dequant_w4b(w, n)
    part, xr = torch.empty(1, m, n, device="cuda"), torch.zeros(K.rows_pad(m) * k * 2, dtype=torch.uint8, device="cuda")
    for at in range(0, k, m):
        x = torch.eye(k, device="cuda")[at: at + m]
        x = torch.nn.functional.pad(x, (0, 0, 0, m - len(x))).bfloat16()
        part.fill_(float("nan"))
        K.stage_rows(x, m, k, xr)
        K.gemm_w4_rows(w, xr, part, m, n, k, 1)
        torch.cuda.synchronize()
        assert torch.equal(part[0, : min(m, k - at)], wf[:, at: at + m].T.float())
    K.check_status()


# router rows around the tiles of 16, rows around the slices of eight, widths that leave pieces of a 32-k chunk; slices side by side or one after another
@pytest.mark.parametrize("tickets", [1, 16])
@pytest.mark.parametrize("m,e,h", [(1, 8, 8), (7, 15, 200), (8, 16, 64), (9, 17, 2056), (33, 257, 2048), (64, 500, 136)])
def test_router_logits(m, e, h, tickets):
    from b200serve.ops import moe as M
    torch.manual_seed(m + e)
    w, x = (torch.randn(e, h, device="cuda") * h ** -0.5).bfloat16(), torch.randn(m, h, device="cuda").bfloat16()
    ld, k = (e + 7) // 8 * 8, 4
    lg = torch.full((m, ld), float("nan"), device="cuda")
    idx, tw, tk = torch.zeros(m * k, dtype=torch.int32, device="cuda"), torch.zeros(m * k, device="cuda"), torch.zeros(tickets, dtype=torch.int32, device="cuda")
    M.router_rows(w, x, lg, m, e, h, ld, e, k, False, False, idx, tw, tk)
    torch.cuda.synchronize()
    ref = x.double() @ w.double().T
    # exact products, fp32 sums of h terms
    assert ((lg[:, :e].double() - ref).abs() <= 16 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-12).all() and torch.isnan(lg[:, e:]).all()
    assert torch.equal(idx.view(m, k).long(), torch.sort(lg[:, :e], dim=-1, descending=True, stable=True).indices[:, :k]) and int(tk.abs().sum()) == 0


@pytest.mark.parametrize("m,e,h", [(1, 256, 2048), (48, 257, 2048), (64, 64, 4096), (5, 64, 512), (20, 33, 1000)])
def test_router_logits_are_fp32_sums(m, e, h):
    """Errors of the size that additions in fp32 make, not a chain of additions that cut off.  Root mean squares in units of 2^-24: a chunk of 32 k is two MMAs that may cut
    off up to 2 units of it each, at most 2 * 4 / 3 over all chunks; three levels of a tree in a warp, three over the warps and a chain of two below 7 / 3."""
    from b200serve.ops import moe as M
    torch.manual_seed(m + e)
    w, x = (torch.randn(e, h, device="cuda") * h ** -0.5).bfloat16(), torch.randn(m, h, device="cuda").bfloat16()
    ld, k = (e + 7) // 8 * 8, 4
    lg = torch.zeros(m, ld, device="cuda")
    idx, tw, tk = torch.zeros(m * k, dtype=torch.int32, device="cuda"), torch.zeros(m * k, device="cuda"), torch.zeros(16, dtype=torch.int32, device="cuda")
    M.router_rows(w, x, lg, m, e, h, ld, e, k, False, False, idx, tw, tk)
    torch.cuda.synchronize()
    ref = x.double() @ w.double().T
    assert (lg[:, :e].double() - ref).norm() <= 5 ** 0.5 * 2.0 ** -24 * ref.norm()
    alone = torch.zeros_like(lg)
    for i in range(m):
        M.router_rows(w, x[i:], alone[i:], 1, e, h, ld, e, k, False, False, idx, tw, tk)
    assert torch.equal(lg, alone)          # whatever the company


# one group, a stage and a lone group, unequal splits; n not a multiple of 128
@pytest.mark.parametrize("n,k,splits", [(128, 64, 1), (300, 320, 1), (1000, 704, 3), (640, 1024, 2)])
@pytest.mark.parametrize("fed", [False, True])
def test_few_rows_have_the_bits_of_eight(n, k, splits, fed):
    """Up to four rows put both limbs into the columns of one integer MMA: the sums of a step of eight rows, bit by bit."""
    from b200serve.utils import quant as Q
    torch.manual_seed(n)
    w, x = Q.random_w4b(n, k, "cuda", 3), torch.randn(8, k, device="cuda").bfloat16()
    x[2, 64:] = 0
    x[1] *= 1e4

    def sums(m):
        out = torch.full((splits, m, n), float("nan"), device="cuda")
        if fed:
            xq, gs = torch.zeros(m * k * 2, dtype=torch.uint8, device="cuda"), torch.zeros(K.quant_slots(m) * (k // 64) * 2, dtype=torch.int32, device="cuda")
            K.quant_x(x[:m].contiguous(), m, k, xq, gs)
            K.gemv_w4_fused(w, xq, out, m, n, k, splits, x_mode=3, norm_ssq=gs)
        else:
            K.gemv_w4(w, x[:m].contiguous(), out, m, n, k, splits)
        torch.cuda.synchronize()
        K.check_status()
        return out
    want = sums(8)
    ref = x.double() @ Q.dequant_w4b(w, n).double().T
    assert (want.double().sum(0) - ref).norm() < 1e-4 * ref.norm()
    for m in range(1, 6):
        assert torch.equal(sums(m), want[:, :m])


@pytest.mark.parametrize("m", [3, 16, 40])
def test_staged_rows_of_every_kind(m):
    """SiLU(gate) * up of split sums, normalised residual rows, and the attention merge's own rows, each against a plain row form of the
    same values."""
    torch.manual_seed(m)
    dev, k, s_in = "cuda", 640, 3
    pad = K.rows_pad(m)

    def unstaged(xr):
        a = xr.view(torch.bfloat16).view(k // 64, pad, 8, 8)[:, :m]                   # [group][row][chunk][element]
        rows = torch.arange(m, device=dev)
        a = torch.stack([a[:, rows, (i ^ (rows & 7))] for i in range(8)], dim=2)      # chunks in order
        out = torch.empty(m, k // 64, 64, dtype=torch.bfloat16, device=dev)
        for i in range(8):
            for t in range(4):
                for e in range(2):
                    out[:, :, 32 * (i >> 2) + 16 * (i & 1) + 4 * t + ((i >> 1) & 1) + 2 * e] = a[:, :, i, 2 * t + e].T
        return out.view(m, k)
    xr = torch.zeros(pad * k * 2, dtype=torch.uint8, device=dev)
    x = torch.randn(m, k, device=dev).bfloat16()
    K.stage_rows(x, m, k, xr)
    assert torch.equal(unstaged(xr), x)
    part = torch.randn(s_in, m, 2 * k, device=dev)
    K.stage_rows(part, m, k, xr, x_mode=1, s_in=s_in, x_slice=m * 2 * k)
    v = part.sum(0).double().view(m, k // 16, 2, 16)
    want = (F.silu(v[:, :, 0]) * v[:, :, 1]).reshape(m, k)
    assert ((unstaged(xr).double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()
    nw = 1 + 0.1 * torch.randn(k, device=dev)
    ssq = (x.float() ** 2).view(m, k // 128, 128).sum(-1).contiguous()
    K.stage_rows(x, m, k, xr, x_mode=2, norm_w=nw, norm_ssq=ssq, norm_eps=1e-6)
    want = x.double() * torch.rsqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-6) * nw.double()
    assert ((unstaged(xr).double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
    heads, ns = k // 128, 5
    o, ml = torch.randn(m, heads, ns, 128, device=dev), torch.rand(m, heads, ns, 2, device=dev) + 0.5
    out = torch.zeros(m, k, dtype=torch.bfloat16, device=dev)
    xr.zero_()
    rc = K.lib().b2_attn_merge_quant(K._p(o), K._p(ml), K._p(out), m, heads, ns, 128, K._p(xr), None, pad, K._stream())
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(unstaged(xr), out) and out.abs().sum() > 0


@pytest.mark.parametrize("m", [17, 31, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("n,k", [(64, 64), (100, 192), (1000, 512), (4160, 1024)])
def test_head_of_many_rows(m, n, k):
    """One pass for up to 64 rows: the bits of the 16-row form, and its arg-max candidates."""
    torch.manual_seed(m + n)
    w, x = (torch.randn(n, k, device="cuda") * 0.05).bfloat16(), torch.randn(m, k, device="cuda").bfloat16()
    w[n // 2] = w[n // 3]                      # ties between rows
    nc = K.head_ncand(n)
    out, cv, ci = torch.full((m, n), float("nan"), device="cuda"), torch.zeros(m, nc, device="cuda"), torch.zeros(m, nc, dtype=torch.int32, device="cuda")
    K.head_gemv(w, x, out, m, n, k, cv, ci, n_valid=n - 3)
    for m0 in range(0, m, 16):
        part = x[m0: m0 + 16].contiguous()
        o1, v1, i1 = torch.zeros(len(part), n, device="cuda"), torch.zeros(len(part), nc, device="cuda"), torch.zeros(len(part), nc, dtype=torch.int32, device="cuda")
        K.head_gemv(w, part, o1, len(part), n, k, v1, i1, n_valid=n - 3)
        torch.cuda.synchronize()
        assert torch.equal(out[m0: m0 + 16], o1) and torch.equal(cv[m0: m0 + 16], v1) and torch.equal(ci[m0: m0 + 16], i1)
    ref = x.double() @ w.double().T
    assert ((out.double() - ref).abs() <= 16 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-9).all()


# two token tiles: k blocks around what a stage and the two groups of warps take in turn, ends of blocks and of the row tiles
@pytest.mark.parametrize("m", [9, 15, 16])
@pytest.mark.parametrize("n,k,splits", [(128, 64, 1), (300, 320, 1), (256, 704, 3), (1000, 1088, 2), (5120, 1024, 4)])
def test_integer_gemv_of_two_token_tiles(m, n, k, splits):
    from b200serve.utils import quant as Q
    torch.manual_seed(n + m)
    w, x = Q.random_w4b(n, k, "cuda", 7), torch.randn(m, k, device="cuda").bfloat16()
    wf = Q.dequant_w4b(w, n).double()
    out, again, one = (torch.full((splits, m, n), float("nan"), device="cuda") for _ in range(3))
    K.gemv_w4(w, x, out, m, n, k, splits)
    K.gemv_w4(w, x, again, m, n, k, splits)
    torch.cuda.synchronize()
    K.check_status()
    # activations are 15-bit integers per 64-k group: half a step of the group's largest, 2^-15, on every weight; fp32 sums
    top = x.double().abs().view(m, k // 64, 64).amax(-1).repeat_interleave(64, -1)
    bound = 2.0 ** -14 * (top @ wf.abs().T) + 16 * 2.0 ** -24 * (x.double().abs() @ wf.abs().T)
    assert ((out.double().sum(0) - x.double() @ wf.T).abs() <= bound).all() and torch.equal(out, again)


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k,splits", [(32, 64, 1), (40, 256, 1), (72, 768, 1), (64, 832, 2), (1000, 2112, 3)])
def test_bf16_gemv_ring(m, n, k, splits):
    """Steps per warp below, at and above the ring's depth, warps without a step, columns that end inside a tile."""
    from b200serve.ops import latent as L
    torch.manual_seed(k + m)
    w, x = (torch.randn(n, k, device="cuda") * 0.05).bfloat16(), torch.randn(m, k, device="cuda").bfloat16()
    out = torch.full((splits, m, n), float("nan"), device="cuda")
    L.gemv_bf16(w, x, out, m, n, k, splits)
    torch.cuda.synchronize()
    K.check_status()
    bound = 16 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((out.double().sum(0) - x.double() @ w.double().T).abs() <= bound + 1e-9).all()


# contexts at the edges of pages, of a warp's keys and of a batch, more batches than are in flight; one, two and four groups of 16
# query rows (the last goes through expanded tiles); rows behind a context hold NaN scales
@pytest.mark.parametrize("ctx", [1, 16, 33, 127, 129, 512, 513, 1900])
@pytest.mark.parametrize("nq,nkv,rows,window", [(5, 1, 1, 0), (16, 4, 4, 0), (16, 1, 1, 0), (20, 4, 5, 100), (12, 2, 5, 0), (16, 2, 8, 0)])
@pytest.mark.parametrize("splits", [1, 3])
def test_attention_on_int8_cache(ctx, nq, nkv, rows, window, splits):
    torch.manual_seed(ctx)
    d, gqa, dev = 128, nq // nkv, "cuda"
    spec = [(0, p) for p in range(max(0, ctx - rows), ctx)] + [(1, ctx // 2)]
    m, blocks = len(spec), ctx // 16 + 2
    table = (torch.randperm(2 * blocks, device=dev) + 1).int().view(2, blocks).contiguous()
    k8, v8 = (torch.randint(-127, 128, (2 * blocks + 1, nkv, 16, d), dtype=torch.int8, device=dev) for _ in range(2))
    ks, vs = (torch.rand(2 * blocks + 1, nkv, 16, device=dev) * 0.03 for _ in range(2))
    for req, last in ((0, ctx - 1), (1, ctx // 2)):       # nothing is stored behind the last position
        pos = torch.arange(last + 1, blocks * 16, device=dev)
        for t in (ks, vs):
            t[table[req].long()[pos // 16], :, pos % 16] = float("nan")
    q = torch.randn(m, nq * d, device=dev).bfloat16()
    ctrl = _ctrl([r for r, _ in spec])
    ctrl[K.CTRL_ROW_POS: K.CTRL_ROW_POS + m] = torch.tensor([p for _, p in spec], dtype=torch.int32, device=dev)
    part, ml = torch.full((m * nq * splits * d,), float("nan"), device=dev), torch.full((m * nq * splits * 2,), float("nan"), device=dev)
    out = torch.full((m, nq * d), float("nan"), dtype=torch.bfloat16, device=dev)
    K.attn_rows(q, k8, v8, table, ctrl, part, ml, out, None, m, nq, nkv, d, splits, blocks, d ** -0.5, k_scale=ks, v_scale=vs, kv_int8=True,
                window=window)
    torch.cuda.synchronize()
    K.check_status()
    for i, (req, pos) in enumerate(spec):
        at = torch.arange(max(0, pos + 1 - window) if window else 0, pos + 1, device=dev)
        pg = table[req].long()[at // 16]
        kk, vv = (c[pg, :, at % 16].double() * s[pg, :, at % 16].double()[..., None] for c, s in ((k8, ks), (v8, vs)))
        qq = q[i].double().view(nkv, gqa, d)
        s = torch.einsum("hgd,khd->hgk", qq, kk) * d ** -0.5
        p = s.softmax(-1)
        want, size = torch.einsum("hgk,khd->hgd", p, vv), torch.einsum("hgk,khd->hgd", p, vv.abs())
        # probabilities (times V's scale) and the result are rounded to bf16, which has eight significant bits: 2^-8 of the
        # value each, 2^-7 together, and a little for fp32 scores and sums.  Expanded tiles round K and V too: 2^-8 of V,
        # and of every product of a score
        bound = 1.05 * 2.0 ** -7 * size
        if rows * gqa > 32:
            ds = 2.0 ** -8 * torch.einsum("hgd,khd->hgk", qq.abs(), kk.abs()).amax(-1, keepdim=True) * d ** -0.5
            bound = bound + (2.0 ** -8 + 2 * ds) * size
        assert ((out[i].double().view(nkv, gqa, d) - want).abs() <= bound + 1e-9).all()


def _shares(spec, gqa, nkv, most, window):
    """Splits of every row: groups of up to eight consecutive rows of a request, by the pages each reads; of all spans that give the
    longest group 1, 2, .. splits the one whose longest piece, or waves of 296 CTAs times the mean piece, takes least."""
    rmax, groups, i = min(8, 64 // gqa), [], 0
    while i < len(spec):
        j = i
        while j < len(spec) and spec[j][0] == spec[i][0] and j - i < rmax:
            j += 1
        last, first = max(p for _, p in spec[i:j]), spec[i][1]
        groups.append((j - i, max(1, last // 16 + 1 - (max(0, first + 1 - window) // 16 if window else 0))))
        i = j
    pages, best = [p for _, p in groups], None
    for k in range(1, min(most, max(pages)) + 1):
        span = -(-max(pages) // k)
        n = [min(most, -(-p // span)) for p in pages]
        if sum(n) <= K.attn_plan_entries(len(spec), nkv):
            t = max(8 + max(-(-p // c) for p, c in zip(pages, n)), -(-sum(n) * nkv // 296) * (8 - (-sum(pages) // sum(n))))
            if best is None or t < best[0]:
                best = (t, n)
    return [c for (r, _), c in zip(groups, best[1]) for _ in range(r)]


# one long context among short ones, the most splits a row may have, several rows of some requests, groups at the 32nd row and behind,
# lone pages, one split of everything, more heads than slots of a wave, a window
@pytest.mark.parametrize("spec,nq,nkv,most,window", [
    ([(i, 40 + 3 * i) for i in range(7)] + [(7, 2900)], 5, 1, 37, 0), ([(0, 2900)] + [(i, 15) for i in range(1, 33)], 4, 2, 16, 0),
    ([(3, p) for p in range(500, 560)] + [(i, 1800 + i) for i in (0, 1, 2, 4)], 10, 2, 64, 0), ([(i, 200 - 3 * i) for i in range(64)], 8, 4, 8, 0),
    ([(i // 3, 100 * (i // 3) + i % 3) for i in range(60)], 16, 1, 12, 0), ([(0, 0), (1, 16)], 2, 2, 37, 0), ([(i, 50 * i) for i in range(9)], 2, 1, 1, 0),
    ([(i, 700) for i in range(33)] + [(i, 5) for i in range(33, 64)], 16, 16, 18, 0), ([(0, 2000), (1, 90), (2, 700), (2, 701), (2, 702)], 6, 2, 9, 100)])
@pytest.mark.parametrize("kv", ["bf16", "int8"])
def test_attention_splits_by_length(spec, nq, nkv, most, window, kv):
    torch.manual_seed(len(spec) + most)
    d, gqa, dev, m = 128, nq // nkv, "cuda", len(spec)
    seqs, blocks = 1 + max(r for r, _ in spec), max(p for _, p in spec) // 16 + 2
    pages = seqs * blocks
    table = (torch.randperm(pages, device=dev) + 1).int().view(seqs, blocks).contiguous()
    if kv == "int8":
        k, v = (torch.randint(-127, 128, (pages + 1, nkv, 16, d), dtype=torch.int8, device=dev) for _ in range(2))
        ks, vs = (torch.rand(pages + 1, nkv, 16, device=dev) * 0.03 for _ in range(2))
    else:
        k, v = (torch.randn(pages + 1, nkv, 16, d, device=dev).bfloat16() for _ in range(2))
        ks = vs = None
    q = torch.randn(m, nq * d, device=dev).bfloat16()
    ctrl = _ctrl([r for r, _ in spec])
    ctrl[K.CTRL_ROW_POS: K.CTRL_ROW_POS + m] = torch.tensor([p for _, p in spec], dtype=torch.int32, device=dev)
    plan = torch.full((K.attn_plan_words(m, nkv),), 1 << 20, dtype=torch.int32, device=dev)
    K.attn_plan(ctrl, m, nq, nkv, most, plan, window=window)
    want = _shares(spec, gqa, nkv, most, window)
    assert plan[:m].tolist() == want
    entries = [(e & 255, e >> 8 & 255, e >> 16) for e in plan[64:].tolist() if e >= 0]
    lead = [i for i in range(m) if i == 0 or spec[i][0] != spec[i - 1][0] or (i - next(j for j in range(m) if spec[j][0] == spec[i][0])) % min(8, 64 // gqa) == 0]
    assert sorted(entries) == [(i, c, want[i]) for i in lead for c in range(want[i])]
    kw = dict(k_scale=ks, v_scale=vs, kv_int8=kv == "int8", window=window)
    pad, kq = K.rows_pad(m), nq * d
    rows, quant = torch.zeros(pad * kq * 2, dtype=torch.uint8, device=dev), torch.zeros(m * kq * 2, dtype=torch.uint8, device=dev)
    gs = torch.zeros(K.quant_slots(m) * kq // 64 * 2, dtype=torch.int32, device=dev)
    outs, tickets = [], torch.zeros(m * nkv, dtype=torch.int32, device=dev)
    for extra in ({}, {"xq": rows}, {"xq": quant, "xq_gs": gs}, None):         # None: the last split's CTA merges
        merge, extra = (tickets, {}) if extra is None else (None, extra)
        part, ml = torch.full((m * nq * most * d,), float("nan"), device=dev), torch.full((m * nq * most * 2,), float("nan"), device=dev)
        out = torch.full((m, kq), float("nan"), dtype=torch.bfloat16, device=dev)
        K.attn_rows(q, k, v, table, ctrl, part, ml, out, merge, m, nq, nkv, d, most, blocks, d ** -0.5, plan=plan, **kw, **extra)
        torch.cuda.synchronize()
        K.check_status()
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]) and int(tickets.abs().sum()) == 0
    again, gs2 = torch.zeros_like(rows), torch.zeros_like(gs)         # the rows as their own launches make them
    K.stage_rows(outs[0], m, kq, again)
    live = [t.view(kq // 64, pad, 128)[:, :m] for t in (rows, again)]
    assert torch.equal(*live)
    again = torch.zeros_like(quant)
    K.quant_x(outs[0], m, kq, again, gs2)
    assert torch.equal(quant, again) and torch.equal(gs, gs2)
    if not window and max(want) == 1:      # nothing is cut: the even form with one split
        even = torch.empty_like(outs[0])
        K.attn_rows(q, k, v, table, ctrl, part, ml, even, None, m, nq, nkv, d, 1, blocks, d ** -0.5, **kw)
        assert torch.equal(even, outs[0])
    for i, (req, pos) in enumerate(spec):
        at = torch.arange(max(0, pos + 1 - window) if window else 0, pos + 1, device=dev)
        pg = table[req].long()[at // 16]
        kk, vv = (c[pg, :, at % 16].double() * (1 if s is None else s[pg, :, at % 16].double()[..., None]) for c, s in ((k, ks), (v, vs)))
        qq = q[i].double().view(nkv, gqa, d)
        p = (torch.einsum("hgd,khd->hgk", qq, kk) * d ** -0.5).softmax(-1)
        want, size = torch.einsum("hgk,khd->hgd", p, vv), torch.einsum("hgk,khd->hgd", p, vv.abs())
        # probabilities (times an int8 V's scale) and the result are rounded to bf16: 2^-8 of the value each, and a little for fp32 sums.
        # Groups above 32 query rows round an int8 cache's K and V too: 2^-8 of V, and of every product of a score
        bound = 1.05 * 2.0 ** -7 * size
        if kv == "int8" and min(8, 64 // gqa, sum(r == req for r, _ in spec)) * gqa > 32:
            ds = 2.0 ** -8 * torch.einsum("hgd,khd->hgk", qq.abs(), kk.abs()).amax(-1, keepdim=True) * d ** -0.5
            bound = bound + (2.0 ** -8 + 2 * ds) * size
        for got in (outs[0], outs[3]):
            assert ((got[i].double().view(nkv, gqa, d) - want).abs() <= bound + 1e-9).all()


@pytest.mark.parametrize("m,h,window", [(2, 64, 0), (17, 512, 0), (64, 5120, 300), (5, 9000, 64), (3, 12224, 0), (3, 12224, 64)])
def test_plan_beside_the_embedding(m, h, window):
    """One launch with the rows and the tables of the launches it stands for, up to the widest row that those take."""
    torch.manual_seed(m)
    nq, nkv, most, vocab = 10, 2, 37, 50
    ctrl = _ctrl([i // 2 for i in range(m)])
    ctrl[K.CTRL_ROW_POS: K.CTRL_ROW_POS + m] = torch.randint(0, 30000, (m,), dtype=torch.int32, device="cuda")
    ctrl[K.CTRL_CUR_TOKEN: K.CTRL_CUR_TOKEN + m] = torch.randint(0, vocab, (m,), dtype=torch.int32, device="cuda")
    embed, w, flag = torch.randn(vocab, h, device="cuda").bfloat16(), 1 + 0.1 * torch.randn(h, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    r0, x0, r1, x1 = (torch.full((m, h), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(4))
    p0, w0, p1, w1 = (torch.full((K.attn_plan_words(m, nkv),), 7, dtype=torch.int32, device="cuda") for _ in range(4))
    K.resid_norm(0, m, h, w, 1e-6, r0, x0, embed=embed, ctrl=ctrl, vocab=vocab, flag=flag)
    K.attn_plan(ctrl, m, nq, nkv, most, p0)
    K.attn_plan(ctrl, m, nq, nkv, most, w0, window=max(1, window))
    K.embed_plan(m, h, w, 1e-6, r1, x1, embed, ctrl, vocab, flag, nq, nkv, most, p1, window=window, plan_win=w1 if window else None)
    torch.cuda.synchronize()
    rows = 64 + K.attn_plan_entries(m, nkv)
    assert torch.equal(r0, r1) and torch.equal(x0, x1) and torch.equal(p0[64:rows], p1[64:rows]) and torch.equal(p0[:m], p1[:m])
    assert (torch.equal(w0[64:rows], w1[64:rows]) and torch.equal(w0[:m], w1[:m])) if window else (w1 == 7).all()
