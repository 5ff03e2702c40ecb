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
