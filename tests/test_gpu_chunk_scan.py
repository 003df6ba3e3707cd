"""-m gpu: the matrix-state recurrence in chunks of 8 positions (yalm_state_scan_rows from 8 rows on) against the recurrence one position at
a time in 64 bits: last chunks of 1 .. 8 positions, portions that carry the state, fewer columns than a CTA has, heads that share keys,
decays of 0 and 1, both scalings, a skip.

Bound: fp32 sums over D <= 128 rows and a state that forgets: 2e-6 of the norm (measured 1.4e-7)."""
import ctypes as C

import pytest
import torch

from yalm_b200 import api

pytestmark = pytest.mark.gpu


def step_by_step(k, q, v, decay, beta, vscale, skip, S, rep):
    out = []
    for i in range(len(k)):
        ki, qi = k[i].repeat_interleave(rep, 0), q[i].repeat_interleave(rep, 0)
        S = S * (decay[i][:, None, :] if decay.dim() == 3 else decay[i][:, None, None])
        e = v[i]
        if beta is not None:
            e = beta[i][:, None] * (e - torch.einsum("hpd,hd->hp", S, ki))
        elif vscale is not None:
            e = vscale[i][:, None] * e
        S = S + e[:, :, None] * ki[:, None, :]
        y = torch.einsum("hpd,hd->hp", S, qi)
        out.append(y + skip[:, None] * v[i] if skip is not None else y)
    return torch.stack(out), S


@pytest.mark.parametrize("D,P", [(128, 128), (64, 64), (128, 4), (64, 20), (64, 36)])
@pytest.mark.parametrize("form", ["delta_channel", "delta_head", "linear_channel", "scaled_head"])
@pytest.mark.parametrize("portions", [(8,), (9, 24), (31, 5, 33), (100, 64)])
def test_chunks_match_steps(D, P, form, portions):
    L, H, rep, n = api.lib(), 4, 2, sum(portions)
    g = torch.Generator(device="cuda")
    g.manual_seed(n + D + P)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    k, q = rnd(n, H // rep, D), rnd(n, H // rep, D) * D ** -0.5
    k = k / k.norm(dim=-1, keepdim=True)
    v = rnd(n, H, P)
    decay = torch.exp(-0.3 * torch.rand((n, H) if form.endswith("head") else (n, H, D), generator=g, device="cuda"))
    decay[3], decay[n // 2] = 1.0, 0.0
    beta = torch.sigmoid(rnd(n, H)) if form.startswith("delta") else None
    vscale = torch.rand((n, H), generator=g, device="cuda") if form == "scaled_head" else None
    skip = rnd(H) if form != "delta_channel" else None
    start = rnd(H, P, D)
    p = lambda t: C.c_void_p(None if t is None else t.data_ptr())
    state, out = start.clone(), torch.full((n, H * P + 4), 7.0, device="cuda")
    at = 0
    for m in portions:
        assert L.yalm_state_scan_rows(p(out[at:]), C.c_int(H * P + 4), p(k[at:]), C.c_int(k[0].numel()), p(q[at:]), C.c_int(k[0].numel()), p(v[at:]), C.c_int(H * P),
                                      p(decay[at:]), C.c_int(decay[0].numel()), C.c_int(int(decay.dim() == 3)), p(vscale[at:] if vscale is not None else None), C.c_int(H),
                                      p(beta[at:] if beta is not None else None), C.c_int(H), p(skip), p(state), C.c_int(m), C.c_int(H), C.c_int(rep), C.c_int(D),
                                      C.c_int(P), C.c_int(7 + at), None, None) == 0
        at += m
    dbl = lambda t: None if t is None else t.double()
    want, S = step_by_step(dbl(k), dbl(q), dbl(v), dbl(decay), dbl(beta), dbl(vscale), dbl(skip), start.double(), rep)
    assert ((out[:, :H * P].reshape(n, H, P).double() - want).norm() / want.norm()).item() < 2e-6
    assert ((state.double() - S).norm() / S.norm()).item() < 2e-6
    assert (out[:, H * P:] == 7.0).all()


@pytest.mark.parametrize("H,D,P", [(40, 128, 64), (40, 64, 36), (148, 64, 8), (149, 64, 8), (37, 128, 4)])
@pytest.mark.parametrize("form", ["delta_channel", "delta_head", "linear_channel"])
def test_columns_four_and_two_a_warp(H, D, P, form):
    """Around the rule between the two: more and fewer column groups than SMs, the last group not full."""
    n = 21
    g = torch.Generator(device="cuda")
    g.manual_seed(H + D + P)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    k, q, v = rnd(n, H, D), rnd(n, H, D) * D ** -0.5, rnd(n, H, P)
    k = k / k.norm(dim=-1, keepdim=True)
    decay = torch.exp(-0.3 * torch.rand((n, H) if form == "delta_head" else (n, H, D), generator=g, device="cuda"))
    beta = torch.sigmoid(rnd(n, H)) if form.startswith("delta") else None
    start = rnd(H, P, D)
    state, out = start.clone(), torch.empty((n, H, P), device="cuda")
    p = lambda t: C.c_void_p(None if t is None else t.data_ptr())
    i = C.c_int
    assert api.lib().yalm_state_scan_rows(p(out), i(H * P), p(k), i(H * D), p(q), i(H * D), p(v), i(H * P), p(decay), i(decay[0].numel()), i(int(decay.dim() == 3)), None, i(0),
                                          p(beta), i(H), None, p(state), i(n), i(H), i(1), i(D), i(P), i(5), None, None) == 0
    want, S = step_by_step(k.double(), q.double(), v.double(), decay.double(), None if beta is None else beta.double(), None, None, start.double(), 1)
    assert ((out.double() - want).norm() / want.norm()).item() < 2e-6
    assert ((state.double() - S).norm() / S.norm()).item() < 2e-6
