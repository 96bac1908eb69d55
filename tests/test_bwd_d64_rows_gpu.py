"""head_dim-64 backward: the tcgen05 kernel subtracts a query row's L and delta inside its MMAs, as three 16-bit parts
each.  Rows whose L is large, small or missing, scales of every kind (those it does not take run the portable kernel) and
rows that are not finite must give the gradients the oracle has."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from mlx_flashattention_steel_b200 import _lib
from mlx_flashattention_steel_b200 import attention as A
from oracle import sdpa_oracle as orc

from .util import assert_close_grad, randn

pytestmark = pytest.mark.gpu


def _grads(dev, q, k, v, do, flags=0, **kw):
    old = A._set_force_flags(flags)
    try:
        t = [x.to(dev).requires_grad_(True) for x in (q, k, v)]
        out = fa.flash_attention(*t, **kw)
        return [g.double().cpu() for g in torch.autograd.grad(out, t, do.to(dev))]
    finally:
        A._set_force_flags(old)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("size,scale", [(1.0, 0.125), (6.0, 0.125), (1.0, -0.125), (0.02, 2.0), (30.0, 1e-3), (1.0, 1e-5),
                                        (1.0, 0.0), (1.0, 1e-9)])
def test_scores_of_every_size(dev, dtype, size, scale):
    """Against the oracle, and no worse than the portable kernel, which subtracts L and delta in float32: its own error (16-bit
    P and dS, 2^-9 or 2^-12 of each) times 1.5, plus the 2^-20 that the parts and the MMAs' sums may add."""
    q, k, v, do = (randn((1, 4, n, 64), dtype, 90 + i) for i, n in enumerate((200, 333, 333, 200)))
    q, k = (q.float() * size).to(dtype), (k.float() * size).to(dtype)
    refs = [r.double() for r in orc.backward(q, k, v, do, causal=True, scale=scale)]
    got = _grads(dev, q, k, v, do, causal=True, scale=scale)
    base = _grads(dev, q, k, v, do, flags=_lib.FLAG_FORCE_MMA_SYNC, causal=True, scale=scale)
    for name, g, b, r in zip(("dQ", "dK", "dV"), got, base, refs):
        n = float(r.norm())
        e, eb = float((g - r).norm()), float((b - r).norm())
        assert e <= 1.5 * eb + 2.0 ** -20 * n, (name, e / max(n, 1e-30), eb / max(n, 1e-30))


@pytest.mark.parametrize("softcap", [0.0, 30.0])
@pytest.mark.parametrize("N,S,causal", [(1, 65, False), (63, 64, True), (65, 127, True), (129, 128, False), (300, 130, True)])
def test_ragged_rows_and_rows_without_keys(dev, N, S, causal, softcap):
    dtype = torch.bfloat16
    q, k, v, do = randn((2, 4, N, 64), dtype, 80), randn((2, 2, S, 64), dtype, 81), randn((2, 2, S, 64), dtype, 82), randn((2, 4, N, 64), dtype, 83)
    got = _grads(dev, q, k, v, do, causal=causal, softcap=softcap)
    first = max(0, N - S) if causal else 0          # the rows before it see no key (the oracle has no gradient for them)
    assert not got[0][:, :, :first].any()
    got[0] = got[0][:, :, first:]
    refs = orc.backward(q[:, :, first:].contiguous(), k, v, do[:, :, first:].contiguous(), causal=causal, softcap=softcap)
    for name, g, r in zip(("dQ", "dK", "dV"), got, refs):
        assert_close_grad(g, r, dtype, name)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_row_that_is_not_finite_stays_a_row(dev, dtype, bad):
    q, k, v, do = (randn((1, 2, 256, 64), dtype, 60 + i) for i in range(4))
    do[0, 1, 150, 7] = bad
    dq, dk, dv = _grads(dev, q, k, v, do, causal=False)
    rows = torch.ones(256, dtype=torch.bool)
    rows[150] = False
    assert torch.isfinite(dq[0, 0]).all() and torch.isfinite(dk[0, 0]).all() and torch.isfinite(dv[0, 0]).all()
    assert torch.isfinite(dq[0, 1, rows]).all() and not torch.isfinite(dq[0, 1, 150]).any()
    assert not torch.isfinite(dk[0, 1]).all()


_FORMS = [dict(), dict(causal=True), dict(causal=True, window_size=(70, 0)), dict(alibi_slopes="4 heads"), dict(softcap=20.0)]


@pytest.mark.parametrize("form", range(len(_FORMS)))
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_channel_of_do_that_is_not_finite_stays_a_channel_of_dv(dev, dtype, form):
    """dV = P^T dO: of a dO row with one infinite channel, that channel of dV has it, and no other."""
    kw = dict(_FORMS[form])
    if "alibi_slopes" in kw:
        kw["alibi_slopes"] = torch.tensor([0.1, 0.2, 0.3, 0.4], device=dev)
    q, k, v, do = randn((1, 4, 200, 64), dtype, 50), randn((1, 2, 200, 64), dtype, 51), randn((1, 2, 200, 64), dtype, 52), randn((1, 4, 200, 64), dtype, 53)
    bad = do.clone()
    bad[0, 1, 150, 7] = float("inf")
    got, base = _grads(dev, q, k, v, bad, **kw), _grads(dev, q, k, v, do, **kw)
    other = [d for d in range(64) if d != 7]
    assert not torch.isfinite(got[2][0, 0, 100:150, 7]).any()
    assert torch.equal(got[2][..., other], base[2][..., other]) and torch.equal(got[2][0, 1], base[2][0, 1])
    assert not torch.isfinite(got[0][0, 1, 150]).any()


@pytest.mark.parametrize("softcap", [0.0, 20.0])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_delta_that_is_not_finite_by_itself(dev, bad, softcap):
    """delta = sum(dO o O) not finite where dO is: dV does not depend on it, that row's dS and what is made of it do."""
    dtype = torch.bfloat16
    q, k, v, do = (randn((1, 2, 150, 64), dtype, 70 + i).to(dev) for i in range(4))
    out, lse = fa.flash_attention(q, k, v, softcap=softcap, return_lse=True)
    base = A._bwd_raw(q, k, v, out, lse, do, 0.125, False, None, softcap=softcap)
    out[0, 1, 77, 3] = bad
    dq, dk, dv = A._bwd_raw(q, k, v, out, lse, do, 0.125, False, None, softcap=softcap)
    assert torch.equal(dv, base[2]) and torch.equal(dk[0, 0], base[1][0, 0])
    assert not torch.isfinite(dk[0, 1]).any() and not torch.isfinite(dq[0, 1, 77]).any()
    rows = torch.ones(150, dtype=torch.bool)
    rows[77] = False
    # dQ is summed over the key tiles in any order
    assert torch.allclose(dq[0, 1, rows].float(), base[0][0, 1, rows].float(), rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.parametrize("dtype,size,scale", [(torch.float16, 2e4, 1e-6), (torch.float16, 2e4, -1e-6), (torch.float16, 5e3, 2e-5),
                                              (torch.bfloat16, 2e4, 1e-6)])
def test_large_rows_under_a_small_scale(dev, dtype, size, scale):
    """Dot products of 2^28 and beyond 2^31 whose scores are ordinary (up to 2^14 in the log2 domain).  The tensor cores sum them to
    2^-21 of sum |q_d k_d| (four steps of 2^-23), forward and backward apart, and L is rounded: a relative error of each P that the
    gradients inherit.  That bound is added to 1.5 times the portable kernel's error, as in test_scores_of_every_size."""
    q, k, v, do = (randn((1, 4, n, 64), torch.float32, 90 + i).clamp(-3, 3) for i, n in enumerate((200, 333, 333, 200)))
    q, k, v, do = (q * size).to(dtype), (k * size).to(dtype), v.to(dtype), do.to(dtype)
    refs = [r.double() for r in orc.backward(q, k, v, do, causal=True, scale=scale)]
    got = _grads(dev, q, k, v, do, causal=True, scale=scale)
    base = _grads(dev, q, k, v, do, flags=_lib.FLAG_FORCE_MMA_SYNC, causal=True, scale=scale)
    Q, K, V, G = (x.double() for x in (q, k, v, do))
    S = (scale * Q @ K.mT).masked_fill(torch.ones(200, 333).triu(134).bool(), -torch.inf)
    P, dP = S.softmax(-1), G @ V.mT
    eP = P * (2 * abs(scale) * 2.0 ** -21 * (Q.abs() @ K.abs().mT) + 2.0 ** -23 * S.logsumexp(-1, keepdim=True).abs())
    eS = eP * (dP - (P * dP).sum(-1, keepdim=True)).abs() + P * (eP * dP.abs()).sum(-1, keepdim=True)
    bounds = abs(scale) * (eS @ K.abs()), abs(scale) * (eS.mT @ Q.abs()), eP.mT @ G.abs()
    for name, g, b, r, bound in zip(("dQ", "dK", "dV"), got, base, refs, bounds):
        assert torch.isfinite(g).all(), name
        e, eb = float((g - r).norm()), float((b - r).norm())
        assert e <= 1.5 * eb + float(bound.norm()), (name, e, eb, float(bound.norm()), float(r.norm()))


def test_float16_scores_up_to_the_largest_that_are_taken(dev):
    """One key per query, q.k = 38016^2 = 1.4e9 (of 2^31; exact), the smallest scale the tcgen05 kernel takes: L is 1.1e7, rounded by up
    to 1/2, and L / scale by 2^-23 of 1.4e9, a score of 1.4: P between 2^-2 and 2^2."""
    eye = torch.eye(64, dtype=torch.float16)[None, None] * 38016
    v, do = randn((1, 1, 64, 64), torch.float16, 20), torch.full((1, 1, 64, 64), 4.0, dtype=torch.float16)
    dv = _grads(dev, eye, eye, v, do, scale=0.0055)[2]
    assert (dv.log2() - 2).abs().max() <= 2.0


def test_float16_parts_keep_float_precision(dev):
    """The same with q.k = 17456^2 = 3.05e8, whose second part is beyond 65504: L is 2.4e6, rounded by up to 1/8, and L / scale by
    2^-23 of 3.05e8, a score of 0.29."""
    eye = torch.eye(64, dtype=torch.float16)[None, None] * 17456
    v, do = randn((1, 1, 64, 64), torch.float16, 20), torch.full((1, 1, 64, 64), 4.0, dtype=torch.float16)
    dv = _grads(dev, eye, eye, v, do, scale=0.0055)[2]
    assert (dv.log2() - 2).abs().max() <= 0.5


@pytest.mark.parametrize("dtype,size", [(torch.bfloat16, 1e34), (torch.float16, 2e3)])
@pytest.mark.parametrize("causal", [False, True])
def test_rows_behind_a_sequence_do_not_matter(dev, dtype, size, causal):
    """Query tiles reach beyond a sequence's end into the next one (or into what pads the packed rows): however large those rows
    are, the gradients of the sequence in front are those it has alone."""
    q, k, v, do = (randn((1, 2, 130, 64), dtype, 30 + i).to(dev) for i in range(4))
    q[:, :, 70:] = (q[:, :, 70:].float() * size).to(dtype)
    cu = torch.tensor([0, 70], dtype=torch.int32, device=dev)
    t = [x.clone().requires_grad_(True) for x in (q, k, v)]
    out = fa.flash_attention_varlen(*t, cu, cu, 70, 70, causal=causal)
    got = torch.autograd.grad(out, t, do)
    t = [x[:, :, :70].contiguous().requires_grad_(True) for x in (q, k, v)]
    want = torch.autograd.grad(fa.flash_attention(*t, causal=causal), t, do[:, :, :70].contiguous())
    for name, g, w in zip(("dQ", "dK", "dV"), got, want):
        assert torch.allclose(g[:, :, :70].double(), w.double(), rtol=2.0 ** -7, atol=2.0 ** -10), name
