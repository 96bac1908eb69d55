"""Work dealt out in another order than one head after the other: causal calls whose heads form several groups (the last
one smaller), and packed sequences that the forward's CTAs take from a counter.  Every item has to be done exactly once:
against the oracle."""
import numpy as np
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from oracle import sdpa_oracle as orc

from .util import LSE_TOL, assert_close, assert_close_grad, randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Hq,Hkv,N,S,D", [(7, 7, 300, 32768, 128), (7, 7, 32768, 300, 128), (14, 7, 20000, 333, 64), (16, 2, 900, 700, 128)])
def test_several_groups_of_heads(dev, Hq, Hkv, N, S, D):
    """48 MB a group: 3 heads of 32768 x 128 K / V (or Q / dO), 9 of 20000 x 64, all of the small ones."""
    dtype = torch.bfloat16
    q, k, v, do = (randn((1, h, n, D), dtype, 900 + i) for i, (h, n) in enumerate(((Hq, N), (Hkv, S), (Hkv, S), (Hq, N))))
    qg, kg, vg = (x.to(dev).requires_grad_(True) for x in (q, k, v))
    out, lse = fa.flash_attention(qg, kg, vg, causal=True, return_lse=True)
    out.backward(do.to(dev))
    O, L, _ = orc.sdpa(q, k, v, causal=True)
    assert_close(out, O, dtype)
    assert_close(lse, L, dtype, "lse", LSE_TOL[dtype])
    blind = max(0, N - S)                # rows that see no key: no gradient, and the oracle's softmax of them is 0 / 0
    assert not qg.grad[:, :, :blind].any()
    refs = orc.backward(q[:, :, blind:], k, v, do[:, :, blind:], causal=True)
    for name, got, ref in zip(("dQ", "dK", "dV"), (qg.grad[:, :, blind:], kg.grad, vg.grad), refs):
        assert_close_grad(got, ref, dtype, name)


@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (128, torch.float16)])
def test_packed_sequences_from_a_counter(dev, D, dtype):
    # enough items for the persistent form: 8 per CTA of 296; uneven, empty and one-row sequences; rows of no sequence
    rng = np.random.default_rng(9)
    lens = [int(x) for x in rng.integers(1, 500, size=40)] + [0, 1, 900, 0, 128]
    cu = [5] + list(5 + np.cumsum(lens))
    T, H = cu[-1] + 70, 32
    q, k, v = randn((1, H, T, D), dtype, 910), randn((1, H // 4, T, D), dtype, 911), randn((1, H // 4, T, D), dtype, 912)
    cu_t = torch.tensor(cu, dtype=torch.int32, device=dev)
    qd, kd, vd = q.to(dev), k.to(dev), v.to(dev)
    torch.full((1, H, T, D), float("nan"), dtype=dtype, device=dev)      # what the next allocation may find
    out = fa.flash_attention_varlen(qd, kd, vd, cu_t, cu_t, max(lens), max(lens), causal=True)
    for i, n in enumerate(lens):
        if n and i in (0, 7, 39, 41, 42, 44):
            O, _, _ = orc.sdpa(q[:, :, cu[i]:cu[i + 1]], k[:, :, cu[i]:cu[i + 1]], v[:, :, cu[i]:cu[i + 1]], causal=True)
            assert_close(out[:, :, cu[i]:cu[i + 1]], O, dtype)
    assert not out[:, :, :5].any() and not out[:, :, cu[-1]:].any()
    assert torch.isfinite(out).all()
    for _ in range(3):
        assert torch.equal(out, fa.flash_attention_varlen(qd, kd, vd, cu_t, cu_t, max(lens), max(lens), causal=True))
    # a max_seqlen_q below the longest sequence: rows beyond its last query tile are zero, as the tiles before them are not
    short = fa.flash_attention_varlen(qd, kd, vd, cu_t, cu_t, 256, max(lens), causal=True)
    i = lens.index(900)
    assert not short[:, :, cu[i] + 256:cu[i + 1]].any()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    other = fa.flash_attention_varlen(qd, kd, vd, cu_t, cu_t, max(lens), max(lens), causal=True, stream=side)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(out, other)
    assert fa.kernel_status() == 0
