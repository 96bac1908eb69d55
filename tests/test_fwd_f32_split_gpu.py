"""The float32 forward with its key tiles shared evenly between CTAs (workspace given) and with one CTA per query tile
(none): shares that begin and end inside a query tile, tiles with no visible key, every mask.  float64 oracle, 1e-5."""
import ctypes as C

import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from mlx_flashattention_steel_b200 import _lib
from mlx_flashattention_steel_b200 import attention as A
from oracle import sdpa_oracle as orc

from .util import assert_close, randn

pytestmark = pytest.mark.gpu

SHAPES = [  # B, Hq, Hkv, N, S, D
    (1, 1, 1, 65, 65, 64), (1, 2, 1, 128, 640, 128), (1, 8, 8, 1024, 1024, 128), (2, 4, 2, 200, 777, 64),
    (1, 3, 3, 1000, 333, 128), (3, 5, 1, 129, 1, 64), (2, 32, 8, 513, 600, 64), (1, 1, 1, 2048, 2048, 128),
]


@pytest.mark.parametrize("B,Hq,Hkv,N,S,D", SHAPES)
@pytest.mark.parametrize("causal,window,softcap", [(False, None, 0.0), (True, None, 0.0), (True, 100, 0.0), (False, 70, 0.0), (True, None, 20.0)])
def test_even_shares(dev, B, Hq, Hkv, N, S, D, causal, window, softcap):
    q, k, v = randn((B, Hq, N, D), torch.float32, 800), randn((B, Hkv, S, D), torch.float32, 801), randn((B, Hkv, S, D), torch.float32, 802)
    qd, kd, vd = q.to(dev), k.to(dev), v.to(dev)
    out, lse = fa.flash_attention(qd, kd, vd, causal=causal, softcap=softcap, return_lse=True,
                                  window_size=None if window is None else (window, 0))
    O, L, _ = orc.sdpa(q, k, v, causal=causal, softcap=softcap, window_left=-1 if window is None else window)
    assert_close(out, O, torch.float32)
    assert_close(lse, L, torch.float32, "lse", 2e-5)
    # without a workspace: one CTA per query tile
    o2, l2 = torch.empty_like(out), torch.empty_like(lse)
    d = A._desc(_lib.F32, _lib.F32, B, Hq, Hkv, N, S, D, D ** -0.5, causal, softcap, -1 if window is None else window, q=qd, k=kd, v=vd, o=o2)
    st = _lib.load().b200fa_fwd(C.byref(d), *(C.c_void_p(x.data_ptr()) for x in (qd, kd, vd, o2, l2)), None, 0,
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == _lib.OK, _lib.last_error()
    assert_close(o2, O, torch.float32)
    assert_close(l2, L, torch.float32, "lse", 2e-5)


def test_even_shares_with_alibi(dev):
    q, k, v = randn((2, 4, 300, 64), torch.float32, 810), randn((2, 4, 500, 64), torch.float32, 811), randn((2, 4, 500, 64), torch.float32, 812)
    slopes = torch.tensor([0.5, 0.25, 0.125, 0.0625])
    out = fa.flash_attention(q.to(dev), k.to(dev), v.to(dev), causal=True, alibi_slopes=slopes.to(dev))
    O, _, _ = orc.sdpa(q, k, v, causal=True, alibi_slopes=slopes)
    assert_close(out, O, torch.float32)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_query_tiles_without_a_key_read_no_values(dev, value):
    """Causal, more queries than keys: the query tiles that see no key are zeros whatever V holds."""
    q, k, v = randn((1, 2, 300, 64), torch.float32, 820), randn((1, 2, 100, 64), torch.float32, 821), randn((1, 2, 100, 64), torch.float32, 822)
    k[0, 0, 0], v[0, 0, 0] = value, value
    out, lse = fa.flash_attention(q.to(dev), k.to(dev), v.to(dev), causal=True, return_lse=True)
    assert not out[:, :, :192].any() and torch.isneginf(lse[:, :, :192]).all()           # rows up to 199 are blind: three tiles of 64
    O, _, _ = orc.sdpa(q[:, 1:, 200:], k[:, 1:], v[:, 1:], causal=True)
    assert_close(out[:, 1:, 200:], O, torch.float32)
    cu_q, cu_k = (torch.tensor([0, n], dtype=torch.int32, device=dev) for n in (300, 100))
    out = fa.flash_attention_varlen(q.to(dev), k.to(dev), v.to(dev), cu_q, cu_k, 300, 100, causal=True)
    assert not out[:, :, :192].any()
