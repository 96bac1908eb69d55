"""The native forms of the plain calls (csrc/host_calls.cpp) take a call only where they do what the Python code does with
it, and give it back (None) everywhere else."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from mlx_flashattention_steel_b200 import _lib, attention as A, kv_cache as K, rope as R

H = _lib.host_calls


def test_what_is_not_a_plain_cuda_call_is_given_back():
    assert H is not _lib._NotBuilt
    q = torch.zeros(1, 2, 64, 64, dtype=torch.float16)
    assert H.fwd(q, q, q, None, False, 0.0, -1, False, 0, True) is None           # not on a GPU
    assert H.fwd(q, q, q, None, False, 0.0, -1, False, 0) is None                 # not the right arguments
    assert H.fwd() is None and H.bwd(1, 2) is None and H.decode(*[None] * 16) is None
    assert H.fwd(None, "q", q, None, False, 0.0, -1, False, 0, True) is None
    assert H.rope(q, q, q, 0, True, None) is None and H.rope(q, q, q, [0], True, 1 << 80) is None
    assert H.append(q, q, q, q, q, None, None) is None
    meta = torch.empty(1, 2, 64, 64, dtype=torch.float16, device="meta")
    assert H.fwd(meta, meta, meta, None, False, 0.0, -1, False, 0, True) is None
    # and what the Python code says about such a call stays as it is
    with pytest.raises(RuntimeError, match="no CPU path"):
        fa.flash_attention(q, q, q)
    with pytest.raises(ValueError, match="4-D"):
        fa.flash_attention(q[0], q[0], q[0])


def _python_only(fn):
    """The call with the native forms out of the way."""
    old = A._H
    A._H = R._H = K._H = _lib._NotBuilt
    try:
        return fn()
    finally:
        A._H = R._H = K._H = old


def _same(fn):
    a, b = fn(), _python_only(fn)
    a, b = (x if isinstance(x, (tuple, list)) else (x,) for x in (a, b))
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert type(x) is type(y) and x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride()
        assert x.requires_grad == y.requires_grad and x.device == y.device
        assert torch.equal(x.nan_to_num(), y.nan_to_num())


class _Counted:
    """The extension, counting the calls it took."""

    def __init__(self):
        self.taken = 0

    def __getattr__(self, name):
        f = getattr(H, name)

        def call(*a):
            r = f(*a)
            self.taken += r is not None
            return r
        return call


@pytest.fixture
def counted():
    old, c = A._H, _Counted()
    A._H = R._H = K._H = c
    yield c
    A._H = R._H = K._H = old


def _r(*s, dt=torch.float16, dev="cuda"):
    return torch.randn(s, device=dev).to(dt)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [64, 128])
def test_dense_forms(dev, dt, D):
    q, k, v = _r(2, 4, 70, D, dt=dt), _r(2, 2, 133, D, dt=dt), _r(2, 2, 133, D, dt=dt)
    bshd = _r(2, 133, 2, D, dt=dt).transpose(1, 2)                    # other strides
    odd = _r(2, 2, 133, D + 1, dt=dt)[..., :D]                        # rows that have to be copied
    for kk, vv in ((k, v), (bshd, bshd), (odd, v), (k[:, :1].expand(2, 2, 133, D), v[:, :1].expand(2, 2, 133, D)), (k[:, :, ::2], v[:, :, ::2])):
        for kw in (dict(), dict(causal=True, return_lse=True), dict(scale=0.3, window_size=(20, 0), causal=True), dict(softcap=20),
                   dict(window_size=[10, -1]), dict(causal=1), dict(scale=2)):
            _same(lambda: fa.flash_attention(q, kk, vv, **kw))
    _same(lambda: fa.flash_attention(q[:, :, :1], k.repeat(1, 1, 4, 1), v.repeat(1, 1, 4, 1), causal=True))      # split-KV route
    _same(lambda: fa.flash_attention(q[:1].expand(2, 4, 70, D), k, v))
    with torch.inference_mode():
        _same(lambda: fa.flash_attention(q, k, v))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        _same(lambda: fa.flash_attention(q, k, v))
    torch.cuda.current_stream().wait_stream(s)


@pytest.mark.gpu
@pytest.mark.parametrize("kv", ["same", "int8", "e4m3"])
@pytest.mark.parametrize("rows", [(8, 2, 1), (8, 2, 4), (16, 2, 4), (4, 4, 1)])
def test_paged_rope_and_append_forms(dev, kv, rows):
    Hq, Hkv, Nq = rows
    B, bs, D, P = 3, 16, 128, 40
    pool = {"same": torch.float16, "int8": torch.int8, "e4m3": torch.float8_e4m3fn}[kv]
    kp, vp = (_r(P, bs, Hkv, D).mul(20).to(pool) for _ in range(2))
    ks, vs = (None, None) if kv == "same" else (torch.rand(P, bs, Hkv, device=dev).half() * 0.05 for _ in range(2))
    table = torch.randperm(P, device=dev)[:B * 12].view(B, 12).int()
    lens = torch.tensor([1, 100, 190], dtype=torch.int32, device=dev)
    q = _r(B, Hq, Nq, D)
    for tt, ll in ((table, lens), (table.long(), lens.long()), (table.t().contiguous().t(), lens)):
        for kw in (dict(max_kv_len=190), dict(), dict(max_kv_len=190, causal=True, return_lse=True, softcap=30.0), dict(max_kv_len=190, scale=0.2, num_splits=2)):
            _same(lambda: fa.flash_attention_paged(q, kp, vp, tt, ll, k_scale=ks, v_scale=vs, **kw))
    _same(lambda: fa.flash_attention_paged(q.transpose(1, 2).contiguous().transpose(1, 2), kp, vp, table, lens, k_scale=ks, v_scale=vs, max_kv_len=190))
    slots = torch.tensor([5, -1, 77], dtype=torch.int64, device=dev)
    kn, vn = _r(B, Hkv, 1, D), _r(B, Hkv, 1, D)

    def append():
        pools = [x.clone() for x in (kp, vp)] + [None if s is None else s.clone() for s in (ks, vs)]
        fa.kv_append(kn[:, :, 0], vn[:, :, 0], slots, *pools)
        return [x.view(torch.uint8) for x in pools if x is not None]
    _same(append)
    cos, sin = torch.rand(300, D // 2, device=dev), torch.rand(300, D // 2, device=dev)
    for off in (0, 7, [1, 2, 290], (1, 2, 3), torch.tensor([4, 5, 6]), torch.tensor([4, 5, 6], device=dev)):
        for x in (q, q.transpose(1, 2).contiguous().transpose(1, 2), q[..., :64]):
            _same(lambda: fa.apply_rope(x, cos[:, :x.shape[-1] // 2], sin[:, :x.shape[-1] // 2], off, interleaved=False))
            _same(lambda: fa.apply_rope(x, cos[:, :16].contiguous(), sin[:, :16].contiguous(), off, rotary_dim=32))
    with pytest.raises(ValueError):
        fa.apply_rope(q, cos, sin, [0, 0, 300])


@pytest.mark.gpu
def test_gradients_and_modes(dev, counted):
    q, k, v = _r(1, 4, 100, 64), _r(1, 2, 100, 64), _r(1, 2, 100, 64)
    do = _r(1, 4, 100, 64)

    def step(g=do, **kw):
        t = [x.detach().clone().requires_grad_(True) for x in (q, k, v)]
        out = fa.flash_attention(*t, causal=True, **kw)
        return [out.detach(), *torch.autograd.grad(out, t, g)]
    _same(step)
    _same(lambda: step(g=do.transpose(1, 2).contiguous().transpose(1, 2)))
    _same(lambda: step(g=do[:, :, :1].expand(1, 4, 100, 64)))
    n = counted.taken
    assert n > 0
    out = fa.flash_attention(q.clone().requires_grad_(True), k, v)
    assert out.requires_grad and out.grad_fn is not None
    with torch.no_grad():
        assert not fa.flash_attention(q.clone().requires_grad_(True), k, v).requires_grad
    # saved-tensor hooks see what the autograd function saves
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t, lambda t: t):
        fa.flash_attention(q.clone().requires_grad_(True), k, v)
    assert len(seen) >= 4
    # subclasses, functorch, forward-mode gradients and modes are not for the native forms
    n = counted.taken

    class Sub(torch.Tensor):
        pass
    fa.flash_attention(q.as_subclass(Sub), k, v)
    assert counted.taken <= n + 1                  # (inside the autograd function the tensors are plain again)
    calls = [lambda: torch.func.vmap(lambda a: fa.flash_attention(a, k, v))(q[None])]

    def dual():
        with torch.autograd.forward_ad.dual_level():
            return fa.flash_attention(torch.autograd.forward_ad.make_dual(q, q), k, v)
    calls.append(dual)
    for f in calls:
        a = b = None
        try:
            f()
        except Exception as e:
            a = type(e)
        try:
            _python_only(f)
        except Exception as e:
            b = type(e)
        assert a is b

    class Mode(torch.overrides.TorchFunctionMode):
        names = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            Mode.names.append(getattr(func, "__name__", str(func)))
            return func(*args, **(kwargs or {}))
    with Mode():
        fa.flash_attention(q, k, v)
    assert "empty" in Mode.names


@pytest.mark.gpu
def test_capture(dev):
    q, k, v = _r(1, 4, 100, 64), _r(1, 2, 100, 64), _r(1, 2, 100, 64)
    want = fa.flash_attention(q, k, v)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = fa.flash_attention(q, k, v)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.gpu
def test_which_calls_are_taken(dev):
    """The comparisons above hold as well where the extension takes nothing: here each plain call has to be taken, once and by the
    form in front of the Python code, and each other one given back."""
    taken = []

    class Named:
        def __getattr__(self, name):
            def call(*a):
                r = getattr(H, name)(*a)
                if r is not None:
                    taken.append(name if name != "fwd" or a[9] else "fwd, behind the checks")
                return r
            return call

    def check(want, fn):
        taken.clear()
        old = A._H
        A._H = R._H = K._H = Named()
        try:
            fn()
        finally:
            A._H = R._H = K._H = old
        assert taken == want, (taken, want)

    for dt in (torch.float16, torch.bfloat16, torch.float32):
        for D in (64, 128):
            q, k = _r(2, 4, 70, D, dt=dt), _r(2, 2, 133, D, dt=dt)
            for kw in (dict(), dict(causal=True, return_lse=True), dict(scale=2, window_size=(20, 0), causal=True), dict(softcap=20)):
                check(["fwd"], lambda: fa.flash_attention(q, k, k, **kw))
            bshd = _r(2, 133, 2, D, dt=dt).transpose(1, 2)
            check(["fwd"], lambda: fa.flash_attention(q, bshd, bshd))
            check(["fwd"], lambda: fa.flash_attention(q[:1].expand(2, 4, 70, D), k, k))
            check(["fwd, behind the checks"], lambda: fa.flash_attention(q, k, k, causal=1))
            check(["fwd, behind the checks"], lambda: fa.flash_attention(q, k, k, window_size=[10, -1]))
            odd, one = _r(2, 2, 133, D + 1, dt=dt)[..., :D], k[:, :1].expand(2, 2, 133, D)
            for x in (odd, one):
                check([], lambda: fa.flash_attention(q, x, x))
            check([], lambda: fa.flash_attention(q, k, k, stream=torch.cuda.current_stream()))

            def train(g):
                t = [x.clone().requires_grad_(True) for x in (q, k, k)]
                torch.autograd.grad(fa.flash_attention(*t), t, g)
            if dt != torch.float32:
                check(["fwd, behind the checks", "bwd"], lambda: train(q))
                check(["fwd, behind the checks"], lambda: train(q[:, :, :1].expand(q.shape)))

    B, P = 3, 40
    table, lens = torch.randperm(P, device=dev)[:B * 12].view(B, 12).int(), torch.tensor([1, 100, 190], dtype=torch.int32, device=dev)
    for pool in (torch.float16, torch.int8, torch.float8_e4m3fn):
        kp = _r(P, 16, 2, 128).mul(20).to(pool)
        s = None if pool == torch.float16 else torch.rand(P, 16, 2, device=dev).half() * 0.05
        for Nq, rows_ok in ((1, True), (4, True), (8, True), (9, False)):        # 4, 16, 32 and 36 query rows per kv head
            q = _r(B, 8, Nq, 128)

            def paged(q=q, table=table, lens=lens, **kw):
                return fa.flash_attention_paged(q, kp, kp, table, lens, k_scale=s, v_scale=s, **kw)
            for kw in (dict(), dict(causal=True, return_lse=True, softcap=30.0), dict(scale=0.2, num_splits=2)):
                check(["decode"] if rows_ok else [], lambda: paged(max_kv_len=190, **kw))
        check([], lambda: paged(q=q[:, :, :2]))
        check([], lambda: paged(q=q[:, :, :2], max_kv_len=190))                  # q strided
        q = _r(B, 8, 1, 128)
        check([], lambda: paged(q=q))
        check([], lambda: paged(q=q, table=table.long(), max_kv_len=190))
        check([], lambda: paged(q=q, lens=lens.long(), max_kv_len=190))
        kn, slots, pools = _r(B, 2, 1, 128)[:, :, 0], torch.tensor([5, -1, 77], device=dev), [kp.clone(), kp.clone(), s, s]
        check(["append"], lambda: fa.kv_append(kn, kn, slots, *pools))
        check([], lambda: fa.kv_append(kn, kn.transpose(0, 1).contiguous().transpose(0, 1), slots, *pools))
    x, cos = _r(B, 8, 1, 128), torch.rand(300, 64, device=dev)
    for off in (0, 7, [1, 2, 290], (1, 2, 3)):
        check(["rope"], lambda: fa.apply_rope(x, cos, cos, off))
        check(["rope"], lambda: fa.apply_rope(x, cos[:, :16].contiguous(), cos[:, :16].contiguous(), off, interleaved=False, rotary_dim=32))
        check([], lambda: fa.apply_rope(x, cos[:, :16], cos[:, :16], off, rotary_dim=32))
    for off in (torch.tensor([4, 5, 6]), torch.tensor([4, 5, 6], device=dev), [True, 1, 2]):
        check([], lambda: fa.apply_rope(x, cos, cos, off))
    check([], lambda: fa.apply_rope(x.requires_grad_(True), cos, cos, 0))
