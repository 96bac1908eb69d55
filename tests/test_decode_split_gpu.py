"""Paged split-KV decode where its launch takes another form: 9 to 32 query rows per kv head (two row tiles per warp, two
warps per head), many partials to merge, more sequences than a CTA scans itself, fixed-point queries of int8 pools,
launches inside a CUDA graph.  Oracle and tolerance (2e-2 max-abs) as in test_decode_gpu.py."""
import pytest
import torch

import mlx_flashattention_steel_b200 as fa
from mlx_flashattention_steel_b200 import attention as A
from oracle import sdpa_oracle as orc

from .test_decode_gpu import _run, _status_checks  # noqa: F401  (the fixture applies to this module too)
from .util import assert_close, make_paged, randn

pytestmark = pytest.mark.gpu

LENS = [0, 1, 2, 16, 17, 31, 33, 500, 2100]


@pytest.mark.parametrize("quant", [None, "int8", "e4m3"])
@pytest.mark.parametrize("Hq,Hkv,Nq", [(6, 2, 3), (32, 8, 3), (32, 8, 4), (16, 16, 17), (8, 2, 6), (16, 2, 4), (3, 1, 11)])
def test_more_than_eight_rows(dev, quant, Hq, Hkv, Nq):
    # 9, 12, 16, 17, 24, 32 and 33 rows (33: the prefill route); sequences shorter than the query chunk among them
    _run(dev, torch.bfloat16, quant, len(LENS), Hq, Hkv, Nq, LENS, 700 + Nq, softcap=30.0 if Nq == 6 else 0.0, holes=True)


@pytest.mark.parametrize("causal,D,block_size,softcap", [(False, 128, 16, 0.0), (True, 64, 16, 0.0), (True, 64, 64, 20.0), (True, 128, 48, 100.0)])
def test_more_than_eight_rows_options(dev, causal, D, block_size, softcap):
    for dtype, Nq in ((torch.float16, 4), (torch.bfloat16, 7)):
        _run(dev, dtype, None, 4, 16, 4, Nq, [700, 5, 1030, 64], 720 + Nq, causal=causal, softcap=softcap, D=D, block_size=block_size)


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("Hq,Hkv,Nq", [(8, 2, 1), (16, 8, 1), (8, 1, 4), (4, 4, 5)])
def test_many_parts_are_merged_in_two_steps(dev, quant, Hq, Hkv, Nq):
    # every CTA holds a part of the long sequence, and a merge block's warps share each row's parts
    _run(dev, torch.float16, quant, 2, Hq, Hkv, Nq, [30000, 1500], 740)


def test_more_sequences_than_a_cta_scans(dev):
    lens = [(7 * i) % 50 for i in range(1030)]                     # every 50th is empty
    _run(dev, torch.bfloat16, "int8", len(lens), 4, 2, 1, lens, 750)
    _run(dev, torch.bfloat16, None, 1024, 4, 2, 1, lens[:1024], 751)


def test_values_beyond_the_end_are_not_read_into_wide_rows(dev):
    pg = make_paged(2, 2, 128, 16, [21, 300], torch.bfloat16, 760)
    for name in ("k", "v"):
        for b, n in enumerate((21, 300)):
            pg[name][int(pg["block_table"][b, n // 16]), n % 16:] = float("nan")
    q = randn((2, 8, 4, 128), torch.bfloat16, 761)
    out = fa.flash_attention_paged(q.to(dev), pg["k"].to(dev), pg["v"].to(dev), pg["block_table"].to(dev), pg["seq_lens"].to(dev), causal=True)
    clean = {n: torch.nan_to_num(pg[n].float()).to(torch.bfloat16) for n in ("k", "v")}
    O, _ = orc.paged_attention(q, clean["k"], clean["v"], pg["block_table"], pg["seq_lens"], causal=True)
    assert_close(out, O, torch.bfloat16)


@pytest.mark.parametrize("Nq", [1, 4])
def test_int8_queries_of_uneven_size(dev, Nq):
    """A row of Q is fixed point below its largest value: rows with one value far above the others, tiny rows, zero rows.
    The step is at most max|q| / 32637, so the scaled score is off by at most sum_d |k_d| * scale * max|q| / 65278: for the outlier
    row (max|q| = 60, sum|k| ~ 128 * 0.8) 0.0083, inside the 2e-2 the outputs are held to."""
    pg = make_paged(3, 2, 128, 16, [40, 700, 333], torch.float16, 770, quant="int8")
    q = randn((3, 8, Nq, 128), torch.float16, 771)
    q[0, :, :, 5] = 60.0
    q[1, 1] = 0.0
    q[1, 2] *= 2.0 ** -12
    args = [x.to(dev) for x in (q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"])]
    out = fa.flash_attention_paged(*args, causal=True, k_scale=pg["k_scale"].to(dev), v_scale=pg["v_scale"].to(dev))
    O, _ = orc.paged_attention(q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"], causal=True, k_scale=pg["k_scale"],
                               v_scale=pg["v_scale"])
    assert_close(out, O, torch.float16)


@pytest.mark.parametrize("Nq", [1, 4])
def test_replayed_from_a_graph(dev, Nq):
    """The main kernel and the merge kernel are joined by a programmatic dependency: it survives capture, and replays on
    changed inputs give what direct calls give."""
    pg = make_paged(3, 2, 128, 16, [900, 65, 333], torch.bfloat16, 780)
    k, v, table = (pg[n].to(dev) for n in ("k", "v", "block_table"))
    lens, q = pg["seq_lens"].to(dev), randn((3, 8, Nq, 128), torch.bfloat16, 781).to(dev)

    def call():
        return fa.flash_attention_paged(q, k, v, table, lens, causal=True, max_kv_len=900)

    from mlx_flashattention_steel_b200 import attention as A
    A._set_check_decode_status(False)                               # the check synchronises, which a capture does not allow
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    for step in range(3):
        q.copy_(randn(tuple(q.shape), torch.bfloat16, 790 + step).to(dev))
        lens.copy_(torch.tensor([900 - 100 * step, 65 - step, 333], dtype=torch.int32, device=dev))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, call())


@pytest.mark.parametrize("Hq,Nq,softcap", [(32, 1, 0.0), (32, 2, 0.0), (8, 1, 30.0)])
def test_two_warps_take_a_heads_units_in_turn(dev, Hq, Nq, softcap):
    """int8 pools, 8 kv heads, 32 or more units per CTA if all sequences were as long as the longest: every CTA leaves two
    partials per sequence, one of them without a unit where a sequence has a single one in the CTA."""
    lens = [2000] + [(13 * i) % 90 for i in range(39)]
    _run(dev, torch.bfloat16, "int8", len(lens), Hq, 8, Nq, lens, 795, softcap=softcap)
    _run(dev, torch.float16, "int8", 1, Hq, 8, Nq, [76000], 796, softcap=softcap)


@pytest.mark.parametrize("peak", [3.0, 30.0, 300.0])
@pytest.mark.parametrize("Hkv,Nq,max_len", [(2, 1, 16), (2, 4, 16), (8, 2, 1200)])
def test_int8_queries_keep_f16_precision(dev, Hkv, Nq, max_len, peak):
    """Scores of int8 pools are at least as exact as with Q rounded to f16, whichever channels K weighs: one channel of Q
    is `peak` and K has a hundredth of its usual size there.  A sequence of one token has its score as its lse.  An f16
    rounding of q_d is off by at most 2^-11 |q_d| and by 2^-11 |q_d| / sqrt(3) in the mean, if evenly spread; the errors
    of the channels add up as squares.  (8, 2, 1200): two warps per head."""
    B, G = 64, 4
    g = torch.Generator().manual_seed(799)
    q = torch.randn((B, Hkv * G, Nq, 128), generator=g)
    q[..., 37] = peak
    q = q.to(torch.float16)
    P = B * ((max_len + 15) // 16)
    k = torch.randint(-127, 128, (P, 16, Hkv, 128), generator=g, dtype=torch.int8)
    k[..., 37] = torch.randint(-1, 2, k.shape[:-1], generator=g, dtype=torch.int8)
    ks = torch.full((P, 16, Hkv), 0.02, dtype=torch.float16)
    table = torch.arange(P, dtype=torch.int32).view(B, -1)
    lens = torch.ones(B, dtype=torch.int32)
    _, lse = fa.flash_attention_paged(*(x.to(dev) for x in (q, k, k, table, lens)), k_scale=ks.to(dev), v_scale=ks.to(dev),
                                      max_kv_len=max_len, return_lse=True)
    kd = (k[table[:, 0].long(), 0].double() * ks[0, 0, 0].double()).repeat_interleave(G, dim=1)      # [B, Hq, 128]
    c = 128 ** -0.5 * 1.4426950408889634
    terms = q.double() * kd.unsqueeze(2) * c
    err = lse.double().cpu() - terms.sum(-1)
    bound = 2.0 ** -11 / 3 ** 0.5 * terms.pow(2).sum(-1).mean().sqrt()
    assert float(err.pow(2).mean().sqrt()) <= float(bound)


@pytest.mark.parametrize("quant", [None, "int8", "e4m3"])
@pytest.mark.parametrize("Nq", [1, 4])
def test_queries_that_are_not_finite(dev, quant, Nq):
    """A NaN or an infinity in a query row makes that row NaN, as the prefill route has it, and no other."""
    pg = make_paged(2, 2, 128, 16, [40, 3000], torch.bfloat16, 775, quant=quant)
    q = randn((2, 8, Nq, 128), torch.bfloat16, 776)
    bad = q.clone()
    bad[0, 1, Nq - 1, 3], bad[1, 6, 0, 127], bad[1, 7, 0, 64] = float("nan"), float("nan"), float("inf")
    rows = torch.zeros(q.shape[:3], dtype=torch.bool)
    rows[0, 1, Nq - 1] = rows[1, 6, 0] = rows[1, 7, 0] = True
    kw = {} if quant is None else dict(k_scale=pg["k_scale"].to(dev), v_scale=pg["v_scale"].to(dev))
    args = [pg[n].to(dev) for n in ("k", "v", "block_table", "seq_lens")]
    out = fa.flash_attention_paged(bad.to(dev), *args, **kw).cpu()
    assert torch.isnan(out[rows]).all()
    assert torch.equal(out[~rows], fa.flash_attention_paged(q.to(dev), *args, **kw).cpu()[~rows])


@pytest.mark.parametrize("quant", ["int8", "e4m3"])
def test_wide_rows_beyond_f16(dev, quant):
    """Queries whose scaled values leave f16's range: 8-bit pools, 16 rows per kv head."""
    pg = make_paged(2, 2, 128, 16, [40, 700], torch.bfloat16, 777, quant=quant)
    q = randn((2, 8, 4, 128), torch.bfloat16, 778)
    q[:, ::2] *= 3e6
    q[:, 1] *= 1e-9
    # a power of two, so that K is the same number in bf16: the largest score is far from the others, not from its rounding
    pg["k_scale"] = torch.full_like(pg["k_scale"], 2.0 ** -5 if quant == "int8" else 2.0 ** -7)
    args = [x.to(dev) for x in (q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"])]
    kw = dict(k_scale=pg["k_scale"], v_scale=pg["v_scale"])
    out = fa.flash_attention_paged(*args, causal=True, **{n: x.to(dev) for n, x in kw.items()})
    O, _ = orc.paged_attention(q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"], causal=True, **kw)
    assert_close(out, O, torch.bfloat16)


@pytest.mark.parametrize("quant", ["int8", "e4m3"])
@pytest.mark.parametrize("Nq", [1, 4])
def test_value_scales_far_apart(dev, quant, Nq):
    """P is multiplied by v_scale over a power of two near the first scale: later scales may be far above it (a first
    token of zeros, stored with the smallest scale there is)."""
    lens = [700, 37, 40]
    pg = make_paged(3, 2, 128, 16, lens, torch.bfloat16, 785, quant=quant)
    for b in range(3):
        page = int(pg["block_table"][b, 0])
        pg["v"][page, 0] = 0
        pg["v_scale"][page, 0] = 2.0 ** -24
    mine = pg["block_table"][2, :3].long()                 # a sequence whose scales are negative, and tiny
    pg["v_scale"][mine] *= -2.0 ** -12
    late = int(pg["block_table"][0, 20])
    pg["v_scale"][late] *= 512.0
    q = randn((3, 8, Nq, 128), torch.bfloat16, 786)
    kw = dict(k_scale=pg["k_scale"], v_scale=pg["v_scale"])
    out, lse = fa.flash_attention_paged(*(x.to(dev) for x in (q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"])), causal=True,
                                        return_lse=True, **{n: x.to(dev) for n, x in kw.items()})
    O, L = orc.paged_attention(q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"], causal=True, **kw)
    assert_close(lse, L, torch.bfloat16, "lse")
    for b in (1, 2):                                       # relative to the sequence's own values
        top = float(O[b].abs().max())
        assert_close(out[b] / top, O[b] / top, torch.bfloat16)
    # the values of one page are 512 times the others': the same 2e-2, relative to the largest
    assert_close(out[:1] / float(O[0].abs().max()), O[:1] / float(O[0].abs().max()), torch.bfloat16)


def test_scales_at_any_address(dev):
    """9 to 32 rows per kv head take the scales of 8-bit pools wherever they lie, as the prefill route does."""
    pg = make_paged(2, 2, 128, 16, [40, 333], torch.bfloat16, 787, quant="int8")
    q = randn((2, 8, 4, 128), torch.bfloat16, 788)

    def odd(x):
        flat = torch.empty(x.numel() + 1, dtype=x.dtype, device=dev)
        flat[1:] = x.flatten().to(dev)
        return flat[1:].view(x.shape)

    args = [x.to(dev) for x in (q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"])]
    out = fa.flash_attention_paged(*args, causal=True, k_scale=odd(pg["k_scale"]), v_scale=odd(pg["v_scale"]))
    O, _ = orc.paged_attention(q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"], causal=True, k_scale=pg["k_scale"],
                               v_scale=pg["v_scale"])
    assert_close(out, O, torch.bfloat16)


def test_what_longer_queries_refuse(dev):
    """Only flash_attention_paged takes more than 8 rows per kv head; a NaN scale and a negative soft cap are errors there
    as on the prefill route."""
    pg = make_paged(1, 2, 128, 16, [40], torch.bfloat16, 789)
    args = [x.to(dev) for x in (randn((1, 8, 4, 128), torch.bfloat16, 790), pg["k"], pg["v"], pg["block_table"], pg["seq_lens"])]
    for kw in (dict(softcap=-1.0), dict(scale=float("nan"))):
        with pytest.raises(ValueError):
            fa.flash_attention_paged(*args, **kw)
    q, k, v, table, lens = args
    with pytest.raises(NotImplementedError):
        A._decode_raw(q, k, v, None, None, table, lens, 40, 0.1, True, 0.0, 16, False, None, packed=True)


def test_more_than_1024_sequences_from_a_graph(dev):
    """Beyond 1024 sequences the merge kernel reads the plan kernel's sums: replays whose lengths change between them."""
    B = 1100
    lens0 = [(11 * i) % 70 for i in range(B)]
    pg = make_paged(B, 2, 128, 16, [69] * B, torch.bfloat16, 782)
    k, v, table = (pg[n].to(dev) for n in ("k", "v", "block_table"))
    lens, q = torch.tensor(lens0, dtype=torch.int32, device=dev), randn((B, 4, 1, 128), torch.bfloat16, 783).to(dev)

    def call():
        return fa.flash_attention_paged(q, k, v, table, lens, causal=True, max_kv_len=69)

    A._set_check_decode_status(False)                               # the check synchronises, which a capture does not allow
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    for step in range(3):
        now = torch.tensor([(n * (step + 3) + 5 * step) % 70 for n in lens0], dtype=torch.int32)
        lens.copy_(now.to(dev))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, call())
        O, _ = orc.paged_attention(q.cpu()[:40], pg["k"], pg["v"], pg["block_table"][:40], now[:40], causal=True)
        assert_close(out[:40], O, torch.bfloat16)


@pytest.mark.parametrize("lens", [[9000], [5000, 0, 40], [3000, 1, 1500, 700, 16], [800, 31, 0] * 3, [400 + 7 * i for i in range(19)]])
@pytest.mark.parametrize("quant,D", [(None, 64), (None, 128), ("int8", 128)])
def test_rows_merged_by_any_number_of_warps(dev, lens, quant, D):
    # 32 down to 1 warps to a row of the output; parts that are few, many, and none at all beside them
    _run(dev, torch.bfloat16, quant, len(lens), 8, 2, 1, lens, 810, D=D)
    _run(dev, torch.float16, quant, len(lens), 8, 8, 3, lens, 811, D=D, softcap=30.0)


def _serve_step(s):
    q, k = (fa.apply_rope(s[n], s["cos"], s["sin"], s["pos"], interleaved=False) for n in ("q", "k"))
    fa.kv_append(k[:, :, 0], s["v"][:, :, 0], s["slots"], s["kp"], s["vp"])
    return fa.flash_attention_paged(q, s["kp"], s["vp"], s["table"], s["lens"], causal=True, max_kv_len=300)


@pytest.mark.parametrize("front", ["nothing", "memset", "copy", "other stream", "lengths"])
def test_launches_that_start_before_the_one_in_front_has_ended(dev, front):
    """Rotation, append, decode and merge are programmatic dependents of what is in front of them, whatever that is: each step
    reads what the one before wrote (rotated rows, appended rows, lengths), directly and from a graph."""
    g = torch.Generator().manual_seed(31)
    B, P = 5, 120
    r = lambda *n: torch.randn(n, generator=g).to(torch.bfloat16).to(dev)    # noqa: E731
    s = dict(kp=r(P, 16, 2, 128), vp=r(P, 16, 2, 128), q=r(B, 8, 1, 128), k=r(B, 2, 1, 128), v=r(B, 2, 1, 128), pos=[10, 299, 16, 17, 100])
    s["table"] = torch.randperm(P, generator=g)[:B * 20].view(B, 20).int().to(dev)
    s["lens"] = torch.tensor([p + 1 for p in s["pos"]], dtype=torch.int32, device=dev)
    s["slots"] = torch.tensor([int(s["table"][b, p // 16]) * 16 + p % 16 for b, p in enumerate(s["pos"])], device=dev)
    ang = torch.arange(300.0)[:, None] * torch.rand(64, generator=g)
    s["cos"], s["sin"] = ang.cos().to(dev), ang.sin().to(dev)
    rot = [torch.cat([x[..., :64] * c - x[..., 64:] * t, x[..., :64] * t + x[..., 64:] * c], -1).to(torch.bfloat16)
           for x in (s["q"].double(), s["k"].double())
           for c, t in [(s["cos"][s["pos"]].double()[:, None, None], s["sin"][s["pos"]].double()[:, None, None])]]
    kp, vp = s["kp"].clone(), s["vp"].clone()
    kp.view(-1, 2, 128)[s["slots"]], vp.view(-1, 2, 128)[s["slots"]] = rot[1][:, :, 0], s["v"][:, :, 0]
    want, _ = orc.paged_attention(*(x.cpu() for x in (rot[0], kp, vp, s["table"], s["lens"])), causal=True)
    A._set_check_decode_status(False)
    side, big, pinned = torch.cuda.Stream(), torch.zeros(1 << 22, device=dev), torch.zeros(256).pin_memory()
    lens = s["lens"].clone()

    def call():
        if front == "memset":
            big.zero_()
        elif front == "copy":
            big[:256].copy_(pinned, non_blocking=True)
        elif front == "other stream":
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                big.add_(1.0)
            torch.cuda.current_stream().wait_stream(side)
        elif front == "lengths":
            s["lens"].zero_()
            big.mul_(1.0)
            s["lens"].add_(lens)
        return _serve_step(s)

    for _ in range(20):
        out = call()
    assert_close(out, want, torch.bfloat16)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    for _ in range(5):
        out.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert_close(out, want, torch.bfloat16)


@pytest.mark.parametrize("quant", [None, "int8"])
@pytest.mark.parametrize("lens", [[17, 400], [0, 0, 5], [16] * 64, [(37 * i) % 200 for i in range(64)], [(37 * i) % 200 for i in range(65)],
                                  [1, 0, 2100, 33, 31, 32] * 5, [5000, 16], [64] * 33, [6200] * 31])
def test_ctas_of_one_sequence_each(dev, quant, lens):
    # few units: no CTA has two sequences; up to 64 of them, more than a lane's first one, empty ones at every place, and sums
    # of units on both sides of the rule
    _run(dev, torch.bfloat16, quant, len(lens), 8, 2, 1, lens, 820)
    _run(dev, torch.bfloat16, quant, len(lens), 32, 8, 3 if len(lens) < 32 else 1, lens, 821)


@pytest.mark.parametrize("Hq,Nq,softcap", [(32, 1, 0.0), (16, 4, 30.0)])
@pytest.mark.parametrize("lens", [[60000, 40000], [60000, 0, 40000], [38000, 1, 0, 17, 30001], [3344 - 150 * (i % 20) for i in range(23)]])
def test_two_warps_per_head_in_ctas_of_one_sequence_each(dev, lens, Hq, Nq, softcap):
    # int8, 8 kv heads: 32 or more units per CTA (two warps take them in turn) of so few sequences that no CTA has two; a
    # sequence of one unit leaves the second warp without any
    _run(dev, torch.bfloat16, "int8", len(lens), Hq, 8, Nq, lens, 830, softcap=softcap)


def test_lengths_written_by_the_launch_directly_in_front(dev):
    """The merge kernel reads the lengths before it waits for the main kernel, which therefore lets it in only after its own wait:
    the append in front, which lets its successor in at once, writes them here (16-bit rows are copied bit for bit)."""
    lens = [700, 16, 0, 333, 1]
    pg = make_paged(len(lens), 2, 128, 16, lens, torch.bfloat16, 840)
    q = randn((len(lens), 8, 1, 128), torch.bfloat16, 841)
    want, _ = orc.paged_attention(q, pg["k"], pg["v"], pg["block_table"], pg["seq_lens"], causal=True)
    buf, other = (torch.zeros(32, dtype=torch.int32, device=dev) for _ in range(2))
    now = torch.zeros(32, dtype=torch.int32)
    now[:len(lens)] = pg["seq_lens"]
    rows = [x.to(dev).view(torch.float16).view(1, 1, 64) for x in (torch.zeros_like(now), now)]
    pools = [x.view(torch.float16).view(1, 1, 1, 64) for x in (buf, other)]
    slot = torch.zeros(1, dtype=torch.int64, device=dev)
    qd, kp, vp, table = q.to(dev), pg["k"].to(dev), pg["v"].to(dev), pg["block_table"].to(dev)
    A._set_check_decode_status(False)

    def call():
        for r in rows:
            fa.kv_append(r, r, slot, *pools)
        return fa.flash_attention_paged(qd, kp, vp, table, buf[:len(lens)], causal=True, max_kv_len=700)

    for _ in range(20):
        assert_close(call(), want, torch.bfloat16)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    for _ in range(20):
        out.fill_(1.0)
        graph.replay()
        assert_close(out, want, torch.bfloat16)
