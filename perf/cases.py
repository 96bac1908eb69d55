"""The attention calls whose speed this repository answers for.

Each case is one call a model makes through the public entry points: a prefill, a training step (forward and
backward), a decode step over a paged cache, a chunk of a paged prefill, a whole serving step of one layer (rotate,
append, attend).  The listed ones are the shapes of the repository's own configurations and benchmark, with the small,
the ragged and the short-query calls that stand beside them in use; ``draw`` gives other sizes of the same ranges.
"""
import math
import random

import torch

import mlx_flashattention_steel_b200 as fa

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
KV_BYTES = {"bf16": 2, "fp16": 2, "int8": 1, "e4m3": 1}


def listed():
    return [
        # config 1: the float32 parity case, also what a float32 user calls at a small model's size
        dict(name="fp32_causal_1k", kind="dense", B=1, Hq=8, Hkv=8, N=1024, S=1024, D=128, dtype="fp32", causal=True,
             softcap=0.0, window=-1, lse=False, grad=False),
        # config 2: grouped-query prefill with a soft cap and the lse kept
        dict(name="gqa_prefill_8k_softcap", kind="dense", B=4, Hq=32, Hkv=8, N=8192, S=8192, D=128, dtype="bf16",
             causal=True, softcap=50.0, window=-1, lse=True, grad=False),
        # config 3: sliding-window prefill of a long document
        dict(name="window_fp16_32k", kind="dense", B=2, Hq=16, Hkv=16, N=32768, S=32768, D=128, dtype="fp16",
             causal=True, softcap=0.0, window=512, lse=False, grad=False),
        # a training step of a grouped-query model at a usual context length
        dict(name="train_gqa_d128_4k", kind="dense", B=2, Hq=32, Hkv=8, N=4096, S=4096, D=128, dtype="bf16",
             causal=True, softcap=0.0, window=-1, lse=False, grad=True),
        # a training step of cross attention: nothing is a multiple of a tile, no mask
        dict(name="train_cross_d64_ragged", kind="dense", B=4, Hq=12, Hkv=12, N=1000, S=777, D=64, dtype="fp16",
             causal=False, softcap=0.0, window=-1, lse=False, grad=True),
        # config 5: packed sequences, training
        dict(name="varlen_train_64k_d64", kind="varlen", tokens=65536, lo=128, hi=4096, Hq=16, Hkv=16, D=64,
             dtype="bf16", causal=True, grad=True, lens_seed=5),
        # config 4: one decode step of a large batch over an int8 pool
        dict(name="decode_int8_b128", kind="paged", B=128, Nq=1, lo=512, hi=32768, Hq=32, Hkv=8, D=128, dtype="bf16",
             kv="int8", page=16, lens_seed=4),
        # one very long sequence, alone
        dict(name="decode_int8_256k_b1", kind="paged", B=1, Nq=1, lo=262144, hi=262144, Hq=32, Hkv=8, D=128,
             dtype="bf16", kv="int8", page=16, lens_seed=0),
        # a few query tokens per sequence: the verification step of speculative decoding
        dict(name="verify_bf16_n4", kind="paged", B=32, Nq=4, lo=512, hi=8192, Hq=32, Hkv=8, D=128, dtype="bf16",
             kv="bf16", page=16, lens_seed=1),
        # a chunk of a prefill against what is already in the pool
        dict(name="chunk_prefill_int8", kind="paged", B=4, Nq=512, lo=1024, hi=8192, Hq=32, Hkv=8, D=128,
             dtype="bf16", kv="int8", page=16, lens_seed=2),
        # one layer of a decode step of a small batch: rotate q and k, append, attend; the smallest call here
        dict(name="serve_step_bf16_b8", kind="serve", B=8, lo=100, hi=1000, Hq=32, Hkv=8, D=128, dtype="bf16",
             kv="bf16", page=16, lens_seed=3),
        # block-sparse attention with the sliding-window mask builder
        dict(name="sparse_window_fp16_8k", kind="sparse", B=2, H=16, N=8192, D=128, dtype="fp16", window=512,
             causal=True),
    ]


def _size(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm, half of the time a multiple of 64."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5 and n >= 128:
        n = n // 64 * 64
    return max(lo, min(hi, n))


def _heads(rng):
    Hkv = rng.choice([1, 2, 4, 8, 16])
    return Hkv * rng.choice([g for g in (1, 2, 4, 8) if Hkv * g <= 32]), Hkv


def _draw(rng):
    kind = rng.choice(["fp32", "prefill", "prefill", "window", "train", "train", "varlen", "decode", "decode", "verify",
                       "chunk", "serve", "serve", "sparse"])
    half = rng.choice(["bf16", "fp16"])
    if kind in ("fp32", "prefill", "window", "train"):
        Hq, Hkv = _heads(rng)
        c = dict(kind="dense", B=rng.randint(1, 4), Hq=Hq, Hkv=Hkv, D=rng.choice([64, 128]), dtype=half,
                 causal=rng.random() < 0.7, softcap=0.0, window=-1, lse=False, grad=False)
        if kind == "fp32":
            c.update(N=_size(rng, 128, 2048), dtype="fp32")
        elif kind == "prefill":
            c.update(N=_size(rng, 128, 8192), D=rng.choice([64, 128, 128, 256]), softcap=rng.choice([0.0, 0.0, 30.0, 50.0]),
                     lse=rng.random() < 0.3)
        elif kind == "window":
            c.update(N=_size(rng, 2048, 32768), window=_size(rng, 128, 4096), causal=True)
        else:
            c.update(N=_size(rng, 128, 8192), grad=True, softcap=rng.choice([0.0, 0.0, 0.0, 30.0]))
        # as many keys as queries, or a prefix before them
        c["S"] = c["N"] if rng.random() < 0.7 else c["N"] + _size(rng, 64, 2048)
        return c
    if kind == "varlen":
        Hq, Hkv = _heads(rng)
        hi = _size(rng, 256, 4096)
        return dict(kind="varlen", tokens=_size(rng, 2048, 65536), lo=min(128, hi), hi=hi, Hq=Hq, Hkv=Hkv,
                    D=rng.choice([64, 128]), dtype=half, causal=rng.random() < 0.8, grad=rng.random() < 0.6,
                    lens_seed=rng.randrange(1 << 20))
    if kind == "sparse":
        return dict(kind="sparse", B=rng.randint(1, 2), H=rng.choice([4, 8, 16]), N=_size(rng, 1024, 16384),
                    D=rng.choice([64, 128]), dtype=half, window=_size(rng, 128, 1024), causal=rng.random() < 0.7)
    kv = rng.choice(["int8", "e4m3", half])
    # head dimension 64 goes with 16-bit pools
    c = dict(kind="paged", Hq=32, Hkv=8, D=64 if kv == half and rng.random() < 0.3 else 128, dtype=half, kv=kv,
             page=rng.choice([16, 16, 16, 32, 64]), lens_seed=rng.randrange(1 << 20))
    c["Hkv"] = rng.choice([2, 4, 8])
    c["Hq"] = c["Hkv"] * rng.choice([4, 8] if c["Hkv"] < 8 else [4])
    if kind == "decode":
        hi = _size(rng, 512, 65536)
        c.update(B=_size(rng, 1, 128), Nq=1, lo=max(64, hi // rng.choice([1, 4, 64])), hi=hi)
    elif kind == "verify":
        hi = _size(rng, 512, 16384)
        c.update(B=_size(rng, 1, 64), Nq=rng.randint(2, 4), lo=max(64, hi // 16), hi=hi)
    elif kind == "chunk":
        hi = _size(rng, 1024, 16384)
        c.update(B=rng.randint(1, 4), Nq=_size(rng, 64, 1024), lo=max(1024, hi // 8), hi=hi)
    else:
        hi = _size(rng, 128, 4096)
        c.update(kind="serve", B=_size(rng, 1, 64), lo=max(64, hi // 8), hi=hi)
    return c


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        if w["flops"] <= (2e10 if c["dtype"] == "fp32" else 1.2e12) and w["bytes"] <= 4e9:
            return c


# ---------------------------------------------------------------------------
# what a case is made of
# ---------------------------------------------------------------------------
def _lens(c):
    """Sequence lengths of a packed or paged case (on the host: a scheduler knows them)."""
    rng = random.Random(c["lens_seed"])
    if c["kind"] == "varlen":
        lens = []
        while sum(lens) < c["tokens"]:
            lens.append(rng.randint(c["lo"], c["hi"]))
        lens[-1] -= sum(lens) - c["tokens"]
        return lens
    return [rng.randint(c["lo"], c["hi"]) for _ in range(c["B"])]


def _pairs(N, S, causal, window):
    """Visible (query, key) pairs of one head; query i stands at key position i + S - N."""
    n = 0
    if not causal and window < 0:
        return N * S
    for i in range(N):
        last = i + S - N if causal else S - 1
        first = max(0, i + S - N - window) if window >= 0 else 0
        n += max(0, last - first + 1)
    return n


def _randn(shape, dtype, gen):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32 if dtype == torch.float32 else dtype)


def _pool(shape, kv, gen):
    """Values of one pool that stand for N(0, 1), and the scales of an 8-bit one."""
    if kv in DTYPES:
        return _randn(shape, DTYPES[kv], gen), None
    scale = (torch.rand(shape[:3], generator=gen, device="cuda") * 0.01 + 0.02).to(torch.float16)
    if kv == "e4m3":
        scale = scale / 4.0      # x / scale reaches about 450, the type's largest value is 448
    out = torch.empty(shape, device="cuda", dtype=torch.int8 if kv == "int8" else torch.float8_e4m3fn)
    step = 8192
    for p in range(0, shape[0], step):
        x = torch.randn(out[p:p + step].shape, generator=gen, device="cuda", dtype=torch.float16)
        x /= scale[p:p + step].unsqueeze(-1)
        out[p:p + step] = x.round_().clamp_(-127, 127).to(torch.int8) if kv == "int8" else x.clamp_(-448, 448).to(out.dtype)
    return out, scale


def prepare(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[c["dtype"]]
    s = {"case": c}
    if c["kind"] in ("dense", "varlen", "sparse"):
        if c["kind"] == "dense":
            qs, ks = (c["B"], c["Hq"], c["N"], c["D"]), (c["B"], c["Hkv"], c["S"], c["D"])
        elif c["kind"] == "varlen":
            qs, ks = (1, c["Hq"], c["tokens"], c["D"]), (1, c["Hkv"], c["tokens"], c["D"])
            lens = _lens(c)
            cu = [0]
            for n in lens:
                cu.append(cu[-1] + n)
            s["cu"] = torch.tensor(cu, dtype=torch.int32, device="cuda")
            s["max"] = max(lens)
        else:
            qs = ks = (c["B"], c["H"], c["N"], c["D"])
            s["mask"] = fa.make_sliding_window_mask(c["N"], c["window"], c["D"], causal=c["causal"], device="cuda")
        s["q"], s["k"], s["v"] = _randn(qs, dt, gen), _randn(ks, dt, gen), _randn(ks, dt, gen)
        if c.get("grad"):
            s["do"] = _randn(qs, dt, gen)
            for n in "qkv":
                s[n].requires_grad_(True)
        return s
    lens = _lens(c)
    page, blocks = c["page"], [-(-n // c["page"]) for n in lens]
    P = sum(blocks)
    perm = torch.randperm(P, generator=gen, device="cuda").to(torch.int32).cpu()
    table = torch.full((c["B"], max(blocks)), -1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(blocks):
        table[b, :n] = perm[at:at + n]
        at += n
    s["table"], s["lens"], s["max"] = table.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), max(lens)
    shape = (P, page, c["Hkv"], c["D"])
    s["kp"], s["ks"] = _pool(shape, c["kv"], gen)
    s["vp"], s["vs"] = _pool(shape, c["kv"], gen)
    s["q"] = _randn((c["B"], c["Hq"], c.get("Nq", 1), c["D"]), dt, gen)
    if c["kind"] == "serve":
        # the new token of every sequence, its slot, its position, and the model's rotary tables
        s["k"] = _randn((c["B"], c["Hkv"], 1, c["D"]), dt, gen)
        s["v"] = _randn((c["B"], c["Hkv"], 1, c["D"]), dt, gen)
        s["slots"] = torch.tensor([int(table[b, (n - 1) // page]) * page + (n - 1) % page for b, n in enumerate(lens)],
                                  dtype=torch.int64, device="cuda")
        s["pos"] = [n - 1 for n in lens]
        freq = 10000.0 ** (-torch.arange(0, c["D"], 2, device="cuda", dtype=torch.float32) / c["D"])
        ang = torch.arange(c["hi"], device="cuda", dtype=torch.float32)[:, None] * freq
        s["cos"], s["sin"] = ang.cos(), ang.sin()
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "serve":
        q = fa.apply_rope(s["q"], s["cos"], s["sin"], s["pos"], interleaved=False)
        k = fa.apply_rope(s["k"], s["cos"], s["sin"], s["pos"], interleaved=False)
        fa.kv_append(k[:, :, 0], s["v"][:, :, 0], s["slots"], s["kp"], s["vp"], s["ks"], s["vs"])
        out = fa.flash_attention_paged(q, s["kp"], s["vp"], s["table"], s["lens"], causal=True, block_size=c["page"],
                                       k_scale=s["ks"], v_scale=s["vs"], max_kv_len=s["max"])
        return [out, s["kp"], s["vp"], s["ks"], s["vs"]]
    if c["kind"] == "paged":
        return fa.flash_attention_paged(s["q"], s["kp"], s["vp"], s["table"], s["lens"], causal=True,
                                        block_size=c["page"], k_scale=s["ks"], v_scale=s["vs"], max_kv_len=s["max"])
    if c["kind"] == "dense":
        out = fa.flash_attention(s["q"], s["k"], s["v"], causal=c["causal"], softcap=c["softcap"],
                                 window_size=(c["window"], 0) if c["window"] >= 0 else None, return_lse=c["lse"])
    elif c["kind"] == "varlen":
        out = fa.flash_attention_varlen(s["q"], s["k"], s["v"], s["cu"], s["cu"], s["max"], s["max"], causal=c["causal"])
    else:
        out = fa.flash_attention_sparse(s["q"], s["k"], s["v"], s["mask"], causal=c["causal"])
    if c.get("grad"):
        return [out.detach(), *torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["do"])]
    return out


def work(c):
    eb = 4 if c["dtype"] == "fp32" else 2
    if c["kind"] in ("paged", "serve"):
        lens, Nq, D = _lens(c), c.get("Nq", 1), c["D"]
        row = D * KV_BYTES[c["kv"]] + (2 if c["kv"] in ("int8", "e4m3") else 0)
        byts = sum(lens) * c["Hkv"] * 2 * row + 2 * c["B"] * c["Hq"] * Nq * D * eb
        pairs = sum(_pairs(min(Nq, n), n, True, -1) for n in lens)
        return {"bytes": float(byts), "flops": 4.0 * c["Hq"] * D * pairs}
    if c["kind"] == "sparse":
        cells = float(fa.make_sliding_window_mask(c["N"], c["window"], c["D"], causal=c["causal"]).sum())
        return {"bytes": 4.0 * c["B"] * c["H"] * c["N"] * c["D"] * eb,
                "flops": 4.0 * c["B"] * c["H"] * c["D"] * cells * 32 * (32 if c["D"] <= 64 else 16)}
    if c["kind"] == "varlen":
        B, N, S, pairs = 1, c["tokens"], c["tokens"], sum(_pairs(n, n, c["causal"], -1) for n in _lens(c))
    else:
        B, N, S, pairs = c["B"], c["N"], c["S"], _pairs(c["N"], c["S"], c["causal"], c["window"])
    q, kv = B * c["Hq"] * N * c["D"], B * c["Hkv"] * S * c["D"]
    # forward: q, k, v in, out out; backward: out's gradient in, three gradients out
    byts = eb * (2 * q + 2 * kv + (2 * q + 2 * kv if c["grad"] else 0)) + (4 * B * c["Hq"] * N if c.get("lse") else 0)
    return {"bytes": float(byts), "flops": 4.0 * B * c["Hq"] * c["D"] * pairs * (3.5 if c["grad"] else 1.0)}


def tolerance(c):
    # Four times what the calls differ by from float64 on the same inputs: 8.5e-7 (fp32, 2000 keys), 3.1e-4 (fp16),
    # 2.6e-3 (bf16); paged calls, which also round the dequantised values, 4.2e-4 and 3.3e-3.  Single values of a
    # gradient are off by up to 0.13 (bf16) and 0.01 (fp16) of the root mean square, those of an output by 0.024.
    if c["dtype"] == "fp32":
        return {"rel": 3.4e-6, "max": 3e-5}
    paged = c["kind"] in ("paged", "serve")
    if c["dtype"] == "fp16":
        return {"rel": 1.7e-3 if paged else 1.25e-3, "max": 0.04}
    return {"rel": 1.3e-2 if paged else 1e-2, "max": 0.5 if c.get("grad") else 0.1}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _attend64(q, k, v, scale, causal, window=-1, softcap=0.0, mask=None, do=None):
    """Attention of one head in float64, [N, D] against [S, D]; with ``do`` also the gradients of q, k and v."""
    N, S, D = q.shape[0], k.shape[0], q.shape[1]
    out, lse = torch.zeros_like(q), torch.full((N,), -math.inf, dtype=torch.float64, device=q.device)
    dq, dk, dv = (torch.zeros_like(x) for x in (q, k, v)) if do is not None else (None, None, None)
    step = max(64, (1 << 26) // max(S, 1))
    if window >= 0:
        step = min(step, 2048)
    for i in range(0, N, step):
        n = min(step, N - i)
        hi = min(S, i + n + S - N) if causal else S
        lo = max(0, i + S - N - window) if window >= 0 else 0
        if hi <= lo:
            continue
        raw = q[i:i + n] @ k[lo:hi].T
        raw *= scale
        s = softcap * torch.tanh(raw / softcap) if softcap > 0 else raw
        qpos = torch.arange(i, i + n, device=q.device)[:, None] + (S - N)
        kpos = torch.arange(lo, hi, device=q.device)[None, :]
        off = torch.zeros((n, hi - lo), dtype=torch.bool, device=q.device)
        if causal:
            off |= kpos > qpos
        if window >= 0:
            off |= kpos < qpos - window
        if mask is not None:
            off |= ~mask(i, i + n, lo, hi)
        s = s.masked_fill(off, -math.inf)
        m = s.amax(1, keepdim=True)
        m[m == -math.inf] = 0.0
        p = torch.exp(s - m)
        total = p.sum(1, keepdim=True)
        lse[i:i + n] = (m + torch.log(total))[:, 0] / math.log(2.0)
        p /= torch.where(total > 0, total, torch.ones_like(total))
        out[i:i + n] = p @ v[lo:hi]
        if do is not None:
            g = do[i:i + n]
            dv[lo:hi] += p.T @ g
            ds = p * (g @ v[lo:hi].T - (g * out[i:i + n]).sum(1, keepdim=True))
            if softcap > 0:
                ds *= 1 - torch.tanh(raw / softcap) ** 2
            dq[i:i + n] = ds @ k[lo:hi] * scale
            dk[lo:hi] += ds.T @ q[i:i + n] * scale
    return out, lse, dq, dk, dv


def _rotated64(x, s):
    half = x.shape[-1] // 2
    pos = torch.tensor(s["pos"], device=x.device)
    cos, sin = s["cos"][pos].double()[:, None, None], s["sin"][pos].double()[:, None, None]
    a, b = x[..., :half].double(), x[..., half:].double()
    return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)


def exact(c, seed):
    """What ``run`` returns for these inputs, in float64.  The bytes of an 8-bit pool have no such value."""
    s = prepare(c, seed)
    D, scale = c["D"], 1.0 / math.sqrt(c["D"])
    if c["kind"] in ("paged", "serve"):
        q, pools = s["q"].double(), []
        for pool, sc in ((s["kp"], s["ks"]), (s["vp"], s["vs"])):
            pools.append((pool.view(-1, c["Hkv"], D), None if sc is None else sc.view(-1, c["Hkv"])))
        new = None
        if c["kind"] == "serve":
            q, new = _rotated64(s["q"], s), (_rotated64(s["k"], s)[:, :, 0], s["v"][:, :, 0].double())
            if c["kv"] in ("int8", "e4m3"):     # the stored row: one float16 scale, values rounded to the pool's type
                top, rounded = (127.0, []) if c["kv"] == "int8" else (448.0, [])
                for x in new:
                    one = (x.abs().amax(-1, keepdim=True) / top).half().double()
                    y = (x / one).clamp(-top, top)
                    rounded.append((y.round() if c["kv"] == "int8" else y.float().to(torch.float8_e4m3fn).double()) * one)
                new = rounded
        out = torch.zeros_like(q)
        group, lens = c["Hq"] // c["Hkv"], s["lens"].tolist()
        for b, n in enumerate(lens):
            pages = s["table"][b, :-(-n // c["page"])].long()
            at = (pages[:, None] * c["page"] + torch.arange(c["page"], device=pages.device)).reshape(-1)[:n]
            kv = []
            for i, (pool, sc) in enumerate(pools):
                x = pool[at].double()
                if sc is not None:
                    x *= sc[at].double().unsqueeze(-1)
                if new is not None:
                    x[n - 1] = new[i][b]
                kv.append(x)
            for h in range(c["Hkv"]):
                for g in range(h * group, (h + 1) * group):
                    out[b, g] = _attend64(q[b, g], kv[0][:, h], kv[1][:, h], scale, True)[0]
        if c["kind"] == "paged":
            return out
        if c["kv"] in ("int8", "e4m3"):
            return [out, None, None, None, None]
        full = []
        for i, pool in enumerate((s["kp"], s["vp"])):
            x = pool.double()
            x.view(-1, c["Hkv"], D)[s["slots"]] = new[i]
            full.append(x)
        return [out, full[0], full[1], None, None]
    q, k, v = (s[n].detach().double() for n in "qkv")
    do = s["do"].double() if c.get("grad") else None
    mask = None
    if c["kind"] == "sparse":
        rows, cols = 32, 32 if D <= 64 else 16
        cells = s["mask"].bool()

        def mask(i0, i1, j0, j1):
            r, t = torch.arange(i0, i1, device=cells.device) // rows, torch.arange(j0, j1, device=cells.device) // cols
            return cells[r[:, None], t[None, :]]
    spans = [(0, q.shape[2], 0, k.shape[2])]
    if c["kind"] == "varlen":
        cu = s["cu"].tolist()
        spans = [(a, b, a, b) for a, b in zip(cu, cu[1:])]
    out, lse = torch.zeros_like(q), torch.zeros(q.shape[:3], dtype=torch.float64, device=q.device)
    dq, dk, dv = (torch.zeros_like(x) for x in (q, k, v))
    group = q.shape[1] // k.shape[1]
    for b in range(q.shape[0]):
        for h in range(q.shape[1]):
            for i0, i1, j0, j1 in spans:
                r = _attend64(q[b, h, i0:i1], k[b, h // group, j0:j1], v[b, h // group, j0:j1], scale, c["causal"],
                              c.get("window", -1) if c["kind"] == "dense" else -1, c.get("softcap", 0.0), mask,
                              None if do is None else do[b, h, i0:i1])
                out[b, h, i0:i1], lse[b, h, i0:i1] = r[0], r[1]
                if do is not None:
                    dq[b, h, i0:i1] = r[2]
                    dk[b, h // group, j0:j1] += r[3]
                    dv[b, h // group, j0:j1] += r[4]
    if do is not None:
        return [out, dq, dk, dv]
    return (out, lse) if c.get("lse") else out
