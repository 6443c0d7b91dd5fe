"""Performance cases: the work a user of this package has it do, over the ranges it is used at.

A case names an operation and its sizes.  `prepare` makes what a program holds before the call, `run` is one pass
through the package's public functions, `work` counts what a pass cannot do without.  Operations:

  step      attention forward and backward (training) over dense [B,H,S,D] tensors, optionally causal, with grouped
            heads, or with key padding lengths per batch entry
  prefill   attention forward alone: S new queries against L >= S keys (a prompt, or a chunk of one behind a cache)
  packed    forward and backward over a packed batch of sequences of different lengths
  decode    one query per sequence against a dense cache
  paged     one query per sequence against a paged cache with ragged lengths
  fc        fully connected layer, forward and backward
  softmax   row softmax, forward and backward
"""
import importlib
import math
import random

import torch

tt = importlib.import_module("pku-aiprogramming_b200")

BF16, F32 = "bf16", "f32"
_DTYPE = {BF16: torch.bfloat16, F32: torch.float32}


def listed():
    return [
        # the reference check: the smallest call, all launches and host work
        dict(name="step_f32_check", op="step", dtype=F32, B=2, H=4, Hkv=4, S=64, L=64, D=32, causal=False, lens=0),
        # training in the reference's own element type
        dict(name="step_f32", op="step", dtype=F32, B=2, H=8, Hkv=8, S=2048, L=2048, D=64, causal=True, lens=0),
        # a batch of ordinary prompts at head dim 64
        dict(name="prefill_d64", op="prefill", dtype=BF16, B=8, H=16, Hkv=16, S=1024, L=1024, D=64, causal=True, lens=0),
        # one chunk of a long prompt behind what the cache holds already; grouped heads, sizes off every tile edge
        dict(name="prefill_chunk", op="prefill", dtype=BF16, B=1, H=32, Hkv=8, S=777, L=5001, D=128, causal=True, lens=0),
        # the training step the forward target is stated on
        dict(name="step_4k", op="step", dtype=BF16, B=4, H=32, Hkv=32, S=4096, L=4096, D=128, causal=True, lens=0),
        # long-sequence training, the largest case
        dict(name="step_32k", op="step", dtype=BF16, B=1, H=64, Hkv=64, S=32768, L=32768, D=128, causal=True, lens=0),
        # training on sequences of different lengths without padding
        dict(name="step_packed", op="packed", n_seq=16, shortest=300, longest=4096, lens=7, H=32, Hkv=32, D=128, causal=True),
        # serving: a full batch with long caches, bound by the cache's bytes
        dict(name="decode_batch", op="decode", dtype=BF16, B=64, H=32, Hkv=32, L=8192, D=128),
        # serving: one sequence, grouped heads, a cache length between two powers of two; bound by latency
        dict(name="decode_single", op="decode", dtype=BF16, B=1, H=32, Hkv=8, L=5001, D=128),
        # serving: pages of 64 rows, grouped heads, every sequence at a length of its own
        dict(name="decode_paged", op="paged", B=32, H=32, Hkv=8, D=128, page=64, shortest=17, longest=8192, lens=11),
        # a layer of a large model
        dict(name="fc_large", op="fc", dtype=BF16, rows=16384, fin=4096, fout=4096),
        # rows of scores
        dict(name="softmax_rows", op="softmax", dtype=F32, rows=262144, cols=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A length: every other one as drawn, the rest at a multiple of 64."""
    n = _log_int(rng, lo, hi)
    return n if rng.random() < 0.5 else max(lo, n // 64 * 64)


def _heads(rng):
    hkv = rng.choice([1, 2, 4, 8, 16, 32])
    group = rng.choice([1, 1, 2, 4, 8])
    return min(64, hkv * group), hkv


def draw(rng):
    op = rng.choice(["step", "step", "prefill", "packed", "decode", "decode", "paged", "fc", "softmax"])
    dtype = rng.choice([BF16, BF16, BF16, F32])
    D = rng.choice([64, 128])
    H, Hkv = _heads(rng)
    if op in ("step", "prefill"):
        if dtype == F32:
            D = rng.choice([32, 64, 128])
        S = _length(rng, 64, 2048 if dtype == F32 else 32768)
        L = S
        if op == "prefill" and rng.random() < 0.5:
            L = S + _log_int(rng, 1, 16384)
        B = _log_int(rng, 1, 16)
        causal = rng.random() < 0.7
        # at most a tenth of the longest listed step (float32: of what takes that long)
        most = 5e10 if dtype == F32 else 5e12
        while B > 1 and 14.0 * B * H * S * L * D > most:
            B -= 1
        while H > Hkv and 14.0 * B * H * S * L * D > most:
            H -= Hkv
        while Hkv > 1 and 14.0 * B * H * S * L * D > most:
            H, Hkv = H // Hkv, 1
        if 14.0 * B * H * S * L * D > most:
            S = L = int(math.sqrt(most / (14.0 * B * H * D)))
        lens = rng.randrange(1, 1 << 16) if B > 1 and not causal and rng.random() < 0.5 else 0
        return dict(op=op, dtype=dtype, B=B, H=H, Hkv=Hkv, S=S, L=L, D=D, causal=causal, lens=lens)
    if op == "packed":
        longest = _log_int(rng, 128, 4096)
        shortest = max(1, longest // rng.randrange(2, 17))
        return dict(op=op, n_seq=_log_int(rng, 2, 32), shortest=shortest, longest=longest, lens=rng.randrange(1, 1 << 16),
                    H=H, Hkv=Hkv, D=D, causal=rng.random() < 0.8)
    if op == "decode":
        B, L = _log_int(rng, 1, 64), _length(rng, 128, 32768)
        while B > 1 and 4.0 * B * Hkv * L * D > 4e9:
            B //= 2
        return dict(op=op, dtype=BF16, B=B, H=H, Hkv=Hkv, L=L, D=D)
    if op == "paged":
        B, longest = _log_int(rng, 1, 64), _log_int(rng, 128, 16384)
        while B > 1 and 4.0 * B * Hkv * longest * D > 4e9:
            B //= 2
        return dict(op=op, B=B, H=H, Hkv=Hkv, D=D, page=rng.choice([16, 32, 64, 128]), shortest=1, longest=longest,
                    lens=rng.randrange(1, 1 << 16))
    if op == "fc":
        rows, fin, fout = _log_int(rng, 32, 16384), _log_int(rng, 64, 8192), _log_int(rng, 10, 8192)
        if dtype == BF16 or rng.random() < 0.5:   # feature counts of real layers
            fin, fout = max(8, fin // 8 * 8), max(8, fout // 8 * 8)
        while dtype == F32 and 6.0 * rows * fin * fout > 3e11:
            rows, fin, fout = max(32, rows // 2), max(64, fin // 16 * 8), max(8, fout // 16 * 8)
        return dict(op=op, dtype=dtype, rows=rows, fin=fin, fout=fout)
    cols = _log_int(rng, 10, 65536)
    rows = _log_int(rng, 32, max(64, min(262144, (1 << 28) // cols)))
    return dict(op=op, dtype=rng.choice([BF16, F32]), rows=rows, cols=cols)


def _lengths(c, n):
    """The n lengths of a packed, paged or padded case: part of the case, not of its data."""
    rng = random.Random(c["lens"])
    return [rng.randint(c["shortest"], c["longest"]) for _ in range(n)]


def _kv_lens(c):
    rng = random.Random(c["lens"])
    return [rng.randint(max(1, c["L"] // 4), c["L"]) for _ in range(c["B"])]


def prepare(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    op = c["op"]
    dt = _DTYPE[c.get("dtype", BF16)]

    def normal(shape, sigma=1.0):
        x = torch.randn(shape, generator=g, device="cuda", dtype=dt)
        return x if sigma == 1.0 else x.mul_(sigma)

    def ints(v):
        return torch.tensor(v, dtype=torch.int32, device="cuda")

    s = {"case": c}
    if op in ("step", "prefill"):
        B, H, Hkv, S, L, D = (c[k] for k in ("B", "H", "Hkv", "S", "L", "D"))
        # scores of a trained layer: a few units wide, so that neither one key nor all of them take the weight
        s.update(q=normal((B, H, S, D), 0.5), k=normal((B, Hkv, L, D), 0.5), v=normal((B, Hkv, L, D), 0.5))
        if op == "step":
            s["dout"] = normal((B, H, S, D))
        s["kv_lens"] = ints(_kv_lens(c)) if c["lens"] else None
    elif op == "packed":
        lens = _lengths(c, c["n_seq"])
        total, H, Hkv, D = sum(lens), c["H"], c["Hkv"], c["D"]
        s.update(q=normal((total, H, D), 0.5), k=normal((total, Hkv, D), 0.5), v=normal((total, Hkv, D), 0.5),
                 dout=normal((total, H, D)), cu=ints([sum(lens[:i]) for i in range(len(lens) + 1)]), longest=max(lens))
    elif op == "decode":
        B, H, Hkv, L, D = (c[k] for k in ("B", "H", "Hkv", "L", "D"))
        s.update(q=normal((B, H, 1, D)), k=normal((B, Hkv, L, D)), v=normal((B, Hkv, L, D)))
    elif op == "paged":
        B, H, Hkv, D, page = (c[k] for k in ("B", "H", "Hkv", "D", "page"))
        lens = _lengths(c, B)
        per = [(n + page - 1) // page for n in lens]
        order = torch.randperm(sum(per), generator=g, device="cuda").to(torch.int32)   # pages as a pool hands them out
        table = torch.zeros((B, (c["longest"] + page - 1) // page), dtype=torch.int32, device="cuda")
        at = 0
        for b, n in enumerate(per):
            table[b, :n] = order[at:at + n]
            at += n
        pool = (sum(per), Hkv, page, D)
        s.update(q=normal((B, H, 1, D)), k=normal(pool), v=normal(pool), table=table, lens=ints(lens))
    elif op == "fc":
        rows, fin, fout = c["rows"], c["fin"], c["fout"]
        s.update(x=normal((rows, fin)), w=normal((fin, fout), fin ** -0.5), bias=normal((fout,)), dy=normal((rows, fout)))
    else:
        s.update(x=normal((c["rows"], c["cols"]), 3.0), dy=normal((c["rows"], c["cols"])))
    return s


def run(s):
    c = s["case"]
    op = c["op"]
    if op in ("step", "prefill"):
        q, k, v, causal, lens = s["q"], s["k"], s["v"], c["causal"], s["kv_lens"]
        out, lse = tt.attention_forward(q, k, v, causal=causal, kv_lens=lens)
        if op == "prefill":
            return out, lse
        dq, dk, dv = tt.attention_backward(q, k, v, out, lse, s["dout"], causal=causal, kv_lens=lens)
        return out, lse, dq, dk, dv
    if op == "packed":
        q, k, v, cu, n, causal = s["q"], s["k"], s["v"], s["cu"], s["longest"], c["causal"]
        out, lse = tt.attention_forward_varlen(q, k, v, cu, cu, n, n, causal=causal)
        dq, dk, dv = tt.attention_backward_varlen(q, k, v, cu, cu, n, n, out, lse, s["dout"], causal=causal)
        return out, lse, dq, dk, dv
    if op == "decode":
        return tt.attention_decode(s["q"], s["k"], s["v"])
    if op == "paged":
        return tt.attention_decode_paged(s["q"], s["k"], s["v"], block_table=s["table"], seq_lens=s["lens"])
    if op == "fc":
        y = tt.fc_forward(s["x"], s["w"], s["bias"])
        return (y,) + tuple(tt.fc_backward(s["x"], s["w"], s["dy"]))
    y = tt.softmax_forward(s["x"])
    return y, tt.softmax_backward(y, s["dy"])


def work(c):
    """Bytes: every input read once, every output written once.  Operations: two per multiply-add of the products over
    the key/query pairs that the mask and the lengths leave (forward two products, backward five)."""
    op = c["op"]
    size = 4 if c.get("dtype", BF16) == F32 else 2

    def pairs(S, L):
        return S * L - S * (S - 1) // 2 if c["causal"] else S * L

    if op in ("step", "prefill"):
        B, H, Hkv, S, L, D = (c[k] for k in ("B", "H", "Hkv", "S", "L", "D"))
        n = sum(pairs(S, x) for x in _kv_lens(c)) if c["lens"] else B * pairs(S, L)
        kept = sum(_kv_lens(c)) if c["lens"] else B * L
        rows, keys = B * H * S, Hkv * D * size
        if op == "prefill":
            return {"bytes": rows * (2 * D * size + 4) + 2 * kept * keys, "flops": 4.0 * H * n * D}
        return {"bytes": rows * (4 * D * size + 4) + 2 * (kept + B * L) * keys, "flops": 14.0 * H * n * D}
    if op == "packed":
        lens, H, Hkv, D = _lengths(c, c["n_seq"]), c["H"], c["Hkv"], c["D"]
        return {"bytes": sum(lens) * (H * (4 * D * size + 4) + 4 * Hkv * D * size),
                "flops": 14.0 * H * D * sum(pairs(n, n) for n in lens)}
    if op in ("decode", "paged"):
        B, H, Hkv, D = (c[k] for k in ("B", "H", "Hkv", "D"))
        keys = B * c["L"] if op == "decode" else sum(_lengths(c, B))
        return {"bytes": 2 * keys * Hkv * D * size + B * H * (2 * D * size + 4), "flops": 4.0 * keys * H * D}
    if op == "fc":
        rows, fin, fout = c["rows"], c["fin"], c["fout"]
        return {"bytes": size * (2 * rows * (fin + fout) + 2 * fin * fout + 2 * fout), "flops": 6.0 * rows * fin * fout}
    n = c["rows"] * c["cols"]
    return {"bytes": size * 4 * n, "flops": 8.0 * n}


def tolerance(c):
    return {"rel": 1e-2} if c.get("dtype", BF16) == BF16 else {"rel": 1e-5}
