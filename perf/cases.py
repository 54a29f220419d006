"""What a program that serves a model over the TQ4 cache has this package do, as timed cases.

``listed()`` names twelve of them, ``draw()`` gives further sizes and options of the same
kinds, ``prepare()`` makes what the program holds before the call, ``run()`` is one pass
through the package's entry points.

Kinds (one attention layer each):
  step    a decode step: the new token of every sequence is compressed into the paged cache,
          then the paged decode runs over all of it (``two_stage``: with the QJL side plane)
  host    the same with the step's inputs and its result in host memory
  spec    a speculative step: the last ``n_q`` tokens of every sequence in one call
  append  a batch of prompt tokens compressed into the paged cache
  prompt  contiguous prefill: keys and values compressed, then causal attention over the codes
  chunk   paged prefill: chunks appended to the cache, then attention over context and chunk
  cache   the contiguous cache behind ``DynamicCache``: one new token and its attention, or a
          prompt that is compressed and read back

Keys and values are N(0,1), four key channels times ten; pages are permuted.
"""

import math
import random

import torch

import flashquant_b200 as fq
from flashquant_b200 import kernels as K
from flashquant_b200.workloads import outlier_channels

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
_BASE = {"hq": 32, "hkv": 8, "d": 128, "block": 16, "dtype": "bf16", "key_bits": 3}


def _case(name, kind, **kw):
    c = {**_BASE, "kind": kind, **kw}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one user at a short context: launches and host time count
        _case("step_1x900", "step", seqs=1, context=900, ragged=False, two_stage=False),
        # the batch of an 8B-shaped layer: 32 sequences of 4096 tokens
        _case("step_32x4096", "step", seqs=32, context=4096, ragged=False, two_stage=False),
        # 70B-shaped long contexts, ragged 32k .. 128k, eight query heads per KV head
        _case("step_long_8x131072", "step", seqs=8, context=131072, ragged=True, two_stage=False,
              hq=64),
        # the same model's layer on one GPU of eight: one KV head, fp16
        _case("step_shard_8x131072", "step", seqs=8, context=131072, ragged=True, two_stage=False,
              hq=8, hkv=1, dtype="fp16"),
        # keys scored with the two-stage estimator
        _case("step_two_stage_16x3000", "step", seqs=16, context=3000, ragged=True, two_stage=True),
        # the scheduler's tensors live on the host
        _case("host_32x2048", "host", seqs=32, context=2048, ragged=True),
        # four tokens a step (speculative decoding)
        _case("spec4_24x2500", "spec", seqs=24, context=2500, ragged=True, n_q=4),
        # a prompt batch goes into the cache, keys two-stage
        _case("append_8192", "append", tokens=8192, slots=65536, two_stage=True),
        # a short prompt, odd length, fp16, the same 16-level table for keys and values
        _case("prompt_1x1000", "prompt", batch=1, length=1000, dtype="fp16", key_bits=4),
        # four long prompts: the largest call
        _case("prompt_4x8192", "prompt", batch=4, length=8192),
        # chunked prefill in a serving batch, every sequence at another point
        _case("chunk_8x512_4096", "chunk", seqs=8, chunk=512, context=4096),
        # one decode step of a contiguous cache, batch of four
        _case("cache_4x4000", "cache", batch=4, context=4000, new=1, key_bits=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "host", "spec", "append", "prompt", "chunk", "cache"],
                       [5, 1, 1, 1, 2, 1, 1])[0]
    c = _case(None, kind, dtype=rng.choice(["bf16", "bf16", "fp16"]))
    if kind in ("step", "host", "spec"):
        c["hq"], c["hkv"] = rng.choice([(32, 8), (32, 8), (64, 8), (8, 1), (16, 2), (16, 4)])
        c["seqs"] = _log(rng, 1, 128)
        most = min(131072, (1 << 19) // c["seqs"])  # 0.6 GB of pages at 8 KV heads
        c["context"] = _log(rng, 20, most)
        c["ragged"] = rng.random() < 0.7
    if kind == "step":
        c["two_stage"] = rng.random() < 0.25
        if not c["two_stage"]:
            c["key_bits"] = rng.choice([3, 3, 4])
            c["block"] = rng.choice([16, 16, 16, 32])
    elif kind == "spec":
        c["n_q"] = rng.choice([2, 3, 4, 5, 8])
        c["context"] = max(c["context"], 2 * c["n_q"])
    elif kind == "append":
        c["hkv"] = rng.choice([8, 8, 4, 1])
        c["tokens"] = _log(rng, 1, 16384)
        c["slots"] = 16 * -(-c["tokens"] * rng.randint(2, 6) // 16)
        c["two_stage"] = rng.random() < 0.5
    elif kind == "prompt":
        c["batch"] = rng.randint(1, 4)
        c["length"] = _log(rng, 20, 8100)
        c["key_bits"] = rng.choice([3, 4])
    elif kind == "chunk":
        c["hq"], c["hkv"] = rng.choice([(32, 8), (64, 8), (16, 4)])
        c["seqs"] = rng.randint(1, 12)
        c["chunk"] = _log(rng, 20, 2048)
        c["context"] = _log(rng, 20, 8192)
    elif kind == "cache":
        c["batch"] = rng.randint(1, 8)
        c["key_bits"] = 4
        c["new"] = 1 if rng.random() < 0.6 else _log(rng, 16, 2048)
        c["context"] = _log(rng, 20, 16384)
    return c


# --------------------------------------------------------------------------------------
# sizes
# --------------------------------------------------------------------------------------
def _lengths(c):
    """Tokens of every sequence, the step's own among them: up to ``context``, ragged ones from
    a quarter of it.  They belong to the case, not to the seed."""
    n, hi = c["seqs"], c["context"]
    r = random.Random(1000003 * n + hi)
    lo = max(2 * c.get("n_q", 1), hi // 4)
    return [r.randint(min(lo, hi), hi) if c["ragged"] else hi for _ in range(n)]


def _chunks(c):
    """(chunk, keys) of every sequence of a chunked prefill: chunks of a quarter of ``chunk``
    upwards behind a context of up to ``context``."""
    r = random.Random(7919 * c["seqs"] + 31 * c["chunk"] + c["context"])
    out = []
    for _ in range(c["seqs"]):
        q = r.randint(max(1, c["chunk"] // 4), c["chunk"])
        out.append((q, q + r.randint(c["context"] // 4, c["context"])))
    return out


def work(case):
    c, d = case, case["d"]
    hq, hkv = c["hq"], c["hkv"]
    row = d // 2 + 4                       # codes and norm of one vector
    rot = 2 * d * d                        # one rotation of one vector
    kind = c["kind"]
    if kind in ("step", "host", "spec"):
        lens, n_q = _lengths(c), c.get("n_q", 1)
        new, total = c["seqs"] * n_q, sum(lens)
        plane = d // 8 + 4 if c.get("two_stage") else 0
        b = total * hkv * (2 * row + plane)             # every cached token once
        b += 2 * new * hq * d * 2                       # q and out
        b += 2 * new * hkv * d * 2 + new * hkv * (2 * row + plane)
        b += 4 * sum(-(-n // c["block"]) for n in lens)
        f = 4 * d * hq * n_q * total * (1.5 if plane else 1)
        f += rot * (2 * new * hq + new * hkv * (4 if plane else 2))
        return {"bytes": b, "flops": f}
    if kind == "append":
        n = c["tokens"] * hkv
        plane = d // 8 + 4 if c["two_stage"] else 0
        return {"bytes": 2 * n * d * 2 + 8 * c["tokens"] + n * (2 * row + plane),
                "flops": n * rot * (4 if plane else 2)}
    if kind == "prompt":
        s, b = c["length"], c["batch"]
        return {"bytes": 2 * b * s * hq * d * 2 + 2 * b * s * hkv * (d * 2 + row),
                "flops": 4 * d * b * hq * (s * (s + 1) // 2) + rot * 2 * b * s * (hq + hkv)}
    if kind == "chunk":
        pairs = _chunks(c)
        new, keys = sum(q for q, _ in pairs), sum(n for _, n in pairs)
        seen = sum(q * (n - q) + q * (q + 1) // 2 for q, n in pairs)
        return {"bytes": 2 * new * hq * d * 2 + 2 * new * hkv * d * 2 + keys * hkv * 2 * row,
                "flops": 4 * d * hq * seen + rot * 2 * new * (hq + hkv)}
    new, b = c["new"], c["batch"]
    if new > 1:                            # compressed and read back
        n = 2 * b * hkv * new
        return {"bytes": n * (d * 2 + row + d * 2), "flops": n * rot * 2}
    keys = c["context"] + 1
    return {"bytes": b * hkv * keys * 2 * row + 2 * b * hq * d * 2 + 2 * b * hkv * d * 2,
            "flops": 4 * d * b * hq * keys + rot * 2 * b * (hq + hkv)}


def tolerance(case):
    """Codes and sign bits next to a decision boundary may fall on either side.  Attention results
    of an fp16 / bf16 path carry two roundings of that type, the tables and weights are fp16."""
    if case["kind"] == "append" or (case["kind"] == "cache" and case["new"] > 1):
        rel = 1e-5 if case["kind"] == "append" else {"bf16": 4e-3, "fp16": 1e-3}[case["dtype"]]
        return {"rel": rel, "differ": 1e-4}
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3}[case["dtype"]], "differ": 1e-4}


# --------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------
_consts = {}


def _constants(c, dev):
    """Rotation, tables and QJL matrix on the device: made once per model."""
    key = (c["d"], c["key_bits"])
    if key not in _consts:
        d = c["d"]
        v = fq.TurboQuantMSE(d, 4, seed=0)
        k = fq.TurboQuantProd(d, c["key_bits"] + 1, seed=0)
        rot_v = fq.haar_orthogonal(d, seed=43)
        _consts[key] = {n: t.contiguous().to(dev) for n, t in dict(
            rot=v.rotation, rot_v=rot_v, bk=k.mse_quantizer.boundaries,
            ck=k.mse_quantizer.centroids, bv=v.boundaries, cv=v.centroids,
            qjl=k.qjl_matrix).items()}
    return _consts[key]


def _randn(g, dev, dtype, *shape):
    return torch.randn(*shape, generator=g, device=dev).to(dtype)


def _kv(g, dev, dtype, *shape):
    k = torch.randn(*shape, generator=g, device=dev)
    k[..., outlier_channels(shape[-1]).to(dev)] *= 10.0
    return k.to(dtype), _randn(g, dev, dtype, *shape)


def _append(c, s, k, v, slots):
    t = s["t"]
    if s["plane"] is None:
        fq.tq4_compress_append(k, v, s["cache"], slots, t["rot"], t["bk"], t["bv"])
    else:
        fq.tq4_compress_append_qjl(k, v, s["cache"], s["plane"], slots, t["rot"], t["bk"],
                                   t["ck"], t["bv"], t["qjl"])


def _rows(c, cache, plane):
    """Codes, norms, sign bits and residual norms of a paged cache, as views of it."""
    h, d = c["hkv"], c["d"]
    a = h * d // 2
    f = cache.view(torch.float32)
    out = {"k_codes": cache[..., :a], "k_norms": f[..., a // 4:a // 4 + h],
           "v_codes": cache[..., a + 4 * h:2 * a + 4 * h], "v_norms": f[..., a // 2 + h:]}
    if plane is not None:
        b = h * d // 8
        out["signs"] = plane[..., :b]
        out["gamma"] = plane.view(torch.float32)[..., b // 4:]
    return out


def _paged(c, g, dev, lens, two_stage):
    """A cache of permuted pages that holds ``lens`` tokens per sequence, and its block table."""
    h, d, bs = c["hkv"], c["d"], c["block"]
    dtype = _DTYPES[c["dtype"]]
    pages = -(-max(lens) // bs)
    n_blocks = pages * len(lens)
    table = torch.randperm(n_blocks, generator=g, device=dev).int().view(len(lens), pages)
    s = {"t": _constants(c, dev), "table": table,
         "lens": torch.tensor(lens, dtype=torch.int32, device=dev),
         "cache": torch.zeros(n_blocks, bs, h * (d + 8), dtype=torch.uint8, device=dev),
         "plane": torch.zeros(n_blocks, bs, h * (d // 8 + 4), dtype=torch.uint8, device=dev)
         if two_stage else None}
    for i, n in enumerate(lens):
        slots = _slots(s, i, 0, n, bs)
        for at in range(0, n, 65536):
            m = min(65536, n - at)
            _append(c, s, *_kv(g, dev, dtype, m, h, d), slots[at:at + m])
    s["rows"] = _rows(c, s["cache"], s["plane"])
    return s


def _slots(s, i, lo, hi, bs):
    at = torch.arange(lo, hi, device=s["table"].device)
    return s["table"][i, at // bs].long() * bs + at % bs


def prepare(case, seed):
    c, kind = case, case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    dtype = _DTYPES[c["dtype"]]
    h, d, hq = c["hkv"], c["d"], c["hq"]

    if kind in ("step", "host", "spec"):
        lens, n_q = _lengths(c), c.get("n_q", 1)
        s = _paged(c, g, dev, lens, c.get("two_stage", False))
        n = c["seqs"]
        k, v = _kv(g, dev, dtype, n * n_q, h, d)
        q = _randn(g, dev, dtype, n, n_q, hq, d)
        slots = torch.cat([_slots(s, i, m - n_q, m, c["block"]) for i, m in enumerate(lens)])
        if kind == "host":
            t = s["t"]
            s["step"] = fq.HostDecodeStep(
                s["cache"], None, t["rot"], t["bk"], t["ck"], t["bv"], t["cv"], None, n, hq, h,
                d, c["block"], s["table"].shape[1], dtype=dtype)
            s["host"] = [x.cpu().pin_memory() for x in
                         (q[:, 0].contiguous(), k, v, slots, s["table"], s["lens"])]
            s["out"] = torch.empty(n, hq, d, dtype=dtype).pin_memory()
        else:
            s.update(k=k, v=v, slots=slots, q=q if kind == "spec" else q[:, 0].contiguous())
        return dict(s, case=c)

    if kind == "append":
        bs = c["block"]
        s = {"t": _constants(c, dev), "case": c,
             "cache": torch.zeros(c["slots"] // bs, bs, h * (d + 8), dtype=torch.uint8, device=dev),
             "plane": torch.zeros(c["slots"] // bs, bs, h * (d // 8 + 4), dtype=torch.uint8,
                                  device=dev) if c["two_stage"] else None}
        s["k"], s["v"] = _kv(g, dev, dtype, c["tokens"], h, d)
        s["slots"] = torch.randperm(c["slots"], generator=g, device=dev)[:c["tokens"]]
        s["rows"] = _rows(c, s["cache"], s["plane"])
        return s

    if kind == "prompt":
        b, n = c["batch"], c["length"]
        k, v = _kv(g, dev, dtype, b, h, n, d)
        t = _constants(c, dev)
        rt = t["rot"].T.contiguous()
        return {"case": c, "t": t, "k": k, "v": v, "q": _randn(g, dev, dtype, b, hq, n, d),
                "even": rt[:, 0::2].contiguous(), "odd": rt[:, 1::2].contiguous()}

    if kind == "chunk":
        pairs = _chunks(c)
        s = _paged(c, g, dev, [n for _, n in pairs], False)
        total = sum(q for q, _ in pairs)
        s["k"], s["v"] = _kv(g, dev, dtype, total, h, d)
        s["q"] = _randn(g, dev, dtype, total, hq, d)
        s["slots"] = torch.cat([_slots(s, i, n - q, n, c["block"])
                                for i, (q, n) in enumerate(pairs)])
        cu = [0]
        for q, _ in pairs:
            cu.append(cu[-1] + q)
        s["cu"] = torch.tensor(cu, dtype=torch.int32, device=dev)
        s["max_q"] = max(q for q, _ in pairs)
        return dict(s, case=c)

    # contiguous cache: keys and values with a rotation each, the tables shared
    b, new, at = c["batch"], c["new"], c["context"]
    cap = at + new + 64
    t = _constants(c, dev)

    def tables(rot):
        rt = rot.T.contiguous()
        return (rt[:, 0::2].contiguous(), rt[:, 1::2].contiguous(), t["bv"], t["cv"], rot)

    s = {"case": c, "tk": tables(t["rot"]), "tv": tables(t["rot_v"]), "at": at}
    for x in ("k", "v"):
        s[x + "_codes"] = torch.zeros(b, h, cap, d // 2, dtype=torch.uint8, device=dev)
        s[x + "_norms"] = torch.zeros(b, h, cap, 1, dtype=torch.float32, device=dev)
    k, v = _kv(g, dev, dtype, b, h, at, d)
    K.cache_update(k, v, s["tk"], s["tv"], s["k_codes"], s["k_norms"], s["v_codes"], s["v_norms"],
                   0)
    s["k"], s["v"] = _kv(g, dev, dtype, b, h, new, d)
    if new > 1:
        s["k_out"] = torch.zeros(b, h, cap, d, dtype=dtype, device=dev)
        s["v_out"] = torch.zeros(b, h, cap, d, dtype=dtype, device=dev)
        s["ws"] = torch.empty(b * h * new * d * 4, dtype=torch.uint8, device=dev)
    else:
        s["q"] = _randn(g, dev, dtype, b, hq, 1, d)
    s["views"] = [s[x][:, :, :at + new] for x in ("k_codes", "k_norms", "v_codes", "v_norms")]
    return s


# --------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    kind, t = c["kind"], state.get("t")
    if kind == "step":
        _append(c, s, s["k"], s["v"], s["slots"])
        geo = (c["hkv"], c["d"], c["block"])
        if s["plane"] is None:
            out = fq.split_k_paged_decode(s["q"], s["cache"], s["table"], s["lens"], t["ck"],
                                          t["cv"], t["rot"], *geo)
        else:
            out = fq.split_k_paged_decode_qjl(s["q"], s["cache"], s["plane"], s["table"],
                                              s["lens"], t["ck"], t["cv"], t["rot"], t["qjl"], *geo)
        return out, s["rows"]
    if kind == "host":
        return s["step"](*s["host"], s["out"]), s["rows"]
    if kind == "spec":
        _append(c, s, s["k"], s["v"], s["slots"])
        out = fq.split_k_paged_decode_multi(s["q"], s["cache"], s["table"], s["lens"], t["ck"],
                                            t["cv"], t["rot"], c["hkv"], c["d"], c["block"])
        return out, s["rows"]
    if kind == "append":
        _append(c, s, s["k"], s["v"], s["slots"])
        return s["rows"]
    if kind == "prompt":
        b, h, n, d = s["k"].shape
        made = []
        for x, bnd in ((s["k"], t["bk"]), (s["v"], t["bv"])):
            codes, norms = fq.tq4_compress(x.view(b * h * n, 1, d), t["rot"], bnd,
                                           rotation_T_even=s["even"], rotation_T_odd=s["odd"])
            made += [codes.view(b, h, n, d // 2), norms.view(b, h, n, 1)]
        return fq.fused_tq_attention(s["q"], *made, t["ck"], t["cv"], t["rot"],
                                     is_causal=True), made
    if kind == "chunk":
        _append(c, s, s["k"], s["v"], s["slots"])
        out = fq.paged_tq4_prefill(s["q"], s["cache"], s["table"], s["lens"], s["cu"], s["max_q"],
                                   t["ck"], t["cv"], t["rot"], c["hkv"], c["d"], c["block"])
        return out, s["rows"]
    K.cache_update(s["k"], s["v"], s["tk"], s["tv"], s["k_codes"], s["k_norms"], s["v_codes"],
                   s["v_norms"], s["at"], s.get("k_out"), s.get("v_out"), s["at"], s.get("ws"))
    if c["new"] > 1:
        return s["views"], s["k_out"], s["v_out"]
    return fq.fused_tq_attention_kv(s["q"], *s["views"], s["tk"][3], s["tv"][3], s["tk"][4],
                                    s["tv"][4]), s["views"]
