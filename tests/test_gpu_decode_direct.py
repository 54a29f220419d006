"""One query token over a contiguous cache, streamed by warps: lengths around the 16-token tiles and the
slices, one to eight query heads per KV head, byte-permute and look-up keys, buffers with room behind
the last token."""

import math

import pytest
import torch

import flashquant_b200 as fq
from oracle import tq_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def reference(q, rot_k, rot_v, deq):
    """The rotated query rounded to its type, everything else in 64 bits; deq: keys and values in their
    rotated space."""
    b, hq, _, d = q.shape
    hkv = deq[0].shape[1]
    q_rot = (q.double() @ rot_k.double().T).to(q.dtype).double().view(b, hkv, hq // hkv, d)
    s = torch.softmax(q_rot @ deq[0].transpose(-1, -2) / math.sqrt(d), dim=-1)
    return ((s @ deq[1]) @ rot_v.double()).view(b, hq, 1, d)


@pytest.mark.parametrize("hq,hkv", [(1, 1), (6, 2), (8, 2), (16, 2), (32, 8), (64, 64)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 255, 273, 4099])
@pytest.mark.parametrize("k_bits,dtype", [(3, torch.float16), (4, torch.bfloat16)])
def test_one_token(consts, hq, hkv, n, k_bits, dtype):
    if hkv == 64 and n > 1000:
        pytest.skip("more than one wave of CTAs is covered by the short ones")
    b, d, cap = 3, 128, n + (5 if n > 1 else 0)
    rot_k, rot_v = consts["rotation_128_0"], fq.haar_orthogonal(d, seed=43)
    bk, ck = consts[f"boundaries_128_{k_bits}"], consts[f"centroids_128_{k_bits}"]
    bv, cv = consts["boundaries_128_4"], consts["centroids_128_4"]
    g = torch.Generator().manual_seed(100 * n + hq)
    k, v = torch.randn(2, b, hkv, n, d, generator=g)
    k[..., 9] *= 10.0
    q = torch.randn(b, hq, 1, d, generator=g).to(dtype)
    bufs, deq = [], []
    for x, r, bnd, c in ((k, rot_k, bk, ck), (v, rot_v, bv, cv)):
        p, nm = O.compress(x.reshape(-1, 1, d), r, bnd)
        deq.append((c.double()[O.nibble_unpack(p).long()] * nm.reshape(-1, 1, 1).double()).view(b, hkv, n, d))
        codes = torch.full((b, hkv, cap, d // 2), 255, dtype=torch.uint8)
        norms = torch.full((b, hkv, cap, 1), math.nan)  # nothing behind the last token counts
        codes[:, :, :n] = p.view(b, hkv, n, -1)
        norms[:, :, :n] = nm.view(b, hkv, n, 1)
        bufs += [codes.to(DEV)[:, :, :n], norms.to(DEV)[:, :, :n]]
    got = fq.fused_tq_attention_kv(q.to(DEV), *bufs, ck, cv, rot_k, rot_v)
    direct = fq.fused_tq_attention_kv(q.to(DEV), *bufs, *(t.to(DEV) for t in (ck, cv, rot_k, rot_v)))
    assert torch.equal(got, direct)
    ref = reference(q, rot_k, rot_v, deq)
    # one rounding of the result (2^-8 or 2^-11 of an entry; its rms is about half of that) and fp16
    # tables and weights (2^-11 at most)
    rel = ((got.cpu().double() - ref).norm() / ref.norm()).item()
    bound = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}[dtype]
    assert rel <= bound, rel


@pytest.mark.parametrize("b", [32, 33])
def test_rows_around_the_switch(consts, b):
    """1024 query rows, the most that this kernel takes, and 1056, which go through the 128-row tile."""
    d, n, hq, hkv = 128, 100, 32, 8
    rot, bnd, c = (consts[x].to(DEV) for x in ("rotation_128_0", "boundaries_128_4", "centroids_128_4"))
    g = torch.Generator(device=DEV).manual_seed(b)
    bufs, deq = [], []
    for _ in range(2):
        p, nm = fq.tq4_compress(torch.randn(b * hkv * n, 1, d, generator=g, device=DEV), rot, bnd)
        codes = torch.stack((p >> 4, p & 15), -1).flatten(-2).long()
        deq.append((c.double()[codes] * nm.double()).view(b, hkv, n, d))
        bufs += [p.view(b, hkv, n, d // 2), nm.view(b, hkv, n, 1)]
    q = torch.randn(b, hq, 1, d, generator=g, device=DEV).half()
    got = fq.fused_tq_attention_kv(q, *bufs, c, c, rot, rot)
    ref = reference(q, rot, rot, deq)
    assert ((got.double() - ref).norm() / ref.norm()).item() <= 2.0 ** -10


@pytest.mark.parametrize("which", [1, 3])
def test_norm_that_is_not_a_number(consts, which):
    """A NaN key (1) or value (3) norm: rows of other heads and sequences are what they were, a value's
    own rows are NaN (a key's have no denominator and come out as zeros, as in the paged decode)."""
    rot, bnd, c = (consts[x].to(DEV) for x in ("rotation_128_0", "boundaries_128_4", "centroids_128_4"))
    bufs = []
    for i in range(2):
        x = torch.randn(2 * 2 * 200, 1, 128, generator=torch.Generator(device=DEV).manual_seed(i), device=DEV)
        p, nm = fq.tq4_compress(x, rot, bnd)
        bufs += [p.view(2, 2, 200, 64), nm.view(2, 2, 200, 1)]
    q = torch.randn(2, 8, 1, 128, device=DEV).half()
    clean = fq.fused_tq_attention_kv(q, *bufs, c, c, rot, rot)
    bufs[which][1, 0, 77] = float("nan")
    got = fq.fused_tq_attention_kv(q, *bufs, c, c, rot, rot)
    assert which == 1 or bool(got[1, :4].isnan().all())
    assert torch.equal(got[0], clean[0]) and torch.equal(got[1, 4:], clean[1, 4:])
