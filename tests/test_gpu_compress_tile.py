"""The 128-vector tcgen05 compressor at the edges of its tiles and of its range: the smallest calls that
reach it, ragged last tiles, every type, sources aligned to four elements only, cache rows that are
only 4-byte aligned, skipped slots, special vectors."""

import pytest
import torch

import flashquant_b200 as fq
from oracle import tq_oracle as O
from parity import check_codes, check_gamma, check_norms, check_signs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [4737, 4864, 4865, 19071, 37890])
@pytest.mark.parametrize("offset", [0, 4])
def test_compress(consts, dtype, n, offset):
    rot, b4 = consts["rotation_128_0"], consts["boundaries_128_4"]
    flat = torch.randn(n * 128 + offset, generator=torch.Generator().manual_seed(n)).to(dtype)
    x = flat[offset:].view(n, 1, 128)
    x[5] = 0.0
    x[7, 0, 3:] = 0.0
    packed, norms = fq.tq4_compress(flat.to(DEV)[offset:].view(n, 1, 128), rot, b4)
    ref_p, ref_n = O.compress(x.float(), rot, b4)
    check_codes(packed, x.float(), rot, b4, ref_p)
    check_norms(norms, ref_n)


@pytest.mark.parametrize("heads,tokens", [(1, 5000), (3, 1603), (8, 600), (8, 2500)])
@pytest.mark.parametrize("two_stage", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_append(consts, heads, tokens, two_stage, dtype):
    """Against single rows of the same call's values through the oracle; slots < 0 and past the
    cache are left alone."""
    rot, S = consts["rotation_128_0"], consts["qjl_128_0"]
    b3, c3, b4 = consts["boundaries_128_3"], consts["centroids_128_3"], consts["boundaries_128_4"]
    g = torch.Generator().manual_seed(tokens + heads)
    pad = 4 if heads == 3 else 0  # a token stride that is a multiple of four elements only
    wide = torch.randn(2, tokens, heads * 128 + pad, generator=g).to(dtype)
    wide[0, :, 7] *= 10.0
    k, v = (w[:, :heads * 128].unflatten(1, (heads, 128)) for w in wide)
    kd, vd = (w[:, :heads * 128].unflatten(1, (heads, 128)) for w in wide.to(DEV))
    blocks = -(-tokens // 16) + 3
    slots = torch.randperm(blocks * 16, generator=g)[:tokens]
    slots[3], slots[tokens - 1] = -1, blocks * 16
    row, qrow = heads * 136, heads * 20
    cache = torch.full((blocks, 16, row), 0xA5, dtype=torch.uint8, device=DEV)
    plane = torch.full((blocks, 16, qrow), 0xA5, dtype=torch.uint8, device=DEV)
    if two_stage:
        fq.tq4_compress_append_qjl(kd, vd, cache, plane, slots.to(DEV), rot, b3, c3, b4, S)
    else:
        fq.tq4_compress_append(kd, vd, cache, slots.to(DEV), rot, b3, b4)
    keep = (slots >= 0) & (slots < blocks * 16)
    rows = cache.cpu().view(-1, row)
    untouched = torch.ones(blocks * 16, dtype=torch.bool)
    untouched[slots[keep]] = False
    assert bool((rows[untouched] == 0xA5).all())
    rows, k, v = rows[slots[keep]], k[keep].float(), v[keep].float()
    h = heads * 64
    for x, at, b in ((k, 0, b3), (v, h + 4 * heads, b4)):
        ref_p, ref_n = O.compress(x, rot, b)
        check_codes(rows[:, at:at + h].reshape(-1, heads, 64), x, rot, b, ref_p)
        check_norms(rows[:, at + h:at + h + 4 * heads].contiguous().view(torch.float32), ref_n)
    if two_stage:
        idx, _, signs, gamma = O.prod_quantize(k, rot, c3, b3, S)
        q = plane.cpu().view(-1, qrow)
        assert bool((q[untouched] == 0xA5).all())
        q = q[slots[keep]]
        codes = O.nibble_unpack(rows[:, :h].reshape(-1, heads, 64))
        norms = rows[:, h:h + 4 * heads].contiguous().view(torch.float32)
        check_gamma(q[:, heads * 16:].contiguous().view(torch.float32), gamma, k, codes, idx, norms,
                    rot, c3)
        check_signs(q[:, :heads * 16].reshape(-1, heads, 16), signs, k, codes, idx, norms, rot, c3, S)


def test_more_rechecks_than_a_group_notes(consts):
    """Every vector has a coordinate next to a boundary: a call of 262 144 of them overflows the groups' lists,
    and each rechecks all of its vectors.  The same bytes as from a call whose lists hold them."""
    rot, b4 = consts["rotation_128_0"].to(DEV), consts["boundaries_128_4"].to(DEV)
    x = torch.randn(131072, 128, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV).bfloat16()
    y = x.double() / x.double().norm(dim=-1, keepdim=True) @ rot.double().T
    close = ((y.unsqueeze(-1) - b4.double()).abs().amin(dim=(1, 2)) < 0.8 * 2.0 ** -22).nonzero().flatten()
    assert close.numel() >= 64
    x = x[close[:64]].repeat(4096, 1).unsqueeze(1).contiguous()
    packed, norms = fq.tq4_compress(x, rot, b4)
    few = 16384  # the smallest call that sums the squares in the same order
    want_p, want_n = fq.tq4_compress(x[:few].contiguous(), rot, b4)
    assert torch.equal(packed[:few], want_p) and torch.equal(norms[:few], want_n)
    assert torch.equal(packed.view(4096, -1), packed[:64].view(1, -1).expand(4096, -1))
