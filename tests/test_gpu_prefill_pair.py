"""The two-tile attention kernel at the edges of its tiles: 64 keys a tile, operand rings of three, 128 or
256 query rows a CTA (even / odd query heads per KV head), contiguous and paged, the sources of key
values (byte permutes, look-ups), and norms that are not finite."""

import pytest
import torch

from flashquant_b200 import kernels as K
from test_gpu_paged_prefill import build, run_and_check
from test_gpu_prefill import DEV, check, make_case, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv", [(2, 1), (3, 1), (4, 4), (6, 2)])
@pytest.mark.parametrize("n", [2, 63, 65, 127, 128, 129, 257, 385, 520])
def test_tile_edges(consts, hq, hkv, n):
    case = make_case(consts, 1, hq, hkv, n, seed=40 + n + hq)
    out = run_gpu(case, is_causal=n != 385)
    check(out, case, is_causal=n != 385)
    on_device = K.fused_tq_attention(*(t.to(DEV) for t in case), is_causal=n != 385)
    assert torch.equal(on_device, out)


@pytest.mark.parametrize("k_bits,scale", [(2, 1.0), (3, 1.0), (4, 1.0), (4, 1.07)])
def test_key_tables(consts, k_bits, scale):
    case = list(make_case(consts, 1, 4, 2, 300, seed=60 + k_bits, dtype=torch.float16, k_bits=k_bits))
    case[5] = case[5] * scale  # 16 levels that are not the values': a table of their own
    check(run_gpu(tuple(case), is_causal=True), tuple(case), is_causal=True)


def test_weights_keep_their_range(consts):
    """Value norms over three orders of magnitude and keys that raise the reference exponent late:
    the accumulator in TMEM is rescaled and no fp16 weight overflows or vanishes."""
    case = list(make_case(consts, 1, 4, 2, 400, seed=77))
    case[4] = case[4] * torch.logspace(-3, 0, 400).reshape(1, 1, 400, 1)
    case[2] = case[2] * torch.linspace(0.1, 3.0, 400).reshape(1, 1, 400, 1)
    check(run_gpu(tuple(case), is_causal=True), tuple(case), is_causal=True)


@pytest.mark.parametrize("chunks", [[300, 200], [256, 257], [129, 1]])
def test_paged_odd_groups(consts, chunks):
    """Three query heads per KV head: a CTA's two tiles are 256 consecutive rows of one head."""
    w, cache, q, cu = build(consts, [300, 460], chunks, hq=12, hkv=4, cfg=44)
    run_and_check(consts, w, cache, q, cu, chunks)


@pytest.mark.parametrize("hq", [4, 6])
@pytest.mark.parametrize("which", [2, 4])
def test_norm_that_is_not_a_number(consts, hq, which):
    """A NaN key (2) or value (4) norm: the rows that see the token are NaN, those of other heads and of
    earlier tokens are what they were."""
    case = list(make_case(consts, 1, hq, 2, 300, seed=91))
    clean = run_gpu(tuple(case), is_causal=True)
    case[which] = case[which].clone()
    case[which][0, 1, 150] = float("nan")
    out = run_gpu(tuple(case), is_causal=True)
    first = hq // 2  # query heads of KV head 1
    assert torch.equal(out[:, :first], clean[:, :first])
    assert torch.equal(out[:, first:, :150], clean[:, first:, :150])
    assert bool(out[:, first:, 150:].isnan().all())
