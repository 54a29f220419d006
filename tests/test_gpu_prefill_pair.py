"""The two-tile attention kernel at the edges of its tiles: 128 keys a tile, value halves of 64 in a
ring of three, 128 or 256 query rows a CTA (even / odd query heads per KV head), and the three
sources of key values (byte permutes, the values' own table, a table of their own)."""

import pytest
import torch

from test_gpu_prefill import check, make_case, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv", [(2, 1), (3, 1), (4, 4), (6, 2)])
@pytest.mark.parametrize("n", [2, 63, 65, 127, 128, 129, 257, 385, 520])
def test_tile_edges(consts, hq, hkv, n):
    case = make_case(consts, 1, hq, hkv, n, seed=40 + n + hq)
    check(run_gpu(case, is_causal=n != 385), case, is_causal=n != 385)


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
