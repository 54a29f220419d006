"""A vector's bytes do not depend on how many vectors a call carries: calls that take the kernel for a few
vectors, the 16-row kernel and the 128-vector kernel store the same codes, norms and sign bits (a coordinate
next to a boundary is decided by one arithmetic in all of them), in both forms of the rotation."""

import pytest
import torch

import flashquant_b200 as fq
from flashquant_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def vectors(n, d, dtype, seed):
    x = torch.randn(n, d, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)
    x[:, [9, d // 2, d - 3]] *= torch.tensor([1.0, 10.0], device=DEV).repeat(n)[:n, None]
    x[5] = 0.0
    return x.to(dtype)


def in_calls_of(size, x, call):
    return [torch.cat(t) for t in zip(*(call(x[i:i + size]) for i in range(0, len(x), size)))]


# few | 16-vector tiles | 128-vector tiles
SIZES = [(128, 1184, 2300), (128, 4700, 16300), (64, 1184, 16000)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("d,small,large", SIZES)
def test_codes_and_norms(consts, d, small, large, dtype):
    """Some 25 million codes per type, a dozen of which two arithmetics would put on
    different sides."""
    rot, b4 = consts[f"rotation_{d}_0"].to(DEV), consts[f"boundaries_{d}_4"].to(DEV)
    rt = rot.T.contiguous()
    split = dict(rotation_T_even=rt[:, 0::2].contiguous(), rotation_T_odd=rt[:, 1::2].contiguous())
    for seed in range(4):
        x = vectors(48000, d, dtype, seed).unsqueeze(1)
        a, b = (in_calls_of(n, x, lambda y: fq.tq4_compress(y, rot, b4, **split)) for n in (small, large))
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d,small,large", SIZES)
def test_two_stage(consts, d, small, large, dtype):
    """Codes, norms and signs of the two-stage quantiser.  Two sums of a reconstructed coordinate differ by
    up to 2^-24 |x|, so the residual by 2^-20.5 |x|, and gamma is about 0.18 |x|: 2^-18 of it."""
    rot, s = consts[f"rotation_{d}_0"].to(DEV), consts[f"qjl_{d}_0"].to(DEV)
    b3, c3 = consts[f"boundaries_{d}_3"].to(DEV), consts[f"centroids_{d}_3"].to(DEV)
    for seed in range(4):
        x = vectors(48000, d, dtype, 10 + seed)
        a, b = (in_calls_of(n, x, lambda y: K.tq_prod_quantize(y, rot, b3, c3, s)) for n in (small, large))
        for i in range(3):
            assert torch.equal(a[i], b[i]), i
        assert bool(((a[3] - b[3]).abs() <= 2.0 ** -18 * b[3]).all())
