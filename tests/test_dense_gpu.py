"""The 1x1x1 product with its epilogue against float64 on the same rounded inputs.

Bound: products are exact in fp32, their sum of c_in terms errs by at most c_in 2^-23 of the sum of
magnitudes, the epilogue by a few units in the last place of fp32, the result is rounded once
(2^-11 relative for fp16, 2^-8 for bf16)."""
import pytest
import torch

from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 80_001])
@pytest.mark.parametrize("c_in,c_out", [(8, 8), (32, 20), (16, 6), (72, 24), (64, 32), (256, 128), (40, 256)])
@pytest.mark.parametrize("dtype,unit", [(torch.float16, 2.0 ** -11), (torch.bfloat16, 2.0 ** -8)])
def test_dense_rows(rows, c_in, c_out, dtype, unit):
    gen = torch.Generator(device=DEV).manual_seed(rows + c_in + c_out)
    rand = lambda *s: torch.randn(*s, generator=gen, device=DEV)
    x, w, res = rand(rows, c_in).to(dtype), rand(c_in, c_out).to(dtype), rand(rows, c_out).to(dtype)
    scale, shift = rand(c_out), rand(c_out)
    want = x.double() @ w.double()
    size = x.double().abs() @ w.double().abs()
    for full in (False, True):
        ref, mag = want, size
        if full:
            ref = (want * scale.double() + shift.double() + res.double()).clamp_min(0)
            mag = size * scale.double().abs() + shift.double().abs() + res.double().abs()
        got = F.dense_forward(x, w, *((scale, shift, res, True) if full else ())).double()
        bound = unit * ref.abs() + (c_in + 4) * 2.0 ** -23 * mag + 2.0 ** -25
        assert bool(((got - ref).abs() <= bound * 1.01).all())
