"""The activations of a feed-forward as a launch of their own, against float64: rows in whole pieces (few rows, where a block has 256 threads; many, where it has as many as a row has pieces),
rows off their pieces, rows of a wider matrix."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, F64 = torch.device("cuda:0"), torch.float64
FORMS = {
    "silu": (None, lambda g, u: g * torch.sigmoid(g) * u),
    "clamped": ((1, 1.702, 2.0), lambda g, u: g.clamp(max=2.0) * torch.sigmoid(1.702 * g.clamp(max=2.0)) * (u.clamp(-2.0, 2.0) + 1)),
    "relu2": ((2, 0.0, 0.0), lambda g, u: g.clamp(min=0.0) ** 2),
    "gelu_erf": ((3, 0.0, 0.0), lambda g, u: torch.nn.functional.gelu(g)),
    "gelu_tanh": ((4, 0.0, 0.0), lambda g, u: torch.nn.functional.gelu(g, approximate="tanh") * u),
}


@pytest.mark.parametrize("name", FORMS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,ff,gap", [(1, 8, 0), (3, 1000, 0), (2367, 264, 8), (2368, 264, 0), (2368, 8, 0), (2369, 2056, 16), (2400, 36, 0), (5, 33, 3)])
def test_activation(name, dtype, rows, ff, gap):
    from promptcache_b200 import _native_seq as nsq
    act, want = FORMS[name]
    wide = torch.randn(rows, 2 * ff + gap, generator=torch.Generator().manual_seed(rows + ff)).mul(2).to(dtype).to(DEV)
    gu = wide[:, :2 * ff]
    got = nsq.glu_mul(gu, ff, act).to(F64)
    g, u = gu[:, :ff].to(F64), gu[:, ff:].to(F64)
    # the result's rounding; a handful of 32-bit operations on numbers of the input's size (differences of 1 in tanh and erf)
    assert bool(((got - want(g, u)).abs() <= want(g, u).abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) + 2.0 ** -22 * g.abs() * (1 + u.abs())).all())
