"""Factors near the ends of the range of fp32, where a third bf16 part of a value (2**-16 of it) is not a normal number, or values lifted for its sake
overflow: the multiplied-out weight is as exact there as elsewhere.  B200CP_GEMM_TC=2 takes the tensor products at every size.

Bound: that of test_weight_planes_gpu.py, 5e-7 in the norm."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def always(monkeypatch):
    monkeypatch.setenv("B200CP_GEMM_TC", "2")


# scales of the factors and of the input: small and large first modes (half of the weight), small and large others, a large weight
WEIGHT = [((1e-36, 1e15, 1e15), 1.0), ((1e30, 1e-18, 1e-18), 1.0), ((1e35, 1e-15, 1e-15), 1.0), ((1e-30, 1e18, 1e17), 1.0), ((1e11, 1e11, 1e11), 1e-5)]


@pytest.mark.parametrize("scales, scale", WEIGHT, ids=str)
@pytest.mark.parametrize("R", [17, 90])
def test_weight(scales, scale, R):
    import paralleltnnlayers_b200 as P
    idims, odims = (15, 13, 16), (13, 14, 15)
    gen = torch.Generator(device="cuda").manual_seed(R)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    F = [normal(i, o, R) * s for i, o, s in zip(idims, odims, scales)]
    x = normal(19, math.prod(idims)) * scale
    A = F[0].double()
    B = torch.einsum("jbr,kcr->jkbcr", F[1].double(), F[2].double()).reshape(13 * 16, 14 * 15, R)
    y = torch.einsum("nij,iar->njar", x.double().view(19, 15, -1), A)
    want = torch.einsum("njar,jbr->nab", y, B).reshape(19, -1)
    assert float((P.dense_cp(x, *F).double() - want).norm() / want.norm()) < 5e-7
    P.device_status()
