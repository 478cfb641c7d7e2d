"""Factors and gradients near the ends of the range of fp32, where a third bf16 part of a value (2**-16 of it) or a product of two factors is not a
normal number, or two of them overflow: the multiplied-out weight and the factor gradients are as exact there as elsewhere.
B200CP_GEMM_TC=2 takes the tensor products at every size.

Bounds: those of test_weight_planes_gpu.py and test_contract_halves_gpu.py, 5e-7 and 1e-6 in the norm."""
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


# scales of x, dy and the factors: a small dense gradient; small factors in one half and the other; a large gradient; factors whose
# product is below every number, and above
GRADIENT = [((1e-18, 1e-18), (1e10, 1e10, 1e10)), ((1e5, 1e5), (1e10, 1e-18, 1e-18)), ((1e5, 1e5), (1e-18, 1e-18, 1e10)), ((1e5, 1e5), (1e-36, 1e10, 1e10)),
            ((1e5, 1e5), (1e10, 1e10, 1e-36)), ((1e17, 1e18), (1e-9, 1e-9, 1e-9)), ((1e15, 1e15), (1.0, 1e-25, 1e-25)), ((1e15, 1e15), (1e-25, 1e-25, 1.0)),
            ((1e-15, 1e-10), (1e-10, 1e22, 1e22)), ((1e-10, 1e-10), (1e22, 1e22, 1e-10))]


@pytest.mark.parametrize("scales, factors", GRADIENT, ids=str)
@pytest.mark.parametrize("idims, odims", [((9, 15, 13), (5, 16, 7)), ((15, 9, 16), (16, 5, 13))], ids=str)
def test_gradients(scales, factors, idims, odims):
    import paralleltnnlayers_b200 as P
    R = 33
    gen = torch.Generator(device="cuda").manual_seed(R)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, dy = normal(70, math.prod(idims)) * scales[0], normal(70, math.prod(odims)) * scales[1]
    F = [normal(i, o, R) * s for i, o, s in zip(idims, odims, factors)]
    G = (x.double().T @ dy.double()).reshape(*idims, *odims)
    V = [f.double() for f in F]
    want = [torch.einsum("ijkabc,jbr,kcr->iar", G, V[1], V[2]), torch.einsum("ijkabc,iar,kcr->jbr", G, V[0], V[2]),
            torch.einsum("ijkabc,iar,jbr->kcr", G, V[0], V[1])]
    for got, w in zip(P.dense_cp_backward(x, dy, *F)[1], want):
        if 1e-37 < float(w.abs().mean()) < 1e36:   # (others are out of range, or below the smallest normal number)
            assert float((got.double() - w).norm() / w.norm()) < 1e-6
    P.device_status()
