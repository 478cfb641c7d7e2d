"""Factor gradients of the dense and reshaped-CP layers where some values of the operands are far above or below the others, finite or not:
none, one, tens, thousands of them, up to 29 binades and more apart in a column.  Every value has its own exponent, so all of them
count with their 24 bits.  B200CP_GEMM_TC=2 takes the tensor products at every size.

Bound: as in test_split_gemm_gpu.py, 1e-6 in the norm (2**-24 of a term left out, sums that are cut off by 2e-7, the contraction
with the other factors)."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def always(monkeypatch):
    monkeypatch.setenv("B200CP_GEMM_TC", "2")


def _kron(F):
    M = torch.ones(1, 1, F[0].shape[2], device=F[0].device, dtype=torch.float64)
    for f in F:
        M = torch.einsum("abr,ijr->aibjr", M, f.double()).reshape(M.shape[0] * f.shape[0], M.shape[1] * f.shape[1], -1)
    return M


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


def _spread(t, count, gen, low, high):
    """`count` values far below (even) and far above (odd) the others"""
    at = torch.randperm(t.numel(), generator=gen, device="cuda")[:count]
    f = torch.full((count,), low, device="cuda")
    f[1::2] = high
    t.view(-1)[at] = f * (torch.randn(count, generator=gen, device="cuda") + 3)


DENSE = [(500, (12, 12), (16, 10)), (131, (13, 9), (7, 11)), (65, (16, 16, 5), (4, 13, 5)), (70, (3, 2), (2, 5)), (1, (5, 4), (4, 4))]


@pytest.mark.parametrize("case", DENSE, ids=str)
@pytest.mark.parametrize("few", [0, 1, 10, 64, 65, 3000])
@pytest.mark.parametrize("where", ["input", "gradient", "both"])
def test_dense(case, few, where):
    import paralleltnnlayers_b200 as P
    B, idims, odims = case
    gen = torch.Generator(device="cuda").manual_seed(B + few)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, dy = normal(B, math.prod(idims)), normal(B, math.prod(odims)) * 1e-6
    if where != "gradient":
        _spread(x, min(few, x.numel()), gen, 1e-11, 1e3)
    if where != "input":
        _spread(dy, min(few, dy.numel()), gen, 1e-18, 1e-3)
    F = [normal(i, o, 9) * 0.35 for i, o in zip(idims, odims)]
    leaves = [f.double().requires_grad_() for f in F]
    ref = torch.autograd.grad(x.double() @ _kron(leaves).sum(-1), leaves, dy.double())
    first = P.dense_cp_backward(x, dy, *F)[1]
    for got, want in zip(first, ref):
        assert _rel(got, want) < 1e-6
    for got, again in zip(first, P.dense_cp_backward(x, dy, *F)[1]):   # whatever the order in which the values are found
        assert torch.equal(got, again)
    P.device_status()


RCP = [(3, 10, 12, (12, 12), (16, 10)), (2, 7, 9, (4, 4), (5, 5)), (1, 9, 5, (5, 13), (16, 4))]


@pytest.mark.parametrize("case", RCP, ids=str)
@pytest.mark.parametrize("few", [0, 1, 10, 64, 65, 3000])
@pytest.mark.parametrize("where", ["input", "gradient", "both"])
def test_rcp(case, few, where):
    import paralleltnnlayers_b200 as P
    N, H, W, cd, td = case
    gen = torch.Generator(device="cuda").manual_seed(H + few)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, dy = normal(N, math.prod(cd), H, W), normal(N, math.prod(td), H, W) * 1e-6
    if where != "gradient":
        _spread(x, min(few, x.numel()), gen, 1e-11, 1e3)
    if where != "input":
        _spread(dy, min(few, dy.numel()), gen, 1e-18, 1e-3)
    x[0, 0, 0, 0], dy[-1, -1, -1, -1] = 1e4, 1.0   # corners: taps beside the image
    A, S = [normal(i, o, 9) * 0.3 for i, o in zip(cd, td)], normal(3, 3, 9) * 0.3
    leaves = [t.double().requires_grad_() for t in (*A, S)]
    K = torch.einsum("ctr,yxr->tcyx", _kron(leaves[:2]), leaves[2])
    y = torch.nn.functional.conv2d(x.double().cpu(), K.cpu(), padding=1)
    ref = torch.autograd.grad(y, leaves, dy.double().cpu())
    _, dA, dS = P.rcp_conv2d_backward(x, dy, *A, S)
    for got, want in zip((*dA, dS), ref):
        assert _rel(got, want) < 1e-6
    P.device_status()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("count", [1, 80])
def test_values_that_are_not_finite(value, count):
    """They reach the gradients of their own column and no other."""
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(3)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, dy = normal(200, 144), normal(200, 160)
    F = [normal(i, o, 9) * 0.35 for i, o in ((12, 16), (12, 10))]
    leaves = [f.double().requires_grad_() for f in F]
    ref = torch.autograd.grad(x.double() @ _kron(leaves).sum(-1), leaves, dy.double())
    x[:count, 5 * 12 + 7] = value
    dF = P.dense_cp_backward(x, dy, *F)[1]
    for f, want, i in zip(dF, ref, (5, 7)):
        keep = [k for k in range(12) if k != i]
        assert not bool(torch.isfinite(f[i]).any())
        assert _rel(f[keep], want[keep]) < 1e-6
    A, S = [normal(8, 8, 9) * 0.3 for _ in range(2)], normal(3, 3, 9) * 0.3
    u, dv = normal(2, 64, 9, 11), normal(2, 64, 9, 11)
    u[0, 3 * 8 + 2, 0, 0] = value   # a corner: the taps beside the image do not meet it
    _, dA, dS = P.rcp_conv2d_backward(u, dv, *A, S)
    assert not bool(torch.isfinite(dA[0][3]).any()) and bool(torch.isfinite(dA[0][4:]).all())
    met = torch.isfinite(dS).all(-1)
    assert not bool(met[:2, :2].any()) and bool(met[2].all()) and bool(met[:, 2].all())
    P.device_status()


def test_whole_numbers_stay_exact():
    """Nothing is cut off where all sums are short: gradients by order-1 factors of rank 1, which are sums of whole numbers."""
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(1)
    integers = lambda *s: torch.randint(-9, 10, s, generator=gen, device="cuda").float()
    x, dy = integers(300, 16), integers(300, 16)
    dF = P.dense_cp_backward(x, dy, integers(16, 16, 1))[1][0]
    assert torch.equal(dF[:, :, 0].double(), x.double().T @ dy.double())
