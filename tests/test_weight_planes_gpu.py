"""The multiplied-out weight written as operand planes: the exponents of its rows from a table of the factors' slices, up to
64 of 256 ranks, at row counts off the 32 of a block and ranks off the 16 of an
instruction and the 64 of a stage, one or two modes in a half, rows in runs of any length.  B200CP_GEMM_TC=2 takes the tensor
product at every size.

Bound: 5e-7 in the norm, as in test_split_gemm_gpu.py; a row's exponent that is too small would overflow its fp16 values, one that is too
large loses a bit of the 22 per binade."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = [((15, 13, 16), (13, 14, 15), 9), ((6, 7, 5, 9), (8, 7, 9, 7), 1), ((16, 16, 16, 2), (8, 4, 9, 16), 33),
         ((15, 13, 16), (13, 14, 15), 250), ((16, 16, 16, 16), (4, 4, 4, 4), 256)]   # the last: 64 KB in one direction


@pytest.mark.parametrize("idims, odims, R", CASES, ids=str)
@pytest.mark.parametrize("turned", [False, True])
def test_weight_planes(idims, odims, R, turned, monkeypatch):
    import paralleltnnlayers_b200 as P
    monkeypatch.setenv("B200CP_GEMM_TC", "2")
    if turned:
        idims, odims = odims, idims
    gen = torch.Generator(device="cuda").manual_seed(R)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = normal(19, math.prod(idims))
    # (a scale per output slice: rows of the weight, each with its exponent, far apart)
    F = [normal(i, o, R) * torch.exp2(torch.randint(-9, 9, (o, 1), generator=gen, device="cuda").float()) for i, o in zip(idims, odims)]
    W = torch.zeros(math.prod(idims), math.prod(odims), device="cuda", dtype=torch.float64)
    for r in range(R):
        y = torch.eye(W.shape[0], device="cuda", dtype=torch.float64).view(-1, *idims)
        for f in F:   # the first mode goes, its outputs come last
            y = torch.tensordot(y, f[:, :, r].double(), dims=([1], [0]))
        W += y.reshape(W.shape)
    ref = x.double() @ W
    off = P.dense_cp(x, *F).double() - ref
    assert float(off.norm() / ref.norm()) < 5e-7
    # an output against its row of the weight (the output itself may be a small difference): no row is worse than four times the mean
    assert float((off.norm(dim=0) / W.norm(dim=0)).max()) < 19 ** 0.5 * 2e-6
    P.device_status()


@pytest.mark.parametrize("turned", [False, True])
def test_rows_off_the_grid(turned, monkeypatch):
    """Runs of 84 neighbours (eight bytes of a plane at a time) and of 63 (a row at a time), the last tile of a half not full."""
    test_weight_planes((9, 7, 7, 12), (8, 7, 9, 7), 21, turned, monkeypatch)
