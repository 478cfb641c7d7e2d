"""Filter gradients of the reshaped-CP layer on the tensor cores where pixels at the edges of an image are not finite: the taps that reach
beside the image meet zeros, not them, and stay finite.  In tiles with all of K and in tiles that are cut; images, the gradient and both.
B200CP_GEMM_TC=2 takes the tensor products at every size.

Bound: 1e-6 of the sum of the magnitudes, as in test_split_gemm_gpu.py; the entries formed anew are fp32 sums over the lanes of a warp."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _weight_gradient(x, dv, F):   # [tap][t][c], over the pixels inside the image only
    H, W, p = x.shape[2], x.shape[3], F // 2
    inside = lambda n, s: slice(max(0, s), max(0, n + min(0, s)))
    taps = [(y, z) for y in range(-p, p + 1) for z in range(-p, p + 1)]
    return torch.stack([torch.einsum("nthw,nchw->tc", dv[:, :, inside(H, -y), inside(W, -z)], x[:, :, inside(H, y), inside(W, z)])
                        for y, z in taps])


# 8 steps of K in tiles cut in two; 2 steps, whole tiles; more tiles than pairs of SMs (25 taps x 3 rows of tiles); many images; a filter
# that reaches beyond the image
@pytest.mark.parametrize("N, cdims, tdims, H, W, F", [(2, (16,), (12,), 9, 11, 3), (1, (16,), (12,), 5, 6, 3), (3, (13, 16, 3), (10, 11, 2), 6, 5, 5),
                                                     (70, (9,), (16,), 7, 7, 3), (2, (16,), (8,), 2, 3, 7)])
@pytest.mark.parametrize("where", ["images", "gradient", "both"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_edges(N, cdims, tdims, H, W, F, where, value, monkeypatch):
    import paralleltnnlayers_b200 as P
    monkeypatch.setenv("B200CP_GEMM_TC", "2")
    gen = torch.Generator(device="cuda").manual_seed(N + F)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    C, T = math.prod(cdims), math.prod(tdims)
    x, dv = normal(N, C, H, W), normal(N, T, H, W)
    if where != "gradient":
        x[0, 3, 0, 0], x[-1, 5, 0, W - 1] = value, -value
    if where != "images":
        dv[0, 2, H - 1, W - 1], dv[-1, T - 1, H - 1, 0] = value, value
    want = _weight_gradient(x.double(), dv.double(), F)
    size = _weight_gradient(x.double().abs(), dv.double().abs(), F)
    # rank 1 and ones: the gradient of S is the sum of the weight's over t and c
    ones = [torch.ones(c, t, 1, device="cuda") for c, t in zip(cdims, tdims)]
    _, dA, dS = P.rcp_conv2d_backward(x, dv, *ones, torch.ones(F, F, 1, device="cuda"))
    got, ref, scale = dS.reshape(-1).double(), want.sum((1, 2)), size.sum((1, 2))
    met = torch.isfinite(want).all(-1).all(-1)
    assert 0 < int(met.sum()) < F * F
    assert bool((torch.isfinite(got) == met).all())
    assert bool(((got - ref)[met].abs() <= 1e-6 * scale[met]).all())
    if len(cdims) == 1:   # and that of the factor the sum over the taps
        got, ref, scale = dA[0][:, :, 0].double(), want.sum(0).T, size.sum(0).T
        met = torch.isfinite(want).all(0).T
        assert bool((torch.isfinite(got) == met).all())
        assert bool(((got - ref)[met].abs() <= 1e-6 * scale[met]).all())
    P.device_status()
