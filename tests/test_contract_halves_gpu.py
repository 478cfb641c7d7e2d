"""Factor gradients from a large dense gradient, the modes in two halves on the tensor cores: halves off the 128 and 64 entries of a tile,
ranks off its 32, four-byte and 16-byte loads (the inputs of the last half a multiple of 4 or not), one or two modes per half, the taps
as a mode; and an infinite gradient, whose sums are formed anew in fp32.  B200CP_GEMM_TC=2 takes the tensor products at every size.

Bound: 1e-6 in the norm, as in test_gradient_window_gpu.py (three bf16 parts leave out 2**-24 of a term, sums of at most 128 terms are cut off by
2**-24 of a partial sum per instruction of 16)."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DENSE = [((5, 4, 7, 5), (4, 3, 5, 8), 1), ((4, 4, 4, 4), (5, 5, 6, 5), 33), ((4, 8, 3, 4), (9, 5, 8, 3), 70), ((15, 9, 7), (16, 5, 13), 31),
         ((16, 10, 6), (12, 12, 4), 65), ((3, 16, 16), (5, 16, 16), 32), ((2, 3, 16, 16), (2, 2, 16, 16), 5)]
RCP = [((16, 9), (16, 5), 16), ((13, 12), (9, 8), 40), ((3, 7, 5), (5, 4, 8), 33), ((4, 4, 4), (3, 16, 2), 7)]


@pytest.fixture(autouse=True)
def always(monkeypatch):
    monkeypatch.setenv("B200CP_GEMM_TC", "2")


def _vectors(F):   # every factor as [pairs][R]
    return [f.double().reshape(-1, f.shape[2]) for f in F]


def _gradients(G, V):
    """d vec_q[p][r] = sum over the other modes of G times their vectors, G by [pairs of each mode]"""
    out = []
    for q in range(len(V)):
        rows = []
        for r in range(V[0].shape[1]):
            t = G
            for k in reversed(range(len(V))):
                if k != q:
                    t = torch.tensordot(t, V[k][:, r], dims=([k], [0]))
            rows.append(t)
        out.append(torch.stack(rows, -1))
    return out


def _by_pairs(G, ins, outs):   # [.., T][C] -> [.., c0 t0, c1 t1, ..]
    m = len(ins)
    lead = G.dim() - 2
    G = G.reshape(*G.shape[:lead], *outs, *ins)
    order = list(range(lead)) + [d for k in range(m) for d in (lead + m + k, lead + k)]
    return G.permute(order).reshape(*G.shape[:lead], *[c * t for c, t in zip(ins, outs)])


def _check(got, want, shapes):
    for g, w, s in zip(got, want, shapes):
        g, w = g.double(), w.reshape(s)
        finite = w.isfinite()
        assert not g[~finite].isfinite().any()
        assert float((g - w)[finite].norm() / w[finite].norm()) < 1e-6


@pytest.mark.parametrize("infinite", [False, True])
@pytest.mark.parametrize("idims, odims, R", DENSE, ids=str)
def test_dense(idims, odims, R, infinite):
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(R)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, dy = normal(70, math.prod(idims)), normal(70, math.prod(odims))
    F = [normal(i, o, R) * 0.35 for i, o in zip(idims, odims)]
    if infinite:
        x[3, 7] = float("inf")
    got = P.dense_cp_backward(x, dy, *F)[1]
    want = _gradients(_by_pairs(dy.double().T @ x.double(), idims, odims), _vectors(F))
    _check(got, want, [f.shape for f in F])
    assert all(g.isfinite().any() for g in got)
    P.device_status()


@pytest.mark.parametrize("idims, odims, R", RCP, ids=str)
def test_rcp(idims, odims, R):
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(R)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    C, T = math.prod(idims), math.prod(odims)
    x, dy = normal(2, C, 9, 7), normal(2, T, 9, 7)
    F, S = [normal(i, o, R) * 0.3 for i, o in zip(idims, odims)], normal(3, 3, R) * 0.3
    _, dF, dS = P.rcp_conv2d_backward(x, dy, *F, S)
    G = torch.nn.grad.conv2d_weight(x.double(), (T, C, 3, 3), dy.double(), padding=1).permute(2, 3, 0, 1).reshape(9, T, C)
    want = _gradients(_by_pairs(G, idims, odims), [S.double().reshape(9, R)] + _vectors(F))
    _check([dS, *dF], want, [S.shape, *[f.shape for f in F]])
    P.device_status()


@pytest.mark.parametrize("idims, odims, R", [((15, 9, 7), (16, 5, 13), 31), ((16, 16, 16), (4, 8, 4), 32), ((8, 4, 4, 4), (4, 8, 4, 4), 20)], ids=str)
def test_sums_of_one_sign(idims, odims, R):
    """What the tensor core cuts off has one sign.  A dense gradient of whole numbers (one sample, exact) and positive factors: a unit of fp32, 2**-23 in the
    norm, half of it for what is rounded (the product of two vectors, sums of tiles and of parts), half for what is cut off."""
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(R)
    whole = lambda n: torch.randint(1, 2048, (1, n), generator=gen, device="cuda").float()
    x, dy = whole(math.prod(idims)), whole(math.prod(odims))
    F = [torch.rand(i, o, R, generator=gen, device="cuda") + 0.01 for i, o in zip(idims, odims)]
    got = P.dense_cp_backward(x, dy, *F)[1]
    want = _gradients(_by_pairs(dy.double().T @ x.double(), idims, odims), _vectors(F))
    for g, w in zip(got, want):
        w = w.reshape(g.shape)
        assert float((g.double() - w).norm() / w.norm()) < 2 ** -23


def _kernels(call):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return " ".join(e.key for e in p.key_averages())


def test_mode(monkeypatch):
    """B200CP_GEMM_TC=0 keeps the contraction off the tensor cores at any size, 2 takes it there at any."""
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(0)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    large = [normal(i, o, 5) for i, o in zip((15, 13, 16), (13, 14, 15))]
    x, dy = normal(3, 15 * 13 * 16), normal(3, 13 * 14 * 15)
    small = [normal(i, o, 7) for i, o in zip(*RCP[-1][:2])]
    S, u, dv = normal(3, 3, 7), normal(2, 64, 6, 5), normal(2, 96, 6, 5)
    calls = [lambda: P.dense_cp_backward(x, dy, *large)[1], lambda: P.rcp_conv2d_backward(u, dv, *small, S)[1]]
    for call in calls:
        out = {}
        for mode, here, other in (("2", "halves_kernel", "peel_"), ("0", "peel_", "halves_")):
            monkeypatch.setenv("B200CP_GEMM_TC", mode)
            out[mode] = call()
            names = _kernels(call)
            assert here in names and other not in names
        for a, b in zip(out["0"], out["2"]):
            assert float((a - b).norm() / b.norm()) < 1e-6
