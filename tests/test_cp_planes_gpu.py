"""CP4 and three-factor CP convolutions over whole rank planes, against the float64 oracle.

Sizes at the edges of the products' tiles (16 / 32 / 64 rows, 64 / 128 pixels, 16 channels or ranks and 32 pixels per
stage): rows, ranks and channels one above and below them, pixel counts that are no multiple of 4 (unaligned rows) and
that straddle images, images of one row or column, one image, splits over a cluster and none, ranks above one tile.
Bound: the one of the other parity tests, 1e-4 relative + 1e-5 of the largest value."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import test_planes_rule as planes_rule
from gpu_util import check
from oracle import cp_oracle as O

# N, C, T, H, W, R
SHAPES = [
    (1, 3, 5, 1, 1, 65), (2, 17, 15, 5, 7, 66), (3, 16, 33, 1, 9, 67), (1, 64, 64, 12, 1, 129), (5, 70, 65, 7, 7, 64),
    (2, 255, 257, 8, 8, 33), (64, 256, 256, 7, 7, 17), (3, 300, 212, 6, 6, 32), (1, 512, 64, 9, 9, 16),
    (4, 500, 12, 5, 13, 3), (2, 12, 500, 11, 6, 5), (33, 64, 64, 23, 23, 40), (1, 4, 4, 64, 64, 128),
    (12, 64, 70, 28, 28, 40),   # only the backward over planes, from the plane another kernel wrote
    (2, 291, 301, 5, 5, 64), (1, 300, 303, 6, 5, 63),   # four gradient entries per thread in the last sum: full blocks, and a ragged end
]


def assert_parity(got, ref):
    check(got, ref, "cp planes", rtol=1e-4, atol=1e-5 * float(np.abs(ref).max()))


def make(shape, cp3):
    N, C, T, H, W, R = shape
    rng = np.random.default_rng(sum(shape))
    X = rng.uniform(-1, 1, (N, C, H, W)).astype(np.float32)
    dU = rng.standard_normal((N, T, H, W)).astype(np.float32)
    dims = [(T, R), (C, R)] + ([(3, 3, R)] if cp3 else [(3, R), (3, R)])
    K = [(rng.standard_normal(d) * (9 * C) ** -0.5).astype(np.float32) for d in dims]
    return X, dU, K


def expect(X, dU, K):
    """Forward, data gradient and factor gradients by float64 autograd of the recomposed convolution."""
    x = torch.tensor(X, dtype=torch.float64, requires_grad=True)
    k = [torch.tensor(f, dtype=torch.float64, requires_grad=True) for f in K]
    w = torch.einsum("tr,cr,yxr->tcyx", *k) if len(k) == 3 else torch.einsum("tr,cr,yr,xr->tcyx", *k)
    u = torch.nn.functional.conv2d(x, w, padding=1)
    g = torch.autograd.grad(u, [x] + k, torch.tensor(dU, dtype=torch.float64))
    return [t.detach().numpy() for t in (u, *g)]


def offset(a):
    """The array on the GPU, contiguous but not 16-byte aligned."""
    buf = torch.empty(a.size + 1, device="cuda")
    t = buf[1:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
def test_cp4(shape, aligned):
    import paralleltnnlayers_b200 as P
    X, dU, K = make(shape, False)
    want = expect(X, dU, K)
    assert np.allclose(want[0], O.cp4_forward(X, *K, 1), rtol=1e-9, atol=1e-9)
    put = (lambda a: torch.from_numpy(a).cuda()) if aligned else offset
    x, du, k = put(X), put(dU), [put(f) for f in K]
    assert_parity(P.cp4_conv2d_forward(x, *k), want[0])
    assert_parity(P.cp4_conv2d_backward_data(du, *k), want[1])
    for got, ref in zip(P.cp4_conv2d_backward_filter(du, x, *k), want[2:]):
        assert_parity(got, ref)
    U, dX, dK = P.cp4_conv2d_step(x, du, *k)
    assert_parity(U, want[0])
    assert_parity(dX, want[1])
    o = 0
    for ref in want[2:]:
        assert_parity(dK[o:o + ref.size].view(ref.shape), ref)
        o += ref.size
    # the layer's node: forward with its plane kept, and the backward from it
    leaves = [t.clone().requires_grad_() for t in (x, *k)]
    y = P.CP4Conv2dFunction.apply(*leaves)
    for got, ref in zip((y, *torch.autograd.grad(y, leaves, du)), want):
        assert_parity(got, ref)


# Shapes near the lines between the kernels, whichever of them the rules choose (test_planes_rule.py says which).
LINES = [
    (45, 96, 144, 14, 14, 32), (44, 96, 144, 14, 14, 32), (45, 96, 145, 14, 14, 32), (45, 95, 142, 14, 14, 32), (46, 96, 96, 20, 16, 17),
    (1, 8, 8, 4, 4, 17), (1, 8, 8, 4, 4, 16), (2, 64, 64, 8, 12, 8), (1, 100, 60, 12, 12, 9), (1, 144, 136, 6, 24, 12), (1, 136, 136, 6, 24, 12),
    (1, 40, 25, 9, 9, 33), (1, 40, 24, 8, 8, 33), (1, 17, 16, 9, 9, 40),
    (11, 40, 40, 21, 22, 18), (10, 40, 40, 21, 22, 18), (11, 40, 41, 21, 22, 18), (11, 40, 40, 21, 24, 18),
]


LINES += sorted({s for _, *both in planes_rule.LINES for s in both if s[0] * s[3] * s[4] * (s[1] + s[2]) < 2e6 and s not in LINES})


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("shape", LINES, ids=str)
def test_lines_between_the_kernels(shape, aligned):
    test_cp4(shape, aligned)


@pytest.mark.parametrize("shape", [s for s in SHAPES if s[5] <= 66])
def test_cp3(shape):
    import paralleltnnlayers_b200 as P
    X, dU, K = make(shape, True)
    want = expect(X, dU, K)
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
    assert_parity(P.cp3_conv2d_forward(x, *k), want[0])
    assert_parity(P.cp3_conv2d_backward_data(du, *k), want[1])
    for got, ref in zip(P.cp3_conv2d_backward_filter(du, x, *k), want[2:]):
        assert_parity(got, ref)
    leaves = [t.clone().requires_grad_() for t in (x, *k)]
    y = P.CP3Conv2dFunction.apply(*leaves)
    for got, ref in zip((y, *torch.autograd.grad(y, leaves, du)), want):
        assert_parity(got, ref)


# Of the tensor-core kernels: tiles of 128 pixels, of 128 channels and 32 or 64 ranks (gradients) and of up to 256 rows (products),
# chunks of 64 terms, sums over clusters of 2, 4 and 8 CTAs (some without a chunk), more pixel tiles than resident CTAs.
TC_SHAPES = SHAPES + [
    (3, 1, 127, 9, 9, 17), (2, 127, 129, 8, 9, 33), (1, 128, 1, 11, 12, 64), (2, 129, 128, 7, 9, 65), (1, 130, 63, 16, 8, 31),
    (1, 320, 320, 9, 9, 40), (1, 600, 130, 9, 9, 35), (1, 140, 200, 20, 20, 100), (1, 1030, 70, 5, 5, 200),
    (16, 65, 33, 49, 51, 33), (10, 33, 130, 63, 61, 17), (64, 5, 6, 28, 22, 70),
]


@pytest.fixture
def form(request):
    from paralleltnnlayers_b200._lib import lib
    lib.b200cp_test_set_planes(2, request.param)
    yield request.param
    lib.b200cp_test_set_planes(-1, -1)


@pytest.mark.parametrize("form", [0, 2], indirect=True, ids=["ffma", "tensor"])
@pytest.mark.parametrize("shape", TC_SHAPES, ids=str)
def test_both_forms(form, shape):
    """Every call over planes, in either arithmetic, whatever the rule would take.  Bound: six products of three bf16 parts leave out
    2**-23 of a term at most, an accumulator of 64 terms is cut off by at most 4 * 2**-23 of its partial sums; the rank plane, the
    stencil and the sum over ranks or pixels follow one another.  In the norm, with random signs, below 4e-7 (measured over drawn
    shapes: 2.4e-7, FFMA 6.5e-7)."""
    import paralleltnnlayers_b200 as P
    X, dU, K = make(shape, False)
    want = expect(X, dU, K)
    x, du, k = offset(X), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]

    def close(got, refs):
        for i, (g, r) in enumerate(zip(got, refs)):
            err = np.linalg.norm(g.detach().double().cpu().numpy() - r) / np.linalg.norm(r)
            assert err < 1e-6, (i, err)

    U, dX, dK = P.cp4_conv2d_step(x, du, *k)
    grads = [g.view(r.shape) for g, r in zip(torch.split(dK.flatten(), [w.size for w in want[2:]]), want[2:])]
    close((U, dX, *grads), want)
    close((P.cp4_conv2d_forward(x, *k), P.cp4_conv2d_backward_data(du, *k), *P.cp4_conv2d_backward_filter(du, x, *k)), want)
    X, dU, K = make(shape, True)
    want = expect(X, dU, K)
    leaves = [torch.from_numpy(a).cuda().requires_grad_() for a in (X, *K)]
    y = P.CP3Conv2dFunction.apply(*leaves)
    close((y, *torch.autograd.grad(y, leaves, torch.from_numpy(dU).cuda())), want)
    P.device_status()


@pytest.mark.parametrize("form", [0, 2], indirect=True, ids=["ffma", "tensor"])
@pytest.mark.parametrize("R", [24, 40])
def test_images_keep_their_own_scale(form, R):
    """An image is as accurate beside any other.  NaN and infinities stay with the pixels that a
    tap reaches."""
    import paralleltnnlayers_b200 as P
    X, dU, K = make((4, 70, 65, 9, 10, R), False)
    scale = np.array([1e-25, 1.0, 1e25, 1e-8], np.float32)[:, None, None, None]
    want = expect(X * scale, dU * scale[::-1], K)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    x, du, k = put(X * scale), put(dU * scale[::-1]), [put(f) for f in K]
    U, dX, _ = P.cp4_conv2d_step(x, du, *k)
    for got, ref in ((U, want[0]), (dX, want[1])):
        for n in range(4):
            assert np.linalg.norm(got[n].double().cpu().numpy() - ref[n]) < 1e-6 * np.linalg.norm(ref[n])
    x[1, 5, 2, 3], x[2, 6, 4, 8] = float("nan"), float("inf")
    hit = torch.zeros(4, 9, 10, dtype=torch.bool, device="cuda")
    hit[1, 1:4, 2:5] = hit[2, 3:6, 7:10] = True
    V = P.cp4_conv2d_forward(x, *k)
    assert not bool(torch.isfinite(V.movedim(1, -1)[hit]).any())
    assert torch.equal(V.movedim(1, -1)[~hit], P.cp4_conv2d_forward(put(X * scale), *k).movedim(1, -1)[~hit])
    P.device_status()


@pytest.mark.parametrize("form", [0, 2], indirect=True, ids=["ffma", "tensor"])
@pytest.mark.parametrize("R", [24, 40])
@pytest.mark.parametrize("where", ["ranks", "channels"])
def test_ranks_and_channels_of_any_scale(form, R, where):
    """The scale of a rank is free to move between the factor matrices, and a channel of any size may have no weight."""
    import paralleltnnlayers_b200 as P
    X, dU, K = make((3, 70, 65, 5, 9, R), False)
    want = expect(X, dU, K)[:2]
    if where == "ranks":
        powers = 2.0 ** np.linspace(-40, 40, R).round()
        K[0], K[1] = (K[0] * powers).astype(np.float32), (K[1] / powers).astype(np.float32)
    else:
        X[:, 3], K[1][3], dU[:, 4], K[0][4] = 1e12, 0, 1e12, 0
        want = expect(X, dU, K)[:2]
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
    for got, ref in zip(P.cp4_conv2d_step(x, du, *k), want):
        assert np.linalg.norm(got.double().cpu().numpy() - ref) < 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("form", [0, 2], indirect=True, ids=["ffma", "tensor"])
@pytest.mark.parametrize("R", [24, 40])
@pytest.mark.parametrize("where", ["input", "gradient"])
def test_factor_gradients_beside_a_large_sample(form, R, where):
    """An image whose gradient (or input) is zero adds nothing to the factor gradients, however large its input (gradient) is."""
    import paralleltnnlayers_b200 as P
    X, dU, K = make((6, 70, 65, 5, 9, R), False)
    big, none = (X, dU) if where == "input" else (dU, X)
    big[1] *= 1e9
    big[4, 3] *= 1e15
    none[[1, 4]] = 0
    want = expect(X, dU, K)[2:]
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
    dK = P.cp4_conv2d_step(x, du, *k)[2].flatten()
    for got, ref in zip(torch.split(dK, [w.size for w in want]), want):
        assert np.linalg.norm(got.view(ref.shape).double().cpu().numpy() - ref) < 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("form", [0, 2], indirect=True, ids=["ffma", "tensor"])
@pytest.mark.parametrize("shape", [(3, 70, 65, 5, 9, 24), (2, 20, 130, 8, 8, 40), (1, 600, 130, 9, 9, 35), (16, 65, 33, 49, 51, 33)], ids=str)
@pytest.mark.parametrize("where, value", [("input", "inf"), ("gradient", "-inf"), ("factor", "inf")])
def test_infinities(form, shape, where, value):
    """An infinite value gives what fp32 arithmetic gives: infinities of its sign, with factors of one sign, and nothing elsewhere."""
    import paralleltnnlayers_b200 as P
    X, dU, K = [[np.abs(a) for a in v] if isinstance(v, list) else np.abs(v) for v in make(shape, False)]
    N, C, T, H, W, R = shape
    at = {"input": X[N - 1, C - 2], "gradient": dU[N - 1, T - 1], "factor": K[1]}[where]
    at[H // 2, W - 3 if where != "factor" else R - 2] = float(value)
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
    # (over rank planes too: with the factors multiplied out, the padding's zeros would meet infinite weights)
    ref = [torch.tensor(a, dtype=torch.float64, requires_grad=True) for a in (X, *K)]
    taps = torch.einsum("yr,xr->ryx", *ref[3:])[:, None]
    Z = torch.nn.functional.conv2d(torch.einsum("cr,nchw->nrhw", ref[2], ref[0]), taps, padding=1, groups=R)
    y = torch.einsum("tr,nrhw->nthw", ref[1], Z)
    want = [g.detach().numpy() for g in (y, *torch.autograd.grad(y, ref, torch.tensor(dU, dtype=torch.float64)))]
    U, dX, dK = P.cp4_conv2d_step(x, du, *k)
    dK = [g.view(r.shape) for g, r in zip(torch.split(dK.flatten(), [w.size for w in want[2:]]), want[2:])]
    many = 0
    for got, ref in zip((U, dX, *dK), want):
        got, fin = got.cpu().double().numpy(), np.isfinite(ref)
        assert not np.isnan(ref).any()
        assert np.array_equal(got[~fin], ref[~fin])
        assert np.abs(got[fin] - ref[fin]).max(initial=0) <= 1e-5 * np.abs(ref[fin]).max(initial=0)
        many += (~fin).sum()
    assert many
    P.device_status()


def test_more_than_7168_channels():
    """The sum over the channels on the tensor cores ends at 7168 channels (ranks); the products take more, on FFMA, in the same
    launches."""
    import paralleltnnlayers_b200 as P
    from paralleltnnlayers_b200._lib import lib
    launches = []
    for C in (7168, 8200):
        X, dU, K = make((1, C, 24, 7, 7, 65), False)
        x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
        before = lib.b200cp_launch_count()
        U, dX, dK = P.cp4_conv2d_step(x, du, *k)
        launches.append(lib.b200cp_launch_count() - before)
        want = expect(X, dU, K)
        assert_parity(U, want[0])
        assert_parity(dX, want[1])
        for got, ref in zip(torch.split(dK.flatten(), [w.size for w in want[2:]]), want[2:]):
            assert_parity(got.view(ref.shape), ref)
    assert launches[0] == launches[1]


def test_streams_and_capture():
    """Two streams at once, and a captured step: the workspace belongs to the call, nothing is shared."""
    import paralleltnnlayers_b200 as P
    X, dU, K = make((4, 96, 40, 9, 9, 70), False)
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
    ref = [t.clone() for t in P.cp4_conv2d_step(x, du, *k)]
    streams, outs = [torch.cuda.Stream(), torch.cuda.Stream()], []
    torch.cuda.synchronize()
    for i in range(6):
        with torch.cuda.stream(streams[i % 2]):
            outs.append(P.cp4_conv2d_step(x, du, *k))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs.append(P.cp4_conv2d_step(x, du, *k))
    graph.replay()
    torch.cuda.synchronize()
    for o in outs:
        for a, b in zip(o, ref):
            assert torch.equal(a, b)   # fixed summation order


@pytest.mark.parametrize("shape", [(4, 96, 40, 9, 9, 70), (8, 64, 64, 14, 14, 8)])   # rank planes; row kernels and their reduction
def test_back_to_back_calls_on_new_inputs(shape):
    """Calls that follow one another without a wait reuse the same scratch: each kernel reads what the one before it wrote
    in this call, not what an earlier call left at the address.  Same bits as with a wait after every call."""
    import paralleltnnlayers_b200 as P
    sets = []
    for i in range(8):
        X, dU, K = make(shape, False)
        rng = np.random.default_rng(i)
        sets.append([torch.from_numpy(np.ascontiguousarray(a * rng.uniform(0.5, 2, a.shape).astype(np.float32))).cuda()
                     for a in (X, dU, *K)])
    alone = []
    for s in sets:
        alone.append([t.clone() for t in P.cp4_conv2d_step(*s)])
        torch.cuda.synchronize()
    for _ in range(5):
        for got, want in zip([P.cp4_conv2d_step(*s) for s in sets], alone):
            for a, b in zip(got, want):
                assert torch.equal(a, b)


def test_cp3_backward_forms_what_is_asked_for():
    """A layer whose input needs no gradient forms the factor gradients only, one product (launch) less; one asked for the
    input's gradient alone runs the data gradient's launches and no others."""
    import paralleltnnlayers_b200 as P
    from paralleltnnlayers_b200._lib import lib
    X, dU, K = make((3, 70, 65, 9, 9, 40), True)
    want = expect(X, dU, K)
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda().requires_grad_() for f in K]

    def launched(run):
        before = lib.b200cp_launch_count()
        out = run()
        return lib.b200cp_launch_count() - before, out

    def backward(x, *leaves):
        y = P.CP3Conv2dFunction.apply(x, *k)
        return launched(lambda: torch.autograd.grad(y, leaves, du))

    xr = x.clone().requires_grad_()
    n_all, g_all = backward(xr, xr, *k)
    n_factors, g_factors = backward(x, *k)
    n_data, g_data = backward(xr, xr)
    for grads, refs in ((g_all, want[1:]), (g_factors, want[2:]), (g_data, want[1:2])):
        for got, ref in zip(grads, refs):
            assert_parity(got, ref)
    assert n_factors == n_all - 1
    with torch.no_grad():
        assert n_data == launched(lambda: P.cp3_conv2d_backward_data(du, *k))[0]


# Which kernels form the factor gradients alone: the tile kernels (two launches per 64 ranks) where their tiles fill the SMs
# once or the channels are few, the plane products (four launches) elsewhere; the times stand beside the rule.
@pytest.mark.parametrize("shape, cp3, launches", [
    ((16, 16, 16, 27, 27, 64), False, 2), ((16, 16, 16, 27, 27, 64), True, 2), ((32, 16, 16, 28, 28, 50), False, 2),
    ((64, 8, 8, 7, 7, 64), True, 2), ((32, 64, 64, 28, 28, 32), True, 2), ((16, 64, 64, 27, 27, 24), True, 2),
    ((32, 24, 24, 28, 28, 64), False, 4), ((8, 256, 256, 14, 14, 33), False, 4), ((4, 96, 96, 28, 28, 32), True, 4),
])
def test_filter_rule(shape, cp3, launches):
    import paralleltnnlayers_b200 as P
    from paralleltnnlayers_b200._lib import lib
    X, dU, K = make(shape, cp3)
    x, du, k = torch.from_numpy(X).cuda(), torch.from_numpy(dU).cuda(), [torch.from_numpy(f).cuda() for f in K]
    before = lib.b200cp_launch_count()
    grads = (P.cp3_conv2d_backward_filter if cp3 else P.cp4_conv2d_backward_filter)(du, x, *k)
    assert lib.b200cp_launch_count() - before == launches
    for got, ref in zip(grads, expect(X, dU, K)[2:]):
        assert_parity(got, ref)


@pytest.mark.parametrize("shape, shared", [((16, 64, 64, 27, 27, 32), False), ((16, 16, 16, 27, 27, 64), False), ((64, 8, 8, 7, 7, 50), False),
                                           ((32, 64, 64, 56, 56, 32), True), ((64, 16, 16, 32, 32, 50), True),
                                           ((64, 512, 512, 7, 7, 16), True)])
def test_cp3_shared_plane_rule(shape, shared):
    from paralleltnnlayers_b200._lib import TensorShape, lib
    import ctypes as C
    N, Cc, T, H, W, R = shape
    s = TensorShape(N=N, H=H, W=W, pad=1, T=T, C=Cc, Y=3, X=3, Rank=R)
    assert bool(lib.b200cp_cp3_shares_planes(C.byref(s), 0)) is shared
