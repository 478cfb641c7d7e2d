"""The tensor-core products of the dense and reshaped-CP layers (scaled fp16 hi / lo operands, in the gradients three bf16 parts) at the
edges of their tiles: 256 x 256 / 128 / 64 results, K steps of 64 (gradients: 32) in instructions of 16, odd row lengths, operands off the 16-byte grid, rows of very
different magnitude.  B200CP_GEMM_TC=2 takes them at every size.

Bound: a product of two 22-bit operands without the product of their low parts is off by at most 2**-21; an accumulator of
n <= 4 instructions is cut off by at most n * 2**-23 of its partial sums, and the totals round by 2**-24 each.  In the norm over a
result, with random signs, that is 2.5e-7 (measured: 1.0 to 2.5e-7); the weight's own fp32 sum adds 1e-7.  The six products of
three bf16 parts leave out 3 * 2**-24 of a term."""
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
REL = 5e-7


@pytest.fixture(autouse=True)
def always(monkeypatch):
    monkeypatch.setenv("B200CP_GEMM_TC", "2")


def _normal(seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=gen, device="cuda")


def _kron(F):
    M = torch.ones(1, 1, F[0].shape[2], device="cuda", dtype=torch.float64)
    for f in F:
        M = torch.einsum("abr,ijr->aibjr", M, f.double()).reshape(M.shape[0] * f.shape[0], M.shape[1] * f.shape[1], -1)
    return M


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


DENSE = [(1, (4, 4), (2, 4)), (63, (3, 5), (3, 3)), (65, (16, 4), (16, 4)), (130, (5, 13), (11, 12)), (257, (16, 8), (16, 16)),
         (300, (16, 12), (16, 9)), (77, (16, 16), (16, 16)), (700, (7, 9), (16, 16)), (40, (16, 16), (13, 7)),
         (33, (13,), (9,)), (50, (4, 3, 5), (5, 4, 3)), (129, (4, 5, 3, 2), (2, 3, 4, 5)), (66, (16, 9), (12, 12)),
         (21, (15, 13, 16), (13, 14, 15)), (22, (6, 7, 5, 9), (8, 7, 9, 7))]   # the last two: the weight written as operand planes


@pytest.mark.parametrize("case", DENSE, ids=str)
@pytest.mark.parametrize("offset", [0, 1])   # floats off the 16-byte grid
def test_dense(case, offset):
    import paralleltnnlayers_b200 as P
    B, idims, odims = case
    normal = _normal(B + offset)
    I, O = math.prod(idims), math.prod(odims)
    x, dy = normal(B * I + offset)[offset:].view(B, I), normal(B * O + offset)[offset:].view(B, O)
    R = {21: 33, 33: 33, 50: 64, 66: 300}.get(B, 9)   # the weight is formed 32 ranks at a time
    F = [normal(i, o, R) * 0.35 for i, o in zip(idims, odims)]
    M = _kron(F).sum(-1)
    n0 = P.launch_count()
    assert _rel(P.dense_cp(x, *F), x.double() @ M) < REL
    assert P.launch_count() - n0 >= 3   # weight, operand planes, product
    dx, dF = P.dense_cp_backward(x, dy, *F)
    assert _rel(dx, dy.double() @ M.T) < REL
    leaves = [f.double().requires_grad_() for f in F]
    ref = torch.autograd.grad(x.double() @ _kron(leaves).sum(-1), leaves, dy.double())
    for got, want in zip(dF, ref):
        assert _rel(got, want) < 1e-6   # and the contraction with the other factors, in fp32
    P.device_status()


RCP = [(1, 3, 5, (3, 3), (4, 3)), (2, 7, 9, (4, 4), (5, 5)), (3, 8, 8, (5, 13), (16, 4)), (1, 16, 17, (16, 8), (13, 10)),
       (5, 9, 4, (16, 12), (16, 16)), (2, 5, 6, (7,), (10,)), (2, 6, 5, (3, 4, 2), (2, 5, 3)), (1, 9, 9, (2, 3, 2, 3), (4, 2, 3, 2))]


@pytest.mark.parametrize("case", RCP, ids=str)
def test_rcp(case):
    import paralleltnnlayers_b200 as P
    N, H, W, cd, td = case
    normal = _normal(H * W)
    C, T, R = math.prod(cd), math.prod(td), 9
    x, dy = normal(N, C, H, W), normal(N, T, H, W)
    A, S = [normal(c, t, R) * 0.3 for c, t in zip(cd, td)], normal(3, 3, R) * 0.3

    def forward(x, A, S):
        K = torch.einsum("ctr,yxr->tcyx", _kron(A), S.double())
        return torch.nn.functional.conv2d(x.cpu(), K.cpu(), padding=1)

    leaves = [t.double().requires_grad_() for t in (x, *A, S)]
    y = forward(leaves[0], leaves[1:-1], leaves[-1])
    ref = torch.autograd.grad(y, leaves, dy.double().cpu())
    assert _rel(P.conv2d_rcp_fused_nchw(x, *A, S).cpu(), y.detach()) < REL
    dx, dA, dS = P.rcp_conv2d_backward(x, dy, *A, S)
    assert _rel(dx, ref[0]) < REL
    for got, want in zip((*dA, dS), ref[1:]):
        assert _rel(got, want) < 1e-6
    P.device_status()


# More tiles than pairs of SMs (74), the last round of them cut in K, and K, M and N that are no multiples of anything.
MANY_DENSE = [(2100, (7, 9, 5), (13, 11, 15)), (100, (13, 11, 15), (13, 11, 15)), (19001, (7, 9), (7, 10)), (19001, (9, 9), (3, 5))]


@pytest.mark.parametrize("case", MANY_DENSE, ids=str)
def test_dense_more_tiles_than_pairs(case):
    test_dense(case, 1)


@pytest.mark.parametrize("case", [(6, 55, 58, (5, 7), (10, 7)), (2, 9, 7, (13, 15, 3), (13, 7, 11))], ids=str)
def test_rcp_more_tiles_than_pairs(case):
    test_rcp(case)


def test_rows_keep_their_own_scale():
    """Every row of the batch has its own power of two, so that a row is as accurate beside any other: magnitudes from 1e-30 to
    the largest float.  Infinities and NaN stay in their row."""
    import paralleltnnlayers_b200 as P
    normal = _normal(5)
    F = [normal(16, 16, 9) * 0.1 for _ in range(2)]
    M = _kron(F).sum(-1)
    scale = torch.tensor([1e-30, 1e-8, 1.0, 1e8, 1e30, 1e-18, 3e37], device="cuda")
    x = normal(7, 256) * scale[:, None]
    ref = x.double() @ M
    y = P.dense_cp(x, *F)
    for i in range(7):
        assert _rel(y[i], ref[i]) < REL, i
    x[2, 3], x[4, 7] = float("nan"), float("inf")
    z = P.dense_cp(x, *F)
    assert bool(torch.isnan(z[2]).all()) and not bool(torch.isfinite(z[4]).any())
    for i in (0, 1, 3, 5):
        assert torch.equal(z[i], y[i]), i
    # the pixels of a convolution
    A, S = [normal(8, 8, 9) * 0.2 for _ in range(2)], normal(3, 3, 9) * 0.3
    u = normal(4, 64, 6, 7) * torch.tensor([1e-25, 1.0, 1e25, 1e-10], device="cuda")[:, None, None, None]
    K = torch.einsum("ctr,yxr->tcyx", _kron(A), S.double()).cpu()
    ref, v = torch.nn.functional.conv2d(u.double().cpu(), K, padding=1), P.conv2d_rcp_fused_nchw(u, *A, S)
    for i in range(4):
        assert _rel(v[i].cpu(), ref[i]) < REL, i
    u[1, 5, 2, 3] = float("nan")
    w = P.conv2d_rcp_fused_nchw(u, *A, S)
    hit = torch.zeros(6, 7, dtype=torch.bool, device="cuda")
    hit[1:4, 2:5] = True
    assert bool(torch.isnan(w[1][:, hit]).all()) and torch.equal(w[1][:, ~hit], v[1][:, ~hit])
    assert torch.equal(w[[0, 2, 3]], v[[0, 2, 3]])


def _bound(x, W, least=2.0 ** -39):
    """Largest error of x W^T (rows: results): 2**-20 of every term, and what values far below the largest of their row may be off."""
    ax, aW = x.double().abs(), W.double().abs()
    far = lambda a: least * a.amax(-1, keepdim=True)
    return 2.0 ** -20 * ax @ aW.T + far(ax) * aW.sum(-1) + ax.sum(-1, keepdim=True) * far(aW).T


@pytest.mark.parametrize("power", [10, 17, 30, 40])
@pytest.mark.parametrize("odims", [(16, 8), (13, 14, 15)])   # the second: the weight written as planes, 2**5 less range
def test_dense_values_far_below_the_largest(power, odims):
    """A feature far above the others that has no weight (an output gradient of an output without one), and small weights along the
    sum: within the stated bound, entry by entry, and unharmed up to 2**17."""
    import paralleltnnlayers_b200 as P
    normal = _normal(power)
    idims = (15, 13, 16)[:len(odims)]
    least = 2.0 ** -39 if len(odims) == 2 else 2.0 ** -34
    F = [normal(i, o, 9) * 0.35 for i, o in zip(idims, odims)]
    I, O = math.prod(idims), math.prod(odims)
    F[0][1] = 0          # inputs without weight
    F[0][2] *= 2.0 ** -power
    F[0][:, 3] = 0       # outputs without weight
    W = _kron(F).sum(-1)
    x, dy = normal(40, I), normal(40, O)
    x[:, I // idims[0] + 2] = 2.0 ** power
    dy[:, 3 * (O // odims[0]) + 1] = -2.0 ** power
    y, ref = P.dense_cp(x, *F).double(), x.double() @ W
    assert bool(((y - ref).abs() <= _bound(x, W.T, least)).all())
    dx, rdx = P.dense_cp_backward(x, dy, *F)[0].double(), dy.double() @ W.T
    assert bool(((dx - rdx).abs() <= _bound(dy, W, least)).all())
    if power <= 17 and len(odims) == 2:
        assert _rel(y, ref) < REL and _rel(dx, rdx) < REL
    P.device_status()


@pytest.mark.parametrize("power", [10, 17, 30, 40])
def test_rcp_values_far_below_the_largest(power):
    import paralleltnnlayers_b200 as P
    normal = _normal(power)
    A, S = [normal(8, 8, 9) * 0.3, normal(9, 10, 9) * 0.3], normal(3, 3, 9) * 0.3
    A[0][1] = 0
    A[0][2] *= 2.0 ** -power
    x = normal(2, 72, 6, 7)
    x[:, 9 + 2] = 2.0 ** power
    K = torch.einsum("ctr,yxr->tcyx", _kron(A), S.double()).cpu()
    conv = lambda u, k: torch.nn.functional.conv2d(u, k, padding=1)
    ref, y = conv(x.double().cpu(), K), P.conv2d_rcp_fused_nchw(x, *A, S).double().cpu()
    ax = x.double().abs().cpu()
    far = ax.amax(1, keepdim=True).expand_as(ax)
    wide = K.abs().amax((1, 2, 3), keepdim=True).expand_as(K)
    bound = 2.0 ** -20 * conv(ax, K.abs()) + 2.0 ** -39 * (conv(far, K.abs()) + conv(ax, wide))
    assert bool(((y - ref).abs() <= bound).all())
    if power <= 17:
        assert _rel(y, ref) < REL


def test_whole_numbers_are_exact():
    """Small integers have no low part and sums below 2**24 are not cut off."""
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(1)
    integers = lambda *s: torch.randint(-3, 4, s, generator=gen, device="cuda").float()
    x, F = integers(130, 144), [integers(12, 12, 2) for _ in range(2)]
    assert torch.equal(P.dense_cp(x, *F).double(), x.double() @ _kron(F).sum(-1))


def test_under_capture_and_on_another_stream():
    import paralleltnnlayers_b200 as P
    normal = _normal(8)
    x, F = normal(128, 256), [normal(16, 16, 12) * 0.35 for _ in range(2)]
    want = P.dense_cp(x, *F)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        assert torch.equal(P.dense_cp(x, *F), want)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = P.dense_cp(x, *F)
    x.copy_(normal(128, 256))
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, P.dense_cp(x, *F))


@pytest.mark.parametrize("size", [1e6, 1e9, 1e20])
@pytest.mark.parametrize("where", ["input", "gradient"])
def test_dense_gradients_beside_a_large_sample(size, where):
    """A sample whose gradient (or input) is zero adds nothing to the factor gradients, however large its input (gradient): every
    value of both operands keeps its own exponent."""
    import paralleltnnlayers_b200 as P
    normal = _normal(7)
    x, dy = normal(500, 144), normal(500, 160)
    big, none = (x, dy) if where == "input" else (dy, x)
    big[7] *= size
    none[7] = 0
    big[300, 3], none[300] = size, 0   # one value of a sample
    F = [normal(i, o, 9) * 0.35 for i, o in ((12, 16), (12, 10))]
    leaves = [f.double().requires_grad_() for f in F]
    ref = torch.autograd.grad(x.double() @ _kron(leaves).sum(-1), leaves, dy.double())
    for got, want in zip(P.dense_cp_backward(x, dy, *F)[1], ref):
        assert _rel(got, want) < 1e-6
    P.device_status()


@pytest.mark.parametrize("size", [1e6, 1e9, 1e20])
@pytest.mark.parametrize("where", ["input", "gradient"])
def test_rcp_gradients_beside_a_large_sample(size, where):
    """The same for a convolution: an image, and a pixel with zeros wherever a tap reaches."""
    import paralleltnnlayers_b200 as P
    normal = _normal(8)
    x, dy = normal(3, 144, 10, 12), normal(3, 160, 10, 12)
    big, none = (x, dy) if where == "input" else (dy, x)
    big[1] *= size
    none[1] = 0
    big[0, :, 4, 5] *= size
    none[0, :, 3:6, 4:7] = 0
    A, S = [normal(i, o, 9) * 0.3 for i, o in ((12, 16), (12, 10))], normal(3, 3, 9) * 0.3
    leaves = [t.double().requires_grad_() for t in (*A, S)]
    K = torch.einsum("ctr,yxr->tcyx", _kron(leaves[:2]), leaves[2])
    y = torch.nn.functional.conv2d(x.double().cpu(), K.cpu(), padding=1)
    ref = torch.autograd.grad(y, leaves, dy.double().cpu())
    _, dA, dS = P.rcp_conv2d_backward(x, dy, *A, S)
    for got, want in zip((*dA, dS), ref):
        assert _rel(got, want) < 1e-6
    P.device_status()
