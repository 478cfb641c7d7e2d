"""Sums that fp32 holds exactly stay exact on the tensor cores: values of all 24 bits that meet one other value, and whole numbers of
12 bits and more whose products and sums stay below 2**24.  Nothing is cut off there, so nothing may be added either.
B200CP_GEMM_TC=2 takes the tensor products at every size."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def always(monkeypatch):
    monkeypatch.setenv("B200CP_GEMM_TC", "2")


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _few(gen, rows, cols):
    """one power of two in every column, the other rows are zero"""
    x = torch.zeros(rows, cols, device="cuda")
    at = torch.randint(rows, (cols,), generator=gen, device="cuda")
    x[at, torch.arange(cols, device="cuda")] = torch.exp2(torch.randint(-9, 10, (cols,), generator=gen, device="cuda").float())
    return x


def _whole(gen, rows, cols, most, count):
    """`count` whole numbers up to `most` in every column"""
    x = torch.zeros(rows, cols, device="cuda")
    for c in range(cols):
        at = torch.randperm(rows, generator=gen, device="cuda")[:count]
        x[at, c] = torch.randint(-most, most + 1, (count,), generator=gen, device="cuda").float()
    return x


# samples and features; the last is cut in K.  (One factor of rank 1: its gradient is the product of the two operands.)
@pytest.mark.parametrize("B, I, O", [(1, 16, 16), (70, 9, 13), (300, 16, 16), (20000, 16, 12)])
def test_gradient_of_single_samples(B, I, O):
    import paralleltnnlayers_b200 as P
    gen = _generator(B)
    one = torch.ones(I, O, 1, device="cuda")
    x, dy = _few(gen, B, I), torch.randn(B, O, generator=gen, device="cuda")
    want = x.double().T @ dy.double()
    assert torch.equal(P.dense_cp_backward(x, dy, one)[1][0][:, :, 0].double(), want)
    x, dy = torch.randn(B, I, generator=gen, device="cuda"), _few(gen, B, O)
    want = x.double().T @ dy.double()
    assert torch.equal(P.dense_cp_backward(x, dy, one)[1][0][:, :, 0].double(), want)


@pytest.mark.parametrize("most, count", [(4095, 1), (2049, 3), (700, 32)])
def test_gradient_of_whole_numbers(most, count):
    import paralleltnnlayers_b200 as P
    gen = _generator(most)
    x, dy = _whole(gen, 300, 16, most, count), _whole(gen, 300, 16, most, 300)
    want = x.double().T @ dy.double()
    assert want.abs().max() < 2 ** 24
    assert torch.equal(P.dense_cp_backward(x, dy, torch.ones(16, 16, 1, device="cuda"))[1][0][:, :, 0].double(), want)


@pytest.mark.parametrize("most, count", [(4095, 1), (2049, 3)])
def test_convolution_gradient_of_whole_numbers(most, count):
    import paralleltnnlayers_b200 as P
    gen = _generator(most)
    N, C, T, H, W = 2, 16, 12, 9, 11
    x = _whole(gen, N * H * W, C, most, count).view(N, H, W, C).permute(0, 3, 1, 2).contiguous()
    dy = _whole(gen, N * H * W, T, most, N * H * W).view(N, H, W, T).permute(0, 3, 1, 2).contiguous()
    S = torch.zeros(3, 3, 1, device="cuda")
    S[1, 1] = 1   # the gradient of the factor is that of the weight in the middle tap
    want = torch.einsum("nchw,nthw->ct", x.double(), dy.double())
    assert want.abs().max() < 2 ** 24
    dA = P.rcp_conv2d_backward(x, dy, torch.ones(C, T, 1, device="cuda"), S)[1][0]
    assert torch.equal(dA[:, :, 0].double(), want)


@pytest.mark.parametrize("R", [9, 64, 100])
def test_weight_of_whole_numbers(R):
    """One rank of whole numbers whose product has 22 bits, the other ranks zero: samples with a single 1 read the weight's rows."""
    import paralleltnnlayers_b200 as P
    gen = _generator(R)
    idims, odims, most = (15, 13, 16), (13, 14, 15), (2047, 45, 45)
    F = [torch.zeros(i, o, R, device="cuda") for i, o in zip(idims, odims)]
    for f, m in zip(F, most):
        f[:, :, R // 2] = torch.randint(-m, m + 1, f.shape[:2], generator=gen, device="cuda").float()
    W = torch.einsum("ai,bj,ck->abcijk", *[f[:, :, R // 2].double() for f in F]).reshape(15 * 13 * 16, 13 * 14 * 15)
    at = torch.randint(len(W), (40,), generator=gen, device="cuda")
    x = torch.zeros(40, len(W), device="cuda")
    x[torch.arange(40, device="cuda"), at] = 1
    assert torch.equal(P.dense_cp(x, *F).double(), W[at])
