"""The multiplied-out forms of the dense and reshaped-CP layers on CUDA cores, at the edges of their tiles."""
import numpy as np
import pytest

from oracle import cp_oracle as O
from tests.gpu_util import check, dev

pytestmark = pytest.mark.gpu

DENSE = [  # B, idims, odims, R: product tiles of 16 / 32 / 64 x 64, K split over 1-8 CTAs, weight tiles of 16 / 32 / 64 x 64
    (1, (5,), (3,), 1), (16, (16, 16), (4, 4), 31), (17, (5, 5, 5), (3, 5, 7), 33), (64, (16, 16, 16), (4, 4, 4), 137),
    (65, (3, 2, 5, 4), (2, 7, 3, 2), 5), (300, (8, 8), (13, 11), 32), (33, (4, 4), (16, 16, 16)[:2], 65),
    (700, (4, 6, 4), (4, 6, 4), 40), (130, (9, 7), (16, 16), 8), (2, (16, 16, 16), (16, 16, 8), 3),
]


@pytest.mark.parametrize("case", DENSE, ids=str)
def test_dense_forward_and_data_gradient(case):
    import paralleltnnlayers_b200 as P
    B, idims, odims, R = case
    X, F, dY = O.make_dense_inputs(11, B, idims, odims, R)
    x, dy = dev(X, dY)
    f = dev(*F)
    ref = O.dense_cp_forward(X, F)
    check(P.dense_cp(x, *f), ref, "dense forward", atol=1e-5 * max(1.0, float(np.abs(ref).max())))
    rX = O.dense_cp_backward(X, dY, F)[0]
    check(P.dense_cp_backward(x, dy, *f, need_dw=False)[0], rX, "dense dX", atol=1e-5 * max(1.0, float(np.abs(rX).max())))


def test_more_row_tiles_than_a_grid_dimension():
    """65536 row tiles of 64: the batch of a wide but shallow input."""
    import torch
    import paralleltnnlayers_b200 as P
    B, R = 65535 * 64 + 1, 64
    x = torch.empty(B, 4, device="cuda").uniform_(-1, 1)
    F = [torch.randn(2, 2, R, device="cuda") * 0.35 for _ in range(2)]
    M = torch.einsum("aoR,bpR->abop", *[f.double() for f in F]).reshape(4, 4)
    for got, ref in ((P.dense_cp(x, *F), x.double() @ M), (P.dense_cp_backward(x, x, *F, need_dw=False)[0], x.double() @ M.T)):
        # sums of 64 then 4 products: (64 + 4) ulp of the terms' size, far below this
        assert float((got.double() - ref).abs().max()) <= 1e-5 * float(ref.abs().max())


RCP = [  # N, cdims, tdims, H, W, R: channel tiles of 16 / 32 / 64, pixel tiles of 256 / 128 / 64, channels split over a cluster
    (1, (3,), (5,), 1, 1, 2), (2, (4, 4), (4, 4), 32, 32, 11), (1, (2, 9), (3, 11), 7, 33, 5), (3, (5, 5), (6, 6), 9, 5, 33),
    (1, (16, 16), (5, 13), 7, 7, 4), (1, (16, 16), (16, 16), 8, 30, 16), (2, (2, 3, 4), (3, 3, 8), 13, 40, 7),
]


@pytest.mark.parametrize("case", RCP, ids=str)
def test_rcp_forward_and_data_gradient(case):
    import paralleltnnlayers_b200 as P
    N, cd, td, H, W, R = case
    X, A, S, dV = O.make_rcp_inputs(12, N, cd, td, H, W, 3, 3, R)
    x, s, dv = dev(X, S, dV)
    a = dev(*A)
    ref = O.rcp_forward(X, A, S)
    check(P.conv2d_rcp_fused_nchw(x, *a, s), ref, "rcp forward", atol=1e-5 * max(1.0, float(np.abs(ref).max())))
    rX = O.rcp_backward(X, dV, A, S)[0]
    check(P.rcp_conv2d_backward(x, dv, *a, s, need_dw=False)[0], rX, "rcp dX", atol=1e-5 * max(1.0, float(np.abs(rX).max())))


# The weight formed by the product's CTAs or by a launch before it: up to 16 ranks, 512 entries (channels of a CTA x its tile of outputs); one to
# four modes, channels that do not fill a CTA's share, a last tile of outputs that is not full.
INSIDE = [
    (2, (4, 4), (4, 4), 9, 8, 16), (2, (4, 4), (4, 4), 9, 8, 17), (1, (2, 2, 2, 2), (2, 2, 2, 3), 5, 6, 16), (1, (13,), (16,), 6, 7, 3),
    (1, (4, 8), (4, 4), 33, 5, 9), (1, (3, 11), (4, 4), 33, 5, 9), (1, (2, 4), (9, 9), 8, 8, 5), (40, (3, 2, 3), (3, 2, 2), 12, 12, 1),
]


@pytest.mark.parametrize("case", INSIDE, ids=str)
def test_rcp_weight_formed_inside(case):
    test_rcp_forward_and_data_gradient(case)


def test_workspace_of_a_weight_formed_inside():
    """The launch that forms the weight itself takes none of the weight's size, and a call without any runs the factored kernels."""
    import ctypes
    import torch
    from paralleltnnlayers_b200._lib import int_array, lib, ptr_array
    N, cd, td, H, W, R = 2, (4, 4), (4, 4), 9, 8, 16
    X, A, S, _ = O.make_rcp_inputs(14, N, cd, td, H, W, 3, 3, R)
    x, s, *a = dev(X, S, *A)
    shape = (N, H, W, 2, int_array(cd), int_array(td), R, 3, 3)
    assert lib.b200cp_rcp_fwd_workspace_bytes(*shape, 8) == 256
    ws = torch.empty(256, dtype=torch.uint8, device="cuda")
    ref = O.rcp_forward(X, A, S)
    for pointer, size in ((ws.data_ptr(), 256), (None, 0)):
        v = torch.empty(ref.shape, device="cuda")
        before = lib.b200cp_launch_count()
        vp = ctypes.c_void_p
        assert lib.b200cp_rcp_fwd_ws(*shape, vp(x.data_ptr()), ptr_array([t.data_ptr() for t in a]), vp(s.data_ptr()), vp(v.data_ptr()),
                                     vp(pointer), size, vp(torch.cuda.current_stream().cuda_stream), 8) == 0
        assert lib.b200cp_launch_count() - before == 1
        check(v, ref, "rcp", atol=1e-5 * max(1.0, float(np.abs(ref).max())))


# The channels split over a cluster whose last CTA has fewer stages than the others: on the other side of the line from which on accumulators
# are added to totals (-1), or on the same side (below it 0, above it 1).
UNEVEN = [
    (4, (6, 6, 2), (6, 6, 2), 9, 9, 16, False, -1), (4, (6, 6, 2), (6, 6, 2), 9, 9, 16, True, -1), (3, (10, 12), (3, 3), 27, 28, 8, False, -1),
    (3, (3, 3), (10, 12), 27, 28, 8, True, -1), (2, (3, 3, 8), (3, 3, 8), 23, 23, 4, False, -1), (4, (10, 5, 3), (3, 4, 3), 11, 11, 24, False, -1),
    (2, (6, 4, 3), (2, 3, 10), 25, 25, 52, False, -1), (14, (6, 12), (6, 12), 7, 7, 20, True, -1), (2, (10, 12), (4, 6), 28, 28, 40, False, -1),
    (2, (7, 8), (6, 12), 20, 20, 20, False, 0), (2, (13, 8), (6, 12), 20, 20, 20, False, 1),
]


@pytest.mark.parametrize("case", UNEVEN, ids=str)
def test_rcp_uneven_shares_of_a_cluster(case):
    import ctypes
    import paralleltnnlayers_b200 as P
    from paralleltnnlayers_b200._lib import int_array, lib
    N, cd, td, H, W, R, transposed, side = case
    out = (ctypes.c_int * 5)()
    assert lib.b200cp_test_rcp_product(N, H, W, len(cd), int_array(cd), int_array(td), R, transposed, 8, out) == 0
    form, ctas, first, last, line = out
    assert form == 1 and ctas > 1 and first > last
    assert (first > line, last > line) == {-1: (True, False), 0: (False, False), 1: (True, True)}[side]
    X, A, S, dV = O.make_rcp_inputs(13, N, cd, td, H, W, 3, 3, R)
    x, s, dv = dev(X, S, dV)
    a = dev(*A)
    if transposed:
        ref, got = O.rcp_backward(X, dV, A, S)[0], lambda: P.rcp_conv2d_backward(x, dv, *a, s, need_dw=False)[0]
    else:
        ref, got = O.rcp_forward(X, A, S), lambda: P.conv2d_rcp_fused_nchw(x, *a, s)
    for _ in range(3):   # (what is left in shared memory differs from call to call)
        check(got(), ref, "rcp", atol=1e-5 * max(1.0, float(np.abs(ref).max())))


def test_rounding_of_long_sums():
    """4096 inputs and 256 channels x 9 taps, not split over CTAs.  A chain of n fp32 additions of random signs is off by about
    2**-24 * sqrt(n / 6) of its result: 1.9e-7 for the 64 to 72 terms of an accumulator, 1.4e-7 for the at most 32 totals,
    1e-7 to 2e-7 for the weight's sum over the ranks; one chain over all terms would be at 8e-7 and 6e-7."""
    import torch
    import paralleltnnlayers_b200 as P
    gen = torch.Generator(device="cuda").manual_seed(3)
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    rel = lambda got, ref: float((got.double() - ref).norm() / ref.norm())
    x, F = normal(256, 4096), [normal(16, 16, 64) * 0.35 for _ in range(3)]
    M = torch.einsum("aor,bpr,cqr->abcopq", *[f.double() for f in F]).reshape(4096, 4096)
    assert rel(P.dense_cp(x, *F), x.double() @ M) < 4e-7
    x, A, S = normal(32, 256, 28, 28), [normal(16, 16, 16) * 0.3 for _ in range(2)], normal(3, 3, 16) * 0.3
    K = torch.einsum("aor,bpr,yxr->opabyx", *[f.double() for f in (*A, S)]).reshape(256, 256, 3, 3)
    ref = torch.nn.functional.conv2d(x[:2].double(), K, padding=1)
    assert rel(P.conv2d_rcp_fused_nchw(x, *A, S)[:2], ref) < 4e-7
