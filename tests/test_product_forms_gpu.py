"""The dense and reshaped-CP layers in both forms -- factored (the C calls without a workspace) and multiplied out (with the
workspace that the library asks for) -- on general shapes, and which of the two the library asks for."""
import ctypes as C
import random

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import cp_oracle as O
from tests.gpu_util import check, dev


def _lib():
    from paralleltnnlayers_b200 import _lib as L
    return L


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _run(L, call, size, out):
    """The call without a workspace, and with the one it asks for (None where it asks for none)."""
    got = []
    for n in (0, size):
        if n == 0 and got:
            return got[0], None
        ws = torch.empty(n // 4, device="cuda") if n else None
        out.fill_(float("nan"))
        L.check(call(_ptr(ws) if n else None, n))
        got.append(out.clone())
    return got


def dense_forms(B, idims, odims, R, X, F, dY):
    """(forward, data gradient), each as the two forms"""
    L = _lib()
    m, i, o = len(idims), L.int_array(idims), L.int_array(odims)
    fp, st = L.ptr_array([f.data_ptr() for f in F]), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    Y, dX = torch.empty(B, int(np.prod(odims)), device="cuda"), torch.empty(B, int(np.prod(idims)), device="cuda")
    return (_run(L, lambda w, n: L.lib.b200cp_dense_fwd_ws(B, m, i, o, R, _ptr(X), fp, _ptr(Y), w, n, st, 0),
                 L.lib.b200cp_dense_fwd_workspace_bytes(B, m, i, o, R, 0), Y),
            _run(L, lambda w, n: L.lib.b200cp_dense_bwd(B, m, i, o, R, None, _ptr(dY), fp, _ptr(dX), None, w, n, st, 0),
                 L.lib.b200cp_dense_bwd_workspace_bytes(B, m, i, o, R, 0), dX))


def rcp_forms(N, H, W, cd, td, R, X, A, S, dV):
    L = _lib()
    m, c, t = len(cd), L.int_array(cd), L.int_array(td)
    ap, st = L.ptr_array([a.data_ptr() for a in A]), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    V, dX = torch.empty(N, int(np.prod(td)), H, W, device="cuda"), torch.empty(N, int(np.prod(cd)), H, W, device="cuda")
    return (_run(L, lambda w, n: L.lib.b200cp_rcp_fwd_ws(N, H, W, m, c, t, R, 3, 3, _ptr(X), ap, _ptr(S), _ptr(V), w, n, st, 0),
                 L.lib.b200cp_rcp_fwd_workspace_bytes(N, H, W, m, c, t, R, 3, 3, 0), V),
            _run(L, lambda w, n: L.lib.b200cp_rcp_bwd(N, H, W, m, c, t, R, 3, 3, None, _ptr(dV), ap, _ptr(S), _ptr(dX), None,
                                                      None, w, n, st, 0),
                 L.lib.b200cp_rcp_bwd_workspace_bytes(N, H, W, m, c, t, R, 3, 3, 0), dX))


def _draw(rng, order, most):
    while True:
        d = tuple(rng.choice((1, 2, 3, 4, 5, 7, 8, 9, 12, 16)) for _ in range(order))
        if np.prod(d) <= most:
            return d


def _dense_cases():
    rng = random.Random(20)
    for _ in range(24):
        order = rng.choice((1, 2, 3, 4))
        yield rng.choice((1, 2, 15, 16, 63, 130, 700)), _draw(rng, order, 1500), _draw(rng, order, 1500), rng.choice((1, 2, 4, 9, 32, 65))
    for B, R in ((1, 32), (3, 159), (70, 160), (1, 170), (300, 200)):   # the register-tiled kernel's shape and where it ends
        yield B, (8, 8, 8, 8), (8, 8, 8, 8), R


def _rcp_cases():
    rng = random.Random(21)
    for _ in range(24):
        order = rng.choice((1, 2, 3, 4))
        yield (rng.choice((1, 3)), rng.choice((1, 2, 7, 13)), rng.choice((1, 3, 8, 35)), _draw(rng, order, 160), _draw(rng, order, 160),
               rng.choice((1, 2, 4, 9, 33)))
    for N, H, R in ((1, 7, 4), (1, 9, 148), (1, 7, 160)):
        yield N, H, H, (4, 8, 8), (4, 8, 8), R


# the bound of the other parity tests: 1e-4 relative + 1e-5 of the largest value
def _check_all(forms, ref, what):
    for form, got in zip(("factored", "multiplied out"), forms):
        if got is not None:
            check(got, ref, f"{what}, {form}", rtol=1e-4, atol=1e-5 * float(np.abs(ref).max()))


@pytest.mark.parametrize("case", list(_dense_cases()), ids=str)
def test_dense_forms(case):
    B, idims, odims, R = case
    X, F, dY = O.make_dense_inputs(B + R, B, idims, odims, R)
    M = np.ones((1, 1, R))
    for f in F:
        M = np.einsum("abr,ijr->aibjr", M, f.astype(np.float64)).reshape(M.shape[0] * f.shape[0], -1, R)
    M = M.sum(-1)
    x, dy = dev(X.reshape(B, -1), dY.reshape(B, -1))
    fwd, bwd = dense_forms(B, idims, odims, R, x, dev(*F), dy)
    _check_all(fwd, X.reshape(B, -1).astype(np.float64) @ M, "dense forward")
    _check_all(bwd, dY.reshape(B, -1).astype(np.float64) @ M.T, "dense data gradient")


@pytest.mark.parametrize("case", list(_rcp_cases()), ids=str)
def test_rcp_forms(case):
    N, H, W, cd, td, R = case
    X, A, S, dV = O.make_rcp_inputs(N + R, N, cd, td, H, W, 3, 3, R)
    K = np.ones((1, 1, R))
    for a in A:
        K = np.einsum("abr,ijr->aibjr", K, a.astype(np.float64)).reshape(K.shape[0] * a.shape[0], -1, R)
    K = torch.from_numpy(np.einsum("ctr,yxr->tcyx", K, S.astype(np.float64)))
    X, dV = X.reshape(N, -1, H, W), dV.reshape(N, -1, H, W)
    x, dv, s = dev(X, dV, S)
    fwd, bwd = rcp_forms(N, H, W, cd, td, R, x, dev(*A), s, dv)
    _check_all(fwd, torch.nn.functional.conv2d(torch.from_numpy(X).double(), K, padding=1).numpy(), "rcp forward")
    _check_all(bwd, torch.nn.functional.conv_transpose2d(torch.from_numpy(dV).double(), K, padding=1).numpy(), "rcp data gradient")


# sizes where one form is far ahead of the other (factored / multiplied out, us): the times stand beside the rule
FACTORED, OUT = False, True


@pytest.mark.parametrize("case", [
    (4096, (16, 16, 16), (16, 16, 16), 4, FACTORED),       # 386 / 3823
    (4096, (16, 16, 16), (16, 16, 16), 256, OUT),          # 15551 / 4095
    (64, (16, 16, 16), (16, 16, 16), 4, FACTORED),         # 49 / 125
    (64, (16, 16, 16), (4, 4, 4), 137, OUT),               # 434 / 17
    (4096, (10, 10, 10), (10, 10, 10), 4, FACTORED),       # 127 / 257
    (4096, (10, 10, 10), (10, 10, 10), 64, OUT),           # 1501 / 264
    (4096, (8, 8, 8, 8), (8, 8, 8, 8), 32, FACTORED),      # 803 / 3850
    (4096, (8, 8, 8, 8), (8, 8, 8, 8), 170, OUT),          # 9721 / 4030: too many ranks for the register-tiled kernel
    (4096, (8, 8, 8, 8), (8, 8, 8, 8), 256, OUT),          # 14484 / 4098
    (1, (8, 8, 8, 8), (8, 8, 8, 8), 16, FACTORED),         # 35 / 82
    (1, (8, 8, 8, 8), (8, 8, 8, 8), 170, OUT),             # 1371 / 250
    (65535 * 64 + 1, (2, 2), (2, 2), 64, OUT),
], ids=str)
def test_dense_rule(case):
    B, idims, odims, R, out = case
    L = _lib()
    assert (L.lib.b200cp_dense_fwd_workspace_bytes(B, len(idims), L.int_array(idims), L.int_array(odims), R, 0) > 0) is out


@pytest.mark.parametrize("case", [
    (32, 28, (16, 16), (16, 16), 4, FACTORED),     # 616 / 968
    (32, 28, (16, 16), (16, 16), 16, OUT),         # 2154 / 968
    (8, 32, (6, 6, 6), (6, 6, 6), 4, FACTORED),    # 161 / 275
    (8, 32, (6, 6, 6), (6, 6, 6), 64, OUT),        # 2250 / 277
    (32, 28, (4, 8, 8), (4, 8, 8), 16, FACTORED),  # 250 / 968
    (8, 32, (4, 4), (4, 4), 11, OUT),              # 223 / 10
], ids=str)
def test_rcp_rule(case):
    N, H, cd, td, R, out = case
    L = _lib()
    assert (L.lib.b200cp_rcp_fwd_workspace_bytes(N, H, H, len(cd), L.int_array(cd), L.int_array(td), R, 3, 3, 0) > 0) is out
