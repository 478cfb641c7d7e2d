"""The native operator bindings: argument errors keep their Python types, and the first call of a thread may be a backward."""
import numpy as np
import pytest
import torch

from oracle import cp_oracle as O

Z = torch.zeros


@pytest.mark.parametrize("call", [
    lambda P: P.cp4_conv2d_forward(Z(1, 2, 4, 4), Z(2, 2), Z(2, 2), Z(3, 2), Z(3, 2)),            # not a CUDA tensor
    lambda P: P.cp4_conv2d_step(None, Z(1, 2, 4, 4), Z(2, 2), Z(2, 2), Z(3, 2), Z(3, 2)),         # not a tensor
    lambda P: P.cp3_conv2d_forward(Z(1, 2, 4, 4), Z(2, 2), Z(2, 2), Z(3, 3, 2)),
    lambda P: P.dense_cp(Z(2, 4), Z(2, 2, 3), Z(2, 2, 3)),
    lambda P: P.conv2d_rcp_fused_nchw(Z(1, 4, 4, 4), Z(2, 2, 3), Z(2, 2, 3), Z(3, 3, 3)),
], ids=["cp4", "step", "cp3", "dense", "rcp"])
def test_wrong_tensors_are_type_errors(lib_built, call):
    import paralleltnnlayers_b200 as P
    with pytest.raises(TypeError, match="must be a float32 CUDA tensor"):
        call(P)


# N, C, T, H, W, R = 2, 4, 6, 5, 5, 3; modes 2x2 -> 3x2.  Each call has one operand whose size or device does not go
# with the others; `c` makes fake CUDA tensors, so that nothing can be launched.
def _k4(c):
    return c(6, 3), c(4, 3), c(3, 3), c(3, 3)


def _k3(c):
    return c(6, 3), c(4, 3), c(3, 3, 3)


def _modes(c):
    return c(2, 3, 3), c(2, 2, 3)


MISFITS = {
    "saved dLdO": lambda P, c: P.cp4_conv2d_backward_filter_saved(c(2, 6, 5, 4), c(2, 4, 5, 5), c(2, 3, 5, 5), c(2, 3, 5, 5), *_k4(c)),
    "saved P": lambda P, c: P.cp4_conv2d_backward_filter_saved(c(2, 6, 5, 5), c(2, 4, 5, 5), c(1, 3, 5, 5), c(2, 3, 5, 5), *_k4(c)),
    "saved Q": lambda P, c: P.cp4_conv2d_backward_filter_saved(c(2, 6, 5, 5), c(2, 4, 5, 5), c(2, 3, 5, 5), c(2, 2, 5, 5), *_k4(c)),
    "cp3 dLdO": lambda P, c: P.cp3_conv2d_backward_filter(c(2, 6, 4, 5), c(2, 4, 5, 5), *_k3(c)),
    "rcp input": lambda P, c: P.rcp_conv2d_backward(c(2, 3, 5, 5), c(2, 6, 5, 5), *_modes(c), c(3, 3, 3)),
    "rcp dV": lambda P, c: P.rcp_conv2d_backward(c(2, 4, 5, 5), c(2, 5, 5, 5), *_modes(c), c(3, 3, 3)),
    "rcp core": lambda P, c: P.rcp_conv2d_backward(c(2, 4, 5, 5), c(2, 6, 5, 5), *_modes(c), c(3, 3, 2)),
    "rcp vector": lambda P, c: P.rcp_conv2d_backward(c(1), c(6), c(1, 6, 3), c(1, 1, 3)),
    "dense input": lambda P, c: P.dense_cp_backward(c(2, 3), c(2, 6), *_modes(c)),
    "dense dV": lambda P, c: P.dense_cp_backward(c(2, 4), c(1, 6), *_modes(c)),
    "cp4 device": lambda P, c: P.cp4_conv2d_forward(c(2, 4, 5, 5), *_k4(c)[:3], c(3, 3, dev=1)),
    "cp4 dLdO device": lambda P, c: P.cp4_conv2d_backward_filter(c(2, 6, 5, 5, dev=1), c(2, 4, 5, 5), *_k4(c)),
    "cp4 pair device": lambda P, c: P.cp4_conv2d_forward_backward_data(c(2, 4, 5, 5), c(2, 6, 5, 5, dev=1), *_k4(c)),
    "step device": lambda P, c: P.cp4_conv2d_step(c(2, 4, 5, 5), c(2, 6, 5, 5, dev=1), *_k4(c)),
    "cp3 device": lambda P, c: P.cp3_conv2d_forward(c(2, 4, 5, 5), *_k3(c)[:2], c(3, 3, 3, dev=1)),
    "rcp device": lambda P, c: P.conv2d_rcp_fused_nchw(c(2, 4, 5, 5), *_modes(c), c(3, 3, 3, dev=1)),
    "dense device": lambda P, c: P.dense_cp(c(2, 4), c(2, 3, 3, dev=1), c(2, 2, 3)),
    "full dLdO": lambda P, c: P.cp4_conv2d_backward_filter_full(c(2, 6, 4, 5), c(2, 4, 5, 5), 3, 3),
    "full device": lambda P, c: P.cp4_conv2d_backward_filter_full(c(2, 6, 5, 5, dev=1), c(2, 4, 5, 5), 3, 3),
    "recompose rank": lambda P, c: P.cp4recom(c(6, 3), c(4, 2), c(3, 3), c(3, 3)),
    "recompose device": lambda P, c: P.cp4recom(c(6, 3), c(4, 3, dev=1), c(3, 3), c(3, 3)),
    "rcp recompose device": lambda P, c: P.rcp_recompose(*_modes(c), c(3, 3, 3, dev=1)),
    "dense recompose device": lambda P, c: P.dense_cp_recompose(c(2, 3, 3), c(2, 2, 3, dev=1)),
    "rebuild device": lambda P, c: P.cp4_conv2d_rebuild_forward(c(2, 4, 5, 5, dev=1), *_k4(c)),
    "conv device": lambda P, c: P.conv2d_dense_forward(c(2, 4, 5, 5), c(6, 4, 3, 3, dev=1)),
    "matmul device": lambda P, c: P.dense_matmul(c(2, 4), c(4, 6, dev=1)),
    "allclose device": lambda P, c: P.allclose(c(2, 4), c(2, 4, dev=1)),
    "dense dV device": lambda P, c: P.dense_cp_backward(c(2, 4), c(2, 6, dev=1), *_modes(c)),
}


@pytest.mark.parametrize("what", MISFITS)
def test_operands_that_do_not_fit_are_value_errors(lib_built, what):
    from torch._subclasses.fake_tensor import FakeTensorMode
    import paralleltnnlayers_b200 as P
    with FakeTensorMode(), pytest.raises(ValueError):
        MISFITS[what](P, lambda *size, dev=0: torch.empty(*size, device=f"cuda:{dev}"))


@pytest.mark.parametrize("dU, fc, out", [((2, 6, 5, 4), (4, 3), None), ((2, 6, 5, 5), (5, 3), None),
                                         ((2, 6, 5, 5), (4, 2), None), ((2, 6, 5, 5), (4, 3), [(2, 6, 5, 4), (2, 4, 5, 5), (48,)]),
                                         ((2, 6, 5, 5), (4, 3), [(2, 6, 5, 5), (2, 4, 5, 5), (47,)])])
def test_host_buffers_that_do_not_fit_are_value_errors(lib_built, dU, fc, out):
    import paralleltnnlayers_b200 as P
    args = (Z(2, 4, 5, 5), Z(*dU), Z(6, 3), Z(*fc), Z(3, 3), Z(3, 3))
    out = out and [Z(*size) for size in out]
    with pytest.raises(ValueError):
        P.cp4_conv2d_step_host(*args, out=out)
    with pytest.raises(ValueError):
        P.cp4_conv2d_step_host_submit(*args, out=out or [Z(2, 6, 5, 5), Z(2, 4, 5, 5), Z(48)])


@pytest.mark.gpu
def test_shape_errors_and_status_errors():
    import paralleltnnlayers_b200 as P
    c = lambda *s: torch.zeros(*s, device="cuda")
    with pytest.raises(TypeError):
        P.dense_cp(c(2, 4).double(), c(2, 2, 3), c(2, 2, 3))
    with pytest.raises(ValueError):
        P.cp4_conv2d_forward(c(1, 3, 4, 4), c(2, 2), c(2, 2), c(3, 2), c(3, 2))     # 3 channels, factor of 2
    with pytest.raises(ValueError):
        P.dense_cp(c(2, 5), c(2, 2, 3), c(2, 2, 3))
    with pytest.raises(ValueError):
        P.conv2d_rcp_fused_nchw(c(1, 4, 4, 4), c(2, 2, 3), c(2, 2, 3), c(3, 3, 2))
    with pytest.raises(P.B200CPError) as e:                                          # refused by the library
        P.cp4_conv2d_backward_filter(c(1, 2, 4, 4), c(1, 2, 4, 4), c(2, 2), c(2, 2), c(3, 2), c(5, 2))
    assert e.value.status == -2


@pytest.mark.gpu
def test_backward_as_the_first_call_of_a_thread():
    """The engine's worker thread has no CUDA context of its own yet when the first backward needs a tensor map."""
    import os
    import subprocess
    import sys
    code = r'''
import numpy as np, torch
import paralleltnnlayers_b200 as P
from oracle import cp_oracle as O
X, K0, K1, KH, KW, dU = O.make_cp4_inputs(5, 2, 8, 16, 16, 16, 3, 3, 4, factor_std=0.3)
t = [torch.from_numpy(a).cuda().requires_grad_(True) for a in (X, K0, K1, KH, KW)]
g = torch.autograd.grad(P.CP4Conv2dFunction.apply(*t), t, torch.from_numpy(dU).cuda())
for a, r in zip(g, (O.cp4_backward_data(dU, K0, K1, KH, KW, 1), *O.cp4_backward_filter(X, dU, K0, K1, KH, KW, 1))):
    assert np.allclose(a.cpu().numpy(), r, rtol=1e-4, atol=1e-5 * max(1.0, float(np.abs(r).max())))
print("ok")
'''
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("make", ["CP4Conv2d", "CPConv2d"])
def test_inference_of_a_module_keeps_no_plane(make):
    """Under no_grad the factors of a module still require a gradient: its forward is the plain operator's, with the
    output as the only allocation, and the same bits."""
    import paralleltnnlayers_b200 as P
    from paralleltnnlayers_b200 import layers
    layer = getattr(layers, make)(512, 512, rank=8).cuda()
    x = torch.randn(2, 512, 50, 50, device="cuda")
    op = P.cp4_conv2d_forward if make == "CP4Conv2d" else P.cp3_conv2d_forward

    def allocations(run):
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        return run(), torch.cuda.memory_stats()["allocation.all.allocated"] - before

    with torch.no_grad():
        allocations(lambda: layer(x))
        y, n = allocations(lambda: layer(x))
        want, n_op = allocations(lambda: op(x, *layer.parameters()))
    assert n == n_op == 1 and torch.equal(y, want)
    y, n = allocations(lambda: layer(x))
    assert n == 2 and y.requires_grad     # with gradients the plane is kept
    with torch.inference_mode():
        assert allocations(lambda: layer(x))[1] == 1
