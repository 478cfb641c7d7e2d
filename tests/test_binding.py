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
