"""Operator-level mirror of the reference's entry points.

C++ order (``Cuda_kernels/cp4Conv2d.cuh:8-28``): ``cp4_conv2d_forward(Input, FT, FC, FY, FX, pad)``
and the backward pair.  TF custom-op order (``Kernels/cp4_conv_nchw.cc:6-13``,
``test/test_conv2d_cp4.py:13-25``): ``cp4_conv2d_nchw(U, K0[C,R], K1[FH,R], K2[FW,R], K3[T,R])``;
``conv2d_rcp_fused_nchw(U, K0, K1, ..., KC)`` (``Kernels/rcp_fused_nchw.cc:6-12``) and
``dense_cp(U, K0, K1, ...)`` (``Kernels/dense_cp.cc:6-12``), generalised from the single shape
each reference op was compiled for.  Arguments are fp32 CUDA tensors; errors raise, like
the reference ops' ``OP_REQUIRES``.
"""
from __future__ import annotations

import ctypes as C

import torch

from ._lib import B200CPError, TensorShape, check, int_array, lib, ptr_array

try:
    from . import _C            # after torch and the library: the hot operators and the autograd nodes
except ImportError as e:
    raise ImportError("the torch binding (_C.so) is missing or does not match: build it with "
                      f"`python -m paralleltnnlayers_b200.build` ({e})") from e
_C.set_error_class(B200CPError)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _dev(t, name, like=None):
    """``t`` contiguous; with ``like`` it has to be on that tensor's device (the kernels read by address)."""
    if not isinstance(t, torch.Tensor) or not t.is_cuda or t.dtype != torch.float32:
        raise TypeError(f"{name} must be a float32 CUDA tensor")
    if like is not None and t.device != like.device:
        raise ValueError(f"{name} is on {t.device}, the first operand on {like.device}")
    return t.contiguous()


def _factors4(ts, like=None):
    """FT, FC, FY, FX ``[dim, rank]`` with one rank, on one device."""
    like = ts[0] if like is None else like
    ts = [_dev(t, n, like) for t, n in zip(ts, ("FT", "FC", "FY", "FX"))]
    if any(f.dim() != 2 or f.shape[1] != ts[0].shape[1] for f in ts):
        raise ValueError("FT, FC, FY and FX must be [dim, rank] with one rank")
    return ts


def _host_shape(X, dU, FT, FC, FY, FX, pad, out):
    """Checked operands of the host-buffer step: contiguous float32 CPU tensors of the sizes the copies take."""
    for t in [X, dU, FT, FC, FY, FX] + list(out or ()):
        if t.is_cuda or t.dtype != torch.float32 or not t.is_contiguous():
            raise TypeError("host entry point takes contiguous float32 CPU tensors")
    s = _shape_from(X, FT, FC, FY, FX, pad)
    n_out = s.N * s.T * s.H * s.W
    if dU.numel() != n_out:
        raise ValueError("dU must be [N,T,H,W]")
    if out is not None:
        U, dX, dK = out
        if U.numel() != n_out or dX.numel() != X.numel() or dK.numel() != (s.T + s.C + s.Y + s.X) * s.Rank:
            raise ValueError("out must be (U [N,T,H,W], dX [N,C,H,W], dK_packed [(T+C+Y+X)*R])")
    return s


def _p(t):
    return C.c_void_p(t.data_ptr())


def tensor_shape(N, C_, H, W, T, Y, X, Rank, pad):
    return TensorShape(N=N, H=H, W=W, pad=pad, T=T, C=C_, Y=Y, X=X, Rank=Rank)


def _shape_from(inp, FT, FC, FY, FX, pad, in_is_upstream=False):
    if inp.dim() != 4:
        raise ValueError("input must be a rank-4 NCHW tensor")
    for f, nm in ((FT, "FT"), (FC, "FC"), (FY, "FY"), (FX, "FX")):
        if f.dim() != 2 or f.shape[1] != FT.shape[1]:
            raise ValueError(f"{nm} must be [dim, rank] with the same rank as FT")
    ch = FT.shape[0] if in_is_upstream else FC.shape[0]
    if inp.shape[1] != ch:
        raise ValueError(f"input has {inp.shape[1]} channels, the factor has {ch}")
    return tensor_shape(inp.shape[0], FC.shape[0], inp.shape[2], inp.shape[3], FT.shape[0], FY.shape[0],
                        FX.shape[0], FT.shape[1], pad)


# ---- CP4, C++ order ---------------------------------------------------------
def cp4_conv2d_forward(Input, FT, FC, FY, FX, pad=1, flags=0):
    """``CP::Conv2dForward`` (Cuda_kernels/cp4Conv2d.cu:14-43): returns Out [N,T,H,W]."""
    return _C.cp4_forward(Input, FT, FC, FY, FX, pad, flags)


def cp4_conv2d_backward_data(Upstream, FT, FC, FY, FX, pad=1, flags=0):
    """``CP::Conv2dBackwardData`` (Cuda_kernels/cp4Conv2d.cu:48-77): returns dX [N,C,H,W]."""
    return _C.cp4_backward_data(Upstream, FT, FC, FY, FX, pad, flags)


def cp4_conv2d_forward_backward_data(Input, Upstream, FT, FC, FY, FX, pad=1, flags=0, save=False):
    """Forward of ``Input`` and backward-data of ``Upstream`` in one call (one launch where the shape allows it): the
    two convolutions of a training step with frozen factors.  Returns ``(Out, dInput)``, with ``save`` also the rank
    planes ``(P, Q)`` for ``cp4_conv2d_backward_filter_saved``."""
    return _C.cp4_forward_backward_data(Input, Upstream, FT, FC, FY, FX, pad, flags, save)


def cp4_conv2d_backward_filter(dLdO, In, FT, FC, FY, FX, pad=1, flags=0, packed=False):
    """The four factor gradients of ``CP::Conv2dBackwardFilter``
    (Cuda_kernels/cp4Conv2d.cu:83-153): returns (dFT, dFC, dFY, dFX), or the
    packed buffer [dFT|dFC|dFY|dFX] with ``packed=True`` (the allreduce unit)."""
    return _C.cp4_backward_filter(dLdO, In, FT, FC, FY, FX, pad, flags, packed)


def cp4_conv2d_backward_filter_full(dLdO, In, Y, X, pad=1):
    """``cp4_conv2d_backward_filter_full_gpu`` (Cuda_kernels/cp4Conv2dBackwardFilter.cu:23-59): dK [T,C,Y,X]."""
    In = _dev(In, "In")
    dLdO = _dev(dLdO, "dLdO", In)
    if In.dim() != 4 or dLdO.dim() < 2 or dLdO.numel() != In.shape[0] * dLdO.shape[1] * In.shape[2] * In.shape[3]:
        raise ValueError("dLdO must be [N,T,H,W] for In [N,C,H,W]")
    s = tensor_shape(In.shape[0], In.shape[1], In.shape[2], In.shape[3], dLdO.shape[1], Y, X, 1, pad)
    dK = torch.empty((s.T, s.C, Y, X), device=In.device, dtype=torch.float32)
    with torch.cuda.device(In.device):
        check(lib.b200cp_cp4_bwd_filter_full(C.byref(s), _p(In), _p(dLdO), _p(dK), _stream()))
    return dK


def cp4recom(FT, FC, FY, FX):
    """``cp4recom`` (Cuda_kernels/Utils.cu:67-98): dense K [T,C,Y,X]."""
    FT, FC, FY, FX = _factors4((FT, FC, FY, FX))
    s = tensor_shape(1, FC.shape[0], 1, 1, FT.shape[0], FY.shape[0], FX.shape[0], FT.shape[1], 0)
    K = torch.empty((s.T, s.C, s.Y, s.X), device=FT.device, dtype=torch.float32)
    with torch.cuda.device(FT.device):
        check(lib.b200cp_cp4_recompose(C.byref(s), _p(FT), _p(FC), _p(FY), _p(FX), _p(K), _stream()))
    return K


def allclose(A, B, tolerance=1e-3):
    """``AllClose`` (Cuda_kernels/Utils.cu:159-180): True when no element's relative difference
    max(|a-b|/|a|, |a-b|/|b|) exceeds ``tolerance``; the count runs on the device."""
    A = _dev(A, "A")
    B = _dev(B, "B", A)
    if A.numel() != B.numel():
        return False
    n = C.c_ulonglong(0)
    with torch.cuda.device(A.device):
        check(lib.b200cp_allclose_count(_p(A), _p(B), A.numel(), C.c_float(tolerance), C.byref(n), _stream()))
    return n.value == 0


def cp4_conv2d_step(X, dU, FT, FC, FY, FX, pad=1, flags=0):
    """One training step on device tensors (``b200cp_cp4_step``): returns (U, dX, dK_packed); the work forward,
    backward-data and backward-filter share is done once."""
    return _C.cp4_step(X, dU, FT, FC, FY, FX, pad, flags)


def cp4_conv2d_forward_save(Input, FT, FC, FY, FX, pad=1, flags=0):
    """Forward that also returns its rank plane ``P = FC^T Input`` [N,R,H,W] (``b200cp_cp4_fwd_save``)."""
    return _C.cp4_forward_save(Input, FT, FC, FY, FX, pad, flags)


def cp4_conv2d_backward_data_save(Upstream, FT, FC, FY, FX, pad=1, flags=0):
    """Backward-data that also returns its rank plane ``Q = FT^T Upstream`` (``b200cp_cp4_bwd_data_save``)."""
    return _C.cp4_backward_data_save(Upstream, FT, FC, FY, FX, pad, flags)


def cp4_conv2d_backward_filter_saved(dLdO, In, P, Q, FT, FC, FY, FX, pad=1, flags=0):
    """The four factor gradients from the saved rank planes (``b200cp_cp4_bwd_filter_saved``)."""
    return _C.cp4_backward_filter_saved(dLdO, In, P, Q, FT, FC, FY, FX, pad, flags)


def cp4_conv2d_step_host(X, dU, FT, FC, FY, FX, pad=1, flags=0, out=None):
    """Forward + both backward passes through the host-buffer entry point
    (``b200cp_cp4_step_host``): CPU tensors in, CPU tensors out, transfers included.
    ``out`` may hold preallocated (pinned) ``(U, dX, dK_packed)``."""
    s = _host_shape(X, dU, FT, FC, FY, FX, pad, out)
    R = s.Rank
    if out is None:
        out = (torch.empty((s.N, s.T, s.H, s.W)), torch.empty((s.N, s.C, s.H, s.W)),
               torch.empty((s.T + s.C + s.Y + s.X) * R))
    U, dX, dK = out
    check(lib.b200cp_cp4_step_host(C.byref(s), _p(X), _p(dU), _p(FT), _p(FC), _p(FY), _p(FX), _p(U), _p(dX), _p(dK),
                                   flags))
    return U, dX, dK


def cp4_conv2d_step_host_submit(X, dU, FT, FC, FY, FX, out, pad=1, flags=0, slot=0):
    """Queue one step on ``slot`` (0 .. 3) through ``b200cp_cp4_step_host_submit``; ``out`` holds the pinned
    ``(U, dX, dK_packed)`` that ``cp4_conv2d_step_host_wait(slot)`` fills.  Inputs and outputs must stay
    alive and untouched until that wait returns."""
    s = _host_shape(X, dU, FT, FC, FY, FX, pad, out)
    U, dX, dK = out
    check(lib.b200cp_cp4_step_host_submit(C.byref(s), _p(X), _p(dU), _p(FT), _p(FC), _p(FY), _p(FX), _p(U), _p(dX),
                                          _p(dK), flags, slot))


def cp4_conv2d_step_host_wait(slot=0):
    """Block until the step queued on ``slot`` has its results in the host tensors."""
    check(lib.b200cp_cp4_step_host_wait(slot))


def device_status():
    """Synchronise and raise if a tensor-path kernel gave up a bounded wait (``b200cp_device_status``)."""
    check(lib.b200cp_device_status())


def set_band_rows(rows):
    """Test hook: force the band height of the row-band CP4 kernel (0: the planner chooses)."""
    lib.b200cp_test_set_band_rows(int(rows))


def set_band_tensor_loads(on):
    """Test hook: the row-band kernel loads its input with 4-D tensor-map boxes (True) or 1-D bulk copies (False)."""
    lib.b200cp_test_set_band_tensor_loads(1 if on else 0)


def set_band_tcgen05(on):
    """Test hook: the row-band kernel's output contraction on tcgen05 (True) or mma.sync (False, default)."""
    lib.b200cp_test_set_band_tcgen05(1 if on else 0)


def set_stream(on):
    """Test hook: the row-stream convolution kernel off (0 / False), on (1 / True) or as the environment says (-1)."""
    lib.b200cp_test_set_stream(int(on))


def debug_cp4_tc(Input, FT, FC, FY, FX, pad=1, terms=3, p_floats=0):
    """Diagnostic forward on the tensor path; also returns the first CTA's rank-R intermediate."""
    Input = _dev(Input, "Input")
    FT, FC, FY, FX = _factors4((FT, FC, FY, FX), Input)
    s = _shape_from(Input, FT, FC, FY, FX, pad)
    out = torch.empty((s.N, s.T, s.H, s.W), device=Input.device, dtype=torch.float32)
    P = torch.zeros(max(p_floats, 1), device=Input.device, dtype=torch.float32)
    with torch.cuda.device(Input.device):
        check(lib.b200cp_debug_cp4_tc(C.byref(s), _p(Input), _p(FT), _p(FC), _p(FY), _p(FX), _p(out),
                                      _p(P) if p_floats else None, terms, _stream()))
    return out, P


# ---- three-factor CP conv -----------------------------------------------------
def cp3_conv2d_forward(Input, KT, KCin, KC, pad=1, flags=0):
    """Three-factor CP conv (``b200cp_cp3_fwd``): ``KT [T,R]``, ``KCin [C,R]``, free core ``KC [Y,X,R]``."""
    return _C.cp3_forward(Input, KT, KCin, KC, pad, flags)


def cp3_conv2d_backward_data(Upstream, KT, KCin, KC, pad=1, flags=0):
    return _C.cp3_backward_data(Upstream, KT, KCin, KC, pad, flags)


def cp3_conv2d_backward_filter(dLdO, In, KT, KCin, KC, pad=1, flags=0):
    """Factor gradients (dKT, dKCin, dKC) of the three-factor CP conv; 3x3 cores with pad 1."""
    return _C.cp3_backward_filter(dLdO, In, KT, KCin, KC, pad, flags)


def conv2d_cp_fused_nchw(U, K0, K1, K2, flags=0):
    """``Conv2dCpFusedNchw`` (Kernels/cp_fused_nchw.cc): K0 [C,R], K1 [FH,FW,R], K2 [R,T], SAME padding
    (test/test_conv2d_cp.py:33-38)."""
    return cp3_conv2d_forward(U, K2.t().contiguous(), K0, K1, pad=(K1.shape[0] - 1) // 2, flags=flags)


# ---- TF custom-op order -----------------------------------------------------
def cp4_conv2d_nchw(U, K0, K1, K2, K3, flags=0):
    """``Cp4Conv2dNchw`` (Kernels/cp4_conv_nchw.cc:6-13): K0 [C,R], K1 [FH,R], K2 [FW,R], K3 [T,R],
    SAME padding (test/test_conv2d_cp4.py:25-33)."""
    return cp4_conv2d_forward(U, K3, K0, K1, K2, pad=(K1.shape[0] - 1) // 2, flags=flags)


def _modes(factors, what):
    a, b = [], []
    R = factors[0].shape[2]
    for k, f in enumerate(factors):
        if f.dim() != 3 or f.shape[2] != R:
            raise ValueError(f"{what}: kernel {k} must be [in, out, rank] with a common rank")
        a.append(f.shape[0])
        b.append(f.shape[1])
    return a, b, R


def conv2d_rcp_fused_nchw(U, *kernels, flags=0):
    """``Conv2dRcpFusedNchw`` (Kernels/rcp_fused_nchw.cc:6-12): ``(U[N,S0..,H,W], K0[S0,T0,R], ..., KC[FH,FW,R])``
    -> ``V[N,T0..,H,W]``.  ``U`` may also be given as [N,C,H,W]."""
    return _C.rcp_forward(flags, U, kernels[-1], *kernels[:-1])


def rcp_conv2d_backward(U, dV, *kernels, flags=0, need_dx=True, need_dw=True):
    """Gradients of ``conv2d_rcp_fused_nchw``: (dU, [dK_k], dKC)."""
    return _C.rcp_backward(flags, need_dx, need_dw, U, dV, kernels[-1], *kernels[:-1])


def dense_cp(U, *kernels, flags=0):
    """``DenseCp`` (Kernels/dense_cp.cc:6-12): ``(U[N,S0,S1,..], K0[S0,T0,R], ...)`` -> ``V[N,T0,T1,..]``
    (output dims are ``kernel_k.dim(1)``, Kernels/dense_cp.cc:86-91).  ``U`` may also be [N, I]."""
    return _C.dense_forward(flags, U, *kernels)


def dense_cp_backward(U, dV, *kernels, flags=0, need_dx=True, need_dw=True):
    """Gradients of ``dense_cp``: (dU, [dK_k])."""
    return _C.dense_backward(flags, need_dx, need_dw, U, dV, *kernels)


# ---- the reference's "rebuild" variants: the undecomposed layer with the recomposed weight --------------------

def conv2d_dense_forward(Input, K, pad=1):
    """Ordinary conv2d with a dense filter ``K [T,C,Y,X]``, H x W output: the ``tf.nn.conv2d(U, K, ..., 'SAME')`` of
    test/benchmark_conv2d_cp4.py:41."""
    Input = _dev(Input, "Input")
    K = _dev(K, "K", Input)
    if Input.dim() != 4 or K.dim() != 4 or K.shape[1] != Input.shape[1]:
        raise ValueError("K must be [T, C, Y, X] with C the input's channel count")
    s = tensor_shape(Input.shape[0], Input.shape[1], Input.shape[2], Input.shape[3], K.shape[0], K.shape[2],
                     K.shape[3], 1, pad)
    U = torch.empty((s.N, s.T, s.H, s.W), device=Input.device, dtype=torch.float32)
    with torch.cuda.device(Input.device):
        wsb = lib.b200cp_conv2d_dense_fwd_workspace_bytes(C.byref(s))
        ws = torch.empty(max(wsb, 4) // 4, device=Input.device, dtype=torch.float32)
        check(lib.b200cp_conv2d_dense_fwd(C.byref(s), _p(Input), _p(K), _p(U), _p(ws), ws.numel() * 4, _stream()))
    return U


def cp4_conv2d_rebuild_forward(Input, FT, FC, FY, FX, pad=1):
    """The CP4 layer's "rebuild" line (test/benchmark_conv2d_cp4.py:35-42): ``cp4recom`` then an ordinary conv2d."""
    Input = _dev(Input, "Input")
    FT, FC, FY, FX = _factors4((FT, FC, FY, FX), Input)
    s = _shape_from(Input, FT, FC, FY, FX, pad)
    U = torch.empty((s.N, s.T, s.H, s.W), device=Input.device, dtype=torch.float32)
    with torch.cuda.device(Input.device):
        wsb = lib.b200cp_cp4_rebuild_fwd_workspace_bytes(C.byref(s))
        ws = torch.empty(max(wsb, 4) // 4, device=Input.device, dtype=torch.float32)
        check(lib.b200cp_cp4_rebuild_fwd(C.byref(s), _p(Input), _p(FT), _p(FC), _p(FY), _p(FX), _p(U), _p(ws),
                                         ws.numel() * 4, _stream()))
    return U


def rcp_recompose(*kernels):
    """Dense filter ``[T, C, FH, FW]`` of the reshaped-CP conv from ``(K0[S0,T0,R], ..., KC[FH,FW,R])``."""
    *A, KC = kernels
    KC = _dev(KC, "kernelc")
    A = [_dev(a, f"kernel{k}", KC) for k, a in enumerate(A)]
    cd, td, R = _modes(A, "rcp_recompose")
    if KC.dim() != 3 or KC.shape[2] != R:
        raise ValueError("kernelc must be [FH, FW, rank]")
    Cc, Tc = 1, 1
    for c, t in zip(cd, td):
        Cc *= c
        Tc *= t
    K = torch.empty((Tc, Cc, KC.shape[0], KC.shape[1]), device=KC.device, dtype=torch.float32)
    with torch.cuda.device(KC.device):
        check(lib.b200cp_rcp_recompose(len(A), int_array(cd), int_array(td), R, KC.shape[0], KC.shape[1],
                                       ptr_array([a.data_ptr() for a in A]), _p(KC), _p(K), _stream()))
    return K


def conv2d_rcp_rebuild_nchw(U, *kernels):
    """The reshaped-CP layer's "rebuild" line: recompose the filter, then an ordinary same-size conv2d."""
    K = rcp_recompose(*kernels)
    U = _dev(U, "input")
    N, H, W = U.shape[0], U.shape[-2], U.shape[-1]
    return conv2d_dense_forward(U.reshape(N, K.shape[1], H, W), K, pad=(K.shape[2] - 1) // 2)


def dense_cp_recompose(*kernels):
    """``M [I, O]`` of the CP dense layer (the einsum + reshape of test/benchmark_dense_cp.py:43-44)."""
    Fk = [_dev(f, f"kernel{k}", kernels[0]) for k, f in enumerate(kernels)]
    idims, odims, R = _modes(Fk, "dense_cp_recompose")
    I, O = 1, 1
    for a, b in zip(idims, odims):
        I *= a
        O *= b
    M = torch.empty((I, O), device=Fk[0].device, dtype=torch.float32)
    with torch.cuda.device(M.device):
        wsb = lib.b200cp_dense_recompose_workspace_bytes(len(Fk), int_array(idims), int_array(odims), R)
        ws = torch.empty(max(wsb, 4) // 4, device=M.device, dtype=torch.float32)
        check(lib.b200cp_dense_recompose(len(Fk), int_array(idims), int_array(odims), R,
                                         ptr_array([f.data_ptr() for f in Fk]), _p(M), _p(ws), ws.numel() * 4,
                                         _stream()))
    return M


def dense_matmul(U, M):
    """``U [B, I] @ M [I, O]`` with fp32-grade results (test/benchmark_dense_cp.py:45-48)."""
    U = _dev(U, "input")
    M = _dev(M, "M", U)
    B = U.shape[0]
    I, O = M.shape
    if U.numel() != B * I:
        raise ValueError("input size does not match M")
    Y = torch.empty((B, O), device=U.device, dtype=torch.float32)
    with torch.cuda.device(U.device):
        wsb = lib.b200cp_dense_matmul_workspace_bytes(B, I, O)
        ws = torch.empty(max(wsb, 4) // 4, device=U.device, dtype=torch.float32)
        check(lib.b200cp_dense_matmul(B, I, O, _p(U), _p(M), _p(Y), _p(ws), ws.numel() * 4, _stream()))
    return Y


def dense_cp_rebuild(U, *kernels):
    """The CP dense layer's "rebuild" line: recompose ``M``, then one matmul."""
    return dense_matmul(U, dense_cp_recompose(*kernels))


# ---- autograd wrappers ----------------------------------------------------------
# The nodes are native (csrc/torch_binding.cpp); each class keeps the ``apply`` its layer calls.
class CP4Conv2dFunction:
    """y = CP4 conv2d(x; FT, FC, FY, FX) with the fused backward kernels: ``apply(x, FT, FC, FY, FX, pad=1, flags=0)``."""
    apply = staticmethod(_C.cp4_apply)


class CP3Conv2dFunction:
    """y = three-factor CP conv2d(x; KT, KCin, KC) with the fused backward kernels: ``apply(x, KT, KCin, KC, pad=1)``."""
    apply = staticmethod(_C.cp3_apply)


class RCPConv2dFunction:
    """y = reshaped-CP conv2d(x; A..., KC): ``apply(x, KC, K0, K1, ...)``."""
    apply = staticmethod(_C.rcp_apply)


class CPDenseFunction:
    """y = CP dense(x; F...): ``apply(x, K0, K1, ...)``."""
    apply = staticmethod(_C.dense_apply)
