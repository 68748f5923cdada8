"""Host-side mirror of the reference's Conv / Gemm / MatMul operator calls for device tensors.

Each function builds the ``params / inputs / outputs`` arrays the way the reference host does
(host/op.h:109-168, host/ops/conv.h:133-157) around torch CUDA tensors (used for device memory
only) and calls the ``eval`` symbol of the drop-in library ``lib<Op>_cu.so``.  Shapes and
layouts are the reference's: NCHW fp32 activations, OIHW weights, [N][K] Gemm weights.

The descriptors a call passes depend on its shapes and options alone, so a bounded table keeps the
``params`` array of each combination of whole numbers (building the ctypes records anew took a fifth of a
small call); the libraries only read them.  Other options (a clip range, a slope: floats, lists, arrays) are
written anew each time.  Pointers go into fresh ``inputs`` / ``outputs`` arrays per call.
"""
import functools

import numpy as np
import torch

from . import abi, capi

_Slots = abi.BUFFER_INFO_S * abi.BUF_MAXNUM
_LUT_SLOT = abi.BUF_MAXNUM - 1


def _dev(a, dtype=torch.float32):
    if isinstance(a, torch.Tensor):
        if a.dtype is dtype and a.is_contiguous() and a.get_device() == torch.cuda.current_device():
            return a
        return a.to("cuda", dtype).contiguous()
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda").to(dtype).contiguous()


def out_hw(H, W, KH, KW, strides, pads):
    return ((H + pads[0] + pads[2] - KH) // strides[1] + 1, (W + pads[1] + pads[3] - KW) // strides[0] + 1)


def _conv_args(x_shape, w_shape, strides, pads, has_bias, act, **cfg_kw):
    """(output shape, params holder) of one conv."""
    N, _, H, W = x_shape
    OC, _, KH, KW = w_shape
    y_shape = (N, OC) + out_hw(H, W, KH, KW, strides, pads)
    cfg = abi.conv_cfg((KH, KW), strides, pads, has_bias=has_bias, act=act, **cfg_kw)
    return y_shape, abi.conv_eval_args(cfg, x_shape, w_shape, y_shape, 0, 0, 0, 0, abi.default_useful_info())


_conv_plan = functools.lru_cache(maxsize=256)(_conv_args)


def _whole(values):
    """Plain whole numbers only: equal keys then write equal records (2.0 == 2, True == 1 and -0.0 == 0.0 would not)."""
    return all(type(v) is int for v in values)


@functools.lru_cache(maxsize=256)
def _gemm_plan(a_shape, w_shape):
    y_shape = (a_shape[-2], w_shape[0])
    return y_shape, abi.gemm_eval_args(a_shape, w_shape, y_shape, 0, 0, 0, 0)


@functools.lru_cache(maxsize=256)
def _matmul_plan(a_shape, b_shape):
    y_shape = a_shape[:-1] + (b_shape[-1],)
    return y_shape, abi.matmul_eval_args(a_shape, b_shape, y_shape, 0, 0, 0)


def _call(op, plan, y_shape, x, w, b=None, lut=None):
    y = torch.empty(y_shape, dtype=torch.float32, device="cuda")
    inputs, outputs = _Slots(), _Slots()
    inputs[0].addr = x.data_ptr()
    inputs[1].addr = w.data_ptr()
    if b is not None:
        inputs[2].addr = b.data_ptr()
    if lut is not None:
        inputs[_LUT_SLOT].addr = lut.data_ptr()
    outputs[0].addr = y.data_ptr()
    capi.check(capi.shim_eval(op)(plan.params, inputs, outputs))
    return y


def conv(x, w, b, strides=(1, 1), pads=(0, 0, 0, 0), act=abi.NOT_ACT, int8=None, lut=None, **cfg_kw):
    """Conv through ``libConv_cu.so:eval``.  ``int8=(input_scale, weight_aux)``: ``w`` is the
    int8 OIHW weight and ``b`` the int32 bias, placed at the start of fp32-sized buffers as the
    reference's quantiser leaves them (tools/optimize/model_quant.hpp:6-29)."""
    xd = _dev(x)
    lutd = _dev(lut) if lut is not None else None
    if int8 is None:
        wd = _dev(w)   # depthwise: pass group=C in cfg_kw, weight [C][1][KH][KW]
        bd = _dev(b) if b is not None else None
        strides, pads = tuple(strides), tuple(pads)
        plan_of = _conv_plan if _whole((*strides, *pads, act, *cfg_kw.values())) else _conv_args
        y_shape, plan = plan_of(tuple(xd.shape), tuple(wd.shape), strides, pads, b is not None, act, **cfg_kw)
        return _call("Conv", plan, y_shape, xd, wd, bd, lutd)
    wd = torch.zeros(int(np.prod(w.shape)), dtype=torch.float32, device="cuda")
    wd.view(torch.int8)[: wd.numel()] = _dev(np.asarray(w, np.int8).ravel(), torch.int8)
    bd = None
    if b is not None:
        bd = _dev(np.asarray(b, np.int32), torch.int32)
    y_shape, plan = _conv_args(tuple(xd.shape), tuple(w.shape), strides, pads, b is not None, act, int8_scale=int8[0], weight_aux=int8[1], **cfg_kw)
    return _call("Conv", plan, y_shape, xd, wd, bd, lutd)


def gemm(a, w, b):
    ad, wd, bd = _dev(a), _dev(w), _dev(b)
    y_shape, plan = _gemm_plan(tuple(ad.shape), tuple(wd.shape))
    return _call("Gemm", plan, y_shape, ad, wd, bd)


def matmul(a, b):
    ad, bd = _dev(a), _dev(b)
    y_shape, plan = _matmul_plan(tuple(ad.shape), tuple(bd.shape))
    return _call("MatMul", plan, y_shape, ad, bd)
