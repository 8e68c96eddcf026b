"""Fused AdamW over flat buckets (one CUDA kernel per bucket, csrc/ops/fused_adamw.cu)."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _ext
from .. import _lib as L


def launches() -> int:
    """Number of fused optimizer kernels launched by this process so far."""
    return _ext.load().launches("optim")


def fused_adamw_(param: torch.Tensor, master: torch.Tensor, exp_avg: torch.Tensor, exp_avg_sq: torch.Tensor,
                 grad: torch.Tensor, *, lr: float, betas=(0.9, 0.95), eps: float = 1e-8, weight_decay: float = 0.0,
                 grad_scale: float = 1.0, step: int = 1, zero_grad: bool = True, norm_sq: torch.Tensor | None = None,
                 max_norm: float = 0.0, stream=None, hyper: torch.Tensor | None = None) -> None:
    """In-place AdamW step on flat tensors: bf16 `param`/`grad`, fp32 `master`/`exp_avg`/`exp_avg_sq`.  With `hyper` (three
    fp32 values on the device: lr, 1 - beta1^t, sqrt(1 - beta2^t)) the kernel reads the schedule when it runs instead of
    taking `lr` and `step` from this call, which is what a launch recorded in a CUDA graph needs."""
    rc = _ext.load().adamw(param, master, exp_avg, exp_avg_sq, grad, lr, betas[0], betas[1], eps, weight_decay, grad_scale, step, zero_grad,
                           norm_sq, max_norm, stream.cuda_stream if stream is not None else None, hyper)
    if rc == L.SUCCESS:
        return
    if not param.is_cuda:
        raise RuntimeError("fused_adamw_ needs CUDA tensors (the kernel is sm_100a code)")
    assert param.dtype == torch.bfloat16 and grad.dtype == torch.bfloat16
    assert master.dtype == exp_avg.dtype == exp_avg_sq.dtype == torch.float32
    n = param.numel()
    assert master.numel() == n and grad.numel() == n and exp_avg.numel() == n and exp_avg_sq.numel() == n
    assert hyper is None or (hyper.is_cuda and hyper.dtype == torch.float32 and hyper.numel() >= 3)
    L.check(rc if rc > 0 else L.INVALID_ARGUMENT, "mcclFusedAdamWDeviceHyper" if hyper is not None else "mcclFusedAdamW")


def sum_squares_(x: torch.Tensor, out: torch.Tensor, scratch: torch.Tensor, accumulate: bool = False, stream=None) -> None:
    """out (one fp32 on the device) = [out +] sum(x**2) for a flat bf16 tensor; `scratch` is fp32 work memory
    (see scratch_floats) whose first element is zero."""
    rc = _ext.load().sum_squares(x, out, scratch, accumulate, stream.cuda_stream if stream is not None else None)
    if rc == L.SUCCESS:
        return
    assert x.is_cuda and x.dtype == torch.bfloat16 and out.dtype == torch.float32 and scratch.dtype == torch.float32
    L.check(rc if rc > 0 else L.INVALID_ARGUMENT, "mcclSumSquaresBf16")


def scratch_floats(n: int) -> int:
    lib = L.load()
    lib.mcclSumSquaresScratchFloats.restype = C.c_uint64
    lib.mcclSumSquaresScratchFloats.argtypes = [C.c_uint64]
    return int(lib.mcclSumSquaresScratchFloats(n))


def adamw_reference(master, exp_avg, exp_avg_sq, grad, *, lr, betas, eps, weight_decay, grad_scale, step):
    """Plain PyTorch fp32 restatement of the kernel, for tests."""
    g = grad.float() * grad_scale
    exp_avg.mul_(betas[0]).add_(g, alpha=1 - betas[0])
    exp_avg_sq.mul_(betas[1]).addcmul_(g, g, value=1 - betas[1])
    bc1 = 1 - betas[0] ** step
    bc2 = 1 - betas[1] ** step
    denom = exp_avg_sq.sqrt() / (bc2 ** 0.5) + eps
    master.mul_(1 - lr * weight_decay).addcdiv_(exp_avg, denom, value=-lr / bc1)
    return master.to(torch.bfloat16)
