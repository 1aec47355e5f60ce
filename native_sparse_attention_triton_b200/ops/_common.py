"""Helpers shared by the Python code that calls the C interface directly (inference step, KV cache)."""
import torch

from .. import _lib


def dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return _lib.DTYPE_BF16
    if t.dtype == torch.float16:
        return _lib.DTYPE_FP16
    raise AssertionError("only bfloat16 and float16 tensors are supported")


def stream_ptr(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


def require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError("native_sparse_attention_triton_b200 ops run on CUDA tensors only (no CPU path)")


def inner_contiguous(t: torch.Tensor) -> torch.Tensor:
    """Kernels need a unit innermost stride, 16-byte aligned rows; copy only when that does not hold."""
    ok = t.stride(-1) == 1 and t.data_ptr() % 16 == 0 and all(s % 8 == 0 for s in t.stride()[:-1])
    return t if ok else t.contiguous()
