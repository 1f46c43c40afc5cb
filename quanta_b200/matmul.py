"""Dense projections (``nn.Linear`` in the reference, src/quanta/minimax/attention.py:166-169): products of a few rows by the framework's
own kernels (``csrc/linear_few.cu`` in bfloat16, ``csrc/linear_rows.cu`` in float32), the others by the library's (cuBLAS via torch).

float32 products run as true float32: TF32 and reduced-precision accumulation are switched off
process-wide when the first engine is built.
"""

from __future__ import annotations

import torch
import torch.autograd.forward_ad as forward_ad
from torch.utils._python_dispatch import _get_current_dispatch_mode

from . import kernels

_configured = False


def configure() -> None:
    global _configured
    if _configured:
        return
    torch.backends.cuda.matmul.allow_tf32 = False
    torch.backends.cudnn.allow_tf32 = False
    torch.set_float32_matmul_precision("highest")
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    _configured = True


# The library's kernels for products of fewer rows than this (of matrices that the kernel for few rows does not take) are slower than its
# kernel for this many (measured on B200, weights from HBM: 3072 x 6144 at 8 rows 37 us, at 32 rows 27 us), so activations of
# small steps are laid out with spare rows and multiplied as MIN_ROWS rows.  Rows do not mix in a
# product: what the spare rows hold never reaches a real row.
MIN_ROWS = 32


def empty_rows(n: int, *cols: int, dtype: torch.dtype, device) -> torch.Tensor:
    """``[n, *cols]`` uninitialised, as the first rows of a buffer of at least MIN_ROWS rows, which
    ``linear`` finds again by the size of the storage."""
    return torch.empty((max(n, MIN_ROWS), *cols), dtype=dtype, device=device)[:n]


def _with_spare_rows(x: torch.Tensor) -> torch.Tensor:
    n, k = x.shape
    if (0 < n < MIN_ROWS and x.is_cuda and x.is_contiguous() and x.storage_offset() == 0
            and x.untyped_storage().nbytes() >= MIN_ROWS * k * x.element_size()):
        return torch.as_strided(x, (MIN_ROWS, k), (k, 1))
    return x


def _plain(x: torch.Tensor, w: torch.Tensor) -> bool:
    """Whether nothing hangs on the product besides its numbers, on the current device.  What torch does with its own product besides
    computing it (gradients, forward mode, vmap, autocast, tracing, the errors of operands that do not fit) stays with torch."""
    if type(x) is not torch.Tensor or type(w) not in (torch.Tensor, torch.nn.Parameter) or _get_current_dispatch_mode() is not None:
        return False
    if torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.is_autocast_enabled("cuda") or forward_ad._current_level >= 0:
        return False
    if any(torch._C._functorch.is_functorch_wrapped_tensor(t) for t in (x, w)):
        return False
    if torch.is_grad_enabled() and (x.requires_grad or w.requires_grad):
        return False
    return (x.is_cuda and w.device == x.device and x.device.index == torch.cuda.current_device() and x.dim() == 2 and w.dim() == 2
            and x.shape[1] == w.shape[1] and x.is_contiguous() and w.is_contiguous())


def _few_float32_rows(x: torch.Tensor, w: torch.Tensor, out_dtype: torch.dtype | None) -> bool:
    """Whether ``kernels.linear_rows`` takes the product: a few float32 rows, bound by the bytes of ``w``."""
    if x.dtype != torch.float32 or w.dtype != torch.float32 or out_dtype not in (None, torch.float32) or not _plain(x, w):
        return False
    return (0 < x.shape[0] <= (kernels.LINEAR_ROWS_MAX if x.shape[1] <= 8192 else 8) and x.shape[1] > 0 and x.shape[1] % 4 == 0
            and x.data_ptr() % 16 == 0 and w.data_ptr() % 16 == 0)


def _few_bfloat16_rows(x: torch.Tensor, w: torch.Tensor, out_dtype: torch.dtype | None) -> bool:
    """Whether ``kernels.linear_few`` takes the product: a few bfloat16 rows, bound by the bytes of ``w``."""
    if (x.dtype != torch.bfloat16 or w.dtype != torch.bfloat16 or out_dtype not in (None, torch.bfloat16, torch.float32)
            or x.dim() != 2 or x.shape[0] > kernels.LINEAR_FEW_MAX or not _plain(x, w)):
        return False
    return x.data_ptr() % 32 == 0 and w.data_ptr() % 32 == 0 and kernels.linear_few_takes(x.shape[0], x.shape[1], w.shape[0])


def linear(x: torch.Tensor, w: torch.Tensor, out_dtype: torch.dtype | None = None, ctx=None) -> torch.Tensor:
    """``x [T, in] @ w [out, in].T``; accumulation is float32; ``out_dtype`` float32 keeps the
    accumulator's precision for bfloat16 operands.  An ``x`` from ``empty_rows`` is multiplied with its
    spare rows and the result cut back to ``T`` rows.  ``ctx``: the step's context, given where the launch before is
    short and leaves the memory idle; where it says that the weights are settled (``StepContext.settled``), the kernel for few rows
    starts to read them before that launch has ended."""
    n = x.shape[0]
    if _few_bfloat16_rows(x, w, out_dtype):
        out = torch.empty((n, w.shape[0]), dtype=out_dtype or x.dtype, device=x.device)
        kernels.linear_few(x, w, out, early=getattr(ctx, "settled", False))
        return out
    if _few_float32_rows(x, w, out_dtype):
        out = torch.empty((n, w.shape[0]), dtype=torch.float32, device=x.device)
        kernels.linear_rows(x, w, out)
        return out
    xp = _with_spare_rows(x)
    if xp is not x:
        return linear(xp, w, out_dtype, ctx)[:n]
    if out_dtype is not None and out_dtype != x.dtype:
        return torch.mm(x, w.t(), out_dtype=out_dtype)
    return torch.mm(x, w.t())


def linear_silu(x: torch.Tensor, w: torch.Tensor, ctx=None) -> torch.Tensor | None:
    """``silu(x @ w[:I].T) * (x @ w[I:].T)`` of a few bfloat16 rows in one launch, both products rounded to bfloat16 first; None where
    ``linear`` would not take its kernel for few rows."""
    if w.dim() != 2 or w.shape[0] % 2 or not _few_bfloat16_rows(x, w, None):
        return None
    out = empty_rows(x.shape[0], w.shape[0] // 2, dtype=torch.bfloat16, device=x.device)
    kernels.linear_few_silu(x, w, out, early=getattr(ctx, "settled", False))
    return out
