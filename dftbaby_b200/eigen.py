"""Symmetric eigensolver of the SCC and of the projected problems: the library's own one-launch kernel for small FP64
matrices on the GPU, torch.linalg.eigh for all others."""
import torch
import torch.autograd.forward_ad as forward_ad

from . import native

SMALL = 128  # largest matrix of dftb_small_eigh: its orthogonal factor fills one SM's shared memory


def _watched():
    """Inside vmap and the other function transforms, forward-mode differentiation or tracing: the values in memory are not
    all that a call has to hand on, so it belongs to torch."""
    return (torch._C._functorch.peek_interpreter_stack() is not None or forward_ad._current_level >= 0
            or torch._C._len_torch_dispatch_stack() > 0 or torch.jit.is_tracing())


def small(A):
    """True for matrices (or batches of them) that dftb_small_eigh takes; autograd, function transforms, tracing and other
    devices than the current one stay with torch."""
    return (type(A) is torch.Tensor and A.is_cuda and A.dtype == torch.float64 and A.dim() in (2, 3)
            and 0 < A.shape[-1] <= SMALL and A.shape[-2] == A.shape[-1] and A.shape[0] > 0
            and A.get_device() == torch.cuda.current_device() and not (A.requires_grad and torch.is_grad_enabled())
            and not A.is_neg() and not _watched())


def small_eigh(A):
    """(eigenvalues, eigenvectors, status per matrix), the lower triangles being read; nothing is synchronised."""
    n = A.shape[-1]
    batch = A.shape[0] if A.dim() == 3 else 1
    w = torch.empty(A.shape[:-1], dtype=A.dtype, device=A.device)
    V = torch.empty(A.shape, dtype=A.dtype, device=A.device)
    info = torch.empty(batch, dtype=torch.int32, device=A.device)
    native.call("dftb_small_eigh", n, batch, native.ptr(A), A.stride(0) if A.dim() == 3 else 0, A.stride(-2), A.stride(-1),
                native.ptr(w), native.ptr(V), native.ptr(info), native.stream())
    return w, V.mT, info


def eigh(A):
    """torch.linalg.eigh(A).  The kernel is the faster one at every size it takes (B200: 0.08 and 0.16 ms at n = 5, 0.39
    and 2.11 ms at n = 128; a batch of 256 at n = 128 0.75 and 3.28 ms); one SM holds no larger matrix."""
    if not small(A):
        return torch.linalg.eigh(A)
    w, V, info = small_eigh(A)
    if bool(info.any()):
        raise torch.linalg.LinAlgError("linalg.eigh: " + ("the input matrix contains non-finite values" if bool(
            (info == 1).any()) else "the eigenvalues did not converge"))
    return w, V
