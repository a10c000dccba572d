"""What stays with torch.linalg.eigh: function transforms, forward-mode differentiation, tracing, and matrices whose memory
holds their negative."""
import pytest
import torch
import torch.autograd.forward_ad as forward_ad

from dftbaby_b200 import eigen

pytestmark = pytest.mark.gpu


def _matrix(*shape):
    g = torch.Generator(device="cuda").manual_seed(len(shape))
    A = torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)
    return A + A.mT


def test_vmap():
    A = _matrix(3, 6, 6)
    w, _ = torch.vmap(eigen.eigh)(A)
    assert torch.allclose(w, torch.linalg.eigvalsh(A), rtol=0, atol=1e-13)


def test_forward_mode():
    A = _matrix(6, 6)
    with forward_ad.dual_level():
        w, _ = eigen.eigh(forward_ad.make_dual(A, torch.eye(6, dtype=A.dtype, device="cuda")))
        tangent = forward_ad.unpack_dual(w).tangent
    assert tangent is not None and torch.allclose(tangent, torch.ones_like(tangent))
    _, tangent = torch.func.jvp(lambda X: eigen.eigh(X)[0], (A,), (torch.eye(6, dtype=A.dtype, device="cuda"),))
    assert torch.allclose(tangent, torch.ones_like(tangent))


def test_tracing():
    from torch.fx.experimental.proxy_tensor import make_fx
    traced = make_fx(lambda X: eigen.eigh(X)[0])(_matrix(6, 6))
    A = _matrix(6, 6) + 2.0
    assert torch.allclose(traced(A), torch.linalg.eigvalsh(A), rtol=0, atol=1e-12)


def test_negative_bit():
    A = torch.complex(torch.zeros(6, 6, dtype=torch.float64, device="cuda"), _matrix(6, 6)).conj().imag
    assert A.is_neg()
    w, _ = eigen.eigh(A)
    assert torch.allclose(w, torch.linalg.eigvalsh(A.resolve_neg()), rtol=0, atol=1e-13)
