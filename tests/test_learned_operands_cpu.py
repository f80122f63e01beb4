"""What the learned preconditioner's training step hands to its residual kernel: the
operands that ``y - target`` and ``scale`` took as tensor expressions, as plain buffers."""

import pytest
import torch

from thick_ptycho_b200.learned import LearnedPreconditioner

V, N = 3, 5
Z = torch.complex(torch.randn(V, N), torch.randn(V, N))
CPU = torch.device("cpu")


def operands(target=Z, scale=torch.ones(V), z=Z, device=CPU):
    return LearnedPreconditioner._residual_operands(z, target, scale, device)


@pytest.mark.parametrize("target", [
    Z, Z.conj(), Z.real, Z[:1], Z[:, :1], Z.real.double(), torch.tensor(2.0), 0.0, 1 + 2j, Z.to(torch.complex128),
    Z.T.contiguous().T, Z.conj().imag,
])
@pytest.mark.parametrize("scale", [torch.rand(V), torch.rand(1), torch.rand(V).half(), torch.rand(V).double(),
                                   torch.arange(V), torch.rand(2 * V)[::2], Z[:, 0].conj().imag])
def test_operands_are_the_values(target, scale):
    z, t, s = operands(target, scale)
    for x, dtype in ((z, torch.complex64), (t, torch.complex64), (s, torch.float32)):
        assert x.dtype == dtype and x.is_contiguous() and not x.is_conj() and not x.is_neg()
    assert z.shape == t.shape == (V, N) and s.shape == (V,)
    assert torch.equal(z - t, (Z - target).to(torch.complex64))
    assert torch.equal(s, (torch.ones(V) * scale).to(torch.float32))


def test_conjugated_input():
    assert torch.equal(operands(z=Z.conj())[0], torch.complex(Z.real, -Z.imag))


@pytest.mark.parametrize("kw", [
    {"target": Z.to("meta")}, {"scale": torch.ones(V, device="meta")}, {"z": Z.to("meta")},
    {"target": Z[:2]}, {"scale": torch.ones(2)}, {"scale": torch.tensor(1.0)}, {"scale": torch.ones(V, 1)},
    {"scale": torch.ones(V, dtype=torch.complex64)}, {"z": Z.to(torch.complex128)},
])
def test_refused(kw):
    with pytest.raises((RuntimeError, TypeError)):
        operands(**kw)
