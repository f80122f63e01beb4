"""Register and in-place transforms at the lengths where their plans change: the 2D
and 3D multislice marches and their adjoints against complex128 NumPy, and the
parallel-in-time z-transforms.

Tolerances: a multislice slice adds FFT round-off (4e-7 relative, two transforms) to
an update |H - 1| |psi| <= 2 |psi| and two roundings of psi, so L slices stay below
L * 1e-6 of the field; the adjoint's transmission gradient, a product of the two
fields, below 2 L * 1e-6.  The space-time solve stops at a 1e-6 residual: 1e-5.
Long marches of white noise: a transform pair's roundings (1e-7 relative, 1.4e-7 on two
axes) add up like their square root over the slices; what the constants and twiddles are
off, the same in every slice, may add 3e-9 per slice and axis.
"""

import numpy as np
import pytest

from oracle import pwe_oracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from thick_ptycho_b200 import SimulationGeometry  # noqa: E402
from thick_ptycho_b200.ms2d import MS2D  # noqa: E402
from thick_ptycho_b200.ms3d import MS3D  # noqa: E402
from thick_ptycho_b200.pit import PWEGpuPiTSolver  # noqa: E402

K = 4 * np.pi
L = 5


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x).astype(np.complex64)).cuda()


def check_march(eng, H, T, probes, src, axes):
    """Forward fields, exits and the adjoint's gradient for T (L, ...) and H (...)."""
    P, shape = probes.shape[0], probes.shape[1:]
    N = int(np.prod(shape))
    u, psi = [probes], probes
    for z in range(L):
        psi = np.fft.ifftn(H * np.fft.fftn(psi * T[z], axes=axes), axes=axes)
        u.append(psi)
    u = np.stack(u, 1)
    lam, grad = src, np.zeros_like(T)
    for z in reversed(range(L)):
        g = np.fft.ifftn(H.conj() * np.fft.fftn(lam, axes=axes), axes=axes)
        grad[z] = np.sum(g * np.conj(T[z] * u[:, z]), 0)
        lam = np.conj(T[z]) * g
    t1 = dev((T - 1).reshape(L, N))
    st = torch.empty((P, L + 1, N), dtype=torch.complex64, device="cuda")
    ex = torch.empty((P, N), dtype=torch.complex64, device="cuda")
    pr = dev(probes.reshape(P, *shape))
    eng.march(t1, pr, u_store=st, exit_out=ex)
    assert rel(st.cpu().numpy().reshape(u.shape), u) < L * 1e-6
    assert torch.equal(ex, st[:, -1])
    ex2 = torch.empty_like(ex)
    eng.march(t1, pr, exit_out=ex2)
    assert torch.equal(ex, ex2)
    gt = torch.zeros((L, N), dtype=torch.complex64, device="cuda")
    eng.backward(t1, st, dev(src.reshape(P, *shape)), gt)
    assert rel(gt.cpu().numpy().reshape(T.shape), grad) < 2 * L * 1e-6


@pytest.mark.parametrize("n,P", [
    (512, 2), (1024, 3), (2048, 1), (4096, 2),  # three register steps
    (12, 3), (18, 5), (25, 2), (36, 3), (128, 4), (243, 3), (256, 2), (270, 2), (625, 2), (960, 5), (1000, 3),
    (1250, 2), (1296, 2), (1500, 3), (1536, 2), (2000, 1), (3000, 2), (3125, 1), (4050, 1),
])
def test_ms2d_lengths(n, P):
    rng = np.random.default_rng(n)
    T = np.exp(1j * 0.02 * rng.standard_normal((L, n)) - 0.01 * rng.random((L, n)))
    check_march(MS2D(n, L + 1, K, 1.0, 1.0), po.ms_kernel(n, 1.0, K, 1.0), T, cplx(rng, P, n), cplx(rng, P, n), (-1,))


@pytest.mark.parametrize("n1,n2,P", [
    (64, 64, 2), (128, 192, 2), (192, 64, 1), (256, 128, 1),  # both axes in registers
    (64, 96, 2), (150, 128, 2), (48, 45, 3), (75, 90, 2), (200, 150, 1), (250, 16, 2), (15, 512, 1),
])
def test_ms3d_lengths(n1, n2, P):
    rng = np.random.default_rng(n1 + n2)
    T = np.exp(1j * 0.02 * rng.standard_normal((L, n1, n2)) - 0.01 * rng.random((L, n1, n2)))
    H = po.ms_kernel_3d(n1, n2, 1.0, 0.8, K, 1.0)
    check_march(MS3D(n1, n2, L + 1, K, 1.0, 0.8, 1.0), H, T, cplx(rng, P, n1, n2), cplx(rng, P, n1, n2), (-2, -1))


@pytest.mark.parametrize("N,nz,P", [
    (97, 33, 3), (64, 60, 2), (260, 130, 2), (33, 257, 9), (600, 70, 1), (40, 513, 2), (24, 1500, 1),
])
def test_pit_block_and_z_lengths(N, nz, P):
    """z-transforms of 64 .. 4096, block solves of one and of several warps' rows, odd sizes."""
    k = 2 * np.pi / 0.5
    rng = np.random.default_rng(N)
    n = 1 - 1e-3 * (rng.standard_normal((N, nz)) + 0.1j * rng.standard_normal((N, nz)))
    x = np.arange(N)[None]
    probes = np.exp(-((x - rng.uniform(0.3 * N, 0.7 * N, (P, 1))) ** 2) / 50.0).astype(complex)
    geo = SimulationGeometry(dimension=2, nx=N, nz=nz, dx=1.0, dz=1.0, k=k, num_probes=P)
    u = PWEGpuPiTSolver(geo, probes[None], bc_type="impedance").solve(n=n)[0, 0]
    co = po.bc_coefficients(k, 1.0, 1.0, bc_type="impedance")
    A, B = po.step_matrices_1d(N, co, "impedance", 1.0)
    C = po.object_contribution(n, k, 1.0)
    for p in range(P):
        ref = po.full_system_solve(A, B, C, po.pit_rhs(B, probes[p], nz - 1)).reshape(nz - 1, N).T
        assert rel(u[p][:, 1:], ref) < 1e-5, (p, rel(u[p][:, 1:], ref))


def march_error(eng, H, T, x, u, axes):
    """Relative errors of the exit and of the last gradient slice, white noise through all slices."""
    Ln, P = T.shape[0], x.shape[0]
    N = int(np.prod(x.shape[1:]))
    psi = lam = x.astype(complex)
    for z in range(Ln):
        psi = np.fft.ifftn(H * np.fft.fftn(psi * T[z], axes=axes), axes=axes)
    for z in reversed(range(Ln)):
        g = np.fft.ifftn(H.conj() * np.fft.fftn(lam, axes=axes), axes=axes)
        lam = np.conj(T[z]) * g
    grad = np.sum(g * np.conj(T[0] * u[:, 0]), 0)
    t1 = dev((T - 1).reshape(Ln, N))
    ex = torch.empty((P, N), dtype=torch.complex64, device="cuda")
    eng.march(t1, dev(x), exit_out=ex)
    gt = torch.zeros((Ln, N), dtype=torch.complex64, device="cuda")
    eng.backward(t1, dev(u.reshape(P, Ln + 1, N)), dev(x), gt)
    return rel(ex.cpu().numpy(), psi.reshape(P, N)), rel(gt[0].cpu().numpy(), grad.reshape(N))


@pytest.mark.parametrize("n", [512, 2048, 243, 270, 625, 960, 1000, 1500])
def test_ms2d_errors_do_not_add_up_over_slices(n):
    rng = np.random.default_rng(n)
    Ln, P = 255, 3
    T = 1 + (np.exp(0.02j * rng.standard_normal((Ln, n))) - 1).astype(np.complex64).astype(complex)
    x, u = cplx(rng, P, n).astype(np.complex64), cplx(rng, P, Ln + 1, n).astype(np.complex64)
    err = march_error(MS2D(n, Ln + 1, K, 1.0, 1.0), po.ms_kernel(n, 1.0, K, 1.0), T, x, u, (-1,))
    assert max(err) < np.sqrt(Ln) * 1e-7 + Ln * 3e-9, err


@pytest.mark.parametrize("n1,n2", [(64, 64), (128, 192), (256, 256), (48, 60), (75, 90)])
def test_ms3d_errors_do_not_add_up_over_slices(n1, n2):
    rng = np.random.default_rng(n1)
    Ln, P = 48, 2
    T = 1 + (np.exp(0.02j * rng.standard_normal((Ln, n1, n2))) - 1).astype(np.complex64).astype(complex)
    x, u = cplx(rng, P, n1, n2).astype(np.complex64), cplx(rng, P, Ln + 1, n1, n2).astype(np.complex64)
    err = march_error(MS3D(n1, n2, Ln + 1, K, 1.0, 1.0, 1.0), po.ms_kernel_3d(n1, n2, 1.0, 1.0, K, 1.0), T, x, u, (-2, -1))
    assert max(err) < np.sqrt(Ln) * 1.4e-7 + Ln * 6e-9, err
