"""Marches whose slices are solved by a fixed polynomial of the scaled
off-diagonals, and the periodic preconditioner evaluated the same way on tiles.

2D: against the complex128 oracle at 1e-5 (the bound of the complex64 form).
3D: against the Krylov march of the same call, both stopping at a residual of
1e-6 of a right-hand side |b| <= 0.4 |u| per step with |(I - P)^-1| ~ 1, over
L <= 12 steps, plus two roundings of u per step: 2 * 12 * 0.4e-6 + 12 * 1.2e-7
< 1.2e-5; gradients, products of two such fields, 2.4e-5.  Preconditioner: one
BiCGStab iteration per step, far from converged, is the same map of the same
inputs to 1e-7 (the polynomial) and 1e-6 (complex64 sums of up to 1e4 terms) of
an update of at most 0.4 |u|: 6 * 0.4 * 1.1e-6 + 6 * 1.2e-7 < 4e-6.
"""

import numpy as np
import pytest

from oracle import pwe_oracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from thick_ptycho_b200.cn2d import CN2D  # noqa: E402
from thick_ptycho_b200.cn3d import CN3D  # noqa: E402

K = 4 * np.pi


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def dev(x, dtype=np.complex64):
    return torch.from_numpy(np.ascontiguousarray(x).astype(dtype)).cuda()


def cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


# ------------------------------------------------------------------ 2D
@pytest.mark.parametrize("N,nz,P,bc,amp", [
    (4, 5, 1, "neumann", 5e-3), (31, 6, 2, "impedance", 5e-3), (240, 7, 3, "dirichlet", 5e-3),
    (241, 7, 3, "impedance", 5e-3), (777, 9, 2, "impedance2", 5e-3), (1023, 6, 2, "impedance", 5e-3),
    (1201, 6, 5, "neumann", 5e-3), (2047, 5, 1, "impedance", 5e-3),
    (241, 7, 3, "impedance", 0.4),  # past the polynomial's bounds: the direct kernel
    (200, 6, 2, "neumann", 2e-2),   # object phases beyond the free-space margin
    (97, 4, 310, "impedance", 5e-3), (512, 6, 3, "impedance", 5e-3),  # large batch; team layout
])
def test_2d_modes_sources_and_gradient(N, nz, P, bc, amp):
    rng = np.random.default_rng(N)
    n = 1 + amp * (rng.standard_normal((N, nz)) + 0.1j * rng.random((N, nz)))
    L = nz - 1
    eng = CN2D(N, nz, K, 1.0, 1.0, bc)
    co = po.bc_coefficients(K, 1.0, 1.0, bc_type=bc)
    A, B = po.step_matrices_1d(N, co, bc, 1.0)
    C = po.object_contribution(n, K, 1.0)
    probes, sh, ex = cplx(rng, P, N), cplx(rng, L, N), cplx(rng, P, N)
    field = dev(n, np.complex128)

    fs = eng.factor(field, "forward")
    store = eng.new_store(P)
    eng.march(fs, P, probes=dev(probes), src_shared=dev(sh), u_store=store)
    u = eng.unchunk(store).cpu().numpy()
    ref = np.array([po.march(A, B, C, probes[p], rhs_block=sh.T) for p in range(P)])
    assert rel(u, ref) < 1e-5

    # the same march in two parts
    state = torch.zeros((P, eng.npad), dtype=torch.complex64, device="cuda")
    out = torch.empty((P, N), dtype=torch.complex64, device="cuda")
    cut = L // 2
    eng.march(fs, P, probes=dev(probes), src_shared=dev(sh), t_begin=1, t_end=cut, state_out=state)
    eng.march(fs, P, src_shared=dev(sh), t_begin=cut + 1, t_end=L, state_in=state.clone(), exit_out=out)
    assert rel(out.cpu().numpy(), ref[:, :, -1]) < 1e-5
    # and from a slice of the stored field
    again = torch.empty_like(out)
    eng.march(fs, P, src_shared=dev(sh), t_begin=cut + 1, t_end=L, state_from=(store, cut), exit_out=again)
    assert torch.equal(again, out)

    plain = eng.new_store(P)
    eng.march(fs, P, probes=dev(probes), u_store=plain)
    gc = eng.new_grad_buffer()
    lam_store = eng.new_store(P)
    fa = eng.factor(field, "adjoint_exact")
    eng.march(fa, P, src_exit=dev(ex), u_fwd=plain, grad_c=gc, u_store=lam_store)
    uf = np.array([po.march(A, B, C, probes[p]) for p in range(P)])
    src = np.zeros((P, N, L), dtype=complex)
    src[:, :, -1] = ex
    lam = po.exact_adjoint_many(A, B, C, src)
    g = eng.unchunk_rows(gc).cpu().numpy().T
    assert rel(g, sum(po.grad_c_from_adjoint(uf[p], lam[p]) for p in range(P))) < 1e-5
    eng.device_status()


# ------------------------------------------------------------------ 3D
@pytest.mark.parametrize("nf,nb,nz,P,bc,dtype,delta", [
    (16, 16, 13, 1, "impedance", np.complex128, False),   # one probe: the slices in chunks
    (33, 47, 6, 3, "neumann", np.complex64, False),       # odd rows: unaligned accesses
    (36, 131, 6, 5, "dirichlet", np.complex128, True),
    (130, 66, 5, 7, "impedance", np.complex64, True),
    (200, 52, 5, 40, "impedance", np.complex128, False),
])
def test_3d_modes_sources_and_gradient(nf, nb, nz, P, bc, dtype, delta):
    rng = np.random.default_rng(nf)
    N, L = nf * nb, nz - 1
    dn = 5e-3 * (rng.standard_normal((N, nz)) + 0.1j * rng.random((N, nz)))
    field = dev(dn if delta else 1 + dn, dtype)
    probes, sh, ex = dev(cplx(rng, P, N)), dev(cplx(rng, L, N)), dev(cplx(rng, P, N))
    got = {}
    for kernels in (0, 8):
        eng = CN3D(nf, nb, nz, K, 1.0, 1.0, 1.0, bc)
        eng.kernels = kernels
        f, a, s = eng.new_store(P), eng.new_store(P), eng.new_store(P)
        out = torch.empty((P, N), dtype=torch.complex64, device="cuda")
        eng.march(field, P, "forward", probes=probes, src_shared=sh, u_store=f, exit_out=out, is_delta=delta)
        eng.march(field, P, "adjoint", probes=probes, src_shared=sh, u_store=a, is_delta=delta)
        eng.march(field, P, "forward", probes=probes, u_store=s, is_delta=delta)
        gc = torch.zeros((L, N), dtype=torch.complex64, device="cuda")
        lam = eng.new_store(P)
        eng.march(field, P, "adjoint_exact", src_exit=ex, u_fwd=s, grad_c=gc, u_store=lam, is_delta=delta)
        sums = eng.new_store(P)
        eng.march(field, P, "forward", probes=probes, u_store=sums, store_sums=True, is_delta=delta)
        gs = torch.zeros_like(gc)
        eng.march(field, P, "adjoint_exact", src_exit=ex, u_fwd=sums, grad_c=gs, store_sums=True, is_delta=delta)
        st = eng.stats.cpu().tolist()
        assert st[2] == 0 and st[1] == 6 * L * P
        assert (st[4] == 2) == (kernels == 0), st
        got[kernels] = [x.cpu().numpy() for x in (f, out, a, s, lam, sums, gc, gs)]
    for i, (x, y) in enumerate(zip(got[0], got[8])):
        assert rel(x, y) < (2.4e-5 if i >= 6 else 1.2e-5), (i, rel(x, y))
    assert rel(got[0][5][:, 1:], got[0][3][:, 1:] + got[0][3][:, :-1]) < 2e-7  # one rounding
    assert rel(got[0][7], got[0][6]) < 1e-6


@pytest.mark.parametrize("nf,nb,P,mu", [
    (8, 8, 2, 0.02), (16, 81, 3, 0.03), (64, 64, 5, 0.04), (128, 128, 2, 0.03), (150, 45, 4, 0.06),
    (192, 192, 3, 0.045), (256, 256, 2, 0.02),
])
@pytest.mark.parametrize("mode", ["forward", "adjoint_exact"])
def test_preconditioner_on_tiles_is_the_transform(nf, nb, P, mu, mode):
    rng = np.random.default_rng(nf + nb)
    nz, N = 7, nf * nb
    field = dev(1 + 5e-3 * rng.standard_normal((N, nz)), np.complex128)
    x = dev(cplx(rng, P, N))
    got = []
    for kernels in (8, 9):
        eng = CN3D(nf, nb, nz, 1 / (4 * mu), 1.0, 1.0, 1.0, "neumann")
        eng.kernels = kernels
        store = eng.new_store(P)
        kw = {"probes": x} if mode == "forward" else {"src_exit": x}
        eng.march(field, P, mode, u_store=store, tol=1e-9, max_iter=1, **kw)
        assert eng.read_stats()["max_iterations"] == 1
        got.append(store.cpu().numpy())
    assert rel(got[0], got[1]) < 4e-6, rel(got[0], got[1])


def test_3d_norms_are_fp64_sums():
    """The right-hand side's norms that solves are judged by: one pixel in 16 of size 1 among
    pixels of 1e-4, whose squares a sum in fp32 drops beside it (2e-7 of the norm).  The
    first exact-adjoint step's right-hand side is its source, and the march leaves the
    norms (fp64 pairs, by step and probe) behind its two state vectors."""
    nf, nb, nz, P = 128, 96, 4, 3
    N = nf * nb
    rng = np.random.default_rng(11)
    src = np.full((P, nb, nf), 1e-4, np.complex64)
    src[:, ::8, ::2] = 1
    src *= np.exp(2j * np.pi * rng.integers(0, 4, src.shape) / 4).round().astype(np.complex64)
    eng = CN3D(nf, nb, nz, K, 1.0, 1.0, 1.0, "impedance")
    field = dev(1 + 5e-3 * rng.standard_normal((N, nz)), np.complex128)
    eng.march(field, P, "adjoint_exact", src_exit=dev(src.reshape(P, N)), exit_out=torch.empty((P, N), dtype=torch.complex64, device="cuda"))
    assert eng.stats.cpu().tolist()[4] == 2
    at = 2 * (-(-P * N * 8 // 256) * 256)
    norms = eng.workspace(P)[at:at + 16 * P].cpu().numpy().view(np.float64).reshape(P, 2)
    exact = np.sum(np.abs(src.astype(complex)) ** 2, axis=(1, 2))
    assert np.all(np.abs(norms[:, 0] - exact) < 1e-12 * exact), norms[:, 0] / exact - 1
    assert np.all(norms[:, 1] < 1e-12 * norms[:, 0])
