"""The polynomial marches away from mu = 0.02 (degrees 4, 8 and 10, other halos and tiles),
the operators and index fields they leave to the other kernels, and the space-time solve
past the basis its fused Gram-Schmidt kernel holds.

Tolerances as in test_polynomial_gpu.py: 2D against the complex128 oracle, 1e-5.  3D
against the Krylov march, both stopping at a residual of 1e-6 of |b| <= 16 mu |u| (0.9 |u|
at mu = 0.055) per step, L = 4: 2 * 4 * 0.9e-6 + 4 * 1.2e-7 < 1e-5, gradients twice that.
"""

import numpy as np
import pytest

from oracle import pwe_oracle as po

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from thick_ptycho_b200 import SimulationGeometry  # noqa: E402
from thick_ptycho_b200.cn2d import CN2D  # noqa: E402
from thick_ptycho_b200.cn3d import CN3D  # noqa: E402
from thick_ptycho_b200.pit import PWEGpuPiTSolver  # noqa: E402


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def dev(x, dtype=np.complex64):
    return torch.from_numpy(np.ascontiguousarray(x).astype(dtype)).cuda()


def cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def verdicts(eng, fs):
    """The slices' verdict words: 0 where the polynomial kernel marches the slice."""
    rows = fs.buf[: (eng.factor_bytes - 256) // eng.L * eng.L].view(eng.L, -1)
    return rows[:, eng.npad * 8:eng.npad * 8 + 4].contiguous().view(torch.float32)[:, 0]


# ------------------------------------------------------------------ 2D
@pytest.mark.parametrize("N,P,mu", [
    (241, 3, 0.005), (777, 2, 0.005), (1201, 3, 0.005), (241, 3, 0.042), (777, 2, 0.042), (1201, 3, 0.042),
    (241, 3, 0.055), (777, 2, 0.055), (1201, 3, 0.055), (1300, 200, 0.02), (1300, 200, 0.055),
])
@pytest.mark.parametrize("bc", ["impedance", "neumann"])
def test_2d_degrees(N, P, mu, bc):
    """Degrees 4 and 8, in 2, 4 and 8 rows per thread; 200 probes of 1300 rows: two CTAs per SM."""
    rng = np.random.default_rng(N)
    nz, k = 6, 1 / (4 * mu)
    L = nz - 1
    n = 1 + 5e-3 * (rng.standard_normal((N, nz)) + 0.1j * rng.random((N, nz)))
    eng = CN2D(N, nz, k, 1.0, 1.0, bc)
    co = po.bc_coefficients(k, 1.0, 1.0, bc_type=bc)
    A, B = po.step_matrices_1d(N, co, bc, 1.0)
    C = po.object_contribution(n, k, 1.0)
    probes, ex = cplx(rng, P, N), cplx(rng, P, N)
    field = dev(n, np.complex128)
    some = range(P) if P < 10 else (0, 63, 148, P - 1)

    fs = eng.factor(field, "forward")
    assert not verdicts(eng, fs).any()
    store = eng.new_store(P)
    out = torch.empty((P, N), dtype=torch.complex64, device="cuda")
    eng.march(fs, P, probes=dev(probes), exit_out=out)
    eng.march(fs, P, probes=dev(probes), u_store=store)
    u = eng.unchunk(store).cpu().numpy()
    assert np.array_equal(out.cpu().numpy(), u[:, :, -1])
    ref = {p: po.march(A, B, C, probes[p]) for p in some}
    for p in some:
        assert rel(u[p], ref[p]) < 1e-5, (p, rel(u[p], ref[p]))

    fa = eng.factor(field, "adjoint_exact")
    assert not verdicts(eng, fa).any()
    lam_store = eng.new_store(P)
    gc = eng.new_grad_buffer()
    eng.march(fa, P, src_exit=dev(ex), u_fwd=store, grad_c=gc, u_store=lam_store)
    lam = eng.unchunk(lam_store).cpu().numpy()
    src = np.zeros((len(ref), N, L), dtype=complex)
    src[:, :, -1] = ex[list(some)]
    want = po.exact_adjoint_many(A, B, C, src)
    if len(ref) == P:
        g = eng.unchunk_rows(gc).cpu().numpy().T
        assert rel(g, sum(po.grad_c_from_adjoint(ref[p], want[p]) for p in range(P))) < 1e-5
    else:  # the sum over probes from the stored fields
        uc, lc = torch.from_numpy(u).cuda().to(torch.complex128), torch.from_numpy(lam).cuda().to(torch.complex128)
        g = eng.unchunk_rows(gc).cpu().numpy().T
        acc = torch.stack([(lc[:, :, L - 1 - s + 1] * (uc[:, :, s + 1] + uc[:, :, s]).conj()).sum(0) for s in range(L)], 1)
        assert rel(g, acc.cpu().numpy()) < 1e-5
    direct = torch.empty_like(out)
    at = eng.npad * 8
    rows = fs.buf[: (eng.factor_bytes - 256) // L * L].view(L, -1)
    rows[:, at:at + 4] = torch.tensor([1.0]).view(torch.uint8).cuda()
    eng.march(fs, P, probes=dev(probes), exit_out=direct)
    assert not torch.equal(direct, out) and rel(direct.cpu().numpy(), out.cpu().numpy()) < 1e-5
    eng.device_status()


# ------------------------------------------------------------------ 3D
def both(nf, nb, nz, P, k, bc, field, rng, garbage=False):
    """Forward exit and pair sums, exact adjoint's exit and gradient by the automatic and by
    the Krylov march, with what stats say of each."""
    N, L = nf * nb, nz - 1
    probes, ex = dev(cplx(rng, P, N)), dev(cplx(rng, P, N))
    got = {}
    for kernels in (0, 8):
        eng = CN3D(nf, nb, nz, k, 1.0, 1.0, 1.0, bc)
        eng.kernels = kernels
        if garbage:
            eng.workspace(P).fill_(0xff)
        out, lam = (torch.empty((P, N), dtype=torch.complex64, device="cuda") for _ in range(2))
        sums = eng.new_store(P)
        gc = torch.zeros((L, N), dtype=torch.complex64, device="cuda")
        eng.march(field, P, "forward", probes=probes, u_store=sums, exit_out=out, store_sums=True)
        eng.march(field, P, "adjoint_exact", src_exit=ex, u_fwd=sums, grad_c=gc, exit_out=lam, store_sums=True)
        eng.device_status()
        got[kernels] = [x.cpu().numpy() for x in (out, sums, lam, gc)], eng.read_stats()
    return got[0][0], got[8][0], got[0][1], got[8][1]


@pytest.mark.parametrize("mu,m", [(0.005, 4), (0.035, 8), (0.055, 10)])
@pytest.mark.parametrize("nf,nb,P", [(130, 97, 3), (131, 60, 2), (57, 140, 2)])
@pytest.mark.parametrize("bc", ["impedance", "neumann"])
def test_3d_degrees_across_tiles(nf, nb, P, mu, m, bc):
    rng = np.random.default_rng(nf + nb)
    nz = 5
    field = dev(1 + 2e-3 * (rng.standard_normal((nf * nb, nz)) + 0.1j * rng.random((nf * nb, nz))), np.complex128)
    a, b, sa, sb = both(nf, nb, nz, P, 1 / (4 * mu), bc, field, rng)
    assert sa["polynomial"] and sa["max_iterations"] == m and sa["failed"] == 0, sa
    assert sb["graph"] and sb["failed"] == 0
    for i, (x, y) in enumerate(zip(a, b)):
        assert rel(x, y) < (2e-5 if i == 3 else 1e-5), (i, rel(x, y))


@pytest.mark.parametrize("what", ["gain", "large mu", "nan", "inf"])
def test_3d_left_to_the_krylov_march(what):
    """Past the polynomial's bounds, or with an index that is not a number, the march is the
    Krylov one, on a workspace full of other bytes."""
    rng = np.random.default_rng(8)
    nf, nb, nz, P = 64, 40, 4, 2
    mu = 0.2 if what == "large mu" else 0.02
    n = 1 + 5e-3 * rng.standard_normal((nf * nb, nz)) + 0j
    if what == "gain":  # |D| of single pixels down to 0.1: |J| sums to 0.8 there
        n += 0.15j * (np.arange(nf * nb) % 101 == 50)[:, None]
    if what in ("nan", "inf"):
        n[777, 1] = float(what)
    a, b, sa, sb = both(nf, nb, nz, P, 1 / (4 * mu), "impedance", dev(n, np.complex128), rng, garbage=True)
    assert sa["graph"] and sb["graph"]
    if what in ("nan", "inf"):
        for x, y in zip(a, b):
            assert np.array_equal(np.isfinite(x), np.isfinite(y))
            assert not np.isfinite(x).all()
        return
    assert sa["failed"] == sb["failed"]
    for i, (x, y) in enumerate(zip(a, b)):  # the same kernels; their sums run in any order
        assert rel(x, y) < 1e-5, (i, rel(x, y))


def test_2d_index_that_is_not_a_number():
    """The slices that read it go to the direct kernel; the others' probes stay finite before it."""
    rng = np.random.default_rng(9)
    N, nz, P = 241, 9, 2
    for bad in (float("nan"), float("inf")):
        n = 1 + 5e-3 * rng.standard_normal((N, nz)) + 0j
        n[100, 4] = bad
        eng = CN2D(N, nz, 4 * np.pi, 1.0, 1.0, "impedance")
        fs = eng.factor(dev(n, np.complex128), "forward")
        assert [s + 1 for s, v in enumerate(verdicts(eng, fs).tolist()) if v] == [4, 5]
        store = eng.new_store(P)
        eng.march(fs, P, probes=dev(cplx(rng, P, N)), u_store=store)
        u = eng.unchunk(store).cpu().numpy()
        assert np.isfinite(u[:, :, :4]).all() and not np.isfinite(u[:, :, 4:]).all()


# ------------------------------------------------------------------ space-time solve
@pytest.mark.parametrize("N,nz,P", [(97, 33, 2), (256, 130, 1)])
def test_pit_past_the_fused_basis(N, nz, P):
    k = 2 * np.pi / 0.5
    rng = np.random.default_rng(N)
    n = 1 + 1.5e-2 * np.cos(np.arange(N) / 9.0)[:, None] * np.sin(np.arange(nz) / 5.0)
    x = np.arange(N)[None]
    probes = np.exp(-((x - rng.uniform(0.3 * N, 0.7 * N, (P, 1))) ** 2) / 50.0).astype(complex)
    geo = SimulationGeometry(dimension=2, nx=N, nz=nz, dx=1.0, dz=1.0, k=k, num_probes=P)
    s = PWEGpuPiTSolver(geo, probes[None], bc_type="impedance")
    u = s.solve(n=n)[0, 0]
    assert 8 < max(s.gmres_iterations), s.gmres_iterations
    co = po.bc_coefficients(k, 1.0, 1.0, bc_type="impedance")
    A, B = po.step_matrices_1d(N, co, "impedance", 1.0)
    C = po.object_contribution(n, k, 1.0)
    for p in range(P):
        ref = po.full_system_solve(A, B, C, po.pit_rhs(B, probes[p], nz - 1)).reshape(nz - 1, N).T
        assert rel(u[p][:, 1:], ref) < 1e-5, (p, rel(u[p][:, 1:], ref))
