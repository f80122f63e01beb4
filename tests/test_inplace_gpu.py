"""Marches whose outputs replace their inputs, and partial marches of one factor set.

A march in place is the march out of place (every input is read before the output that
replaces it is written): to the bit where both run the same kernel; in 3D, where a march
whose outputs lie on its sources runs the Krylov solves, to 1.2e-5 (test_polynomial_gpu.py).
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from thick_ptycho_b200 import _native  # noqa: E402
from thick_ptycho_b200.cn2d import CN2D  # noqa: E402
from thick_ptycho_b200.cn3d import CN3D  # noqa: E402

K = 4 * np.pi


def cplx(rng, *shape):
    return torch.from_numpy((rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)).cuda()


def index(rng, N, nz, amp=5e-3):
    return torch.from_numpy(1 + amp * (rng.standard_normal((N, nz)) + 0.1j * rng.random((N, nz)))).cuda()


@pytest.mark.parametrize("N,P", [(20, 3), (97, 40), (777, 20), (1201, 7), (2047, 9), (97, 310), (1024, 5)])
@pytest.mark.parametrize("mode", ["forward", "adjoint_exact"])
def test_2d_slice_by_slice_in_place(N, P, mode):
    rng = np.random.default_rng(N)
    nz = 9
    L = nz - 1
    eng = CN2D(N, nz, K, 1.0, 1.0, "impedance")
    fs = eng.factor(index(rng, N, nz), mode)
    src = {"src_shared": cplx(rng, L, N)}
    probes = None if mode == "adjoint_exact" else cplx(rng, P, N)
    if mode == "adjoint_exact":
        src["src_exit"] = cplx(rng, P, N)
    whole = torch.zeros((P, eng.npad), dtype=torch.complex64, device="cuda")
    ex = torch.empty((P, N), dtype=torch.complex64, device="cuda")
    eng.march(fs, P, probes=probes, state_out=whole, exit_out=ex, **src)
    for _ in range(20):
        state = torch.zeros_like(whole)
        out = torch.empty_like(ex)
        for t in range(1, L + 1):
            eng.march(fs, P, probes=probes if t == 1 else None, t_begin=t, t_end=t,
                      state_in=None if t == 1 else state, state_out=state, exit_out=out, **src)
        assert torch.equal(state, whole)
        assert torch.equal(out, ex)
    eng.device_status()


@pytest.mark.parametrize("N,P", [(97, 40), (777, 20), (2047, 9), (97, 310), (1024, 5)])
def test_2d_one_slice_exit_on_its_input(N, P):
    rng = np.random.default_rng(N + 1)
    eng = CN2D(N, 2, K, 1.0, 1.0, "impedance")
    field = index(rng, N, 2)
    probes, src = cplx(rng, P, N), cplx(rng, P, N)
    for mode in ("forward", "adjoint", "adjoint_exact"):
        fs = eng.factor(field, mode)
        runs = [{"src_exit": src}]
        if mode != "adjoint_exact":
            runs += [{"probes": probes}, {"probes": probes, "src_exit": src}, {"probes": probes, "src_probe": src[:, None]}]
        for kw in runs:
            ref = torch.empty((P, N), dtype=torch.complex64, device="cuda")
            eng.march(fs, P, exit_out=ref, **kw)
            for name in kw:
                for _ in range(10):
                    got = {k: v.clone() for k, v in kw.items()}
                    eng.march(fs, P, exit_out=got[name].view(P, N), **got)
                    assert torch.equal(got[name].view(P, N), ref), (mode, sorted(kw), name)
    eng.device_status()


# ------------------------------------------- which kernel a partial march runs
def slice_size(eng):
    return (eng.factor_bytes - 256) // eng.L


def verdicts(eng, fs):
    """The slices' verdict words (the first entry of the forward multipliers)."""
    rows = fs.buf[: slice_size(eng) * eng.L].view(eng.L, -1)
    return rows[:, eng.npad * 8:eng.npad * 8 + 4].contiguous().view(torch.float32)[:, 0]


def set_verdict(eng, fs, s, value):
    at = (s - 1) * slice_size(eng) + eng.npad * 8
    fs.buf[at:at + 4] = torch.tensor([value], dtype=torch.float32).view(torch.uint8).cuda()


@pytest.mark.parametrize("N", [97, 777])
@pytest.mark.parametrize("mode", ["forward", "adjoint", "adjoint_exact"])
def test_2d_partial_march_decides_by_its_own_slices(N, mode):
    """A slice outside the polynomial's bounds (here by its verdict, set from the host)
    sends the marches that read it, and only those, to the direct kernel, in place as well,
    and no march writes the factor set."""
    rng = np.random.default_rng(N + 2)
    nz, P = 13, 4
    L = nz - 1
    eng = CN2D(N, nz, K, 1.0, 1.0, "impedance")
    fs = eng.factor(index(rng, N, nz), mode)
    assert verdicts(eng, fs).tolist() == [0.0] * L
    start = torch.zeros((P, eng.npad), dtype=torch.complex64, device="cuda")
    eng.march(fs, P, probes=None if mode == "adjoint_exact" else cplx(rng, P, N),
              src_exit=cplx(rng, P, N) if mode == "adjoint_exact" else None, t_begin=1, t_end=4, state_out=start)
    grad = mode == "adjoint_exact"
    fwd = eng.new_store(P).copy_(cplx(rng, P, nz, eng.npad)) if grad else None

    def part():
        """Steps 5..8 in place; the state and the gradient of four probes."""
        before = fs.buf.clone()
        state = start.clone()
        gc = eng.new_grad_buffer() if grad else None
        eng.march(fs, P, t_begin=5, t_end=8, state_in=state, state_out=state, u_fwd=fwd, grad_c=gc)
        assert torch.equal(fs.buf, before)
        return [state] + ([torch.view_as_real(gc)] if grad else [])

    slices = range(5, 9) if mode == "forward" else range(L + 1 - 8, L + 1 - 4)
    poly = part()
    for s in range(1, L + 1):
        set_verdict(eng, fs, s, 1.0)
    direct = part()
    assert not torch.equal(poly[0], direct[0])
    scale = max(float(direct[0].abs().max()), 1.0)
    assert float((poly[0] - direct[0]).abs().max()) < 1e-5 * scale
    for s in range(1, L + 1):
        set_verdict(eng, fs, s, 0.0)
    for s in range(1, L + 1):
        set_verdict(eng, fs, s, 1.0)
        got, want = part(), (direct if s in slices else poly)
        assert torch.equal(got[0], want[0]), s
        if grad:  # sums over probes in any order
            assert float((got[1] - want[1]).abs().max()) < 1e-5 * float(want[1].abs().max())
        set_verdict(eng, fs, s, 0.0)
    eng.device_status()


def test_2d_verdicts_follow_the_factorised_slices():
    rng = np.random.default_rng(7)
    N, nz = 241, 40
    eng = CN2D(N, nz, K, 1.0, 1.0, "impedance")
    weak = index(rng, N, nz)
    strong = weak.clone()
    strong[100, 20] += 1.5  # nodes 20: slices 20 and 21
    fs = eng.factor(strong, "forward")
    assert [s + 1 for s, v in enumerate(verdicts(eng, fs).tolist()) if v] == [20, 21]
    eng.factor_range(weak, "forward", 10, 30, out=fs.buf)
    assert not verdicts(eng, fs).any()
    for bad in (float("nan"), float("inf")):
        strong[100, 20] = bad
        eng.factor_range(strong, "forward", 15, 25, out=fs.buf)
        assert [s + 1 for s, v in enumerate(verdicts(eng, fs).tolist()) if v] == [20, 21]


@pytest.mark.parametrize("N", [97, 1024])
def test_2d_march_arguments_refused(N):
    """store_sums is 0 or 1; the stride of state_in is an argument of its own entry."""
    rng = np.random.default_rng(N)
    eng = CN2D(N, 5, K, 1.0, 1.0, "impedance")
    fs = eng.factor(index(rng, N, 5), "forward")
    state = torch.zeros((2, 3, eng.npad), dtype=torch.complex64, device="cuda")
    for sums, slices, with_state, ok in [(0, None, True, True), (0, None, False, True), (0, 3, True, True),
                                         (0, 1, True, True), (0, 3, False, False), (0, 0, True, False),
                                         (0, -1, True, False), (2, None, True, False), (-1, None, True, False),
                                         (256, None, True, False), (768, None, True, False), (768, 3, True, False),
                                         (1, None, True, N == 1024), (1, 3, True, N == 1024)]:
        a = _native.TpCn2dMarchArgs()
        a.num_probes, a.mode, a.t_begin, a.t_end = 2, _native.MODE_FORWARD, 2, 3
        a.store_sums = sums
        if with_state:
            a.state_in = ctypes.c_void_p(state.data_ptr())
        op, buf = eng.op(), ctypes.c_void_p(fs.buf.data_ptr())
        if slices is None:
            rc = eng.lib.tp_cn2d_march(ctypes.byref(op), buf, ctypes.byref(a), None)
        else:
            rc = eng.lib.tp_cn2d_march_from(ctypes.byref(op), buf, ctypes.byref(a), slices, None)
        assert (rc == 0) == ok, (sums, slices, with_state, rc)
    torch.cuda.synchronize()


# ------------------------------------------------------------------ 3D
@pytest.mark.parametrize("case", ["exit on src_exit", "exit on src_exit, exact", "exit on src_shared", "store on src_exit",
                                  "exit on src_exit, later", "exit on probes"])
def test_3d_outputs_on_sources(case):
    rng = np.random.default_rng(3)
    nf, nb, P = 130, 66, 1 if "shared" in case or "store" in case else 5
    nz = 4 if "shared" in case or "later" in case else 2
    N, L = nf * nb, nz - 1
    field = index(rng, N, nz)
    mode = "adjoint_exact" if "exact" in case else "adjoint" if case.startswith("exit on src_exit") else "forward"
    src = cplx(rng, P, N)
    kw = {}
    if "src_exit" in case:
        kw["src_exit"] = src
    if "shared" in case:
        kw["src_shared"] = cplx(rng, L, N)
    if mode == "forward":
        kw["probes"] = cplx(rng, P, N)
    eng = CN3D(nf, nb, nz, K, 1.0, 1.0, 1.0, "impedance")
    ref, store = torch.empty((P, N), dtype=torch.complex64, device="cuda"), eng.new_store(P)
    eng.march(field, P, mode, exit_out=ref, u_store=store, **kw)
    assert (eng.stats.cpu().tolist()[4] == 2) == (nz > 2)
    if "store" in case:
        again = eng.new_store(P)
        again[:, 1] = src
        eng.march(field, P, mode, u_store=again, **{**kw, "src_exit": again[0, 1:2]})
        got, want = again, store
    else:
        kw = {k: v.clone() for k, v in kw.items()}
        got = kw["src_shared"][L - 1:L] if "shared" in case else kw["probes" if "probes" in case else "src_exit"]
        eng.march(field, P, mode, exit_out=got, **kw)
        want = ref
    # a march of several steps has used src_exit before it writes the exit
    assert (eng.stats.cpu().tolist()[4] == 2) == ("later" in case)
    assert float(torch.linalg.vector_norm(got - want)) < 1.2e-5 * float(torch.linalg.vector_norm(want))
    eng.device_status()


@pytest.mark.parametrize("kernels,launch,how", [(0, 0, "polynomial"), (8, 0, "graph"), (8, 1, None)])
def test_3d_stats_name_the_march(kernels, launch, how):
    rng = np.random.default_rng(4)
    eng = CN3D(32, 32, 4, K, 1.0, 1.0, 1.0, "impedance")
    eng.kernels, eng.launch = kernels, launch
    eng.march(index(rng, 1024, 4), 2, "forward", probes=cplx(rng, 2, 1024), u_store=eng.new_store(2))
    st = eng.read_stats()
    assert [st["graph"], st["polynomial"]] == [how == "graph", how == "polynomial"]
