"""Marches whose outputs replace their inputs, and partial marches of one factor set.

A march in place is the march out of place (every input is read before the output that
replaces it is written): to the bit where both run the same kernel.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from thick_ptycho_b200.cn2d import CN2D  # noqa: E402

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


@pytest.mark.parametrize("N,P", [(97, 40), (777, 20), (2047, 9)])
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
