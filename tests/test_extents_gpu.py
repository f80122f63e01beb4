"""Calls whose slices, rows or images outnumber a grid's y or z extent (65535 blocks):
against the same call on a part of them, to the bit where each output is computed alone.
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
from thick_ptycho_b200.learned import unpack_padded  # noqa: E402

K = 4 * np.pi
LIB = _native.load()


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def c64(*shape):
    return torch.randn(shape, dtype=torch.complex64, device="cuda")


def test_factor_and_march_of_two_million_slices():
    nz = 32 * 65535 + 40
    field = torch.ones((4, nz), dtype=torch.complex128, device="cuda") + 1e-3 * torch.randn((4, nz), dtype=torch.float64, device="cuda")
    eng, tail = CN2D(4, nz, K, 1.0, 1.0, "neumann"), CN2D(4, 60, K, 1.0, 1.0, "neumann")
    fs, ft = eng.factor(field, "forward"), tail.factor(field[:, -60:].contiguous(), "forward")
    size = (eng.factor_bytes - 256) // eng.L
    assert torch.equal(fs.buf[size * (eng.L - 59):size * eng.L], ft.buf[:size * 59])
    state, a, b = c64(3, eng.npad), c64(3, eng.npad), c64(3, eng.npad)
    eng.march(fs, 3, state_in=state, state_out=a, t_begin=eng.L - 58, t_end=eng.L)
    tail.march(ft, 3, state_in=state, state_out=b, t_begin=1, t_end=59)
    assert torch.equal(a, b)


def test_natural_layout_of_four_million_slices():
    nz = 64 * 65535 + 70
    eng = CN2D(4, nz, K, 1.0, 1.0, "neumann")
    store = torch.empty((1, nz, eng.npad), dtype=torch.complex64, device="cuda").copy_(c64(1, nz, 1))
    store[:, :, 1] += 1
    out = eng.unchunk(store)
    assert torch.equal(out[0], store[0, :, :4].T)


def test_filter_passes_of_many_rows_and_images():
    # a column of 70000 x 8 rows: filters of the centre tap alone are one product per pixel
    nb = 65536 * 8 + 3
    F, z, y = torch.zeros((13, nb), dtype=torch.complex64, device="cuda"), c64(2, nb), c64(2, nb)
    F[0] = c64(nb)
    assert LIB.tp_cnn_filter_apply(1, nb, 2, 0, 0, ptr(F), ptr(z), ptr(y), None) == 0
    want = z + F[0] * z
    assert float((y - want).abs().max()) < 4e-7 * float(want.abs().max())
    # 70000 images of 2 x 3: their gradients are those of a few of them alone
    nf, nb, n, m = 3, 2, 70000, 5
    z, e = c64(n, nf * nb), c64(n, nf * nb)
    out = []
    for cnt, first in ((n, 0), (m, n - m)):
        g = torch.zeros(int(LIB.tp_cnn_act_bytes(nf, nb, cnt, 32)), dtype=torch.uint8, device="cuda")
        assert LIB.tp_cnn_filter_grad(nf, nb, cnt, 1, ptr(z[first:]), ptr(e[first:]), ctypes.c_float(1.0), ptr(g), None) == 0
        out.append(g)
    torch.cuda.synchronize()
    a, b = (unpack_padded(g.cpu(), 32, cnt, nb, nf) for g, cnt in zip(out, (n, m)))
    assert torch.equal(torch.as_tensor(a)[-m:], torch.as_tensor(b)) and torch.as_tensor(b).abs().sum() > 0
