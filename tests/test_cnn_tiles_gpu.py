"""Tiled filter kernels and the tensor-core weight gradient of the learned
preconditioner at sizes where tiles (64 x 8) are ragged, against the float64 oracle.

Tolerances: a filtered value is a sum of 14 complex64 products (28 roundings of at
most 6e-8 of a term: below 2e-6 of the result's norm); residuals subtract an
independent target of the same size, 4e-6; the loss is their squared sum, 1e-5; the
filter gradient is stored as bf16 (1e-2 of its largest value); weight gradients add up
to 1.3e4 exact bf16 products in fp32, 1e-4.
"""

import ctypes

import numpy as np
import pytest

from oracle import cnn_oracle as co

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from thick_ptycho_b200 import _native  # noqa: E402
from thick_ptycho_b200.learned import pack_padded, unpack_padded  # noqa: E402

LIB = _native.load()


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def c64(x):
    return torch.from_numpy(np.ascontiguousarray(x).astype(np.complex64)).cuda()


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nf,nb,nimg,per", [(3, 2, 1, 1), (63, 7, 2, 2), (64, 8, 1, 3), (65, 9, 3, 1), (130, 33, 2, 5),
                                            (256, 3, 1, 2)])
def test_filter_kernels_on_ragged_tiles(nf, nb, nimg, per):
    rng = np.random.default_rng(nf)
    N, V = nf * nb, nimg * per
    F = 0.1 * cplx(rng, nimg, 13, nb, nf)
    z, t = cplx(rng, V, nb, nf), cplx(rng, V, nb, nf)
    Fd = c64(F.transpose(1, 0, 2, 3).reshape(13, nimg * N))
    zd, td = c64(z.reshape(V, N)), c64(t.reshape(V, N))
    out = torch.empty_like(zd)
    for conj in (0, 1):
        _native.check(LIB.tp_cnn_filter_apply(nf, nb, V, per, conj, ptr(Fd), ptr(zd), ptr(out), stream()), "apply")
        assert rel(out.cpu().numpy().reshape(z.shape), co.filter_apply(F, z, per, bool(conj))) < 2e-6
    if nimg == 1:  # per_image = 0: image 0 for all
        _native.check(LIB.tp_cnn_filter_apply(nf, nb, V, 0, 0, ptr(Fd), ptr(zd), ptr(out), stream()), "apply")
        assert rel(out.cpu().numpy().reshape(z.shape), co.filter_apply(F, z, per)) < 2e-6
    scale = (0.5 + rng.random(V)).astype(np.float32)
    sd = torch.from_numpy(scale).cuda()
    loss = torch.full((1,), 3.0, dtype=torch.float64, device="cuda")
    _native.check(LIB.tp_cnn_filter_residual(nf, nb, V, per, ptr(Fd), ptr(zd), ptr(td), ptr(sd), ptr(out), ptr(loss),
                                             stream()), "residual")
    d = co.filter_apply(F, z, per) - t
    assert rel(out.cpu().numpy().reshape(z.shape), d * scale[:, None, None]) < 4e-6
    want = float(np.sum(scale[:, None, None] * np.abs(d) ** 2))
    assert abs(loss.item() - 3.0 - want) < 1e-5 * want
    e = out.cpu().numpy().reshape(z.shape).astype(complex)
    dy = torch.zeros(int(LIB.tp_cnn_act_bytes(nf, nb, nimg, 32)), dtype=torch.uint8, device="cuda")
    _native.check(LIB.tp_cnn_filter_grad(nf, nb, nimg, per, ptr(zd), ptr(out), 0.5, ptr(dy), stream()), "grad")
    got = unpack_padded(dy, 32, nimg, nf, nb).cpu().numpy()
    ref = np.zeros((nimg, 32, nb, nf))
    for v in range(V):
        for k, (ddy, ddx) in enumerate(co.TAPS):
            g = np.conj(co.shift(z[v], ddy, ddx)) * e[v]
            ref[v // per, 2 * k] += g.real
            ref[v // per, 2 * k + 1] += g.imag
    assert np.abs(got - ref).max() <= 1e-2 * np.abs(ref).max()


@pytest.mark.parametrize("cin", [16, 32])
@pytest.mark.parametrize("nf,nb,batch", [(5, 3, 1), (64, 64, 1), (129, 50, 2), (33, 31, 5)])
def test_weight_gradient_sizes(cin, nf, nb, batch):
    rng = np.random.default_rng(nf + cin)
    x, dy = rng.standard_normal((batch, cin, nb, nf)), rng.standard_normal((batch, 32, nb, nf))
    bf = lambda a: torch.as_tensor(a).to(torch.bfloat16).double().numpy()  # noqa: E731
    dw = torch.zeros((9, cin, 32), dtype=torch.float32, device="cuda")
    db = torch.zeros(32, dtype=torch.float32, device="cuda")
    xb, dyb = pack_padded(torch.from_numpy(x)).cuda(), pack_padded(torch.from_numpy(dy)).cuda()
    _native.check(LIB.tp_conv3x3_wgrad(nf, nb, batch, cin, ptr(xb), ptr(dyb), ptr(dw), ptr(db), stream()), "wgrad")
    got = dw.view(3, 3, cin, 32).permute(3, 2, 0, 1).cpu().numpy()
    assert rel(got, co.conv3x3_wgrad(bf(x), bf(dy))) < 1e-4
    assert np.allclose(db.cpu().numpy(), bf(dy).sum(axis=(0, 2, 3)), rtol=1e-4, atol=1e-3)


def test_training_step_operands():
    """Lazily conjugated, real and broadcast operands give what their values give; operands
    of another device are refused."""
    from thick_ptycho_b200.learned import LearnedPreconditioner

    rng = np.random.default_rng(5)
    nf, nb, nimg, per = 24, 10, 2, 3
    N, V = nf * nb, nimg * per
    m = LearnedPreconditioner(nf, nb, kappa=20.0)
    d, z, t = c64(0.01 * cplx(rng, nimg, N)), c64(cplx(rng, V, N)), c64(cplx(rng, V, N))
    sc = torch.rand(V, device="cuda")
    same = [((t, sc), (t.conj().resolve_conj().conj(), sc.double())),
            ((t.real.to(torch.complex64), torch.ones_like(sc)), (t.real, torch.ones(1, device="cuda"))),
            ((torch.zeros_like(t), sc), (0.0, sc)), ((torch.zeros_like(t), sc), (torch.tensor(0.0), sc))]
    for a, b in same:
        la, wa, ba = m.loss_and_grads(d, z, *a, per)
        lb, wb, bb = m.loss_and_grads(d, z, *b, per)
        assert abs(float(la) - float(lb)) <= 1e-6 * float(la)
        for x, y in zip(wa + ba, wb + bb):  # sums in any order
            assert float((x - y).abs().max()) <= 1e-4 * float(x.abs().max())
    for bad in ((t.cpu(), sc), (t, sc.cpu())):
        with pytest.raises(RuntimeError):
            m.loss_and_grads(d, z, *bad, per)
    with pytest.raises(RuntimeError):
        m.loss_and_grads(d, z.cpu(), t, sc, per)


@pytest.mark.parametrize("nf,nb", [(1, 1), (2, 3), (5, 2), (65, 9)])
def test_filter_taps_that_leave_the_image(nf, nb):
    """They have no part in the sum, whatever the filter holds there."""
    rng = np.random.default_rng(nf)
    dy = [0, 0, 0, -1, 1, -1, -1, 1, 1, 0, 0, -2, 2]
    dx = [0, -1, 1, 0, 0, -1, 1, -1, 1, -2, 2, 0, 0]
    y, x = np.mgrid[:nb, :nf]
    F = cplx(rng, 13, nb, nf).astype(np.complex64)
    for t in range(13):
        out = (y + dy[t] < 0) | (y + dy[t] >= nb) | (x + dx[t] < 0) | (x + dx[t] >= nf)
        F[t][out] = 0
    hole = F.copy()
    hole[F == 0] = np.nan
    z, t = c64(cplx(rng, 2, nb * nf)), c64(cplx(rng, 2, nb * nf))
    res = []
    for f in (F, hole):
        f, a, e = c64(f.reshape(13, -1)), torch.empty_like(z), torch.empty_like(z)
        loss, sc = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.ones(2, device="cuda")
        assert LIB.tp_cnn_filter_apply(nf, nb, 2, 0, 0, ptr(f), ptr(z), ptr(a), stream()) == 0
        assert LIB.tp_cnn_filter_residual(nf, nb, 2, 0, ptr(f), ptr(z), ptr(t), ptr(sc), ptr(e), ptr(loss), stream()) == 0
        res.append((a, e, loss))
    assert torch.isfinite(torch.view_as_real(res[1][0])).all()
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    assert abs(float(res[0][2]) - float(res[1][2])) <= 1e-12 * float(res[0][2])
