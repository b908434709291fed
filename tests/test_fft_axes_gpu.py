"""The local term's FFT kernels at every axis length, against torch's float64 transforms."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [n for n in range(2, 129) if all(n % p for p in range(11, n + 1) if all(p % q for q in range(2, p)))]


def _handle(shape, flat, nk, npw_max, npw, v, t):
    from gradwave_b200 import _lib
    geom = _lib.Geometry()
    geom.nk, geom.npw_max, geom.nproj = nk, npw_max, 0
    for a in range(3):
        geom.n[a] = shape[a]
    npw = np.ascontiguousarray(npw, dtype=np.int64)
    flat = np.ascontiguousarray(flat, dtype=np.int64)
    geom.npw = npw.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    geom.flat_idx = flat.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    h = ctypes.c_void_p()
    _lib.call("gwb_ham_create", ctypes.byref(geom), 0, ctypes.byref(h))
    s = _lib.stream_ptr()
    _lib.call("gwb_ham_set_kinetic", h, t.data_ptr(), s)
    _lib.call("gwb_ham_set_potential", h, v.data_ptr(), s)
    _lib.call("gwb_ham_set_projectors", h, None, None, s)
    return h


def _check(shape, sel, dev, seed, nb=3):
    """Two k: the points ``sel`` of the box (box indices), the second k short of a third of them. Returns the applies
    (complex128 and complex64 rows in both precisions) and the density."""
    from gradwave_b200 import _lib
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    npw_max = len(sel)
    npw = [npw_max, max(1, npw_max - npw_max // 3)]
    flat = np.zeros((2, npw_max), dtype=np.int64)
    for k in range(2):
        flat[k, :npw[k]] = rng.permutation(sel)[:npw[k]]
    g = torch.Generator().manual_seed(seed)
    v = torch.randn(shape, dtype=torch.float64, generator=g).to(dev)
    t = torch.rand(2, npw_max, dtype=torch.float64, generator=g).to(dev)
    c = torch.randn(2, nb, npw_max, dtype=torch.complex128, generator=g).to(dev)
    h = _handle(shape, flat, 2, npw_max, npw, v, t)
    ref = torch.zeros_like(c)
    rho = torch.zeros(shape, dtype=torch.float64, device=dev)
    w = torch.rand(2, nb, dtype=torch.float64, generator=g).to(dev)
    for k in range(2):
        idx = torch.as_tensor(flat[k, :npw[k]], device=dev)
        box = torch.zeros(nb, n, dtype=torch.complex128, device=dev)
        box[:, idx] = c[k, :, :npw[k]]
        psi = torch.fft.ifftn(box.view(nb, *shape), dim=(1, 2, 3), norm="forward")
        rho += (w[k, :, None, None, None] * psi.abs() ** 2).sum(0)
        loc = torch.fft.fftn(psi * v, dim=(1, 2, 3)).reshape(nb, n)[:, idx] / n
        ref[k, :, :npw[k]] = t[k, :npw[k]] * c[k, :, :npw[k]] + loc
    got = []
    try:
        # a transform's error is a few eps sqrt(log N) of its norm: 1e-14 and 1e-6 leave a factor of ten
        for dt, prec, tol in ((torch.complex128, 1, 1e-14), (torch.complex128, 0, 1e-6), (torch.complex64, 0, 1e-6),
                              (torch.complex64, 1, 1e-6)):
            ci = c.to(dt).contiguous()
            out = torch.full_like(ci, float("nan"))
            _lib.call("gwb_ham_apply", h, ci.data_ptr(), out.data_ptr(), nb, _lib.io_dtype(ci), prec,
                      _lib.stream_ptr())
            err = float((out.to(torch.complex128) - ref).norm() / ref.norm())
            assert err < tol, (shape, dt, prec, err)
            for k in range(2):
                assert not out[k, :, npw[k]:].any()
            got.append(out)
        r = torch.empty(shape, dtype=torch.float64, device=dev)
        _lib.call("gwb_ham_density", h, c.data_ptr(), nb * npw_max, nb, 1, w.data_ptr(), nb, 1.0, r.data_ptr(),
                  _lib.stream_ptr())
        assert float((r - rho).norm() / rho.norm()) < 1e-14
        return got + [r]
    finally:
        torch.cuda.synchronize()
        _lib.load().gwb_ham_destroy(h)


@pytest.mark.parametrize("n", LENGTHS)
def test_every_axis_length(n, cuda_device):
    """Length n on each axis in turn (the others unequal and short), the whole axis occupied, then a few low
    Miller indices only."""
    for axis in range(3):
        shape = [6, 5, 4]
        shape[axis] = n
        full = np.arange(int(np.prod(shape)))
        _check(shape, full[::2] if full.size > 4 else full, cuda_device, n)
        m = np.stack(np.meshgrid(*[np.rint(np.fft.fftfreq(k, 1 / k)) for k in shape], indexing="ij"), -1).reshape(-1, 3)
        few = full[(np.abs(m[:, axis]) <= max(1, n // 5)) & (np.abs(m).sum(1) <= n // 5 + 2)]
        _check(shape, few, cuda_device, n + 1, nb=5)


@pytest.mark.parametrize("n", LENGTHS)
def test_bands_of_one_block(n, cuda_device):
    """Length n on axis 0 with so many pencils that a block of the axis-0 kernel takes several bands (10 bands in
    groups of 3 or 4, the last one short), the next band's points arriving while one is transformed."""
    shape = [n, 96, 100]
    sel = np.random.default_rng(n).choice(n * 9600, 1500, replace=False)
    _check(shape, sel, cuda_device, n, nb=10)


def test_unequal_axes_and_chunks(cuda_device, monkeypatch):
    """A large box with unequal axes, in one chunk and band by band: bit for bit the same."""
    sel = np.random.default_rng(0).choice(30 * 108 * 49, 9000, replace=False)
    monkeypatch.setenv("GWB_W_BUDGET_MB", "1")
    bands = _check([30, 108, 49], sel, cuda_device, 1, nb=7)
    monkeypatch.delenv("GWB_W_BUDGET_MB")
    chunk = _check([30, 108, 49], sel, cuda_device, 1, nb=7)
    assert all(torch.equal(x, y) for x, y in zip(bands, chunk))


def test_slots_of_one_box_cell(cuda_device):
    """Two slots that name the same box cell: the later one enters the transform, both receive the local term."""
    from gradwave_b200 import _lib
    shape, flat = [8, 8, 8], np.array([[0, 9, 9, 70]])
    g = torch.Generator().manual_seed(1)
    v = torch.randn(shape, dtype=torch.float64, generator=g).to(cuda_device)
    t = torch.rand(1, 4, dtype=torch.float64, generator=g).to(cuda_device)
    c = torch.randn(1, 2, 4, dtype=torch.complex128, generator=g).to(cuda_device)
    h = _handle(shape, flat, 1, 4, [4], v, t)
    box = torch.zeros(2, 512, dtype=torch.complex128, device=cuda_device)
    for s in (0, 2, 3):
        box[:, int(flat[0, s])] = c[0, :, s]
    loc = torch.fft.fftn(torch.fft.ifftn(box.view(2, 8, 8, 8), dim=(1, 2, 3)) * v, dim=(1, 2, 3)).reshape(2, -1)
    ref = t[0] * c[0] + loc[:, torch.as_tensor(flat[0], device=cuda_device)]
    out = torch.empty_like(c)
    _lib.call("gwb_ham_apply", h, c.data_ptr(), out.data_ptr(), 2, 1, 1, _lib.stream_ptr())
    assert float((out[0] - ref).abs().max()) < 1e-13
    torch.cuda.synchronize()
    _lib.load().gwb_ham_destroy(h)


def test_scratch_of_a_destroyed_handle(cuda_device):
    """A handle that takes over another's scratch (larger, then smaller than it needs) gives the same result."""
    points = {n: np.random.default_rng(n).choice(n ** 3, n * n, replace=False) for n in (12, 20)}
    keep = _handle([4, 4, 4], np.zeros((1, 1)), 1, 1, [1], torch.zeros(4, 4, 4, dtype=torch.float64, device=cuda_device),
                   torch.zeros(1, 1, dtype=torch.float64, device=cuda_device))
    for n in (20, 12, 20, 12):
        _check([n] * 3, points[n], cuda_device, n)
    from gradwave_b200 import _lib
    torch.cuda.synchronize()
    _lib.load().gwb_ham_destroy(keep)
