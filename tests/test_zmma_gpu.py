"""Float64 tensor-instruction products (split-K A B^H, nonlocal update) at tile edges, against torch."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, generator=g).cuda()


@pytest.mark.parametrize("M,N,K,batch", [(1, 1, 1, 1), (7, 9, 63, 2), (8, 8, 64, 1), (24, 65, 749, 3), (33, 31, 1001, 2),
                                         (129, 256, 515, 1), (160, 64, 4097, 1), (25, 1, 130, 4)])
def test_a_bh_products(M, N, K, batch, cuda_device):
    """C = alpha A B^H + beta C with strides wider than the matrices. Error bound: K eps sum |a||b|, far above
    the eps sqrt(K) growth of random sums."""
    from gradwave_b200 import _lib
    A, B, C = _rand(batch, M + 1, K + 3, seed=1), _rand(batch, N + 2, K + 5, seed=2), _rand(batch, M, N + 1, seed=3)
    ref = (2.0 + 0.5j) * A[:, :M, :K] @ B[:, :N, :K].mH + (0.25 - 1j) * C[:, :, :N]
    keep = C[:, :, N].clone()
    work = torch.empty(8 << 20, dtype=torch.uint8, device=cuda_device)
    _lib.call("gwb_zgemm_nh", M, N, K, 2.0, 0.5, A.data_ptr(), K + 3, (M + 1) * (K + 3), B.data_ptr(), K + 5,
              (N + 2) * (K + 5), 0.25, -1.0, C.data_ptr(), N + 1, M * (N + 1), batch, work.data_ptr(), work.numel(),
              _lib.stream_ptr())
    bound = K * 2.3e-16 * 2.2 * (A[:, :M, :K].abs() @ B[:, :N, :K].abs().mT) + 1e-15
    assert bool(((C[:, :, :N] - ref).abs() <= bound + 4e-16 * ref.abs()).all())
    assert torch.equal(C[:, :, N], keep)


@pytest.mark.parametrize("nproj,nb", [(1, 1), (8, 9), (33, 17), (130, 40)])
def test_nonlocal_of_both_outputs(nproj, nb, cuda_device):
    """H c and S c of random projectors (ragged counts, two k of unequal size) against torch."""
    from gradwave_b200.basis import BatchedK
    from gradwave_b200.hamiltonian import BatchedHamiltonian
    from gradwave_b200.uspp import BatchedHS
    npw, n = [71, 60], 10
    g = torch.Generator().manual_seed(nproj)
    mask = torch.zeros(2, 71, dtype=torch.bool)
    flat = torch.zeros(2, 71, dtype=torch.int64)
    for k in range(2):
        mask[k, :npw[k]] = True
        flat[k, :npw[k]] = torch.randperm(n ** 3, generator=g)[:npw[k]]
    d, q = (torch.randn(nproj, nproj, dtype=torch.float64, generator=g) for _ in range(2))
    d, q = d + d.T, q + q.T
    t = torch.rand(2, 71, dtype=torch.float64, generator=g) * mask
    bk = BatchedK(torch.tensor(npw), mask, flat, torch.zeros(2, 71, 3, dtype=torch.float64), t,
                  torch.zeros(0, dtype=torch.complex128), torch.zeros(nproj, dtype=torch.int64), d).to(cuda_device)
    p = _rand(2, nproj, 71, seed=5) * bk.mask[:, None, :]
    c = _rand(2, nb, 71, seed=6) * bk.mask[:, None, :]
    v = torch.zeros(n, n, n, dtype=torch.float64, device=cuda_device)
    b = c @ p.mH
    ref_h = bk.t[:, None] * c + (b @ d.to(b)) @ p
    ref_s = c + (b @ q.to(b)) @ p
    h, s = BatchedHS(bk, (n, n, n), v, p, d, q).hs(c)
    assert torch.equal(BatchedHamiltonian(bk, (n, n, n), v, p).apply(c), h)
    for got, ref in ((h, ref_h), (s, ref_s)):
        assert float((got - ref).norm() / ref.norm()) < 1e-14
        assert not got[1, :, 60:].any()


@pytest.mark.parametrize("op", [0, 1])
@pytest.mark.parametrize("M,N,K,batch", [(1, 8, 1, 1), (7, 63, 9, 2), (8, 64, 8, 3), (24, 193, 72, 2), (33, 1001, 17, 1),
                                         (64, 513, 64, 2), (65, 600, 5, 1)])
def test_short_row_products(op, M, N, K, batch, cuda_device):
    """C = alpha op(A) B + beta C of few rows (own tiles; 64 and 65: cuBLAS) with strides wider than the matrices; C is
    not read where beta = 0. Bound as above."""
    from gradwave_b200 import _lib
    A = _rand(batch, M, K + 2, seed=1) if op == 0 else _rand(batch, K, M + 2, seed=1)
    a = A[:, :, :K] if op == 0 else A[:, :, :M].mT
    B, C0 = _rand(batch, K + 1, N + 3, seed=2), _rand(batch, M, N + 1, seed=3)
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (0.5 - 2j, 0.25j)):
        C = C0.clone() if beta != 0.0 else torch.full_like(C0, float("nan"))
        alpha, beta = complex(alpha), complex(beta)
        _lib.call("gwb_zgemm", op, 0, M, N, K, alpha.real, alpha.imag, A.data_ptr(), A.shape[2], A.shape[1] * A.shape[2],
                  B.data_ptr(), N + 3, (K + 1) * (N + 3), beta.real, beta.imag, C.data_ptr(), N + 1, M * (N + 1), batch,
                  _lib.stream_ptr())
        ref = alpha * (a @ B[:, :K, :N]) + (beta * C0[:, :, :N] if beta != 0.0 else 0.0)
        bound = (K + 2) * 2.3e-16 * abs(alpha) * 2.2 * (a.abs() @ B[:, :K, :N].abs()) + 1e-15 * (1 + abs(beta) * C0[:, :, :N].abs())
        assert bool(((C[:, :, :N] - ref).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(8, 64, 128), (8, 63, 128), (24, 192, 128), (24, 192, 129), (25, 200, 25), (25, 200, 26),
                                   (40, 320, 40), (41, 328, 41)])
def test_short_row_rule(M, N, K, cuda_device):
    """Both sides of every line between the own tiles and cuBLAS, and which side it is (the own tiles count their
    launches)."""
    from gradwave_b200 import _lib
    A, B, C = _rand(2, M, K, seed=1), _rand(2, K, N, seed=2), torch.empty(2, M, N, dtype=torch.complex128, device=cuda_device)
    before = _lib.launch_count()
    _lib.call("gwb_zgemm", 0, 0, M, N, K, 1.0, 0.0, A.data_ptr(), K, M * K, B.data_ptr(), N, K * N, 0.0, 0.0, C.data_ptr(), N,
              M * N, 2, _lib.stream_ptr())
    own = N >= 8 * M and K <= (128 if M <= 24 else M if M <= 40 else 0)
    assert _lib.launch_count() - before == int(own)
    bound = (K + 2) * 2.3e-16 * 2.2 * (A.abs() @ B.abs())   # as above
    assert bool(((C - A @ B).abs() <= bound).all())


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 63, 64])
def test_cholesky_and_inverse(n, cuda_device):
    """L L^H = G and L^-1 L = 1 for two matrices (n eps cond: the random Gram matrices have cond below 1e4), the
    third one indefinite: its pivot is reported, the others unaffected."""
    from gradwave_b200 import _lib
    X = _rand(3, n, 4 * n + 4, seed=n)
    G = X @ X.mH
    G[2, n - 1, n - 1] = -1.0
    F, Li = G.clone(), torch.full((3, n, n), 7.0, dtype=torch.complex128, device=cuda_device)
    info, flag = torch.zeros(3, dtype=torch.int32, device=cuda_device), torch.zeros(1, dtype=torch.int32, device=cuda_device)
    _lib.call("gwb_chol_inv", 3, n, F.data_ptr(), n, n * n, Li.data_ptr(), n * n, info.data_ptr(), flag.data_ptr(),
              _lib.stream_ptr())
    assert info.tolist() == [0, 0, n] and int(flag) == 2
    L = torch.tril(F[:2])
    eye = torch.eye(n, dtype=torch.complex128, device=cuda_device)
    assert float((L @ L.mH - G[:2]).norm() / G[:2].norm()) < n * 2.3e-16 * 4
    assert float((Li[:2] @ L - eye).abs().max()) < n * 2.3e-16 * 1e4
    assert not torch.triu(Li[:2], 1).any()
    assert bool((Li[2] == 7.0).all())


def _err_extended(got, a, b):
    """Relative 2-norm error of got against a b in extended precision."""
    g, ar, br = [(v.real.astype(np.longdouble), v.imag.astype(np.longdouble))
                 for v in (np.asarray(x.resolve_conj().cpu()) for x in (got, a, b))]
    re, im = ar[0] @ br[0] - ar[1] @ br[1], ar[0] @ br[1] + ar[1] @ br[0]
    return float(np.sqrt(((g[0] - re) ** 2 + (g[1] - im) ** 2).sum() / (re ** 2 + im ** 2).sum()))


# rounding of one operation on numbers of the result's size: uniform in half a unit
_ROUND = 2.0 ** -53 / np.sqrt(3.0)


@pytest.mark.parametrize("op,M,N,K", [(0, 24, 256, 96), (1, 24, 256, 96), (0, 8, 512, 128), (1, 8, 512, 128), (0, 40, 512, 40)])
def test_short_row_products_rounding(op, M, N, K, cuda_device):
    """Rounding of a random product. A sum that grows like sqrt(k) errs by sqrt(n / 2) roundings of its final size
    after n of them: chains of 16 and one addition per 8 terms give sqrt(8 + K / 16), plus the last operations;
    one chain of 2 K roundings would give sqrt(K)."""
    from gradwave_b200 import _lib
    A, B = _rand(*((M, K) if op == 0 else (K, M)), seed=1), _rand(K, N, seed=2)
    C = torch.empty(M, N, dtype=torch.complex128, device=cuda_device)
    _lib.call("gwb_zgemm", op, 0, M, N, K, 1.0, 0.0, A.data_ptr(), A.shape[1], 0, B.data_ptr(), N, 0, 0.0, 0.0,
              C.data_ptr(), N, 0, 1, _lib.stream_ptr())
    assert _err_extended(C, A if op == 0 else A.T, B) < _ROUND * np.sqrt(10 + K / 16)


@pytest.mark.parametrize("M,N,K", [(24, 24, 100), (24, 24, 128), (33, 61, 250)])
def test_a_bh_products_rounding(M, N, K, cuda_device):
    """As above with chains of 32 terms (64 roundings) and slices of at least 64 terms: sqrt(32 + K / 64 + 2)."""
    from gradwave_b200 import _lib
    A, B = _rand(M, K, seed=1), _rand(N, K, seed=2)
    C, work = torch.empty(M, N, dtype=torch.complex128, device=cuda_device), torch.empty(8 << 20, dtype=torch.uint8, device=cuda_device)
    _lib.call("gwb_zgemm_nh", M, N, K, 1.0, 0.0, A.data_ptr(), K, 0, B.data_ptr(), K, 0, 0.0, 0.0, C.data_ptr(), N, 0, 1,
              work.data_ptr(), work.numel(), _lib.stream_ptr())
    assert _err_extended(C, A, B.mH) < _ROUND * np.sqrt(34 + K / 64)


@pytest.mark.parametrize("nproj", [320, 321, 864])
def test_nonlocal_rounding(nproj, cuda_device):
    """S c where the projector sum outweighs c: the contraction (as above, 500 plane waves), and the update with one
    chain up to 320 projectors (2 nproj roundings), chains of 8 beyond."""
    from gradwave_b200.basis import BatchedK
    from gradwave_b200.uspp import BatchedHS
    npw, nb, n = 500, 8, 12
    g = torch.Generator().manual_seed(1)
    z = torch.zeros(1, npw, dtype=torch.float64)
    d = torch.eye(nproj, dtype=torch.float64)
    bk = BatchedK(torch.tensor([npw]), torch.ones(1, npw, dtype=torch.bool), torch.randperm(n ** 3, generator=g)[None, :npw],
                  torch.zeros(1, npw, 3, dtype=torch.float64), z, torch.zeros(0, dtype=torch.complex128),
                  torch.zeros(nproj, dtype=torch.int64), d).to(cuda_device)
    p, c = _rand(1, nproj, npw, seed=5), _rand(1, nb, npw, seed=6)
    v = torch.zeros(n, n, n, dtype=torch.float64, device=cuda_device)
    s = BatchedHS(bk, (n, n, n), v, p, d, d).hs(c)[1]
    pe, ce = np.asarray(p[0].cpu()), np.asarray(c[0].cpu())
    pr, pi, cr, ci = (x.astype(np.longdouble) for x in (pe.real, pe.imag, ce.real, ce.imag))
    br, bi = cr @ pr.T + ci @ pi.T, ci @ pr.T - cr @ pi.T
    re, im = cr + br @ pr - bi @ pi, ci + br @ pi + bi @ pr
    got = np.asarray(s[0].cpu())
    err = float(np.sqrt(((got.real - re) ** 2 + (got.imag - im) ** 2).sum() / (re ** 2 + im ** 2).sum()))
    update = nproj if nproj <= 320 else 8 + nproj / 16
    assert err < _ROUND * np.sqrt(34 + npw / 64 + update + 4)


def test_cholesky_of_pivots(cuda_device):
    """1 x 1 matrices: the factor is the rounded square root and its inverse the rounded quotient, to the last bit."""
    from gradwave_b200 import _lib
    g = torch.rand(4096, dtype=torch.float64, generator=torch.Generator().manual_seed(1)) * 100.0
    F = g.to(torch.complex128).to(cuda_device)
    Li, info = torch.empty_like(F), torch.zeros(4096, dtype=torch.int32, device=cuda_device)
    _lib.call("gwb_chol_inv", 4096, 1, F.data_ptr(), 1, 1, Li.data_ptr(), 1, info.data_ptr(), None, _lib.stream_ptr())
    root = np.sqrt(g.numpy())
    assert np.array_equal(F.cpu().numpy(), root.astype(np.complex128))
    assert np.array_equal(Li.cpu().numpy(), (1.0 / root).astype(np.complex128))
