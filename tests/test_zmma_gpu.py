"""Float64 tensor-instruction products (split-K A B^H, nonlocal update) at tile edges, against torch."""

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
