"""The generalized (USPP/PAW) band solve on the GPU (``gradwave_b200.uspp``)
against the reference's own ``BatchedHS.s`` and ``davidson_gen_batched``
(gradwave ``scf/uspp_batch.py``).

Golden values come from the reference on the si2 and si8 cells with a seeded
augmentation matrix q (``tests/golden/make_golden.py uspp``): checksums of S on
a seeded block (float64, bar 1e-12 relative) and the eigenvalues of
H x = eps S x from the identity start at tol 1e-10 eV (bar 1e-8 Ha, the
band-solve parity bar, with 1e-9 eV reached in practice). Size-independent
checks: S-orthogonality of the returned Ritz vectors and their residuals.
"""

import numpy as np
import pytest
import torch

from tests.conftest import load_golden
from tests.golden.make_golden import checksums, random_block

pytestmark = pytest.mark.gpu

HA = 27.211386245988


def _hs(name, dev):
    from gradwave_b200.cells import make_cell
    from gradwave_b200.uspp import BatchedHS
    g = load_golden(f"uspp_{name}")
    ci = make_cell(name)
    bk = ci.bk.to(dev)
    hs = BatchedHS(bk, ci.shape, ci.v_eff_r, ci.p, bk.dij_full, torch.from_numpy(g["q"]))
    return g, ci, hs


@pytest.mark.parametrize("name", ["si2_fcc", "si8_cubic"])
def test_overlap_apply_matches_reference(cuda_device, name):
    g, ci, hs = _hs(name, cuda_device)
    seed = int(g["seed"])
    c = torch.from_numpy(random_block(seed, ci.bk.nk, 2, ci.bk.npw_max)).to(cuda_device)
    chk = checksums(hs.s(c).cpu().numpy(), seed)
    assert np.abs(chk - g["s_chk"]).max() <= 1e-12 * np.abs(g["s_chk"]).max()


@pytest.mark.parametrize("name", ["si2_fcc", "si8_cubic"])
def test_generalized_davidson_matches_reference(cuda_device, name):
    from gradwave_b200.uspp import davidson_gen_batched
    g, ci, hs = _hs(name, cuda_device)
    x0 = ci.identity_start().to(cuda_device)
    eig, x = davidson_gen_batched(hs, x0, ci.nbands, tol=1e-10, max_iter=200)
    err = np.abs(eig.cpu().numpy() - g["eigenvalues"]).max()
    assert err < 1e-8 * HA
    assert err < 1e-9
    # Ritz vectors: S-orthogonal (up to their norms) with residual below tol
    hx, sx = hs.h(x), hs.s(x)
    r = hx - eig[..., None].to(x.dtype) * sx
    assert float(torch.linalg.vector_norm(r, dim=-1).max()) < 1e-10
    m = torch.matmul(x.conj(), sx.transpose(-1, -2))
    d = torch.diagonal(m, dim1=-2, dim2=-1).real
    off = m - torch.diag_embed(torch.diagonal(m, dim1=-2, dim2=-1))
    assert float(off.abs().max()) < 1e-8 * float(d.max())


@pytest.mark.parametrize("name", ["si2_fcc", "si8_cubic"])
def test_fused_hs_apply(cuda_device, name):
    """gwb_ham_apply_hs: H c from the fused pass equals the plain apply (the
    same arithmetic in the same order), and S c equals the float64 oracle's
    overlap apply; float32 arithmetic within its bar."""
    from oracle.uspp import s_apply
    g, ci, hs = _hs(name, cuda_device)
    c = torch.from_numpy(random_block(int(g["seed"]) + 3, ci.bk.nk, 5, ci.bk.npw_max)).to(cuda_device)
    c = c * hs.mask[:, None, :]
    h_out, s_out = hs.hs(c)
    h_ref = hs.h(c)
    scale = float(h_ref.abs().max())
    assert float((h_out - h_ref).abs().max()) <= 1e-14 * scale
    s_ref = s_apply(ci.p.numpy(), g["q"], ci.bk.mask.numpy(), c.cpu().numpy())
    assert np.abs(s_out.cpu().numpy() - s_ref).max() <= 1e-12 * np.abs(s_ref).max()
    h32, s32 = hs.hs(c.to(torch.complex64))
    assert float((h32.to(torch.complex128) - h_ref).abs().max()) <= 3e-6 * scale
    assert np.abs(s32.cpu().numpy() - s_ref).max() <= 3e-6 * np.abs(s_ref).max()


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
def test_fused_hs_apply_without_projectors(cuda_device, dtype):
    """No projectors: H c is the plain apply, S c the masked block; many small applies in a row, so that the kernel
    that copies c runs close behind the local term's last one."""
    from gradwave_b200.basis import BatchedK
    from gradwave_b200.hamiltonian import BatchedHamiltonian
    from gradwave_b200.uspp import BatchedHS
    npw, nb, n = [300, 211], 70, 12
    g = torch.Generator().manual_seed(3)
    mask = torch.zeros(2, 300, dtype=torch.bool)
    flat = torch.zeros(2, 300, dtype=torch.int64)
    for k in range(2):
        mask[k, :npw[k]] = True
        flat[k, :npw[k]] = torch.randperm(n ** 3, generator=g)[:npw[k]]
    bk = BatchedK(torch.tensor(npw), mask, flat, torch.zeros(2, 300, 3, dtype=torch.float64),
                  torch.rand(2, 300, dtype=torch.float64, generator=g) * mask, torch.zeros(0, dtype=torch.complex128),
                  torch.zeros(0, dtype=torch.int64), torch.zeros(0, 0, dtype=torch.float64)).to(cuda_device)
    v = torch.randn(n, n, n, dtype=torch.float64, generator=g).to(cuda_device)
    p = torch.zeros(2, 0, 300, dtype=torch.complex128, device=cuda_device)
    hs = BatchedHS(bk, (n, n, n), v, p, bk.dij_full, bk.dij_full)
    c = torch.randn(2, nb, 300, dtype=torch.complex128, generator=g).to(cuda_device).to(dtype)
    ref = BatchedHamiltonian(bk, (n, n, n), v, p).apply(c)
    for _ in range(20):
        h, s = hs.hs(c)
        assert torch.equal(h, ref)
        assert torch.equal(s, c * bk.mask[:, None, :])
