"""The dense orbital kernels at the edges of their tiles: the overlap and rotation tiles
(16, 32 and 64 wide), the blocks of 32 of the Cholesky factor and its inverse, and JADE in
one cluster (rows spread over 16 CTAs, 2 or 4 elements a lane) and, above 128 states, step by
step, against numpy and the oracle.

Tolerances: a sum of n rounded FP64 products is within about sqrt(n) 1.1e-16 of its
2-norm; the factor's condition number (below 10 for these sets) multiplies it once."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 129]


def _ham(pb, n=16, precision="fp64"):
    return pb.KSHamiltonian(np.eye(3) * 6.0, (n, n, n), precision)


def _block(h, M, ld, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((h.N, ld, 2), generator=g, device="cuda", dtype=torch.float64)
    return torch.view_as_complex(x).to(dtype)[:, :M]


@pytest.mark.parametrize("M", SIZES)
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-6)])
def test_orthonormalize_edges(pb, M, precision, tol):
    h = _ham(pb, precision=precision)
    x = _block(h, M, M + 3, M, h.dtype)
    pad = x.as_strided((h.N, 3), (M + 3, 1), M).clone()
    ref = x.to(torch.complex128)
    u = torch.linalg.cholesky(h.volume_element * (ref.conj().T @ ref), upper=True)
    ref = torch.linalg.solve_triangular(u, ref, upper=True, left=False)
    h.orthonormalize_(x)
    assert float((x - ref).norm() / ref.norm()) < tol
    assert torch.equal(x.as_strided((h.N, 3), (M + 3, 1), M), pad)  # past the block: untouched


@pytest.mark.parametrize("Ma,Mb", [(1, 1), (5, 33), (33, 5), (17, 64), (65, 100)])
def test_overlap_and_rotate_blocks(pb, Ma, Mb):
    h = _ham(pb)
    a, b = _block(h, Ma, Ma + 1, 1, h.dtype), _block(h, Mb, Mb, 2, h.dtype)
    S = h.overlap_block(a, b)
    ref = h.volume_element * (a.conj().T @ b)
    assert float((S - ref).norm() / ref.norm()) < 1e-13
    got = h.rotate_block(a, S)
    assert float((got - a @ S).norm() / (a @ S).norm()) < 1e-14


@pytest.mark.parametrize("M", SIZES)
def test_cholesky_inverse_edges(pb, M):
    h = _ham(pb)
    x = _block(h, M, M, 7, torch.complex128)
    S = (x.conj().T @ x) / h.N + 0.1 * torch.eye(M, device="cuda")
    big = torch.full((M, M + 2), 5.0 + 1.0j, dtype=torch.complex128, device="cuda")
    big[:, :M] = S
    ref = torch.linalg.inv(torch.linalg.cholesky(S, upper=True))
    got = h.cholesky_inverse_(big[:, :M])
    assert float((got - ref).norm() / ref.norm()) < 1e-13
    assert float(torch.tril(got, -1).abs().sum()) == 0.0
    assert torch.all(big[:, M:] == 5.0 + 1.0j)


@pytest.mark.parametrize("M,zero", [(40, 0), (40, 31), (40, 32), (100, 97)])
def test_cholesky_reports_the_first_failing_pivot(pb, M, zero):
    h = _ham(pb)
    x = _block(h, M, M, 3, torch.complex128).clone()
    x[:, zero] = 0  # an exact zero pivot
    keep = x.clone()
    with pytest.raises(pb.InqbError) as e:
        h.orthonormalize_(x)
    assert f"pivot {zero}" in str(e.value)
    assert torch.equal(x, keep)


@pytest.mark.parametrize("M", [1, 2, 3, 16, 17, 32, 33, 64, 65, 97, 129, 150, 190])
def test_jade_sizes(pb, oracle_mod, M):
    """Hermitian matrices diagonal up to a small unitary mixing: the sweeps of the oracle,
    and its rotation to the accuracy the convergence threshold leaves."""
    rng = np.random.default_rng(M)
    g = 0.3 / np.sqrt(M) * (rng.standard_normal((M, M)) + 1j * rng.standard_normal((M, M)))
    w, v = np.linalg.eigh(1j * (g - g.conj().T))
    q = v @ np.diag(np.exp(-1j * w)) @ v.conj().T
    a = np.stack([q @ np.diag(rng.uniform(-1, 1, M)) @ q.conj().T for _ in range(6)])
    h = _ham(pb)
    maxsweep = 100 if M < 100 else 2  # the CPU oracle multiplies dense rotations
    u, adiag, sweeps = h.jade(torch.as_tensor(a).cuda(), maxsweep, 1e-8)
    _, u_ref, d_ref, sw_ref = oracle_mod.jade(a, maxsweep, 1e-8)
    assert sweeps == sw_ref
    assert np.abs(u.cpu().numpy() - u_ref).max() < 1e-10
    assert np.abs(adiag.cpu().numpy() - d_ref).max() < 1e-10


@pytest.mark.parametrize("Ma,Mb,n", [(33, 33, 16), (40, 72, 16), (136, 41, 16), (70, 200, 32)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-13)])
def test_wide_tiles_of_ragged_blocks(pb, Ma, Mb, n, precision, tol):
    """64-wide tiles whose row blocks, column blocks or both end inside the tile, from
    complex128 and complex64 orbitals; one slab of points to many."""
    h = _ham(pb, n, precision)
    a, b = _block(h, Ma, Ma + 1, 1, h.dtype), _block(h, Mb, Mb + 2, 2, h.dtype)
    wa, wb = a.to(torch.complex128), b.to(torch.complex128)
    ref = h.volume_element * (wa.conj().T @ wb)
    assert float((h.overlap_block(a, b) - ref).norm() / ref.norm()) < tol
    rot = _block(h, Mb, Mb, 3, torch.complex128)[:Ma].contiguous()
    ref = wa @ rot
    # complex64 results are rounded once to 6e-8
    assert float((h.rotate_block(a, rot) - ref).norm() / ref.norm()) < (1e-14 if precision == "fp64" else 1e-7)


@pytest.mark.parametrize("Ma,Mb", [(1, 1), (7, 9), (33, 8), (31, 33), (64, 65), (70, 100)])
def test_gram_and_adjoint_rotation(pb, Ma, Mb):
    """The weighted Gram matrices and psi u^H of complex128 orbitals at the edges of their
    64-wide tiles."""
    h = _ham(pb, 18)
    a, b = _block(h, Ma, Ma + 1, 1, h.dtype), _block(h, Mb, Mb, 2, h.dtype)
    i = torch.arange(18, device="cuda", dtype=torch.float64)
    f = torch.where(i >= 9, i - 18, i) / 18
    for d, Z in enumerate(h.mlwf_gram_block(a, b)):
        shape = [1, 1, 1]
        shape[d] = 18
        w = torch.exp(2j * np.pi * f).reshape(shape).expand(18, 18, 18).reshape(-1, 1)
        ref = a.conj().T @ (w * b)
        assert float((Z - ref).norm() / ref.norm()) < 1e-13
    u = _block(h, Mb, Mb, 4, torch.complex128)[:Mb].contiguous()
    ref = b @ u.conj().T
    assert float((h.mlwf_rotate_(b.clone(), u) - ref).norm() / ref.norm()) < 1e-14
