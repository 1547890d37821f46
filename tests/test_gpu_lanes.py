"""The tile passes' 16-byte lanes and the flat vector kernels at their edges: blocks whose
rows are and are not 16-byte aligned give the same numbers bit for bit (the same arithmetic
on other accesses), orbital counts around a lane and a group, and atoms beyond what a
tile's accumulators and staged projections hold."""
import numpy as np
import pytest
import torch

from helpers import make_oracle, make_product, rel_max, small_system

pytestmark = pytest.mark.gpu


def _pair(h, M, pad, seed=0):
    """The same random block contiguous and with `pad` more columns a row."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.view_as_complex(torch.randn((h.N, M, 2), generator=g, device="cuda", dtype=torch.float64)).to(h.dtype)
    wide = torch.full((h.N, M + pad), 3.0, dtype=h.dtype, device="cuda")
    wide[:, :M] = x
    return x.clone(), wide, wide[:, :M]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("M,pad", [(8, 1), (8, 2), (16, 3), (7, 1), (1, 1), (9, 0)])
def test_row_alignment_does_not_change_the_numbers(pb, precision, M, pad):
    sysd = small_system(pb, n=20, a=6.4, M=1)
    h = make_product(pb, sysd, precision, (0.02, 0.0, 0.01))
    h.set_fourier_sphere_mask(True)
    k = [h.cart_to_cov([0.01 * i, 0.0, 0.0]) for i in (1, 2)]
    occ = np.full(M, 2.0)
    rho0 = h.density(_pair(h, M, 0)[0], occ)
    V = sysd["V"]
    vion = torch.as_tensor(V).cuda()

    def scf(p):
        rho = rho0.clone()
        h.set_scalar_potential(V)
        h.ks_potential(rho, vion, 2, energies=False)
        h.etrs_scf_step_(p, rho, 0.05, k[0], k[1], occ, vion, 2, nscf=1)

    runs = [lambda p: h.exponential_(p, 0.05j, 3), lambda p: h.exponential_(p, 0.05j, 1),
            lambda p: h.etrs_step_terms_(p, 0.05, k[0], k[1]),
            lambda p: h.crank_nicolson_step_(p, 0.05, k[0], k[1], 1, 0.0), scf]
    for run in runs:
        x, wide, view = _pair(h, M, pad)
        if pad == 0:  # an odd FP32 row count still is one aligned run or none: compare with a padded copy
            _, wide, view = _pair(h, M, 1)
        edge = wide[:, M:].clone()
        run(x)
        run(view)
        assert torch.isfinite(torch.view_as_real(x)).all()
        assert torch.equal(x, view)
        assert torch.equal(wide[:, M:], edge)


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 15, 16, 17, 33])
@pytest.mark.parametrize("n", [16, 18])
def test_density_sizes(pb, n, M):
    h = pb.KSHamiltonian(np.eye(3) * 6.0, (n, n, n), "mixed")
    x, _, view = _pair(h, M, 3, seed=M)
    occ = np.linspace(0.5, 2.0, M)
    ref = (x.to(torch.complex128).abs() ** 2 @ torch.as_tensor(occ).cuda())
    for p in (x, view):
        assert float((h.density(p, occ) - ref).abs().max() / ref.max()) < 1e-14


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-5)])
@pytest.mark.parametrize("atoms", [200, 400])
def test_more_atoms_than_a_tile_stages(pb, oracle_mod, precision, tol, atoms):
    """Up to 400 atoms over every plane and tile of a 16^3 grid: past the accumulators (192
    atoms a plane) and past the staged projections (320 segments a tile), with many entries
    a grid point."""
    sysd = small_system(pb, n=16, a=5.0, M=5)
    sysd["positions"] = np.random.default_rng(3).uniform(0, 5.0, (atoms, 3))
    h = make_product(pb, sysd, precision, (0.1, 0.2, 0.3))
    o = make_oracle(oracle_mod, sysd, (0.1, 0.2, 0.3))
    x = torch.as_tensor(sysd["psi"]).to(h.dtype).cuda()
    # up to 360 entries a point: their FP32 sum is within about sqrt(360) 6e-8 of its terms' norm
    assert rel_max(h(x).cpu().numpy(), o.apply_h(x.cpu().numpy().astype(np.complex128))) < tol
    assert torch.equal(h(x), h(x))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-6)])
@pytest.mark.parametrize("n,M", [(80, 1), (80, 7), (80, 17), (128, 5)])
def test_long_axes(pb, precision, tol, n, M):
    """Axes whose transforms are longer than 12 values: one orbital a lane in FP32, 512
    threads in the first and third pass, against the same passes with 64 and 256 threads
    (sums of the projections in another order), in rows of both alignments."""
    sysd = small_system(pb, n=n, a=0.3 * n, M=1)
    h = make_product(pb, sysd, precision, (0.02, 0.0, 0.01))
    x, _, view = _pair(h, M, 1)
    y = h(x)
    assert torch.isfinite(torch.view_as_real(y)).all()
    assert torch.equal(y, h(view))
    for threads in (64, 256):
        h.set_schedule(M, (1, threads, threads, threads))
        assert float((h(x) - y).norm() / y.norm()) < tol
    picked = h.autotune(M)
    h.set_schedule(M, picked)  # what the tuner picks can be set again
    assert float((h(x) - y).norm() / y.norm()) < tol
