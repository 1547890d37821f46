"""The 3 x 3 eigenproblem of a JADE rotation (FP32 iteration, refined in FP64) by itself: two
states have one pair and one rotation, so one sweep returns it.  The reference is the FP64
iteration's steps in extended precision (64-bit mantissa): the same column and sign, and the
same rotation to FP64 rounding, no further off than the FP64 iteration itself."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 2.0**-52


def jacobi_top(G, dtype):
    """Top eigenvector of each G [B, 3, 3] as the cyclic Jacobi iteration leaves it, in dtype."""
    S, B = G.astype(dtype), len(G)
    V = np.tile(np.eye(3, dtype=dtype), (B, 1, 1))
    d = S[:, range(3), range(3)].copy()
    one = dtype(1)
    with np.errstate(all="ignore"):
        for _ in range(60):
            off = S[:, 0, 1]**2 + S[:, 0, 2]**2 + S[:, 1, 2]**2
            thresh = np.sqrt(off) / 12
            if not (off > 0).any():
                break
            for p, q in ((0, 1), (0, 2), (1, 2)):
                x = S[:, p, q].copy()
                small = np.abs(x) <= np.finfo(dtype).eps**2 * np.minimum(np.abs(d[:, p]), np.abs(d[:, q]))
                go = (np.abs(x) >= thresh) & (off > 0) & (x != 0) & ~small
                S[small, p, q] = 0
                h, e2 = d[:, q] - d[:, p], 2 * np.abs(x)
                dd = np.abs(h) + np.sqrt(h * h + e2 * e2)
                sg = np.where((h != 0) & ((h < 0) != (x < 0)), -one, one)
                r = np.sqrt(dd * dd + e2 * e2)
                t, c, s = sg * e2 / dd, dd / r, sg * e2 / r
                tau = s / (1 + c)
                t, s, tau = (np.where(go, v, 0) for v in (t, s, tau))
                d[:, p] -= t * x
                d[:, q] += t * x
                S[go, p, q] = 0

                def rot(M, a, b):
                    g, f = M[a].copy(), M[b].copy()
                    M[a], M[b] = g - s * (f + g * tau), f + s * (g - f * tau)

                j = 3 - p - q
                up = lambda a, b: (slice(None), min(a, b), max(a, b))
                rot(S, up(j, p), up(j, q))
                for j in range(3):
                    rot(V, (slice(None), j, p), (slice(None), j, q))
    w = np.sort(d, axis=1)
    return V[np.arange(B), :, d.argmax(1)], ((w[:, 2] - w[:, 1]) / w[:, 2]).astype(float)


def rotation(v):
    x, y, z = np.abs(v[:, 0]), np.where(v[:, 0] < 0, -v[:, 1], v[:, 1]), v[:, 2]
    c = np.sqrt((x + 1) / 2)
    return np.stack([c, y / (2 * c), -z / (2 * c)], 1)


def orthogonal(rng, n):
    q, r = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    return q * np.sign(r[:, range(3), range(3)])[:, None, :]


def spectra(rng, n, kind):
    """Vectors h [n, 6, 3], whole multiples of 2^-20 so that G = sum h h^T is exact in FP64."""
    h = np.zeros((n, 6, 3))
    if kind == "random":
        h = rng.standard_normal((n, 6, 3)) * rng.uniform(0.01, 1, (n, 6, 1))
    else:
        lo = {"apart": rng.uniform(0, 0.9, (n, 2)), "close below": rng.uniform(0, 0.9, (n, 1)) + rng.uniform(0, 1e-6, (n, 2)),
              "near the gap": rng.uniform(0.96, 0.985, (n, 2)), "close on top": 1 - rng.uniform(1e-3, 1e-2, (n, 2)),
              "one vector": rng.uniform(0, 1e-8, (n, 2)), "near 45 degrees": rng.uniform(0, 0.9, (n, 2))}[kind]
        q = orthogonal(rng, n)
        if kind == "near 45 degrees":
            a = np.pi / 4 + rng.uniform(-1e-3, 1e-3, n)
            q = np.zeros((n, 3, 3))
            q[:, 0, 0] = q[:, 1, 1] = np.cos(a)
            q[:, 1, 0], q[:, 0, 1], q[:, 2, 2] = np.sin(a), -np.sin(a), 1
            q = q[np.arange(n)[:, None], np.argsort(rng.random((n, 3)), 1)]
        lam = np.concatenate([np.ones((n, 1)), lo], 1)
        h[:, :3] = np.sqrt(lam)[:, :, None] * q.transpose(0, 2, 1)
    return np.round(h * 2.0**20) * 2.0**-20


KINDS = ["random", "apart", "close below", "near the gap", "close on top", "one vector", "near 45 degrees"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("scale", [1.0, 2.0**-100, 2.0**100])
def test_rotation_of_a_pair(pb, kind, scale):
    """Error bound: a dozen rotations' rounding, 64 eps of |G|, over the relative gap below the
    top eigenvalue."""
    rng = np.random.default_rng(KINDS.index(kind))
    h = spectra(rng, 400, kind)
    G = np.einsum("bki,bkj->bij", h, h)
    v, gap = jacobi_top(G, np.longdouble)
    keep = np.abs(v[:, 0]) > 1e-4  # at 0 the rotation's sign changes sides
    h, v, gap, G = h[keep], v[keep], gap[keep], G[keep]
    ref = rotation(v)
    fp64 = rotation(jacobi_top(G, np.float64)[0])
    a = np.zeros((len(h), 6, 2, 2), complex)
    a[:, :, 0, 0], a[:, :, 1, 1] = h[:, :, 0] / 2, -h[:, :, 0] / 2
    a[:, :, 0, 1] = (h[:, :, 1] + 1j * h[:, :, 2]) / 2
    a[:, :, 1, 0] = a[:, :, 0, 1].conj()
    ham = pb.KSHamiltonian(np.eye(3) * 6.0, (16, 16, 16), "fp64")
    dev = torch.as_tensor(a * scale).cuda()
    u = torch.stack([ham.jade(m, 1, 1e-300)[0] for m in dev]).cpu().numpy()
    got = np.stack([u[:, 0, 0].real, -u[:, 1, 0].real, -u[:, 1, 0].imag], 1)
    err, err64 = (np.abs(x - ref).max(1).astype(float) for x in (got, fp64))
    assert (err < 64 * EPS / gap).all()
    # no further off than the FP64 iteration, up to three standard errors of the root mean
    # squares of 250 and more rotations
    assert np.sqrt((err**2).mean()) < 1.15 * np.sqrt((err64**2).mean())
