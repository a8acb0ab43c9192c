"""twoematel and reducedpot of hermitian pairs without the diagonal pairs' imaginary rows,
through the A-vector orbital-RHS call, at the orbital counts where the kernels and their
tiles change: one symmetric tile (up to 12 orbitals), patches of the triangle (13 to 16),
several tiles (17); column tiles of 32 to 128, with the apply in the epilogue up to 10.

Tolerance 1e-11, as the other parity tests against the oracle (sums of N^3 = 343 products
after two transforms)."""
import numpy as np
import pytest

from oracle import sinc_oracle as orc
from oracle.walks_oracle import CIWalks

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / np.abs(np.asarray(b)).max())


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17])
def test_rhs_from_avector(built_lib, n):
    import torch
    from sincgpu import SincProject, WalkTables
    N, d = 7, 0.5
    sysm = orc.SincSystem(N, d, [[0, 0, 2]], [2.0], toothnbig=16, toothnsmall=6)
    phi = orc.seeded_orbitals(sysm, n, seed=n)
    ww = CIWalks(2, n, 0)
    rng = np.random.default_rng(n)
    a = rng.standard_normal(ww.numconfig) + 1j * rng.standard_normal(ww.numconfig)
    a /= np.linalg.norm(a)
    den, tally = ww.getdenmat00(a), ww.get_tworeducedx(a)
    inv = orc.invmatsmooth(den)
    mat, red = sysm.call_twoe_matel00(phi, phi)
    rp = orc.get_reducedpot(red, tally)
    out = orc.actreduced00(sysm, phi, phi, den, inv, rp)
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(np.asarray(v).T)).cuda()  # noqa: E731
    z = lambda *s: torch.zeros(*s, dtype=torch.complex128, device="cuda")  # noqa: E731
    with SincProject(N, d, [[0, 0, 2]], [2.0], n, toothnbig=16, toothnsmall=6) as gpu:
        gpu.ci_attach(WalkTables(2, n, 0))
        bufs = [z(n, n), z(n, n), z(n, n, n, n), z(n, n, n, n), z(n, n, N ** 3), z(n, N ** 3)]
        gpu.orbital_rhs_avec_dev(dev(phi), dev(a), *bufs)
        gpu.synchronize()
        got = [b.cpu().numpy().T for b in bufs]
    for g, r in zip(got[2:], (tally, mat, rp, out)):
        assert relerr(g, r) < 1e-11
