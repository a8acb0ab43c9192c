"""The one-CTA kernels of the small matrices at the edges of their tiles: the matrix
exponential behind the Krylov propagators (8 x 8 tiles; shared memory up to order 64, global
beyond) and the symmetric orthogonalisation (a column pair per warp, odd counts with a bye).

Tolerances: a Krylov step is accepted at a local error of 1e-12 and a propagation takes some
ten of them, with FP64 roundoff of the same size: 1e-10 of the unit norm.  The overlap sums
343 products of order 1/343 and its root n <= 32 of order 1: 1e-12, as the other
orthogonalisation test."""
import numpy as np
import pytest
import scipy.linalg as sl

from oracle import orbprop_oracle as op
from oracle import sinc_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ci(built_lib):
    from sincgpu import SincProject, WalkTables
    n = 5
    sysm = orc.SincSystem(11, 0.5, [[0, 0, 0]], [2.0])
    with SincProject(11, 0.5, [[0, 0, 0]], [2.0], n) as gpu:
        walks = WalkTables(4, n, 0)
        gpu.ci_attach(walks)
        phi = orc.seeded_orbitals(sysm, n, seed=3)
        mat, _ = sysm.call_twoe_matel00(phi, phi)
        ph = np.conj(phi).T
        gpu.assemble_sparsemats(mat, ph @ sysm.mult_pot(phi), ph @ sysm.mult_ke(phi), ph @ sysm.mult_zdipole(phi))
        nc = 100
        H = np.column_stack([gpu.sparseconfigmult(e) for e in np.eye(nc, dtype=np.complex128)])
        rng = np.random.default_rng(4)
        a = rng.standard_normal(nc) + 1j * rng.standard_normal(nc)
        yield gpu, H, a / np.linalg.norm(a)


# the exponential has the order m + 2
@pytest.mark.parametrize("m", [4, 5, 6, 7, 14, 15, 30, 31, 61, 62, 63, 70, 100])
def test_matrix_exponential(ci, m):
    gpu, H, a = ci
    tf = -0.02j * m
    w, _, _ = gpu.expoavecprop(a, 1.0, krylovdim=m, tol=1e-12, anorm=abs(tf), stepguess=1.0, timefac=tf)
    assert np.abs(w - sl.expm(tf * H) @ a).max() < 1e-10


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 15, 16, 17, 31, 32])
def test_orthogonalisation(built_lib, n):
    import torch
    from sincgpu import SincProject
    sysm = orc.SincSystem(7, 0.5, [[0, 0, 0]], [2.0])
    rng = np.random.default_rng(n)
    phi = orc.seeded_orbitals(sysm, n, seed=n)
    bad = phi + 0.05 * (rng.standard_normal(phi.shape) + 1j * rng.standard_normal(phi.shape)) * np.abs(phi)
    ref, err_ref = op.spf_orthogit(bad)
    d = torch.from_numpy(np.ascontiguousarray(bad.T)).cuda()
    with SincProject(7, 0.5, [[0, 0, 0]], [2.0], n) as gpu:
        err = gpu.spf_orthogit_dev(d)
    out = d.cpu().numpy().T
    assert np.abs(out - ref).max() < 1e-12
    assert np.abs(np.conj(out).T @ out - np.eye(n)).max() < 1e-12
    assert err == pytest.approx(err_ref, abs=1e-12)


# 784 determinants: four warps a configuration; 3025: one; 14400: the general kernel, and
# vectors whose rows beyond the eleventh stay outside shared memory
@pytest.mark.parametrize("numelec,n,m", [(4, 8, 20), (4, 11, 20), (4, 16, 18)])
def test_krylov_forms(built_lib, numelec, n, m):
    from sincgpu import SincProject, WalkTables
    sysm = orc.SincSystem(9, 0.5, [[0, 0, 0]], [2.0])
    with SincProject(9, 0.5, [[0, 0, 0]], [2.0], n) as gpu:
        walks = WalkTables(numelec, n, 0)
        nc = walks.numconfig
        gpu.ci_attach(walks)
        phi = orc.seeded_orbitals(sysm, n, seed=5)
        rng = np.random.default_rng(6)
        mat = rng.standard_normal((n,) * 4) + 1j * rng.standard_normal((n,) * 4)
        mat = (mat + np.conj(mat.transpose(2, 3, 0, 1))) / n
        ph = np.conj(phi).T
        gpu.assemble_sparsemats(np.asfortranarray(mat), ph @ sysm.mult_pot(phi), ph @ sysm.mult_ke(phi),
                                ph @ sysm.mult_zdipole(phi))
        a = rng.standard_normal(nc) + 1j * rng.standard_normal(nc)
        a /= np.linalg.norm(a)
        outs = []
        for cluster in (1, 0):
            gpu.set_option("kry_cluster", cluster)
            outs.append(gpu.expoavecprop(a, 1.0, krylovdim=m, tol=1e-10, anorm=0.02, stepguess=1.0, timefac=-0.02j,
                                         ezfield=0.1))
        assert outs[0][2] == outs[1][2]
        # two roundings of the same recurrence, as test_matrix_exponential
        assert np.abs(outs[0][0] - outs[1][0]).max() < 1e-10
