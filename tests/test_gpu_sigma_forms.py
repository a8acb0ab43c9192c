"""The sigma product's kernels by the size of the space: four warps a configuration (784
determinants), one (3025), the general kernel with its matrix kept in the caches (4356) and
read past them (8281): <A|H|A> against the contraction with the reduced density matrices,
for two random vectors and their sums, which fix the off-diagonal elements between them.

Tolerance 1e-10 of the energy, as the other test of this identity (both sides sum some 1e6
products of either sign)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 11, 12, 14])
@pytest.mark.parametrize("ez", [0.0, 0.05])
def test_energy_through_sigma_and_density_matrices(built_lib, n, ez):
    from sincgpu import SincProject, WalkTables
    from oracle import sinc_oracle as orc
    sysm = orc.SincSystem(9, 0.5, [[0, 0, 0]], [4.0])
    phi = orc.seeded_orbitals(sysm, n, seed=n)
    ph = np.conj(phi).T
    pot, ke, z = ph @ sysm.mult_pot(phi), ph @ sysm.mult_ke(phi), ph @ sysm.mult_zdipole(phi)
    with SincProject(9, 0.5, [[0, 0, 0]], [4.0], n) as gpu:
        walks = WalkTables(4, n, 0)
        gpu.ci_attach(walks)
        mat, _ = gpu.call_twoe_matel00(phi)
        gpu.assemble_sparsemats(mat, pot, ke, z)
        rng = np.random.default_rng(n)
        a, b = (rng.standard_normal(walks.numconfig) + 1j * rng.standard_normal(walks.numconfig) for _ in range(2))
        for v in (a, b, a + b, a + 1j * b):
            v = v / np.linalg.norm(v)
            e_sigma = np.vdot(v, gpu.sparseconfigmult(v, ezfield=ez))
            den, _ = gpu.getdenmat(v)
            tally = gpu.get_tworeducedx(v)
            e_rdm = np.sum((pot + ke + ez * z) * den.T) + 0.5 * np.sum(mat * tally)
            assert abs(e_sigma - e_rdm) < 1e-10 * abs(e_rdm)
