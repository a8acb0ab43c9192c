"""The five-pass Coulomb solve's z-pass forms at length 162 (81 points a side) against its
plain z pass, and the cluster form of its y and z passes, with the half-length form off:
that form is the default at this size and would serve as the baseline else.

Tolerances: the same transforms in another order of threads, 1e-14 of the largest value, as
the tests of the forms at shorter lengths; 1e-13 between other factorisations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / np.abs(np.asarray(b)).max())


@pytest.fixture(scope="module")
def solver(built_lib):
    from sincgpu import SincProject
    rng = np.random.default_rng(81)
    dens = rng.standard_normal((81 ** 3, 2)) + 1j * rng.standard_normal((81 ** 3, 2))
    with SincProject(81, 0.3, [[0, 0, 0]], [1.0], 2) as gpu:
        half = gpu.op_tinv(dens)
        gpu.set_option("coul_half", 0)
        yield gpu, dens, gpu.op_tinv(dens), half


def test_default_is_the_half_length_form(solver):
    _, _, plain, half = solver
    assert not np.array_equal(half, plain) and relerr(half, plain) < 1e-13


@pytest.mark.parametrize("option", ["coul_z2", "coul_tma"])
def test_z_pass_forms(solver, option):
    gpu, dens, plain, _ = solver
    gpu.set_option(option, 1)
    try:
        other = gpu.op_tinv(dens)
    finally:
        gpu.set_option(option, -1 if option == "coul_tma" else 0)
    assert relerr(other, plain) < 1e-14
    assert gpu.kernel_timeouts() == [0, 0]
    assert np.array_equal(gpu.op_tinv(dens), plain)


def test_cluster_planes(solver):
    gpu, dens, plain, _ = solver
    gpu.set_option("coul_fused", 1)
    try:
        fused = gpu.op_tinv(dens)
    finally:
        gpu.set_option("coul_fused", 0)
    assert relerr(fused, plain) < 1e-13
