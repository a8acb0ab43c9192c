"""Krylov chains whose vectors lose their orthogonality, far above rounding: under an
operator whose mean is large against its spread (a long chain's Gram-Schmidt then has to
solve its triangular system in full: cut after the first power of the loss, the Hessenberg
matrix and the result grew without bound), and close to a breakdown under a large norm.
Against the exact exponential and the sequential projections, in all launch forms.

Tolerances: as test_gpu_small_matrices (1e-10 of a unit vector: the accepted local errors
and a rounding of eps t |A|), as test_gpu_orbital_algebra (1e-12 between two roundings of the
same recurrence) for the short orbital chain."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [300.0, 3000.0])
@pytest.mark.parametrize("m,ta", [(30, 15.0), (60, 40.0), (100, 70.0)])
def test_avector_large_mean(built_lib, mean, m, ta):
    from sincgpu import SincProject, WalkTables
    n = 10
    rng = np.random.default_rng(5)
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    levels = (np.where(np.arange(n) < n // 2, -1, 1) + 0.1 * np.linspace(-1, 1, n)) / 2
    h = (Q * levels) @ Q.T + mean / 2 * np.eye(n)
    with SincProject(5, 0.5, [[0, 0, 0]], [0.0], n) as gpu:
        walks = WalkTables(2, n, 0)
        nc = walks.numconfig
        gpu.ci_attach(walks)
        zero = np.zeros((n, n), dtype=np.complex128)
        gpu.assemble_sparsemats(np.zeros((n,) * 4, dtype=np.complex128), (h + h.T) / 2 + zero, zero, zero)
        w, U = np.linalg.eigh(np.column_stack([gpu.sparseconfigmult(e) for e in np.eye(nc, dtype=np.complex128)]))
        t = ta / np.abs(w).max()
        for seed in range(4):
            a = np.random.default_rng(seed).standard_normal((2, nc))
            a = (a[0] + 1j * a[1]) / np.linalg.norm(a)
            ref = U @ (np.exp(-1j * t * w) * (U.conj().T @ a))
            steps = []
            for cluster in (1, 0):
                gpu.set_option("kry_cluster", cluster)
                out, _, nstep = gpu.expoavecprop(a, t, krylovdim=m, tol=1e-12, anorm=mean, stepguess=t, timefac=-1j)
                steps.append(nstep)
                assert np.abs(out - ref).max() < 1e-10
            assert steps[0] == steps[1]


@pytest.mark.parametrize("m,ta", [(60, 40.0), (100, 70.0)])
def test_orbitals_large_mean(built_lib, m, ta):
    import torch
    from sincgpu import SincProject
    N, mean = 5, 1000.0
    rng = np.random.default_rng(m)
    phi = rng.standard_normal((N ** 3, 2)) + 1j * rng.standard_normal((N ** 3, 2))
    phi = np.linalg.qr(phi)[0]
    rp = np.zeros((2, 2, N ** 3), dtype=np.complex128)
    rp[0, 0] = rp[1, 1] = mean + rng.standard_normal(N ** 3)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    one = np.eye(2, dtype=np.complex128)
    dt = ta / (mean + 5.0)
    outs = []
    with SincProject(N, 2.0, [[0, 0, 0]], [0.0], 2, toothnbig=16, toothnsmall=6) as gpu:
        slot = (dev(one), dev(one), dev(rp))
        for onepass, fused in ((0, 0), (1, 1), (1, 0)):
            gpu.set_option("orth_onepass", onepass)
            gpu.set_option("orth_fused", fused)
            gpu.orbprop_setup(m, m, 1.2, dt)
            d = dev(phi.T.copy())
            gpu.expospfprop_dev(d, slot, slot, 0.0, dt, 0.0, dt, True, expotol=1e-12)
            outs.append(d.cpu().numpy())
    assert np.abs(outs[1] - outs[0]).max() < 1e-10
    assert np.array_equal(outs[1], outs[2])


@pytest.mark.parametrize("scale", [1.0, 1e3, 1e5])
@pytest.mark.parametrize("small", [1.5e-7, 1e-5])
def test_avector_chain(built_lib, scale, small):
    from sincgpu import SincProject, WalkTables
    n = 16
    couplings = np.array([1, 1, small / scale, 1, 1, small / scale, 1, 1, 0.0])
    T = np.zeros((n, n))
    for i, x in enumerate(couplings):
        T[i, i + 1] = T[i + 1, i] = x
    T[10:, 10:] = np.diag(np.linspace(-1, 1, n - 10))
    rng = np.random.default_rng(int(scale))
    U = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    H = scale * (U @ T @ U.conj().T)
    H = (H + H.conj().T) / 2
    with SincProject(5, 0.5, [[0, 0, 0]], [0.0], n) as gpu:
        walks = WalkTables(1, n, 1)
        assert walks.numconfig == n
        gpu.ci_attach(walks)
        zero = np.zeros((n, n), dtype=np.complex128)
        gpu.assemble_sparsemats(np.zeros((n,) * 4, dtype=np.complex128), H, zero, zero)
        full = np.column_stack([gpu.sparseconfigmult(e) for e in np.eye(n, dtype=np.complex128)])
        assert np.abs(full - H).max() < 1e-12 * scale
        a = np.ascontiguousarray(U[:, 0])
        t = 1.0 / scale
        ref = sl.expm(-1j * t * full) @ a
        for cluster in (1, 0):
            gpu.set_option("kry_cluster", cluster)
            w, _, _ = gpu.expoavecprop(a, t, krylovdim=14, tol=1e-12, anorm=scale, stepguess=t, timefac=-1j)
            assert np.abs(w - ref).max() < 1e-10


@pytest.mark.parametrize("norm", [1.0, 1e3])
def test_orbital_chain(built_lib, norm):
    """One orbital of full cubic symmetry: the Krylov space has 20 real dimensions but for a
    perturbation of 1e-7 of the operator."""
    import torch
    from sincgpu import SincProject
    N = 5
    p = np.arange(N) - 2.0
    r2 = p[:, None, None] ** 2 + p[None, :, None] ** 2 + p[None, None, :] ** 2
    rng = np.random.default_rng(3)
    phi = (np.exp(-0.3 * r2) * (1.0 + 0.2j * r2)).reshape(-1, 1)
    phi /= np.linalg.norm(phi)
    rp = (1.0 / (1.0 + r2) + 0.1 * r2).reshape(-1) + 1e-7 * rng.standard_normal(N ** 3)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    one = np.ones((1, 1), dtype=np.complex128)
    dt = 0.2 / norm
    outs = []
    with SincProject(N, 0.5, [[0, 0, 0]], [1.0], 1, toothnbig=16, toothnsmall=6) as gpu:
        slot = (dev(one), dev(norm * one), dev(rp.astype(np.complex128).reshape(1, 1, -1)))
        for onepass, fused in ((1, 1), (1, 0), (0, 1), (0, 0)):
            gpu.set_option("orth_onepass", onepass)
            gpu.set_option("orth_fused", fused)
            gpu.orbprop_setup(26, 30, 1.2, dt)
            d = dev(phi.T.copy())
            it = gpu.expospfprop_dev(d, slot, slot, 0.0, dt, 0.0, dt, True, expotol=1e-9)
            outs.append((d.cpu().numpy(), it))
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[2][0], outs[3][0])
    assert outs[0][1] == outs[2][1]
    assert np.abs(outs[0][0] - outs[2][0]).max() < 1e-12
