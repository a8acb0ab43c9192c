"""The half-length Coulomb form (option coul_half = 1, the FP64 default on the grids of
csrc/coul_half.h) against numpy's FFT convolution and the five passes: the smallest and
largest grid of plans of every kind (coprime, equal odd and even factors), densities,
hermitian pairs and ordered pairs, and a kernel that is not even in each axis.

Tolerance: each of the three forms rounds a transform of L^3 <= 200^3 points twice, an
error of some eps * log2(L^3) = 23 eps of the largest value; 1e-13 is 450 eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-13


def relerr(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / np.abs(np.asarray(b)).max())


def convolve(kernel, dens):
    """Linear convolution of densities (x, y, z, m) with kernel(1-N..N-1 per axis)."""
    N = dens.shape[0]
    L = 2 * N
    k = np.zeros((L, L, L))
    at = np.arange(1 - N, N) % L
    k[np.ix_(at, at, at)] = kernel
    f = np.fft.fftn(dens, s=(L, L, L), axes=(0, 1, 2)) * np.fft.fftn(k)[..., None]
    return np.fft.ifftn(f, axes=(0, 1, 2))[:N, :N, :N]


def project(N, n):
    from sincgpu import SincProject
    return SincProject(N, 0.3, [[0, 0, 0]] if N % 2 else [[1, 1, 1]], [1.0], n, toothnbig=max(N, 16), toothnsmall=8)


@pytest.mark.parametrize("N", [46, 49, 55, 56, 61, 63, 64, 65, 72, 73, 81, 97])
def test_densities(built_lib, N):
    m = 2 if N > 60 else 5
    rng = np.random.default_rng(N)
    dens = rng.standard_normal((N ** 3, m)) + 1j * rng.standard_normal((N ** 3, m))
    with project(N, 2) as gpu:
        ref = convolve(gpu.get_tables()["tempcoulomb"], dens.reshape(N, N, N, m, order="F")).reshape(-1, m, order="F")
        half = gpu.op_tinv(dens)
        gpu.set_option("coul_chunk", 2)
        chunked = gpu.op_tinv(dens)
        gpu.set_option("coul_half", 0)
        five = gpu.op_tinv(dens)
    assert relerr(half, ref) < TOL
    assert relerr(half, five) < TOL
    assert np.array_equal(half, chunked)


@pytest.mark.parametrize("N", [47, 49, 55, 61, 64])
def test_pairs(built_lib, N):
    n = 3
    rng = np.random.default_rng(100 + N)
    bra, ket = (rng.standard_normal((N ** 3, n)) + 1j * rng.standard_normal((N ** 3, n)) for _ in range(2))
    with project(N, n) as gpu:
        for other in (None, ket):
            gpu.set_option("coul_half", 1)
            mat, red = gpu.call_twoe_matel00(bra, other)
            gpu.set_option("coul_half", 0)
            mat5, red5 = gpu.call_twoe_matel00(bra, other)
            assert relerr(red, red5) < TOL
            assert relerr(mat, mat5) < 1e-12  # sums of N^3 products


@pytest.mark.parametrize("N", [46, 55])
def test_uneven_kernel_keeps_the_five_passes(built_lib, N):
    """A caller's kernel that is not even in each axis: the result of the five passes, bit for bit."""
    from sincgpu import SincProject
    rng = np.random.default_rng(7 * N)
    d = np.arange(-N, N, dtype=np.float64)
    even = 1.0 / np.sqrt(1.0 + d[:, None, None] ** 2 + d[None, :, None] ** 2 + d[None, None, :] ** 2)
    skew = even * (1.0 + 1e-3 * d[:, None, None])
    dens = rng.standard_normal((N ** 3, 2)) + 1j * rng.standard_normal((N ** 3, 2))
    for table, same in ((skew, True), (even, False)):
        with SincProject.from_tables(N, 0.3, 2, table, np.zeros(N ** 3)) as gpu:
            out = gpu.op_tinv(dens)
            gpu.set_option("coul_half", 0)
            five = gpu.op_tinv(dens)
        assert np.array_equal(out, five) == same
        assert relerr(out, five) < TOL
