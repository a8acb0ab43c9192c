"""The tensor-core orbital products (mix, projection, Jacobian's combination) and dots at
the edges of their tiles, and the one-pass Arnoldi coefficients in both launch forms.

Tolerances: the products sum 2n <= 64 and the dots N^3 <= 216 terms in FP64, some 216 eps =
5e-14 of the largest value at the worst; actreduced chains five of them with a kinetic
contraction whose terms are ten times its result: 1e-11, as the other parity tests."""
import numpy as np
import pytest

from oracle import sinc_oracle as orc

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / np.abs(np.asarray(b)).max())


# one to eight fragments of four orbitals, full and ragged; beyond 16 the dots' other form
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 21, 25, 29, 32])
def test_actreduced(built_lib, n):
    from sincgpu import SincProject
    N = 6
    sysm = orc.SincSystem(N, 0.5, [[1, 1, 1]], [2.0], toothnbig=16, toothnsmall=6)
    phi, proj = orc.seeded_orbitals(sysm, n, seed=n), orc.seeded_orbitals(sysm, n, seed=50 + n)
    den = orc.seeded_hermitian_psd(n, seed=n)
    inv = orc.invmatsmooth(den)
    rng = np.random.default_rng(n)
    rp = np.asfortranarray(rng.standard_normal((N ** 3, n, n)) + 1j * rng.standard_normal((N ** 3, n, n)))
    ref = orc.actreduced00(sysm, phi, proj, den, inv, rp, ztdpot=0.3)
    with SincProject(N, 0.5, [[1, 1, 1]], [2.0], n, toothnbig=16, toothnsmall=6) as gpu:
        assert relerr(gpu.actreduced00(phi, proj, den, inv, rp, ztdpot=0.3), ref) < 1e-11


# 41^3 x 16: vectors longer than the registers of the one-launch form; 17: the Jacobian's
# two dots as separate passes; 4: one launch
@pytest.mark.parametrize("N,n", [(15, 4), (11, 17), (41, 16)])
def test_one_pass_orthogonalisation(built_lib, N, n):
    import torch
    from sincgpu import SincProject
    from sincgpu import inputs
    phi = inputs.seeded_orbitals(N, 0.4, n, seed=N)
    den = inputs.seeded_hermitian_psd(n, 3)
    inv = inputs.regularized_inverse(den)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()  # noqa: E731
    with SincProject(N, 0.4, [[0, 0, 0]], [1.0], n, toothnbig=max(N, 20), toothnsmall=8) as gpu:
        rp = torch.zeros(n, n, N ** 3, dtype=torch.complex128, device="cuda")
        mat = torch.zeros(n ** 4, dtype=torch.complex128, device="cuda")
        tally = torch.from_numpy(np.ascontiguousarray(inputs.seeded_tally(n, 4).T)).cuda() / n
        gpu.mean_field_dev(dev(phi), tally, mat, rp)
        gpu.synchronize()
        slot = (dev(den), dev(inv), rp)
        outs = []
        for onepass in (1, 0):
            gpu.set_option("orth_onepass", onepass)
            gpu.orbprop_setup(6, 12, 1.2, 0.002)
            d = dev(phi)
            it = gpu.expospfprop_dev(d, slot, slot, 0.0, 0.004, 0.0, 0.004, True, expotol=1e-9)
            outs.append((d.cpu().numpy(), it, gpu.orbprop_state()))
        assert outs[0][1] == outs[1][1]
        assert outs[0][2]["thisexpodim"] == outs[1][2]["thisexpodim"]
        assert relerr(outs[0][0], outs[1][0]) < 1e-12
