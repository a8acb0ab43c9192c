"""The orbital Arnoldi orthogonalisation's launch forms: with orth_fused = 0 (the request
server's setting) no cooperative launch is made, with either source of the coefficients,
and the separate launches give the same bits as the one launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# vectors of less than one element a thread and of several, Krylov dimensions that are no
# multiple of four rows
@pytest.mark.parametrize("onepass", [1, 0])
@pytest.mark.parametrize("N,n", [(9, 3), (21, 4), (31, 8)])
def test_launch_forms_are_bitwise(built_lib, N, n, onepass):
    import torch
    from sincgpu import SincProject, inputs
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
        gpu.set_option("orth_onepass", onepass)
        outs, launches = [], []
        for fused in (1, 0):
            gpu.set_option("orth_fused", fused)
            gpu.orbprop_setup(5, 11, 1.2, 0.002)
            d = dev(phi)
            before = gpu.launch_count()
            it = [gpu.expospfprop_dev(d, slot, slot, t, t + 0.004, t, t + 0.004, True, expotol=1e-9)
                  for t in (0.0, 0.004)]
            launches.append(gpu.launch_count() - before)
            outs.append((d.cpu().numpy(), it, gpu.orbprop_state()))
    assert np.array_equal(outs[0][0], outs[1][0])
    assert outs[0][1] == outs[1][1] and outs[0][2] == outs[1][2]
    assert launches[1] > launches[0]  # the one launch is replaced by several
