"""Evaluations whose kernels start before the one in front has ended, at the sizes where the
form changes (41 points a side live; in a captured graph 25 for fewer than 8 orbitals): live
calls and graph replays against one stream with the overlap off, bit for bit, with the
buffers overwritten in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n", [(25, 4), (26, 5), (27, 8), (33, 6), (41, 3), (42, 4)])
def test_live_and_captured_evaluations(built_lib, N, n):
    import torch
    from sincgpu import SincProject, WalkTables, inputs
    phi = torch.from_numpy(np.ascontiguousarray(inputs.seeded_orbitals(N, 0.4, n, seed=N).T)).cuda()
    z = lambda *s: torch.zeros(*s, dtype=torch.complex128, device="cuda")  # noqa: E731
    with SincProject(N, 0.4, [[0, 0, 0]] if N % 2 else [[1, 1, 1]], [2.0], n, toothnbig=max(N, 20),
                     toothnsmall=8) as gpu:
        gpu.set_stream(torch.cuda.current_stream().cuda_stream)
        walks = WalkTables(2, n, 0)
        gpu.ci_attach(walks)
        rng = np.random.default_rng(n)
        a = rng.standard_normal(walks.numconfig) + 1j * rng.standard_normal(walks.numconfig)
        a = torch.from_numpy(a / np.linalg.norm(a)).cuda()
        bufs = [z(n, n), z(n, n), z(n, n, n, n), z(n, n, n, n), z(n, n, N ** 3), z(n, N ** 3)]

        def result(call):
            for b in bufs:
                b.fill_(float("nan"))
            call()
            gpu.synchronize()
            return [b.cpu().numpy() for b in bufs]

        live = lambda: gpu.orbital_rhs_avec_dev(phi, a, *bufs)  # noqa: E731
        gpu.set_option("rhs_overlap", 0)
        ref = result(live)
        assert all(np.isfinite(r).all() for r in ref)
        gpu.set_option("rhs_overlap", 1)
        outs = [result(live) for _ in range(3)]
        gpu.rhs_graph_capture(phi, a, *bufs)
        outs += [result(gpu.rhs_graph_launch) for _ in range(3)]
        outs.append(result(lambda: [live() for _ in range(4)]))
    for out in outs:
        assert all(np.array_equal(o, r) for o, r in zip(out, ref))
