"""The benchmark's work of the two dense contractions against the least work that the measured
cases declare for the same evaluation (n^2 real rows and columns, no diagonal zeros)."""
import sys
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(REPO))

import bench  # noqa: E402


@pytest.mark.parametrize("N,n", [(41, 10), (81, 16)])
def test_contractions_count_the_rows_in_use(N, n):
    G = N ** 3
    fl = bench.contraction_flops(n, G)
    assert fl["rp_gemm"] == 2.0 * G * n ** 4
    assert fl["twoe_gemm"] == G * (n ** 4 + n ** 2)  # upper triangle with the diagonal


def test_evaluation_roofline_uses_them(monkeypatch):
    from sincgpu.inputs import WORKLOADS
    monkeypatch.setattr(bench, "_dgemm_tflops", lambda dev: 37.0)
    w = WORKLOADS["C"]
    prof = {"twoe_gemm": (2.2, 1), "rp_gemm": (2.7, 1)}
    r = bench.eval_roofline(w, prof, 1, None, 162, 12.5)
    fl = bench.contraction_flops(w.nspf, w.G)
    for k in prof:
        assert r["stages"][k]["roof_ms"] == pytest.approx(fl[k] / 37e12 * 1e3)
        one = bench.make_roofline(w, {k: prof[k]}, 1, None, 162)
        assert one["achieved"] == pytest.approx(fl[k] / (prof[k][0] / 1e3) / 1e12)
