"""The mixed form's fit at the edges of its row quads and workspace sizes, and
on columns without a finite depth, against the FP64 form on the same noise.

Tolerance: the mixed form's own bounds (test_gpu_mixed.py: RMS 2e-3 cells
horizontally, 1 % of the mean water depth vertically, status equal for 99 %
of the particles), which hold for any point count: the fit's sweeps carry
FP32 rounding (6e-8) of values whose factor is formed in FP64.
"""
import numpy as np
import pytest

import harness

pytestmark = pytest.mark.gpu


# int((N + 1) * sub) points: 4 (no quad, no further row), the remainders of the
# quads, both sides of each workspace size and the largest
@pytest.mark.parametrize("N,sub", [(3, 1.0), (4, 1.0), (3, 1.5), (6, 1.0), (7, 1.0), (8, 1.0), (9, 1.0), (10, 1.0),
                                   (21, 4.0), (21, 4.05), (31, 4.0), (31, 4.04), (35, 4.0)])
@pytest.mark.parametrize("variant", ["fused", "smem"])
def test_point_counts(N, sub, variant):
    case = harness.make_case("tiny", 200, seed=5, spec_over={"N": N}, param_over={"sub": sub})
    hook = harness.noise_array(case, 6)
    ref, T0 = harness.run_gpu(case, 6, noise="hook", hook=hook)
    mix, T1 = harness.run_gpu(case, 6, noise="hook", hook=hook, field_dtype="mixed", variant=variant)
    T0.close()
    T1.close()
    ok = np.isin(ref["status"], [1.0, np.float32(1.1), np.float32(1.2)]) & (np.floor(mix["status"]) == 1.0)
    assert ok.sum() > 150 and np.mean(np.floor(mix["status"]) == np.floor(ref["status"])) >= 0.99
    d = np.hypot(mix["x"][ok] - ref["x"][ok], mix["y"][ok] - ref["y"][ok])
    assert np.sqrt(np.mean(d * d)) < 2e-3
    dz = mix["z"][ok] - ref["z"][ok]
    assert np.sqrt(np.mean(dz * dz)) < 0.01 * np.mean(ref["wd"][ok])


# one cell's zeta NaN or infinite: the walk up the column ends, and particles
# elsewhere are those of the plain run
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("variant", ["fused", "smem"])
def test_column_without_depth(bad, variant):
    case = harness.make_case("tiny", 200, seed=6)
    ref, T0 = harness.run_gpu(case, 1, field_dtype="mixed", variant=variant)
    plain = case.frame

    def frame(k, ng=1):
        z = plain(k, ng)["zeta"].copy(order="F")
        z[12, 10] = bad
        return dict(plain(k, ng), zeta=z)
    case.frame = frame
    got, T1 = harness.run_gpu(case, 1, field_dtype="mixed", variant=variant)
    T0.close()
    T1.close()
    far = np.hypot(ref["x"] - 13.0, ref["y"] - 11.0) > 4.0
    assert far.sum() > 100
    for k in ("x", "y", "z", "status", "zeta"):
        assert np.array_equal(got[k][far], ref[k][far]), k
