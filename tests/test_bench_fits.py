"""The benchmark's accuracy summaries count the solves that ended in NaN or
infinity and take their errors over the others."""
import json

import numpy as np

import bench


def test_nonfinite_fits_are_counted_wherever_they_stand():
    want = [0.5, 0.25, 0.125, 1.0]
    for at in range(4):
        got = list(want)
        got[(at + 1) % 4] += 0.1
        got[at] = float("nan")
        err, bad, bad64 = bench.finite_errors(got, want)
        assert (len(err), bad, bad64) == (3, 1, 0)
        np.testing.assert_allclose(bench.stat(np.max, err), 0.1)
        json.dumps({"max": bench.stat(np.max, err)}, allow_nan=False)
    err, bad, bad64 = bench.finite_errors([np.inf, 1.0], [1.0, np.nan])
    assert (len(err), bad, bad64) == (0, 1, 1) and bench.stat(np.max, err) is None
