"""The 113-bit integer integrand's layouts: batches of low orders (a warp per
configuration), order 1 alone, and a mixed batch so large that its small
configurations get a launch of their own, against the same configurations in a
batch of one, bit for bit, on one and two spins, with and without the LU
fallback."""
import dataclasses
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from helpers import GOLDEN, bits_equal, load_case  # noqa: E402

DD = np.load(os.path.join(GOLDEN, "dd_mode.npz"))


@pytest.mark.parametrize("case", ["physical_2x2", "column_3x3"])
@pytest.mark.parametrize("tol_fpm", [None, "1"])
def test_layouts_give_the_same_values(case, tol_fpm):
    params, tables, _ = load_case(case)
    if tol_fpm:
        params = dataclasses.replace(params, tol_fpm=tol_fpm)
    gpu = CdetIntegrand(params, tables)
    gpu.set_integrand_real("double_double", significand_bits=113)
    gpu.set_assembly("split")
    v, o = DD[f"{case}.vertices"], DD[f"{case}.orders"]
    keep = np.concatenate([np.flatnonzero(o == n)[:4] for n in range(1, 11)])
    one = np.array([gpu.integrand_batch(v[c:c + 1, :o[c]], o[c:c + 1])[0][0] for c in keep])
    single_status = np.array([gpu.integrand_batch(v[c:c + 1, :o[c]], o[c:c + 1])[1][0] for c in keep])
    for top in (1, 2, 6, 7, 8, 10):
        which = np.flatnonzero(o[keep] <= top)
        reps = 1 + (7000 if top > 7 and not tol_fpm else 500) // len(which)
        idx = np.tile(which, reps)
        vertices = np.ascontiguousarray(v[keep][idx][:, :top])
        got, status = gpu.integrand_batch(vertices, o[keep][idx])
        assert bits_equal(got, one[idx]), top
        assert np.array_equal(np.asarray(status), single_status[idx]), top
        assert gpu.last_launch_count() >= 6
