"""The second launch of the 113-bit integrand: a mixed batch so large that its
small configurations run as a warp each behind the four-warp blocks. It is one
launch more than the same mixture below the line takes, and the values and
statuses are those of batches of one, with every matrix on the Schur recursion
and with every matrix on the LU fallback (whose scratch a warp indexes by the
batch's largest order, while the arena holds orders up to 7). A batch as large
with few small configurations finds nothing left for that launch."""
import dataclasses
import os

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from cdet_gb300 import lib as L  # noqa: E402
from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from helpers import GOLDEN, bits_equal, load_case  # noqa: E402

DD = np.load(os.path.join(GOLDEN, "dd_mode.npz"))
ABOVE = 8 * 152 * 12 + 77  # more than eight configurations for every block that could be resident


@pytest.mark.parametrize("case", ["physical_2x2", "column_3x3"])
@pytest.mark.parametrize("tol_fpm", [None, "10"])
def test_second_launch(case, tol_fpm):
    params, tables, _ = load_case(case)
    if tol_fpm:
        params = dataclasses.replace(params, tol_fpm=tol_fpm)
    gpu = CdetIntegrand(params, tables)
    gpu.set_integrand_real("double_double", significand_bits=113)
    gpu.set_assembly("split")
    v, o = DD[f"{case}.vertices"], DD[f"{case}.orders"]
    small = np.concatenate([np.flatnonzero(o == n)[:5] for n in range(1, 8)])
    large = np.concatenate([np.flatnonzero(o == n)[:4] for n in range(8, 11)])
    idx = np.concatenate([large, np.resize(small, ABOVE - len(large))])
    idx = idx[np.random.default_rng(3).permutation(len(idx))]
    assert o[idx].max() == 10
    want, want_status = {}, {}
    for c in np.unique(idx):
        value, status = gpu.integrand_batch(v[c:c + 1, :o[c]], o[c:c + 1])
        want[c], want_status[c] = value[0], np.asarray(status)[0]
    if tol_fpm:
        assert all(want_status[c] & L.CONFIG_FPM_FALLBACK for c in want if o[c] >= 2)
    few = np.concatenate([large, np.resize(small, 600)])
    eights = np.flatnonzero(o == 8)[:4]
    mostly_large = np.concatenate([large, np.resize(eights, 6400), np.resize(small, 60)])
    launches = {}
    for name, part in (("few", few), ("many", idx), ("mostly large", mostly_large)):
        got, status = gpu.integrand_batch(np.ascontiguousarray(v[part]), o[part])
        launches[name] = gpu.last_launch_count()
        assert bits_equal(got, np.array([want[c] for c in part])), name
        assert np.array_equal(np.asarray(status), np.array([want_status[c] for c in part])), name
    assert launches["many"] == launches["mostly large"] == launches["few"] + 1, launches
