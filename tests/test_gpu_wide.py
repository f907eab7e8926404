"""The 113-bit integer integrand behind the split assembly against the
reference's double-double values (dd_mode.npz): orders 1..10 on both golden
cases (two spins and one), with the filter on and off and the LU fallback
forced, in batches of one, of a few blocks and of several rounds of the queue.
The Green matrices are the split assembly's (entries within 1e-15), whose effect
on these cases is below 1e-12 relative; the same values in every batch."""
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
VARIANTS = {"default": {}, "nofilter": {"z_safety": "0"}, "fallback": {"tol_fpm": "1"}}


@pytest.mark.parametrize("case", ["physical_2x2", "column_3x3"])
@pytest.mark.parametrize("variant", sorted(VARIANTS))
def test_wide_integrand(case, variant):
    params, tables, _ = load_case(case)
    gpu = CdetIntegrand(dataclasses.replace(params, **VARIANTS[variant]), tables)
    gpu.set_integrand_real("double_double", significand_bits=113)
    gpu.set_assembly("split")
    v, o = DD[f"{case}.vertices"], DD[f"{case}.orders"]
    want = DD[f"{case}.{variant}.values"]
    got, st = gpu.integrand_batch(v, o)
    assert (st & ~L.CONFIG_FPM_FALLBACK).max() == 0
    if variant == "fallback":
        assert np.all(st[o >= 2] & L.CONFIG_FPM_FALLBACK)
    rel = np.abs(got - want) / np.maximum(np.abs(want), 1e-300)
    assert rel[o >= 2].max() <= 1e-12, (rel[o >= 2].max(), o[o >= 2][np.argmax(rel[o >= 2])])
    assert np.abs(got - want)[o == 1].max() <= 1e-13
    for c in np.flatnonzero(o >= 2)[::17]:  # a batch of one, of its own order
        one, _ = gpu.integrand_batch(v[c:c + 1, :o[c]], o[c:c + 1])
        assert bits_equal(one, got[c:c + 1]), (c, o[c])
    reps = 2 if variant == "fallback" else 13
    many, _ = gpu.integrand_batch(np.tile(v, (reps, 1, 1)), np.tile(o, reps))
    assert bits_equal(many, np.tile(got, reps))

