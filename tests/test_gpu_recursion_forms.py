"""The all-subsets recursion's block form and the step kernels against the
oracle and the lane form, bit for bit, where their layout changes: one, two and
four configurations per block, a last block that is not full, orders 2 to 11,
the round-off filter off, at its default and at thresholds that put many masks
near it (the decision from exponent fields, and the sum where they do not
decide); chains from one to several per block, and the thread-per-chain step
of large batches."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bindings import Oracle  # noqa: E402
from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.mcmcmc import McmcmcChains  # noqa: E402
from cdet_gb300.synthetic import uniform_configurations  # noqa: E402
from helpers import bits_equal, load_case  # noqa: E402


@pytest.mark.parametrize("case", ["physical_2x2", "column_3x3"])
@pytest.mark.parametrize("z_safety", ["0", "1e4", "1e9", "1e13", "3e15"])
@pytest.mark.parametrize("order,batch", [(2, 3), (5, 130), (7, 1301), (9, 6), (10, 700), (11, 2)])
def test_all_subsets_block_form(case, z_safety, order, batch):
    params, tables, _ = load_case(case)
    params = dataclasses.replace(params, z_safety=z_safety)
    gpu = CdetIntegrand(params, tables)
    v = uniform_configurations(order * 31 + batch, batch, order)
    gpu.set_all_subsets_form("warp")
    got, _ = gpu.all_subsets_batch(v)
    gpu.set_all_subsets_form("lane")
    want, _ = gpu.all_subsets_batch(v)
    assert bits_equal(got, want)
    some = np.arange(batch)[:: max(1, batch // 5)]
    ref, _ = Oracle(params.runtime_scalars(), tables).all_subsets_batch(v[some], threads=8)
    assert bits_equal(got[some], ref)


@pytest.mark.parametrize("z_safety", ["0", "1e4", "1e9", "1e13"])
def test_queue_form_filter(z_safety):
    params, tables, _ = load_case("column_3x3")
    params = dataclasses.replace(params, z_safety=z_safety)
    gpu = CdetIntegrand(params, tables)
    orders = (np.arange(200) % 9 + 2).astype(np.int32)
    v = uniform_configurations(99, 200, 10)
    gpu.set_integrand_form("queue")
    got, _ = gpu.integrand_batch(v, orders)
    want, _ = Oracle(params.runtime_scalars(), tables).integrand_batch(v, orders, threads=8)
    assert bits_equal(got, want)


@pytest.mark.parametrize("env", [3, 6, 9])
def test_chains_do_not_depend_on_the_batch(env):
    """Chains are independent, so a chain's masks, vertices and generator are
    the same whatever shares its block: alone, one per block, two to eight per
    block, and in the thread-per-chain step (16,384 chains)."""
    params, tables, _ = load_case("column_3x3")
    lambdas = [0.0] + [1.0] * (env - 1) + [0.0]
    counts = [1, 5, 400, 1300, 2500] + ([16384] if env == 3 else [])
    steps = 80  # several generator transitions
    seeds = np.arange(1, max(counts) + 1, dtype=np.uint64) * np.uint64(7919)
    first = None
    for chains in counts:
        gpu = CdetIntegrand(params, tables)
        m = McmcmcChains(gpu, 1, env - 1, env, seeds[:chains], lambdas)
        rec = m.run(steps, record=True)
        v, _, rng = m.state()
        got = (rec["chosen"][:, 0], rec["norms"][:, 0], rec["signal"][:, 0], v[0], rng[0])
        if first is None:
            first = got
        for x, y in zip(got, first):
            assert np.array_equal(np.asarray(x).view(np.uint64), np.asarray(y).view(np.uint64)), chains
        last = (rec["chosen"][:, -1], v[-1], rng[-1])
        alone = McmcmcChains(gpu, 1, env - 1, env, seeds[chains - 1:chains], lambdas)
        rec1 = alone.run(steps, record=True)
        v1, _, rng1 = alone.state()
        for x, y in zip(last, (rec1["chosen"][:, 0], v1[0], rng1[0])):
            assert np.array_equal(np.asarray(x).view(np.uint64), np.asarray(y).view(np.uint64)), chains
        alone.close()
        m.close()
