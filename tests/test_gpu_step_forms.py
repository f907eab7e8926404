"""The MCMCMC step's two forms meet at a number of chains that depends on the
envelope and the seed kernel: a run just above it (a thread per chain) and runs
of the same chains below it (a warp per chain) give the same masks, norms,
signals, vertices and generators."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.mcmcmc import McmcmcChains  # noqa: E402
from helpers import load_case  # noqa: E402


@pytest.mark.parametrize("env,chains,hist", [(2, 2048, False), (2, 2100, True), (3, 8192, True), (4, 16384, False),
                                             (11, 3072, True), (11, 12288, False)])
def test_forms_agree_at_their_line(env, chains, hist):
    params, tables, _ = load_case("physical_2x2")
    gpu = CdetIntegrand(params, tables)
    sites = params.n1 * params.n2
    rng = np.random.default_rng(env)

    def rows(n):
        x = rng.uniform(0.5, 1.0, (n, n))
        return x / x.sum(1, keepdims=True)

    probabilities = rows(12), rows(sites), rows(2)
    lambdas = [0.0] + [1.0] * (env - 1) + [0.0]
    seeds = np.arange(1, chains + 1, dtype=np.uint64) * np.uint64(7919)

    def run(part):
        m = McmcmcChains(gpu, 1, env - 1, env, seeds[part], lambdas)
        if hist:
            m.set_histogram(12, *probabilities)
        rec = m.run(3, record=True)
        v, _, mt = m.state()
        out = (np.asarray(rec["chosen"]), np.asarray(rec["norms"]).view(np.uint64),
               np.asarray(rec["signal"]).view(np.uint64), v.view(np.uint64), np.asarray(mt))
        m.close()
        return out

    whole = run(slice(0, chains))
    for part in (slice(0, 700), slice(chains - 300, chains)):
        got = run(part)
        for k, (a, b) in enumerate(zip(got, whole)):
            assert np.array_equal(a, b[:, part] if k < 3 else b[part]), (env, part, k)
