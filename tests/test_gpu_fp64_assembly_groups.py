"""The FP64 Green assembly's blocks of several configurations (low orders in large
batches) against the same configurations in small batches, where a block has one
configuration or a part of it, bit for bit, and some of them against the oracle:
full and partial last blocks, more configurations per block than a warp could
scan, mixed orders with rejected ones among them, rejected vertices, corner
entries, one and two spins, few and many rows, and Green-pair reuse."""
import numpy as np
import pytest

from bindings import Oracle
from cdet_gb300 import lib as L
from cdet_gb300.integrand import CdetIntegrand
from cdet_gb300.mcmcmc import McmcmcChains
from cdet_gb300.params import CdetParams, named_mask
from cdet_gb300.synthetic import uniform_configurations
from test_gpu_fp64_assembly import _tables

pytestmark = pytest.mark.gpu


def _params(nu, nv, shared=True):
    return CdetParams(n1=2, n2=2, beta="2", mu="0", u="2", alpha_up="0" if shared else "0.55",
                      alpha_down="0" if shared else "0.4", mask_sites=named_mask("first_column", 2, 2), cheb_nu=nu,
                      cheb_nv=nv)


@pytest.mark.parametrize("order,nu,nv,batch,shared", [
    (1, 12, 12, 90001, True), (1, 1, 1, 200000, True), (1, 4, 3, 45007, False), (2, 2, 9, 45000, True),
    (2, 5, 8, 30011, False), (3, 7, 7, 30000, True), (1, 33, 16, 40009, True), (2, 130, 6, 20000, True),
    (4, 3, 4, 12345, True),
])
def test_grouped_blocks_equal_single_ones(order, nu, nv, batch, shared):
    import torch
    rng = np.random.default_rng(order * 100 + nu)
    params = _params(nu, nv, shared)
    tables = _tables(rng, nu, nv, shared, False)
    v = uniform_configurations(nu * 31 + nv, batch, order)
    v[::5, 0, 0] = 0.0     # corner entries
    v[3::97, 0, 1] = np.nan  # rejected vertices
    orders = rng.integers(1, order + 1, batch).astype(np.int32)
    orders[7::41] = 0        # rejected orders
    orders[9::43] = order + 1
    gpu = CdetIntegrand(params, tables)
    dv, do = torch.from_numpy(v).cuda(), torch.from_numpy(orders).cuda()
    got = [x.cpu().numpy() for x in gpu.assemble(dv, do)]
    status = got[2]
    bad = (orders < 1) | (orders > order)
    assert np.all(status[bad] & L.CONFIG_BAD_INPUT)
    nan = np.isnan(v[:, 0, 1])
    assert np.array_equal((status & L.CONFIG_BAD_INPUT) != 0, bad | nan)
    good = np.flatnonzero(~(bad | nan))
    step = 600
    for start in range(0, batch, step):
        if (start // step) % 7 and start + step < batch:  # the first, every seventh and the last
            continue
        part = slice(start, min(batch, start + step))
        want = [x.cpu().numpy() for x in gpu.assemble(dv[part].contiguous(), do[part].contiguous())]
        for c in good[(good >= part.start) & (good < part.stop)]:
            n = orders[c]
            assert np.array_equal(got[0][c, :, :, :n * n].view(np.uint64),
                                  want[0][c - start, :, :, :n * n].view(np.uint64)), c
            assert np.array_equal(got[1][c, :, :, :n].view(np.uint64),
                                  want[1][c - start, :, :, :n].view(np.uint64)), c
        assert np.array_equal(status[part], want[2])
    orc = Oracle(params.runtime_scalars(), tables)
    for c in good[::len(good) // 40]:
        n = int(orders[c])
        for s, (replicas, twisted) in enumerate(((2, True), (1, False))):
            up, down, diag_up, diag_down, _ = orc.green(v[c, :n], replicas, twisted)
            for spin, (g, d) in enumerate(((up, diag_up), (down, diag_down))):
                assert np.array_equal(got[0][c, s, spin, :n * n].view(np.uint64), g.reshape(-1).view(np.uint64)), c
                assert np.array_equal(got[1][c, s, spin, :n].view(np.uint64), d.view(np.uint64)), c


@pytest.mark.parametrize("envelope", [2, 3])
def test_grouped_blocks_with_reuse(envelope):
    import torch
    params = _params(6, 7)
    gpu = CdetIntegrand(params, _tables(np.random.default_rng(5), 6, 7, True, False))
    chains = 12000
    seeds = np.arange(1, chains + 1, dtype=np.uint64) * np.uint64(7919)
    runs = []
    for reuse in (True, False):
        c = McmcmcChains(gpu, 1, envelope - 1, envelope, seeds, [0.0] + [1.0] * envelope)
        c.set_green_reuse(reuse)
        rec = c.run(5, record=True)
        runs.append((np.asarray(rec["chosen"]), np.asarray(rec["norms"]).view(np.uint64),
                     np.asarray(rec["signal"]).view(np.uint64)))
        c.close()
    torch.cuda.synchronize()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
