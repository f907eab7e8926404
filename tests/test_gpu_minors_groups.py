"""The staged form's minors on two and four warps per workspace, against the
oracle bit for bit where the grouping changes: batches that leave an SM at most
seven workspaces and more, orders 2 to 10 and, with the chunked recursion, up
to 13, with and without the LU fallback; and the split assembly's key scan
where a block takes more than one round of keys."""
import dataclasses

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bindings import Oracle  # noqa: E402
from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.params import CdetParams, named_mask  # noqa: E402
from cdet_gb300.synthetic import uniform_configurations  # noqa: E402
from cdet_gb300.tables import build_tables  # noqa: E402
from helpers import bits_equal, load_case  # noqa: E402


@pytest.mark.parametrize("case", ["physical_2x2", "column_3x3"])
@pytest.mark.parametrize("tol_fpm", [None, "1"])
@pytest.mark.parametrize("nmax,batch", [(2, 1), (5, 40), (9, 533), (10, 532), (10, 900), (11, 3), (13, 5)])
def test_minors_of_a_group_of_warps(case, tol_fpm, nmax, batch):
    params, tables, _ = load_case(case)
    if tol_fpm:
        params = dataclasses.replace(params, tol_fpm=tol_fpm)
    gpu = CdetIntegrand(params, tables)
    gpu.set_integrand_form("staged")
    orders = (nmax - np.arange(batch) % min(nmax, 4)).astype(np.int32)
    v = uniform_configurations(nmax * 77 + batch, batch, nmax)
    got, status = gpu.integrand_batch(v, orders)
    some = np.unique(np.concatenate([np.arange(batch)[:: max(1, batch // 12)], [batch - 1]]))
    want, want_status = Oracle(params.runtime_scalars(), tables).integrand_batch(v[some], orders[some], threads=8)
    assert bits_equal(got[some], want)
    assert np.array_equal(np.asarray(status)[some], np.asarray(want_status))


def test_key_scan_of_several_rounds_per_block():
    """12x12 sites: 207,360 sub-blocks, more than 1,024 per SM."""
    params = CdetParams(n1=12, n2=12, beta="4", mu="0", u="2", mask_sites=named_mask("origin_square", 12, 12, 1),
                        cheb_nu=8, cheb_nv=8)
    tables = build_tables(params, device="cuda")
    gpu = CdetIntegrand(params, tables)
    v = torch.from_numpy(uniform_configurations(12, 300, 6)).cuda()
    orders = torch.full((300,), 6, dtype=torch.int32, device="cuda")
    g64, _, s64 = gpu.assemble(v, orders)
    gpu.set_assembly("split")
    gsp, _, ssp = gpu.assemble(v, orders)
    assert int(s64.max()) == 0 and int(ssp.max()) == 0
    # both assemblies are FP64-level evaluations of the same series: 2e-15 of the set's largest entry
    scale = g64.abs().amax(dim=-1, keepdim=True)
    assert bool(((g64 - gsp).abs() <= 2e-15 * scale).all())
