"""The FP64 Green assembly against the oracle, bit for bit, at rows around one
staged chunk of eight columns: seven (a partial chunk alone), eight (one full
chunk that both begins and ends the recurrence) and nine (a partial chunk of one
column before a full one), odd and even row counts up to several row blocks, with
ordinary coefficients and with those that leave the integer-pipe path."""
import numpy as np
import pytest

from bindings import Oracle
from cdet_gb300.integrand import CdetIntegrand
from cdet_gb300.params import CdetParams, named_mask
from cdet_gb300.synthetic import uniform_configurations
from test_gpu_fp64_assembly import _tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("nv", [7, 8, 9, 10, 16, 17])
@pytest.mark.parametrize("nu,order,batch,shared", [(5, 4, 30, True), (129, 2, 9, False), (8, 1, 40, True)])
def test_rows_around_one_chunk(nu, nv, order, batch, shared, special):
    import torch
    rng = np.random.default_rng(nu * 1000 + nv)
    params = CdetParams(n1=2, n2=2, beta="2", mu="0", u="2", alpha_up="0" if shared else "0.55",
                        alpha_down="0" if shared else "0.4", mask_sites=named_mask("first_column", 2, 2), cheb_nu=nu,
                        cheb_nv=nv)
    tables = _tables(rng, nu, nv, shared, special)
    v = uniform_configurations(nu * 17 + nv, batch, order)
    if special:
        v[::3, :, 0] = np.round(v[::3, :, 0] * 8) / 8
    orders = np.full(batch, order, dtype=np.int32)
    gpu = CdetIntegrand(params, tables)
    green, diag, status = gpu.assemble(torch.from_numpy(v).cuda(), torch.from_numpy(orders).cuda())
    green, diag = green.cpu().numpy(), diag.cpu().numpy()
    assert int(status.max()) == 0
    orc = Oracle(params.runtime_scalars(), tables)
    for c in range(batch):
        for s, (replicas, twisted) in enumerate(((2, True), (1, False))):
            up, down, diag_up, diag_down, _ = orc.green(v[c], replicas, twisted)
            for spin, (want, want_diag) in enumerate(((up, diag_up), (down, diag_down))):
                for got, ref in ((green[c, s, spin, :order * order], want.reshape(-1)),
                                 (diag[c, s, spin, :order], want_diag)):
                    same = got.view(np.uint64) == ref.view(np.uint64)
                    assert np.all(same | (np.isnan(got) & np.isnan(ref))), (c, s, spin)
