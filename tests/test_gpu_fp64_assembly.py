"""The FP64 Green assembly on the GPU against the oracle, bit for bit, at the
edges of its tiling: rows shorter, equal and longer than a staged chunk of 16
columns, more rows than one row block of 128, odd rows (8-byte copies) and even
ones (16-byte copies), blocks with fewer lookups than 16, both spin layouts, and
coefficients and vertices whose products leave the integer-pipe path (zeros,
ties, extreme exponents, infinities)."""
import numpy as np
import pytest

from bindings import Oracle
from cdet_gb300.integrand import CdetIntegrand
from cdet_gb300.params import CdetParams, named_mask
from cdet_gb300.synthetic import uniform_configurations

pytestmark = pytest.mark.gpu


def _tables(rng, nu, nv, shared, special):
    count = 4 * 4 * 4

    def table():
        t = {}
        for key in ("upper", "lower"):
            c = rng.standard_normal((count, nu, nv)) * 2.0 ** rng.integers(-40, 3, (count, nu, nv))
            if special:
                c[::5] = 0.0                                          # zero blocks: every product exceptional
                c[1::7] = np.round(c[1::7] * 4) / 4                   # short significands: ties
                c[2::9, :, nv // 2] *= 1e-250                         # tiny and huge exponents
                c[3::11, nu // 2, :] *= 1e200
                c[4::13, 0, 0] = np.inf
            t[key] = np.ascontiguousarray(c.reshape(-1))
            t[key + "_corners"] = rng.standard_normal(count)
        return t

    up, ordinary = table(), table()
    return {"twisted_up": up, "twisted_down": up if shared else table(),
            "ordinary_up": ordinary, "ordinary_down": ordinary if shared else table()}


@pytest.mark.parametrize("nu,nv,order,batch,shared,special", [
    (1, 1, 2, 3, True, False), (2, 2, 3, 5, False, False), (5, 3, 1, 70, True, False), (3, 15, 4, 9, True, False),
    (7, 16, 3, 33, True, False), (33, 17, 5, 4, False, False), (18, 31, 9, 2, True, False), (127, 32, 4, 3, True, False),
    (128, 33, 2, 11, False, False), (129, 48, 3, 7, True, False), (300, 49, 2, 2, True, False),
    (16, 32, 6, 40, True, True), (20, 45, 5, 40, False, True), (131, 64, 6, 400, True, True),
])
def test_green_matrices_bitwise(nu, nv, order, batch, shared, special):
    import torch
    rng = np.random.default_rng(nu * 1000 + nv)
    params = CdetParams(n1=2, n2=2, beta="2", mu="0", u="2", alpha_up="0" if shared else "0.55",
                        alpha_down="0" if shared else "0.4", mask_sites=named_mask("first_column", 2, 2),
                        cheb_nu=nu, cheb_nv=nv)
    tables = _tables(rng, nu, nv, shared, special)
    v = uniform_configurations(nu * 17 + nv, batch, order)
    if special:
        v[::3, :, 0] = np.round(v[::3, :, 0] * 8) / 8  # u and v with short significands, 0 and +-1 among them
    v[::4, 0, 0] = 0.0                                # corner entries
    orders = rng.integers(1, order + 1, batch).astype(np.int32)
    orders[0] = order
    gpu = CdetIntegrand(params, tables)
    green, diag, status = gpu.assemble(torch.from_numpy(v).cuda(), torch.from_numpy(orders).cuda())
    green, diag = green.cpu().numpy(), diag.cpu().numpy()
    assert int(status.max()) == 0
    orc = Oracle(params.runtime_scalars(), tables)
    for c in range(batch):
        n = int(orders[c])
        for s, (replicas, twisted) in enumerate(((2, True), (1, False))):
            up, down, diag_up, diag_down, _ = orc.green(v[c, :n], replicas, twisted)
            for spin, (want, want_diag) in enumerate(((up, diag_up), (down, diag_down))):
                for got, ref in ((green[c, s, spin, :n * n], want.reshape(-1)), (diag[c, s, spin, :n], want_diag)):
                    same = got.view(np.uint64) == ref.view(np.uint64)
                    assert np.all(same | (np.isnan(got) & np.isnan(ref))), (c, s, spin)
