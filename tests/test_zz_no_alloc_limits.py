"""cdet_integrand_device_noalloc where the batch leaves its fixed scratch with the
fewest LU-fallback regions it accepts (8 to 11 warps', fewer than a block of the
shared-memory minors kernel can hold workspaces): every matrix takes the LU
fallback, and the values and statuses equal the ordinary entry point's bit for
bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from cdet_gb300 import lib as L  # noqa: E402
from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.params import CdetParams, named_mask  # noqa: E402
from cdet_gb300.synthetic import uniform_configurations  # noqa: E402
from cdet_gb300.tables import build_tables  # noqa: E402


@pytest.mark.parametrize("order,batch", [(7, 11355), (4, 57810)])
def test_lu_fallback_on_the_smallest_scratch(order, batch):
    params = CdetParams(n1=3, n2=3, beta="4", mu="0", u="2", mask_sites=named_mask("first_column", 3, 3), cheb_nu=8,
                        cheb_nv=8, tol_fpm="10")
    gpu = CdetIntegrand(params, build_tables(params, device="cuda"))
    v = torch.from_numpy(uniform_configurations(31 + order, batch, order)).cuda()
    o = torch.full((batch,), order, dtype=torch.int32, device="cuda")
    values = [torch.full((batch,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    status = [torch.full((batch,), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
    gpu.integrand_device(v, o, values[0], status[0])
    assert gpu.integrand_device_noalloc(v, o, values[1], status[1]) == L.CDET_OK, L.last_error()
    torch.cuda.synchronize()
    want = values[0].cpu().numpy()
    assert np.all(np.isfinite(want))
    assert np.array_equal(values[1].cpu().numpy().view(np.uint64), want.view(np.uint64))
    assert np.array_equal(status[1].cpu().numpy(), status[0].cpu().numpy())
    assert np.all(status[1].cpu().numpy() & L.CONFIG_FPM_FALLBACK)
