"""Device memory of the double-double integrand: behind the split assembly it has
no lane form, so a context takes no more than the FP64 integrand behind the same
assembly does; switched to the FP64 assembly later, it takes the lane region then
and gives the values of a context that never left it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.params import CdetParams, named_mask  # noqa: E402
from cdet_gb300.synthetic import uniform_configurations  # noqa: E402
from cdet_gb300.tables import build_tables  # noqa: E402

ORDER, BATCH = 10, 8192
LANES = 3 * (BATCH // 32) * 2 * (1 << ORDER) * 32 * 8  # bytes of the lane region


def test_no_lane_region_behind_the_split_assembly():
    params = CdetParams(n1=3, n2=3, beta="4", mu="0", u="2", mask_sites=named_mask("first_column", 3, 3), cheb_nu=16,
                        cheb_nv=16)
    tables = build_tables(params, device="cuda")
    v = torch.from_numpy(uniform_configurations(8, BATCH, ORDER)).cuda()
    o = torch.full((BATCH,), ORDER, dtype=torch.int32, device="cuda")
    out = torch.empty(BATCH, dtype=torch.float64, device="cuda")
    st = torch.empty(BATCH, dtype=torch.int32, device="cuda")

    def taken(gpu):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        gpu.integrand_device(v, o, out, st)
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0], out.cpu().numpy().copy()

    def context(assembly, real):
        gpu = CdetIntegrand(params, tables)
        gpu.set_assembly(assembly)
        if real != "double":
            gpu.set_integrand_real(real)
        return gpu

    for gpu in (context("split", "double"), context("split", "double_double")):
        gpu.integrand_device(v[:32], o[:32], out[:32], st[:32])  # (the library's own set-up)
    double, _ = taken(context("split", "double"))
    switched = context("split", "double_double")
    wide, _ = taken(switched)
    assert wide <= double + LANES // 8, (wide, double, LANES)
    switched.set_assembly("fp64")
    _, got = taken(switched)
    fp64, want = taken(context("fp64", "double_double"))
    assert fp64 >= LANES
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
