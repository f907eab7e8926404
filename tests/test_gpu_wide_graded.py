"""The 113-bit integrand behind the split assembly on graded Green matrices: one
vertex whose row and column are 2^-s of the others. The tables of the site it
sits on are scaled by powers of two, so the Green matrix is D G D exactly, every
subset value with the vertex carries 2^-4s (rows and columns of both spins), and
so does the integrand: the graded value must be the ungraded one times 2^-4s.

Bound: the minors are formed from a matrix with a uniform shift p, to 112 bits of
the shifted minors, which do not shrink with the vertex; its minors are 2^-2s of
them, so their relative error is about 2^(2s - 112) times the rounding steps (6
levels, 6 shift removals) and the cancellation in the connected sum (some tens on
these diagonally dominant matrices): 2^14 in all. Where that is small, what the
double-double result and its difference of two sets leave: 2^-46."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.params import CdetParams, named_mask  # noqa: E402

SIDE, ORDER, BATCH, NU, NV = 3, 6, 48, 8, 10
VARIANTS = {"default": {}, "nofilter": {"z_safety": "0"}, "fallback": {"tol_fpm": "1"},
            "filter": {"z_epsilon0": "0.05", "z_safety": "1"}}


def _tables(rng, shared):
    sites = SIDE * SIDE

    def table():
        t = {}
        for key in ("upper", "lower"):
            c = rng.uniform(-0.5, 0.5, (4, sites, sites, NU, NV)) * 0.1
            c[..., 0, 0] = rng.uniform(-0.5, 0.5, (4, sites, sites))
            for x in range(sites):
                c[:, x, x, 0, 0] = 1.5
            t[key] = c
            t[key + "_corners"] = rng.uniform(-0.5, 0.5, (4, sites, sites))
        return t

    up, ordinary = table(), table()
    return {"twisted_up": up, "twisted_down": up if shared else table(),
            "ordinary_up": ordinary, "ordinary_down": ordinary if shared else table()}


def _graded(tables, site, s):
    d = np.ones(SIDE * SIDE)
    d[site] = 2.0 ** -s
    pair = d[:, None] * d[None, :]
    done, out = {}, {}
    for kind, t in tables.items():
        if id(t) not in done:
            done[id(t)] = {k: np.ascontiguousarray((c * (pair[..., None, None] if c.ndim == 5 else pair)).reshape(-1))
                           for k, c in t.items()}
        out[kind] = done[id(t)]
    return out


@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("variant", sorted(VARIANTS))
def test_graded_vertex(shared, variant):
    rng = np.random.default_rng(606 + shared)
    # (no diagonal shifts: alpha / U would not scale with the tables)
    params = CdetParams(n1=SIDE, n2=SIDE, beta="2", mu="0", u="2", alpha_up="0", alpha_down="0",
                        mask_sites=named_mask("first_column", SIDE, SIDE), cheb_nu=NU, cheb_nv=NV, **VARIANTS[variant])
    tables = _tables(rng, shared)
    small = 4
    v = np.empty((BATCH, ORDER, 4))
    for c in range(BATCH):  # distinct sites, the small one at a place that moves through the vertices
        others = rng.permutation([x for x in range(SIDE * SIDE) if x != small])[:ORDER]
        others[c % ORDER] = small
        v[c, :, 0] = rng.uniform(0.05, 0.95, ORDER)
        v[c, :, 1] = (others // SIDE + 0.5) / SIDE
        v[c, :, 2] = (others % SIDE + 0.5) / SIDE
        v[c, :, 3] = rng.uniform(0, 1, ORDER)
    orders = np.full(BATCH, ORDER, dtype=np.int32)

    def values(s):
        gpu = CdetIntegrand(params, _graded(tables, small, s))
        gpu.set_integrand_real("double_double")
        gpu.set_assembly("split")
        got, status = gpu.integrand_batch(v, orders)
        assert int(np.max(np.asarray(status) & ~2)) == 0
        return got

    flat = values(0)
    assert np.all(np.isfinite(flat))
    # (at the filter's threshold here it cuts many values to zero, not all)
    assert 0 < np.count_nonzero(flat) < BATCH if variant == "filter" else np.all(flat != 0)
    for s in (20, 40, 44):
        want, got = flat * 2.0 ** (-4 * s), values(s)
        assert np.array_equal(want == 0, got == 0), s
        rel = np.abs(got - want)[want != 0] / np.abs(want)[want != 0]
        assert rel.max() <= 2.0 ** -46 + 2.0 ** (2 * s - 98), (s, rel.max())
