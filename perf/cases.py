"""The workloads this framework is measured on.

Each case is one call (or one run of Markov-chain steps) through the public
Python interface: `CdetIntegrand` (single configurations, host and device
batches, all-subset envelopes, Green matrices) and `McmcmcChains`. A context
(tables in device memory, split slices, scratch) is the handle a program keeps
for a parameter set, so contexts live in a small cache here and each
preparation draws new vertices, orders or chain seeds.
"""
import collections
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "cdet-renyi-entanglement-hpc_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from cdet_gb300.integrand import CdetIntegrand  # noqa: E402
from cdet_gb300.mcmcmc import McmcmcChains  # noqa: E402
from cdet_gb300.params import CdetParams, half_lattice_mask, named_mask  # noqa: E402
from cdet_gb300.synthetic import truncated_geometric_orders  # noqa: E402
from cdet_gb300.tables import build_tables  # noqa: E402

# Parameter sets of the benchmark and the tests, by lattice side: beta, mu, U,
# subsystem mask.
_PHYSICS = {
    2: ("2", "0", "2", "column"),
    3: ("4", "0", "2", "column"),
    4: ("6", "0", "2", "square"),
    6: ("5", "0", "4", "half"),
    8: ("8", "0", "4", "square2"),
}


def _case(name, entry, side, nu, nv, order, batch, assembly="fp64", real="double", mixed=False, two_spins=False,
          steps=0):
    return {"name": name, "entry": entry, "side": side, "nu": nu, "nv": nv, "order": order, "batch": batch,
            "assembly": assembly, "real": real, "mixed": mixed, "two_spins": two_spins, "steps": steps}


def listed():
    return [
        # the reference's own entry: one configuration per call, as a driver
        # that swaps the integrand in calls it once per proposal
        _case("single_6x6_n6", "single", 6, 96, 96, 6, 1),
        # a small device batch of the default form on an odd, ragged table,
        # distinct spin-up and spin-down tables (ALPHA_UP != ALPHA_DOWN)
        _case("fp64_two_spins_4x4_n7", "device", 4, 45, 37, 7, 391, two_spins=True),
        # 64 chains x 64 proposals, orders 1..10 truncated-geometric, default form
        _case("fp64_mixed_6x6", "device", 6, 96, 96, 10, 4096, mixed=True),
        # the headline lattice in the default (bit-identical) form
        _case("fp64_8x8_n10", "device", 8, 128, 128, 10, 4096),
        # Green matrices alone, default form (a caller with its own recursion)
        _case("green_fp64_6x6_n8", "assemble", 6, 96, 96, 8, 1531),
        # the headline: 65,536 proposals of order 10 on the tensor-core assembly
        _case("split_8x8_n10", "device", 8, 128, 128, 10, 65536, assembly="split"),
        # a driver's mixed batch from host memory to host memory
        _case("split_mixed_host_6x6", "host", 6, 96, 96, 10, 16384, assembly="split", mixed=True),
        # a latency-bound split batch
        _case("split_small_6x6_n8", "device", 6, 96, 96, 8, 250, assembly="split"),
        # high order on a table of several sub-blocks
        _case("split_3x3_n14", "device", 3, 192, 192, 14, 512, assembly="split"),
        # the reference's double-double integrand mode behind the split assembly
        _case("dd_split_6x6_n10", "device", 6, 96, 96, 10, 8192, assembly="split", real="double_double"),
        # Markov chains resident on the GPU: the chains of one node, default form
        _case("chains_fp64_6x6_e9", "chains", 6, 96, 96, 9, 128, steps=16),
        # the same on the split assembly with many chains
        _case("chains_split_6x6_e9", "chains", 6, 96, 96, 9, 2048, assembly="split", steps=16),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: lattices 2x2..8x8, degrees 12..128 (192 on the small ones;
    equal or not), orders 1..14, batches from 1 up to what costs as much as the largest listed cases."""
    entry = rng.choice(["single", "host", "device", "device", "device", "device", "subsets", "assemble", "chains"])
    side = rng.choice(sorted(_PHYSICS))
    top = 192 if side <= 3 else 128
    nu = _log_int(rng, 12, top)
    nv = nu if rng.random() < 0.5 else _log_int(rng, 12, top)
    assembly = rng.choice(["fp64", "split"])
    two_spins = rng.random() < 0.25
    real = "double"
    if entry in ("device", "host") and rng.random() < 0.15:
        real = "double_double"
    if entry == "subsets":
        order = rng.randint(2, 10)
    elif entry == "chains":
        order = rng.randint(4, 9)
    elif real == "double_double":
        order = rng.randint(1, 10)
    else:
        order = rng.randint(1, 14)
    # the most configurations that stay below the largest listed cases: FP64
    # Chebyshev terms, split lookups, subset pairs and output values
    spins = 2 if two_spins else 1
    terms = 2 * spins * order * order * nu * nv
    cap = 65536
    cap = min(cap, (1.2e10 if assembly == "fp64" else 1.0e12) / terms)
    cap = min(cap, (8.0e8 if entry in ("subsets", "chains") else 2.0e9) / 3 ** order)
    if real == "double_double":
        cap = min(cap, 2.0e8 / 3 ** order)
    if order > 10:
        cap = min(cap, 1024)
    steps = 0
    if entry == "single":
        batch, order = 1, min(order, 10)
    elif entry == "chains":
        steps = rng.randint(3, 16)
        batch = _log_int(rng, 1, max(1, min(2048, int(cap / steps))))
    else:
        batch = _log_int(rng, 1, max(1, int(cap)))
    mixed = entry in ("device", "host") and order > 1 and rng.random() < 0.4
    c = _case("", entry, side, nu, nv, order, batch, assembly, real, mixed, two_spins, steps)
    del c["name"]
    return c


def _params(case):
    side = case["side"]
    beta, mu, u, mask = _PHYSICS[side]
    sites = {"column": lambda: named_mask("first_column", side, side),
             "square": lambda: named_mask("origin_square", side, side, 1),
             "square2": lambda: named_mask("origin_square", side, side, 2),
             "half": lambda: half_lattice_mask(side, side)}[mask]()
    alpha = ("0.55", "0.4") if case["two_spins"] else ("0", "0")
    return CdetParams(n1=side, n2=side, beta=beta, mu=mu, u=u, alpha_up=alpha[0], alpha_down=alpha[1],
                      mask_sites=sites, cheb_nu=case["nu"], cheb_nv=case["nv"])


_tables = collections.OrderedDict()
_contexts = collections.OrderedDict()


def _table_set(case):
    key = (case["side"], case["nu"], case["nv"], case["two_spins"])
    if key not in _tables:
        while len(_tables) >= 4:
            old, _ = _tables.popitem(last=False)
            for k in [k for k in _contexts if k[0] == old]:
                del _contexts[k]
        _tables[key] = build_tables(_params(case), device="cuda")
    _tables.move_to_end(key)
    return key, _tables[key]


def _context(case):
    tkey, tables = _table_set(case)
    key = (tkey, case["assembly"], case["real"])
    if key not in _contexts:
        ctx = CdetIntegrand(_params(case), tables, device=0)
        if case["assembly"] != "fp64":
            ctx.set_assembly(case["assembly"])
            ctx.prepare_split()
        if case["real"] != "double":
            ctx.set_integrand_real(case["real"])
        _contexts[key] = ctx
    return _contexts[key]


def _inputs(case, seed):
    """Uniform unit-cube vertices [batch][order][4] and orders [batch] on the device."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    batch, order = case["batch"], case["order"]
    v = torch.rand((batch, order, 4), dtype=torch.float64, device="cuda", generator=g)
    if case["mixed"]:
        o = torch.from_numpy(truncated_geometric_orders(seed * 7919 + 17, batch, 0.3, order)).cuda()
    else:
        o = torch.full((batch,), order, dtype=torch.int32, device="cuda")
    return v, o


def prepare(case, seed):
    ctx = _context(case)
    state = {"case": case, "ctx": ctx}
    entry, batch, order = case["entry"], case["batch"], case["order"]
    if entry == "chains":
        seeds = np.random.RandomState(seed % (1 << 32)).randint(1, 1 << 62, size=batch, dtype=np.int64)
        lambdas = [0.0] + [1.0] * (order - 1) + [0.0]
        state["chains"] = McmcmcChains(ctx, 1, order - 1, order, seeds.astype(np.uint64), lambdas)
        return state
    v, o = _inputs(case, seed)
    if entry in ("single", "host"):
        state["v"] = v.cpu().numpy()
        state["o"] = o.cpu().numpy()
        return state
    state["v"], state["o"] = v, o
    if entry in ("device", "subsets"):
        shape = (batch, 1 << order) if entry == "subsets" else (batch,)
        state["values"] = torch.empty(shape, dtype=torch.float64, device="cuda")
        state["status"] = torch.empty(batch, dtype=torch.int32, device="cuda")
    return state


def run(state):
    ctx, entry = state["ctx"], state["case"]["entry"]
    if entry == "single":
        return ctx.evaluate_cdet_density_integrand_double(state["v"][0])
    if entry == "host":
        values, status = ctx.integrand_batch(state["v"], state["o"])
        return {"values": values, "status": status}
    if entry == "device":
        ctx.integrand_device(state["v"], state["o"], state["values"], state["status"])
        return {"values": state["values"], "status": state["status"]}
    if entry == "subsets":
        ctx.all_subsets_device(state["v"], state["values"], state["status"])
        return {"values": state["values"], "status": state["status"]}
    if entry == "assemble":
        green, diag, status = ctx.assemble(state["v"], state["o"])
        return {"green": green, "diag": diag, "status": status}
    rec = state["chains"].run(state["case"]["steps"], record=True)
    return {"chosen": rec["chosen"].astype(np.int64), "norms": rec["norms"], "signal": rec["signal"]}


def work(case):
    """Each reached coefficient block and each input read once, each output
    written once; two flops per coefficient of a lookup, the minors' Schur
    updates and one multiply-add per subset pair of the recursion."""
    n, batch, sites = case["order"], case["batch"], case["side"] ** 2
    spins = 2 if case["two_spins"] else 1
    evals = batch * max(1, case["steps"])
    if case["mixed"]:  # mean over the truncated geometric distribution
        w = [0.3 * 0.7 ** k for k in range(n)]
        mix = [(k + 1, x / sum(w)) for k, x in enumerate(w)]
    else:
        mix = [(n, 1.0)]
    mean = lambda f: sum(x * f(k) for k, x in mix)  # noqa: E731
    block = case["nu"] * case["nv"]
    pairs = mean(lambda k: k * k)
    blocks = 2 * 5 * sites * sites * spins  # both branches: 4 S^2 twisted, S^2 ordinary
    lookups = 2 * spins * evals * pairs
    out = {"subsets": 8 << n, "assemble": 8 * 4 * (n * n + n), "chains": 8 * (n + 3)}.get(case["entry"], 12)
    flops = lookups * 2 * block
    if case["entry"] != "assemble":
        full = case["entry"] in ("subsets", "chains")
        schur = lambda k: sum(2 ** l * (k - l - 1) ** 2 for l in range(k - 1)) + k * 2 ** (k - 1)  # noqa: E731
        pair = lambda k: 3 ** k / 2 if full else 3 ** (k - 1)  # noqa: E731
        flops += 2 * 2 * evals * mean(lambda k: spins * schur(k) + pair(k))
    return {"bytes": min(lookups, blocks) * block * 8 + evals * (32 * n + 4 + out), "flops": flops}


# ------------------------------------------------------------------ exact ---
def _cheb(x, degree):
    """T_0..T_{degree-1} at x, [len(x)][degree]."""
    return torch.cos(torch.acos(x)[:, None] * torch.arange(degree, dtype=torch.float64, device=x.device)[None])


def _exact_green(case, p, tables, v):
    """Unscaled Green values [2 sets][2 spins][batch][n][n] (shifts not added)
    of configurations v [batch][n][4], by T_a(u)^T C T_b(v)."""
    b, n = v.shape[0], v.shape[1]
    side, s = case["side"], case["side"] ** 2
    beta = float(p.beta)
    tau = beta * v[..., 0]
    site = ((side * v[..., 1]).floor().clamp(0, side - 1) * side + (side * v[..., 2]).floor().clamp(0, side - 1)).long()
    ti, tj = tau[:, :, None].expand(b, n, n), tau[:, None, :].expand(b, n, n)
    off = ~torch.eye(n, dtype=torch.bool, device=v.device)[None]
    upper = (v[:, :, None, 0] > v[:, None, :, 0]) & off
    outer, inner = torch.where(upper, ti, tj), torch.where(upper, tj, ti)
    u = (2.0 * outer / beta - 1.0).clamp(-1, 1).reshape(-1)
    w = torch.where(outer > 0, 2.0 * inner / outer.clamp(min=1e-300) - 1.0, torch.ones_like(outer)).clamp(-1, 1).reshape(-1)
    corner = (outer < float(p.branch_epsilon)).reshape(-1)
    up = upper.reshape(-1)
    out = torch.empty((2, 2, b * n * n), dtype=torch.float64, device=v.device)
    nu, nv = case["nu"], case["nv"]
    for k, kind in enumerate(("twisted", "ordinary")):
        rep = (2.0 * v[..., 3]).floor().clamp(0, 1).long() if k == 0 else torch.zeros_like(site)
        pair = (((rep[:, :, None] * 2 + rep[:, None, :]) * s + site[:, :, None]) * s + site[:, None, :]).reshape(-1)
        for spin, name in enumerate(("up", "down")):
            if spin == 1 and not case["two_spins"]:
                out[k, 1] = out[k, 0]
                continue
            t = tables[kind + "_" + name]
            step = max(1, (1 << 28) // (nu * nv))
            for branch, sel in (("upper", up & ~corner), ("lower", ~up & ~corner)):
                where = sel.nonzero()[:, 0]
                coeffs = t[branch].reshape(-1, nu, nv)
                for i in range(0, where.numel(), step):
                    at = where[i:i + step]
                    rows = torch.bmm(coeffs[pair[at]], _cheb(w[at], nv)[:, :, None])[:, :, 0]
                    out[k, spin, at] = (rows * _cheb(u[at], nu)).sum(1)
            for branch, sel in (("upper", up & corner), ("lower", ~up & corner)):
                out[k, spin, sel] = t[branch + "_corners"][pair[sel]]
    return out.reshape(2, 2, b, n, n)


def _all_minors(a):
    """Principal minors [batch][2^n] (bit i of the index: row i) of a [batch][n][n]."""
    b, n = a.shape[0], a.shape[1]
    shift = a.abs().amax((1, 2)) / (n * n)  # a uniform shift keeps the pivots away from zero
    a = a + shift[:, None, None] * torch.eye(n, dtype=a.dtype, device=a.device)
    m = torch.ones((b, 1), dtype=a.dtype, device=a.device)
    level = a[:, None]
    for _ in range(n):
        pivot = level[:, :, 0, 0]
        rest = level[:, :, 1:, 1:]
        schur = rest - level[:, :, 1:, :1] * (level[:, :, :1, 1:] / pivot[..., None, None])
        m = torch.cat([m, m * pivot], 1)
        level = torch.cat([rest, schur], 1)
    m = m.reshape([b] + [2] * n)
    for axis in range(1, n + 1):  # remove the shift, row by row: the minor is linear in each diagonal entry
        m0, m1 = m.select(axis, 0), m.select(axis, 1)
        m = torch.stack([m0, m1 - shift.reshape([b] + [1] * (n - 1)) * m0], axis)
    return m.reshape(b, 1 << n)


def _connected(a, n, anchored_everywhere, threshold):
    """The connected sums dp [batch][2^n] of a [batch][2^n]; only the masks with
    vertex 0 unless anchored_everywhere."""
    b = a.shape[0]
    dp = torch.zeros((1 << n, b), dtype=a.dtype, device=a.device)
    at = a.t().contiguous()
    for mask in sorted(range(1, 1 << n), key=lambda x: bin(x).count("1")):
        anchor = mask & -mask
        if anchor != 1 and not anchored_everywhere:
            continue
        rest, subs = mask ^ anchor, []
        x = rest
        while x:
            x = (x - 1) & rest
            subs.append(x | anchor)
        acc = at[mask].clone()
        if subs:
            i = torch.tensor(subs, device=a.device)
            rhs = acc.abs()
            for k in range(0, len(subs), 512):
                terms = dp[i[k:k + 512]] * at[mask ^ i[k:k + 512]]
                acc -= terms.sum(0)
                rhs += terms.abs().sum(0)
            if threshold > 0:
                acc[acc.abs() < threshold * rhs] = 0.0
        dp[mask] = acc
    return dp.t()


def exact(case, seed):
    """The same values by dense Chebyshev sums, minors and subset sums in 64
    bits. None for Markov chains and the double-double mode (more than 64
    bits), and where it would take long."""
    if case["entry"] == "chains" or case["real"] != "double":
        return None
    n, batch = case["order"], case["batch"]
    if n > 10 and case["entry"] != "assemble":
        return None  # 64 bits do not hold the cancellation of these orders
    p = _params(case)
    _, tables = _table_set(case)
    v, orders = _inputs(case, seed)
    sc = math.sqrt(float(p.u) * p.sites * float(p.beta))
    shifts = (float(p.alpha_down) / float(p.u), float(p.alpha_up) / float(p.u))
    threshold = 2.0e-16 * float(p.z_safety)
    subsets = case["entry"] == "subsets"
    if case["entry"] == "assemble":
        g = _exact_green(case, p, tables, v)
        for spin in range(2):
            g[:, spin].diagonal(dim1=-2, dim2=-1).add_(shifts[spin])
        g = g.permute(2, 0, 1, 3, 4)
        diag = g.diagonal(dim1=-2, dim2=-1).contiguous()
        return {"green": (g * sc).reshape(batch, 2, 2, n * n), "diag": diag, "status": None}
    values = torch.zeros((batch, 1 << n) if subsets else (batch,), dtype=torch.float64, device="cuda")
    for k in sorted(set(orders.tolist())):
        which = (orders == k).nonzero()[:, 0]
        for part in which.split(max(1, 16384 * 1024 >> k)):
            g = _exact_green(case, p, tables, v[part, :k])
            for spin in range(2):
                g[:, spin].diagonal(dim1=-2, dim2=-1).add_(shifts[spin])
            total = 0.0
            for q, r in enumerate((2, 1)):
                one = -r * float(p.u) * float(p.beta) * (g[q, 0].diagonal(dim1=-2, dim2=-1) *
                                                        g[q, 1].diagonal(dim1=-2, dim2=-1) - shifts[0] * shifts[1])
                if k == 1:
                    x = one if not subsets else None
                    x = x[:, 0]
                else:
                    a = _all_minors(g[q, 0] * sc) * _all_minors(g[q, 1] * sc)
                    dp = _connected(a, k, subsets, threshold)
                    if subsets:
                        bits = [bin(m).count("1") for m in range(1 << k)]
                        pref = torch.tensor([float(-r) ** c / (math.factorial(c) * p.sites) for c in bits],
                                            dtype=torch.float64, device="cuda")
                        x = dp * pref
                        for i in range(k):
                            x[:, 1 << i] = one[:, i]
                        x[:, 0] = 0.0
                    else:
                        x = dp[:, -1] * (float(-r) ** k / (math.factorial(k) * p.sites))
                total = total + x if q == 0 else total - 2.0 * x
            values[part] = total
    if case["entry"] == "single":
        return float(values[0])
    return {"values": values, "status": None}
