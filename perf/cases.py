"""The work that users have this framework do, as measurable cases.

A case is one call a program makes over and over: a forcing interval of a
routing model (`set_inputs`, `step_advance`, and `collect_statistics` where
output is saved), a forward and backward pass of a calibration window
(`AdjointRouting.window`), or a chunk of gridded runoff mapped onto the
catchments (`shard_forcing`).  Sizes, intervals and networks are those of
`cmfb200.synthetic.CONFIGS`, the tests and bench.py, and odd sizes between
them; the networks are seeded synthetic ones, and the seed of `prepare` draws
the model's state (nine cells in ten above their banks, as after a week of
rain) and its forcing.

`exact` restates the routing equations in plain 64-bit torch (and, for the
windows, differentiates them with autograd); only the order in which a model
lays out its catchments is taken from the framework.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "cama-flood-gpu_b200"))

from cmfb200 import CaMaFlood, synthetic as syn, topology  # noqa: E402
from cmfb200.adjoint import CELL_STATE, PARAMS, PATH_STATE, AdjointRouting  # noqa: E402
from cmfb200.forcing import build_local_mapping, shard_forcing  # noqa: E402

DEVICE = "cuda"
DAY, HOUR = 86400.0, 3600.0
MM_PER_DAY = 86400000.0          # mm/day x m^2 -> m^3/s
GRAVITY, ALPHA, MIN_KINEMATIC = 9.8, 0.7, 1e-5
SAVED = {"mean": ["total_outflow"], "last": ["river_depth"]}  # what the reference's run script saves


def _route(name, n, full, interval, cap=0.0, precision="float32", members=1, basins=0, stats=False):
    return {"name": name, "kind": "route", "n": n, "full": full, "interval": interval, "cap": cap,
            "precision": precision, "members": members, "basins": basins, "stats": stats}


def listed():
    return [
        # one hourly interval of a regional model, the smallest call: launches and latency
        _route("hour_4k_full", 4_000, True, HOUR),
        # a day of the plain 60k network with the 3600 s sub-step cap
        _route("day_60k_plain", 60_000, False, DAY, cap=3600.0),
        # a day of a global 15-arcmin model with every module
        _route("day_250k_full", 250_000, True, DAY),
        # the same physics at an odd size with the daily mean and last-value output on
        _route("day_100k_full_saved", 100_003, True, DAY, stats=True),
        # an fp64 run, as calibration checks its gradients against
        _route("day_30k_full_fp64", 30_011, True, DAY, precision="float64"),
        # an hour of a 2M-catchment map of large single-mouth basins, no extra module
        _route("hour_2m_plain", 2_000_003, False, HOUR, basins=166),
        # an hour of the 3-arcmin global model with every module: the largest
        _route("hour_6m_full", 6_000_000, True, HOUR),
        # 64 members of a regional ensemble in large basins, runoff and Manning perturbed
        _route("hour_64x60k_plain", 60_000, False, HOUR, members=64, basins=5),
        # a few members with every module, neither count a power of two
        _route("hour_6x50k_full", 50_021, True, HOUR, members=6),
        # calibration: one day of the 250k full-physics model, forward and backward
        {"name": "window_250k_full", "kind": "window", "n": 250_000, "full": True, "interval": DAY,
         "intervals": 1},
        # calibration of a small basin set over hourly forcing: launch-bound
        {"name": "window_20k_plain", "kind": "window", "n": 20_011, "full": False,
         "interval": HOUR, "intervals": 6},
        # a day of hourly quarter-degree runoff onto 2M catchments
        {"name": "forcing_2m", "kind": "forcing", "n": 2_000_000, "ny": 720, "nx": 1440,
         "steps": 24, "members": 0, "grid": "float32", "out": "float32", "missing": False},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randint(0, 1)


def draw(rng):
    kind = rng.choice(("route", "route", "route", "ensemble", "window", "forcing"))
    full = rng.random() < 0.6
    if kind == "route":
        wide = rng.random() < 0.2
        interval = rng.choice((HOUR, 6 * HOUR, DAY))
        n = _size(rng, 1_000, {HOUR: 3_000_000, 6 * HOUR: 800_000, DAY: 250_000}[interval] // (3 if wide else 1))
        c = _route("", n, full, interval, cap=rng.choice((0.0, 0.0, 600.0, 3600.0)),
                   precision="float64" if wide else "float32",
                   basins=0 if full else rng.choice((0, max(1, n // 12_000))),
                   stats=n < 500_000 and rng.random() < 0.3)
    elif kind == "ensemble":
        members = rng.choice((2, 3, 8, 12, 16, 24, 32, 64))
        n = _size(rng, 1_000, 3_000_000 // members)
        c = _route("", n, full, HOUR, members=members, basins=0 if full else max(1, n // 12_000))
    elif kind == "window":
        interval = rng.choice((HOUR, DAY))
        c = {"kind": "window", "n": _size(rng, 2_000, 100_000), "full": full, "interval": interval,
             "intervals": 1 if interval == DAY else rng.randint(1, 12)}
    else:
        ny = rng.choice((180, 360, 720))
        members = rng.choice((0, 0, 3, 8))
        c = {"kind": "forcing", "n": _size(rng, 5_000, 2_000_000), "ny": ny, "nx": 2 * ny,
             "steps": rng.choice((1, 5, 8, 24)) if members == 0 else rng.randint(1, 2), "members": members,
             "grid": rng.choice(("float32", "float64")), "out": rng.choice(("float32", "float64")),
             "missing": rng.random() < 0.3}
    c.pop("name", None)
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=3)
def _network(n, full, basins):
    """The map of a case: the shares of paths, levees and reservoirs are those
    of the 250k and 6M configurations."""
    if basins:
        return syn.generate_basins(basins, n, seed=3, min_size=1000)
    extra = dict(bifurcation_paths=max(2, n // 30), levee_fraction=0.2,
                 reservoirs=max(1, n // 700)) if full else {}
    return syn.generate(syn.NetworkSpec(n, seed=2, **extra))


def _net(case):
    return _network(case["n"], case["full"], case.get("basins", 0))


def _generator(case, seed):
    g = torch.Generator(DEVICE)
    g.manual_seed(1_000_003 * (seed + 1) + case["n"])
    return g


def _d(a):
    return torch.as_tensor(np.asarray(a), device=DEVICE).double()


def _fields(net, g):
    """The map's fields with a state drawn from `g`: river and floodplain
    filled to one depth each, water in motion along the surface slope."""
    f = dict(net.fields)
    n = net.num_catchments
    rand = lambda: torch.rand(n, generator=g, device=DEVICE, dtype=torch.float64)  # noqa: E731
    w, length, rh = _d(f["river_width"]), _d(f["river_length"]), _d(f["river_height"])
    area, elev, table = _d(f["catchment_area"]), _d(f["catchment_elevation"]), _d(f["flood_depth_table"])
    K = table.shape[1]
    h = torch.where(rand() < 0.9, -0.3 * torch.log1p(-rand()), 0.0).minimum(table[:, -1])
    depth = torch.where(h > 0, rh + h, rh * (0.2 + 0.8 * rand()))
    dw = area / length / K
    below, lo, top = torch.zeros_like(h), torch.zeros_like(h), torch.zeros_like(h)
    for k in range(K):
        layer = (table[:, k] - lo).clamp(min=1e-6)
        x = (h - lo).clamp(min=0.0).minimum(layer)
        below += length * x * (w + k * dw + 0.5 * dw * x / layer)
        top += x / layer
        lo = table[:, k]
    flood = (below - length * w * h).clamp(min=0.0)
    dn = torch.as_tensor(f["downstream_id"], device=DEVICE)
    mouth = dn == torch.arange(n, device=DEVICE)
    eta = depth + elev - rh
    eta_dn = torch.where(mouth, elev, eta[dn])
    surface = torch.where(mouth, eta, torch.maximum(eta, eta_dn))
    slope = ((eta - eta_dn) / _d(f["downstream_distance"])).clamp(-1e-3, 1e-3)
    flow_depth = surface - (elev - rh)
    out = w * flow_depth ** (5.0 / 3.0) * slope.sign() * slope.abs().sqrt() / _d(f["river_manning"])
    state = {"river_storage": length * w * depth, "flood_storage": flood, "river_depth": depth,
             "flood_depth": h, "protected_depth": h, "flood_fraction": (top * dw * length / area).clamp(0, 1),
             "river_outflow": out, "river_cross_section_depth": flow_depth,
             "flood_cross_section_depth": (surface - elev).clamp(min=0.0),
             "flood_cross_section_area": (flood / length - h * w).clamp(min=0.0)}
    for k, v in state.items():
        f[k] = (v if k.endswith("storage") else v.float()).cpu().numpy()
    return f


def _rain(net, g, *lead):
    """Runoff in m^3/s, gamma(0.5) about a mean of 2 mm/day, [*lead, N]."""
    z = torch.randn(*lead, net.num_catchments, generator=g, device=DEVICE)
    return 2.0 * z * z * torch.as_tensor(net.fields["catchment_area"], device=DEVICE) / MM_PER_DAY


def _members(case, net, g, runoff):
    """Per-member runoff [N, M] and Manning fields of the ensemble workload."""
    shape = (net.num_catchments, case["members"])
    factor = torch.exp(0.3 * torch.randn(shape, generator=g, device=DEVICE))
    spread = 0.8 + 0.4 * torch.rand(shape, generator=g, device=DEVICE)
    manning = torch.as_tensor(net.fields["river_manning"], device=DEVICE)[:, None] * spread
    return runoff[:, None] * factor, manning.cpu().numpy()


def _inputs(case, seed):
    """(network, fields, runoff in the map's order, per-member Manning)."""
    net, g = _net(case), _generator(case, seed)
    fields = _fields(net, g)
    if case["kind"] == "window":
        return net, fields, _rain(net, g, case["intervals"]).double(), None
    runoff = _rain(net, g)
    if case["members"] == 1:
        return net, fields, runoff, None
    return net, fields, *_members(case, net, g, runoff)


def _prepare_route(case, seed):
    net, fields, runoff, manning = _inputs(case, seed)
    many = case["members"] > 1
    large = case["n"] * case["members"] > 1_000_000   # the CTA size the tuner picks there
    model = CaMaFlood(device=DEVICE, input_proxy=fields, opened_modules=net.opened_modules,
                      step_duration=case["interval"], precision=case["precision"],
                      num_members=case["members"], max_sub_step_seconds=case["cap"],
                      batched_fields={"river_manning": manning} if many else None,
                      variables_to_save=SAVED if case["stats"] else None,
                      **({"BLOCK_SIZE": 64} if large else {}))
    if many:
        model.set_member_tile(math.gcd(case["members"], 16))
    order = torch.as_tensor(model.order, device=DEVICE)
    return {"kind": "route", "model": model, "stats": case["stats"],
            "runoff": runoff.index_select(0, order).to(model.base.runoff.dtype)}


def _gauges(net, order):
    """Forty cells with a large upstream area, and a discharge level at each."""
    area = net.info["upstream_area_km2"][order]
    at = np.flatnonzero(area > np.quantile(area, 0.8))
    at = at[:: max(1, at.size // 40)][:40]
    return at, area[at] * 1e6 * 2e-3 / 86400.0


def _prepare_window(case, seed):
    net, fields, runoff, _ = _inputs(case, seed)
    model = CaMaFlood(device=DEVICE, input_proxy=fields, opened_modules=net.opened_modules,
                      step_duration=case["interval"], precision="float64")
    gauges, level = _gauges(net, model.order)
    engine = AdjointRouting(model, gauges)
    params = {k: v.requires_grad_() for k, v in engine.parameters().items()}
    forcing = runoff.index_select(1, torch.as_tensor(model.order, device=DEVICE)).requires_grad_()
    return {"kind": "window", "engine": engine, "params": params, "forcing": forcing,
            "state0": engine.initial_state().requires_grad_(), "level": _d(level)}


def _prepare_forcing(case, seed):
    table, ids = _mapping(case["n"], case["ny"], case["nx"])
    lead = (case["steps"], case["members"]) if case["members"] else (case["steps"],)
    grid = torch.randn(*lead, case["ny"], case["nx"], generator=_generator(case, seed), device=DEVICE,
                       dtype=getattr(torch, case["grid"]))
    grid = 2.0 * grid * grid
    if case["missing"]:
        grid = torch.where(grid > 8.0, -9999.0, grid)
    return {"kind": "forcing", "grid": grid, "mapping": build_local_mapping(table, ids, DEVICE),
            "options": dict(dtype=getattr(torch, case["out"]), unit_factor=MM_PER_DAY,
                            **({"missing_value": -9999.0, "clamp_negative": True} if case["missing"] else {}))}


@functools.lru_cache(maxsize=2)
def _mapping(n, ny, nx):
    net = _network(n, False, 0)
    order, _ = topology.bfs_order(net.fields["downstream_id"].astype(np.int32))
    return syn.runoff_mapping(net, (ny, nx), seed=2), net.fields["catchment_id"][order]


def prepare(case, seed):
    return {"route": _prepare_route, "window": _prepare_window, "forcing": _prepare_forcing}[case["kind"]](case, seed)


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(state):
    if state["kind"] == "forcing":
        return shard_forcing(state["grid"], state["mapping"], **state["options"])
    if state["kind"] == "window":
        p = state["params"]
        q, final = state["engine"].window(p, state["forcing"], state["state0"])
        loss = ((q / state["level"] - 1.0) ** 2).sum()
        wrt = [p[k] for k in PARAMS] + [state["forcing"], state["state0"]]
        return {"discharge": q.detach(), "final": final.detach(),
                "gradients": list(torch.autograd.grad(loss, wrt))}
    model = state["model"]
    model.set_inputs(state["runoff"])
    model.step_advance()
    out = dict(model.state_tensors())
    out.update(river_inflow=model.base.river_inflow, flood_inflow=model.base.flood_inflow,
               sub_steps=model.sub_step_counts())
    if state["stats"]:
        out.update(model.collect_statistics())
    return out


def work(case):
    """Bytes: a state beyond the 126 MB L2 has to pass through memory once per
    sub-step, a smaller one once per interval.  Flops: about 250 per catchment
    and sub-step, the sub-steps by the length of a typical CFL step."""
    n = case["n"]
    if case["kind"] == "forcing":
        series = case["steps"] * max(1, case["members"])
        item = {"float32": 4, "float64": 8}
        return {"bytes": 8 * n + 12 * 2.5 * n + series * (case["ny"] * case["nx"] * item[case["grid"]]
                                                           + n * item[case["out"]]),
                "flops": series * 2 * 2.5 * n}
    steps = case["interval"] * case.get("intervals", 1) / 160.0
    if case["kind"] == "window":
        # the state, the parameters and every interval's runoff once in, and
        # the final state and all gradients once out, with two checkpointed
        # forward passes and one reverse pass of arithmetic
        state = (12 * n + (2 * 5 * (n // 30) if case["full"] else 0)) * 8
        return {"bytes": 3 * state + 14 * 8 * n + 2 * 8 * n * case["intervals"], "flops": steps * n * 250.0 * 4}
    wide = 2 if case["precision"] == "float64" else 1
    cell = (172 if not case["full"] else 207) * wide * n * case["members"]
    return {"bytes": cell * (max(1.0, steps) if cell > 126e6 else 1.0),
            "flops": steps * n * case["members"] * 250.0}


# --------------------------------------------------------------------------
# the same in plain 64-bit torch
# --------------------------------------------------------------------------
def _root(x, power=0.5):
    """x ** power of a non-negative tensor, with derivative 0 at 0."""
    live = x > 0
    return torch.where(live, torch.where(live, x, 1.0).pow(power), 0.0)


def _floored_root(x):
    live = x > 1e-12
    return torch.where(live, torch.where(live, x, 1.0).sqrt(), 1e-6)


def _larger(a, b):
    return torch.where(a >= b, a, b)


def _smaller(a, b):
    return torch.where(a <= b, a, b)


class _Routing:
    """The routing equations of CaMa-Flood over tensors in one catchment order."""

    def __init__(self, fields, order, modules, cap=0.0):
        order = torch.as_tensor(np.asarray(order), dtype=torch.long, device=DEVICE)
        n = order.numel()
        inverse = torch.empty_like(order)
        inverse[order] = torch.arange(n, device=DEVICE)
        cells = lambda k: _d(fields[k])[order]                                   # noqa: E731
        index = lambda k: inverse[torch.as_tensor(fields[k], device=DEVICE)]     # noqa: E731
        self.dn = inverse[torch.as_tensor(fields["downstream_id"], device=DEVICE)[order]]
        self.mouth = self.dn == torch.arange(n, device=DEVICE)
        self.inner = ~self.mouth
        self.to = self.dn[self.inner]
        self.length, self.elev, self.area = cells("river_length"), cells("catchment_elevation"), cells("catchment_area")
        self.dist, self.table, self.cap = cells("downstream_distance"), cells("flood_depth_table"), cap
        self.params = {k: cells(k) for k in PARAMS}
        none = torch.zeros(n, dtype=torch.bool, device=DEVICE)
        self.levee, self.dam, self.above_dam = none, none, none
        self.state = {k: cells(k) if k in fields else torch.zeros(n, device=DEVICE, dtype=torch.float64)
                      for k in CELL_STATE}
        self.paths = "bifurcation" in modules
        if "levee" in modules:
            self.lc = index("levee_catchment_id")
            self.levee = none.index_fill(0, self.lc, True)
            self.crown, self.frac = _d(fields["levee_crown_height"]), _d(fields["levee_fraction"])
            K = self.table.shape[1]
            # base height: the profile read at frac x K, rounded to 32 bits as the model holds it
            rows = torch.cat([torch.zeros_like(self.table[self.lc, :1]), self.table[self.lc]], 1).float()
            at = (self.frac.float() * K).clamp(0, K)
            low = at.floor().long()
            a, b = (rows.gather(1, i[:, None])[:, 0] for i in (low, (low + 1).clamp(max=K)))
            self.base = (a + (at - low.float()) * (b - a)).double()
        if "reservoir" in modules:
            self.rc = index("reservoir_catchment_id")
            self.dam = none.index_fill(0, self.rc, True)
            self.above_dam = ~self.dam & self.inner & self.dam[self.dn]
            single = lambda k: torch.as_tensor(fields[k], device=DEVICE)         # noqa: E731
            cons, emerg, norm, flood = (single(k) for k in ("conservation_volume", "emergency_volume",
                                                             "normal_outflow", "flood_control_outflow"))
            year, half = 365.0 * 86400.0, 180.0 * 86400.0
            eff = torch.minimum(norm, (cons * 0.7 + norm * year / 4.0) / half) * 1.5
            self.rule = [v.double() for v in (cons, emerg, cons + (emerg - cons) / 0.95 * 0.1, eff,
                                              (eff + flood) * 0.5, flood)]
            rs, fs = self.state["river_storage"], self.state["flood_storage"]
            low = rs[self.rc] + fs[self.rc] < self.rule[0]
            rs[self.rc] = torch.where(low, self.rule[0], rs[self.rc])
            fs[self.rc] = torch.where(low, 0.0, fs[self.rc])
        if self.paths:
            self.a, self.b = index("bifurcation_catchment_id"), index("bifurcation_downstream_id")
            self.sill, self.path_w = _d(fields["bifurcation_elevation"]), _d(fields["bifurcation_width"])
            self.path_n, self.path_len = _d(fields["bifurcation_manning"]), _d(fields["bifurcation_length"])
            near = self.dam | self.above_dam
            self.sill[near[self.a] | near[self.b]] = 1e20
            self.state.update({k: torch.zeros_like(self.sill) for k in PATH_STATE})

    def sub_steps(self, s, interval):
        dt = ALPHA * self.dist / (GRAVITY * s["river_depth"].detach().clamp(min=0.01)).sqrt()
        dt = dt.clamp(max=min(interval, self.cap) if self.cap > 0 else interval)
        n = torch.where(self.dam | self.above_dam, 1.0, torch.floor(interval / dt - 0.01) + 1.0)
        return int(n.max().item())

    def momentum(self, s, p, runoff, dt):
        rh, w, n_riv, n_fld = p["river_height"], p["river_width"], p["river_manning"], p["flood_manning"]
        rs, fs, hr, hf = s["river_storage"], s["flood_storage"], s["river_depth"], s["flood_depth"]
        bed = self.elev - rh
        eta = hr + bed
        eta_dn = torch.where(self.mouth, self.elev, eta[self.dn])
        high = torch.maximum(eta, eta_dn)
        slope = (eta - eta_dn) / self.dist
        r_now = torch.where(self.mouth, hr, high - bed)
        f_now = (torch.where(self.mouth, eta, high) - self.elev).clamp(min=0.0)
        a_now = (fs / self.length - hf * w).clamp(min=0.0)
        r_mid = _floored_root(r_now * s["river_cross_section_depth"])
        f_mid = _floored_root(f_now * s["flood_cross_section_depth"])
        a_mid = _floored_root(a_now * s["flood_cross_section_area"].clamp(min=1e-6))
        gdt = GRAVITY * dt
        unit = s["river_outflow"] / w
        qr = w * (unit + gdt * r_mid * slope) / (1.0 + gdt * n_riv ** 2 * unit.abs() * r_mid ** (-7.0 / 3.0))
        qr = torch.where((r_mid > 1e-5) & (r_now * w > 1e-5), qr, 0.0)
        qf = ((s["flood_outflow"] + gdt * a_mid * slope.clamp(-0.005, 0.005))
              / (1.0 + gdt * n_fld ** 2 * s["flood_outflow"].abs() * f_mid ** (-4.0 / 3.0) / a_mid))
        qf = torch.where((f_mid > 1e-5) & (a_now > 1e-5), qf, 0.0)
        qf = torch.where(qr * qf < 0.0, 0.0, qf)
        back = (qr < 0.0) & self.inner
        moved = torch.where(back, (-qr - qf) * dt, 1.0)
        rate = (0.05 * (rs + fs + s["protected_storage"]) / moved).clamp(max=1.0)
        qr, qf = torch.where(back, qr * rate, qr), torch.where(back, qf * rate, qf)
        if self.dam.any():
            zero = torch.zeros_like(qr)
            fall = ((self.elev - self.elev[self.dn]) / self.dist).clamp(min=MIN_KINEMATIC)
            kr = _larger(_smaller(w * hr * (fall.sqrt() / n_riv) * _root(hr * hr, 1 / 3), rs / dt), zero)
            kf = _larger(fs / self.length - hf * w, zero) * (fall.clamp(max=0.005).sqrt() / n_fld) * _root(hf * hf, 1 / 3)
            kf = _larger(_smaller(kf, fs / dt), zero)
            qr, qf = torch.where(self.above_dam, kr, qr), torch.where(self.above_dam, kf, qf)
            release = self.release((rs + fs)[self.rc], (s["reservoir_total_inflow"] + runoff)[self.rc], dt)
            qr = qr.index_put((self.rc,), release)
            qf = qf.index_put((self.rc,), torch.zeros_like(release))
        return qr, qf, r_now, f_now, a_now

    def release(self, total, inflow, dt):
        cons, emerg, adjust, q_norm, q_adj, q_flood = self.rule
        first, second, third = total <= cons, total <= adjust, total <= emerg
        q1 = q_norm * _root(total / cons)
        x = torch.where(second & ~first, (total - cons) / (adjust - cons), 1.0)
        q2 = q_norm + x ** 3 * (q_adj - q_norm)
        x = torch.where(third & ~second, (total - adjust) / (emerg - adjust), 1.0)
        ramp = q_adj + x ** 0.1 * (q_flood - q_adj)
        share = q_norm + (total - cons) / (emerg - cons) * (inflow - q_norm)
        q3 = torch.where(inflow >= q_flood, _larger(share, ramp), ramp)
        q4 = torch.where(inflow >= q_flood, inflow, q_flood)
        q = torch.where(first, q1, torch.where(second, q2, torch.where(third, q3, q4)))
        return _smaller(_larger(q, torch.zeros_like(q)), total / dt)

    def path_flux(self, s, p, dt):
        eta = s["river_depth"] + self.elev - p["river_height"]
        behind = torch.where(self.levee, _smaller(self.elev + s["protected_depth"], eta), eta)
        held = s["river_storage"] + s["flood_storage"]
        held = torch.where(self.dam, held, held + s["protected_storage"])
        a, b = self.a, self.b
        top, top_behind = _larger(eta[a], eta[b]), _larger(behind[a], behind[b])
        slope = ((eta[a] - eta[b]) / self.path_len).clamp(-0.005, 0.005)[:, None]
        before = s["bifurcation_cross_section_depth"]
        if self.levee.any():
            surface = torch.cat([top[:, None], top_behind[:, None].expand(-1, self.sill.shape[1] - 1)], 1)
            h = _larger(surface - self.sill, torch.zeros_like(self.sill))
            first = _root(h[:, :1] * before[:, :1])
            mid = torch.cat([torch.where(first <= 0.0, h[:, :1], first), h[:, 1:]], 1)
        else:
            h = _larger(top[:, None] - self.sill, torch.zeros_like(self.sill))
            mid = _larger(_root(h * before), _root(h * 0.01))
        live = mid > 1e-5
        m = torch.where(live, mid, 1.0)
        unit = s["bifurcation_outflow"] / self.path_w
        gdt = GRAVITY * dt
        q = self.path_w * (unit + gdt * m * slope) / (1.0 + gdt * self.path_n ** 2 * unit.abs() * m ** (-7.0 / 3.0))
        q = torch.where(live, q, 0.0)
        total = q.sum(1)
        moved = total.abs() * dt
        flows = moved > 0
        rate = torch.where(flows, (0.05 * _smaller(held[a], held[b]) / torch.where(flows, moved, 1.0)).clamp(max=1.0), 1.0)
        return q * rate[:, None], total * rate, h

    def stage(self, total, rh, w):
        length, K = self.length, self.table.shape[1]
        bank, dw = length * w * rh, self.area / self.length / K
        over = total > bank
        low = torch.cat([torch.zeros_like(self.table[:, :1]), self.table[:, :-1]], 1)
        k = torch.arange(K, device=DEVICE, dtype=torch.float64)
        layer = length[:, None] * (w[:, None] + (k + 0.5) * dw[:, None]) * (self.table - low)
        marks = torch.cat([bank[:, None], bank[:, None] + torch.cumsum(layer, 1)], 1)
        full = (total[:, None] > marks[:, 1:]).long().cumprod(1).sum(1)
        above = full == K
        at = full.clamp(max=K - 1)[:, None]
        d_lo = torch.where(above, self.table[:, -1], low.gather(1, at)[:, 0])
        extra = total - marks.gather(1, full[:, None])[:, 0]
        grad = torch.where(above, 1.0, (self.table.gather(1, at)[:, 0] - d_lo) / dw)
        wide = w + full * dw
        inside = torch.where(above | ~over, 1.0, wide * wide + 2.0 * extra / (grad * length))
        more = inside.sqrt() - wide
        h = torch.where(above, d_lo + extra / (wide * length), d_lo + more * grad)
        column = bank + length * w * h
        rs = torch.where(over & (column < total), column, total)
        rest = total - rs
        fs = torch.where(over & (rest > 0), rest, 0.0)
        part = torch.where(above, 1.0, ((wide + more - w) * length / self.area).clamp(0.0, 1.0))
        return rs, fs, rs / (length * w), torch.where(over, h, 0.0), torch.where(over, part, 0.0)

    def behind_levees(self, rs, fs, rd, fd, part, rh, w):
        """River, flood and protected storage of the levee cells again."""
        c, crown, base, frac = self.lc, self.crown, self.base, self.frac
        length, table, K = self.length[c], self.table[c], self.table.shape[1]
        span = self.area[c] / length
        dw, dist = span / K, frac * span
        zero, total = torch.zeros_like(rs), rs + fs
        bank = length * w * rh
        lows = torch.cat([torch.zeros_like(table[:, :1]), table[:, :-1]], 1)
        layers = _larger(table - lows, torch.full_like(table, 1e-6))
        widths = w[:, None] + torch.arange(K, device=DEVICE, dtype=torch.float64) * dw[:, None]
        tops = bank[:, None] + torch.cumsum(length[:, None] * (widths + 0.5 * dw[:, None]) * layers, 1)
        starts = torch.cat([bank[:, None], tops[:, :-1]], 1)

        def filled(z):
            """Profile storage up to height z."""
            inside = (z[:, None] > lows) & (z[:, None] <= table)
            hit = inside.any(1)
            at = inside.long().argmax(1, keepdim=True)
            pick = lambda t: t.gather(1, at)[:, 0]  # noqa: E731
            r = (z - pick(lows)) / pick(layers)
            within = pick(starts) + length * (pick(widths) + 0.5 * r * dw) * r * pick(layers)
            beyond = tops[:, -1] + length * (w + K * dw) * (z - table[:, -1])
            return torch.where(hit, within, torch.where(z > table[:, -1], beyond, bank)), torch.where(hit, at[:, 0], K)

        s_base, base_layer = filled(base)
        s_crown, _ = filled(crown)
        wedge = (dist + w) * length
        s_top = s_base + wedge * (crown - base)
        first = (frac * K).long()
        marks = tops + wedge[:, None] * (crown[:, None] - table)
        layer = torch.arange(K, device=DEVICE)
        stop = (layer >= first[:, None]) & (total[:, None] < marks)
        found = stop.any(1)
        at = torch.where(found, stop.long().argmax(1), K)
        prior = (at - 1).clamp(min=0)[:, None]
        fresh = at <= first
        s_first = torch.where(base_layer <= first, s_base, bank) + wedge * (crown - base)
        s_fill = torch.where(fresh, s_first, marks.gather(1, prior)[:, 0])
        w_fill = torch.where(fresh, 0.0, dw * at - dist)
        d_fill = torch.where(fresh, 0.0, table.gather(1, prior)[:, 0] - base)
        grad = layers.gather(1, at.clamp(max=K - 1)[:, None])[:, 0] / dw
        more = total - s_fill
        in_table = w_fill * w_fill + 2.0 * more / length / (grad + 1e-9)
        pd_fill = base + d_fill + torch.where(found, (_root(_larger(in_table, zero)) - w_fill) * grad,
                                              more / (w_fill * length + 1e-9))
        part_fill = torch.where(found, ((w_fill + dist) / (dw * K)).clamp(0.0, 1.0), 1.0)
        over = total >= s_crown
        filling = ~over & (total >= s_top)
        rising = ~over & ~filling & (total >= s_base)
        fd_rise = base + (total - s_base) / wedge
        level = torch.where(rising, fd_rise, crown)
        column = bank + length * w * level
        rs1 = torch.where(rising | filling, _smaller(column, total), rs)
        rest = (total - rs1).clamp(min=0.0)
        fs1 = torch.where(over, _smaller(_larger(s_top + (fd - crown) * wedge - rs, zero), rest),
                          torch.where(filling, _smaller(_larger(s_top - column, zero), rest),
                                      torch.where(rising, rest, fs)))
        ps1 = (rest - fs1).clamp(min=0.0)
        shift = rising | filling
        active = total >= bank
        keep = lambda new, old: torch.where(active, new, old)  # noqa: E731
        return (keep(rs1, rs), keep(fs1, fs), keep(ps1, zero), keep(torch.where(shift, column / length / w, rd), rd),
                keep(torch.where(shift, level, fd), fd),
                keep(torch.where(over, fd, torch.where(filling, pd_fill, zero)), zero),
                keep(torch.where(rising, frac, torch.where(filling, part_fill, part)), part))

    def sub_step(self, s, p, runoff, dt):
        """(state, diagnostics) after one sub-step."""
        qr, qf, r_now, f_now, a_now = self.momentum(s, p, runoff, dt)
        rs, fs, zero = s["river_storage"], s["flood_storage"], torch.zeros_like(qr)
        out = (qr.clamp(min=0.0) + qf.clamp(min=0.0)) * dt
        out = out.index_add(0, self.to, -(qr.clamp(max=0.0) + qf.clamp(max=0.0))[self.inner] * dt)
        new = {}
        if self.paths:
            q, total, h = self.path_flux(s, p, dt)
            none = torch.zeros_like(total)
            out = out.index_add(0, self.a, _larger(total, none) * dt).index_add(0, self.b, -_smaller(total, none) * dt)
        live = out > 1e-8
        rate = torch.where(live, ((rs + fs) / torch.where(live, out, 1.0)).clamp(max=1.0), 1.0)
        rate_dn = rate[self.dn]
        ur, uf = torch.where(qr >= 0.0, qr * rate, qr * rate_dn), torch.where(qf >= 0.0, qf * rate, qf * rate_dn)
        rin = zero.index_add(0, self.to, ur[self.inner])
        fin = zero.index_add(0, self.to, uf[self.inner])
        new["reservoir_total_inflow"] = torch.where(self.dam, rin + fin, s["reservoir_total_inflow"])
        lost = zero
        if self.paths:
            ra, rb = rate[self.a], rate[self.b]
            new["bifurcation_outflow"] = torch.where(q >= 0.0, q * ra[:, None], q * rb[:, None])
            new["bifurcation_cross_section_depth"] = h
            net = q.sum(1)
            net = torch.where(net >= 0.0, net * ra, net * rb)
            lost = zero.index_add(0, self.a, net).index_add(0, self.b, -net)
        river = rs + (rin - ur) * dt
        flood = fs + river.clamp(max=0.0) + (fin - uf - lost) * dt
        river = torch.where(river > 0.0, river, zero)
        both = river + flood
        river = torch.where(flood < 0.0, torch.where(both > 0.0, both, zero), river)
        flood = torch.where(flood > 0.0, flood, zero)
        total = river + flood + s["protected_storage"] + runoff * dt
        total = torch.where(total > 0.0, total, zero)
        rs, fs, rd, fd, part = self.stage(total, p["river_height"], p["river_width"])
        ps, pd = zero, fd
        if self.levee.any():
            c = (self.lc,)
            again = self.behind_levees(*(x[self.lc] for x in (rs, fs, rd, fd, part, p["river_height"], p["river_width"])))
            rs, fs, ps, rd, fd, pd, part = (x.index_put(c, y) for x, y in zip((rs, fs, ps, rd, fd, pd, part), again))
        new.update(river_storage=rs, flood_storage=fs, river_outflow=ur, flood_outflow=uf, river_depth=rd,
                   flood_depth=fd, river_cross_section_depth=r_now, flood_cross_section_depth=f_now,
                   flood_cross_section_area=a_now, protected_storage=ps, protected_depth=pd)
        return new, {"flood_fraction": part, "river_inflow": rin, "flood_inflow": fin}


def _exact_route(case, seed):
    net, fields, runoff, manning = _inputs(case, seed)
    order, _ = topology.bfs_order(fields["downstream_id"].astype(np.int32))
    got = []
    for m in range(case["members"]):
        r = _Routing(fields, order, net.opened_modules, case["cap"])
        rain = _d((runoff if manning is None else runoff[:, m]).cpu())[_d(order).long()]
        if manning is not None:
            r.params["river_manning"] = _d(manning[order, m])
        s, n = r.state, r.sub_steps(r.state, case["interval"])
        mean = 0.0
        for _ in range(n):
            s, more = r.sub_step(s, r.params, rain, case["interval"] / n)
            mean = mean + (s["river_outflow"] + s["flood_outflow"]) / n
        out = {**s, **more}
        if "reservoir" not in net.opened_modules:
            del out["reservoir_total_inflow"]
        if case["stats"]:
            out.update(total_outflow_mean=mean, river_depth_last=s["river_depth"])
        got.append(out)
    if manning is None:
        return {**got[0], "sub_steps": None}
    return {**{k: torch.stack([o[k] for o in got], -1) for k in got[0]}, "sub_steps": None}


def _exact_window(case, seed):
    from torch.utils.checkpoint import checkpoint
    net, fields, runoff, _ = _inputs(case, seed)
    order, _ = topology.bfs_order(fields["downstream_id"].astype(np.int32))
    r = _Routing(fields, order, net.opened_modules)
    gauges, level = _gauges(net, order)
    gauges = torch.as_tensor(gauges, device=DEVICE)
    params = {k: v.requires_grad_() for k, v in r.params.items()}
    forcing = runoff[:, torch.as_tensor(np.asarray(order), dtype=torch.long, device=DEVICE)].requires_grad_()
    names = CELL_STATE + (PATH_STATE if r.paths else ())
    first = [r.state[k].requires_grad_() for k in names]
    state, q = first, []

    def step(rain, dt, *values):
        new, _ = r.sub_step(dict(zip(names, values)), params, rain, dt)
        return tuple(new[k] for k in names)

    for t in range(case["intervals"]):
        n = r.sub_steps(dict(zip(names, state)), case["interval"])
        for _ in range(n):
            state = checkpoint(step, forcing[t], case["interval"] / n, *state, use_reentrant=False)
        now = dict(zip(names, state))
        q.append((now["river_outflow"] + now["flood_outflow"])[gauges])
    q = torch.stack(q)
    loss = ((q / _d(level) - 1.0) ** 2).sum()
    grads = torch.autograd.grad(loss, [params[k] for k in PARAMS] + [forcing] + first, allow_unused=True)
    grads = [torch.zeros_like(x) if d is None else d
             for d, x in zip(grads, [params[k] for k in PARAMS] + [forcing] + first)]
    flat = lambda parts: torch.cat([x.detach().reshape(-1) for x in parts])  # noqa: E731
    return {"discharge": q.detach(), "final": flat(state), "gradients": grads[:5] + [flat(grads[5:])]}


def _exact_forcing(case, seed):
    s = _prepare_forcing({**case}, seed)
    table, ids = _mapping(case["n"], case["ny"], case["nx"])
    grid = s["grid"].double().flatten(-2)
    if case["missing"]:
        grid = torch.where(grid == -9999.0, 0.0, grid)
    place = torch.empty(int(table["catchment_ids"].max()) + 1, dtype=torch.long, device=DEVICE)
    place[torch.as_tensor(ids, device=DEVICE)] = torch.arange(ids.size, device=DEVICE)
    rows = place[torch.as_tensor(table["catchment_ids"], device=DEVICE)]
    rows = rows.repeat_interleave(torch.as_tensor(np.diff(table["sparse_indptr"]), device=DEVICE))
    cols, weights = torch.as_tensor(table["sparse_indices"], device=DEVICE), _d(table["sparse_data"])
    out = [torch.zeros(ids.size, dtype=torch.float64, device=DEVICE).index_add(0, rows, g[cols] * weights)
           for g in grid.reshape(-1, grid.shape[-1])]
    out = torch.stack(out) / MM_PER_DAY
    return out if not case["members"] else out.reshape(case["steps"], case["members"], -1).transpose(1, 2)


def exact(case, seed):
    return {"route": _exact_route, "window": _exact_window, "forcing": _exact_forcing}[case["kind"]](case, seed)
