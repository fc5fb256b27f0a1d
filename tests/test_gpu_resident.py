"""The resident interval kernel, which step_advance takes for one member whose
state fits in the SMs' shared memory, against the four sub-step kernels
launched one by one (use_cuda_graph=False), which no interval form shares: the
state, the diagnostics and the statistics must be the same bits, at sizes
around the tile edges, from one catchment to several tiles per feature case."""
import numpy as np
import pytest
import torch

from cmfb200 import synthetic as syn

import parity as P

pytestmark = pytest.mark.gpu

DIAGNOSTICS = ("river_inflow", "flood_inflow", "total_storage", "water_surface_elevation",
               "protected_water_surface_elevation", "time_step", "outer_time_step", "current_step")
SAVED = {"mean": ["total_outflow", "flood_fraction"], "max": ["river_depth", "river_storage"],
         "min": ["flood_storage"], "last": ["flood_depth"]}


def _run(net, graph, days=2, fixed=None, saved=None, **kw):
    m = P.model_for(net, use_cuda_graph=graph, variables_to_save=saved, **kw)
    assert (m.resident_tiles > 0) == graph
    counts = []
    for d in range(days):
        m.set_inputs(torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda())
        m.step_advance(num_sub_steps=fixed)
        counts.append(int(m.sub_step_counts()[0].item()))
    torch.cuda.synchronize()
    m.check_status()
    out = dict(m.state_tensors())
    out.update({k: getattr(m.base, k) for k in DIAGNOSTICS if getattr(m.base, k) is not None})
    if m.bifurcation is not None:
        out.update(limit_rate=m.bifurcation.limit_rate, net=m.bifurcation.global_bifurcation_outflow)
    if saved:
        out.update(m.collect_statistics())
    return {k: v.cpu().numpy() for k, v in out.items()}, counts


def _same(net, **kw):
    a, ca = _run(net, True, **kw)
    b, cb = _run(net, False, **kw)
    assert ca == cb
    assert a.keys() == b.keys()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("case", list(P.CASES))
def test_resident_equals_direct_launches(case, precision, device):
    _same(P.make_network(case), precision=precision)


@pytest.mark.parametrize("n", [1, 31, 256, 257, 2049])
def test_resident_small_networks(n, device):
    _same(syn.generate(syn.NetworkSpec(n, seed=3)))


@pytest.mark.parametrize("n, precision", [(45_001, "float64"), (150_001, "float32"), (250_007, "float32")])
def test_resident_several_cells_per_thread(n, precision, device):
    """Rows in shared memory, several cells per thread, and (250k) rows in L2."""
    net = syn.generate(syn.NetworkSpec(n, seed=5, bifurcation_paths=n // 30, levee_fraction=0.2,
                                       reservoirs=n // 700))
    _same(net, precision=precision, days=1, fixed=30)


def test_resident_statistics(device):
    _same(P.make_network("full", n=9001), saved={**SAVED, "mean": SAVED["mean"] + ["protected_storage"]})


def test_resident_sub_step_cap_and_dt_cap(device):
    _same(P.make_network("bif"), max_sub_step_seconds=600.0)
    net = P.make_network("plain")
    m = P.model_for(net, max_sub_steps_cap=3)
    m.step_advance()
    assert int(m.sub_step_counts()[0].item()) == 3
    with pytest.raises(RuntimeError):
        m.check_status()


def test_resident_is_left_to_what_it_runs(device):
    """Members, the budget, the persistent kernel and a network beyond the
    SMs' shared memory take their own forms."""
    net = P.make_network("plain", n=2000)
    assert P.model_for(net).resident_tiles == 16
    assert P.model_for(net, budget=True).resident_tiles == 0
    assert P.model_for(net, persistent=True).resident_tiles == 0
    assert P.model_for(net, num_members=2).resident_tiles == 0
    assert P.model_for(syn.generate(syn.NetworkSpec(400_000, seed=1))).resident_tiles == 0


def test_resident_models_on_streams_of_their_own(device):
    """Two models, each on its own stream, one of high priority, their intervals
    in flight together: each equals its own run on one stream."""
    nets = [P.make_network("full", n=40_000, seed=2), P.make_network("bif", n=23_000, seed=6)]
    alone = [_run(net, True, days=3)[0] for net in nets]
    models = [P.model_for(net) for net in nets]
    runoff = [[torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda() for d in range(3)]
              for m, net in zip(models, nets)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-1)]
    for d in range(3):
        for m, s, r in zip(models, streams, runoff):
            with torch.cuda.stream(s):
                m.set_inputs(r[d])
                m.step_advance()
    torch.cuda.synchronize()
    for m, a in zip(models, alone):
        m.check_status()
        for k, v in m.state_tensors().items():
            np.testing.assert_array_equal(v.cpu().numpy(), a[k], err_msg=k)
