"""The interval graph of one member, which serves the networks that do not fit
the SMs' shared memory, at sizes where the resident kernel would be taken: with
that kernel turned off, the state, the diagnostics and the statistics are the
bits of the sub-step kernels launched one by one and of the other forms of an
interval, in every feature case, with adaptive and fixed sub-step counts and
intervals of several lengths, which change the nodes of an instantiated graph."""
import numpy as np
import pytest
import torch

from cmfb200 import _lib, synthetic as syn

import parity as P

pytestmark = pytest.mark.gpu

DIAGNOSTICS = ("river_inflow", "flood_inflow", "total_storage", "water_surface_elevation",
               "protected_water_surface_elevation", "time_step", "outer_time_step", "current_step")
SAVED = {"mean": ["total_outflow", "flood_fraction", "river_storage"], "max": ["river_depth", "flood_storage"],
         "min": ["river_storage"], "last": ["flood_depth"]}
# (interval in seconds, fixed sub-steps or None): node parameters, and the
# graph rebuilt where the CFL comes or goes; counts odd and even
PLAN = ((86400.0, None), (86400.0, None), (3600.0, None), (3600.0, 7), (3600.0, 8), (7200.0, 8), (86400.0, None))


def _model(net, form, **kw):
    m = P.model_for(net, use_cuda_graph=form != "direct", resident=form == "resident",
                    persistent=form == "persistent", **kw)
    assert (m.resident_tiles > 0) == (form == "resident")
    return m


def _run(net, form, plan=PLAN, **kw):
    m = _model(net, form, **kw)
    counts = []
    for d, (seconds, fixed) in enumerate(plan):
        m.step_seconds = seconds
        m.set_inputs(torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda())
        m.step_advance(num_sub_steps=fixed)
        counts.append(int(m.sub_step_counts()[0].item()))
    torch.cuda.synchronize()
    m.check_status()
    out = dict(m.state_tensors())
    out.update({k: getattr(m.base, k) for k in DIAGNOSTICS if getattr(m.base, k) is not None})
    if m.bifurcation is not None:
        out.update(limit_rate=m.bifurcation.limit_rate, net=m.bifurcation.global_bifurcation_outflow)
    if m.variables_to_save:
        out.update(m.collect_statistics())
    return {k: v.cpu().numpy() for k, v in out.items()}, counts


def _same(a, b):
    assert a[1] == b[1]
    assert a[0].keys() == b[0].keys()
    for k in a[0]:
        np.testing.assert_array_equal(a[0][k], b[0][k], err_msg=k)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("case", list(P.CASES))
def test_graph_equals_direct_launches(case, precision, device):
    net = P.make_network(case)
    _same(_run(net, "graph", precision=precision), _run(net, "direct", precision=precision))


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("form", ["persistent", "resident"])
def test_graph_equals_the_other_forms(form, precision, device):
    net = P.make_network("full", n=20_000, seed=8)
    _same(_run(net, "graph", precision=precision), _run(net, form, precision=precision))


@pytest.mark.parametrize("block", [64, 256])
def test_graph_on_a_large_network(block, device):
    net = P.make_network("full", n=200_000, seed=8)
    plan = ((86400.0, None), (3600.0, 5))
    _same(_run(net, "graph", plan=plan, BLOCK_SIZE=block), _run(net, "direct", plan=plan, BLOCK_SIZE=block))


@pytest.mark.parametrize("case, precision", [("plain", "float32"), ("full", "float32"), ("full", "float64")])
def test_graph_statistics(case, precision, device):
    net = P.make_network(case, n=9001)
    _same(_run(net, "graph", precision=precision, variables_to_save=SAVED),
          _run(net, "direct", precision=precision, variables_to_save=SAVED))


def test_graph_sub_step_cap(device):
    m = _model(P.make_network("plain"), "graph", max_sub_steps_cap=3)
    m.step_advance()
    assert int(m.sub_step_counts()[0].item()) == 3
    with pytest.raises(RuntimeError):
        m.check_status()


def test_forms_change_between_intervals(device):
    """One model that goes through the forms in turn, a statistic attached
    where the form takes one, equals one that stays with the direct launches."""
    net = P.make_network("full", n=9001, seed=4)
    ref, mix = _model(net, "direct"), P.model_for(net)
    for d, (resident, persistent, saved) in enumerate(
            [(True, False, None), (False, False, None), (False, False, SAVED), (True, False, SAVED),
             (True, True, None), (False, False, None), (True, False, None), (False, True, None)]):
        mix.set_persistent(False)
        mix.set_variables_to_save(saved)
        mix.set_persistent(persistent)
        mix.set_resident(resident)
        assert (mix.resident_tiles > 0) == (resident and not persistent)
        r = torch.as_tensor(ref.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda()
        for m in (ref, mix):
            m.set_inputs(r)
            m.step_advance(num_sub_steps=9 + d if d % 3 == 2 else None)
        if d == 5:
            mix._rebuild_plan(128)      # the choice outlives the plan
            assert mix.resident_tiles == 0
    torch.cuda.synchronize()
    mix.check_status()
    for k, v in ref.state_tensors().items():
        np.testing.assert_array_equal(mix.state_tensors()[k].cpu().numpy(), v.cpu().numpy(), err_msg=k)


def test_switch_refuses_a_null_plan(device):
    assert _lib.lib().cmf_plan_set_resident(None, 0) == _lib.CMF_ERR_ARG
