"""Plans made while their tensors are still on their way: a model built, and
rebuilt, on a side stream with work queued ahead of its uploads, in memory that
holds other bits, and stepped at once, equals a model built on an idle device; and a plan made with another device
current than its tensors'."""
import numpy as np
import pytest
import torch

from cmfb200 import CaMaFlood, synthetic as syn

import parity as P

pytestmark = pytest.mark.gpu

BUSY_CYCLES = 40_000_000  # some 20 ms of a stream


def _dirty_pool(mib=64):
    """Memory that the stream's next allocations come from, with every bit pattern non-zero."""
    for _ in range(4):
        torch.full((mib << 20,), 0x7F, dtype=torch.uint8, device="cuda")


def _steps(m, net, days):
    for d in days:
        m.set_inputs(torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda())
        m.step_advance()


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("case", ["plain", "bif", "full"])
def test_plan_made_behind_queued_work(case, graph, device):
    net = P.make_network(case, n=9001)
    ref = P.model_for(net, use_cuda_graph=graph)
    _steps(ref, net, range(3))
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        _dirty_pool()
        torch.cuda._sleep(BUSY_CYCLES)
        m = P.model_for(net, use_cuda_graph=graph)
        _steps(m, net, [0])
        _dirty_pool()
        torch.cuda._sleep(BUSY_CYCLES)
        m._rebuild_plan(128)
        _steps(m, net, [1, 2])
    torch.cuda.synchronize()
    assert m.resident_tiles == ref.resident_tiles
    m.check_status()
    for k, v in ref.state_tensors().items():
        np.testing.assert_array_equal(m.state_tensors()[k].cpu().numpy(), v.cpu().numpy(), err_msg=k)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")
@pytest.mark.parametrize("case", ["plain", "full"])
def test_plan_made_with_another_device_current(case, device):
    """The plan's own work runs on the device of its tensors, and the caller's
    current device is what it was."""
    net = P.make_network(case, n=5000)
    ref = P.model_for(net)
    _steps(ref, net, range(2))
    m = CaMaFlood(device="cuda:1", input_proxy=net.fields, opened_modules=net.opened_modules)
    assert torch.cuda.current_device() == 0
    with torch.cuda.device(1):
        assert m.resident_tiles == ref.resident_tiles
        for d in range(2):
            m.set_inputs(torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, d))))
            m.step_advance()
        m.check_status()
    for k, v in ref.state_tensors().items():
        np.testing.assert_array_equal(m.state_tensors()[k].cpu().numpy(), v.cpu().numpy(), err_msg=k)
