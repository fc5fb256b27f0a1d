"""The waits of the resident interval kernel are bounded: a tile that leaves in
the middle of an interval (and posts nothing more) makes those that need its
values give up after their polls, report it in the status word and leave; the
kernel returns, the context stays usable, and the plan runs on from a restored
state."""
import time

import numpy as np
import pytest
import torch

from cmfb200 import _lib, synthetic as syn

import parity as P

pytestmark = pytest.mark.gpu

POLLS = 20_000      # some 10 ms
SUB_STEPS = 8
INTERVAL = 3600.0


def _model(case, precision):
    net = P.make_network(case, n=20_000)
    m = P.model_for(net, precision=precision)
    m.set_inputs(torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, 0))).cuda())
    # the last tile's cells flow into cells of other tiles, which therefore wait for it
    first = (m.resident_tiles - 1) * 160
    assert m.resident_tiles == 125 and bool((m.base.downstream_idx[first:] < first).any())
    return net, m


def _give_up(m, leave):
    lib = _lib.lib()
    t0 = time.perf_counter()
    rc = lib.cmf_probe_resident_timeout(m._plan, m._stream(), INTERVAL, SUB_STEPS, leave, POLLS)
    assert rc == _lib.CMF_OK
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 10.0
    assert m.status() & _lib.STATUS_SYNC_TIMEOUT
    with pytest.raises(RuntimeError):
        m.check_status()


@pytest.mark.parametrize("leave", [0, 3, SUB_STEPS - 1])
@pytest.mark.parametrize("case, precision", [("plain", "float32"), ("full", "float32"), ("full", "float64")])
def test_resident_wait_gives_up_and_reports(case, precision, leave, device):
    _, m = _model(case, precision)
    _give_up(m, leave)
    x = torch.arange(100, device=device, dtype=torch.float32)
    assert float(x.sum().item()) == 4950.0


@pytest.mark.parametrize("case, precision", [("plain", "float32"), ("full", "float32"), ("full", "float64")])
def test_resident_plan_runs_on_after_a_give_up(case, precision, device):
    """The words that the abandoned interval left are not taken for the next
    one's: with the state restored, the plan equals one that never failed."""
    net, m = _model(case, precision)
    ref = _model(case, precision)[1]
    before = {k: v.clone() for k, v in m.state_tensors().items()}
    for leave in (0, 1, SUB_STEPS - 1):
        _give_up(m, leave)
        for k, v in m.state_tensors().items():
            v.copy_(before[k])
        m._status.zero_()
    for d in range(2):
        for x in (m, ref):
            x.set_inputs(torch.as_tensor(x.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda())
            x.step_advance()
    torch.cuda.synchronize()
    m.check_status()
    for k, v in ref.state_tensors().items():
        np.testing.assert_array_equal(m.state_tensors()[k].cpu().numpy(), v.cpu().numpy(), err_msg=k)


def test_resident_probe_refuses_what_it_does_not_run(device):
    lib = _lib.lib()
    _, m = _model("plain", "float32")
    for sub_steps, leave, polls in ((0, 0, 100), (4, 4, 100), (4, -1, 100), (4, 0, 0), (4, 0, (1 << 22) + 1)):
        rc = lib.cmf_probe_resident_timeout(m._plan, m._stream(), INTERVAL, sub_steps, leave, polls)
        assert rc == _lib.CMF_ERR_ARG
    assert lib.cmf_probe_resident_timeout(None, None, INTERVAL, 4, 0, 100) == _lib.CMF_ERR_ARG
    direct = P.model_for(P.make_network("plain", n=2000), use_cuda_graph=False)
    rc = lib.cmf_probe_resident_timeout(direct._plan, direct._stream(), INTERVAL, 4, 0, 100)
    assert rc == _lib.CMF_ERR_UNSUPPORTED
