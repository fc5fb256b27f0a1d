"""An interval inside a stream capture is refused, as CUDA refuses a graph with
a conditional node there, without spoiling the capture or the plan."""
import numpy as np
import pytest
import torch

from cmfb200 import _lib, synthetic as syn

import parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [True, False])
@pytest.mark.parametrize("form", [dict(), dict(resident=False), dict(num_members=2)])
def test_captured_interval_is_refused(form, warm, device):
    net = P.make_network("full", n=3000)
    m, ref = P.model_for(net, **form), P.model_for(net, **form)
    if warm:
        m.step_advance()
        ref.step_advance()
    x = torch.zeros(4, device=device)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1)
        rc = _lib.lib().cmf_step_interval(m._plan, m._stream(), 3600.0, 0)
        x.add_(1)
    assert rc == _lib.CMF_ERR_UNSUPPORTED
    g.replay()
    m.step_advance()
    ref.step_advance()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 4
    m.check_status()
    for k, v in ref.state_tensors().items():
        np.testing.assert_array_equal(m.state_tensors()[k].cpu().numpy(), v.cpu().numpy(), err_msg=k)
