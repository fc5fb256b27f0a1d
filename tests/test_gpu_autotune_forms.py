"""The autotuner says whether step_advance uses what it picked."""
import pytest

import parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("resident", [True, False])
def test_autotune_says_whether_its_choice_is_used(resident, device, tmp_path):
    m = P.model_for(P.make_network("plain", n=5000), resident=resident)
    cache = str(tmp_path / "tune.json")
    for cached in (False, True):
        res = m.autotune_block_size(candidates=(64, 256), sub_steps=2, cache_path=cache)
        assert res["cached"] == cached
        assert res["used_by_step_advance"] == (not resident)
        assert (m.resident_tiles > 0) == resident
