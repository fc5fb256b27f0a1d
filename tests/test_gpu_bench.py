"""The small-configuration leg of bench.py times the forms of an interval that
it names, and their end states agree."""
import pytest

import bench as B

pytestmark = pytest.mark.gpu


def test_small_network_leg_names_the_forms_it_runs(device):
    out = B.small_network_measure(device, "plain_60k", 1)
    for mode in ("resident", "graph", "persistent"):
        assert out[mode]["sub_steps"] == out["graph"]["sub_steps"] > 0
        assert out[mode]["us_per_substep"] > 0
    for mode in ("resident", "persistent"):
        assert out[f"{mode}_state_equal"]
        assert out[f"{mode}_over_graph"] == out[mode]["value"] / out["graph"]["value"]
