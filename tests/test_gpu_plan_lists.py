"""Lists of a view in a form that the resident interval kernel cannot index by:
a levee list that is not ascending, a levee cell that no levee lists, a path end
in a cell that is not flagged for bifurcation, a mouth whose downstream index is not
its own.  The plan leaves such a view to the interval graph, whose results are
those of the same view with the sub-step kernels launched one by one; it does the
same where a cell or a tile has more path ends than the resident kernel is fast
with.  Flag bits that the library does not define change nothing."""
import numpy as np
import pytest
import torch

from cmfb200 import _lib, synthetic as syn

import parity as P

pytestmark = pytest.mark.gpu


def _run(m, net, days=2):
    for d in range(days):
        m.set_inputs(torch.as_tensor(m.to_model_order(20.0 * syn.daily_runoff(net, d))).cuda())
        m.step_advance()
    torch.cuda.synchronize()
    m.check_status()
    return {k: v.cpu().numpy() for k, v in m.state_tensors().items()}


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def _shuffled_levees(m):
    """The same levees listed in another order."""
    lm = m.levee
    perm = torch.randperm(lm.num_levees, generator=torch.Generator().manual_seed(4)).to(m.device)
    for k in ("levee_catchment_idx", "levee_crown_height", "levee_fraction", "levee_base_height"):
        getattr(lm, k).copy_(getattr(lm, k)[perm])
    m.base.levee_slot[lm.levee_catchment_idx.long()] = torch.arange(lm.num_levees, dtype=torch.int32,
                                                                    device=m.device)


def _unlisted_levee(m):
    """The last levee taken off the list, its cell still flagged."""
    m.base.levee_slot[m.levee.levee_catchment_idx[-1].long()] = -1
    m.levee.num_levees -= 1


def _unflagged_path_ends(m):
    cells = m.bifurcation.bifurcation_downstream_idx[:20].long()
    m.base.cell_flags[cells] &= 255 - _lib.CELL_BIFURCATION


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_levees_in_any_order(precision, device):
    net = P.make_network("full", n=9001)
    plain = P.model_for(net, precision=precision)
    assert plain.resident_tiles > 0
    mixed = P.model_for(net, precision=precision)
    _shuffled_levees(mixed)
    mixed._rebuild_plan(mixed.block_size)
    assert mixed.resident_tiles == 0
    _same(_run(plain, net), _run(mixed, net))


def _mouths_into_another_cell(m):
    """The downstream index of a mouth, which its flag keeps from being used."""
    mouths = (m.base.cell_flags & _lib.CELL_MOUTH) != 0
    m.base.downstream_idx[mouths] = 7


def _foreign_upstream_cell(m):
    """A leaf's upstream range made to hold a cell of another one."""
    up = m.base.upstream_ptr
    last = int(up.numel()) - 2
    up[last] = last - 1
    up[last + 1] = last


@pytest.mark.parametrize("change", [_unlisted_levee, _unflagged_path_ends, _mouths_into_another_cell])
def test_lists_that_disagree_with_the_flags(change, device):
    net = P.make_network("full", n=5000)
    runs = []
    for graph in (True, False):
        m = P.model_for(net, use_cuda_graph=graph)
        change(m)
        m._rebuild_plan(m.block_size)
        assert m.resident_tiles == 0
        runs.append(_run(m, net))
    _same(*runs)


def test_upstream_range_with_a_foreign_cell(device):
    """The plan only: the sub-step kernels would add that cell's flow twice."""
    m = P.model_for(P.make_network("plain", n=5000))
    assert m.resident_tiles > 0
    _foreign_upstream_cell(m)
    m._rebuild_plan(m.block_size)
    assert m.resident_tiles == 0


def test_undefined_flag_bits_are_ignored(device):
    net = P.make_network("full", n=5000)
    plain, marked = P.model_for(net), P.model_for(net)
    marked.base.cell_flags |= 192
    marked._rebuild_plan(marked.block_size)
    assert marked.resident_tiles > 0
    _same(_run(plain, net), _run(marked, net))


def _paths(n, count, hub_ends, seed=5):
    """`count` paths between random cells, `hub_ends` of them into the last cell."""
    net = syn.generate(syn.NetworkSpec(n, seed=1, bifurcation_paths=count, levee_fraction=0.2))
    rng = np.random.default_rng(seed)
    net.fields["bifurcation_catchment_id"] = rng.integers(0, n - 1, size=count)
    to = rng.integers(0, n - 1, size=count)
    to[:hub_ends] = n - 1
    net.fields["bifurcation_downstream_id"] = to
    return net


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("n, count, hub_ends, resident", [
    (6000, 400, 48, True), (6000, 400, 49, False),         # the most path ends of a cell
    (2500, 8000, 0, True), (2500, 12_000, 0, False)])      # 819 and 1,229 in a tile
def test_cells_and_tiles_with_many_path_ends(n, count, hub_ends, resident, precision, device):
    net = _paths(n, count, hub_ends)
    runs = []
    for graph in (True, False):
        m = P.model_for(net, precision=precision, use_cuda_graph=graph)
        assert (m.resident_tiles > 0) == (graph and resident)
        runs.append(_run(m, net, days=1))
    _same(*runs)


def test_path_in_the_wrong_cells_list(device):
    """Two cells' lists exchanged: the resident kernel takes one end's cell from the list
    and the other's from the path."""
    net = P.make_network("bif", n=5000)
    runs = []
    for graph in (True, False):
        m = P.model_for(net, use_cuda_graph=graph)
        b = m.bifurcation
        n_ends = (b.bif_cell_ptr[1:] - b.bif_cell_ptr[:-1]).cpu().numpy()
        i, j = np.flatnonzero(n_ends == 1)[[3, 40]]
        x, y = int(b.bif_cell_ptr[i]), int(b.bif_cell_ptr[j])
        b.bif_cell_paths[[x, y]] = b.bif_cell_paths[[y, x]]
        m._rebuild_plan(m.block_size)
        assert m.resident_tiles == 0
        runs.append(_run(m, net, days=1))
    _same(*runs)
