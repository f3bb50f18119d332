"""The three routes to the dual grid of a reconstruction -- rank bitmap, two-level rank bitmap, sorted corner keys -- each
forced, seen to run, and giving the same dual grid and mesh; the two for deep scenes against the FP64 oracle as well;
and the boxes that are refused."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
ROUTES = {"bitmap": (1 << 27, 1 << 27), "two_level": (0, 1 << 27), "sorted_keys": (0, 0)}


@pytest.fixture
def taken(monkeypatch):
    """The routes that ran, in order ("bitmap" leaves no entry)."""
    from jspsr.core.pipeline import DualMesher
    out = []
    for name, route in (("_dual_cubes_two_level", "two_level"), ("_dual_centres_by_sort", "sorted_keys")):
        def run(self, *a, _f=getattr(DualMesher, name), _route=route):
            out.append(_route)
            return _f(self, *a)
        monkeypatch.setattr(DualMesher, name, run)
    return out


@pytest.mark.parametrize("name", ["torus_adaptive", "sq_noisy"])
def test_routes_agree(golden, name, taken):
    from jspsr.core.pipeline import Reconstruction
    g = golden(name)
    vs, depth, md, alpha = g["params"]
    rec = Reconstruction(torch.from_numpy(g["xyz"]).cuda(), torch.from_numpy(g["nrm"]).cuda(), vs, int(depth), md, alpha,
                         solver="pcg-mixed@tol=1e-9")
    rec.build_tree().assemble().solve()
    out = []
    for route, (plain, two) in ROUTES.items():
        rec.dual_grid_max_words, rec.dual_grid2_max_words = plain, two
        v, f = rec.extract_mesh()
        assert taken == ([] if route == "bitmap" else [route])
        taken.clear()
        out.append((rec.dual_cubes().cpu().numpy(), v.cpu().numpy(), f.cpu().numpy()))
    for other in out[1:]:
        assert np.array_equal(out[0][0], other[0]) and np.array_equal(out[0][2], other[2])
        assert np.abs(out[0][1] - other[1]).max() <= 1e-5


@pytest.mark.parametrize("route", ["two_level", "sorted_keys"])
def test_deep_hierarchy_against_the_oracle(route, taken, monkeypatch):
    """A room scene at 2 cm with 7 levels: coarse cells of 64 voxels in the dual grid."""
    from jspsr import synthetic
    from jspsr.core.pipeline import DualMesher
    from test_gpu_timed_config import check_parity, run_both
    plain, two = ROUTES[route]
    monkeypatch.setattr(DualMesher, "dual_grid2_max_words", two)
    xyz, nrm = synthetic.room(n=200_000, seed=0, n_objects=12)
    ref, rec, v, f = run_both(xyz, nrm, 0.02, 7, 2.0, 4.0, "pcg-mixed@tol=1e-7", dual_grid_max_words=plain)
    assert taken == [route]
    check_parity(ref, rec, v, f, 7, {})


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("two", [0, 1 << 27])
def test_boxes_of_2_21_cells_an_axis_are_refused(axis, two):
    """Where a plain bitmap does not hold the box."""
    from jspsr.core.pipeline import DualMesher
    m = DualMesher()
    m.levels = [SimpleNamespace(stride=1)]
    m.vs, m.dev, m.dual_grid_max_words, m.dual_grid2_max_words = 1.0, DEV, 0, two
    cells = torch.zeros(2, 3, dtype=torch.int32, device=DEV)
    cells[1, axis] = 1 << 20
    with pytest.raises(ValueError, match="2\\^21"):
        m.mesh_from_leaves({0: cells}, 1, 2, lambda p: torch.sin(p.sum(1)))


@pytest.mark.parametrize("cells,apart,route", [(500, 4200, "sorted_keys"), (500, 3000, "two_level"), (60000, 4200, "two_level")])
def test_route_follows_the_cells_in_the_box(cells, apart, route, taken):
    """Two clusters of cells far apart: an outer grid of 18 or 9 million words, for few cells or for many."""
    from jspsr.core.pipeline import DualMesher
    g = torch.Generator(device=DEV).manual_seed(cells)
    c = torch.unique(torch.randint(0, 60, (cells, 3), generator=g, device=DEV), dim=0)
    c = torch.unique(torch.cat([c, c + apart // 2]), dim=0).int()
    out = []
    for two in (1 << 27, 0):
        m = DualMesher()
        m.levels = [SimpleNamespace(stride=1)]
        m.vs, m.dev, m.dual_grid_max_words, m.dual_grid2_max_words = 1.0 / 64, DEV, 0, two
        v, f = m.mesh_from_leaves({0: c}, 1, 2, lambda p: torch.sin(97.0 * p.sum(1) + 1.0))
        out.append((m.mesh_info["cnt"], m.mesh_info["acc_ids"], f, v))
    assert taken == [route, "sorted_keys"]
    for a, b in zip(*out):
        assert torch.equal(a, b)
