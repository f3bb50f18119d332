"""Which form of a level's matrix the solver reads: packed from 40 entries a row on (mixed mode: from 8,192 rows on),
the CSR for shorter rows and for the reference mode, with 2-byte column deltas where the vector is staged in shared
memory.  Either way the solutions agree."""
import pytest
import torch

from jspsr import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["pcg-mixed@tol=1e-10", "pcg-fp64@tol=1e-10", "pcg@tol=1e-6"])
@pytest.mark.parametrize("n,voxel", [(2000, 1 / 512), (20000, 1 / 512), (20000, 1 / 128)])
def test_form_follows_the_rows(solver, n, voxel):
    from jspsr import synthetic
    from jspsr.core.pipeline import Reconstruction
    xyz, nrm = synthetic.torus(n=n)
    xyz, nrm = torch.from_numpy(xyz).cuda(), torch.from_numpy(nrm).cuda()
    rec = Reconstruction(xyz, nrm, voxel, 4, None, solver=solver).build_tree().assemble().solve()
    rec.check_solves()
    plain = Reconstruction(xyz, nrm, voxel, 4, None, solver="plain-fp64@tol=1e-10").build_tree().assemble().solve()
    kinds = set()
    for lv, ref in zip(rec.levels, plain.levels):
        if lv.n == 0:
            continue
        packed = (solver != "pcg@tol=1e-6" and lv.nnz >= 40 * lv.n and (solver.startswith("pcg-fp64") or lv.n >= 8192))
        window = L.load().ngs_pcg_window(lv.n, lv.nnz, lv.band, rec.solver.mode) == 1
        assert (lv.pk_vals is not None) == packed
        assert (lv.col_delta is not None) == (not packed and window and lv.band <= 32767)
        kinds.add((packed, lv.col_delta is not None))
        # tolerance of the solves times a bound of the levels' condition (1e3; CG needs some 60 iterations for 1e-10)
        tol = 1e3 * (1e-6 if solver.startswith("pcg@") else 1e-10) + 1e-6
        assert float((lv.x64 - ref.x64).norm() / ref.x64.norm()) <= tol
    assert kinds
