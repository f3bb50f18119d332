"""A reconstruction assembled for one solver and solved with another: the packed matrix of a mode is read by no other
mode, and the solutions are those of a reconstruction assembled for the second solver."""
import pytest
import torch

pytestmark = pytest.mark.gpu
SPECS = ["pcg-mixed@tol=1e-10", "pcg-fp64@tol=1e-10", "pcg@tol=1e-6", "plain-fp64@tol=1e-10"]


@pytest.mark.parametrize("first", SPECS)
@pytest.mark.parametrize("then", SPECS)
def test_solver_changed_after_assembly(first, then):
    from jspsr import synthetic
    from jspsr.core.pipeline import Reconstruction, parse_solver
    xyz, nrm = synthetic.torus(n=20000)
    xyz, nrm = torch.from_numpy(xyz).cuda(), torch.from_numpy(nrm).cuda()

    def assembled(spec):
        return Reconstruction(xyz, nrm, 1 / 128, 3, 4.0, 4.0, solver=spec).build_tree().assemble()
    rec, want = assembled(first), assembled(then).solve()
    rec.solver = parse_solver(then)
    rec.solve()
    rec.check_solves()
    # both solve the same system to the solver's tolerance: FP64 forms to 1e-10 of the right-hand side, the FP32
    # reference form to 1e-6 (coarse levels' errors reach the finer ones' right-hand sides), times the condition of a
    # level's matrix (1e3 bounds it: CG needs some 60 iterations for 1e-10)
    tol = 1e3 * (1e-6 if then.startswith("pcg@") else 1e-10) + 1e-6
    for a, b in zip(rec.levels, want.levels):
        assert float((a.x64 - b.x64).norm() / b.x64.norm()) <= tol
