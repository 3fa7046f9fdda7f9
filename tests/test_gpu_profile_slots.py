"""The profiler's phases: each launch of a solve is counted once, and every
phase of the sort, the iterations and the final energy is named; without
correspondences the node set-up stands alone."""
import pytest
import torch

from cudafusion_b200 import synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("corrs", [0, 2000])
def test_phases(corrs):
    p = synth.sphere_problem(num_nodes=64, num_corrs=2000, node_radius=0.13, seed=1)
    p.corrs, p.canon = p.corrs[:corrs], p.canon[:corrs]
    s = GaussNewtonSolver(Params(gn_iterations=2, pcg_iterations=3, lambda_damping=1.0), max_nodes=64, max_corrs=2000)
    dp = DeviceProblem(p)
    s.profile_enable(True)
    n0 = s.launch_count()
    s.gn_solve(dp, dp.init_transforms.clone())
    torch.cuda.synchronize()
    ph = s.profile_read()
    assert sum(n for _, n in ph.values()) == s.launch_count() - n0
    assert {k: ph[k][1] for k in ("residual", "assemble", "pcg")} == {"residual": 2, "assemble": 2, "pcg": 2}
    sort = {"key_count", "bin_scan", "bin_scatter", "bucket_sort", "node_lists"}
    assert set(ph) == {"residual", "assemble", "pcg", "final_energy"} | (sort if corrs else {"node_plain"})
