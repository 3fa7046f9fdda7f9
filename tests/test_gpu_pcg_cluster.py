"""The single-cluster PCG at the sizes where its layout changes: one row per
CTA, 8 CTAs, a ragged last CTA, the last size of four and of two lanes per row
element and the first past each, and the largest of five rows per warp; the
solve against the FP64 oracle within the bar of the other solves (1e-5 per
transform component, or 1.5 times what FP32 in the reference's order is off)."""
import numpy as np
import pytest
import torch

from cudafusion_b200 import _lib, synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params
from cudafusion_b200.types import DQ_DTYPE, dq_as_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [9, 16, 17, 31, 250, 384, 400, 768, 800, 1600])
def test_sizes_match_the_oracle(oracle, nodes):
    kw = dict(gn_iterations=2, pcg_iterations=9, pcg_tolerance=0.0, lambda_smooth=10.0, lambda_damping=1.0)
    p = synth.sphere_problem(num_nodes=nodes, num_corrs=40 * nodes + 7, node_radius=0.3 * (12.6 / nodes) ** 0.5, seed=nodes)
    s = GaussNewtonSolver(Params(**kw), max_nodes=nodes, max_corrs=p.num_corrs)
    s.set_option(_lib.CF_OPT_PCG_MODE, 2)
    dp = DeviceProblem(p)
    T = dp.init_transforms.clone()
    st = s.gn_solve(dp, T, max_rot=0.12, max_trans=0.04)
    torch.cuda.synchronize()
    assert st["error_flags"] == 0 and s.get_option(_lib.CF_OPT_PCG_ACTIVE) == 2
    prm = oracle.params(**kw)
    T64, E64, _ = oracle.gn_solve(p, prm, 0.12, 0.04, precision="f64")
    T32, _, _ = oracle.gn_solve(p, prm, 0.12, 0.04, precision="f32")
    spread = float(np.abs(dq_as_array(T64) - dq_as_array(T32)).max())
    err = float(np.abs(dq_as_array(T.cpu().numpy().view(DQ_DTYPE)) - dq_as_array(T64)).max())
    assert err < max(1e-5, 1.5 * spread), (err, spread)
    assert abs(st["energy_final"] - E64[-1]) / E64[-1] < 1e-4
