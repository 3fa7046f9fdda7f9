"""The grid-wide PCG's exchanged sums: one CTA, two, an odd number and all of
them, several problems with their own CTA groups, and a right-hand side of
zeros (no scale for the sums: they are exchanged as stored partials); against
the FP64 oracle within the bar of the other solves (1e-5 per transform component,
or 1.5 times what FP32 in the reference's order is off)."""
import numpy as np
import pytest
import torch

from cudafusion_b200 import _lib, synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params
from cudafusion_b200.types import DQ_DTYPE, dq_as_array

pytestmark = pytest.mark.gpu

KW = dict(gn_iterations=2, pcg_iterations=9, pcg_tolerance=0.0, lambda_smooth=10.0, lambda_damping=1.0)


def check(oracle, p, T):
    prm = oracle.params(**KW)
    T64, _, _ = oracle.gn_solve(p, prm, 0.12, 0.04, precision="f64")
    T32, _, _ = oracle.gn_solve(p, prm, 0.12, 0.04, precision="f32")
    spread = float(np.abs(dq_as_array(T64) - dq_as_array(T32)).max())
    err = float(np.abs(dq_as_array(T.cpu().numpy().view(DQ_DTYPE)) - dq_as_array(T64)).max())
    assert err < max(1e-5, 1.5 * spread), (err, spread)


def problem(nodes):
    return synth.sphere_problem(num_nodes=nodes, num_corrs=40 * nodes, node_radius=0.3 * (12.6 / nodes) ** 0.5, seed=nodes)


@pytest.mark.parametrize("ctas", [1, 2, 37, 0])
def test_cta_counts(oracle, ctas):
    p = problem(300)
    s = GaussNewtonSolver(Params(**KW), max_nodes=300, max_corrs=p.num_corrs)
    s.set_option(_lib.CF_OPT_PCG_MODE, 1)
    s.set_option(_lib.CF_OPT_PCG_CTAS, ctas)
    dp = DeviceProblem(p)
    T = dp.init_transforms.clone()
    st = s.gn_solve(dp, T, max_rot=0.12, max_trans=0.04)
    torch.cuda.synchronize()
    assert st["error_flags"] == 0
    check(oracle, p, T)


def test_groups(oracle):
    ps = [problem(n) for n in (20, 90, 41)]
    s = GaussNewtonSolver(Params(**KW), max_nodes=151, max_corrs=sum(p.num_corrs for p in ps))
    s.set_option(_lib.CF_OPT_PCG_MODE, 1)
    dps = [DeviceProblem(p) for p in ps]
    Ts = [d.init_transforms.clone() for d in dps]
    s.gn_solve_batched(dps, Ts, max_rot=0.12, max_trans=0.04)
    torch.cuda.synchronize()
    for p, T in zip(ps, Ts):
        check(oracle, p, T)


def test_zero_right_hand_side():
    p = problem(300)
    p.corrs["dst"] = p.corrs["src"]
    s = GaussNewtonSolver(Params(**KW), max_nodes=300, max_corrs=p.num_corrs)
    s.set_option(_lib.CF_OPT_PCG_MODE, 1)
    dp = DeviceProblem(p)
    T = dp.init_transforms.clone()
    st = s.gn_solve(dp, T, max_rot=0.12, max_trans=0.04)
    torch.cuda.synchronize()
    assert st["error_flags"] == 0
    a = dq_as_array(T.cpu().numpy().view(DQ_DTYPE))
    assert np.abs(a - dq_as_array(p.init_transforms)).max() < 1e-6
