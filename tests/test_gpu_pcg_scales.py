"""The grid-wide PCG's exchanged sums where they change by many binary orders
from one iteration to the next, so that they do not fit the words they are
exchanged in and are taken from the stored partials: a system without coupling
(the first step leaves rounding errors of the right-hand side, r.r falls by
2^40 and more) and one whose nodes' weights differ by 10^3 (||r|| rises and falls
by 2^8 in turn: 2^17 in r.r).  The residual against that of the single cluster,
whose sums are FP64 throughout, and the solve against the FP64 oracle within the
bar of the other solves."""
import numpy as np
import pytest
import torch

from cudafusion_b200 import _lib, synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params
from cudafusion_b200.types import DQ_DTYPE, dq_as_array

pytestmark = pytest.mark.gpu

N = 300


def problem(kind):
    p = synth.sphere_problem(num_nodes=N, num_corrs=12000, node_radius=0.3 * (12.6 / N) ** 0.5, seed=3)
    c = p.corrs
    ids = c["node_ids"].copy()
    c["node_ids"] = -1
    c["node_ws"] = 0
    if kind == "uncoupled":
        # points all around their node, with normals in all directions: blocks near multiples of the identity
        rng = np.random.default_rng(5)
        d, n = rng.normal(size=(2, len(ids), 3))
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        c["node_ids"][:, 0] = ids[:, 0]
        c["node_ws"][:, 0] = 1
        p.canon[:] = c["src"] = p.nodes["pos"][ids[:, 0]] + d
        c["normal"] = n
        c["dst"] = c["src"] + 0.1 * rng.normal(size=(len(ids), 1)) * n
        return p
    # light nodes have the residuals alone, and share quiet correspondences with heavy ones
    light = ids % 2 == 1
    rows = np.arange(len(ids))
    c["valid"] = light.any(1) & ~light.all(1)
    c["node_ids"][:, 0] = ids[rows, light.argmax(1)]
    c["node_ws"][:, 0] = 1e-3
    pair = rows % 2 == 1
    c["node_ids"][pair, 1] = ids[rows, (~light).argmax(1)][pair]
    c["node_ws"][pair, 1] = 1
    c["dst"][pair] = c["src"][pair]
    return p


def solve(p, kw, mode, ctas=0):
    s = GaussNewtonSolver(Params(**kw), max_nodes=N, max_corrs=p.num_corrs)
    s.set_option(_lib.CF_OPT_PCG_MODE, mode)
    s.set_option(_lib.CF_OPT_PCG_CTAS, ctas)
    dp = DeviceProblem(p)
    T = dp.init_transforms.clone()
    st = s.gn_solve(dp, T, max_rot=0.12, max_trans=0.04)
    torch.cuda.synchronize()
    assert st["error_flags"] == 0
    return st, dq_as_array(T.cpu().numpy().view(DQ_DTYPE))


@pytest.mark.parametrize("ctas", [1, 37, 0])
def test_residual_far_below_the_one_before(ctas):
    p = problem("uncoupled")
    kw = dict(gn_iterations=1, pcg_iterations=1, pcg_tolerance=0.0, lambda_smooth=1e-9, lambda_damping=1e-6)
    got, want = solve(p, kw, 1, ctas)[0]["pcg_residual"][0], solve(p, kw, 2)[0]["pcg_residual"][0]
    # the same FP32 residuals, summed in FP64 in another order
    assert want > 0 and abs(got - want) < 1e-9 * want


@pytest.mark.parametrize("kind", ["uncoupled", "uneven"])
@pytest.mark.parametrize("ctas", [1, 37, 0])
def test_solve_matches_the_oracle(oracle, kind, ctas):
    p = problem(kind)
    kw = dict(gn_iterations=2, pcg_iterations=6, pcg_tolerance=0.0, lambda_smooth=1e-9, lambda_damping=1e-6)
    st, T = solve(p, kw, 1, ctas)
    prm = oracle.params(**kw)
    T64, E64, _ = oracle.gn_solve(p, prm, 0.12, 0.04, precision="f64")
    T32, _, _ = oracle.gn_solve(p, prm, 0.12, 0.04, precision="f32")
    spread = float(np.abs(dq_as_array(T32) - dq_as_array(T64)).max())
    err = float(np.abs(T - dq_as_array(T64)).max())
    assert err < max(1e-5, 1.5 * spread), (err, spread)
