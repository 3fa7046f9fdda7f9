"""Failure detection of the single-cluster PCG without a GPU fault: exchanges
that also wait for a message nobody sends give up after their (short) poll
limit; the solve reports CF_ERR_TIMEOUT, and the next one on the same handle is
exact.  16 CTAs, 8, and the three lane layouts."""
import pytest
import torch

from cudafusion_b200 import _lib, synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [9, 300, 600, 1200])
def test_timeout_is_reported_and_the_handle_survives(nodes):
    p = synth.sphere_problem(num_nodes=nodes, num_corrs=40 * nodes, node_radius=0.3 * (12.6 / nodes) ** 0.5, seed=nodes)
    prm = Params(gn_iterations=2, pcg_iterations=10, pcg_tolerance=0.0, lambda_smooth=10.0, lambda_damping=1.0)
    dp = DeviceProblem(p)

    def make():
        s = GaussNewtonSolver(prm, max_nodes=nodes, max_corrs=p.num_corrs)
        s.set_option(_lib.CF_OPT_PCG_MODE, 2)
        return s

    def run(s):
        T = dp.init_transforms.clone()
        st = s.gn_solve(dp, T, max_rot=0.12, max_trans=0.04)
        torch.cuda.synchronize()
        return st, T

    s = make()
    s.set_option(_lib.CF_OPT_SPIN_LIMIT, 2000)
    s.set_option(_lib.CF_OPT_TEST_BARRIER_EXTRA, 1)
    with pytest.raises(_lib.CFError) as e:
        run(s)
    assert e.value.status == _lib.CF_ERR_TIMEOUT
    assert s.get_option(_lib.CF_OPT_PCG_ACTIVE) == 2
    s.set_option(_lib.CF_OPT_TEST_BARRIER_EXTRA, 0)
    s.set_option(_lib.CF_OPT_SPIN_LIMIT, 0)
    st, T = run(s)
    assert st["error_flags"] == 0
    assert torch.equal(T, run(make())[1])
