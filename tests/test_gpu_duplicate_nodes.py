"""Correspondences that name a node in two or three of their slots: every slot
is blended at its own place (kernels/solver_kernels.cu:52-111 walks the slots),
so the sign that a node gets there depends on the slots before it.  Nodes whose
rotations are up to 180 degrees apart make that sign matter.  The energy at the
first linearisation point and after the step's twist of zero against the FP64
oracle, within the 1e-4 of the other energies; records (large sets) and
correspondences taken one by one (small sets)."""
import numpy as np
import pytest
import torch

from cudafusion_b200 import synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_set", [1, 3, 40])
@pytest.mark.parametrize("slots", [(0, 1, 2, 0), (0, 1, 0, 2), (1, 0, 0, 1), (2, 2, 0, 2), (0, 1, 2, 3)])
def test_energy_matches_the_oracle(oracle, slots, per_set):
    sets = 12
    rng = np.random.default_rng(100 * per_set + slots[1])
    p = synth.sphere_problem(num_nodes=24, num_corrs=sets * per_set, node_radius=0.2, seed=per_set)
    q = rng.normal(size=(24, 4))
    T = synth.centred_dq(q / np.linalg.norm(q, axis=1, keepdims=True), 0.02 * rng.normal(size=(24, 3)))
    ids = np.stack([rng.choice(24, 4, replace=False) for _ in range(sets)])[:, list(slots)]
    p.corrs["node_ids"] = np.repeat(ids, per_set, axis=0)
    p.corrs["node_ws"] = rng.uniform(0.05, 1.0, size=(sets * per_set, 4)) ** 2
    s = GaussNewtonSolver(Params(gn_iterations=1, pcg_iterations=1, pcg_tolerance=0.0, lambda_smooth=1e-6,
                                 lambda_damping=1.0), max_nodes=24, max_corrs=p.num_corrs)
    dp = DeviceProblem(p)
    Td = torch.from_numpy(T.view(np.uint8).reshape(-1).copy()).cuda()
    st = s.gn_solve(dp, Td, update_scale=0.0)
    torch.cuda.synchronize()
    E = oracle.energy(p, T, 1e-6, precision="f64")
    assert abs(st["energy"][0] - E) < 1e-4 * E
    assert abs(st["energy_final"] - E) < 1e-4 * E
