"""The data term by node set (cf_cells.cu) where its units change: sets of 1..5
correspondences (without a record below 4), of a window of 32 and one less or
more, of a task of 64, of a sort chunk of 512, buckets past 1024 positions, the
two row widths of the gather, and shares shorter than a warp.  The assembled
matrix against the FP64 oracle: FP32 products summed over at most 32 of a
half-task before the rows are compensated, (32 + 4) 2^-24 of the largest entry.
(The right-hand side is held on config1: with so few correspondences it is the
edges', whose residuals in FP32 are 5e-5 of it off in the reference's order.)
"""
import numpy as np
import pytest
import torch

from cudafusion_b200 import synth
from cudafusion_b200.solver import GaussNewtonSolver, Params, to_device

pytestmark = pytest.mark.gpu


def sets(p, counts, seed):
    """p's correspondences with node sets of the given sizes, in random order."""
    rng = np.random.default_rng(seed)
    c = p.corrs[: sum(counts)].copy()
    base = p.corrs["node_ids"][rng.choice(p.num_corrs, len(counts), replace=False)]
    c["node_ids"] = np.repeat(base, counts, axis=0)
    c["node_ids"] = rng.permuted(c["node_ids"], axis=1)  # a set's slots in any order
    dup = rng.choice(c.shape[0], c.shape[0] // 10, replace=False)
    c["node_ids"][dup, 3] = c["node_ids"][dup, 0]
    gone = rng.choice(c.shape[0], c.shape[0] // 12, replace=False)
    c["node_ids"][gone, 1] = -1
    return c[rng.permutation(c.shape[0])]


CASES = {
    "single": (24, [1]),
    "five": (24, [2, 3]),
    "small sets": (300, [1, 2, 3, 4, 5] * 60),
    "window edges": (24, [31, 32, 33, 63, 64, 65, 95, 96, 97]),
    "task and chunk edges": (24, [127, 128, 129, 511, 512, 513]),
    "long buckets": (8, [1023, 1024, 1025, 2500, 3]),
    "four warps a row": (1024, [7] * 1200),
    "two warps a row": (1025, [7] * 1200),
}


@pytest.mark.parametrize("name", list(CASES))
def test_system_matches_the_oracle(oracle, name):
    nodes, counts = CASES[name]
    p = synth.sphere_problem(num_nodes=nodes, num_corrs=max(sum(counts), 2 * len(counts)),
                             node_radius=0.3 * (12.6 / nodes) ** 0.5, seed=3)
    c = sets(p, counts, seed=len(counts))
    s = GaussNewtonSolver(Params(pcg_iterations=2, pcg_tolerance=0.0, lambda_smooth=3.0), max_nodes=nodes, max_corrs=c.shape[0])
    s.solve(to_device(c), c.shape[0], to_device(p.nodes), to_device(p.gt_transforms), nodes)
    torch.cuda.synchronize()
    row_ptr, col_idx, vals, rhs = s.system()
    A, _, _ = oracle.assemble(c, p.nodes, p.gt_transforms, row_ptr, col_idx, 3.0, 1e-2, precision="f64")
    assert np.abs(vals - A).max() <= 36 * 2.0**-24 * np.abs(A).max()
    assert np.isfinite(rhs).all()
