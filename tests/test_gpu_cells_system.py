"""The assembled system and the energies of the data term by node set, where its
units change (tests/test_gpu_cells.py) and where its lists are long: rows with
more blocks than a pass of the gather takes (a hub of the graph) and a node in
more than 4096 tasks.  Large residuals and no smoothness term, so that every
value is the data term's.

Bound of an entry: (32 + 32) 2^-24 of the sum of its terms' magnitudes: FP32
sums of at most 32 of a half-task, what is left for the factors, the move from the
set's lowest node to the row's (a term counts with the largest distance of its
point to a node of its set) and the compensated sum of the tasks; and one
rounding of the damping, which is at least lambda 1e-2 on the diagonal of a node
without correspondences."""
import numpy as np
import pytest
import torch

from cudafusion_b200 import synth
from cudafusion_b200.solver import DeviceProblem, GaussNewtonSolver, Params, to_device

from test_gpu_cells import CASES, sets

pytestmark = pytest.mark.gpu

U = 64 * 2.0**-24
DAMPING = 2.0**-24 * 1e-2 * 1e-2


def scene(nodes, corrs, seed=3):
    p = synth.sphere_problem(num_nodes=nodes, num_corrs=corrs, node_radius=0.3 * (12.6 / nodes) ** 0.5, seed=seed)
    rng = np.random.default_rng(seed)
    c = p.corrs
    c["dst"] = c["src"] + (0.3 * rng.normal(size=(corrs, 1)) * c["normal"]).astype(np.float32)
    c["weight"] = rng.uniform(0.2, 1.0, corrs)
    return p


def magnitudes(c, nodes):
    """Per block and per row the sums of the terms' magnitudes: (uu, un, nn), (u, n)."""
    N = len(nodes)
    x, src = nodes["pos"].astype(np.float64), c["src"].astype(np.float64)
    r = np.abs(np.sum(c["normal"].astype(np.float64) * (src - c["dst"]), 1))
    fw = np.where(c["valid"] != 0, c["weight"], 0) * np.minimum(1.0, 0.2 / np.maximum(r, 1e-30))
    ids, ws = c["node_ids"], np.where(c["node_ids"] >= 0, c["node_ws"], 0).astype(np.float64)
    dist = np.where(ids >= 0, np.linalg.norm(src[:, None] - x[np.maximum(ids, 0)], axis=2), 0).max(1)
    A, b = np.zeros((3, N, N)), np.zeros((2, N))
    for s in range(4):
        i = np.maximum(ids[:, s], 0)
        np.add.at(b[0], i, fw * ws[:, s] * r * dist)
        np.add.at(b[1], i, fw * ws[:, s] * r)
        for t in range(4):
            j = np.maximum(ids[:, t], 0)
            for k in range(3):
                np.add.at(A[k], (i, j), fw * ws[:, s] * ws[:, t] * dist ** (2 - k))
    return A, b


def check(oracle, c, nodes, T):
    N, M = len(nodes), len(c)
    s = GaussNewtonSolver(Params(pcg_iterations=2, pcg_tolerance=0.0, lambda_smooth=1e-9), max_nodes=N, max_corrs=M)
    s.solve(to_device(c), M, to_device(nodes), to_device(T), N)
    torch.cuda.synchronize()
    row_ptr, col_idx, vals, rhs = s.system()
    A, b, e = oracle.assemble(c, nodes, T, row_ptr, col_idx, 1e-9, 1e-2, precision="f64")
    mA, mb = magnitudes(c, nodes)
    row = np.repeat(np.arange(N), np.diff(row_ptr))
    half = np.add.outer(np.arange(6) // 3, np.arange(6) // 3)  # 0: uu, 1: un, 2: nn
    bound = U * 1.01 * mA[:, row, col_idx][half].transpose(2, 0, 1)  # [block][6][6]
    assert (np.abs(vals.reshape(-1, 6, 6) - A.reshape(-1, 6, 6)) <= bound + DAMPING).all()
    assert (np.abs(rhs.reshape(N, 6) - b.reshape(N, 6)) <= U * mb[np.arange(6) // 3].T).all()
    assert abs(s.last_stats()["energy_initial"] - e) < 1e-4 * e


@pytest.mark.parametrize("name", list(CASES))
def test_edges_of_the_units(oracle, name):
    nodes, counts = CASES[name]
    p = scene(nodes, max(sum(counts), 2 * len(counts)))
    c = sets(p, counts, seed=len(counts))
    check(oracle, c, p.nodes, p.init_transforms)


@pytest.mark.parametrize("name", list(CASES))
def test_energies(oracle, name):
    nodes, counts = CASES[name]
    p = scene(nodes, max(sum(counts), 2 * len(counts)))
    c = sets(p, counts, seed=len(counts))
    p.corrs, p.canon = c, c["src"].copy()
    s = GaussNewtonSolver(Params(gn_iterations=1, pcg_iterations=1, pcg_tolerance=0.0, lambda_smooth=1e-9),
                          max_nodes=nodes, max_corrs=len(c))
    dp = DeviceProblem(p)
    T = torch.from_numpy(np.ascontiguousarray(p.gt_transforms).view(np.uint8).reshape(-1).copy()).cuda()
    st = s.gn_solve(dp, T, update_scale=0.0)
    E = oracle.energy(p, p.gt_transforms, 1e-9, precision="f64")
    assert abs(st["energy"][0] - E) < 1e-4 * E and abs(st["energy_final"] - E) < 1e-4 * E


@pytest.mark.parametrize("nodes", [300, 1100])  # four and two warps per row
@pytest.mark.parametrize("spokes", [15, 16, 17, 32, 33, 60])
def test_hub_of_the_graph(oracle, nodes, spokes):
    p = scene(nodes, 4000)
    rng = np.random.default_rng(spokes)
    nd = p.nodes
    nd["neighbors"][0] = -1  # the hub's blocks are those of the nodes that list it
    nd["num_neighbors"][0] = 0
    for i in range(1, nodes):
        nb = nd["neighbors"][i]
        nb[nb == 0] = (i % (nodes - 1)) + 1
    ends = rng.choice(np.arange(1, nodes), spokes, replace=False)
    nd["neighbors"][ends, 0] = 0
    nd["num_neighbors"][ends] = np.maximum(nd["num_neighbors"][ends], 1)
    hub = rng.random(len(p.corrs)) < 0.5
    p.corrs["node_ids"][hub, 1] = 0
    p.corrs["node_ids"][hub, 2] = rng.choice(ends, hub.sum())
    p.corrs["node_ws"] = rng.uniform(0.1, 1.0, (len(p.corrs), 4))
    # both sets of one correspondence and sets of many
    p.corrs["node_ids"][::2] = p.corrs["node_ids"][:: 100].repeat(50, axis=0)[: len(p.corrs[::2])]
    check(oracle, p.corrs, nd, p.init_transforms)


@pytest.mark.parametrize("nodes", [300, 1100])
def test_node_in_many_tasks(oracle, nodes):
    p = scene(nodes, 9000)
    rng = np.random.default_rng(nodes)
    p.corrs["node_ids"][:] = np.stack([rng.permutation(nodes)[:4] for _ in range(9000)])
    p.corrs["node_ids"][:7000, 2] = 5  # sets of one correspondence, almost all different
    p.corrs["node_ws"] = rng.uniform(0.1, 1.0, (9000, 4))
    check(oracle, p.corrs, p.nodes, p.init_transforms)
