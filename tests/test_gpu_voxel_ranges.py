"""Voxel activation over the ranges of its kernels, bit-exact against the
oracle (getNumberVoxelsUsedPerNode and generateVoxelIDs, particles.cu:88-321):
a lane a node (65,536 nodes and more, few particles in each), eight lanes, a
warp; nodes of more than 1,024 particles (positions clamped to the domain's
faces, which several warps share); positions on a lattice whose distances to
the voxel faces' points equal the radius exactly, where the FP32 test leaves
the decision to the FP64 one; positions a few 1e-7 from that radius; particles
outside the box, whose keys alias past its upper faces."""
import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = {
    # name: (particles, root cells per axis, cell size, corner)
    "lane_a_node": (150001, (50, 52, 48), 1.0, (0.0, 0.0, 0.0)),
    "eight_lanes": (20011, (24, 24, 24), 1.0 / 3.0, (-1.7, 2.1, 0.3)),
    "warp_a_node": (40003, (9, 7, 8), 0.7, (0.0, -3.0, 0.0)),
    "piled": (60001, (10, 10, 10), 1.0, (0.0, 0.0, 0.0)),
    "lattice": (30000, (12, 12, 12), 1.0, (0.0, 0.0, 0.0)),
    "at_the_radius": (30000, (16, 16, 16), 1.0, (0.0, 0.0, 0.0)),
    "outside": (20003, (14, 15, 16), 0.5, (0.0, 0.0, 0.0)),
    "one": (1, (4, 4, 4), 1.0, (0.0, 0.0, 0.0)),
}


def positions(name, n, size, cell, corner):
    rng = np.random.default_rng(len(name) + n)
    ext = np.array(size) * cell
    u = rng.random((n, 3))
    h = cell / 4
    if name == "piled":
        u = np.clip(rng.normal(0.05, 0.1, (n, 3)), 0.0, 1.0 - 2.0 ** -24)
    if name == "outside":
        u = u * 1.3 - 0.15
    p = u * ext
    if name == "lattice":
        p = np.round(p / (h / 2)) * (h / 2)
    if name == "at_the_radius":
        v = rng.normal(size=(n, 3))
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        p = np.floor(p / h) * h + np.array([0.0, 0.5, 0.5]) * h + 2 * h * v * (1 + 1e-7 * rng.normal(size=(n, 1)))
    return p + np.array(corner)


@pytest.mark.parametrize("name", list(CASES))
def test_voxels_match_the_oracle(name):
    import torch
    n, size, cell, corner = CASES[name]
    pos = positions(name, n, size, cell, corner)
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), O.grid(*corner, *size, cell))
    grid = F.make_grid(*corner, *size, cell)
    p = [torch.from_numpy(pos[:, k].copy()).cuda() for k in range(3)]
    keys, perm = F.sort_pairs(F.ref_keys(*p, grid))
    p = [a[perm.long()].contiguous() for a in p]
    _, starts, _, nodes = F.segment_heads(keys, want_flags=False)
    assert nodes == b["nodes"]
    _, node_voxels, ids, solids = F.ref_voxels(starts.contiguous(), keys, nodes, *p, grid)
    assert np.array_equal(node_voxels.cpu().numpy().view(np.uint32), b["node_voxels"])
    assert np.array_equal(ids.cpu().numpy().view(np.uint32), b["voxel_ids"])
    assert np.array_equal(solids.cpu().numpy(), b["solids"])
