"""Voxel counts by eight lanes a node in dense boxes, and the compaction of
voxel ids on both sides of its lines (particles.cu:88-321), bit-exact against the
oracle: a warp a node (below 16,384 nodes), four nodes a warp and 32 (524,288
nodes and more), warps whose nodes have more voxels than a list holds and warps
whose nodes have not, four nodes that do not fit one either, and a last warp with
nodes missing."""
import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
LIST = 1280


def groups(b, size):
    """Voxels of each run of `size` nodes."""
    ends = np.append(b["node_voxels"][size - 1:: size], b["node_voxels"][-1] if b["nodes"] % size else [])
    return np.diff(np.concatenate([[0], ends.astype(np.int64)]))


CASES = {
    # name: particles, root cells, share of the particles in the box's lowest eighth
    "one node": (3, (4, 4, 4), 0.0),
    "dense, a warp a node": (12001, (7, 6, 5), 0.0),
    "dense, four a warp": (1200001, (28, 26, 27), 0.9),
    "sparse": (30017, (60, 61, 62), 0.0),
    "eight lanes, dense": (300007, (27, 28, 26), 0.0),
    "eight lanes, nearly too dense": (2000003, (26, 25, 26), 0.0),
    "many, some of them dense": (1400003, (101, 100, 99), 0.35),
}


@pytest.mark.parametrize("name", list(CASES))
def test_ids_match_the_oracle(name):
    import torch
    n, size, low = CASES[name]
    rng = np.random.default_rng(n)
    u = rng.random((n, 3))
    k = int(low * n)
    u[:k, 2] /= 8
    if name == "one node":
        u = 0.5 + 0.01 * u
    pos = u * np.array(size)
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), O.grid(0.0, 0.0, 0.0, *size, 1.0))
    four, all32 = groups(b, 4), groups(b, 32)
    if name == "dense, four a warp":
        assert b["nodes"] >= 16384 and (four > LIST).any() and (four <= LIST).any()
    if name == "sparse":
        assert b["nodes"] >= 16384 and b["nodes"] % 4
    if name.startswith("eight"):
        assert b["nodes"] >= 16384 and 8 <= n / b["nodes"] < 128
    if name.startswith("many"):
        assert b["nodes"] >= 1 << 19 and b["nodes"] % 32
        assert (all32 > LIST).any() and (all32 <= LIST).any()
    grid = F.make_grid(0.0, 0.0, 0.0, *size, 1.0)
    p = [torch.from_numpy(pos[:, a].copy()).cuda() for a in range(3)]
    keys, perm = F.sort_pairs(F.ref_keys(*p, grid))
    p = [a[perm.long()].contiguous() for a in p]
    _, starts, _, nodes = F.segment_heads(keys, want_flags=False)
    assert nodes == b["nodes"]
    _, node_voxels, ids, solids = F.ref_voxels(starts.contiguous(), keys, nodes, *p, grid)
    assert np.array_equal(node_voxels.cpu().numpy().view(np.uint32), b["node_voxels"])
    assert np.array_equal(ids.cpu().numpy().view(np.uint32), b["voxel_ids"])
    assert np.array_equal(solids.cpu().numpy(), b["solids"])
