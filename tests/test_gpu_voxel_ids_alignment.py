"""flip_ref_voxel_ids on masks that a caller carved out of a larger buffer: a
pointer of any 4-byte alignment, in the compaction by lanes (65,536 nodes and
more) and in the one by warps, bit-exact against the oracle."""
import ctypes as C

import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O
from tests.test_gpu_voxel_ranges import CASES, positions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["lane_a_node", "eight_lanes"])
@pytest.mark.parametrize("words", [0, 1, 2, 3])
def test_masks_at_any_word(name, words):
    import torch
    n, size, cell, corner = CASES[name]
    pos = positions(name, n, size, cell, corner)
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), O.grid(*corner, *size, cell))
    assert (b["nodes"] >= 65536) == (name == "lane_a_node")
    grid = F.make_grid(*corner, *size, cell)
    p = [torch.from_numpy(pos[:, k].copy()).cuda() for k in range(3)]
    keys, perm = F.sort_pairs(F.ref_keys(*p, grid))
    p = [a[perm.long()].contiguous() for a in p]
    _, starts, _, nodes = F.segment_heads(keys, want_flags=False)
    starts = starts.contiguous()
    masks = torch.zeros(16 * nodes + 8, dtype=torch.int32, device="cuda")[words:]
    assert masks.data_ptr() % 16 == 4 * words
    counts = torch.empty(nodes, dtype=torch.int32, device="cuda")

    def ptr(t):
        return C.c_void_p(t.data_ptr())

    L = F.lib()
    assert L.flip_ref_voxel_counts(ptr(starts), ptr(keys), nodes, n, *map(ptr, p), C.byref(grid), ptr(counts), ptr(masks),
                                   None) == 0
    node_voxels = F.inclusive_scan(counts)
    nvox = int(node_voxels[-1].item())
    assert nvox == int(b["node_voxels"][-1])
    ids = torch.empty(nvox, dtype=torch.int32, device="cuda")
    solids = torch.empty(nvox, dtype=torch.int8, device="cuda")
    assert L.flip_ref_voxel_ids(ptr(keys), nodes, ptr(masks), ptr(node_voxels), C.byref(grid), ptr(ids), ptr(solids), None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(ids.cpu().numpy().view(np.uint32), b["voxel_ids"])
    assert np.array_equal(solids.cpu().numpy(), b["solids"])
    assert int(masks[16 * nodes:].abs().sum().item()) == 0
