"""The reference's P2G and G2P over the ranges of their kernels, against the
oracle (particles.cu:370-662): sparse nodes (scattered with atomics), dense
ones (cell by cell), nodes of several rounds of 512 particles, particles on
the box's upper faces and outside it (keys that alias into other nodes), and
one particle.  FP64 on both sides; a voxel's sums run over at most some 5,000
terms of a few roundings each, in another order: 5,000 x 2^-52 = 1.1e-12 of
the sum of their absolute values, which the weighted mean of velocities in
[-1, 1] turns into the same relative to 1."""
import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1.2e-12

CASES = {
    # name: (particles, root cells per axis, cell size, positions as a share of the box)
    "sparse": (6000, (12, 10, 11), 1.0, (0.0, 1.0)),
    "dense": (40001, (6, 5, 7), 1.0 / 3.0, (0.0, 1.0)),
    "several_rounds": (20000, (2, 2, 2), 0.5, (0.0, 1.0)),
    "upper_faces_and_outside": (30000, (5, 5, 5), 1.0, (0.1, 1.25)),
    "one": (1, (4, 4, 4), 1.0, (0.3, 0.6)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_transfers_match_the_oracle(name):
    import torch
    n, size, cell, (lo, hi) = CASES[name]
    rng = np.random.default_rng(n)
    pos = (lo + (hi - lo) * rng.random((n, 3))) * np.array(size) * cell
    vel = rng.uniform(-1.0, 1.0, (n, 3))
    og = O.grid(0.0, 0.0, 0.0, *size, cell)
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), og)
    dev = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a).view(dt)).cuda()  # noqa: E731
    p = [dev(b[k], np.float64) for k in ("spx", "spy", "spz")]
    v = [dev(vel[:, k].copy(), np.float64) for k in range(3)]
    starts, keys = dev(b["starts"], np.int32), dev(b["sorted_keys"], np.int32)
    nv, ids, sol = dev(b["node_voxels"], np.int32), dev(b["voxel_ids"], np.int32), dev(b["solids"], np.int8)
    grid = F.make_grid(0.0, 0.0, 0.0, *size, cell)
    U = F.ref_p2g(starts, keys, b["nodes"], *p, *v, nv, ids, sol, grid)
    want = [O.ref_p2g(b, vel[:, d], og, d) for d in range(3)]
    for d in range(3):
        assert np.max(np.abs(U[d].cpu().numpy() - want[d])) <= TOL
    V = F.ref_g2p(starts, keys, b["nodes"], *p, nv, ids, *(dev(u, np.float64) for u in want), grid)
    for d in range(3):
        vo = O.ref_g2p(b, b["spx"], b["spy"], b["spz"], want[d], og, d)
        assert np.max(np.abs(V[d].cpu().numpy() - vo)) <= TOL
