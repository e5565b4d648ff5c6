"""The invariant that ref_gs_long_kernel rests on: a listed voxel of a tile's
plane y = 0 is a solid one.  The oracle's lists (particles.cu:88-321) for
positions that would break it if anything did: on the voxels' faces and
midpoints, a rounding step to either side of them, on the domain's faces and
clamped onto them, and at random."""
import numpy as np
import pytest

from oracle import oracle as O


def box_scene(kind, seed, n=20000):
    """n particles in a box of 5 x 4 x 6 root cells, and N(0, 1) velocities."""
    rng = np.random.default_rng(seed)
    g = (-0.5, 0.25, 1.0, 5, 4, 6, 0.25)
    lo, ext = np.array(g[:3]), np.array(g[3:6]) * g[6]
    u = rng.random((n, 3))
    if kind == "faces":  # a sixth of the span beyond the faces: clamped onto them
        u = u * 1.2 - 0.1
    if kind in ("lattice", "beside"):  # half voxels: corners, midpoints and the faces
        h = g[6] / 8
        u = np.round(u * ext / h) * h / ext
    pos = lo + u * ext
    if kind == "beside":
        pos = np.where(rng.random((n, 3)) < 0.5, np.nextafter(pos, -10.0), np.nextafter(pos, 10.0))
    return pos, rng.normal(size=(n, 3)), g


@pytest.mark.parametrize("kind", ["inside", "faces", "lattice", "beside"])
@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("cell,corner", [(0.25, None), (1.0 / 3.0, 0.0), (0.7, -1.7), (1e-3, 0.1)])
def test_listed_voxels_of_the_bottom_plane_are_solid(kind, seed, cell, corner):
    pos, _, g = box_scene(kind, seed)
    if corner is not None:  # the same relative places in a box of another size and corner
        pos = corner + (pos - np.array(g[:3])) / g[6] * cell
        g = (corner,) * 3 + g[3:6] + (cell,)
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), O.grid(*g))
    bottom = (b["voxel_ids"] % 64) // 8 == 0
    assert bottom.any()
    assert (b["solids"][bottom] != 0).all()
