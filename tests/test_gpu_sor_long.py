"""The reference's pressure solve where its sweeps run in long chunks
(ref_gs_long_kernel), against the oracle's sweeps in index order: solid
voxels at all of the domain's faces, particles on its upper faces, positions
on the voxels' corners.  The oracle sweeps the engine's own divergence (its
divergence of particles past the last z row reads its row table out of
bounds, as the reference does).  After some 1,000 sweeps both sides are at
the system's solution, so p agrees to the rounding of one sweep, amplified by
the system: the bound is the one of test_gpu_ref_step.py for p."""
import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O
from tests.test_ref_bottom_plane import box_scene
from tests.util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,seed", [("inside", 8), ("faces", 12), ("faces", 17), ("faces", 21), ("lattice", 3)])
def test_long_chunks_against_the_oracle(kind, seed):
    pos, vel, g = box_scene(kind, seed)
    og = O.grid(*g)
    P = F.Particles(pos.shape[0], mode=F.MODE_REFERENCE)
    P.setDomain(*g)
    P.upload(pos, vel)
    P.initialize()
    P.particleVelToVoxels()
    P.pressureSolve()
    info = P.info()
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), og)
    div = P.read(F.BUF_DIVU)
    _, iters, p, _ = O.ref_gs_solve(b, div, np.zeros(b["voxels"]), info.dt, og)
    assert iters >= 1025  # one long chunk at least
    assert info.pressure_iters == iters  # the first dt was kept
    assert rel_err(P.read(F.BUF_P), p, floor=1e-30) < 1e-8
    P.close()
