"""The reference engine on few particles with many voxels each: the block
maxima of the residual, one per 512 voxels, have room of their own (they were
held in a buffer sized by the particles and ran past its end into whatever was
allocated behind it, the voxel ids for one).  After a sub-step's pressure solve the
voxel lists are still the oracle's, and p is its sweeps' on the engine's own
divergence, to the bound of test_gpu_ref_step.py."""
import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O
from tests.test_ref_bottom_plane import box_scene
from tests.util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [60, 500, 3000])
@pytest.mark.parametrize("kind", ["inside", "faces"])
def test_voxel_lists_survive_the_pressure_solve(n, kind):
    pos, vel, g = box_scene(kind, 2, n=n)
    og = O.grid(*g)
    b = O.ref_bin(pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), og)
    assert b["voxels"] // 512 + 1 > 2 * (n // 512 + 2)  # more blocks than the particles' buffer holds
    P = F.Particles(n, mode=F.MODE_REFERENCE)
    P.setDomain(*g)
    P.upload(pos, vel)
    P.initialize()
    P.particleVelToVoxels()
    P.pressureSolve()
    info = P.info()
    assert np.array_equal(P.read(F.BUF_VOXEL_IDS), b["voxel_ids"])
    assert np.array_equal(P.read(F.BUF_SOLIDS), b["solids"])
    assert np.array_equal(P.read(F.BUF_NODE_VOXELS), b["node_voxels"])
    div = P.read(F.BUF_DIVU)
    _, iters, p, _ = O.ref_gs_solve(b, div, np.zeros(b["voxels"]), info.dt, og)
    if info.pressure_iters == iters:  # the first dt was kept: this solve's sweeps are all there were
        assert rel_err(P.read(F.BUF_P), p, floor=1e-30) < 1e-8
    P.updateVoxelVelocities()
    P.voxelVelsToParticles()
    P.advectParticles()
    P.moveSolidParticles()
    assert all(np.isfinite(a).all() for a in P.download())
    P.close()
