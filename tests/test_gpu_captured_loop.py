"""Captured steps and frames on more tiles than the resident pressure solve
holds: the solve's kernel leaves at once and the graph's loop of launches runs,
in the step's graph, inside a frame's loop over sub-steps, and in the restart
branch of a learned solve.  As in test_gpu_graph.py each captured form must
give what the launch-by-launch form gives."""
import os

import numpy as np
import pytest

import flip2_b200 as F

pytestmark = pytest.mark.gpu
BOX = 256


@pytest.fixture(scope="module")
def block():
    """A particle a cell in the lowest 104 cell layers: 32 x 13 x 32 tiles."""
    rng = np.random.default_rng(5)
    x, y, z = np.meshgrid(np.arange(BOX), np.arange(104), np.arange(BOX), indexing="ij")
    pos = np.stack([x.ravel(), y.ravel(), z.ravel()], 1).astype(np.float32)
    pos += rng.uniform(0.05, 0.95, pos.shape).astype(np.float32)
    pos /= BOX
    vel = 0.1 * np.sin(2 * np.pi * pos[:, ::-1]).astype(np.float32)
    return pos, vel


def run(block, timing, frame, method):
    import torch
    pos, vel = block
    kw = dict(pressure_method=method)
    if method:
        kw["learned_max_iter"] = 1  # misses tol: the restart branch runs
    P = F.Particles(pos.shape[0], mode=F.MODE_NATIVE, params=F.default_params(F.MODE_NATIVE, **kw))
    P.setDomain(0.0, 0.0, 0.0, BOX // 4, BOX // 4, BOX // 4, 4.0 / BOX)
    if method:
        P.lp_set_weights(np.load(os.path.join(os.path.dirname(F.__file__), "data", "mg_weights.npy")))
    P.set_timing(timing)
    P.upload(pos, vel)
    P.solveFrame(120.0) if frame else P.step(1.0 / 240)
    P.sync()
    info, solve = P.info(), P.solve_info()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert info.nodes > 88 * min(sms, 160)
    assert info.error_flags == 0 and info.converged == 1 and info.residual <= 1e-6
    assert solve.fell_back == (1 if method else 0)
    out = P.download()
    P.close()
    return out, info, solve


@pytest.mark.parametrize("frame", [False, True])
@pytest.mark.parametrize("method", [0, 2])
def test_the_loop_past_the_resident_solve(block, frame, method):
    (pe, ve), ie, se = run(block, True, frame, method)
    (pg, vg), ig, sg = run(block, False, frame, method)
    assert ie.graph_steps == 0 and ig.graph_steps == ig.solves == ie.solves >= (2 if frame else 1)
    # one chunk of slack, as in test_gpu_graph.py
    assert abs(ie.pressure_iters - ig.pressure_iters) <= 64
    assert abs(ie.pressure_iters_total - ig.pressure_iters_total) <= 64 * ig.solves
    assert se.plain_iters == pytest.approx(sg.plain_iters, abs=64)
    if not frame:  # rows stay in the order of the same first keys
        assert np.max(np.abs(pe - pg)) < 1e-4 / BOX
        assert np.max(np.abs(ve - vg)) < 1e-4 * max(1.0, float(np.max(np.abs(ve))))
    assert np.max(np.abs(np.sort(pe, axis=0) - np.sort(pg, axis=0))) < 1e-4 / BOX
