"""The resident pressure solve gives up on a wait that nothing ends, reports it,
and the engine solves on.  flip_test_solve_timeout makes one CTA poll for a
word that nothing publishes, a bounded number of times: in hop 1 of an
exchange, in hop 2, and for a neighbouring CTA's face cells; in a cluster and
in a cooperative grid; in a call, in a captured step and in a captured frame.
Nothing here faults or hangs the GPU: every wait ends by its own limit (some
10 ms here) and every access stays inside the buffers.  The solve after it
gives the solution of the solve before it, bit for bit: no packet or face cell
of the abandoned solve reaches it."""
import numpy as np
import pytest

import flip2_b200 as F
from flip2_b200 import scenes
from tests.test_gpu_resident_pcg import TOL, problem

pytestmark = pytest.mark.gpu
FLIP_ERR_TIMEOUT = 4
GRID_TIMEOUT = 1 << 4
POLLS = 1 << 14
CLUSTER, TWO_HOPS = (32, 24, 32), (64, 72, 64)


@pytest.mark.parametrize("shape,which", [(CLUSTER, 0), (CLUSTER, 2), (TWO_HOPS, 0), (TWO_HOPS, 1), (TWO_HOPS, 2)])
@pytest.mark.parametrize("exchange", [1, 7])
def test_a_lost_word_ends_the_solve(shape, which, exchange):
    typ, b = problem(shape, seed=3)
    P = F.Particles(1, mode=F.MODE_NATIVE)
    P.setDomain(0.0, 0.0, 0.0, shape[0] // 4, shape[1] // 4, shape[2] // 4, 1.0)
    P.poisson_set(typ.ravel(), b.ravel())
    before = P.poisson_solve(0, TOL, 4000)
    x = P.poisson_solution()
    for _ in range(2):
        P._call("flip_test_solve_timeout", which, exchange, POLLS)
        with pytest.raises(F.FlipError) as err:
            P.poisson_solve(0, TOL, 4000)
        assert err.value.status == FLIP_ERR_TIMEOUT
        assert "pressure solve timed out" in str(err.value)
        assert P.info().error_flags & GRID_TIMEOUT
        P._call("flip_test_solve_timeout", which, 0, 0)
        after = P.poisson_solve(0, TOL, 4000)
        assert after.converged == 1 and after.iters == before.iters
        assert np.array_equal(P.poisson_solution(), x)
    P.close()


@pytest.mark.parametrize("frame", [False, True])
@pytest.mark.parametrize("method", [0, 2])
def test_captured_steps_report_it(frame, method):
    """method 2: the restart of a learned solve that may take no iterations.  No
    warm start: the second upload's problem is the first one's, solved already."""
    nc = 32
    pos, vel = scenes.dam_break(nc, seed=0)
    params = F.default_params(F.MODE_NATIVE, pressure_method=method, learned_max_iter=1 if method else 400,
                              pcg_warm_start=0)
    P = F.Particles(pos.shape[0], mode=F.MODE_NATIVE, params=params)
    P.setDomain(0.0, 0.0, 0.0, nc // 4, nc // 4, nc // 4, 4.0 / nc)
    if method:
        P.lp_init(1)

    def advance():
        P.upload(pos, vel)
        P.solveFrame(60.0) if frame else P.step(1.0 / 240)
        P.sync()

    advance()
    assert P.info().converged == 1
    P._call("flip_test_solve_timeout", 0, 5, POLLS)
    with pytest.raises(F.FlipError) as err:
        advance()
    assert err.value.status == FLIP_ERR_TIMEOUT
    assert P.info().error_flags & GRID_TIMEOUT
    P._call("flip_test_solve_timeout", 0, 0, 0)
    advance()
    info = P.info()
    assert info.converged == 1 and info.residual <= 1e-6
    assert info.graph_steps >= 1
    out = P.download()
    assert all(np.isfinite(a).all() for a in out)
    P.close()


def test_bad_arguments():
    P = F.Particles(1, mode=F.MODE_NATIVE)
    P.setDomain(0.0, 0.0, 0.0, 2, 2, 2, 1.0)
    for args in ((3, 1, POLLS), (-1, 1, POLLS), (0, 1, 1023)):
        with pytest.raises(F.FlipError) as err:
            P._call("flip_test_solve_timeout", *args)
        assert err.value.status == 1
    P.close()
