"""The resident Jacobi-PCG solve claims nothing before its first step: a
right-hand side with an infinity or a NaN in it has no solution (r.r <= tol^2
b.b holds as inf <= inf), and a tolerance above 1 gets the one step that a
cold solve takes before it looks at its residual.  In a cluster, in a
cooperative grid and in the loop of launches past it."""
import numpy as np
import pytest

import flip2_b200 as F
from tests.test_gpu_resident_pcg import problem, relative_residual

pytestmark = pytest.mark.gpu
SHAPES = [(16, 16, 16), (40, 48, 40), (120, 104, 128), (200, 192, 192)]


def engine(shape, typ, b):
    P = F.Particles(1, mode=F.MODE_NATIVE)
    P.setDomain(0.0, 0.0, 0.0, shape[0] // 4, shape[1] // 4, shape[2] // 4, 1.0)
    P.poisson_set(typ.ravel(), b.ravel())
    return P


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_no_solution_is_not_converged(shape, value):
    typ, b = problem(shape, seed=sum(shape))
    b[1, 1, 1] = value
    typ[1, 1, 1] = 1
    P = engine(shape, typ, b)
    for _ in range(2):
        s = P.poisson_solve(0, 1e-6, 200)
        assert s.converged == 0
    P.close()


@pytest.mark.parametrize("shape", SHAPES)
def test_a_loose_tolerance_takes_one_step(shape):
    typ, b = problem(shape, seed=sum(shape))
    P = engine(shape, typ, b)
    s = P.poisson_solve(0, 3.0, 200)
    x = P.poisson_solution().reshape(typ.shape)
    P.close()
    assert s.converged == 1 and s.iters == 1
    # one step of steepest descent in D^-1: the residual is the solver's own to rounding
    assert abs(relative_residual(typ, b, x) - s.rel_residual) <= 1e-6 * s.rel_residual
