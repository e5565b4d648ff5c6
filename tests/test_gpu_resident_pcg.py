"""The resident Jacobi-PCG solve (pcg_resident.cu) at the edges of its ranges:
one tile, one group of CTAs and several, every vector on the chip and not,
faces without room on the chip, and more tiles than it holds (the solve then
runs as a loop of launches).  The solution of each problem is put back into
the 7-point system in numpy, in FP64: |b - A x| <= tol |b|, the solver's own
stopping rule evaluated independently, with 1e-9 for the rounding of that
evaluation (x and b are exact inputs; every product and sum is FP64)."""
import numpy as np
import pytest

import flip2_b200 as F

pytestmark = pytest.mark.gpu
TOL = 1e-6


def problem(shape, seed):
    """Fluid below 90% of the height, 2% of the cells solid in a quarter of
    the box, b = N(0, 1) on the fluid: (nz, ny, nx) arrays."""
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    typ = np.zeros((nz, ny, nx), np.uint8)
    typ[:, : max(1, int(0.9 * ny)), :] = 1
    part = typ[: (nz + 1) // 2, :, : (nx + 1) // 2]
    part[rng.random(part.shape, dtype=np.float32) < 0.02] = 2
    b = rng.standard_normal(typ.shape, dtype=np.float32) * (typ == 1)
    return typ, b  # (2% of solid cells wall in no fluid cell: 0.02^6 a cell)


def relative_residual(typ, b, x):
    fluid = typ == 1
    xp = np.pad(np.where(fluid, x, 0.0), 1)
    sp = np.pad(typ == 2, 1, constant_values=True)
    diag = np.zeros(typ.shape)
    total = np.zeros(typ.shape)
    mid = slice(1, -1)
    for ax in range(3):
        for lo in (0, 2):
            at = [mid, mid, mid]
            at[ax] = slice(lo, lo + typ.shape[ax])
            diag += ~sp[tuple(at)]
            total += xp[tuple(at)]
    r = np.where(fluid, b.astype(np.float64) - (diag * x - total), 0.0)
    return np.linalg.norm(r) / np.linalg.norm(b.astype(np.float64))


@pytest.mark.parametrize("shape", [
    (8, 8, 8),        # one tile, one CTA
    (40, 16, 24),     # 30 tiles, 8 CTAs: one hop
    (64, 72, 64),     # 576 tiles, 144 CTAs: two hops
    (120, 104, 128),  # 3,120 tiles, 22 a CTA: the most with every vector on the chip
    (128, 112, 128),  # 3,584 tiles, 25 a CTA: w in registers, the rest through L2
    (184, 184, 184),  # 12,167 tiles, 83 a CTA: faces and w without room on the chip
    (200, 192, 192),  # 14,400 tiles: more than the chip holds
])
def test_solution_satisfies_the_system(shape):
    typ, b = problem(shape, seed=sum(shape))
    P = F.Particles(1, mode=F.MODE_NATIVE)
    P.setDomain(0.0, 0.0, 0.0, shape[0] // 4, shape[1] // 4, shape[2] // 4, 1.0)
    P.poisson_set(typ.ravel(), b.ravel())
    first = P.poisson_solve(0, TOL, 20000)
    x = P.poisson_solution().reshape(typ.shape)
    again = P.poisson_solve(0, TOL, 20000)  # the exchange's tags go on from the first solve's
    y = P.poisson_solution().reshape(typ.shape)
    P.close()
    for s in (first, again):
        assert s.converged == 1 and s.rel_residual <= TOL and s.fell_back == 0
    assert first.iters == again.iters  # every sum is taken in a fixed order
    assert np.array_equal(x, y)
    assert relative_residual(typ, b, x) <= TOL + 1e-9
