"""The resident Jacobi-PCG solve (pcg_resident.cu) on the tile counts where it
changes form, every listed tile with fluid in it: S CTAs (one per SM) hold
21 tiles each with every vector on the chip, unless their tiles have more
faces towards other CTAs than half of the most -- then some CTAs keep all on the
chip and some do not --, from 22 on none does, up to 29 in a box no larger no
face lies in global memory, 40 have their w in registers, 88 is the most, and
one tile more goes to the loop of launches.  Checked as in
test_gpu_resident_pcg.py: |b - A x| <= tol |b| in FP64, twice, bit for bit."""
import numpy as np
import pytest

import flip2_b200 as F
from tests.test_gpu_resident_pcg import TOL, relative_residual

pytestmark = pytest.mark.gpu


def tiled_problem(dims, count, seed):
    """Fluid in the first `count` of a box of dims tiles, all but the top
    voxel row of the box; 2% of the cells solid in a quarter of it, none of
    them in a tile's first cells; b = N(0, 1) on the fluid."""
    nx, ny, nz = (8 * d for d in dims)
    rng = np.random.default_rng(seed)
    tile = np.arange(dims[0] * dims[1] * dims[2]).reshape(dims[2], dims[1], dims[0])
    listed = (tile < count).repeat(8, 0).repeat(8, 1).repeat(8, 2)
    typ = listed.astype(np.uint8)
    part = typ[: nz // 2, :, : nx // 2]
    part[(rng.random(part.shape, dtype=np.float32) < 0.02) & (part == 1)] = 2
    typ[::8, ::8, ::8][tile < count] = 1
    typ[:, ny - 1, :] = 0
    b = rng.standard_normal(typ.shape, dtype=np.float32) * (typ == 1)
    return typ, b


CASES = {
    # name: S -> (tiles a box axis, listed tiles)
    "21 a CTA, all on the chip": lambda S: ((8, 20, S // 7), 21 * S),
    "21 a CTA, some on the chip": lambda S: ((22, 12, S // 12), 21 * S),
    "one more": lambda S: ((37, 11, S // 18), 21 * S + 1),
    "29 a CTA in a box of 29 a CTA": lambda S: ((29, S // 4, 4), 29 * (S // 4) * 4),
    "30 a CTA": lambda S: ((22, 12, S // 8), 29 * S + 1),
    "40 a CTA": lambda S: ((16, 16, S // 6), 40 * S),
    "41 a CTA": lambda S: ((16, 16, S // 6), 41 * S),
    "88 a CTA, the box full": lambda S: ((22, S // 4, 16), 88 * (S // 4) * 4),
    "88 a CTA, the most": lambda S: ((37, 11, S // 4), 88 * S),
    "one too many": lambda S: ((37, 11, S // 4), 88 * S + 1),
    "nine tiles, three CTAs of a cluster": lambda S: ((1, 9, 1), 9),
    "64 tiles, the largest cluster": lambda S: ((4, 4, 4), 64),
}


@pytest.mark.parametrize("name", list(CASES))
def test_at_the_line(name):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    dims, count = CASES[name](min(sms, 160))
    assert count <= dims[0] * dims[1] * dims[2]
    typ, b = tiled_problem(dims, count, seed=count)
    P = F.Particles(1, mode=F.MODE_NATIVE)
    P.setDomain(0.0, 0.0, 0.0, *(2 * d for d in dims), 1.0)
    P.poisson_set(typ.ravel(), b.ravel())
    assert np.array_equal(P.read(F.BUF_TILE_LIST), np.arange(count))
    first = P.poisson_solve(0, TOL, 20000)
    x = P.poisson_solution().reshape(typ.shape)
    again = P.poisson_solve(0, TOL, 20000)
    y = P.poisson_solution().reshape(typ.shape)
    assert P.info().error_flags == 0
    P.close()
    for s in (first, again):
        assert s.converged == 1 and s.rel_residual <= TOL and s.fell_back == 0
    assert first.iters == again.iters
    assert np.array_equal(x, y)
    assert relative_residual(typ, b, x) <= TOL + 1e-9
