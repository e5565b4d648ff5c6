"""The tensor-core backward pass where its tiles can go wrong: one tile, a row
of tiles (every box with faces outside the grid), tiles without activations
next to active ones, and more tiles than three rounds of a CTA per SM (both
stages of the pipeline reused).  Weight gradients of all four layers against
the CUDA-core kernels, FP32 throughout; the tensor cores take input gradients
as BF16 operands (relative error 2^-9 each, averaged over the products), so
3e-3 in L2 over all weights and 5e-3 per layer, with room for the ReLU masks
that a BF16 rounding of the activations flips."""
import numpy as np
import pytest

import flip2_b200 as F
from tests.test_gpu_lprec import engine, random_types

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,fill", [((8, 8, 8), 1.0), ((56, 8, 8), 1.0), ((64, 64, 64), 0.4), ((72, 64, 64), 1.0)])
def test_backward_on_ranges_of_tiles(shape, fill):
    typ = random_types(shape, 3)
    nx, ny, nz = shape
    # fluid only in the lower part: tiles above hold air and are not listed
    j = (np.arange(typ.size) // nx) % ny
    typ = np.where((typ == 1) & (j >= fill * ny), 0, typ).astype(np.uint8)
    rng = np.random.default_rng(4)
    r = (rng.standard_normal(typ.size) * (typ == 1)).astype(np.float32)
    ev = (r + 0.5 * rng.standard_normal(typ.size) * (typ == 1)).astype(np.float32)
    w = (rng.standard_normal(F.lib().flip_lp_num_weights()) * 0.15).astype(np.float32)
    gs = []
    for cc in (0, 1):
        P = engine(shape, lp_cuda_cores=cc)
        P.poisson_set(typ, np.zeros(typ.size, np.float32))
        P.lp_set_weights(w)
        P.lp_eval(r, ev, want_grad=True)
        assert P.info().error_flags == 0
        gs.append(P.lp_grad())
        P.close()
    offs = [0, 27 * 3 * 16, 27 * 3 * 16 + 27 * 256, 27 * 3 * 16 + 2 * 27 * 256, gs[0].size]
    assert np.linalg.norm(gs[0] - gs[1]) <= 3e-3 * np.linalg.norm(gs[1])
    for l in range(4):
        a, b = gs[0][offs[l]:offs[l + 1]], gs[1][offs[l]:offs[l + 1]]
        assert np.linalg.norm(a - b) <= 5e-3 * np.linalg.norm(b), l
