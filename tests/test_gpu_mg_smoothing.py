"""The multilevel smoothing kernels where a tile can go wrong: one tile along
an axis, ragged boxes whose coarse levels are padded, and a second problem on
the same engine, whose coarse fluid tiles are others than the first one's
(corrections off the list of tiles read as zero, not as what the first
problem left there).  One V-cycle without the network against the oracle's
FP64 restatement."""
import os

import numpy as np
import pytest

import flip2_b200 as F
from oracle import oracle as O
from tests.test_gpu_lprec import engine, problem_arrays
from tests.util import rel_err

pytestmark = pytest.mark.gpu
WEIGHTS = os.path.join(os.path.dirname(F.__file__), "data", "mg_weights.npy")


@pytest.mark.parametrize("shape", [(32, 8, 8), (8, 40, 24), (72, 16, 104), (64, 64, 64)])
def test_vcycle_on_changing_problems(shape):
    P = engine(shape, mg_coarse=1)
    W = np.load(WEIGHTS)
    for seed, radius in ((3, (1.0, 3.0)), (4, (8.0, 20.0)), (5, (2.0, 6.0))):
        P.poisson_generate(seed=seed, radius=radius)
        P.lp_set_weights(W)
        typ, _ = problem_arrays(P, shape)
        if not np.any(typ == 1):
            continue
        r = np.where(typ == 1, np.random.default_rng(seed).standard_normal(typ.size), 0.0).astype(np.float32)
        z = P.mg_apply(r)
        assert P.info().error_flags == 0
        zo = O.mg_apply(typ, r, W, shape, mode=1)
        assert np.all(z[typ != 1] == 0.0)
        # some 30 FP32 operations per cell and level at 6e-8 each, no more
        # than five levels, every sweep a contraction: below 1e-5
        assert rel_err(z, zo) < 1e-5
        assert np.linalg.norm(z - zo) <= 1e-5 * np.linalg.norm(zo)
    P.close()
