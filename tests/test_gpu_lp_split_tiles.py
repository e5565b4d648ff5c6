"""The network's tensor-core layers where their CTAs share a tile's slices:
four CTAs a tile, two, and one, on both sides of each line (tiles against CTAs
of a launch: one a SM for the weight gradients and dilation 4, three for
dilation 2).  Against the CUDA-core kernels, with the bounds of
test_gpu_lp_backward_ranges.py for the gradients and of test_gpu_lprec.py for
the output."""
import numpy as np
import pytest

import flip2_b200 as F
from tests.test_gpu_lprec import engine

pytestmark = pytest.mark.gpu


def box_of(tiles):
    """A box of that many tiles, as nearly square in x and y as it gets."""
    k = max(d for d in range(1, int(tiles ** 0.5) + 1) if tiles % d == 0)
    return 8 * (tiles // k), 8 * k, 8


@pytest.mark.parametrize("ctas,parts,past", [(1, 4, 0), (1, 4, 1), (1, 2, 0), (1, 2, 1), (3, 4, 0), (3, 4, 1), (3, 2, 0), (3, 2, 1)])
def test_split_tiles_match_cuda_cores(ctas, parts, past):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shape = box_of(ctas * sms // parts + past)
    rng = np.random.default_rng(6)
    typ = np.where(rng.random(shape[::-1]) < 0.08, 2, 1).astype(np.uint8)  # fluid in every tile
    typ[:, -1, :] = 0
    typ = typ.ravel()
    r = (rng.standard_normal(typ.size) * (typ == 1)).astype(np.float32)
    ev = (r + 0.5 * rng.standard_normal(typ.size) * (typ == 1)).astype(np.float32)
    w = (rng.standard_normal(F.lib().flip_lp_num_weights()) * 0.15).astype(np.float32)
    zs, gs = [], []
    for cc in (0, 1):
        P = engine(shape, lp_cuda_cores=cc)
        P.poisson_set(typ, np.zeros(typ.size, np.float32))
        P.lp_set_weights(w)
        zs.append(P.lp_eval(r, ev, want_grad=True)[0])
        assert P.info().error_flags == 0
        gs.append(P.lp_grad())
        P.close()
    assert np.linalg.norm(zs[0] - zs[1]) <= 1e-3 * np.linalg.norm(zs[1])
    offs = [0, 27 * 3 * 16, 27 * 3 * 16 + 27 * 256, 27 * 3 * 16 + 2 * 27 * 256, gs[0].size]
    assert np.linalg.norm(gs[0] - gs[1]) <= 3e-3 * np.linalg.norm(gs[1])
    for l in range(4):
        a, b = gs[0][offs[l]:offs[l + 1]], gs[1][offs[l]:offs[l + 1]]
        assert np.linalg.norm(a - b) <= 5e-3 * np.linalg.norm(b), l
