"""The resident Jacobi-PCG solve on both sides of the line between one cluster
and a cooperative grid, clusters with CTAs that have no tile, and engines on
several threads and streams at once.  As in test_gpu_resident_pcg.py the
solution is put back into the system in FP64: |b - A x| <= tol |b|, the
solver's own stopping rule, with 1e-9 for the rounding of that evaluation."""
import threading

import numpy as np
import pytest

import flip2_b200 as F
from tests.test_gpu_resident_pcg import TOL, problem, relative_residual

pytestmark = pytest.mark.gpu


def solve(shape, seed, repeat=1):
    typ, b = problem(shape, seed)
    P = F.Particles(1, mode=F.MODE_NATIVE)
    P.setDomain(0.0, 0.0, 0.0, shape[0] // 4, shape[1] // 4, shape[2] // 4, 1.0)
    P.poisson_set(typ.ravel(), b.ravel())
    out = []
    for _ in range(repeat):
        info = P.poisson_solve(method=0, tol=TOL, max_iter=4000)
        x = P.poisson_solution().reshape(typ.shape)
        out.append((info.converged, info.iters, relative_residual(typ, b, x), P.info().error_flags))
    P.close()
    return out


@pytest.mark.parametrize("shape", [
    (24, 8, 8),    # three tiles, one CTA
    (8, 72, 8),    # nine tiles, three CTAs in a cluster of four
    (32, 24, 32),  # 48 tiles, 12 CTAs in a cluster of 16
    (32, 32, 32),  # 64 tiles, 16 CTAs: the largest cluster
    (8, 8, 520),   # 65 tiles, 17 CTAs: a cooperative grid
])
def test_cluster_edges(shape):
    first, second = solve(shape, seed=sum(shape), repeat=2)
    assert first[0] == 1 and first[3] == 0 and first[2] <= TOL + 1e-9
    assert second[1] == first[1] and second[2] <= TOL + 1e-9


def test_engines_on_several_threads():
    got = {}

    def work(k):
        got[k] = solve((32, 32, 32) if k % 2 else (40, 40, 40), seed=k, repeat=3)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 4
    for k, runs in got.items():
        for converged, iters, residual, flags in runs:
            assert converged == 1 and flags == 0 and residual <= TOL + 1e-9, k
        assert len({r[1] for r in runs}) == 1
