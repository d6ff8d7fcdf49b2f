"""One V-cycle at the sizes where the level kernels change form, against the
oracle's cycle on the same operator (all rows distinct): odd and mixed-parity
coarsenings (stencils of 45 to 125 points, below and above 32768 cells), levels
of a few cells, slivers, levels on both sides of the one-launch forms.

Bounds: FP64 1e-12, as for the reference's own V-cycle fixtures.  FP32: the
cycle is some hundred dependent FP32 operations per value (9 line solves per
level, rounding 6e-8, errors partly cancelling): 2e-5."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _case(dims, seed, scale=(1.0, 1.0, 1.0)):
    from lsstag_b200 import cases
    N, M, K = dims
    n = N * M * K
    r = np.random.default_rng(seed)
    i = np.arange(n)
    x, y, z = i % N, (i // N) % M, i // (N * M)
    e, f, g = (c * r.uniform(0.5, 1.5, n) for c in scale)
    e[x == N - 1] = 0.0
    f[y == M - 1] = 0.0
    g[z == K - 1] = 0.0
    P = np.zeros((7, n))
    P[4], P[5], P[6] = e, f, g
    P[2, 1:], P[1, N:], P[0, N * M:] = e[:-1], f[:-N], g[:-N * M]
    P[3] = -P.sum(axis=0)
    P[3, ::97] -= 0.5
    rp, col, val = cases.planes_to_csr(P, dims)
    return P, sp.csr_matrix((val, col, rp), shape=(n, n)), r.standard_normal(n)


DIMS = [(66, 65, 64), (52, 51, 50), (33, 17, 9), (17, 19, 21), (64, 48, 32), (16, 16, 16), (130, 6, 8), (6, 130, 10),
        (24, 20, 12), (128, 32, 16), (5, 4, 7), (96, 80, 64), (300, 6, 5), (430, 5, 6), (600, 5, 4)]


@pytest.mark.parametrize("dims", DIMS)
def test_cycle_matches_oracle(dims):
    import lsg_oracle as lo
    from lsstag_b200 import _lib as L
    from lsstag_b200 import solver as S
    P, A, b = _case(dims, 1)
    want = lo.MultiGrid(A, dims).apply(b)
    for prec, bound in ((L.FP64, 1e-12), (L.FP32, 2e-5)):
        s = S.MGFGMRES(mg_precision=prec)
        s.set_planes(P, dims)
        for _ in range(2):                   # recorded, then replayed
            got = s.precondition(b)
            assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want)
        s.close()


@pytest.mark.parametrize("schedule", ["fused", "reference"])
@pytest.mark.parametrize("scale", [(1e3, 1.0, 1.0), (1.0, 1e3, 1.0), (1.0, 1.0, 1e3)])
@pytest.mark.parametrize("dims", [(64, 48, 40), (50, 45, 36)])
def test_strongly_coupled_lines(dims, scale, schedule):
    """Lines coupled a thousand times more strongly along one direction: the
    segments' maps remember what enters them over the whole line, so the scans
    run to their end, in the fused steps and in the separate line solves."""
    import lsg_oracle as lo
    from lsstag_b200 import _lib as L
    from lsstag_b200 import solver as S
    P, A, b = _case(dims, 3, scale)
    want = lo.MultiGrid(A, dims).apply(b)
    # as above, times the lines' conditioning (about 1e3 / 1); FP32: a
    # rounding of 6e-8 times that a line solve, 6e-5, a few of which add up
    for prec, bound in ((L.FP64, 1e-10), (L.FP32, 2e-4)):
        s = S.MGFGMRES(mg_precision=prec, adlj_schedule=L.ADLJ_FUSED if schedule == "fused" else L.ADLJ_REFERENCE)
        s.set_planes(P, dims)
        got = s.precondition(b)
        s.close()
        rel = np.linalg.norm(got - want) / np.linalg.norm(want)
        print(f"{dims} {scale} {schedule} {'fp64' if prec == L.FP64 else 'fp32'}: {rel:.1e}")
        assert rel <= bound


@pytest.mark.parametrize("dims", [(32, 32, 32), (24, 20, 12), (17, 19, 21), (64, 16, 8)])
def test_gauss_seidel_cycle_matches_oracle(dims):
    import lsg_oracle as lo
    from lsstag_b200 import _lib as L
    from lsstag_b200 import solver as S
    P, A, b = _case(dims, 2)
    want = lo.MultiGridGS(A, dims).apply(b)
    for prec, bound in ((L.FP64, 1e-12), (L.FP32, 2e-5)):
        s = S.MGFGMRES(mg_precision=prec, smoother=L.SMOOTHER_RBGS, n_pre=2)
        s.set_planes(P, dims, S.Task(n_post=2))
        for _ in range(2):
            got = s.precondition(b)
            assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want)
        s.close()
