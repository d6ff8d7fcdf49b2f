"""One V-cycle at the sizes where the level kernels change form, in both smoother
schedules, against the oracle's cycle on the same operator (all rows distinct):
odd and mixed-parity coarsenings (stencils of 45 to 125 points, below and above
32768 cells), levels of a few cells, slivers, levels on both sides of the
one-launch forms.

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
        for schedule in (L.ADLJ_FUSED, L.ADLJ_REFERENCE):
            s = S.MGFGMRES(mg_precision=prec, adlj_schedule=schedule)
            s.set_planes(P, dims)
            for _ in range(2):               # recorded, then replayed
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


def _prolong_1d(y, axis):
    """3/4 - 1/4 interpolation to twice the cells along one axis, copied at the ends."""
    y = np.moveaxis(y, axis, 0)
    lo, hi = np.concatenate([y[:1], y[:-1]]), np.concatenate([y[1:], y[-1:]])
    out = np.stack([0.25 * lo + 0.75 * y, 0.75 * y + 0.25 * hi], 1).reshape(-1, *y.shape[1:])
    return np.moveaxis(out, 0, axis)


def _unprolong_1d(x, axis):
    """y with _prolong_1d(y) = x, from the means of the cell pairs (1/8, 3/4,
    1/8; 7/8 at the ends)."""
    from scipy.linalg import solve_banded
    x = np.moveaxis(x, axis, 0)
    m = 0.5 * (x[0::2] + x[1::2])
    ab = np.full((3, m.shape[0]), 0.125)
    ab[1] = 0.75
    ab[1, 0] = ab[1, -1] = 0.875
    return np.moveaxis(solve_banded((1, 1), ab, m.reshape(m.shape[0], -1)).reshape(m.shape), 0, axis)


@pytest.mark.parametrize("dims", [(30, 20, 18), (128, 128, 66), (256, 176, 196)])
def test_prolongation_of_even_grids(dims):
    """One, four and eight coarse planes a thread, with remainders: an
    unsmoothed cycle ends with the prolongation of some coarse vector, so the
    vector read back from the pair means prolongs to it again.  FP32: rounding
    6e-8 times 8, the inverse of the means' smallest eigenvalue, a few times."""
    from lsstag_b200 import _lib as L
    from lsstag_b200 import solver as S
    N, M, K = dims
    n = N * M * K
    i = np.arange(n)
    P = np.ones((7, n))
    for k, out in zip((0, 1, 2, 4, 5, 6), (i // (N * M) == 0, i // N % M == 0, i % N == 0, i % N == N - 1,
                                           i // N % M == M - 1, i // (N * M) == K - 1)):
        P[k][out] = 0.0
    P[3] = -P.sum(axis=0) + 0.9
    b = np.random.default_rng(5).standard_normal(n)
    for prec, bound in ((L.FP64, 1e-13), (L.FP32, 5e-6)):
        s = S.MGFGMRES(mg_precision=prec)
        s.set_planes(P, dims, S.Task(n_post=0))
        x = s.precondition(b).reshape(K, M, N)
        s.close()
        y = x
        for axis in range(3):
            y = _unprolong_1d(y, axis)
        for axis in range(3):
            y = _prolong_1d(y, axis)
        assert np.linalg.norm(x) > 0 and np.linalg.norm(y - x) <= bound * np.linalg.norm(x)


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
