"""ILU(0) applications at the edges of the sweeps' tiles (16 x 16 lines in y
and z, chunks of 4 steps in x), on slabs and in the natural order that tight
memory leaves, against the oracle's factorisation and triangular solves.

Bound: each entry of the two solves is a sum of at most three products and a
quotient in FP64; on these diagonally dominant rows (off-diagonals at most
0.8 of the diagonal in sum) rounding stays within a few hundred units of 1e-16
of the largest entry: 1e-13."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _planes(dims, seed):
    N, M, K = dims
    n = N * M * K
    r = np.random.default_rng(seed)
    P = r.uniform(-0.13, 0.13, (7, n))
    P[3] = r.choice([-1.0, 1.0], n) * r.uniform(1.0, 2.0, n)
    i = np.arange(n)
    x, y, z = i % N, (i // N) % M, i // (N * M)
    for k, out in zip((0, 1, 2, 4, 5, 6), (z == 0, y == 0, x == 0, x == N - 1, y == M - 1, z == K - 1)):
        P[k][out] = 0.0
    return P


@pytest.mark.parametrize("dims", [(3, 3, 3), (5, 16, 17), (17, 15, 33), (34, 16, 16), (33, 31, 18), (70, 17, 5),
                                  (4, 1030, 3)])
def test_ilu_apply_at_tile_edges(dims):
    import lsg_oracle as lo
    from lsstag_b200 import cases
    from lsstag_b200 import solver as S
    P = _planes(dims, sum(dims))
    n = P.shape[1]
    rp, col, val = cases.planes_to_csr(P, dims)
    LU = lo.ilu0(sp.csr_matrix((val, col, rp), shape=(n, n)))
    s = S.ILUFGMRES()
    s.set_planes(P, dims)
    for k in range(3):                       # repeated applications reuse the tickets and the face values
        b = np.random.default_rng(k).standard_normal(n)
        want = lo.ilu_solve(LU, b)
        got = s.precondition(b)
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    s.close()


def _application(dims, P, b):
    """One application, and the launches of a solve of two iterations."""
    from lsstag_b200 import solver as S
    s = S.ILUFGMRES()
    s.set_planes(P, dims, S.Task(eps=0.0, MAX_ITER=2))
    x = s.precondition(b)
    s.solve(b, np.zeros(b.size))
    launches = s.stats.kernel_launches
    s.close()
    return x, launches


@pytest.mark.parametrize("dims,leave", [((4, 1024, 600), 2600 << 20), ((3, 64, 1400), 420 << 20)])
def test_slabs_run_the_tiles_and_tight_memory_the_natural_order(dims, leave):
    """Grids that the tile layout pads nine- and twelvefold run the tiled
    sweeps (a solve of tens of launches, not of two per hyperplane and
    application); with less than twice the layout's memory left on the GPU
    they run in natural order: the same arithmetic, the same bits.  The
    smaller one also against the oracle, every coupling present."""
    import torch
    P = _planes(dims, 7)
    n = P.shape[1]
    planes = sum(dims) - 2
    b = np.random.default_rng(3).standard_normal(n)
    x, launches = _application(dims, P, b)
    assert launches < 100
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - leave, dtype=torch.uint8, device="cuda")
    y, launches = _application(dims, P, b)
    del hog
    torch.cuda.empty_cache()
    assert launches > 4 * planes             # two applications of two sweeps
    assert np.array_equal(x, y)
    if n < 500000:
        import lsg_oracle as lo
        from lsstag_b200 import cases
        rp, col, val = cases.planes_to_csr(P, dims)
        want = lo.ilu_solve(lo.ilu0(sp.csr_matrix((val, col, rp), shape=(n, n))), b)
        assert np.abs(y - want).max() <= 1e-13 * np.abs(want).max()


def test_rebuild_allocates_nothing():
    """A rebuild on the same grid finds every array in place: it succeeds with
    less than one vector's memory left."""
    import torch
    from lsstag_b200 import solver as S
    dims = (96, 128, 128)
    P = _planes(dims, 5)
    s = S.ILUFGMRES()
    s.set_planes(P, dims)
    b = np.random.default_rng(4).standard_normal(P.shape[1])
    x = s.precondition(b)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free // (2 << 20) * (2 << 20) - (8 << 20), dtype=torch.uint8, device="cuda")
    try:
        s.rebuildPreconditioner()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.array_equal(s.precondition(b), x)
    s.close()


def test_concurrent_contexts_give_the_same_bits():
    """Three contexts whose sweeps together have more tiles than the GPU has
    SMs, solving at once: every solve gives the bits of a solve alone (a ring
    slot released while its loads were in flight gave other values in one
    solve of fifty)."""
    import ctypes as C
    import threading

    import torch
    from lsstag_b200 import solver as S
    dims = (96, 128, 128)
    P = _planes(dims, 11)
    ctx = []
    for k in range(3):
        s = S.ILUFGMRES()
        s.set_planes(P, dims, S.Task(eps=0.0, MAX_ITER=4))
        b = torch.as_tensor(np.random.default_rng(k).standard_normal(P.shape[1]), device="cuda")
        ctx.append((s, b, torch.empty_like(b)))

    def solve(k):
        s, b, x = ctx[k]
        x.zero_()
        torch.cuda.current_stream().synchronize()
        s.ctx.check(s.ctx.lib.lsg_solve_device(s.ctx.h, C.c_void_p(b.data_ptr()), C.c_void_p(x.data_ptr()),
                                               C.byref(s.stats)))
        return x

    want = [solve(k).clone() for k in range(3)]
    differ = [0, 0, 0]

    def many(k):
        for _ in range(120):
            differ[k] += not torch.equal(solve(k), want[k])

    threads = [threading.Thread(target=many, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, _, _ in ctx:
        s.close()
    assert differ == [0, 0, 0]
