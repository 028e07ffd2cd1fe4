"""3-D gridding at the edges of its tiles, items and windows, against the oracle.

The spread's tiles have 8 cells per axis and its items at most 512 samples,
staged 64 at a time; a window has 8 taps per axis, and samples of one window
are summed before they reach the tile.  Tolerance: 1e-5 relative L2, the
operator tolerance of the other parity tests (float windows and tables; the
sums themselves are 32-bit)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

OP_TOL = 1e-5


def _trajectory(kind, n, nz):
    r = np.random.default_rng(5)
    if kind == "cluster":        # many samples per tile: several items, runs of equal windows
        k = r.random((3, 3000)) * 1.5 - 0.75
        k[:, ::7] = k[:, :1]
    elif kind == "stack":        # one in-plane position over all kz, on and off the grid's planes
        k = np.stack([np.full(4 * nz, 1.3), np.full(4 * nz, -2.6), np.linspace(-nz / 2, nz / 2 - 0.25, 4 * nz)])
    elif kind == "tile_edges":   # window starts on both sides of every tile edge
        c = (np.arange(2 * n) / 2.0 - n / 2)[:, None] + np.array([-0.01, 0.0, 0.01])
        c = np.clip(c.ravel(), -n / 2, n / 2 - 0.01)
        k = np.stack([c, r.permutation(c), r.random(c.size) * (nz - 0.1) - nz / 2])
    else:                        # the border of k-space, and samples whose window is cut or lies past the grid
        e = np.array([-1.0, -0.999, 0.98, 0.999, 1.0, 1.02, 1.04])
        g = np.stack(np.meshgrid(e * n / 2, e * n / 2, e * nz / 2, indexing="ij")).reshape(3, -1)
        k = g
    return k.astype(np.float32)


@pytest.mark.parametrize("n,nz,kind", [(16, 8, "cluster"), (16, 8, "stack"), (24, 9, "tile_edges"), (88, 8, "border"),
                                       (16, 16, "border")])
def test_gridding_3d_vs_oracle(pg, oracle, n, nz, kind):
    from powergrid_b200 import synthetic as S
    kx, ky, kz = _trajectory(kind, n, nz)
    M, N = kx.size, n * n * nz
    G, ref = pg.Gnufft(M, 2.0, n, n, nz, kx, ky, kz), oracle.gnufft(0, M, n, n, nz, kx, ky, kz)
    x, y = S.image(S.Rng(3), N), S.image(S.Rng(4), M)
    assert rel_l2(G * x, ref.forward(x)) <= OP_TOL
    for _ in range(2):           # the second adjoint finds the grids as the first one left them
        assert rel_l2(G / y, ref.adjoint(y)) <= OP_TOL


@pytest.mark.parametrize("L,interp,nc", [(1, 1, 1), (1, 1, 2), (1, 1, 5), (4, 1, 1), (4, 1, 3), (3, 2, 2), (2, 1, 9)])
def test_gridding_3d_planes_vs_oracle(pg, oracle, L, interp, nc):
    """Every number of planes per item: window widths K = 1, 2, 3 and odd coil counts."""
    from powergrid_b200 import synthetic as S
    n, nz = 16, 8
    kx, ky, kz, t = S.stack_of_spirals(n, nz, 2, 200, 8e-3)
    M, N = kx.size, n * n * nz
    fm, sm = S.field_map(S.Rng(1), n, n, nz, 60.0), S.coil_maps(S.Rng(2), n, n, nz, nc)
    A, Ao = pg.Gnufft(M, 2.0, n, n, nz, kx, ky, kz), oracle.gnufft(0, M, n, n, nz, kx, ky, kz)
    if L > 1:
        A = pg.TimeSegmentation(A, fm, t, M, N, L, interp, 1)
        Ao = oracle.timeseg(Ao, fm, t, M, N, L) if interp == 1 else None
    x, y = S.image(S.Rng(3), N), S.image(S.Rng(4), M * nc)
    Sg = pg.SENSE(A, sm, M, N, nc)
    if Ao is None:               # dense windows: forward and adjoint are each other's transpose
        a, b = np.vdot(Sg * x, y), np.vdot(x, Sg / y)
        assert abs(a - b) <= OP_TOL * abs(a) + 1e-6 * np.linalg.norm(Sg * x) * np.linalg.norm(y)
        return
    So = oracle.sense(Ao, sm, M, N, nc)
    assert rel_l2(Sg * x, So.forward(x)) <= OP_TOL
    assert rel_l2(Sg / y, So.adjoint(y)) <= OP_TOL


@pytest.mark.parametrize("L,nc", [(1, 1), (1, 4), (4, 3)])
def test_spread_hands_cells_between_lanes(pg, oracle, L, nc):
    """Windows that move by one cell from sample to sample, in every direction: each
    cell of the tile passes between the lanes that add to it."""
    from powergrid_b200 import synthetic as S
    n, nz = 16, 8
    c = (np.arange(-20, 20) / 10.0).astype(np.float32)      # 8 windows per axis, several samples in each
    kx, ky = (a.ravel() for a in np.meshgrid(c, c, indexing="ij"))
    kz = np.resize(np.float32([-0.6, -0.1, 0.3]), kx.size)
    t = np.linspace(0, 8e-3, kx.size).astype(np.float32)
    M, N = kx.size, n * n * nz
    fm, sm = S.field_map(S.Rng(5), n, n, nz, 60.0), S.coil_maps(S.Rng(6), n, n, nz, nc)
    A, Ao = pg.Gnufft(M, 2.0, n, n, nz, kx, ky, kz), oracle.gnufft(0, M, n, n, nz, kx, ky, kz)
    if L > 1:
        A, Ao = pg.TimeSegmentation(A, fm, t, M, N, L, 1, 1), oracle.timeseg(Ao, fm, t, M, N, L)
    Sg, So = pg.SENSE(A, sm, M, N, nc), oracle.sense(Ao, sm, M, N, nc)
    y = S.image(S.Rng(7), M * nc)
    want = So.adjoint(y)
    for _ in range(3):
        assert rel_l2(Sg / y, want) <= OP_TOL


def test_tuning_skips_what_the_3d_spread_ignores(pg):
    """The first operator of a shape times its candidates.  The 3-D spread has no choice of
    coils per item: one adjoint per bin size and repetition, none per number of coils."""
    from powergrid_b200 import _lib, synthetic as S
    n, nz, nc = 40, 24, 4
    kx, ky, kz, t = S.stack_of_spirals(n, nz, 1, 150, 8e-3)
    M, N = kx.size, n * n * nz
    sm = S.coil_maps(S.Rng(2), n, n, nz, nc)
    counts = []
    for _ in range(2):                     # a search, then its result from the cache
        G = pg.Gnufft(M, 2.0, n, n, nz, kx, ky, kz)
        before = _lib.launches()
        Sg = pg.SENSE(G, sm, M, N, nc)
        counts.append(_lib.launches() - before)
    x = S.image(S.Rng(3), N)
    fwd, adj = [_count(_lib, f, v) for f, v in ((Sg.forward, x), (Sg.adjoint, S.image(S.Rng(4), M * nc)))]
    builds = 4 * 14                        # at most 14 launches per binning, one per bin size and the default
    assert counts[0] <= 3 * 3 * (fwd + adj) + 3 * 9 * fwd + builds < 3 * 3 * (fwd + adj) + 3 * 9 * (fwd + adj)
    assert counts[1] <= 14


def _count(_lib, f, v):
    f(v)
    before = _lib.launches()
    f(v)
    return _lib.launches() - before


@pytest.mark.parametrize("M", [1000, 56800, 56900, 113600, 113700])
def test_item_sizes_vs_oracle(pg, oracle, M):
    """Items of 64, 128 and 256 samples (the rule's steps for one coil), full and ragged: half of
    the samples share the central tiles, as in a radial stack."""
    from powergrid_b200 import synthetic as S
    n, nz = 16, 8
    r = np.random.default_rng(8)
    k = (r.random((3, M)) - 0.5) * np.array([[n], [n], [nz]]) * 0.99
    k[:, ::2] *= 0.1
    kx, ky, kz = k.astype(np.float32)
    G, ref = pg.Gnufft(M, 2.0, n, n, nz, kx, ky, kz), oracle.gnufft(0, M, n, n, nz, kx, ky, kz)
    x, y = S.image(S.Rng(9), n * n * nz), S.image(S.Rng(10), M)
    # one coil is built untuned; SENSE over it takes the items of four coils
    Sg = pg.SENSE(G, np.ones(4 * x.size, np.complex64), M, x.size, 4)
    want = ref.adjoint(y)
    assert rel_l2(G * x, ref.forward(x)) <= OP_TOL
    assert rel_l2(G / y, want) <= OP_TOL
    assert rel_l2(Sg / np.tile(y, 4), 4 * want) <= OP_TOL
