"""SENSE<Gdft> where its sums run on the tensor cores (3 or more coils, at least
2^25 sample-voxel pairs, and up to 8 coils enough outputs for its CTAs), against
the sums in 64 bits.

Tolerance 2e-6 relative L2: cos and sin to 2^-21 (the fast intrinsics' bound on
[-pi, pi]), operands to 2^-23 in two 16-bit parts, sums in FP32; measured
2.6e-7.  The plain kernels below the size and coil limits meet the same bound."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 2e-6


def _inputs(M, shape, nc, seed=1, kmax=None):
    from powergrid_b200 import synthetic as S
    nx, nz = shape
    N = nx * nx * nz
    r = np.random.default_rng(seed)
    kmax = kmax or nx / 2
    k = (r.random((3, M)) * 2 - 1) * np.array([[kmax], [kmax], [nz / 2]])
    k = k.astype(np.float32)
    t = np.sort(r.random(M)).astype(np.float32) * np.float32(20e-3)
    fm = S.field_map(S.Rng(seed), nx, nx, nz, 120.0)
    sm = S.coil_maps(S.Rng(seed + 1), nx, nx, nz, nc).reshape(nc, N)
    sm = (sm * (1 + 0.1 * r.standard_normal((nc, 1)))).astype(np.complex64)
    return k, t, S.image_coords(nx, nx, nz), fm, sm


def _exact(k, t, r, fm, grad=None):
    """M x N matrix of the operator in 64 bits, by chunks of samples."""
    k, t = k.astype(np.float64), t.astype(np.float64)
    r, fm = np.stack(r).astype(np.float64), fm.astype(np.float64)
    for a in range(0, t.size, 512):
        q = slice(a, min(t.size, a + 512))
        e = np.exp(-1j * (2 * np.pi * (k[:, q].T @ r) + np.outer(t[q], fm)))
        if grad is not None:
            for d in range(3):
                e *= np.sinc(np.outer(k[d, q] / grad["n"][d], np.ones(fm.size)) + np.outer(t[q], grad["g"][d]))
        yield q, e


def _both(k, t, r, fm, sm, x, y, grad=None):
    nc, M = sm.shape[0], t.size
    fwd, adj = np.empty((nc, M), np.complex128), np.zeros((nc, x.size), np.complex128)
    xs = (sm * x).astype(np.complex128).T
    for q, e in _exact(k, t, r, fm, grad):
        fwd[:, q] = (e @ xs).T
        adj += y.reshape(nc, M)[:, q].astype(np.complex128) @ e.conj()
    return fwd.ravel(), (adj * sm.conj()).sum(0)


def _operator(pg, k, t, r, fm, sm):
    nc, N = sm.shape
    return pg.SENSE(pg.Gdft(t.size, N, *k, *r, fm, t), sm.ravel(), t.size, N, nc)


def _on_tensor_cores(pg, S, x, y):
    """Whether the forward and the adjoint run there, by their kernel launches per group of
    coils: largest entry, packing, sums, finish; the plain kernels have 3 and 2 (groups of 8)."""
    from powergrid_b200 import _lib
    nc, out = S.n_data // _samples(S), []
    for f, v, plain in ((S.forward, x, 3), (S.adjoint, y, 2)):
        before = _lib.launches()
        f(v)
        n = _lib.launches() - before
        tensor, other = 4 * -(-nc // (8 if nc <= 8 else 16)), plain * -(-nc // 8)
        assert n in (tensor, other), n
        out.append(n == tensor)
    return tuple(out)


def _samples(S):
    return S._keep[0].n_data


# outputs and inputs at the edges of tiles (128 inputs, 512 or 1024 outputs),
# padded and full coil groups, a second group
@pytest.mark.parametrize("M,shape,nc", [(8192, (16, 16), 3), (8193, (23, 8), 8), (1025, (32, 33), 4), (9999, (24, 6), 9),
                                        (2100, (26, 24), 16), (3001, (33, 11), 17), (1025, (32, 33), 9)])
def test_tensor_sums_against_64_bits(pg, M, shape, nc):
    k, t, r, fm, sm = _inputs(M, shape, nc)
    g = np.random.default_rng(2)
    N = sm.shape[1]
    assert M * N >= 1 << 25
    tensor = (M, nc) != (1025, 4)    # few outputs and coils: the plain kernels at the same size
    x = (g.standard_normal(N) + 1j * g.standard_normal(N)).astype(np.complex64)
    y = (g.standard_normal(M * nc) + 1j * g.standard_normal(M * nc)).astype(np.complex64)
    # coils of very different size share no scale
    y.reshape(nc, M)[1] *= np.float32(1e-12)
    sm[2] *= np.float32(1e15)
    S = _operator(pg, k, t, r, fm, sm)
    fwd, adj = _both(k, t, r, fm, sm, x, y)
    assert _on_tensor_cores(pg, S, x, y) == (tensor, tensor)
    got = (S * x).reshape(nc, M)
    for c in range(nc):
        assert rel_l2(got[c], fwd.reshape(nc, M)[c]) <= TOL
    assert rel_l2(S / y, adj) <= TOL


def test_tensor_sums_with_gradients(pg, oracle):
    k, t, r, fm, sm = _inputs(8190, (32, 9), 4)
    n, N, M = (32, 32, 9), sm.shape[1], t.size
    gd = []
    for off in (1, 32, 1024):   # GdftR2.cpp:62-110
        d = np.zeros(N, np.float32)
        d[off:N - off] = fm[2 * off:] - fm[:N - 2 * off]
        d[:off] = fm[off:2 * off] - fm[:off]
        d[N - off:] = fm[N - off:] - fm[N - 2 * off:N - off]
        gd.append(d)
    S = pg.SENSE(pg.GdftR2(M, N, *k, *r, fm, t, *n), sm.ravel(), M, N, 4)
    g = np.random.default_rng(3)
    x = (g.standard_normal(N) + 1j * g.standard_normal(N)).astype(np.complex64)
    y = (g.standard_normal(M * 4) + 1j * g.standard_normal(M * 4)).astype(np.complex64)
    fwd, adj = _both(k, t, r, fm, sm, x, y, dict(n=n, g=gd))
    assert _on_tensor_cores(pg, S, x, y) == (True, True)
    assert rel_l2(S * x, fwd) <= 2 * TOL    # plus the three sinc factors in FP32
    assert rel_l2(S / y, adj) <= 2 * TOL


def test_phases_past_the_fixed_point_range(pg):
    """k r of some 2^20 turns: the plain kernels, whose FP64 phase still resolves them."""
    k, t, r, fm, sm = _inputs(2200, (32, 16), 3, kmax=4e6)
    M, N = t.size, sm.shape[1]
    g = np.random.default_rng(4)
    x = (g.standard_normal(N) + 1j * g.standard_normal(N)).astype(np.complex64)
    y = (g.standard_normal(M * 3) + 1j * g.standard_normal(M * 3)).astype(np.complex64)
    S = _operator(pg, k, t, r, fm, sm)
    assert _on_tensor_cores(pg, S, x, y) == (False, False)
    fwd, adj = _both(k, t, r, fm, sm, x, y)
    assert rel_l2(S * x, fwd) <= TOL
    assert rel_l2(S / y, adj) <= TOL


def test_non_finite_data_stays_non_finite(pg):
    k, t, r, fm, sm = _inputs(8190, (32, 9), 4)
    M, N = t.size, sm.shape[1]
    S = _operator(pg, k, t, r, fm, sm)
    y = np.ones((4, M), np.complex64)
    assert _on_tensor_cores(pg, S, np.ones(N, np.complex64), y.ravel()) == (True, True)
    clean = S / y.ravel()
    assert np.isfinite(clean).all()
    for bad in (np.nan, np.inf):
        z = y.copy()
        z[1, 77] = bad
        assert not np.isfinite(S / z.ravel()).any()
    zero = S / np.zeros(4 * M, np.complex64)
    assert (zero == 0).all()


@pytest.mark.parametrize("M,N,nc,grad,want", [
    (1100, 30505, 3, 0, (False, False)), (1100, 30505, 8, 0, (False, True)), (1100, 30505, 9, 0, (True, True)),
    (700, 47935, 5, 0, (False, True)), (8192, 16385, 3, 0, (True, True)), (3472, 15376, 4, 1, (False, False)),
    (8192, 16385, 4, 1, (True, True)), (400, 83887, 8, 0, (False, False)), (400, 83887, 12, 0, (True, True))])
def test_few_outputs_or_inputs_stay_on_the_plain_kernels(pg, M, N, nc, grad, want):
    """Up to 8 coils the tensor kernel's 1024-output CTAs and whole 128-input tiles have to
    fill the GPU; measured times on both sides are beside the rule (use_tensor)."""
    g = np.random.default_rng(6)
    k = ((g.random((3, M)) - 0.5) * 32).astype(np.float32)
    r = (g.random((3, N)) - 0.5).astype(np.float32)
    t, fm = np.linspace(0, 10e-3, M).astype(np.float32), (g.random(N) * 300).astype(np.float32)
    a = (M, N, *k, *r, fm, t)
    G = pg.GdftR2(*a, N, 1, 1) if grad else pg.Gdft(*a)
    S = pg.SENSE(G, np.ones(N * nc, np.complex64), M, N, nc)
    assert _on_tensor_cores(pg, S, np.ones(N, np.complex64), np.ones(M * nc, np.complex64)) == want
