"""The oversampled-FFT stage in all of its forms, and gridding edge cases.

Operators with N a multiple of 8 (up to 256, and 512; 2-D and 3-D) run the
library's own pruned FFT passes with the pre/post kernels fused in; PG_CUFFT=1 at
construction keeps the cuFFT form, which other N always take.  The own passes
have forms that the batch's shape chooses: both passes of a small 2-D grid in one
block, and the sum over an image's grids in one block, in a cluster or through
images in memory.  Every form must agree with cuFFT's and with the reference CPU
path at the supported grid sizes, and the gridding must handle the
trajectory edges the reference's clamped windows define (samples on the
-N/2 border, a single sample, all samples in one tile).

Tolerances (relative L2): operator application <= 1e-5 vs the reference CPU
path (the oracle with the reference's kernels, or its restatement), and the
two FFT forms within 2e-6 of each other.
"""
import os

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

OP_TOL = 1e-5
FORMS_TOL = 2e-6


def _ts_sense(pg, n, M, L, nc, seed, nz=1):
    from powergrid_b200 import synthetic as S
    rng = S.Rng(seed)
    inter = max(1, M // 2048)
    if nz == 1:
        kx, ky, t = S.spiral(n, inter, M // inter, 10e-3)
        kz = np.zeros_like(kx)
    else:
        kx, ky, kz, t = S.stack_of_spirals(n, nz, inter, M // inter, 10e-3)
    fm = S.field_map(rng, n, n, nz, 80.0)
    sm = S.coil_maps(rng, n, n, nz, nc)
    N = n * n * nz
    G = pg.Gnufft(kx.size, 2.0, n, n, nz, kx, ky, kz)
    A = pg.TimeSegmentation(G, fm, t, kx.size, N, L, 1, 1)
    Sg = pg.SENSE(A, sm, kx.size, N, nc)
    return (kx, ky, kz, t, fm, sm), (G, A, Sg)


def _cufft_form(build):
    old = os.environ.get("PG_CUFFT")
    os.environ["PG_CUFFT"] = "1"
    try:
        return build()
    finally:
        if old is None:
            del os.environ["PG_CUFFT"]
        else:
            os.environ["PG_CUFFT"] = old


@pytest.mark.parametrize("n", [32, 64, 128, 256, 512])
def test_own_fft_passes_match_cufft(pg, n):
    """Forward and adjoint of SENSE<TS<Gnufft>> (L=4, 2 coils) with the own FFT
    passes and with cuFFT, at grids 64^2 ... 1024^2."""
    from powergrid_b200 import synthetic as S
    M = 8192 if n <= 128 else 32768
    arrays, own = _ts_sense(pg, n, M, 4, 2, 40 + n)
    _, ref = _cufft_form(lambda: _ts_sense(pg, n, M, 4, 2, 40 + n))
    x = S.image(S.Rng(7), n * n)
    y1, y2 = own[2] * x, ref[2] * x
    e_f = rel_l2(y1, y2)
    a1, a2 = own[2] / y2, ref[2] / y2
    e_a = rel_l2(a1, a2)
    print(f"n={n}: forward {e_f:.2e}, adjoint {e_a:.2e}")
    assert e_f <= FORMS_TOL and e_a <= FORMS_TOL


@pytest.mark.parametrize("n", list(range(8, 257, 8)) + [512])
def test_own_fft_passes_every_length(pg, n):
    """Every supported length 2n (each has its own factorisation), with and
    without segments: their supports differ, and the second adjoint of a plan
    finds the grids as the first one left them."""
    from powergrid_b200 import synthetic as S
    arrays, own = _ts_sense(pg, n, 4096, 3, 2, 90 + n)
    _, ref = _cufft_form(lambda: _ts_sense(pg, n, 4096, 3, 2, 90 + n))
    x = S.image(S.Rng(7), n * n)
    for a, b in ((own[2], ref[2]), (own[0], ref[0])):
        y = b * x
        assert rel_l2(a * x, y) <= FORMS_TOL
        for _ in range(2):
            assert rel_l2(a / y, b / y) <= FORMS_TOL


@pytest.mark.parametrize("n,nz,L", [(24, 24, 1), (40, 56, 3), (104, 8, 5), (48, 24, 12)])
def test_own_fft_passes_3d_odd_factors(pg, n, nz, L):
    """3-D with lengths that are no powers of two, one segment and many."""
    from powergrid_b200 import synthetic as S
    _, own = _ts_sense(pg, n, 600, L, 3, 50 + n, nz=nz)
    _, ref = _cufft_form(lambda: _ts_sense(pg, n, 600, L, 3, 50 + n, nz=nz))
    x = S.image(S.Rng(9), n * n * nz)
    y = ref[2] * x
    assert rel_l2(own[2] * x, y) <= FORMS_TOL
    for _ in range(2):
        assert rel_l2(own[2] / y, ref[2] / y) <= FORMS_TOL


def _launches(f, v):
    from powergrid_b200 import _lib
    f(v)                                   # binning and workspaces of a first call
    before = _lib.launches()
    out = f(v)
    return out, _lib.launches() - before


# The adjoint's launches: spread, both inverse passes, and the sum of the images where
# they go through memory; 1, 2, 4 and 8 grids per image add up in one block or a
# cluster, more are shared out over images in memory (12: one each, 64 and 120: several).
@pytest.mark.parametrize("L,nc,launches", [(1, 1, 3), (2, 1, 3), (4, 1, 3), (8, 1, 3), (2, 3, 3), (4, 3, 4), (8, 8, 4),
                                           (10, 12, 4)])
def test_sums_over_an_images_grids_match_cufft(pg, L, nc, launches):
    """SENSE<TS<Gnufft>> 128^2: every form of the last inverse pass."""
    from powergrid_b200 import synthetic as S
    n = 128
    _, own = _ts_sense(pg, n, 8192, L, nc, 77)
    _, ref = _cufft_form(lambda: _ts_sense(pg, n, 8192, L, nc, 77))
    x = S.image(S.Rng(78), n * n)
    y, fwd = _launches(own[2].forward, x)
    xa, adj = _launches(own[2].adjoint, y)
    assert (fwd, adj) == (3, launches)
    assert rel_l2(y, ref[2] * x) <= FORMS_TOL and rel_l2(xa, ref[2] / y) <= FORMS_TOL


# Up to one grid per SM both passes of a grid run in one block (forward 2 launches with
# the gather; adjoint 2 with the spread, 3 where the images go through memory); a larger
# batch runs separate passes.
@pytest.mark.parametrize("n,L,nc,fwd,adj", [(32, 1, 1, 2, 2), (32, 4, 2, 2, 2), (32, 3, 2, 2, 3), (16, 8, 12, 2, 3),
                                            (32, 4, 48, 3, 4), (24, 5, 32, 3, 4)])
def test_small_grids_in_one_block_match_separate_passes(pg, n, L, nc, fwd, adj):
    """Small 2-D grids: the batch's form against one coil at a time (one block per grid)
    and against cuFFT."""
    from powergrid_b200 import synthetic as S
    arrays, own = _ts_sense(pg, n, 2048, L, nc, 31)
    _, ref = _cufft_form(lambda: _ts_sense(pg, n, 2048, L, nc, 31))
    x = S.image(S.Rng(32), n * n)
    y, lf = _launches(own[2].forward, x)
    xa, la = _launches(own[2].adjoint, y)
    assert (lf, la) == (fwd, adj)
    assert rel_l2(y, ref[2] * x) <= FORMS_TOL and rel_l2(xa, ref[2] / y) <= FORMS_TOL
    A, sm, M = own[1], arrays[5].reshape(nc, n * n), arrays[0].size
    one = [A * (c * x).astype(np.complex64) for c in sm]
    assert rel_l2(y, np.concatenate(one)) <= FORMS_TOL
    back = sum(np.conj(c) * (A / d).astype(np.complex128) for c, d in zip(sm, y.reshape(nc, M)))
    assert rel_l2(xa, back) <= FORMS_TOL


@pytest.mark.parametrize("n", [128, 256])
def test_own_fft_passes_vs_reference(pg, oracle, n):
    """Gnufft 2-D against the reference CPU path at 256^2 and 512^2 grids."""
    from powergrid_b200 import synthetic as S
    kx, ky, t = S.spiral(n, 4, 2048, 10e-3)
    kz = np.zeros_like(kx)
    M = kx.size
    G = pg.Gnufft(M, 2.0, n, n, 1, kx, ky, kz)
    ref = oracle.gnufft(0, M, n, n, 1, kx, ky, kz)
    x = S.image(S.Rng(11), n * n)
    y = (S.image(S.Rng(12), M)).astype(np.complex64)
    e_f = rel_l2(G * x, ref.forward(x))
    e_a = rel_l2(G / y, ref.adjoint(y))
    print(f"n={n}: forward {e_f:.2e}, adjoint {e_a:.2e}")
    assert e_f <= OP_TOL and e_a <= OP_TOL


@pytest.mark.parametrize("n,nz", [(8, 8), (16, 32), (32, 16), (64, 8), (128, 64)])
def test_own_fft_passes_3d_match_cufft(pg, n, nz):
    """3-D SENSE<TS<Gnufft>> (L=3, 2 coils) with the own FFT passes and with
    cuFFT, from 16 x 16 x 16 up to the 256 x 256 x 128 grid of a 128^2 x 64
    volume; the z length differs from the in-plane one in most cases."""
    from powergrid_b200 import synthetic as S
    per_plane = 1024
    _, own = _ts_sense(pg, n, per_plane, 3, 2, 70 + n + nz, nz=nz)
    _, ref = _cufft_form(lambda: _ts_sense(pg, n, per_plane, 3, 2, 70 + n + nz, nz=nz))
    x = S.image(S.Rng(9), n * n * nz)
    y1, y2 = own[2] * x, ref[2] * x
    e_f = rel_l2(y1, y2)
    e_a = rel_l2(own[2] / y2, ref[2] / y2)
    print(f"{n}x{n}x{nz}: forward {e_f:.2e}, adjoint {e_a:.2e}")
    assert e_f <= FORMS_TOL and e_a <= FORMS_TOL


@pytest.mark.parametrize("n,nz", [(16, 8), (32, 16)])
def test_own_fft_passes_3d_vs_reference(pg, oracle, n, nz):
    """Gnufft 3-D on the own FFT passes against the reference CPU path."""
    from powergrid_b200 import synthetic as S
    kx, ky, kz, t = S.stack_of_spirals(n, nz, 2, 256, 5e-3)
    M = kx.size
    G = pg.Gnufft(M, 2.0, n, n, nz, kx, ky, kz)
    ref = oracle.gnufft(0, M, n, n, nz, kx, ky, kz)
    x = S.image(S.Rng(13), n * n * nz)
    y = S.image(S.Rng(14), M)
    e_f = rel_l2(G * x, ref.forward(x))
    e_a = rel_l2(G / y, ref.adjoint(y))
    print(f"{n}x{n}x{nz}: forward {e_f:.2e}, adjoint {e_a:.2e}")
    assert e_f <= OP_TOL and e_a <= OP_TOL


def _edge_case(kind, n):
    rng = np.random.default_rng(3)
    if kind == "border":          # samples on the -N/2 edge and just inside +N/2
        k = np.linspace(-n / 2, n / 2 - 1e-3, 64).astype(np.float32)
        kx = np.concatenate([np.full(64, -n / 2, np.float32), k])
        ky = np.concatenate([k, np.full(64, -n / 2, np.float32)])
    elif kind == "single":
        kx = np.array([3.25], np.float32)
        ky = np.array([-7.5], np.float32)
    else:                         # every sample in one tile: a dense cluster
        kx = (rng.random(3000) * 2.0 - 1.0).astype(np.float32)
        ky = (rng.random(3000) * 2.0 - 1.0).astype(np.float32)
    return kx, ky, np.zeros_like(kx)


@pytest.mark.parametrize("kind", ["border", "single", "cluster"])
def test_gridding_edge_cases_vs_reference(pg, oracle, kind):
    from powergrid_b200 import synthetic as S
    n = 32
    kx, ky, kz = _edge_case(kind, n)
    M = kx.size
    G = pg.Gnufft(M, 2.0, n, n, 1, kx, ky, kz)
    ref = oracle.gnufft(0, M, n, n, 1, kx, ky, kz)
    x = S.image(S.Rng(5), n * n)
    y = S.image(S.Rng(6), M)
    e_f = rel_l2(G * x, ref.forward(x))
    e_a = rel_l2(G / y, ref.adjoint(y))
    print(f"{kind}: forward {e_f:.2e}, adjoint {e_a:.2e}")
    assert e_f <= OP_TOL and e_a <= OP_TOL


def test_adjoint_of_zero_data_is_zero(pg):
    from powergrid_b200 import synthetic as S
    n = 64
    kx, ky, t = S.spiral(n, 2, 1024, 5e-3)
    G = pg.Gnufft(kx.size, 2.0, n, n, 1, kx, ky, np.zeros_like(kx))
    x = G / np.zeros(kx.size, np.complex64)
    assert np.all(x == 0)


def test_first_application_allocates_four_buffers(pg, monkeypatch):
    """A new operator's first forward and adjoint wait for their workspaces, some 0.34 ms
    each: the forward's grids, the passes' scratch (with the images of the last inverse
    pass), the spread's queue and its grids."""
    import torch
    from powergrid_b200 import _lib
    monkeypatch.setenv("PG_AUTOTUNE", "0")
    _, own = _ts_sense(pg, 104, 4096, 4, 12, 61)
    A = own[2]
    x = torch.ones(A.n_image, dtype=torch.complex64, device="cuda")
    y = torch.ones(A.n_data, dtype=torch.complex64, device="cuda")
    out = [torch.zeros_like(y), torch.zeros_like(x)]
    _lib.load().pg_debug_fail_allocation_after(5)
    try:
        A.forward(x, out=out[0])
        A.adjoint(y, out=out[1])
    finally:
        _lib.load().pg_debug_fail_allocation_after(0)
    assert all(bool(o.abs().max() > 0) for o in out)
