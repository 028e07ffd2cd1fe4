"""Tensors on PyTorch's default stream (CUDA's legacy stream): operators, solves and
penalties are ordered with the work before and after them on that stream.

Equality is exact: the same kernels run on the same values, only the order of
streams is at stake (the exact DFT's sums have a fixed order; the gridded solve is
compared with its own copy)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dft(pg, torch):
    """An operator whose application takes some milliseconds, far longer than its call."""
    from powergrid_b200 import synthetic as S
    n, nz, nc, M = 32, 32, 4, 60000
    N = n * n * nz
    r = np.random.default_rng(1)
    k = ((r.random((3, M)) - 0.5) * n).astype(np.float32)
    t = np.sort(r.random(M)).astype(np.float32) * np.float32(10e-3)
    G = pg.Gdft(M, N, *k, *S.image_coords(n, n, nz), S.field_map(S.Rng(2), n, n, nz, 60.0), t)
    A = pg.SENSE(G, S.coil_maps(S.Rng(3), n, n, nz, nc), M, N, nc)
    v = lambda m: torch.from_numpy((r.standard_normal(m) + 1j * r.standard_normal(m)).astype(np.complex64))  # noqa: E731
    return A, v(N).cuda(), v(M * nc).cuda(), G


def test_results_are_ordered_with_the_default_stream(pg):
    import torch
    A, x, y, G = _dft(pg, torch)
    for f, v in ((A.forward, x), (A.adjoint, y)):
        f(v)                                      # workspaces
        torch.cuda.synchronize()
        out = torch.zeros_like(y if f == A.forward else x)
        f(v, out=out)
        taken = out.clone()                       # on the default stream, at once
        torch.cuda.synchronize()
        assert torch.equal(torch.view_as_real(taken), torch.view_as_real(out))
        assert float(out.abs().max()) > 0


def test_inputs_are_ordered_with_the_default_stream(pg):
    import torch
    A, x, y, G = _dft(pg, torch)
    want = A * x
    torch.cuda.synchronize()
    late = torch.zeros_like(x)
    torch.cuda._sleep(20_000_000)                 # some 10 ms of the default stream
    late.copy_(x)
    got = A * late
    torch.cuda.synchronize()
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))


def test_host_calls_follow_tensor_calls(pg):
    """Both share the operator's workspaces."""
    import torch
    A, x, y, G = _dft(pg, torch)
    a, b = x.cpu().numpy(), (2 * x).cpu().numpy()
    want_a, want_b = A * a, A * b
    for _ in range(3):
        t = A * x
        h = A * b
        assert np.array_equal(h, want_b)
        assert np.array_equal(t.cpu().numpy(), want_a)


def test_solves_beside_another_threads_default_stream_work(pg):
    """The solver captures its iteration as a graph; another thread's work on the
    default stream meanwhile is no part of the capture and does not fail it."""
    import torch
    from powergrid_b200 import synthetic as S
    n = 32
    kx, ky, t = S.spiral(n, 4, 512, 8e-3)
    M, N = kx.size, n * n
    stop, bad = threading.Event(), []

    def busy():
        try:
            v = torch.zeros(1 << 16, device="cuda")
            while not stop.is_set():
                v.add_(1.0)
                v.sum().item()
        except Exception as e:                    # noqa: BLE001
            bad.append(e)

    th = threading.Thread(target=busy)
    th.start()
    try:
        for k in range(12):                       # new operators: each captures its graph
            G = pg.Gnufft(M, 2.0, n, n, 1, kx, ky, np.zeros_like(kx))
            y = torch.from_numpy((G * S.image(S.Rng(k), N)).astype(np.complex64)).cuda()
            x = torch.zeros(N, dtype=torch.complex64, device="cuda")
            it = torch.zeros(1, dtype=torch.int32, device="cuda")
            for _ in range(2):
                pg.solve_pwls_pcg_device(G, y, pg.QuadPenalty(n, n, 1, 1e-3), 8, x, iters=it)
                taken = x.clone()
                torch.cuda.synchronize()
                assert int(it) == 8
                assert torch.equal(torch.view_as_real(taken), torch.view_as_real(x))
                assert float(x.abs().max()) > 0
    finally:
        stop.set()
        th.join()
    assert not bad, bad
