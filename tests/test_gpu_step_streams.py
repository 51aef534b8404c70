"""GPU: solve_step does not wait for its residual, but what the caller does next
comes after it on whatever stream, as if it had: the steps of one simulation
issued from several streams in turn, fields written and read on others."""
import time

import numpy as np
import pytest

from test_gpu_gang import _kw, _mesh, _sdfs

pytestmark = pytest.mark.gpu


def _solver(dims, **over):
    from xpbd_gpu.neohookean_solver import XPBDNeoHookeanSolver
    return XPBDNeoHookeanSolver(_mesh(dims), _sdfs(), young_modulus=2e5, poisson_ratio=0.4, density=1000.0,
                                **_kw(constraints_iter=6, **over))


def _busy(stream):
    """Some tens of milliseconds of work ahead of what follows on the stream."""
    import torch
    with torch.cuda.stream(stream):
        torch.cuda._sleep(60_000_000)


# one launch per substep (clusters, grid), launch per phase, the gather: bitwise the same in every run
@pytest.mark.parametrize("dims,scatter", [((5, 4, 4), "patch"), ((9, 9, 9), "gather")])
def test_steps_from_several_streams_in_turn(dims, scatter):
    import torch
    a, b = _solver(dims, scatter=scatter), _solver(dims, scatter=scatter)
    s = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    rest = a.mesh.verts.x.to_numpy()
    got, want, r_hat = [], [], []
    for k in range(4):
        for sol, streams, out in ((a, s, got), (b, [torch.cuda.current_stream()] * 3, want)):
            if sol is a:
                _busy(s[k % 3])
            with torch.cuda.stream(streams[k % 3]):
                sol.apply_external_forces(1 / 120)
                sol.solve_step(1 / 120)
            with torch.cuda.stream(streams[(k + 1) % 3]):
                sol.advance(1 / 120, sol.damping)
                out.append(sol.mesh.verts.x.to_torch())
            if k == 1:  # a field written on a third stream
                with torch.cuda.stream(streams[(k + 1) % 3]):
                    sol.solve_step(1 / 120)
                with torch.cuda.stream(streams[(k + 2) % 3]):
                    sol.mesh.verts.x.from_numpy(rest)
                    sol.mesh.cells.lambda_D.fill(0.0)
                    out.append(sol.mesh.verts.pred_x.to_torch())
            r_hat.append(sol.prev_r_hat)
            torch.cuda.synchronize()
    for x, y in zip(got, want):
        torch.testing.assert_close(x, y, rtol=0, atol=1e-6 if scatter == "patch" else 0)
    np.testing.assert_allclose(r_hat[0::2], r_hat[1::2], rtol=1e-3)


def test_a_field_is_read_on_another_stream():
    import torch
    a = _solver((5, 4, 4))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    _busy(s)
    with torch.cuda.stream(s):
        a.apply_external_forces(1 / 120)
        a.solve_step(1 / 120)
    lam = a.mesh.cells.lambda_D.to_numpy()  # on the default stream
    assert np.abs(lam).max() > 0.0


def test_a_capture_on_another_stream_comes_after_the_step():
    """The residual can be read, and the solver used, while another stream captures."""
    import torch
    a = _solver((5, 4, 4))
    side = torch.cuda.Stream()
    a.solve()
    torch.cuda.synchronize()
    t = time.perf_counter()
    _busy(side)  # 29 ms at the highest clock
    with torch.cuda.stream(side):
        a.apply_external_forces(1 / 120)
        a.solve_step(1 / 120)
    g, cap = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(cap):
        g.capture_begin()
        a.advance(1 / 120, a.damping)
        waited = time.perf_counter() - t
        r_hat = a.prev_r_hat
        g.capture_end()
    assert waited > 0.02 and r_hat > 0.0
    x = a.mesh.verts.x.to_torch()
    g.replay()
    torch.cuda.synchronize()
    assert not torch.equal(x, a.mesh.verts.x.to_torch())
