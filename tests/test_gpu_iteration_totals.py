"""GPU: solve_compute_iterations over a change from a fixed count to stop mode: the
host counts fixed frames and the device the iterations of stop mode, so a fixed
frame without a residual sweep must not be in both, whatever form it took."""
import pytest

from test_gpu_gang import _kw, _mesh, _sdfs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,profiled,form", [((2, 2, 2), False, 1), ((12, 11, 11), False, 2), ((12, 11, 11), True, 0)])
def test_plain_frames_then_stop_mode(dims, profiled, form):
    from xpbd_gpu.neohookean_solver import XPBDNeoHookeanSolver
    s = XPBDNeoHookeanSolver(_mesh(dims), _sdfs(), young_modulus=2e5, poisson_ratio=0.4, density=1000.0,
                             **_kw(cheb_enable=False))
    s.set_profiling(profiled)
    assert s.launch_info()["form"] == form
    s.solve()
    s.solve()
    assert s.solve_compute_iterations == 2 * 2 * 9
    s.target_rel_residual = 0.5
    assert s.solve_compute_iterations == 2 * 2 * 9
    s.solve()
    assert s.solve_compute_iterations == 2 * 2 * 9 + int(s.iterations_per_substep().sum())
