"""GPU: the recurrence from r_hat to rho_hat and omega (neohookean_solver.py:495-504,
:537-546) of every form that evaluates it, replayed in FP64 from the recorded
r_hat, also where a residual is infinite.

The kernels hold it in two-float numbers, whose operations err by a few units of
2^-44 (test_gpu_two_float.py).  A step of rho_hat takes three of them, one of omega
four; rho_hat's own error is damped by 0.8 per step, omega = 4 / (4 - rho^2 omega')
passes on less than omega^2 / 4 < 1 times that of omega' and 2 times rho's: 40 x 2^-44,
2.3e-12, bounds them; 1e-11 here."""
import numpy as np
import pytest

from test_gpu_gang import _kw, _mesh, _sdfs

pytestmark = pytest.mark.gpu
RTOL = 1e-11


def _replay(r, rho, warmup, rho_min=0.00001, rho_max=0.99999, beta=0.2):
    """(omega of every iteration, rho_hat after them)."""
    om, prev, out = 1.0, None, []
    with np.errstate(all="ignore"):
        for k, rk in enumerate(np.asarray(r, dtype=np.float64)):
            if prev is not None and prev > 1e-12:
                rho = (1.0 - beta) * rho + beta * np.fmax(rho_min, np.fmin(rho_max, rk / (prev + 1e-12)))
            prev = rk
            om = 1.0 if k < warmup else 2.0 / (2.0 - rho * rho) if k == warmup else 4.0 / (4.0 - rho * rho * om)
            out.append(om)
    return np.array(out), rho


def _single(dims, **over):
    from xpbd_gpu.neohookean_solver import XPBDNeoHookeanSolver
    s = XPBDNeoHookeanSolver(_mesh(dims), _sdfs(), young_modulus=2e5, poisson_ratio=0.4, density=1000.0,
                             **_kw(constraints_iter=40, **over))
    return s, lambda: s.read_history()[None], lambda: np.array([s.rho_hat])


def _batch(all_dims, **over):
    from xpbd_gpu.batched import Body, XPBDBatchedSolver
    s = XPBDBatchedSolver([Body(_mesh(d, seed=k, x=3.0 * k), young_modulus=2e5, poisson_ratio=0.4, density=1000.0)
                           for k, d in enumerate(all_dims)], _sdfs(), **_kw(constraints_iter=40, **over))
    return s, s.read_history, lambda: np.array(s.rho_hat)


SMALL = [(4, 4, 4), (1, 1, 1), (7, 5, 6)]
# what evaluates it: k_gang (clusters, grid, a batch's clusters, its grid), the update of one
# body in each variant, the update of a batch
FORMS = {
    "clusters": (1, lambda **o: _single((5, 4, 4), **o)), "grid": (2, lambda **o: _single((12, 11, 11), **o)),
    "tiles": (0, lambda **o: _single((5, 4, 4), tets_per_thread=1, **o)),
    "large tiles": (0, lambda **o: _single((28, 26, 27), **o)),
    "gather": (0, lambda **o: _single((5, 4, 4), scatter="gather", **o)),
    "atomic": (0, lambda **o: _single((5, 4, 4), scatter="atomic", **o)),
    "batch clusters": (1, lambda **o: _batch(SMALL, **o)), "batch grid": (2, lambda **o: _batch([(12, 12, 12)] + SMALL, **o)),
    "batch tiles": (0, lambda **o: _batch(SMALL, tets_per_thread=1, **o)),
    "large batch": (0, lambda **o: _batch([(16, 16, 16)] * 5 + [(9, 8, 7)], **o)),
}


def _check(rows, rho0, rho1, warmup=3, K=40):
    for b in range(len(rows)):
        rho = rho0[b]
        for s in range(rows.shape[1] // K):
            r = rows[b, s * K:(s + 1) * K]
            om, rho = _replay(r[:, 0], rho, warmup)
            np.testing.assert_allclose(r[:, 1], om, rtol=RTOL, err_msg="body %d substep %d" % (b, s))
        np.testing.assert_allclose(rho1[b], rho, rtol=RTOL)


@pytest.mark.parametrize("name", FORMS)
def test_recurrence_equals_its_replay_in_fp64(name):
    form, make = FORMS[name]
    s, rows, rho = make()
    assert s.launch_info()["form"] == form
    for _ in range(3):
        before = rho()
        s.solve()
        _check(rows(), before, rho())
    s.check_status()


def _blow_up(s):
    """Uniformly scaled bodies: det F near 1e21 and a residual beyond the range of
    FP32 squares (infinite), positions and projections finite."""
    if hasattr(s, "set_positions"):
        x = s.positions()
        s.set_positions((x - x.min(0)) * 1e7 + 1.0)
    else:
        x = s.mesh.verts.x.to_numpy()
        s.mesh.verts.x.from_numpy((x - x.min(0)) * 1e7 + 1.0)


@pytest.mark.parametrize("name", FORMS)
def test_infinite_residual_in_the_recurrence(name):
    _, make = FORMS[name]
    s, rows, rho = make(substeps_num=1, dt=1e-6, frame_dt=1e-6)
    _blow_up(s)
    before = rho()
    s.solve()
    h = rows()
    assert np.isposinf(h[:, 0, 0]).all()
    _check(h, before, rho())
    with pytest.raises(RuntimeError, match="non-finite"):
        s.check_status()


@pytest.mark.parametrize("name", FORMS)
def test_infinite_residual_meets_its_target(name):
    """inf <= target * inf: the substep ends after its first iteration."""
    _, make = FORMS[name]
    s, rows, _ = make(substeps_num=1, dt=1e-6, frame_dt=1e-6, target_rel_residual=1e-2)
    _blow_up(s)
    s.solve()
    assert np.isposinf(rows()[:, 0, 0]).all()
    assert (np.atleast_2d(s.iterations_per_substep()) == 1).all()


@pytest.mark.parametrize("name", FORMS)
def test_recorded_residuals_have_fp64_digits(name):
    """r_hat is the FP64 sum over the tet count: its last two bits are set as often as
    not.  A two-float value of 48 bits has them clear unless its parts lie apart."""
    _, make = FORMS[name]
    s, rows, _ = make(substeps_num=4)
    s.solve()
    r = rows()[:, :, 0].ravel()
    low = np.ascontiguousarray(r).view(np.uint64) & np.uint64(3)
    assert len(r) >= 160 and (low != 0).mean() > 0.5
