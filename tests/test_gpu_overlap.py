"""GPU: the launch-per-phase forms as they ship, beyond the sizes of the one-launch
form: frame graph and overlapping launches (programmatic dependent launch),
against the same kernels one after the other (XPBD_NO_PDL=1).  Positions within the
parity tolerance of two FP32 runs that differ by the order of their sums, 1e-4 of
the bounding-box diagonal; r_hat 2e-3 relative plus 2e-4 of its maximum; the
deterministic gather 1e-6 of the diagonal (only r_hat's sum, and with it omega's
last bits, depends on an order)."""
import numpy as np
import pytest

from test_gpu_gang import POS_TOL, RES_RTOL, _kw, _mesh, _sdfs

pytestmark = pytest.mark.gpu
LARGE = (28, 26, 27)  # 117,936 tets, 461 patches


def _compare(pair, positions, frames, diag, tol, hist=True):
    a, b = pair
    assert a.launch_info()["form"] == 0 and b.launch_info()["form"] == 0
    for f in range(frames):
        a.solve()
        b.solve()
        assert np.abs(positions(a) - positions(b)).max() <= tol * diag, f
    for s in pair:
        s.check_status()
    if hist:
        ha, hb = a.read_history()[..., 0].reshape(-1), b.read_history()[..., 0].reshape(-1)
        np.testing.assert_allclose(ha, hb, rtol=RES_RTOL, atol=2e-4 * hb.max())
    assert a.launch_info()["overlapped"] > 0 and b.launch_info()["overlapped"] == 0


SINGLE = dict(block={}, split=dict(block_neohookean_enable=False), precise=dict(precise_hydro=True),
              plain=dict(cheb_enable=False), plain_split=dict(cheb_enable=False, block_neohookean_enable=False),
              warm=dict(cheb_warmup=50), monitored=dict(monitor_convergence=True),
              plain_monitored=dict(cheb_enable=False, monitor_convergence=True), direct=dict(use_graph=False),
              gather=dict(scatter="gather"), gather_plain=dict(scatter="gather", cheb_enable=False),
              gather_monitored=dict(scatter="gather", monitor_convergence=True), atomic=dict(scatter="atomic"),
              atomic_split=dict(scatter="atomic", block_neohookean_enable=False))


@pytest.mark.parametrize("mode", SINGLE)
def test_single_body(mode, monkeypatch):
    from xpbd_gpu.neohookean_solver import XPBDNeoHookeanSolver
    m, pair = _mesh(LARGE), []
    for no_pdl in ("0", "1"):
        monkeypatch.setenv("XPBD_NO_PDL", no_pdl)
        s = XPBDNeoHookeanSolver(m, _sdfs(), young_modulus=2e5, poisson_ratio=0.4, density=1000.0, **_kw(**SINGLE[mode]))
        v = np.zeros((s.n_verts, 3), dtype=np.float32)
        v[:, 1] = -1.5
        v[:, 0] = 0.4 * np.sin(9.0 * m.points[:, 1])
        s.mesh.verts.v.from_numpy(v)
        pair.append(s)
    diag = float(np.linalg.norm(np.ptp(m.points, axis=0)))
    # the plain gather has no sum whose order is open
    tol = 0.0 if mode == "gather_plain" else 1e-6 if mode.startswith("gather") else POS_TOL
    _compare(pair, lambda s: s.mesh.verts.x.to_numpy(), 2, diag, tol, hist="plain" not in mode)
    if "monitored" in mode:
        for key in ("hydro_error", "dev_error"):
            u, w = (np.array([r[key] for r in s.convergence_history]) for s in pair)
            np.testing.assert_allclose(u, w, rtol=5e-3, atol=2e-4 * w.max())


BATCH = dict(block={}, split=dict(block_neohookean_enable=False), precise=dict(precise_hydro=True),
             plain=dict(cheb_enable=False), monitored=dict(monitor_convergence=True), one_tet=dict(tets_per_thread=1),
             direct=dict(use_graph=False), materials={})


@pytest.mark.parametrize("mode", BATCH)
def test_batch(mode, monkeypatch):
    from xpbd_gpu.batched import Body, XPBDBatchedSolver
    pair = []
    bodies = []
    for k, d in enumerate([(16, 16, 16), (9, 8, 7), (20, 11, 13), (16, 17, 18), (1, 1, 1), (19, 18, 17), (16, 15, 16)]):
        m = _mesh(d, seed=k, x=3.0 * k)
        mat = dict(tet_young_modulus=np.exp(np.random.default_rng(k).uniform(11, 13, m.n_tets))) if mode == "materials" else {}
        bodies.append(Body(m, young_modulus=2e5, poisson_ratio=0.3 + 0.03 * k, density=1000.0, **mat))
    for no_pdl in ("0", "1"):
        monkeypatch.setenv("XPBD_NO_PDL", no_pdl)
        s = XPBDBatchedSolver(bodies, _sdfs(), **_kw(**BATCH[mode]))
        v = np.zeros((s.n_verts, 3), dtype=np.float32)
        v[:, 1] = -1.5
        v[:, 0] = 0.4 * np.sin(9.0 * s.positions()[:, 1])
        s.set_velocities(v)
        pair.append(s)
    _compare(pair, lambda s: s.positions(), 2, 0.4, POS_TOL, hist=mode != "plain")  # the small bodies' diagonals


@pytest.mark.parametrize("scatter", ["atomic", "gather"])
@pytest.mark.parametrize("omega_grad", [True, False])
def test_gradients_beyond_the_one_launch_form(scatter, omega_grad, monkeypatch):
    """Taping launches and reverse kernels that overlap, against the same one after
    the other: gradients within 1e-3 relative, as two forwards that differ by rounding."""
    import torch
    from xpbd_gpu.differentiable import DiffSim, xpbd_simulate
    m = _mesh(LARGE, y=0.02)
    E = np.log(1e5) + 0.3 * np.random.default_rng(3).normal(size=m.n_tets)
    out = []
    for no_pdl in ("0", "1"):
        monkeypatch.setenv("XPBD_NO_PDL", no_pdl)
        sim = DiffSim(m, _sdfs(), E, np.full(m.n_tets, 0.4), omega_grad=omega_grad, scatter=scatter, density=1000.0,
                      **_kw(constraints_iter=6, cheb_warmup=2))
        assert sim.solver.launch_info()["form"] == 0
        v0 = np.zeros_like(m.points) + [0.2, -1.0, 0.1]
        t = [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=True)
             for a in (m.points, v0, E, np.full(m.n_tets, 0.4))]
        xf = xpbd_simulate(sim, *t, 1)
        (xf ** 2).sum().backward()
        out.append([xf.detach().cpu().numpy()] + [a.grad.cpu().numpy() for a in t])
        assert (sim.solver.launch_info()["overlapped"] > 0) == (no_pdl == "0")
    for u, w in zip(*out):
        assert np.isfinite(u).all()
        assert np.linalg.norm(u - w) <= 1e-3 * np.linalg.norm(w)
