"""GPU: stop mode of batches that launch per phase.  The update's listing CTAs
say which patches and vertex blocks the next iteration sweeps; a patch left
out, listed twice or listed too long moves its body.  So every body is compared
with a single-body solver run for the iteration counts that the batch
recorded (one, two and three listing CTAs, overlapping launches on and off,
frame graph and direct launches), within the parity tolerance: positions 1e-4
of the bounding-box diagonal, r_hat 2e-3 relative plus 2e-4 of its maximum.
"""
import numpy as np
import pytest

from test_gpu_stop_mode import POS_TOL, _batch_scene, _check_counts, _fixed_substeps, _sdfs, _single_for

pytestmark = pytest.mark.gpu
TARGET, K, SUBSTEPS = 2e-2, 40, 2


def _velocities(pts):
    v = np.zeros((len(pts), 3), dtype=np.float32)
    v[:, 1] = -3.0 + 0.5 * np.sin(9.0 * pts[:, 0])
    v[:, 0] = np.sin(7.0 * pts[:, 1])
    return v


def _run(bodies, compared, frames, target, floor, cap, substeps, **kw):
    """A batch's frames against the compared bodies alone, by the batch's counts."""
    from xpbd_gpu.batched import XPBDBatchedSolver
    step = dict(frame_dt=1 / 60, dt=1 / 60, substeps_num=substeps, constraints_iter=cap, cheb_enable=True, cheb_warmup=5,
                cheb_gamma=0.6666)
    batch = XPBDBatchedSolver(bodies, _sdfs(), target_rel_residual=target, residual_floor=floor, **step, **kw)
    assert batch.launch_info()["form"] == 0
    v = np.concatenate([_velocities(b.rest_pose.points) for b in bodies])
    batch.set_velocities(v)
    singles = {}
    for k in compared:
        s = _single_for(bodies[k], substeps_num=substeps, constraints_iter=cap, cheb_warmup=5)
        s.mesh.verts.v.from_numpy(v[batch.body_vert_slices[k]])
        singles[k] = s
    seen = set()
    for f in range(frames):
        batch.solve()
        counts, hist, X = batch.iterations_per_substep(), batch.read_history(), batch.positions()
        for k in range(len(bodies)):
            _check_counts(hist[k], counts[k], cap, target, floor)
        for k, s in singles.items():
            _fixed_substeps(s, counts[k], 1 / 60 / substeps)
            x = s.mesh.verts.x.to_numpy()
            diag = float(np.linalg.norm(x.max(0) - x.min(0)))
            err = np.abs(X[batch.body_vert_slices[k]] - x).max()
            assert err <= POS_TOL * diag, "frame %d body %d: %.3e" % (f, k, err / diag)
            n = int(counts[k][-1])  # the rows of the last substep
            a, b = hist[k, (substeps - 1) * cap:(substeps - 1) * cap + n, 0], s.read_history(n)[:, 0]
            np.testing.assert_allclose(a, b, rtol=2e-3, atol=max(2e-4 * b.max(), 1e-6))
        seen.update(counts.ravel().tolist())
    batch.check_status()
    assert len(seen) > 1
    return batch, counts


# bodies whose patches lie in each listing CTA's share, the first and the last
@pytest.mark.parametrize("n,patches,compared", [(21, 2016, (0, 3, 7, 20)), (22, 2112, (0, 2, 5, 10, 21)),
                                                (44, 4224, (0, 3, 6, 14, 27, 43))])
@pytest.mark.parametrize("no_pdl,graph", [("0", True), ("1", True), ("0", False)])
def test_large_batch_equals_truncated_single_bodies(n, patches, compared, no_pdl, graph, monkeypatch):
    from xpbd_gpu.batched import Body
    from xpbd_gpu.mesh import kuhn_grid
    monkeypatch.setenv("XPBD_NO_PDL", no_pdl)
    m = kuhn_grid(16, 16, 16, 0.05, origin=(0.0, 0.004, 0.0), jitter=0.1, seed=0)
    bodies = [Body(m, young_modulus=1e4 * 1.3 ** (k % 16), poisson_ratio=0.3 + 0.01 * (k % 19), total_mass=300.0)
              for k in range(n)]
    batch, _ = _run(bodies, compared, 2, TARGET, 0.0, K, SUBSTEPS, use_graph=graph)
    assert batch.n_patches == patches
    assert (batch.launch_info()["overlapped"] > 0) == (no_pdl == "0")


@pytest.mark.parametrize("no_pdl", ["0", "1"])
def test_small_bodies_launched_per_phase(no_pdl, monkeypatch):
    """Uneven bodies, one of which stops after every first iteration (free fall)."""
    monkeypatch.setenv("XPBD_NO_PDL", no_pdl)
    bodies = _batch_scene()
    _, counts = _run(bodies, range(len(bodies)), 3, 3e-2, 1e-2, 60, 3, tets_per_thread=1)
    assert counts.min() >= 1 and counts.max() <= 60
