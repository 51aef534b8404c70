"""GPU: the reverse pass goes by what the tape recorded: vertices pinned or freed
between a forward and its backward (as for the next simulation) do not change its
gradients (1e-3 relative, the tolerance of the adjoint tests for two forwards that
differ by rounding)."""
import numpy as np
import pytest

from test_gpu_gang import _kw, _mesh, _sdfs

pytestmark = pytest.mark.gpu


# the one-launch form's tape, the launch-per-phase one, the gather
@pytest.mark.parametrize("profiled,scatter", [(False, "atomic"), (True, "atomic"), (False, "gather")])
@pytest.mark.parametrize("change", ["pin", "free"])
def test_masses_changed_before_the_backward(profiled, scatter, change):
    import torch
    from xpbd_gpu.differentiable import DiffSim, xpbd_simulate
    m = _mesh((5, 4, 4), y=0.02)
    E = np.full(m.n_tets, np.log(1e5))
    sim = DiffSim(m, _sdfs(), E, np.full(m.n_tets, 0.4), scatter=scatter, use_graphs=False, tape_memory="store", density=1000.0,
                  **_kw(constraints_iter=6, cheb_warmup=2))
    sim.solver.set_profiling(profiled)
    free = sim.solver.mesh.verts.inv_m.to_numpy()
    pinned = free.copy()
    pinned[::5] = 0.0
    masses = dict(pin=(free, pinned), free=(pinned, free))[change]
    v0 = np.zeros_like(m.points) + [0.2, -1.0, 0.1]
    grads = []
    for later in (masses[0], masses[1]):
        sim.solver.mesh.verts.inv_m.from_numpy(masses[0])
        t = [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=True)
             for a in (m.points, v0, E, np.full(m.n_tets, 0.4))]
        loss = (xpbd_simulate(sim, *t, 2) ** 2).sum()
        sim.solver.mesh.verts.inv_m.from_numpy(later)
        loss.backward()
        grads.append([a.grad.cpu().numpy() for a in t])
    for u, w in zip(*grads):
        assert np.linalg.norm(u - w) <= 1e-3 * np.linalg.norm(u)
