"""GPU: which form a body or a batch takes (launch_info), on both sides of every
line of the dispatch: the tests that compare two forms with each other are
only tests of both if these hold."""
import numpy as np
import pytest

from test_gpu_gang import SIZES, _kw, _mesh, _sdfs

pytestmark = pytest.mark.gpu


def _solver(mesh, **over):
    from xpbd_gpu.neohookean_solver import XPBDNeoHookeanSolver
    return XPBDNeoHookeanSolver(mesh, _sdfs(), young_modulus=2e5, poisson_ratio=0.4, density=1000.0, **_kw(**over))


def _form(s):
    i = s.launch_info()
    return i["form"], i["ctas"], i["patches_per_cta"]


# clusters of one and of two patches per CTA, the grid
FORMS = [(1, 1, 1), (1, 1, 1), (1, 2, 1), (1, 16, 1), (1, 9, 2), (1, 16, 2), (2, 35, 1)]


@pytest.mark.parametrize("dims,form", list(zip(SIZES, FORMS)))
def test_form_of_a_body(dims, form):
    s = _solver(_mesh(dims))
    assert _form(s) == form
    s.set_profiling(True)
    assert _form(s) == (0, 0, 0)
    s.set_profiling(False)
    s.constraints_iter = 0
    assert _form(s) == (0, 0, 0)


@pytest.mark.parametrize("dims,form", [((27, 26, 27), (2, 445, 1)), ((28, 26, 27), (0, 0, 0))])
def test_form_of_the_largest_resident_body_and_the_next(dims, form):
    assert _form(_solver(_mesh(dims))) == form


@pytest.mark.parametrize("over", [dict(scatter="gather"), dict(scatter="atomic"), dict(tets_per_thread=1),
                                  dict(patch_pipeline=1), dict(patch_reduce=1)])
def test_other_variants_launch_per_phase(over):
    assert _form(_solver(_mesh((9, 9, 9)), **over)) == (0, 0, 0)


def test_body_with_an_unused_vertex_launches_per_phase():
    from xpbd_gpu.mesh import TetMesh
    m = _mesh((3, 3, 3))
    assert _form(_solver(TetMesh(np.concatenate([m.points, [[0.5, 1.0, 0.5]]]), m.tets))) == (0, 0, 0)


@pytest.mark.parametrize("dims,bodies,form", [((4, 4, 4), 20, (1, 40, 1)), ((4, 4, 4), 150, (1, 300, 1)),
                                              ((4, 4, 4), 160, (2, 320, 1)), ((4, 4, 4), 228, (2, 456, 1)),
                                              ((4, 4, 4), 229, (1, 458, 1)),
                                              ((8, 8, 8), 37, (2, 444, 1)), ((8, 8, 8), 48, (0, 0, 0)),
                                              ((10, 10, 10), 19, (2, 456, 1)), ((16, 16, 16), 21, (0, 0, 0))])
def test_form_of_a_batch_of_equal_bodies(dims, bodies, form):
    from xpbd_gpu.batched import Body, XPBDBatchedSolver
    m = _mesh(dims)
    s = XPBDBatchedSolver([Body(m, young_modulus=2e5, poisson_ratio=0.4, density=1000.0)] * bodies, _sdfs(), **_kw())
    assert _form(s) == form
    if bodies != 150:  # the clusters that fit at once decide
        assert s.launch_info()["rounds"] == (2 if bodies == 229 else 1 if form[0] else 0)
    s.set_profiling(True)
    assert _form(s) == (0, 0, 0)


@pytest.mark.parametrize("dims,form", [((8, 8, 8), 1), ((11, 11, 11), 1), ((12, 12, 12), 2)])
def test_form_of_an_uneven_batch(dims, form):
    from xpbd_gpu.batched import Body, XPBDBatchedSolver
    s = XPBDBatchedSolver([Body(_mesh(d, seed=k, x=3.0 * k), young_modulus=2e5, poisson_ratio=0.4, density=1000.0)
                           for k, d in enumerate([dims, (1, 1, 1), (43, 1, 1), (5, 4, 6), (7, 6, 1)])], _sdfs(), **_kw())
    assert _form(s)[0] == form


@pytest.mark.parametrize("dims,form", [((3, 2, 2), 1), ((43, 1, 1), 1), ((9, 9, 9), 1), ((12, 12, 12), 2)])
def test_form_of_a_body_with_per_tet_materials(dims, form):
    from xpbd_gpu.differentiable import DiffSim
    m = _mesh(dims)
    sim = DiffSim(m, _sdfs(), np.full(m.n_tets, np.log(1e5)), np.full(m.n_tets, 0.4), density=1000.0, use_graphs=False,
                  **_kw())
    assert _form(sim.solver)[0] == form
    sim = DiffSim(m, _sdfs(), np.full(m.n_tets, np.log(1e5)), np.full(m.n_tets, 0.4), density=1000.0, use_graphs=False,
                  scatter="gather", **_kw())
    assert _form(sim.solver)[0] == 0


@pytest.mark.parametrize("dims", [(4, 4, 4), (18, 18, 20), (19, 18, 19), (22, 22, 22)])
@pytest.mark.parametrize("graph", [True, False])
def test_gather_overlaps_the_projection_up_to_one_cta_per_sm(dims, graph):
    """Every kernel of an iteration but the substep's first may overlap the one
    before; the gather only where the projection leaves the SMs room."""
    import torch
    s = _solver(_mesh(dims), scatter="gather", substeps_num=1, use_graph=graph)
    small = -(-s.n_tets // 256) <= torch.cuda.get_device_properties(0).multi_processor_count
    assert small == (dims in ((4, 4, 4), (18, 18, 20)))
    s.solve()
    assert s.launch_info()["overlapped"] == (4 if small else 3) * 9 - 1


@pytest.mark.parametrize("kind", ["gather", "atomic", "patch", "gradient", "gradient over the gather", "batch"])
def test_the_switch_turns_every_overlap_off(kind, monkeypatch):
    """XPBD_NO_PDL=1 when the solver is made: no launch overlaps, whatever layouts it has."""
    import torch
    from xpbd_gpu.batched import Body, XPBDBatchedSolver
    from xpbd_gpu.differentiable import DiffSim, xpbd_simulate
    counts = []
    for off in ("0", "1"):
        monkeypatch.setenv("XPBD_NO_PDL", off)
        m = _mesh((9, 9, 9) if "gradient" in kind else (28, 26, 27))
        if "gradient" in kind:
            sim = DiffSim(m, _sdfs(), np.full(m.n_tets, np.log(1e5)), np.full(m.n_tets, 0.4), density=1000.0,
                          use_graphs=False, scatter="gather" if "gather" in kind else "atomic", **_kw())
            t = [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=True)
                 for a in (m.points, np.zeros_like(m.points), np.full(m.n_tets, np.log(1e5)), np.full(m.n_tets, 0.4))]
            (xpbd_simulate(sim, *t, 1) ** 2).sum().backward()
            s = sim.solver
        elif kind == "batch":
            s = XPBDBatchedSolver([Body(m, young_modulus=2e5, poisson_ratio=0.4, density=1000.0)], _sdfs(), **_kw())
            s.solve()
        else:
            s = _solver(m, scatter=kind)
            s.solve()
        counts.append(s.launch_info()["overlapped"])
    assert counts[0] > 0 and counts[1] == 0
