"""The host side of building a solver: the patch lists take time in proportion to
the tets, a small multiple of the plain counting pass over the same corners
(xpbd_build_patch_csr), as a per-tet body now needs them too."""
import ctypes
import time

import numpy as np

from xpbd_gpu.mesh import kuhn_grid


def test_patch_lists_cost_a_few_passes_over_the_corners(native_lib):
    m = kuhn_grid(20, 20, 20, 0.05, jitter=0.1, seed=0)
    V, T, P = m.n_verts, m.n_tets, 256
    tt = np.ascontiguousarray(m.tets, dtype=np.int32)
    npat = -(-T // P)
    voff, pv = np.empty(npat + 1, np.int32), np.empty(4 * T, np.int32)
    lid, mx = np.zeros(npat * P, np.uint32), ctypes.c_int32()
    build, csr = [], []
    for _ in range(7):
        t = time.perf_counter()
        assert native_lib.xpbd_build_patches(tt.ctypes.data, T, V, P, voff.ctypes.data, pv.ctypes.data, lid.ctypes.data,
                                             ctypes.byref(mx)) == 0
        build.append(time.perf_counter() - t)
        start, slots = np.empty(int(voff[-1]), np.uint16), np.empty(4 * npat * P, np.uint16)
        t = time.perf_counter()
        assert native_lib.xpbd_build_patch_csr(voff.ctypes.data, lid.ctypes.data, T, P, start.ctypes.data,
                                               slots.ctypes.data) == 0
        csr.append(time.perf_counter() - t)
    # sorting every corner took 30 to 40 times as long, sorting the lists 3
    assert min(build) < 12 * min(csr), (min(build), min(csr))
    # the lists: every patch's vertices once, ascending, and each corner's place in them
    for p in (0, npat // 2, npat - 1):
        want = np.unique(tt[p * P:(p + 1) * P])
        np.testing.assert_array_equal(pv[voff[p]:voff[p + 1]], want)
        loc = lid[p * P:min(T, (p + 1) * P), None] >> (8 * np.arange(4, dtype=np.uint32)) & 0xff
        np.testing.assert_array_equal(want[loc], tt[p * P:(p + 1) * P])


def test_resident_bodies_are_those_of_the_device(monkeypatch):
    """Three patches of 256 tets per SM, as the library asks the device for it."""
    import torch
    from types import SimpleNamespace
    from xpbd_gpu import neohookean_solver as n
    for sms in (132, 148, 152, 160):
        monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device: SimpleNamespace(multi_processor_count=sms))
        assert n.resident_tets("cuda:0") == 768 * sms
