"""A program built before bem_assembly_args got its last member passes a shorter
struct: whatever lies behind it must not be taken for a pointer."""
import ctypes

import numpy as np
import pytest

from capytaine_b200 import _lib
from capytaine_b200.meshes import mesh_vertical_cylinder

pytestmark = pytest.mark.gpu

ENTRY_POINTS = ["bem_assemble", "bem_assemble_symmetric", "bem_assemble_finite_depth", "bem_assemble_rankine_part",
                "bem_assemble_wave_symmetric", "bem_assemble_wave_symmetric_batched", "bem_assemble_wave_cached"]


class _EarlierHost:
    """The library as a program with the earlier struct calls it; what lies
    behind the struct would be refused as a pointer (not 32-byte aligned)."""

    def __init__(self, lib):
        self.lib, self.calls = lib, 0

    def __getattr__(self, name):
        real = getattr(self.lib, name)
        if name not in ENTRY_POINTS:
            return real

        def call(args, *rest):
            size = _lib.AssemblyArgs.packed_table_dev.offset
            args.tabulation_grid_shape &= 1
            buf = ctypes.create_string_buffer(b"\x01" * (size + 64), size + 64)
            ctypes.memmove(buf, ctypes.byref(args), size)
            self.calls += 1
            return real(ctypes.cast(buf, ctypes.POINTER(_lib.AssemblyArgs)), *rest)
        return call


@pytest.mark.parametrize("water_depth,reuse", [(np.inf, True), (np.inf, False), (20.0, False)])
@pytest.mark.parametrize("points", [False, True])
def test_shorter_struct(monkeypatch, points, water_depth, reuse):
    import torch
    from capytaine_b200.green_function import Delhommeau
    gf = Delhommeau(tabulation_cache_dir=None)
    mesh = mesh_vertical_cylinder(length=10.0, radius=2.0, resolution=(2, 12, 4)).immersed_part()
    m1 = mesh.faces_centers[:7] + [6.0, 0.0, -1.0] if points else mesh
    n, N = (7 if points else mesh.nb_faces), mesh.nb_faces

    def assemble():
        S = torch.zeros((N, n), dtype=torch.complex128, device="cuda")
        K = torch.zeros_like(S)
        gf.assemble_into(m1, mesh, S, K, wavenumber=0.8, water_depth=water_depth, reuse_rankine=reuse)
        return S.cpu().numpy(), K.cpu().numpy()
    want = assemble()
    host = _EarlierHost(_lib.load())
    monkeypatch.setattr(_lib, "load", lambda: host)
    got = assemble()
    assert host.calls > 0
    # float64 sums of about 60 terms from the plain table and from the packed one
    for g, w in zip(got, want):
        assert np.abs(g - w).max() <= 1e-13 * np.abs(w).max()
