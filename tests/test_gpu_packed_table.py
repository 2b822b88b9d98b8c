"""The wave term from the packed table (wave_pairs_kernel, the kernel that the
engine's assemblies take) against the plain-table kernels, at the sizes where a
tile, a warp or a share of columns ends, for one wavenumber (in place) and
sweeps, both table grids and both variants.  Both sides are float64 with the
same stencil nodes, so the largest difference is a few roundings of sums of
about 60 terms of the largest entry's size: the bar is 1e-13 of it."""
import numpy as np
import pytest

from capytaine_b200.meshes import Mesh, mesh_sphere

pytestmark = pytest.mark.gpu


def _faces(count, radius=2.0):
    whole = mesh_sphere(radius=radius, resolution=(24, 25)).immersed_part()
    return Mesh(whole.vertices, [list(map(int, f)) for f in whole.faces[:count]], clean=False)


def _assemble(gf, m1, m2, ks, packed, reuse):
    import torch
    gf._device_tabulation()
    keep = gf._dev_tab_packed
    assert keep
    if not packed:
        gf._dev_tab_packed = 0
    n, N = m1.nb_faces, m2.nb_faces
    S = torch.full((len(ks), n * N), 7.0, dtype=torch.complex128, device="cuda")
    K = torch.full_like(S, 7.0)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    gf.assemble_into(m1, m2, S[0], K[0], wavenumber=ks[0], sweep=(ks, n * N, n * N), reuse_rankine=reuse,
                     nan_flag=flag)
    gf._dev_tab_packed = keep
    assert int(flag.item()) == 0
    return S.cpu().numpy(), K.cpu().numpy()


@pytest.mark.parametrize("grid", ["scaled_nemoh3", "legacy"])
@pytest.mark.parametrize("sing", ["low_freq", "high_freq"])
@pytest.mark.parametrize("n", [1, 8, 31, 33, 127, 129, 260])
def test_packed_and_plain_tables_give_the_same_matrices(n, sing, grid):
    from capytaine_b200.green_function import Delhommeau
    shape = dict(tabulation_nr=328, tabulation_nz=46, tabulation_nb_integration_points=251) \
        if grid == "legacy" else {}
    gf = Delhommeau(gf_singularities=sing, tabulation_grid_shape=grid, tabulation_cache_dir=None, **shape)
    mesh, other = _faces(n), _faces(max(1, 250 - n), radius=1.3)
    ks = [0.02, 0.9, 6.0, 45.0]  # tabulated, and past the table's end
    for m2, reuse in ((mesh, True), (mesh, False), (other, True)):  # sweep, in place, points against a mesh
        got = _assemble(gf, mesh, m2, ks, True, reuse)
        want = _assemble(gf, mesh, m2, ks, False, reuse)
        for g, w in zip(got, want):
            assert np.abs(g - w).max() <= 1e-13 * np.abs(w).max()
