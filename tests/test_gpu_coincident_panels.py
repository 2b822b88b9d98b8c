"""Two panels of the free surface with one centre and different areas, in
different tiles of the pair kernel: each entry of the pair takes the area of its
own panel, as the entry kernel does (both float64, 1e-13 of the largest entry)."""
import numpy as np
import pytest

from capytaine_b200.meshes import Mesh, mesh_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adjoint", [True, False])
@pytest.mark.parametrize("places", [(0, 200), (130, 5), (3, 9)])
def test_concentric_panels_of_the_free_surface(places, adjoint):
    import torch
    from capytaine_b200.green_function import Delhommeau
    hull = mesh_sphere(radius=2.0, resolution=(24, 25)).immersed_part()
    faces = [list(map(int, f)) for f in hull.faces[:210]]
    square = np.array([[-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]], dtype=float)
    vertices = np.concatenate([hull.vertices, 0.25 * square, 0.5 * square])
    for i, place in enumerate(places):
        faces[place] = list(range(len(hull.vertices) + 4 * i, len(hull.vertices) + 4 * i + 4))
    mesh = Mesh(vertices, faces, clean=False)
    n = mesh.nb_faces
    assert np.array_equal(mesh.faces_centers[places[0]], mesh.faces_centers[places[1]])

    def assemble(symmetric):
        gf = Delhommeau(tabulation_cache_dir=None)
        gf.symmetric_assembly = symmetric
        S = torch.zeros((n, n), dtype=torch.complex128, device="cuda")
        K = torch.zeros_like(S)
        gf.assemble_into(mesh, mesh, S, K, wavenumber=0.9, adjoint_double_layer=adjoint, reuse_rankine=symmetric)
        return S.cpu().numpy(), K.cpu().numpy()
    for pairs, entries in zip(assemble(True), assemble(False)):
        assert np.abs(pairs - entries).max() <= 1e-13 * np.abs(entries).max()
