"""Entries at the limits of float64: collocation points that meet a quadrature
point of a panel on the free surface, points that are no numbers."""
import numpy as np
import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gf():
    from capytaine_b200.green_function import Delhommeau
    return Delhommeau(tabulation_cache_dir=None)


def _hull():
    from capytaine_b200.meshes import mesh_vertical_cylinder
    return mesh_vertical_cylinder(length=10.0, radius=2.0, resolution=(2, 12, 4)).immersed_part()


def test_point_on_a_quadrature_point_of_the_free_surface(gf):
    # 2 / r1 with r1 = 0: the vertical derivative is infinite there, nothing is a NaN
    from capytaine_b200.meshes import Mesh
    xy = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [2, 0, 0], [2, 1, 0]], dtype=float)
    lid = Mesh(xy, np.array([[0, 1, 2, 3], [1, 4, 5, 2]]), quadrature_method="Gauss-Legendre 2")
    points = lid.quadrature_points[0][0]
    assert not np.any(np.all(points == lid.faces_centers[0], axis=1))
    S, D = gf.evaluate(points, lid, wavenumber=1.0, adjoint_double_layer=False)
    assert np.all(np.isfinite(S))
    assert np.all(np.isinf(D[:, 0].real)) and np.all(np.isfinite(D[:, 1]))


@pytest.mark.parametrize("free_surface,wavenumber", [(np.inf, 1.0), (0.0, 0.0), (0.0, np.inf), (0.0, 1.0)])
@pytest.mark.parametrize("axis", [0, 2])
def test_point_that_is_no_number_is_reported(gf, axis, free_surface, wavenumber):
    points = np.array([[100.0, 0.0, -1.0], [50.0, 60.0, -2.0]])
    points[1, axis] = np.nan
    with pytest.raises(_lib.GreenFunctionEvaluationError):
        gf.evaluate(points, _hull(), free_surface=free_surface, wavenumber=wavenumber)



@pytest.mark.parametrize("depth", [np.inf, 9.0])
@pytest.mark.parametrize("free_surface,wavenumber", [(np.inf, 1.0), (0.0, 0.0), (0.0, np.inf), (0.0, 0.5)])
@pytest.mark.parametrize("points", [[[1e160, 0, -1], [0, -1e170, -2]], [[1e160, 0, -1], [3.0, 0, -2]]])
def test_points_beyond_the_range_of_squares(gf, points, free_surface, wavenumber, depth):
    if depth != np.inf and (free_surface == np.inf or wavenumber == 0.0):
        pytest.skip("refused: a finite depth without a free surface or with k h below 0.1")
    hull = _hull()
    kw = dict(free_surface=free_surface, water_depth=depth, wavenumber=wavenumber, diagonal_term_in_double_layer=False)
    S, K = gf.evaluate(np.array(points, dtype=float), hull, early_dot_product=False, **kw)
    # 1 / r, and the wave term's 1 / sqrt(r), are all that is left
    far = np.max(np.abs(points), axis=1) > 1e150
    assert np.all(np.abs(S[far]) < 1e-60) and np.all(np.abs(K[:, far]) < 1e-60)
    # a point beside them keeps its entries (other sums of a pair's terms: 1e-12 of the largest)
    if not np.all(far):
        s, k = gf.evaluate(np.array(points, dtype=float)[~far], hull, early_dot_product=False, **kw)
        assert np.abs(S[~far] - s).max() <= 1e-12 * np.abs(s).max()
        assert np.abs(K[:, ~far] - k).max() <= 1e-12 * np.abs(k).max()
