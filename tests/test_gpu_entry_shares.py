"""The entry kernel (collocation points against panels, infinite and finite
depth) at the edges of its shares: rows around a warp and a CTA, columns around
the 4 to 32 of a CTA, pairs that are all near their panel (the warp's queue fills
and empties many times), none near (it never fills) and some.  Both sides are
float64 with the same table and the same Prony terms: 1e-10 of the largest entry,
as the assembly tests.  An entry does not depend on the share it is computed in."""
import os

import numpy as np
import pytest

from capytaine_b200.meshes import Mesh, mesh_sphere

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gf(default_oracle_gf, tmp_path_factory):
    from capytaine_b200.green_function import Delhommeau
    d = str(tmp_path_factory.mktemp("table"))
    g = Delhommeau(tabulation_cache_dir=d)
    np.savez(os.path.join(d, g._cache_filename), r_range=default_oracle_gf.tabulated_r_range,
             z_range=default_oracle_gf.tabulated_z_range, values=default_oracle_gf.tabulated_integrals)
    return g


def _faces(count):
    whole = mesh_sphere(radius=2.0, resolution=(36, 60)).immersed_part()
    assert whole.nb_faces >= count
    return Mesh(whole.vertices, [list(map(int, f)) for f in whole.faces[:count]], clean=False)


def _points(rng, n, mesh, spread):
    if spread == "near":  # within seven radii of every panel, as the panels lie close together
        return mesh.faces_centers[rng.integers(0, mesh.nb_faces, n)] + rng.uniform(-0.01, 0.0, (n, 3))
    p = rng.uniform(-3.0, 3.0, (n, 3)) - [0, 0, 3.1]
    if spread == "far":
        p[:, 0] += 60.0
    return p


def _close(got, want):
    for a, b in zip(got, want):
        assert a.shape == b.shape and np.abs(a - b).max() <= 1e-10 * np.abs(b).max()


@pytest.mark.parametrize("depth", [np.inf, 9.0])
@pytest.mark.parametrize("spread", ["near", "far", "some"])
@pytest.mark.parametrize("n,N", [(1, 1), (31, 3), (32, 4), (33, 5), (127, 31), (128, 33), (129, 7), (260, 9)])
def test_edges_against_the_oracle(gf, default_oracle_gf, n, N, spread, depth):
    rng = np.random.default_rng(n + N)
    mesh = _faces(N)
    points = _points(rng, n, mesh, spread)
    kw = dict(free_surface=0.0, water_depth=depth, wavenumber=0.7, early_dot_product=False)
    for adjoint in (True, False):
        got = gf.evaluate(points, mesh, adjoint_double_layer=adjoint, **kw)
        _close(got, default_oracle_gf.evaluate(points, mesh, adjoint_double_layer=adjoint, **kw))


@pytest.mark.parametrize("depth", [np.inf, 9.0])
@pytest.mark.parametrize("N", [250, 500, 1000])  # 8, 16 and 32 columns per CTA at 61 blocks of rows; 4 at two
def test_entries_do_not_depend_on_the_share(gf, N, depth):
    rng = np.random.default_rng(N)
    mesh = _faces(N)
    points = _points(rng, 61 * 128 - 5, mesh, "some")
    kw = dict(water_depth=depth, wavenumber=0.7, early_dot_product=False, diagonal_term_in_double_layer=False)
    S, K = gf.evaluate(points, mesh, **kw)
    rows = rng.choice(len(points), 200, replace=False)
    s, k = gf.evaluate(points[rows], mesh, **kw)
    assert np.array_equal(s, S[rows]) and np.array_equal(k, K[:, rows])
