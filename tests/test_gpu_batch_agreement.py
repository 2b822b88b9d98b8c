"""A frequency solved alone and in a batch: the block steps of the mixed LU and the
splits of sums follow the batch's size, so the coefficients agree to the solves'
relative residual (1e-10 mixed, 1e-13 float64) times the condition, below 100 here."""
import numpy as np
import pytest

from capytaine_b200.bodies import FloatingBody, rigid_body_dofs
from capytaine_b200.meshes import mesh_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bar", [("mixed", 1e-8), ("fp64", 1e-11)])
def test_alone_and_in_a_batch(precision, bar):
    from capytaine_b200.engine import B200Engine
    body = FloatingBody(mesh_sphere(resolution=(30, 34)).immersed_part(), rigid_body_dofs())
    omegas = np.linspace(0.8, 3.0, 30)
    engine = B200Engine(precision=precision, max_batch=30)
    together = engine.solve_frequencies(body, omegas, wave_directions=(0.0, 0.7))
    for i in (0, 13, 29):
        alone = engine.solve_frequencies(body, omegas[i:i + 1], wave_directions=(0.0, 0.7))
        for name in ("added_mass", "radiation_damping", "diffraction"):
            a, t = getattr(alone, name)[0], getattr(together, name)[i]
            assert np.abs(a - t).max() <= bar * np.abs(t).max(), name
