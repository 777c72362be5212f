"""Particle objects to an array: rows of floats by records, everything else as numpy converts it."""

from decimal import Decimal

import numpy as np
import pytest

from particuology_hydraulic_penalty_b200 import engine
from particuology_hydraulic_penalty_b200.psc3d import Particle3D


def _numpy(particles):
    return np.array([engine._particle_row(p) for p in particles], dtype=np.float64).reshape(-1, 10)


@pytest.mark.parametrize("count", [0, 1, 2, 257])
def test_float_particles(count):
    rng = np.random.default_rng(count)
    scale = 10.0 ** rng.integers(-300, 300, (count, 10))
    parts = [Particle3D(*r) for r in (rng.normal(size=(count, 10)) * scale).tolist()]
    got = engine.particles_array(iter(parts))
    assert got.dtype == np.float64 and got.shape == (count, 10) and got.flags.c_contiguous and got.flags.writeable
    assert got.tobytes() == _numpy(parts).tobytes()
    assert (engine._float_rows([engine._particle_row(p) for p in parts]) is not None) == (count > 0)


@pytest.mark.parametrize("where", [0, 3])
@pytest.mark.parametrize("value", [1, True, np.float64(1.5), np.float32(1.5), np.array(2.0), "1.5", Decimal("2.5"),
                                   2 ** 70, -0.0, 5e-324])
def test_other_values_convert_as_before(value, where):
    parts = [Particle3D(1.0, 2.0, 3.0, 0.5) for _ in range(5)]
    parts[where].vx = value
    assert engine.particles_array(parts).tobytes() == _numpy(parts).tobytes()


@pytest.mark.parametrize("value", [np.array([1.0]), [1.0], 1j, "x", None, float("nan"), float("inf"), b"\0" * 8])
def test_refused_values(value):
    parts = [Particle3D(1.0, 2.0, 3.0, 0.5) for _ in range(5)]
    parts[2].wy = value
    with pytest.raises((ValueError, TypeError)):
        engine.particles_array(parts)
