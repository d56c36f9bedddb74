"""Fast-mode results of the models that work on the stretches of F (linear
elasticity, both sands, snow) against recorded ones: 16 steps of a sparse box of
strained, moving particles, velocities as the SVD forms with the hardware
logarithm gave them when they were recorded.  What these forms round away (the
strain of a stretch near one) shows in such a scene as 5e-5 to 1e-4 of the
velocities, so another form of the same model, nearer to 64 bits or not, changes
the results of programs; it has to keep within the 1e-5 of 32-bit sums."""
import os

import numpy as np
import pytest

from nexus_b200 import scenes
from nexus_b200.models import BoundaryCondition, ParticleModel
from nexus_b200.particles import ParticleBatch, box_walls, collider_array

RECORDED = os.path.join(os.path.dirname(os.path.abspath(__file__)), "data", "stretch_models.npz")
MATERIALS = {"elastic": (1000.0, ParticleModel.elastic(2.0e5, 0.25)),
             "sand": (2700.0, ParticleModel.sand_with_friction_angle(3.5e5, 0.3, 30.0)),
             "sand_neo_hookean": (2700.0, ParticleModel.sand_neo_hookean(3.5e5, 0.3)),
             "snow": (400.0, ParticleModel.snow(1.4e5, 0.2))}
N, DX, STEPS = 400, 1.0 / 64.0, 16


def strained_box(material):
    """About a particle a cell, falling, each with a strain of its own."""
    rng = np.random.default_rng(17)
    pos = (0.4 + 0.11 * rng.random((N, 3))).astype(np.float32)
    density, model = MATERIALS[material]
    b = ParticleBatch.from_positions(pos, np.float32(0.5 * 0.11 / N ** (1.0 / 3.0)), density, model)
    b.vel[:, 2] -= np.float32(0.5)
    b.vel += rng.random((N, 3), dtype=np.float32) * np.float32(0.1) - np.float32(0.05)
    b.def_grad += rng.random((N, 9), dtype=np.float32) * np.float32(0.008) - np.float32(0.005)
    cols = collider_array(box_walls(0.0, 1.0, BoundaryCondition.stick(), BoundaryCondition.slip()))
    return scenes.Scene("strained box", DX, 5.0e-5, (0.0, 0.0, -9.81), b, cols, STEPS, 1024)


def velocities(material):
    from nexus_b200.mpm import MpmPipeline, state_from_scene
    pipe, st = MpmPipeline(), state_from_scene(strained_box(material))
    for _ in range(STEPS):
        pipe.step(st)
    return st.read_velocities()


@pytest.mark.gpu
@pytest.mark.parametrize("material", sorted(MATERIALS))
def test_stretch_models_keep_their_results(gpu_lib, material):
    want = np.load(RECORDED)[material].astype(np.float64)
    got = velocities(material).astype(np.float64)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
