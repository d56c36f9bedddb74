"""The kernels at the sizes where their splits change: the gather P2G's stages and
blocks of every shape, long and short canonical buckets.  Against the CPU oracle,
bit for bit."""
import numpy as np
import pytest

from nexus_b200 import scenes
from nexus_b200.models import BoundaryCondition, ParticleModel
from nexus_b200.mpm import MpmPipeline, state_from_scene
from nexus_b200.particles import ParticleBatch, box_walls, collider_array
from tests.parity import compare_sort, nodes_in_oracle_order

pytestmark = pytest.mark.gpu

DX = 1.0 / 64.0


@pytest.fixture(scope="module")
def pipe(gpu_lib, oracle_built):
    return MpmPipeline()


def _cells_scene(counts, seed=3, block=(6, 7, 8), model=None):
    """One particle set per cell of one block: counts[c] particles in associated
    cell c (x fastest), with random velocities and affine matrices."""
    rng = np.random.default_rng(seed)
    pos = []
    for c, n in enumerate(counts):
        cell = np.array([c & 3, (c >> 2) & 3, c >> 4]) + 4 * np.array(block)
        # associated cell = round(x / dx) - 1: x / dx in (cell + 0.5, cell + 1.5)
        pos.append((cell + 0.55 + 0.9 * rng.random((n, 3))) * DX)
    pos = np.concatenate(pos).astype(np.float32)
    b = ParticleBatch.from_positions(pos, np.float32(DX / 4), 1000.0,
                                     model or ParticleModel.elastic_neo_hookean(1.0e5, 0.3))
    b.vel[:] = rng.standard_normal(b.vel.shape).astype(np.float32)
    b.aff[:] = (0.1 * rng.standard_normal(b.aff.shape)).astype(np.float32)
    cols = collider_array(box_walls(0.0, 1.0, BoundaryCondition.slip(), BoundaryCondition.slip()))
    return scenes.Scene("cells", DX, 1.0e-4, (0.0, 0.0, -9.81), b, cols, 1, 256)


def _counts(kind):
    rng = np.random.default_rng(11)
    c = np.zeros(64, int)
    if kind == "one cell":
        c[37] = 301
    elif kind == "32 cells":
        c[rng.permutation(64)[:32]] = 5
    elif kind == "33 cells":
        c[rng.permutation(64)[:33]] = rng.integers(1, 4, 33)
    elif kind == "all equal":
        c[:] = 3
    elif kind == "one heavy":
        c[:] = rng.integers(0, 9, 64)
        c[63] = 700
    elif kind == "corners":
        c[[0, 3, 12, 15, 48, 51, 60, 63]] = 1
    return c


@pytest.mark.parametrize("kind", ["one cell", "32 cells", "33 cells", "all equal", "one heavy", "corners"])
@pytest.mark.parametrize("deterministic", [True])
def test_p2g_over_cell_counts(pipe, kind, deterministic):
    from oracle.oracle import OracleScene
    counts = _counts(kind)
    sc = _cells_scene(counts)
    sc.particles.enabled[::7] = 0  # disabled particles carry nothing
    st = state_from_scene(sc, deterministic=deterministic)
    pipe.debug_sort(st, with_p2g=True)
    h, ids = st.headers(), st.sorted_ids()
    o = OracleScene(sc)
    o.sort()
    o.p2g()
    errs = compare_sort(h, ids, o.headers(), o.sorted_ids(), exact_order=deterministic)
    assert not errs, "\n".join(errs[:10])
    g = nodes_in_oracle_order(h, st.nodes(), o.headers())
    want = o.nodes()[:, :, :4]
    assert np.array_equal(g.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("per_slab", [300, 600, 1500])
def test_canonical_buckets_of_every_length(pipe, per_slab):
    """Buckets a warp sorts (up to 512 ids) and buckets the CTA sorts."""
    from oracle.oracle import OracleScene
    counts = np.zeros(64, int)
    counts[::16] = per_slab
    sc = _cells_scene(counts)
    perm = np.random.default_rng(1).permutation(sc.n)
    sc.particles = sc.particles.take(perm)
    st = state_from_scene(sc, deterministic=True)
    pipe.debug_sort(st, with_p2g=True)
    o = OracleScene(sc)
    o.sort()
    o.p2g()
    errs = compare_sort(st.headers(), st.sorted_ids(), o.headers(), o.sorted_ids(), exact_order=True)
    assert not errs, "\n".join(errs[:10])
    g = nodes_in_oracle_order(st.headers(), st.nodes(), o.headers())
    assert np.array_equal(g.view(np.uint32), o.nodes()[:, :, :4].view(np.uint32))
