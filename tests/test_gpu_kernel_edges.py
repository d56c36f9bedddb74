"""The kernels at the sizes where their splits change: P2G's two rounds of 32
cells, the cell-ordered sort list and its two scans, strains of every size,
the gather P2G's stages, long and short canonical buckets, mesh searches with
more leaves than a warp keeps, render data at partial warps.  Against the CPU oracle, with the bounds of
tests/parity.py (or bit for bit where the mode promises it)."""
import numpy as np
import pytest

from nexus_b200 import scenes
from nexus_b200.models import BoundaryCondition, ParticleModel
from nexus_b200.mpm import MpmPipeline, state_from_scene
from nexus_b200.particles import Collider, ParticleBatch, box_walls, collider_array
from tests.parity import FAST_BOUNDS, assert_run_matches, compare_sort, nodes_in_oracle_order, rel_l2, start_state

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
@pytest.mark.parametrize("deterministic", [False, True])
def test_p2g_over_cell_counts(pipe, kind, deterministic):
    from oracle.oracle import OracleScene
    counts = _counts(kind)
    sc = _cells_scene(counts)
    sc.particles.enabled[::7] = 0  # disabled particles carry nothing
    st = state_from_scene(sc, deterministic=deterministic)
    pipe.debug_sort(st, with_p2g=True)
    h, ids = st.headers(), st.sorted_ids()
    o = OracleScene(sc, "f32" if deterministic else "f64")
    o.sort()
    o.p2g()
    errs = compare_sort(h, ids, o.headers(), o.sorted_ids(), exact_order=deterministic)
    assert not errs, "\n".join(errs[:10])
    if not deterministic:  # the block's list is in cell order
        row = h[np.argmax(h[:, 4])]
        cell_of = np.repeat(np.arange(64), counts)
        listed = cell_of[ids[row[3]:row[3] + row[4]]]
        assert np.array_equal(listed, np.sort(listed))
    g = nodes_in_oracle_order(h, st.nodes(), o.headers())
    want = o.nodes()[:, :, :4]
    if deterministic:
        assert np.array_equal(g.view(np.uint32), want.view(np.uint32))
    else:
        # 32-bit sums of at most a few hundred products a node
        assert rel_l2(g[..., 3], want[..., 3]) < 1e-6
        assert rel_l2(g[..., :3], want[..., :3]) < 1e-5


@pytest.mark.parametrize("blocks", [40, 1200])
def test_p2g_shares_heavy_cells_over_a_warp(pipe, blocks):
    """Cells far fuller than their block's others, in either half of the block's cells,
    alone or several, at counts about multiples of 32; with few blocks (two warps each)
    and with many (one warp each)."""
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(23)
    at = rng.permutation(14 ** 3)[:blocks]
    pos = []
    for i, b in enumerate(at):
        lo = 4 * (1 + np.array([b % 14, b // 14 % 14, b // 196]))
        counts = rng.integers(0, 4, 64) * (rng.random(64) < 0.7)
        for c in rng.permutation(64)[:(0, 0, 0, 1, 2, 5)[i % 6]]:
            counts[c] = rng.choice([33, 63, 64, 65, 96, 127, 200])
        if i % 50 == 7:  # nothing but heavy cells
            counts = np.zeros(64, int)
            counts[[5, 40]] = [70, 161]
        cell = np.repeat(np.arange(64), counts)
        pos.append((lo + np.stack([cell & 3, (cell >> 2) & 3, cell >> 4], 1) + 0.55 + 0.9 * rng.random((len(cell), 3))) * DX)
    sc = _cells_scene(np.zeros(64, int))
    sc.particles = ParticleBatch.from_positions(np.concatenate(pos).astype(np.float32), np.float32(DX / 4), 1000.0,
                                                ParticleModel.elastic_neo_hookean(1.0e5, 0.3))
    b = sc.particles
    b.vel[:] = rng.standard_normal(b.vel.shape).astype(np.float32)
    b.aff[:] = (0.1 * rng.standard_normal(b.aff.shape)).astype(np.float32)
    b.enabled[::7] = 0
    sc.grid_capacity = 8192
    st = state_from_scene(sc)
    pipe.debug_sort(st, with_p2g=True)
    o = OracleScene(sc, "f64")
    o.sort()
    o.p2g()
    g = nodes_in_oracle_order(st.headers(), st.nodes(), o.headers())
    want = o.nodes()[:, :, :4]
    # 32-bit sums of at most a few thousand products a node
    assert rel_l2(g[..., 3], want[..., 3]) < 1e-6
    assert rel_l2(g[..., :3], want[..., :3]) < 1e-5


@pytest.mark.parametrize("model", ["elastic", "sand", "sand_neo_hookean", "snow"])
@pytest.mark.parametrize("strain", ["none", "tiny", "small", "edge", "large", "far"])
def test_strain_forms_match_the_oracle(pipe, model, strain):
    """One step from given deformation gradients: rotated, unstrained to strongly
    strained, and with stretches far apart (far)."""
    from oracle.oracle import OracleScene
    mat = {"elastic": ParticleModel.elastic(2.0e4, 0.25), "sand": ParticleModel.sand(3.5e5, 0.3),
           "sand_neo_hookean": ParticleModel.sand_neo_hookean(2.0e5, 0.3), "snow": ParticleModel.snow(1.4e5, 0.2)}[model]
    sc = _cells_scene(np.full(64, 4), model=mat)
    sc.dt = 1.0e-5
    b = sc.particles
    b.aff[:] = 0.0
    rng = np.random.default_rng(5)
    size = {"none": 0.0, "tiny": 1e-5, "small": 1e-2, "edge": 0.09, "large": 0.3, "far": 0.3}[strain]
    for p in range(b.n):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        r, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        q, r = q * np.sign(np.linalg.det(q)), r * np.sign(np.linalg.det(r))
        s = 1.0 + size * (2.0 * rng.random(3) - 1.0)
        if strain == "far":
            s[0] *= 0.05
        b.def_grad[p] = (q @ np.diag(s) @ r).T.reshape(9)
    st = state_from_scene(sc)
    pipe.step(st)
    st.synchronize()
    o32, o64 = OracleScene(sc, "f32"), OracleScene(sc, "f64")
    o32.step(1)
    o64.step(1)
    g, want, o = st.read_particles(), o64.particles(), o32.particles()
    for k in ("def_grad", "aff"):
        # no further from 64 bits than a few times the 32-bit oracle is, or float rounding of the field's scale
        scale = np.linalg.norm(want[k])
        noise = np.linalg.norm(o[k] - want[k])
        assert np.linalg.norm(g[k] - want[k]) <= 4.0 * noise + 4e-6 * scale, k
    sg, sw = g["model"].view(np.float32)[:, 1:4], want["model"].view(np.float32)[:, 1:4]
    assert np.allclose(sg, sw, rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("per_slab", [300, 600, 1500, (1, 2, 3, 5), (33, 0, 4051, 7), (1013, 1013, 1013, 1013),
                                      (1013, 1013, 1013, 1014), (1, 4095, 2, 4096)])
def test_canonical_buckets_of_every_length(pipe, per_slab):
    """A block's list sorted whole, up to 4,052 ids, and bucket by bucket above, on both
    sides of the switch, with buckets of every remainder by four and up to 4,096 ids."""
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


@pytest.mark.parametrize("vertices", [5, 21, 41])
def test_mesh_floor_of_every_fineness(pipe, vertices):
    """From a few triangles a block to more than a warp keeps (41 x 41 vertices:
    about 600 triangles within reach of a warp's nodes, each node searches alone)."""
    from oracle.oracle import OracleScene
    sc = scenes.trimesh_floor(n_side=8, steps=20)
    tri = scenes.height_field(vertices, 5, lo=0.3, hi=0.55)
    walls = box_walls(0.0, 1.0, BoundaryCondition.slip(), BoundaryCondition.slip())
    mesh = Collider.trimesh(0, len(tri), (0.0, 0.0, 0.0), BoundaryCondition.separate(0.3))
    sc.colliders = collider_array(walls + [mesh])
    sc.tri_vertices = tri.reshape(-1, 3)
    st = state_from_scene(sc)
    for _ in range(sc.steps):
        pipe.step(st)
    st.synchronize()
    o32, o64 = OracleScene(sc, "f32"), OracleScene(sc, "f64")
    o32.step(sc.steps)
    o64.step(sc.steps)
    p64 = o64.particles()
    p64["pos"] = o64.positions_f64()
    assert_run_matches(f"mesh floor {vertices}", st.read_particles(), o32.particles(), p64, start_state(sc), FAST_BOUNDS)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000])
def test_render_buffers_equal_the_records(pipe, n):
    import torch
    sc = scenes.elastic_cube(n_side=10)
    sc.particles = sc.particles.take(np.arange(n))
    st = state_from_scene(sc)
    for _ in range(2):
        pipe.step(st)
    p, d, c = (torch.zeros((n, k), device="cuda") for k in (3, 9, 4))
    torch.cuda.synchronize()
    st.prep_render(2, p.data_ptr(), d.data_ptr(), c.data_ptr())
    st.synchronize()
    rec = st.prep_readback(2)
    assert np.array_equal(p.cpu().numpy(), rec["position"])
    assert np.array_equal(c.cpu().numpy(), rec["color"])
    assert np.array_equal(d.cpu().numpy().reshape(n, 3, 3), rec["deformation"][:, :3, :3])


@pytest.mark.parametrize("capacity", [2048, 4096])
def test_step_headers_of_both_scans(pipe, capacity):
    """A step lists primaries only, by one kernel up to 2,048 blocks and by two
    above: the blocks of the full sort, the same particles in each, and the
    blocks without particles empty at the list's end."""
    sc = scenes.elastic_cube(n_side=12)
    step, full = (state_from_scene(sc, grid_capacity=capacity) for _ in range(2))
    pipe.step(step)
    pipe.debug_sort(full)
    hs, hf = step.headers(), full.headers()
    ids, ids_f = step.sorted_ids(), full.sorted_ids()
    assert len(ids) == sc.n and len(hs) == len(hf)
    by_key = {tuple(h[:3]): h for h in hf}
    at = 0
    for h in hs:
        f = by_key[tuple(h[:3])]
        assert h[3] == at and h[4] == h[5] == f[4] and h[15] == at + h[4]
        assert sorted(ids[at:at + h[4]]) == sorted(ids_f[f[3]:f[3] + f[4]])
        assert all((a < 0) == (b < 0) and (a < 0 or tuple(hs[a][:3]) == tuple(hf[b][:3])) for a, b in zip(h[16:], f[16:]))
        at += h[4]
    assert at == sc.n


@pytest.mark.parametrize("axes", [[0], [2], [0, 1], [0, 1, 2]])
def test_gather_of_positions_that_are_no_numbers(pipe, axes):
    """Deterministic P2G: a weight that is no number along one axis makes the node's
    product no number wherever the other axes' weights are zero too."""
    from oracle.oracle import OracleScene
    sc = _cells_scene(np.full(64, 2), block=(0, 0, 0))
    sc.particles.pos[37, axes] = np.nan
    st = state_from_scene(sc, deterministic=True)
    pipe.debug_sort(st, with_p2g=True)
    o = OracleScene(sc)
    o.sort()
    o.p2g()
    g, want = nodes_in_oracle_order(st.headers(), st.nodes(), o.headers()), o.nodes()[:, :, :4]
    assert np.array_equal(np.isnan(g), np.isnan(want))
    assert np.isnan(want).any()
    assert np.array_equal(np.nan_to_num(g), np.nan_to_num(want))


def test_gather_of_short_and_long_lists(pipe):
    """Deterministic P2G of blocks with no entry, a few, one chunk of the reference (64)
    or just more, primaries and extras in every proportion, bit for bit."""
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(31)
    pos = []
    for i, b in enumerate(rng.permutation(14 ** 3)[:400]):
        lo = 4 * (1 + np.array([b % 14, b // 14 % 14, b // 196]))
        n = (0, 1, 2, 3, 7, 8, 9, 31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 257)[i % 18]
        pos.append((lo + 0.5 + 4.0 * rng.random((n, 3))) * DX)
    sc = _cells_scene(np.zeros(64, int))
    sc.particles = ParticleBatch.from_positions(np.concatenate(pos).astype(np.float32), np.float32(DX / 4), 1000.0,
                                                ParticleModel.elastic_neo_hookean(1.0e5, 0.3))
    b = sc.particles
    b.vel[:] = rng.standard_normal(b.vel.shape).astype(np.float32)
    b.aff[:] = (0.1 * rng.standard_normal(b.aff.shape)).astype(np.float32)
    b.enabled[::7] = 0
    sc.grid_capacity = 4096
    st = state_from_scene(sc, deterministic=True)
    pipe.debug_sort(st, with_p2g=True)
    o = OracleScene(sc)
    o.sort()
    o.p2g()
    lists = o.headers()[:, 5]
    assert (lists <= 64).sum() > 100 and (lists > 64).sum() > 100
    g = nodes_in_oracle_order(st.headers(), st.nodes(), o.headers())
    assert np.array_equal(g.view(np.uint32), o.nodes()[:, :, :4].view(np.uint32))
