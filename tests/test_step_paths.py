"""Paths that a step can take give the same bits: the packed two-cell collision and the flat mapping of
threads to cells against one thread per cell by rows, for every dynamics, on lattices whose cell pairs
mix bulk cells with solid and bounce-back ones; fused moving walls against the link kernel."""
import numpy as np
import pytest

from openlb_b200 import lbx

pytestmark = pytest.mark.gpu

DYNAMICS = ["bgk", "trt", "smagorinsky_bgk", "forced_bgk", "smagorinsky_forced_bgk"]


def lattice(q, core, periodic, storage, dynamics, solid=0.0, bounce=0.0, lid=None, seed=11):
    """A lattice with random populations, a share `solid` of cells without dynamics behind halfway
    bounce-back links, a share `bounce` of bounce-back cells, and with `lid` a moving top layer."""
    rng = np.random.default_rng(seed)
    lat = lbx.BlockLattice(q, core, periodic, storage)
    lat.define_dynamics(dynamics, omega=1.35, magic=0.2, smagorinsky=0.14, force=(1e-4, -3e-5, 2e-5))
    full = lat.core
    mat = np.ones(full, np.int32)
    if solid:
        mat[rng.random(full) < solid] = 2
    if lid is not None:
        mat[:, -1, :] = 3
    ids = np.where(mat == 1, lbx.CELL_BULK, lbx.CELL_NONE)
    if bounce:
        ids[(rng.random(full) < bounce) & (mat == 1)] = lbx.CELL_BOUNCE_BACK
    if solid or bounce or lid is not None:
        lat.set_cell_dynamics(ids.astype(np.uint8))
    if solid or lid is not None:
        fluid = np.where(ids == lbx.CELL_BULK, 1, np.where(mat == 1, 4, mat)).astype(np.int32)
        lat.set_bouzidi_boundary(fluid, 1, (2, 3), wall_velocity=[(0, 0, 0), lid] if lid is not None else None)
    lat.set_populations((rng.random((q, lat.n_core)) - 0.5) * 1e-2)
    lat.bulk = (ids == lbx.CELL_BULK).reshape(-1)
    return lat


def populations(lat):
    out = lat.get_populations(np.float64)
    lat.close()
    return out


@pytest.mark.parametrize("dynamics", DYNAMICS)
@pytest.mark.parametrize("q,core,storage", [(19, (5, 6, 67), "f32"), (27, (4, 5, 97), "f16dev"),
                                            (9, (7, 130), "f32"), (19, (3, 4, 33), "bf16dev"),
                                            (19, (3, 4, 64), "f32"), (9, (8, 128), "f32"), (9, (5, 96), "f16dev")])
def test_packed_pairs_match_single_cells(dynamics, q, core, storage):
    """Variant 2 runs rows of a multiple of 64 cells as rows and the ragged ones flat; variant 5 runs
    them all as rows, with lanes and second cells beyond a row's end."""
    for kw in ({}, {"solid": 0.3}, {"bounce": 0.1, "solid": 0.1}):
        ref = None
        for variant, cells in ((1, 1), (2, 1), (2, 2), (5, 1), (5, 2)):
            lat = lattice(q, core, (1, 1, 1 if q != 9 else 0), storage, dynamics, **kw)
            lat.set_launch_config(variant, 32, 4, cells)
            for _ in range(6):
                lat.collide_and_stream(1)
            # cells without dynamics hold what streams into them, and a bounce-back cell beside one
            # returns it to them; variant 1 carries that across a periodic face, variant 2 does not
            f = populations(lat)[:, lat.bulk]
            assert np.isfinite(f).all()
            ref = f if ref is None else ref
            assert np.array_equal(ref, f)


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("q,core", [(19, (3, 4, 1)), (19, (2, 3, 32)), (19, (5, 7, 33)), (19, (4, 9, 161)),
                                    (27, (3, 5, 65)), (9, (5, 31)), (9, (1, 97)), (9, (40, 129))])
def test_ragged_rows_match_one_thread_per_cell(q, core, storage):
    """Rows that fill their lanes and rows that do not (the step then runs flat through the padded
    cells), periodic on all axes and on some."""
    for periodic in ((1, 1, 1), (0, 1, 0), (1, 0, 1)):
        periodic = periodic if q != 9 else (periodic[0], periodic[1], 0)
        ref = None
        for variant, block in ((1, (32, 8)), (2, (32, 4)), (2, (128, 1)), (2, (256, 1))):
            lat = lattice(q, core, periodic, storage, "bgk")
            lat.set_launch_config(variant, *block, 1)
            for _ in range(5):
                lat.collide_and_stream(1)
            f = populations(lat)
            ref = f if ref is None else ref
            assert np.array_equal(ref, f)


@pytest.mark.parametrize("storage", ["f64", "f32", "f16dev"])
@pytest.mark.parametrize("q,core", [(19, (9, 8, 34)), (19, (5, 9, 67)), (19, (5, 8, 64)), (27, (6, 7, 33)), (9, (40, 37)),
                                    (9, (35, 64))])
def test_fused_moving_walls_match_the_link_kernel(q, core, storage):
    """Links of a moving wall, fused into the step's store, against the link kernel (variant 1), with
    one and two cells a thread, by rows and flat; with a wall velocity that differs from cell to cell
    there are more wall terms than classes, and the step fuses some and leaves the others."""
    configs = ((1, 32, 8, 1), (2, 32, 8, 1), (2, 64, 4, 1), (2, 32, 4, 2), (5, 32, 8, 1), (5, 32, 4, 2))
    ref = None
    for config in configs:
        lat = lattice(q, core, (0, 0, 0), storage, "bgk", solid=0.1, lid=(0.05, 0.0, 0.01))
        lat.set_launch_config(*config)
        lat.post_process()
        for _ in range(5):
            lat.collide_and_stream(1)
        f = populations(lat)
        ref = f if ref is None else ref
        assert np.array_equal(ref, f)
    ref = None
    for config in configs:
        lat = lattice(q, core, (0, 0, 0), storage, "bgk", lid=(0.05, 0.0, 0.01))
        mat = np.ones(lat.core, np.int32)
        mat[:, -1, :] = 3
        cells, dirs, wall = lbx.build_bouzidi_links(q, lat.core, mat, 1, (3,), [(1.0, 0.0, 0.0)])
        assert len(np.unique(cells[wall != 0])) > 31
        wall = wall * (0.02 + 1e-4 * np.arange(len(cells)))
        lat.set_bouzidi_links(cells, dirs, wall)
        lat.set_launch_config(*config)
        for _ in range(5):
            lat.collide_and_stream(1)
        f = populations(lat)
        ref = f if ref is None else ref
        assert np.array_equal(ref, f)


def test_wall_terms_are_told_apart_bit_for_bit():
    """Cells whose wall terms differ in one direction only, and there by a NaN or an infinity, are of
    different classes: the fused step sends back what the link kernel does."""
    ref = None
    for config in ((1, 32, 8, 1), (2, 32, 8, 1), (2, 32, 4, 2)):
        lat = lattice(19, (12, 6, 40), (0, 0, 0), "f32", "bgk", lid=(0.05, 0.0, 0.01))
        mat = np.ones(lat.core, np.int32)
        mat[:, -1, :] = 3
        cells, dirs, wall = lbx.build_bouzidi_links(19, lat.core, mat, 1, (3,), [(0.05, 0.0, 0.01)])
        rng = np.random.default_rng(3)
        for value in (np.nan, np.inf, -0.0):
            wall[rng.choice(np.flatnonzero(wall), 4, replace=False)] = value
        lat.set_bouzidi_links(cells, dirs, wall)
        lat.set_launch_config(*config)
        lat.collide_and_stream(1)
        f = populations(lat)
        assert not np.isfinite(f).all()
        ref = f if ref is None else ref
        assert np.array_equal(ref, f, equal_nan=True)


@pytest.mark.parametrize("variant", [(2, 64, 2, 1), (2, 32, 4, 2), (5, 32, 8, 1), (5, 32, 4, 2), (1, 64, 2, 1),
                                     (0, 256, 1, 1), (3, 256, 1, 1)])
@pytest.mark.parametrize("storage", ["f64", "f16dev"])
@pytest.mark.parametrize("name", ["geo_cavity2d_d2q9_ivel_bgk_rest_f64", "geo_cavity_d3q27_ivel_trt_f64",
                                  "geo_step_d3q19_lvel_bgk_f64", "geo_channel_d3q19_lvel_lpres_f64",
                                  "geo_channel_d3q27_trt_f64"])
def test_steps_at_once_match_single_steps_with_boundary_cells(name, storage, variant):
    """Within a call a step collides the boundary cells for the next one as it rebuilds them; steps
    called one by one collide them on their own.  The last step's statistics count them either way."""
    import lbcases as L
    from test_boundaries import build_from_materials
    fx = L.load_fixture(name)
    out = []
    for chunks in ((1,) * 7, (7,), (3, 4)):
        lat = build_from_materials(fx, storage)
        lat.set_launch_config(*variant)
        lat.set_populations(np.asarray(fx["f0"], np.float64))
        for i, k in enumerate(chunks):
            lat.collide_and_stream(k, statistics=i == len(chunks) - 1)
        stats = lat.get_statistics()
        out.append((populations(lat), stats))
    for f, stats in out[1:]:
        assert np.array_equal(out[0][0], f)
        assert stats == out[0][1]
