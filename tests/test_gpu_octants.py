"""Octant subsampling (power-of-two grids from 8 to 128) at the sizes where its
units change shape: the smallest and largest grids, children split in parts,
leaves of more points than one unit's ranks hold, points without a cell proof,
and points that two levels put on different sides of an octant boundary.
Compared with the CPU oracle bit for bit."""
import numpy as np
import pytest

from helpers import case_from_points, compare_results, make_case, run_gpu, run_oracle

pytestmark = pytest.mark.gpu

MODES = {
    "first": dict(),
    "first_intra": dict(intra=True),
    "first_inter": dict(inter=True),
    "first_weighted": dict(inter=True, weighting=True),
    "random": dict(random=True),
    "random_intra": dict(random=True, intra=True),
    "random_inter": dict(random=True, inter=True),
    "random_weighted": dict(random=True, inter=True, weighting=True),
}


def points(name, n=60_000, seed=3):
    rng = np.random.default_rng(seed)
    if name == "volume":        # occupied cells in every direction, every octant
        xyz = rng.random((n, 3))
    elif name == "corner":      # most points in one leaf of the smallest tree
        xyz = rng.random((n, 3))
        xyz[: n * 4 // 5] *= 0.45
    elif name == "plane":       # cells along both sides of an octant boundary
        xyz = rng.random((n, 3))
        xyz[:, 0] = 0.5 + (xyz[:, 0] - 0.5) * 0.02
    elif name == "one_octant":  # nodes with a single child
        xyz = rng.random((n, 3)) * 0.1 + 0.6
    return xyz, rng.integers(0, 256, (n, 3), dtype=np.uint8)


def check(case, cfg, passes=None):
    ref = run_oracle(case, cfg)
    s = run_gpu(case, cfg)
    compare_results(ref, s)
    # (a staging area that was too small also repeats the pass)
    assert passes is None or s.stats()["subsample_passes"] == passes
    s.close()


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("shape,cloud_type,n,chunk,sub,threshold", [
    ("volume", 0, 60_000, 16, 8, 300), ("volume", 1, 60_000, 16, 128, 300), ("plane", 0, 60_000, 32, 64, 400),
    ("one_octant", 1, 20_000, 64, 16, 200), ("corner", 0, 200_000, 2, 128, 20_000),
    ("corner", 1, 150_000, 8, 32, 5_000)])
def test_units(shape, cloud_type, n, chunk, sub, threshold, mode):
    xyz, rgb = points(shape, n)
    case = case_from_points(xyz * 50.0, rgb, cloud_type, scale=0.001, bbox=[0, 0, 0, 50.5, 50.5, 50.5])
    check(case, dict(chunk_grid=chunk, sub_grid=sub, merge_threshold=threshold, **MODES[mode]))


@pytest.mark.parametrize("sub", [4, 100, 256])
def test_other_grids(sub):
    """Grids that octant subsampling does not take."""
    case = make_case(0, 1, 40_000, seed=8)
    check(case, dict(chunk_grid=32, sub_grid=sub, merge_threshold=600, inter=True))


def middle_sides(p, mn, side, sub):
    """Whether the counting grid (512) and the grid of the root's upper child put x coordinates p in the upper half of
    that child (the binary64 formula)."""
    cubic = (mn + side) - mn
    m1 = mn + cubic / 2
    count = np.floor((p - mn) / (cubic / 512)) >= 384
    child = np.floor((p - m1) / (((m1 + cubic / 2) - m1) / sub)) >= sub // 2
    return count, child


@pytest.mark.parametrize("mode", ["first", "first_inter", "random_intra", "random_weighted"])
def test_points_on_an_octant_boundary(mode):
    """Points at the middle of a node whose formula puts them on the other side than the counting grid's."""
    rng = np.random.default_rng(12)
    side = 100.0
    for _ in range(4000):
        mn = float(rng.uniform(-60, 100))
        p = np.array([mn + side * 0.75])
        for _ in range(6):
            p = np.unique(np.concatenate([p, np.nextafter(p, -np.inf), np.nextafter(p, np.inf)]))
        a, b = middle_sides(p, mn, side, 128)
        if (a != b).any():
            break
    assert (a != b).any()
    n = 100_000
    xyz = rng.random((n, 3)) * side
    xyz[:, 0] += mn
    xyz[:64, 0] = p[a != b][0]
    rgb = rng.integers(0, 256, (n, 3), dtype=np.uint8)
    case = case_from_points(xyz, rgb, 1, scale=0.01, bbox=[mn, 0, 0, mn + side, side, side])
    check(case, dict(chunk_grid=512, sub_grid=128, merge_threshold=1000, output_factor=12.0, **MODES[mode]), passes=2)


def test_grids_in_turn_on_one_session():
    """One session through grids of both kinds and back: they share the scratch buffers."""
    from helpers import octree_api

    case = make_case(1, 0, 80_000, seed=31)
    s = octree_api.OctreeSession(0)
    s.set_cloud(case.cloud, n=case.n, stride=case.stride, cloud_type=case.cloud_type, scale=case.scale,
                bb_min=case.bb_min, bb_max=case.bb_max)
    for sub, mode in ((64, "first_inter"), (100, "random_weighted"), (32, "random_weighted"), (64, "first")):
        cfg = dict(chunk_grid=64, sub_grid=sub, merge_threshold=1000, **MODES[mode])
        s.configure(**cfg)
        s.init()
        s.generate()
        compare_results(run_oracle(case, cfg), s)
    s.close()


def test_pyramid_left_zero_between_builds():
    """Builds in turn that find the count pyramid zero, or not: a dense one with a pyramid large enough to be zeroed
    beside subsampling, again on the same state, a small dense grid, the sparse kind, and back."""
    from helpers import octree_api

    case = make_case(1, 1, 1_100_000, seed=41)
    s = octree_api.OctreeSession(0)
    s.set_cloud(case.cloud, n=case.n, stride=case.stride, cloud_type=case.cloud_type, scale=case.scale,
                bb_min=case.bb_min, bb_max=case.bb_max)
    want = {}
    for grid in (256, 256, 64, 512, 256, 64):
        cfg = dict(chunk_grid=grid, sub_grid=64, merge_threshold=20_000)
        s.configure(**cfg)
        s.init()
        for _ in range(2):
            s.generate()
            if grid not in want:
                want[grid] = run_oracle(case, cfg)
            compare_results(want[grid], s)
    s.close()


@pytest.mark.parametrize("n", [500, 60_000])
@pytest.mark.parametrize("grid", [2, 4, 8, 16, 32, 64, 128, 256])
def test_pyramid_levels(grid, n):
    """Counts of every level and the number of occupied cells, where the pyramid's top (32^3 cells and fewer) is the
    whole of it, starts after one or two launches, and for sparse and dense clouds."""
    xyz, rgb = points("volume", n)
    case = case_from_points(xyz * 50.0, rgb, 1, scale=0.001, bbox=[0, 0, 0, 50.5, 50.5, 50.5])
    cfg = dict(chunk_grid=grid, sub_grid=32, merge_threshold=300)
    ref = run_oracle(case, cfg, keep_levels=True)
    s = run_gpu(case, dict(cfg, debug=1))
    assert s.stats()["sparse_nodes"] == ref.stats["sparse_nodes"]
    level, g = 0, grid
    while g >= 1:
        np.testing.assert_array_equal(s.level_counts(level, g), ref.level_counts[level])
        level, g = level + 1, g // 2
    s.close()


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("n,chunk,sub", [(60_000, 16, 32), (150_000, 64, 128)])
def test_wait_that_runs_out(n, chunk, sub, mode):
    """A unit that gives up waiting for its node's earlier ones ends the call with an error, and nothing after it reads
    what it left (levels of both kinds: with colours spread over blocks, and not); the session goes on."""
    from helpers import octree_api

    xyz, rgb = points("volume", n)
    case = case_from_points(xyz * 50.0, rgb, 1, scale=0.001, bbox=[0, 0, 0, 50.5, 50.5, 50.5])
    cfg = dict(chunk_grid=chunk, sub_grid=sub, merge_threshold=300, output_factor=12.0, **MODES[mode])
    s = octree_api.OctreeSession(0)
    s.set_cloud(case.cloud, n=case.n, stride=case.stride, cloud_type=case.cloud_type, scale=case.scale,
                bb_min=case.bb_min, bb_max=case.bb_max)
    out = np.zeros(12 * n * 18, np.uint8), np.zeros(12 * n, np.uint32)
    s.set_output_host(*out)
    s.configure(debug=2, **cfg)
    s.init()
    for _ in range(2):
        with pytest.raises(octree_api.OctreeError, match="wait on the device"):
            s.generate()
    s.configure(**cfg)
    s.init()
    s.generate()
    compare_results(run_oracle(case, cfg), s)
    s.close()


def foreign_side(sub, chunk=512, side=100.0):
    """A box minimum and a coordinate at the middle of the root's upper child that the counting grid and the child's grid
    put on different sides."""
    rng = np.random.default_rng(12)
    for _ in range(4000):
        mn = float(rng.uniform(-60, 100))
        p = np.array([mn + side * 0.75])
        for _ in range(6):
            p = np.unique(np.concatenate([p, np.nextafter(p, -np.inf), np.nextafter(p, np.inf)]))
        a, b = middle_sides(p, mn, side, sub)
        if (a != b).any():
            return mn, p[a != b][0]
    raise AssertionError("no such coordinate")


def check_repeat(case, cfg, repeat):
    """Against the oracle; `repeat`: what the pass was repeated with, by the names of the stages."""
    ref = run_oracle(case, cfg)
    s = run_gpu(case, cfg)
    names = [k for k in s.timings() if k.startswith("repeat")]
    compare_results(ref, s)
    assert names == repeat and s.stats()["subsample_passes"] == 1 + len(repeat)
    s.close()


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("chunk,sub,n", [(512, 128, 60_000), (512, 64, 20_000), (512, 16, 20_000)])
def test_wall_in_another_octant(chunk, sub, n, mode):
    """A wall whose points all belong to octants without a child, among other points."""
    mn, p = foreign_side(sub)
    xyz, rgb = points("volume", 2 * n)
    xyz = xyz * 100.0
    xyz[:, 0] += mn
    xyz[:n, 0] = p
    keep = (xyz[:, 0] < mn + 50.0) | (xyz[:, 0] == p)   # nothing else in the child's other half
    case = case_from_points(xyz[keep], rgb[keep], 1, scale=0.01, bbox=[mn, 0, 0, mn + 100.0, 100.0, 100.0])
    check_repeat(case, dict(chunk_grid=chunk, sub_grid=sub, merge_threshold=700, output_factor=12.0, **MODES[mode]),
                 ["repeat_octants"])


def test_more_foreign_points_than_the_list_holds():
    mn, p = foreign_side(8)
    n = 90_000
    xyz, rgb = points("volume", n)
    xyz = xyz * 50.0          # all in one child of the root
    xyz[:, 0] = p
    case = case_from_points(xyz, rgb, 1, scale=0.01, bbox=[mn, 0, 0, mn + 100.0, 100.0, 100.0])
    check_repeat(case, dict(chunk_grid=512, sub_grid=8, merge_threshold=80_000, output_factor=12.0, inter=True),
                 ["repeat_octants", "repeat_nodes"])


@pytest.mark.parametrize("mode", ["first", "first_intra", "first_inter", "random_inter", "first_weighted"])
@pytest.mark.parametrize("off,side,chunk,sub", [(437000.0, 51.2, 64, 128), (123456.78, 51.2, 64, 32),
                                                (0.1, 102.4, 128, 64), (5412345.67, 25.6, 32, 16)])
def test_lattice_cloud(off, side, chunk, sub, mode):
    """Coordinates that are multiples of 1 cm from an offset, as scans are stored, in a box whose octant planes are
    among them."""
    rng = np.random.default_rng(5)
    n = 80_000
    steps = int(round(side / 0.01))
    q = rng.integers(0, steps, (n, 3))
    q[:, 2] = (q[:, 0] // 7 + q[:, 1] // 5) % steps
    rgb = rng.integers(0, 256, (n, 3), dtype=np.uint8)
    case = case_from_points(off + q * 0.01, rgb, 1, scale=0.01, bbox=[off] * 3 + [off + side] * 3)
    cfg = dict(chunk_grid=chunk, sub_grid=sub, merge_threshold=600, output_factor=12.0, **MODES[mode])
    check_repeat(case, cfg, ["repeat_octants"])


@pytest.mark.parametrize("mode", ["first", "first_intra", "random_inter", "random_weighted"])
@pytest.mark.parametrize("cloud_type,steps,scale,sub", [(1, 4096, 0.01, 128), (0, 4096, 0.01, 64), (1, 512, 1 / 64, 32),
                                                        (0, 65536, 1 / 1024, 128)])
def test_points_on_cell_boundaries(cloud_type, steps, scale, sub, mode):
    """Coordinates that are exact multiples of a fraction of the box, most of them on boundaries between cells of some
    level, at both ends of the box too; output coordinates that lie on integers."""
    rng = np.random.default_rng(9)
    n = 70_000
    xyz = rng.integers(0, steps + 1, (n, 3)) * (64.0 / steps)
    xyz[:, 2] = np.floor(xyz[:, 0] + xyz[:, 1]) / 2
    rgb = rng.integers(0, 256, (n, 3), dtype=np.uint8)
    case = case_from_points(xyz, rgb, cloud_type, scale=scale, bbox=[0, 0, 0, 64.0, 64.0, 64.0])
    check(case, dict(chunk_grid=64, sub_grid=sub, merge_threshold=500, output_factor=12.0, **MODES[mode]))


@pytest.mark.parametrize("box", [64.0, 40.0])
@pytest.mark.parametrize("off", [0.0, 1e12])
def test_points_beyond_the_box(box, off):
    """Points above the box (clamped to its last cells), and a box whose coordinates prove no cell."""
    rng = np.random.default_rng(10)
    n = 40_000
    xyz = off + np.floor(rng.random((n, 3)) * 64 * 64) / 64
    rgb = rng.integers(0, 256, (n, 3), dtype=np.uint8)
    case = case_from_points(xyz, rgb, 1, scale=0.125, bbox=[off] * 3 + [off + box] * 3)
    check(case, dict(chunk_grid=32, sub_grid=64, merge_threshold=400, output_factor=12.0, inter=True))


@pytest.mark.parametrize("sub", [64, 100])
def test_output_coordinate_beyond_int32(sub):
    """A scale for which the far points' output coordinates do not fit: an error found before subsampling, after which
    nothing is subsampled or placed, and the session goes on."""
    from helpers import octree_api

    rng = np.random.default_rng(11)
    xyz = np.round(rng.random((20_000, 3)) * 1000)
    rgb = rng.integers(0, 256, (20_000, 3), dtype=np.uint8)
    cfg = dict(chunk_grid=32, sub_grid=sub, merge_threshold=400, output_factor=12.0)
    for scale in (1e-7, 1e-9):
        case = case_from_points(xyz, rgb, 1, scale=scale, bbox=[0, 0, 0, 1000.0, 1000.0, 1000.0])
        with pytest.raises(octree_api.OctreeError, match="does not fit int32"):
            run_gpu(case, cfg)
    check(case_from_points(xyz, rgb, 1, scale=0.001, bbox=[0, 0, 0, 1000.0, 1000.0, 1000.0]), cfg)


@pytest.mark.parametrize("mode", ["first_intra", "first_inter", "random_intra", "random_inter"])
@pytest.mark.parametrize("shape,n,chunk,sub,threshold", [("plane", 150_000, 8, 8, 9_000), ("volume", 150_000, 8, 16, 9_000),
                                                         ("corner", 200_000, 8, 32, 20_000), ("plane", 250_000, 2, 64, 200_000)])
def test_many_candidates_per_cell(shape, n, chunk, sub, threshold, mode):
    """Cells of more than 257 candidates (the shared sums' limit), and of more than 1024 (the packed count's)."""
    xyz, rgb = points(shape, n)
    if shape == "plane":
        xyz[:, 0] = 0.3
    rgb[: n // 3] = 255
    case = case_from_points(xyz * 50.0, rgb, 0, scale=0.001, bbox=[0, 0, 0, 50.5, 50.5, 50.5])
    check(case, dict(chunk_grid=chunk, sub_grid=sub, merge_threshold=threshold, output_factor=4.0, **MODES[mode]))


@pytest.mark.parametrize("mode", ["first_weighted", "random_weighted"])
def test_more_face_cells_than_their_sums_have_room_for(mode):
    """A small grid, most of whose cells lie on faces between units, with few points per cell: the level is repeated
    with more room for their weighted sums, by the same kernels, and a later build has the room."""
    xyz, rgb = points("volume", 40_000)
    case = case_from_points(xyz * 50.0, rgb, 1, scale=0.001, bbox=[0, 0, 0, 50.5, 50.5, 50.5])
    cfg = dict(chunk_grid=32, sub_grid=8, merge_threshold=24, output_factor=12.0, **MODES[mode])
    ref = run_oracle(case, cfg)
    s = run_gpu(case, cfg)
    assert [k for k in s.timings() if k.startswith("repeat")] == ["repeat_partials"]
    compare_results(ref, s)
    s.generate()
    assert s.stats()["subsample_passes"] == 1
    compare_results(ref, s)
    s.close()


@pytest.mark.parametrize("cloud_type,stride", [(0, 15), (0, 16), (0, 20), (0, 28), (0, 64), (0, 65), (0, 80), (1, 27), (1, 28),
                                               (1, 32), (1, 64), (1, 72), (1, 100)])
@pytest.mark.parametrize("scattered", [False, True])
def test_strides(cloud_type, stride, scattered):
    """Record strides on both sides of what the grouped distribution takes, in leaf order and scattered, with enough
    points (262,144) for the choice by the sampled order."""
    from helpers import Case

    n = 270_001
    case = make_case(2, cloud_type, n, seed=17, stride=stride)
    if scattered:
        rec = case.cloud.reshape(n, stride)
        case = Case(np.ascontiguousarray(rec[np.random.default_rng(4).permutation(n)]).reshape(-1), n, stride, cloud_type,
                    case.scale, case.bb_min, case.bb_max)
    check(case, dict(chunk_grid=128, sub_grid=64, merge_threshold=1500, random=True, inter=True))


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("cloud_type,chunk,sub,around", [(0, 2, 128, 0), (1, 4, 64, 0), (0, 8, 32, 20_000), (1, 16, 128, 60_000),
                                                         (1, 16, 8, 30_000)])
def test_large_leaves(cloud_type, chunk, sub, around, mode):
    """Leaves of more points than one block takes: a few alone (colours spread over blocks where the grid allows it), and
    one among the units of a level of many, with points beyond both count limits of a cell."""
    rng = np.random.default_rng(21)
    n = 160_000
    xyz = rng.random((n, 3)) ** 2 * 0.06 + 0.52 if around else rng.random((n, 3)) * 0.9 * rng.random((n, 1))
    xyz[: n // 8] = xyz[0]                     # one cell of very many
    xyz = np.concatenate([xyz, rng.random((around, 3))])
    xyz = xyz[rng.permutation(len(xyz))]
    rgb = rng.integers(0, 256, (len(xyz), 3), dtype=np.uint8)
    case = case_from_points(xyz * 50.0, rgb, cloud_type, scale=0.001, bbox=[0, 0, 0, 50.5, 50.5, 50.5])
    cfg = dict(chunk_grid=chunk, sub_grid=sub, merge_threshold=100, output_factor=12.0, **MODES[mode])
    ref = run_oracle(case, cfg)
    assert ref.stats["max_leaf_points"] > 65536
    s = run_gpu(case, cfg)
    compare_results(ref, s)
    assert not [k for k in s.timings() if k.startswith("repeat")]
    s.close()


@pytest.mark.parametrize("mode", ["first", "first_intra", "random_inter", "first_weighted"])
@pytest.mark.parametrize("sub", [16, 64])
def test_large_leaves_with_points_of_other_octants(sub, mode):
    """Eight large leaves of one node whose points are multiples of 1 cm, some of them on the planes between the leaves
    where the node's grid puts them on another side than the counting grid."""
    rng = np.random.default_rng(22)
    side, steps = 51.2, 5120
    for _ in range(1000):
        off = float(np.round(rng.uniform(1e5, 9e5), 2))
        p = off + (steps * 3 // 8) * 0.01
        cubic = (off + side) - off
        m = off + cubic / 4
        if (np.floor((p - off) / (cubic / 8)) >= 3) != (np.floor((p - m) / (((m + cubic / 4) - m) / sub)) >= sub // 2):
            break
    else:
        raise AssertionError("no such offset")
    n = 620_000
    q = rng.integers(-60, 60, (n, 3)) + steps * 3 // 8
    rgb = rng.integers(0, 256, (n, 3), dtype=np.uint8)
    case = case_from_points(off + q * 0.01, rgb, 1, scale=0.01, bbox=[off] * 3 + [off + side] * 3)
    cfg = dict(chunk_grid=8, sub_grid=sub, merge_threshold=1000, output_factor=4.0, **MODES[mode])
    assert run_oracle(case, cfg).stats["max_leaf_points"] > 65536
    check_repeat(case, cfg, ["repeat_octants"])
