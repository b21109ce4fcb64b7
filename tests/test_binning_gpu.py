"""GPU parity of projection, tile counts, keys, sorted indices and ranges.

The CUDA path (fvgs_project_bin) must match the CPU restatement bit for bit
(tile keys, ranges and sorted indices: exact; projection outputs: exact, both
sides use the same FP32 operation order).
"""
import numpy as np
import pytest

from conftest import crossing_layers, scaled_camera
from f_vigs_slam_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


SORT_PATHS = {"tile": 0, "radix": 0x8}


def _gpu_binning(fv, scene, pose, K, W, H, params, sort_path="tile"):
    s = fv.Session(max(scene.n, 1), W, H, params)
    s.set_debug(fv.DEBUG_PROJECTION | SORT_PATHS[sort_path])
    s.upload(scene)
    n_inst = s.project_bin(pose, K, W, H)
    proj = s.download_projection() if scene.n else None
    keys, vals, ranges = s.download_binning(W, H)
    s.close()
    return n_inst, proj, keys, vals, ranges


def _check(oracle, fv, scene, pose, K, W, H, quirks, sort_path="tile"):
    P = oracle.default_params(quirks)
    b = oracle.prepare(scene, pose, K, W, H, P)
    n_inst, proj, keys, vals, ranges = _gpu_binning(fv, scene, pose, K, W, H, fv.default_params(quirks), sort_path)
    assert n_inst == b.keys.shape[0]
    if scene.n:
        vis = b.proj.visible.astype(bool)
        np.testing.assert_array_equal(proj["visible"], b.proj.visible)
        for name in ("uv", "depth", "phat"):
            g = proj[name][vis]
            o = getattr(b.proj, name)[vis]
            np.testing.assert_array_equal(g.view(np.uint32), o.view(np.uint32), err_msg=name)
        np.testing.assert_array_equal(proj["cov2d"][vis].view(np.uint32), b.proj.cov2d[vis].view(np.uint32))
        np.testing.assert_array_equal(proj["inv2d"][vis].view(np.uint32), b.proj.inv2d[vis].view(np.uint32))
        np.testing.assert_array_equal(proj["counts"], b.cnt)
    np.testing.assert_array_equal(keys, b.keys)
    np.testing.assert_array_equal(vals, b.vals)
    np.testing.assert_array_equal(ranges, b.ranges)
    return b


@pytest.mark.parametrize("sort_path", ["tile", "radix"])
@pytest.mark.parametrize("quirks", [0x4 | 0x8, 0x0, 0x1 | 0x4, 0x2 | 0x4])
def test_binning_small(oracle, fvgs_lib, quirks, sort_path):
    W, H, K = scaled_camera(0.25)
    scene = S.cam_box(3000, seed=11)
    pose = S.perturb((np.zeros(3), S.IDENTITY_Q), 1.0, 2.0, np.random.default_rng(1))
    _check(oracle, fvgs_lib, scene, pose, K, W, H, quirks, sort_path)


@pytest.mark.parametrize("sort_path", ["tile", "radix"])
def test_binning_vga_50k(oracle, fvgs_lib, sort_path):
    """Full small plain-method workload: N=50k at 640x480 (bit-exact)."""
    W, H, K = scaled_camera(1.0)
    scene = S.cam_box(50_000, seed=0)
    pose = S.perturb((np.zeros(3), S.IDENTITY_Q), 1.0, 2.0, np.random.default_rng(0))
    b = _check(oracle, fvgs_lib, scene, pose, K, W, H, 0x4 | 0x8, sort_path)
    assert b.keys.shape[0] > 100_000  # several sort tiles and passes exercised


def _full_frame_splats(n, seed):
    rng = np.random.default_rng(seed)
    pos = np.stack([rng.uniform(-0.1, 0.1, n), rng.uniform(-0.1, 0.1, n), rng.uniform(1.0, 1.2, n)], 1)
    return S.Scene(pos.astype(np.float32), np.full((n, 3), 1.5, np.float32),
                   np.tile(S.IDENTITY_Q, (n, 1)).astype(np.float32),
                   rng.uniform(0, 1, (n, 3)).astype(np.float32), np.full(n, 0.5, np.float32))


def test_binning_large_tiles(oracle, fvgs_lib):
    """Every tile holds more than 4096 instances: the per-tile sort must hand
    them to the global merge path and still match bit for bit."""
    W, H, K = scaled_camera(0.25)
    scene = _full_frame_splats(9000, 5)
    b = _check(oracle, fvgs_lib, scene, (np.zeros(3), S.IDENTITY_Q), K, W, H, 0x4 | 0x8)
    assert (b.ranges[:, 1] - b.ranges[:, 0]).min() > 4096


def test_binning_culled_slots_pile_into_tile0(oracle, fvgs_lib):
    """With the reference's culled slots, 20k Gaussians behind the camera all
    land in tile 0 with key 0 (one huge bucket of equal depth bits)."""
    W, H, K = scaled_camera(0.25)
    sc = S.cam_box(22_000, seed=8)
    sc.positions[:20_000, 2] *= -1.0
    b = _check(oracle, fvgs_lib, sc, (np.zeros(3), S.IDENTITY_Q), K, W, H, 0x1 | 0x4)
    assert b.ranges[0, 1] - b.ranges[0, 0] >= 20_000


def test_binning_empty_and_culled(oracle, fvgs_lib):
    W, H, K = scaled_camera(0.25)
    scene = S.cam_box(500, seed=2)
    behind = S.Scene(scene.positions * np.array([1, 1, -1], np.float32), scene.scales, scene.orientations,
                     scene.colors, scene.opacities)
    pose = (np.zeros(3), S.IDENTITY_Q)
    # all culled: no instances (intended) / one instance per Gaussian in tile 0 (reference slots)
    _check(oracle, fvgs_lib, behind, pose, K, W, H, 0x4)
    b = _check(oracle, fvgs_lib, behind, pose, K, W, H, 0x1 | 0x4)
    assert b.keys.shape[0] == behind.n and np.all(b.keys == 0)
    empty = S.Scene(*(a[:0] for a in (scene.positions, scene.scales, scene.orientations, scene.colors)),
                    scene.opacities[:0])
    _check(oracle, fvgs_lib, empty, pose, K, W, H, 0x4)


def test_binning_capacity_growth(oracle, fvgs_lib):
    """Large splats (every Gaussian covers the frame) overflow the initial
    instance capacity; the library must grow and return the exact result."""
    W, H, K = scaled_camera(1.0)
    rng = np.random.default_rng(4)
    n = 1500
    pos = np.stack([rng.uniform(-0.1, 0.1, n), rng.uniform(-0.1, 0.1, n), rng.uniform(1.0, 1.2, n)], 1)
    scene = S.Scene(pos.astype(np.float32), np.full((n, 3), 1.5, np.float32),
                    np.tile(S.IDENTITY_Q, (n, 1)).astype(np.float32),
                    rng.uniform(0, 1, (n, 3)).astype(np.float32), np.full(n, 0.5, np.float32))
    b = _check(oracle, fvgs_lib, scene, (np.zeros(3), S.IDENTITY_Q), K, W, H, 0x4 | 0x8)
    assert b.keys.shape[0] > (1 << 20)


@pytest.mark.parametrize("equal", [False, True], ids=["spread", "equal_depths"])
@pytest.mark.parametrize("n", [1, 126, 127, 128, 512, 1536, 1537, 3072, 3073, 4096, 4097, 8192, 8193, 16384, 16385,
                               40000, (1 << 20) + 5])
def test_one_tile_sort_sizes(oracle, fvgs_lib, n, equal):
    """One tile's list around the capacities of the per-tile sort's forms, full
    and incremental (members leaving and entering between poses), and keys
    that tie in depth and fall back to the index."""
    W, H, K = 16, 16, (40.0, 40.0, 7.5, 7.5)
    rng = np.random.default_rng(n)
    scene = S.cam_box(n, seed=n)
    z = scene.positions[:, 2]
    scene.positions[:, :2] = rng.uniform(-0.21, 0.21, (n, 2)) * z[:, None]
    if equal:
        scene.positions[:] = [0.01, -0.02, 2.0]
    P = oracle.default_params()
    poses = [(np.zeros(3, np.float32), S.IDENTITY_Q)]
    for deg, cm in ((0.05, 0.1), (1.0, 2.0), (0.0, 0.0)):
        poses.append(S.perturb(poses[-1], deg, cm, rng))
    with fvgs_lib.Session(n, W, H) as s:
        s.upload(scene)
        for pose in poses:
            n_inst = s.project_bin(pose, K, W, H)
            b = oracle.prepare(scene, pose, K, W, H, P)
            keys, vals, ranges = s.download_binning(W, H)
            assert n_inst == b.keys.shape[0]
            np.testing.assert_array_equal(ranges, b.ranges)
            np.testing.assert_array_equal(vals, b.vals)
            np.testing.assert_array_equal(keys, b.keys)


def _expect_binning(oracle, s, scene, pose, K, W, H):
    n_inst = s.project_bin(pose, K, W, H)
    b = oracle.prepare(scene, pose, K, W, H, oracle.default_params())
    keys, vals, ranges = s.download_binning(W, H)
    assert n_inst == b.keys.shape[0]
    np.testing.assert_array_equal(ranges, b.ranges)
    np.testing.assert_array_equal(vals, b.vals)
    np.testing.assert_array_equal(keys, b.keys)
    return b


def _alternating(n, every, near, far):
    """Two layers, the near one taking every `every`-th place, each spread over 0.05."""
    i = np.arange(n)
    return np.where(i % every == 0, near, far) + 0.05 * i / n


@pytest.mark.parametrize("n,every", [(32768, 2), (40960, 2), (65536, 2), (65536, 16), (131072, 2), (131072, 32),
                                     (262144, 64)])
def test_one_tile_sort_alternating_layers(oracle, fvgs_lib, n, every):
    """A tile above one CTA's capacity whose depths alternate with the Gaussian
    index: samples at even places of its list may then all come from one layer,
    and the other holds most of the tile between two of them."""
    W, H, K = 16, 16, (40.0, 40.0, 7.5, 7.5)
    rng = np.random.default_rng(n + every)
    scene = S.cam_box(n, seed=n)
    scene.scales[:] = 0.005
    z = _alternating(n, every, 1.5, 2.5)
    scene.positions[:] = np.stack([rng.uniform(-0.1, 0.1, n) * z, rng.uniform(-0.1, 0.1, n) * z, z], 1)
    pose = (np.zeros(3, np.float32), S.IDENTITY_Q)
    with fvgs_lib.Session(n, W, H) as s:
        s.upload(scene)
        for _ in range(2):
            assert _expect_binning(oracle, s, scene, pose, K, W, H).keys.shape[0] == n
        pose = S.perturb(pose, 0.5, 1.0, rng)
        assert _expect_binning(oracle, s, scene, pose, K, W, H).keys.shape[0] == n


@pytest.mark.parametrize("tiles", [1, 32])
@pytest.mark.parametrize("n", [32768, 65536])
def test_one_tile_sort_alternating_layers_incremental(oracle, fvgs_lib, n, tiles):
    """The same for a list that is carried over and whose order the next camera
    sees alternate.  With 32 tiles, all but one empty, the mean length picks the
    sort's forms for short lists."""
    W, H, K = (16, 16, (40.0, 40.0, 7.5, 7.5)) if tiles == 1 else (128, 64, (40.0, 40.0, 55.5, 23.5))
    scene, front, side = crossing_layers(oracle, n, K, W, H)
    with fvgs_lib.Session(n, W, H) as s:
        s.upload(scene)
        for k, pose in enumerate((front, side, front)):
            _expect_binning(oracle, s, scene, pose, K, W, H)
            assert bool(s.binning_info()["incremental"]) == (k > 0)


@pytest.mark.parametrize("fill", [100, 1200])
@pytest.mark.parametrize("dense", [2049, 4097, 8193, 16384, 20000])
def test_dense_tile_among_short_lists(oracle, fvgs_lib, dense, fill):
    """One tile far above the grid's mean, which picks the sort's forms for
    short lists (means up to 1024 and 2048) once a binning has set it; the dense
    tile's layers alternate by index.  A re-upload makes a full binning."""
    W, H, K = 128, 64, (40.0, 40.0, 63.5, 31.5)
    tiles = [(tx, ty) for ty in range(4) for tx in range(8)]
    n_tile = [dense if t == (3, 1) else fill for t in tiles]
    order = sorted(range(len(tiles)), key=lambda k: tiles[k] != (3, 1))  # the dense tile's Gaussians first
    n = sum(n_tile)
    rng = np.random.default_rng(dense + fill)
    scene = S.cam_box(n, seed=dense)
    scene.scales[:] = 0.005
    at = np.concatenate([np.tile(tiles[k], (n_tile[k], 1)) for k in order])
    uv = 16.0 * at + 8.0 + rng.uniform(-0.5, 0.5, (n, 2))
    z = np.concatenate([_alternating(dense, 2, 1.8, 2.2), rng.uniform(1.5, 2.5, n - dense)])
    scene.positions[:] = np.stack([(uv[:, 0] - K[2]) / K[0] * z, (uv[:, 1] - K[3]) / K[1] * z, z], 1)
    poses = [(np.zeros(3, np.float32), S.IDENTITY_Q)]
    for deg, cm in ((0.0, 0.0), (0.05, 0.1), (0.3, 1.0)):
        poses.append(S.perturb(poses[-1], deg, cm, rng))
    with fvgs_lib.Session(n, W, H) as s:
        s.upload(scene)
        b = _expect_binning(oracle, s, scene, poses[0], K, W, H)
        assert b.keys.shape[0] // len(tiles) <= (1024 if fill < 1000 else 2048)
        assert (b.ranges[:, 1] - b.ranges[:, 0]).max() >= dense
        s.upload(scene)
        for pose in poses:
            _expect_binning(oracle, s, scene, pose, K, W, H)
            _expect_binning(oracle, s, scene, pose, K, W, H)
