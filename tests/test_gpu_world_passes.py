"""The bit-parallel world passes at the sizes where a tile can go wrong: worlds and boxes
one voxel short of, at and beyond the tiles' edges, sparse solids (offsets at the rim of
the depth field's radius) and dense ones, against the oracle, word for word."""
import numpy as np
import pytest

from helpers import make_world

pytestmark = pytest.mark.gpu


def sparse_words(W, H, seed, density):
    """Random solids; the air carries old depth-field words in places, which a refresh that
    finds a near solid has to leave alone."""
    rng = np.random.default_rng(seed)
    n = W * H * W
    words = np.full(n, -1, np.int32)
    old = rng.random(n) < 0.2
    words[old] = np.float32(-2.5).view(np.int32)
    solid = rng.random(n) < density
    words[solid] = rng.integers(0, 1 << 24, int(solid.sum())).astype(np.int32) | 0x01000000
    return words


@pytest.mark.parametrize("W,H", [(1, 1), (5, 70), (31, 15), (32, 16), (33, 17), (66, 47), (97, 33)])
@pytest.mark.parametrize("density", [0.0, 0.0006, 0.01, 0.7, 1.0])
def test_depth_field_of_boxes(cuda, oracle, W, H, density):
    words = sparse_words(W, H, 7 * W + H, density)
    boxes = [(0, 0, 0, W, H, W), (W // 3, H // 4, W // 2, W, H, W), (1, 1, 1, W - 1, H - 1, W - 2),
             (-9, -9, -9, W // 2 + 1, H // 2 + 1, 2), (W - 1, H - 1, W - 1, W + 40, H + 40, W + 40)]
    for box in boxes:
        w = make_world(words, W, H)
        w.fix_depth_field(box)
        ref = words.copy()
        x0, y0, z0, x1, y1, z1 = box
        oracle.fix_depth_field_box(ref, W, H, (max(x0, 0), max(y0, 0), max(z0, 0), min(x1, W), min(y1, H), min(z1, W)))
        got = w.download(np.empty_like(ref))
        assert np.array_equal(got, ref), (box, np.flatnonzero(got != ref)[:4])


@pytest.mark.parametrize("W,H", [(31, 15), (64, 48), (97, 33)])
def test_removed_spheres_refresh_the_depth_field(cuda, oracle, W, H):
    words = sparse_words(W, H, W + H, 0.3)
    w = make_world(words, W, H)
    rng = np.random.default_rng(W)
    ref = words.copy()
    for r in (0, 1, 2, 5, 8, 13, 30):
        c = [int(rng.integers(-4, n + 4)) for n in (W, H, W)]
        w.remove_sphere(*c, r, 1)
        oracle.remove_sphere(ref, W, H, *c, r, 1)
        got = w.download(np.empty_like(ref))
        assert np.array_equal(got, ref), (c, r)
