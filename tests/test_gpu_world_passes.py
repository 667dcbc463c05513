"""The bit-parallel world passes at the sizes where a tile can go wrong: worlds and boxes
one voxel short of, at and beyond the tiles' edges, sparse solids (offsets at the rim of
the depth field's radius) and dense ones, against the oracle, word for word."""
import numpy as np
import pytest

import vrt
from helpers import assert_same_frame, expected_distances, expected_masks, gpu_render, make_world

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


def check_structures(w, words, W, H):
    bricks, regions, supers = w.masks()
    eb, er, es = expected_masks(words, W, H)
    assert np.array_equal(bricks, eb) and np.array_equal(regions, er) and np.array_equal(supers, es)
    bdir, rdist = w.distances()
    ed, erd = expected_distances(words, W, H)
    assert np.array_equal(bdir, ed) and np.array_equal(rdist, erd)


@pytest.mark.parametrize("W,H", [(3, 130), (64, 64), (70, 47), (129, 20), (257, 65)])
def test_structures_follow_uploads_and_edits(cuda, W, H):
    """Masks of every level and both distance fields after whole and partial uploads from
    host and device memory at odd offsets (bricks fill and empty in one pass), removed
    spheres and placed voxels, against the model built from the words."""
    rng = np.random.default_rng(W)
    n = W * H * W
    words = sparse_words(W, H, W, 0.0002)
    w = make_world(words, W, H)
    check_structures(w, words, W, H)
    for k, density in enumerate((0.0001, 0.02, 0.0)):
        first = int(rng.integers(0, n // 2))
        part = sparse_words(W, H, 10 + k, density)[: int(rng.integers(1, n - first))]
        if k == 1:
            w.upload(part, first)
        else:
            pad = 1 + k  # a source address that is not 16-byte aligned
            d = cuda.from_numpy(np.concatenate([np.zeros(pad, np.int32), part])).cuda()
            w.upload_device(d.data_ptr() + 4 * pad, first, part.size)
        words[first:first + part.size] = part
        got = w.download(np.empty_like(words))
        assert np.array_equal(got, words)
        check_structures(w, words, W, H)
        assert w.info().has_depth_field == int((words < -1).any())
    w.place_voxel(W - 1, H - 1, 0, 0x01FFFFFF)
    words[W - 1 + W * (H - 1)] = 0x01FFFFFF
    w.remove_sphere(W // 2, H // 2, W // 2, 9, 0)
    z, y, x = np.meshgrid(np.arange(W) - W // 2, np.arange(H) - H // 2, np.arange(W) - W // 2, indexing="ij")
    words.reshape(W, H, W)[x * x + y * y + z * z < 81] = -1
    assert np.array_equal(w.download(np.empty_like(words)), words)
    check_structures(w, words, W, H)


@pytest.mark.parametrize("W,H", [(37, 33), (64, 48)])
def test_frames_after_edits_that_write_the_z_major_copy(cuda, oracle, W, H):
    """Small edits change the word kernel's z-major copy with the words; uploads and large
    spheres leave it to the next frame.  In any order between two frames, each frame equals
    the oracle's on the words of that moment."""
    words = sparse_words(W, H, W, 0.2)
    w = make_world(words, W, H)
    w.fix_depth_field()
    u = vrt.default_uniforms()
    u.camPos[:] = [2.5, H - 2.25, 3.5]
    u.rotateMatrix[:] = vrt.rotate_matrix(0.4, 0.6)
    u.lightPos[:] = [W / 2, 300.0, W / 3]
    u.aspectRatio = 1.5
    rng = np.random.default_rng(3)

    def small():
        w.remove_sphere(*[int(rng.integers(0, n)) for n in (W, H, W)], 4, 1)

    def voxel():
        w.place_voxel(int(rng.integers(0, W)), int(rng.integers(0, H)), int(rng.integers(0, W)), 0x01FF8000)

    def slab():
        w.upload(sparse_words(W, H, 5, 0.3)[: 2 * W * H + 7], first=5 * W * H + 3)

    def large():
        w.remove_sphere(W, H, W, 22, 1)

    for edits in ((), (small, voxel), (slab, small), (small, slab, voxel), (large, small), (voxel, large)):
        for e in edits:
            e()
        now = w.download(np.empty(W * H * W, np.int32))
        assert_same_frame(oracle.render(now, W, H, u, 60, 40), gpu_render(w, u, 60, 40, kernel=vrt.KERNEL_WORD))


@pytest.mark.parametrize("W,H", [(33, 17), (97, 41)])
@pytest.mark.parametrize("density", [0.0006, 0.01, 0.2])
def test_edits_with_small_and_large_depth_field_tiles(cuda, oracle, W, H, density):
    """Edits whose boxes end on either side of the tiles' edges, take a few small tiles or, from
    radius 34 in the larger world, the large ones; solids at the rim of the depth field's radius."""
    words = sparse_words(W, H, 3 * W + H, density)
    w = make_world(words, W, H)
    ref = words.copy()
    centres = [(0, 0, 0), (8, 8, 8), (W - 1, H - 1, W - 1), (15, 9, 24), (16, 7, 25), (W // 2, H // 2, W // 2)]
    for r in (0, 1, 4, 5, 12, 34):
        for c in centres if r < 34 else centres[-1:]:
            w.remove_sphere(*c, r, 1)
            oracle.remove_sphere(ref, W, H, *c, r, 1)
            got = w.download(np.empty_like(ref))
            assert np.array_equal(got, ref), (c, r, np.flatnonzero(got != ref)[:4])


@pytest.mark.parametrize("W,H", [(33, 17), (64, 20)])
@pytest.mark.parametrize("where", ["pageable", "page-locked", "device"])
def test_uploads_from_any_byte_address(cuda, W, H, where):
    """Words at addresses that no 4-byte load can read, in every memory an upload takes them from."""
    n = W * H * W
    words = sparse_words(W, H, W, 0.02)
    w = make_world(words, W, H)
    for off in (1, 2, 3, 4, 6):
        first = 5 * off
        part = sparse_words(W, H, off, 0.05)[: n - first - off]
        raw = np.zeros(part.nbytes + 16, np.uint8)
        if where == "pageable":
            raw[off:off + part.nbytes] = part.view(np.uint8)
            w.upload(np.frombuffer(raw.data, np.int32, part.size, off), first)
        else:
            raw[off:off + part.nbytes] = part.view(np.uint8)
            t = cuda.from_numpy(raw)
            t = t.pin_memory() if where == "page-locked" else t.cuda()
            if where == "page-locked":
                w.upload(t.numpy()[off:off + part.nbytes].view(np.int32), first)
            else:
                w.upload_device(t.data_ptr() + off, first, part.size)
        words[first:first + part.size] = part
        assert np.array_equal(w.download(np.empty_like(words)), words), off
        check_structures(w, words, W, H)
