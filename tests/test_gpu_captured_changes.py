"""World changes captured into a CUDA graph: its runs change the words without the host's knowledge,
and every frame after a run, by either kernel, shows the words of that moment, whatever was drawn,
uploaded or looked at between capture and run."""
import numpy as np
import pytest

import vrt
from helpers import INEXACT_OUTPUTS, assert_same_frame, expected_masks, gpu_render, make_world

pytestmark = pytest.mark.gpu

W, H = 96, 64
KERNELS = (vrt.KERNEL_WORD, vrt.KERNEL_MASK_PIXEL)


def some_words(seed, depth):
    rng = np.random.default_rng(seed)
    n = W * H * W
    words = np.where(rng.random(n) < 0.01, 0x01000000 | rng.integers(0, 1 << 24, n), -1).astype(np.int32)
    words.reshape(W, H, W)[:, :3, :] = 0x01808080
    if depth:  # jumps that are not fixDepthField's: a frame has to go by the words themselves
        far = (words == -1) & (rng.random(n) < 0.3)
        words[far] = np.float32(-2.5).view(np.int32)
    return words


def camera():
    u = vrt.default_uniforms()
    u.camPos[:] = (20.3, 24.6, 9.7)
    u.rotateMatrix[:] = vrt.rotate_matrix(0.25, 0.5)
    u.lightPos[:] = [40.0, 160.0, 30.0]
    u.maxSteps = 300
    u.aspectRatio = 1.5
    return u


CHANGES = {
    "small sphere": lambda w, s: w.remove_sphere(40, 12, 40, 7, 1, s),
    "large sphere": lambda w, s: w.remove_sphere(48, 20, 48, 33, 1, s),
    "depth field": lambda w, s: w.fix_depth_field(stream=s),
    "voxels": lambda w, s: [w.place_voxel(24 + k, 21, 18 + 3 * k, 0x01FF8000, s) for k in range(6)],
}


def capture(torch, calls):
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g.capture_begin()
        try:
            calls(s.cuda_stream)
        finally:  # a capture left open would fail every later test
            g.capture_end()
    torch.cuda.synchronize()
    return g


def draw_all(oracle, w, now, kernels=KERNELS):
    want = oracle.render(now, W, H, camera(), 60, 40)
    for kernel in kernels:
        assert_same_frame(want, gpu_render(w, camera(), 60, 40, kernel=kernel))


@pytest.mark.parametrize("drawn_before", [False, True])
@pytest.mark.parametrize("change", CHANGES)
def test_frames_after_runs_of_a_captured_change(cuda, oracle, change, drawn_before):
    w = make_world(some_words(0, True), W, H)
    if drawn_before:
        draw_all(oracle, w, some_words(0, True))
    g = capture(cuda, lambda s: CHANGES[change](w, s))
    for k in range(3):
        words = some_words(k, True)
        w.upload(words)
        draw_all(oracle, w, words)
        g.replay()
        cuda.cuda.synchronize()
        now = w.download(np.empty_like(words))
        assert not np.array_equal(now, words)
        draw_all(oracle, w, now)
        bricks, regions, supers = w.masks()
        eb, er, es = expected_masks(now, W, H)
        assert np.array_equal(bricks, eb) and np.array_equal(regions, er) and np.array_equal(supers, es)


def test_a_captured_voxel_outside_the_solid_box(cuda, oracle):
    """Frames end rays at the box of the solid voxels, which the host knows from the last upload."""
    words = np.full(W * H * W, -1, np.int32)
    words.reshape(W, H, W)[:, :3, :] = 0x01808080
    w = make_world(words, W, H)
    g = capture(cuda, lambda s: [w.place_voxel(20 + x, y, 30 + x, 0x01FF8000, s) for x in range(4) for y in (20, 21, 29)])
    for again in (lambda: w.upload(words), lambda: w.sync_flags()):
        w.upload(words)
        again()
        g.replay()
        cuda.cuda.synchronize()
        now = w.download(np.empty_like(words))
        want = oracle.render(now, W, H, camera(), 60, 40)
        assert (np.asarray(want["hit"]).ravel() >= 3 * W).any()
        for kernel in KERNELS + (vrt.KERNEL_BITMASK,):
            got = gpu_render(w, camera(), 60, 40, kernel=kernel, outputs=INEXACT_OUTPUTS)
            assert_same_frame(want, got, outputs=INEXACT_OUTPUTS)


@pytest.mark.parametrize("change", ["small sphere", "depth field", "jump"])
def test_captured_depth_field_words_of_a_world_without(cuda, oracle, change):
    """The kernels that follow jumps are picked by a flag that the host knows from the last upload."""
    words = some_words(1, False)
    w = make_world(words, W, H)
    word = int(np.float32(-2.5).view(np.int32))
    g = capture(cuda, lambda s: [w.place_voxel(24 + k, 22, 18 + k, word, s) for k in range(9)]
                if change == "jump" else CHANGES[change](w, s))
    for again in (lambda: w.upload(words), lambda: w.sync_flags()):
        w.upload(words)
        again()
        g.replay()
        cuda.cuda.synchronize()
        now = w.download(np.empty_like(words))
        assert (now < -1).any()
        draw_all(oracle, w, now, KERNELS + (vrt.KERNEL_AUTO,))


@pytest.mark.parametrize("change", CHANGES)
@pytest.mark.parametrize("kernel", KERNELS)
def test_frames_captured_behind_a_change(cuda, oracle, change, kernel):
    """Two changes with a frame behind each in one graph, run again and again on other words, and
    plain frames after it."""
    w = make_world(some_words(0, True), W, H)
    draw_all(oracle, w, some_words(0, True))  # made before: what a kernel allocates on its first use
    r, u, n = vrt.Renderer(), camera(), 60 * 40 * 4
    imgs = [cuda.zeros(n, dtype=cuda.uint8, device="cuda") for _ in range(3)]
    opts = vrt.RenderOpts()
    opts.kernel = kernel

    def calls(s):
        CHANGES[change](w, s)
        r.render(w, u, 60, 40, imgs[0].data_ptr(), None, 0, opts, s)
        r.render(w, u, 60, 40, imgs[1].data_ptr(), None, 0, opts, s)
        w.remove_sphere(30, 12, 30, 9, 1, s)
        r.render(w, u, 60, 40, imgs[2].data_ptr(), None, 0, opts, s)

    g = capture(cuda, calls)
    for k in range(3):
        words = some_words(5 + k, True)
        w.upload(words)
        if k == 1:
            draw_all(oracle, w, words)
        between = make_world(words, W, H)  # the words of the two frames ahead of the sphere
        CHANGES[change](between, 0)
        mid = between.download(np.empty_like(words))
        g.replay()
        cuda.cuda.synchronize()
        now = w.download(np.empty_like(words))
        for img, at in zip(imgs, (mid, mid, now)):
            want = np.asarray(oracle.render(at, W, H, u, 60, 40)["rgba"]).reshape(-1)
            assert np.array_equal(img.cpu().numpy(), want)
        draw_all(oracle, w, now)


@pytest.mark.parametrize("kernel", KERNELS)
def test_frames_captured_behind_a_plain_change(cuda, oracle, kernel):
    """The first frames after a large plain change, captured on two streams of one graph: they rebuild
    what they read in each run, and plain frames before and after the runs do so for themselves."""
    words = some_words(3, True)
    w = make_world(words, W, H)
    draw_all(oracle, w, words)
    w.remove_sphere(48, 20, 48, 33, 1)
    renderers, u, n = [vrt.Renderer(), vrt.Renderer()], camera(), 60 * 40 * 4
    imgs = [cuda.zeros(n, dtype=cuda.uint8, device="cuda") for _ in range(2)]
    opts = vrt.RenderOpts()
    opts.kernel = kernel
    side = cuda.cuda.Stream()

    def calls(s):
        here = cuda.cuda.current_stream()
        renderers[0].render(w, u, 60, 40, imgs[0].data_ptr(), None, 0, opts, s)
        side.wait_stream(here)
        renderers[1].render(w, u, 60, 40, imgs[1].data_ptr(), None, 0, opts, side.cuda_stream)
        here.wait_stream(side)

    g = capture(cuda, calls)
    for k in range(3):
        if k:
            w.remove_sphere(20 + 30 * k, 12, 70 - 30 * k, (0, 33, 6)[k], 1)
        now = w.download(np.empty_like(words))
        if k != 1:
            draw_all(oracle, w, now)
        g.replay()
        cuda.cuda.synchronize()
        want = np.asarray(oracle.render(now, W, H, u, 60, 40)["rgba"]).reshape(-1)
        for img in imgs:
            assert np.array_equal(img.cpu().numpy(), want), k
            img.zero_()
        draw_all(oracle, w, now)
