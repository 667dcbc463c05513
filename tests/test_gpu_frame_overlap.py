"""Frames in a row on one stream, where the next one may begin before the last has ended:
each leaves its own image, side outputs and counters, whatever is put between two of them."""
import numpy as np
import pytest

import vrt
from helpers import make_world

pytestmark = pytest.mark.gpu

W, H = 96, 64


def scene(jumps):
    rng = np.random.default_rng(5)
    words = np.where(rng.random(W * H * W) < 0.004, 0x01000000 | rng.integers(0, 1 << 24, W * H * W), -1).astype(np.int32)
    words.reshape(W, H, W)[:, :3, :] = 0x01808080
    w = make_world(words, W, H)
    if jumps:
        w.fix_depth_field()
    return w


def views(n, steps=300):
    us = []
    for i in range(n):
        u = vrt.default_uniforms()
        u.camPos[:] = (20.3 + i, 12.6 + 3 * (i % 5), 19.7)
        u.rotateMatrix[:] = vrt.rotate_matrix(0.1 * (i % 4), 0.9 * i)
        u.lightPos[:] = [20.0 + 5 * i, 120.0, 3.0]
        u.maxSteps = steps
        u.aspectRatio = 1.0
        us.append(u)
    return us


def frame(torch, r, w, u, width, height, kernel, out, stream, stats=None):
    opts = vrt.RenderOpts()
    opts.kernel = kernel
    r.render(w, u, width, height, out.data_ptr(), None, stats.data_ptr() if stats is not None else 0, opts, stream)


def alone(torch, w, u, width, height, kernel):
    out = torch.zeros(width * height * 4, dtype=torch.uint8, device="cuda")
    stats = torch.zeros(vrt.STAT_COUNT, dtype=torch.int64, device="cuda")
    frame(torch, vrt.Renderer(), w, u, width, height, kernel, out, torch.cuda.current_stream().cuda_stream, stats)
    torch.cuda.synchronize()
    return out.cpu(), stats.cpu()[:4]


# a grid of one CTA, one that fits at once, and one several times as large
@pytest.mark.parametrize("size", [(5, 3), (320, 200), (1501, 700)])
@pytest.mark.parametrize("kernel,jumps", [(vrt.KERNEL_MASK_PIXEL, False), (vrt.KERNEL_MASK_PIXEL, True),
                                          (vrt.KERNEL_WORD, True)])
@pytest.mark.parametrize("own_stream", [False, True])
def test_frames_in_a_row(cuda, size, kernel, jumps, own_stream):
    torch = pytest.importorskip("torch")
    w, us = scene(jumps), views(6)
    n = size[0] * size[1] * 4
    expect = [alone(torch, w, u, *size, kernel) for u in us]
    s = torch.cuda.Stream() if own_stream else torch.cuda.current_stream()
    side = torch.cuda.Stream()
    r = vrt.Renderer()
    img = torch.zeros(n, dtype=torch.uint8, device="cuda")
    host = [torch.zeros(n, dtype=torch.uint8).pin_memory() for _ in range(40)]
    copies, stats = [], torch.zeros(vrt.STAT_COUNT, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        order = []
        for k in range(40):  # one image: copied away by the copy engine, a kernel, another stream, or overwritten
            i = (k * k + k // 7) % 6
            order.append(i)
            frame(torch, r, w, us[i], *size, kernel, img, s.cuda_stream, stats)
            if k % 4 == 0:
                host[k].copy_(img, non_blocking=True)
            elif k % 4 == 1:
                copies.append((i, img.clone()))
            elif k % 4 == 2:
                ev = s.record_event()
                side.wait_event(ev)
                with torch.cuda.stream(side):
                    torch.cuda._sleep(200000)
                    copies.append((i, img.clone()))
                    done = side.record_event()
                s.wait_event(done)
    torch.cuda.synchronize()
    for k in range(0, 40, 4):
        assert torch.equal(host[k], expect[order[k]][0]), k
    for i, c in copies:
        assert torch.equal(c.cpu(), expect[i][0])
    assert torch.equal(img.cpu(), expect[order[-1]][0])
    assert torch.equal(stats.cpu()[:4], sum(expect[i][1] for i in order))


@pytest.mark.parametrize("kernel,jumps", [(vrt.KERNEL_MASK_PIXEL, False), (vrt.KERNEL_MASK_PIXEL, True),
                                          (vrt.KERNEL_WORD, True)])
def test_changes_between_frames(cuda, kernel, jumps):
    """Edits, uploads and other worlds between frames: no frame sees a change from behind it
    or misses one ahead of it."""
    torch = pytest.importorskip("torch")
    size = (1301, 700)
    us = views(3)
    n = size[0] * size[1] * 4
    s = torch.cuda.current_stream().cuda_stream

    def run(together):
        w, other = scene(jumps), scene(not jumps if kernel == vrt.KERNEL_MASK_PIXEL else jumps)
        r = vrt.Renderer()
        imgs = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(24)]
        row = torch.full((W,), 0x01ff0000, dtype=torch.int32, device="cuda")
        for k, img in enumerate(imgs):
            if not together:
                torch.cuda.synchronize()
                r = vrt.Renderer()
            frame(torch, r, other if k % 5 == 3 else w, us[k % 3], *size, kernel, img, s)
            if not together:
                torch.cuda.synchronize()
            if k % 3 == 1:
                w.remove_sphere(10 + 3 * k, 3, 30 + k, 6, 1 if jumps else 0)
            if k % 8 == 6:
                w.place_voxel(20 + k, 20, 30, 0x0100ff00)
            if k == 13:
                w.upload_device(row.data_ptr(), 5 * W, W)
        torch.cuda.synchronize()
        return [i.cpu() for i in imgs]

    for k, (a, b) in enumerate(zip(run(True), run(False))):
        assert torch.equal(a, b), k


def test_captured_frames(cuda):
    """A captured frame replays alone, after its renderer is gone, between frames of others."""
    torch = pytest.importorskip("torch")
    size, us, kernel = (801, 600), views(3), vrt.KERNEL_MASK_PIXEL
    n = size[0] * size[1] * 4
    w = scene(False)
    expect = [alone(torch, w, u, *size, kernel)[0] for u in us]
    img = torch.zeros(n, dtype=torch.uint8, device="cuda")
    out = torch.zeros(n, dtype=torch.uint8, device="cuda")
    r, gone, s = vrt.Renderer(), vrt.Renderer(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        frame(torch, r, w, us[0], *size, kernel, img, s.cuda_stream)
        frame(torch, gone, w, us[0], *size, kernel, img, s.cuda_stream)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        g.capture_begin()
        frame(torch, gone, w, us[1], *size, kernel, out, s.cuda_stream)
        g.capture_end()
        s.synchronize()
        gone.close()
        kept = []
        for k in range(40):
            frame(torch, r, w, us[k % 3], *size, kernel, img, s.cuda_stream)
            kept.append(img.clone())
            out.zero_()
            g.replay()
            kept.append(out.clone())
            frame(torch, r, w, us[k % 2], *size, kernel, img, s.cuda_stream)
            g.replay()
    torch.cuda.synchronize()
    assert torch.equal(img.cpu(), expect[39 % 2])
    for k in range(40):
        assert torch.equal(kept[2 * k].cpu(), expect[k % 3]), k
        assert torch.equal(kept[2 * k + 1].cpu(), expect[1]), k


def test_changes_and_probes_in_a_row(cuda):
    """Edits, probes of what they left and uploads queued without a wait give the words, masks
    and answers of the same calls one by one."""
    torch = pytest.importorskip("torch")
    xyz = torch.tensor([[x, 2, z] for x in range(0, W, 5) for z in range(0, W, 5)], dtype=torch.int32, device="cuda")
    row = torch.full((3 * W + 1,), 0x01ff0000, dtype=torch.int32, device="cuda")

    def run(together, jumps):
        w = scene(jumps)
        found = [torch.zeros(len(xyz), dtype=torch.int32, device="cuda") for _ in range(30)]
        torch.cuda.synchronize()
        for k, f in enumerate(found):
            w.remove_sphere(7 + 11 * k % 80, 3, 9 + 17 * k % 80, 5 + k % 4, 1 if jumps else 0)
            if not together:
                torch.cuda.synchronize()
            w.probe(xyz.data_ptr(), len(xyz), f.data_ptr())
            if k % 6 == 2:
                w.place_voxel(5 * (k % 19), 2, 10, 0x0100ff00)
            if k % 10 == 5:
                w.upload_device(row.data_ptr(), 2 * W + 9 + k, row.numel() - 1)
            if not together:
                torch.cuda.synchronize()
        words = np.empty(W * H * W, np.int32)
        w.download(words)
        return [f.cpu() for f in found], words, w.masks(), w.distances()

    for jumps in (False, True):
        a, b = run(True, jumps), run(False, jumps)
        assert all(torch.equal(x, y) for x, y in zip(a[0], b[0]))
        assert np.array_equal(a[1], b[1])
        for p, q in zip(a[2:], b[2:]):
            assert all(np.array_equal(x, y) for x, y in zip(p, q))


UNDRAWN = 7  # fills an image before its frame; a pixel's fourth byte is 255


def fresh_images(torch, n, count):
    return [torch.full((n,), UNDRAWN, dtype=torch.uint8, device="cuda") for _ in range(count)]


# Grids whose CTAs all fit at once: a frame, the changes behind it and the frames behind those
# can all be in place while the first still runs.
ONE_WAVE = [(5, 3), (96, 96), (228, 120), (320, 200)]


@pytest.mark.parametrize("size", ONE_WAVE)
def test_small_word_frames_of_a_turning_camera(cuda, size):
    """A renderer's first 71 word frames on a grid, nothing between them, each into an image of
    its own: the plain frames that record the tiles' classes and those that go by them draw
    every tile."""
    torch = pytest.importorskip("torch")
    w, us = scene(True), views(12)
    n = size[0] * size[1] * 4
    expect = [alone(torch, w, u, *size, vrt.KERNEL_WORD)[0] for u in us]
    s = torch.cuda.current_stream().cuda_stream
    r, imgs = vrt.Renderer(), fresh_images(torch, n, 71)
    order = [(k * k + k // 7) % 12 for k in range(71)]
    torch.cuda.synchronize()
    for i, img in zip(order, imgs):
        frame(torch, r, w, us[i], *size, vrt.KERNEL_WORD, img, s)
    torch.cuda.synchronize()
    for k, (i, img) in enumerate(zip(order, imgs)):
        assert torch.equal(img.cpu(), expect[i]), k


# the kernels of the three frames behind each change: word frames on a world with jumps, and a word
# frame followed by tile frames on one without
@pytest.mark.parametrize("size", ONE_WAVE)
@pytest.mark.parametrize("kernels,jumps", [((vrt.KERNEL_WORD,) * 3, True),
                                           ((vrt.KERNEL_WORD, vrt.KERNEL_MASK_PIXEL, vrt.KERNEL_MASK_PIXEL), False)])
def test_small_frames_behind_changes(cuda, size, kernels, jumps):
    """Changes of the world, each with three frames behind it, all queued without a wait: no frame
    sees the world of before the change, the second and third ones included."""
    torch = pytest.importorskip("torch")
    us, n, rounds = views(3), size[0] * size[1] * 4, 16
    s = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(8)
    slabs = [torch.from_numpy(np.where(rng.random(W * H * 40) < 0.01, 0x01ff0000 + k, -1).astype(np.int32)).cuda()
             for k in range(rounds)]

    def change(w, k):
        if k % 4 == 3:
            w.upload_device(slabs[k].data_ptr(), (7 + 2 * k) * W * H + 11, W * H * 40 - 13)
        if jumps and k % 3 == 0:
            w.fix_depth_field()
        if k % 5 != 4:  # else the frames follow the slab or the whole depth field directly
            w.remove_sphere(10 + 5 * k, 6, 30 + 3 * k, (9, 21, 12)[k % 3], 1 if jumps else 0)
            w.place_voxel(20 + k, 13, 21 + k, 0x0100ff00)

    def run(together):
        w, r = scene(jumps), vrt.Renderer()
        imgs = fresh_images(torch, n, 3 * rounds)
        for k in range(4):  # the renderer's first frames on the grid are plain ones
            frame(torch, r, w, us[k % 3], *size, kernels[0], torch.empty_like(imgs[0]), s)
        for k in range(rounds):
            change(w, k)
            for j in range(3):
                if not together:
                    torch.cuda.synchronize()
                    r = vrt.Renderer()
                frame(torch, r, w, us[(k + j) % 3], *size, kernels[j], imgs[3 * k + j], s)
        torch.cuda.synchronize()
        return [i.cpu() for i in imgs]

    for k, (a, b) in enumerate(zip(run(True), run(False))):
        assert torch.equal(a, b), k
