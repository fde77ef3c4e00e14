"""The forward pass's checkpoints are optional memory: a frame, its gradients and a graph
capture go on where there is none, without asking for it again; the buffer stays where
it is for frames that need no more room; a frame's own buffers come before it; and a
renderer whose first frame no backward pass reads gives it back. A first frame, which is
bound by its allocations, takes no more of them than one per buffer. Allocations are
counted and refused on the host, through the library's allocation hook."""
import ctypes

import numpy as np
import pytest

import gsn
import scenes
from helpers import dev, empty, host, sync, torch
from test_backward_segments_gpu import faint_scene

pytestmark = pytest.mark.gpu

HOOK = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t)
CUDA_ERROR_MEMORY_ALLOCATION = 2
W, H, COUNT, CAPACITY = 64, 48, 1500, 1 << 20
# CAPACITY / 128 blocks of 256 float4: 32 MB; every other buffer here is below 5 MB
LARGE = 16 << 20


class Allocations:
    """Sizes of the library's device allocations while the context is open; `refuse` says
    which of them fail."""

    def __init__(self, refuse=lambda size: False):
        self.refuse, self.sizes = refuse, []
        self.alloc = ctypes.CDLL("libcuda.so.1").cuMemAlloc_v2
        self.alloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
        self.set = getattr(gsn.lib(), "_ZN9gs_native18SetDeviceAllocHookEPF9cudaErrorPPvmE")
        self.set.argtypes = [ctypes.c_void_p]
        self.set.restype = None
        self.hook = HOOK(self.call)

    def call(self, pointer, size):
        self.sizes.append(size)
        if self.refuse(size):
            return CUDA_ERROR_MEMORY_ALLOCATION
        return 0 if self.alloc(pointer, size) == 0 else CUDA_ERROR_MEMORY_ALLOCATION

    def __enter__(self):
        self.set(ctypes.cast(self.hook, ctypes.c_void_p))
        return self

    def __exit__(self, *_):
        self.set(None)

    def large(self):
        return sum(s > LARGE for s in self.sizes)


def scene():
    params = faint_scene(COUNT, 3)
    cam = scenes.make_camera(W, H, fx=60.0, fy=60.0)
    target = np.random.default_rng(4).integers(0, 256, (H, W, 3), dtype=np.uint8)
    return dev(params), cam, dev(target)


def gradients(renderer, solver, p, cam, target, image):
    assert renderer.render(p.data_ptr(), COUNT, cam, [0, 0, 0], image.data_ptr(), 0) == 0
    solver.image_gradients(cam, image.data_ptr(), target.data_ptr())
    ptr = solver.screen_gradients(cam, renderer, image.data_ptr(), p.data_ptr(), COUNT)
    sync()
    return host(ptr, np.float32, 12 * COUNT).reshape(COUNT, 12)


def close(a, b):
    # the same fp32 terms, summed in float atomics over segments or whole lists
    scale = np.abs(b).max(0)
    return np.all(np.abs(a - b) <= 1e-4 * np.abs(b) + 1e-5 * scale)


def steps():
    """Three eager frames with gradients, a capture and three replays."""
    t = torch()
    p, cam, target = scene()
    image = empty((H, W, 3), t.float32)
    r, s, g = gsn.Renderer(), gsn.Solver(), gsn.Graph()
    assert r.set_record_capacity(CAPACITY) == 0
    screens = [gradients(r, s, p, cam, target, image) for _ in range(3)]
    g.capture(r, s, p.data_ptr(), COUNT, [cam], target.data_ptr(), W * H * 3, [0, 0, 0], image.data_ptr(), 0, CAPACITY)
    g.run([0, 0, 0], [1e-4] * 3)
    status = g.check()
    out = screens, p.cpu().numpy(), status
    g.close()
    return out


def test_a_step_and_a_capture_go_on_without_checkpoints():
    screens, params, status = steps()
    with Allocations(lambda size: size > LARGE) as none:
        without, params_without, status_without = steps()
    assert none.large() == 1  # asked for once, not per frame and not inside the capture
    assert status == status_without == 0
    for a, b in zip(without, screens):
        assert close(a, b)
    start = scene()[0].cpu().numpy()
    moved = np.abs(params - start)
    assert moved.max() > 0
    assert np.mean(np.abs(params_without - params) <= 1e-6 + 1e-3 * moved) > 0.999


def test_checkpoints_stay_in_place_for_frames_of_fewer_tiles_than_reserved():
    t = torch()
    p, cam, target = scene()
    r, s = gsn.Renderer(), gsn.Solver()
    assert r.set_record_capacity(CAPACITY) == 0
    image = empty((1024, 1040, 3), t.float32)
    wide = scenes.make_camera(1040, 1024, fx=60.0, fy=60.0)  # 65 x 64 tiles: keeps none
    middle = scenes.make_camera(800, 700, fx=60.0, fy=60.0)
    big_target = empty((1024, 1040, 3), t.uint8)
    gradients(r, s, p, wide, big_target, image)
    for _ in range(2):
        gradients(r, s, p, cam, target, image)
    with Allocations() as seen:
        gradients(r, s, p, middle, big_target, image)
        gradients(r, s, p, cam, target, image)
    assert seen.sizes == []


def test_the_frames_own_buffers_come_before_checkpoints():
    t = torch()
    p, cam, target = scene()
    image = empty((H, W, 3), t.float32)
    r, s = gsn.Renderer(), gsn.Solver()
    for _ in range(2):
        gradients(r, s, p, cam, target, image)  # grow mode, checkpoints held
    n = 40000
    more = dev(faint_scene(n, 8))
    fresh = gsn.Renderer()
    expected, got = empty((H, W, 3), t.float32), empty((H, W, 3), t.float32)
    assert fresh.render(more.data_ptr(), n, cam, [0, 0, 0], expected.data_ptr(), 0) == 0
    refusals = []

    def once(size):  # as if the memory that checkpoints hold were the last
        if size > 1 << 17 and not refusals:
            refusals.append(size)
            return True
        return False

    with Allocations(once):
        assert r.render(more.data_ptr(), n, cam, [0, 0, 0], got.data_ptr(), 0) == 0
    sync()
    assert refusals and torch().equal(expected, got)


def test_a_renderer_that_only_renders_keeps_no_checkpoints():
    t = torch()
    p, cam, target = scene()
    image = empty((H, W, 3), t.float32)
    r, s = gsn.Renderer(), gsn.Solver()

    def render():
        assert r.render(p.data_ptr(), COUNT, cam, [0, 0, 0], image.data_ptr(), 0) == 0
        sync()
        return t.cuda.mem_get_info()[0]

    with Allocations() as seen:
        assert r.set_record_capacity(CAPACITY) == 0
        first = render()
        assert seen.large() == 1  # a first frame may be the first of a step
        for _ in range(2):
            assert render() - first >= LARGE  # it was not: given back
        assert seen.large() == 1
        whole = gradients(r, s, p, cam, target, image)
        assert seen.large() == 2  # by the backward pass, for the frames from now on
        segments = gradients(r, s, p, cam, target, image)
        assert render() < first + LARGE and seen.large() == 2
    assert close(whole, segments)


def test_a_trainers_evaluation_keeps_no_checkpoints():
    p, cam, target = scene()
    rng = np.random.default_rng(6)
    trainer = gsn.Trainer()
    assert trainer.initialize([cam], [target.cpu().numpy()], rng.normal(0, 0.3, (200, 3)) + [0, 0, 3],
                              rng.random((200, 3)), gsn.TrainingOptions.defaults()) == 0
    image = empty((H, W, 3), torch().float32)
    with Allocations() as seen:
        assert trainer.render(cam, image.data_ptr()) == 0
        sync()
    # the first evaluation makes its buffers; whole blocks of 4,096 bytes are checkpoints, or
    # the contributors
    assert [size for size in seen.sizes if size % 4096 == 0] == [4 * W * H]


@pytest.mark.parametrize("culled", [False, True])
@pytest.mark.parametrize("capacity", [0, CAPACITY])
def test_a_first_frame_takes_one_allocation_per_buffer(culled, capacity):
    """12 per-Gaussian buffers (13 with culled counts), offsets with bounds, contributors, five
    record buffers, two scratches (one again for the records in grow mode) and checkpoints."""
    t = torch()
    p, cam, _ = scene()
    image = empty((H, W, 3), t.float32)
    r = gsn.Renderer()
    r.set_exact_culling(culled)
    with Allocations() as seen:
        if capacity:
            assert r.set_record_capacity(capacity) == 0
        assert r.render(p.data_ptr(), COUNT, cam, [0, 0, 0], image.data_ptr(), 0) == 0
        sync()
        assert len(seen.sizes) == 22 + (1 if culled else 0) + (0 if capacity else 1)


def test_an_empty_first_frame_keeps_no_checkpoints():
    t = torch()
    _, cam, _ = scene()
    image = empty((H, W, 3), t.float32)
    r = gsn.Renderer()
    with Allocations() as seen:
        assert r.render(0, 0, cam, [0.25, 0.5, 0.75], image.data_ptr(), 0) == 0
        sync()
        assert len(seen.sizes) == 21
    assert torch().equal(image, t.tensor([0.25, 0.5, 0.75], device="cuda").expand(H, W, 3))
