"""The calls whose speed matters to a user of this library, over their real range.

A case is one pass through the public binding (gs-native_b200/gsn.py):

* ``step``: Renderer.render + Solver.iterate, one training iteration of a model
  held by the caller (or ``steps`` of them through a captured Graph), from the
  4,096-Gaussian single-step scene to 3.0M Gaussians at 2048x1360, in the plain
  fp32 form and in the forms the trainer's options select (exact culling, sparse
  Adam, fast blend arithmetic, bf16 SH storage);
* ``train``: Trainer.train, the whole training loop on host images and points;
* ``render``: a held-out view rendered and scored (Renderer.render + eval_metrics);
* ``views``: MultiView.render of views of uneven resolution;
* ``loss``: the L1 + SSIM gradient alone (Solver.image_gradients), fp32 or tcgen05;
* ``knn``: the 3-NN search that sets the initial scales, on device points;
* ``policy``: the learned density policy, a few fit steps and one inference;
* ``order``: the Morton order of a model and the gather that applies it.

Models follow the seeded distribution of gs-native_b200/scenes.py
(random_gaussians); target images are smooth random photographs with noise.
``exact`` restates every pass in plain torch in 64 bits.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gs-native_b200"))

import gsn  # noqa: E402
import scenes  # noqa: E402

SH_C0 = 0.28209479177387814
VIEWS = 4  # training views a step's state rotates through
# Learning rates of the end of a schedule, so that a model that is stepped a
# thousand times stays the workload it was.
RATES = dict(scale=5e-5, rotation=1e-5, opacity=2.5e-4, sh_dc=2.5e-5, sh_rest=1.25e-6)
POSITION_RATE = 1.5e-5


# ------------------------------------------------------------------ the cases
def step_case(name, n, width, height, focal, radius, sigma, **form):
    case = dict(kind="step", n=n, width=width, height=height, focal=focal, radius=radius, sigma=sigma, log_scale=-3.5,
                logit=0.0, sh=3, bf16=False, cull=False, sparse=False, fast=False, graph=False, steps=1)
    case.update(form)
    if name:
        case["name"] = name
    return case


def listed():
    chosen = dict(bf16=True, cull=True, sparse=True, fast=True)
    return [
        # the smallest call: the 4,096-Gaussian 128x128 scene, where launches and latency count
        step_case("step_tiny", 4096, 128, 128, 140.0, 4.0, 1.0),
        # the start of a run: 100k initial points, half resolution, faint large Gaussians, SH degree 1, fp32 with the
        # trainer's culled / sparse / fast options
        step_case("step_early", 100_003, 800, 532, 700.0, 8.0, 3.0, log_scale=-2.5, logit=-2.0, sh=1, cull=True,
                  sparse=True, fast=True),
        # the plain fp32 form at the model cap of the ring scene (bench.py's baseline form)
        step_case("step_plain", 1_200_000, 1600, 1064, 1400.0, 8.0, 3.0),
        # the same in the form bench.py selects, four steps as graph replays
        step_case("step_graph", 1_200_000, 1600, 1064, 1400.0, 8.0, 3.0, graph=True, steps=4, **chosen),
        # the largest: the two-ring large scene's model and resolution, eager
        step_case("step_large", 3_000_000, 2048, 1360, 1800.0, 10.0, 4.0, **chosen),
        # the whole loop through the Trainer: 20 steady-state iterations per call on a ragged resolution
        dict(name="train_call", kind="train", points=30_011, width=979, height=546, views=12, iterations=20),
        # held-out evaluation of a mid-size model on a ragged resolution
        dict(name="render_eval", kind="render", n=300_007, width=979, height=546, sh=3, sigma=3.0),
        # views of uneven resolution in one call
        dict(name="multiview", kind="views", n=300_007, views=12, sh=3, sigma=3.0),
        # the precision form's tensor-core SSIM gradient on the ring scene's frame
        dict(name="loss_precision", kind="loss", width=1600, height=1064, tensor_core=True),
        # initial scales of a 100k-point cloud
        dict(name="knn_points", kind="knn", n=100_003),
        # the learned density policy: four fit steps on logged samples, then proposals for as many Gaussians
        dict(name="policy", kind="policy", n=300_007, steps=4),
        # the spatial order after a density step at the model cap
        dict(name="spatial_order", kind="order", n=1_200_000, bf16=False),
    ]


def log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "train", "render", "views", "loss", "knn", "policy", "order"])
    width, height = log_uniform(rng, 120, 2048), 0
    height = max(90, int(width * rng.uniform(0.55, 1.0)))
    if kind == "step":
        # the share of the frame and of the model grow together, as the configurations' do
        n = log_uniform(rng, 3000, 1_200_000)
        width = min(2048, max(100, int(150 * (n / 4096.0) ** 0.42 * rng.uniform(0.7, 1.3))))
        height = int(width * rng.uniform(0.55, 1.0))
        small = n < 30_000
        bf16, fast, graph = rng.random() < 0.5, rng.random() < 0.5, n < 400_000 and rng.random() < 0.4
        return step_case(None, n, width, height, width * 0.875, 4.0 if small else 8.0, 1.0 if small else 3.0,
                         log_scale=-3.5, logit=rng.choice([0.0, -1.0]), sh=rng.choice([0, 1, 2, 3, 3]), bf16=bf16,
                         cull=rng.random() < 0.5, sparse=rng.random() < 0.5, fast=fast, graph=graph,
                         steps=3 if graph else 1)
    if kind == "train":
        return dict(kind=kind, points=log_uniform(rng, 5000, 60_000), width=min(width, 1300), height=min(height, 900),
                    views=rng.randint(5, 16), iterations=rng.randint(8, 24))
    if kind == "render":
        return dict(kind=kind, n=log_uniform(rng, 3000, 1_200_000), width=width, height=height, sh=rng.randint(0, 3),
                    sigma=3.0)
    if kind == "views":
        return dict(kind=kind, n=log_uniform(rng, 10_000, 600_000), views=rng.randint(3, 16), sh=rng.randint(0, 3),
                    sigma=3.0)
    if kind == "loss":
        return dict(kind=kind, width=width, height=height, tensor_core=rng.random() < 0.5)
    if kind == "knn":
        return dict(kind=kind, n=log_uniform(rng, 1000, 300_000))
    if kind == "policy":
        return dict(kind=kind, n=log_uniform(rng, 2000, 800_000), steps=rng.randint(2, 6))
    return dict(kind="order", n=log_uniform(rng, 3000, 1_500_000), bf16=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000 + int(seed))


def normal(g, shape, mean=0.0, sigma=1.0):
    return torch.randn(shape, generator=g, device="cuda") * sigma + mean


def morton_order(xyz):
    lo, hi = xyz.amin(1, keepdim=True), xyz.amax(1, keepdim=True)
    q = ((xyz - lo) / (hi - lo).clamp_min(1e-20) * 1023.0).long().clamp(0, 1023)
    key = torch.zeros_like(q[0])
    for bit in range(10):
        for axis in range(3):
            key |= ((q[axis] >> bit) & 1) << (3 * bit + axis)
    return torch.argsort(key, stable=True)


def model_of(n, sigma, g, log_scale=-3.5, logit=0.0, ordered=False):
    """A (58, n) fp32 block of the distribution of scenes.random_gaussians."""
    p = torch.empty((58, n), device="cuda")
    p[0:3] = normal(g, (3, n), 0.0, sigma)
    p[3:6] = normal(g, (3, n), log_scale, 0.5)
    axis = normal(g, (3, n))
    p[6:9] = axis / axis.norm(dim=0, keepdim=True) * (torch.rand(n, generator=g, device="cuda") * math.pi)
    p[9] = normal(g, (n,), logit, 1.0)
    p[10:] = normal(g, (48, n), 0.0, 0.05)
    p[10::16] = normal(g, (3, n), 0.5, 0.2)
    return p[:, morton_order(p[0:3])].contiguous() if ordered else p


def photograph(g, height, width):
    """A u8 HWC target: smooth structure of several scales plus sensor noise."""
    image = torch.zeros((1, 3, height, width), device="cuda")
    for cells, weight in ((4, 0.35), (16, 0.2), (64, 0.12)):
        coarse = torch.rand((1, 3, cells, cells), generator=g, device="cuda")
        image += weight * torch.nn.functional.interpolate(coarse, (height, width), mode="bilinear")
    image += 0.1 + normal(g, image.shape, 0.0, 0.03)
    return (image[0].permute(1, 2, 0).clamp(0, 1) * 255).round().to(torch.uint8).contiguous()


def ring_view(width, height, focal, radius, k, count):
    az, el = 2.0 * math.pi * k / count, math.radians(15.0 if k % 2 == 0 else -15.0)
    R, t = scenes.look_at((radius * math.cos(el) * math.cos(az), radius * math.cos(el) * math.sin(az),
                           radius * math.sin(el)))
    return scenes.pinhole(width, height, focal, focal, R, t)



class DeviceArray:
    def __init__(self, pointer, shape, kind, owner):
        self.owner = owner  # the handle that frees this memory lives as long as the tensor
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=kind, data=(pointer, False), version=3,
                                             strides=None)


def view_of(owner, pointer, shape, kind="<f4"):
    """A handle's device memory as a tensor, without a copy."""
    return torch.as_tensor(DeviceArray(pointer, shape, kind, owner), device="cuda")


def rows_of(block, n, bf16):
    """A parameter or moment block as tensors of its stored types."""
    if not bf16:
        return block.view(58, n)
    flat = block.view(-1)
    return [flat[:10 * n].view(10, n), flat[10 * n:34 * n].view(torch.bfloat16).view(24, n, 2)]


def step_inputs(case, seed):
    g = generator(seed)
    p = model_of(case["n"], case["sigma"], g, case["log_scale"], case["logit"], case["sparse"])
    first = int(seed) % 40
    cams = [ring_view(case["width"], case["height"], case["focal"], case["radius"], first + 7 * k, 40)
            for k in range(VIEWS)]
    targets = torch.stack([photograph(g, case["height"], case["width"]) for _ in range(VIEWS)])
    return p, cams, targets


def uneven_views(case, seed):
    """Poses on a sphere by the seed; the resolutions go round those of scenes.MULTIVIEW_SIZES."""
    sizes = scenes.MULTIVIEW_SIZES
    return [scenes.multiview_cameras(1, seed=100 * int(seed) + k, sizes=(sizes[(3 * k + 2) % len(sizes)],))[0]
            for k in range(case["views"])]


def policy_inputs(case, seed):
    g, n = generator(seed), case["n"]
    f = normal(g, (n, 16)).abs() * torch.rand((n, 16), generator=g, device="cuda") * 2.0
    f[:, 3:6] = normal(g, (n, 3), -1.0, 1.0)
    score = f @ normal(g, (16, 4)) + normal(g, (n, 4), 0.0, 0.5)
    score[:, 0] += 2.0  # most Gaussians are kept
    labels = score.argmax(1).to(torch.int32)
    weights = 1.0 + 2.0 * torch.rand(n, generator=g, device="cuda")
    master = (normal(g, (5508,)) * 0.1).cpu().numpy()
    return f.contiguous(), labels.contiguous(), weights, master


def cloud(case, seed):
    """Half a volume, half two shells, as a reconstruction's point cloud clusters."""
    g, n = generator(seed), case["n"]
    p = normal(g, (n, 3), 0.0, 3.0)
    half = n // 2
    shell = p[:half] / p[:half].norm(dim=1, keepdim=True)
    p[:half] = shell * (2.0 + 2.0 * (torch.arange(half, device="cuda") % 2)[:, None]) + normal(g, (half, 3), 0.0, 0.02)
    return p.contiguous()


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return prepare_step(case, seed)
    if kind == "train":
        return prepare_train(case, seed)
    if kind == "render":
        g = generator(seed)
        s = dict(p=model_of(case["n"], case["sigma"], g), cam=ring_view(case["width"], case["height"],
                 0.875 * case["width"], 8.0, int(seed) % 40, 40), target=photograph(g, case["height"], case["width"]),
                 renderer=gsn.Renderer(), image=torch.empty((case["height"], case["width"], 3), device="cuda"))
    elif kind == "views":
        cams = uneven_views(case, seed)
        s = dict(p=model_of(case["n"], case["sigma"], generator(seed)), cams=cams, mv=gsn.MultiView(),
                 images=[torch.empty((c.height, c.width, 3), device="cuda") for c in cams])
    elif kind == "loss":
        s = loss_inputs(case, seed)
        s["cam"] = scenes.make_camera(case["width"], case["height"])
        s["solver"] = gsn.Solver()
        s["solver"].set_compute_loss(True)
        s["solver"].set_tensor_core_loss(case["tensor_core"])
    elif kind == "knn":
        n = case["n"]
        s = dict(points=cloud(case, seed), dist=torch.empty(n, device="cuda"),
                 near=torch.empty((n, 3), dtype=torch.int32, device="cuda"))
        size = gsn.ctypes.c_size_t()
        gsn.declare("gsn_knn3_workspace", [gsn.ctypes.c_int, gsn.ctypes.POINTER(gsn.ctypes.c_size_t)])(
            n, gsn.ctypes.byref(size))
        s["workspace"] = torch.empty(size.value, dtype=torch.uint8, device="cuda")
        vp = gsn.ctypes.c_void_p
        s["call"] = gsn.declare("gsn_knn3", [vp, gsn.ctypes.c_int, vp, vp, vp, vp])
    elif kind == "policy":
        f, labels, weights, master = policy_inputs(case, seed)
        s = dict(f=f, labels=labels, weights=weights, mlp=gsn.Mlp(), probs=torch.empty((case["n"], 4), device="cuda"),
                 actions=torch.empty(case["n"], dtype=torch.int8, device="cuda"))
        s["mlp"].set_weights(master)
    else:
        p = model_of(case["n"], 3.0, generator(seed))
        block = gsn.to_precision_layout(p, torch) if case["bf16"] else p
        s = dict(p=p, block=block, out=torch.empty_like(block),
                 perm=torch.empty(case["n"], dtype=torch.int32, device="cuda"))
    s["case"] = case
    return s


def prepare_step(case, seed):
    p, cams, targets = step_inputs(case, seed)
    renderer, solver = gsn.Renderer(), gsn.Solver()
    renderer.set_exact_culling(case["cull"])
    renderer.set_fast_blend(case["fast"])
    renderer.set_bf16_sh(case["bf16"])
    solver.set_sparse_adam(case["sparse"])
    solver.set_bf16_sh(case["bf16"])
    solver.set_tensor_core_loss(False)
    solver.set_learning_rates(**RATES)
    block = gsn.to_precision_layout(p, torch) if case["bf16"] else p
    s = dict(case=case, block=block, cams=cams, targets=targets, renderer=renderer, solver=solver, k=0, graph=None,
             image=torch.empty((case["height"], case["width"], 3), device="cuda"))
    if case["graph"]:
        # a captured step needs the record capacity of its largest view
        records = 0
        for c in cams:
            assert renderer.render(block.data_ptr(), case["n"], c, [0, 0, 0], s["image"].data_ptr(), case["sh"]) == 0
            records = max(records, int(renderer.buffers().record_count_host))
        s["graph"] = gsn.Graph()
        s["graph"].capture(renderer, solver, block.data_ptr(), case["n"], cams, targets.data_ptr(),
                           case["width"] * case["height"] * 3, [0, 0, 0], s["image"].data_ptr(), case["sh"],
                           records + records // 2 + 65536)
    return s


def train_inputs(case, seed):
    g = generator(seed)
    images = [photograph(g, case["height"], case["width"]).cpu().numpy() for _ in range(case["views"])]
    points = cloud(dict(n=case["points"]), seed).cpu().numpy()
    colors = torch.rand((case["points"], 3), generator=g, device="cuda").cpu().numpy()
    cams = [ring_view(case["width"], case["height"], 0.875 * case["width"], 8.0, k, case["views"])
            for k in range(case["views"])]
    return images, points, colors, cams


def prepare_train(case, seed):
    images, points, colors, cams = train_inputs(case, seed)
    # the steady state of the schedule (densification over, SH degree at its maximum) in the chosen form
    options = gsn.TrainingOptions.defaults(
        sh_degree_interval=1, densify_until=0, position_lr_init=1.6e-6, position_lr_final=1.6e-6, lr_scale=5e-5,
        lr_rotation=1e-5, lr_opacity=2.5e-4, lr_sh_dc=2.5e-5, lr_sh_rest=1.25e-6, precision=1, graph=1,
        exact_culling=1, sparse_adam=1, spatial_order=1, fast_blend=1, fp32_ssim=1)
    trainer = gsn.Trainer()
    assert trainer.initialize(cams, images, points, colors, options) == 0
    return dict(case=case, trainer=trainer)


def run(s):
    case = s["case"]
    return RUN[case["kind"]](s, case)


def run_step(s, case):
    n, block, image = case["n"], s["block"], s["image"]
    if s["graph"] is not None:
        steps = case["steps"]
        s["graph"].run([(s["k"] + j) % VIEWS for j in range(steps)], [POSITION_RATE] * steps)
        s["k"] += steps
    else:
        v = s["k"] % VIEWS
        s["k"] += 1
        ok = s["renderer"].render(block.data_ptr(), n, s["cams"][v], (0, 0, 0), image.data_ptr(), case["sh"])
        ok = ok or s["solver"].iterate(s["cams"][v], s["renderer"], image.data_ptr(), s["targets"][v].data_ptr(),
                                       block.data_ptr(), n, POSITION_RATE, case["sh"])
        if ok:
            raise RuntimeError("step failed with status %d" % ok)
    if "outputs" not in s:  # the solver's buffers, which the first step made
        m, v, _ = s["solver"].moments()
        stats, absolute = s["solver"].statistics()
        rows = 34 if case["bf16"] else 58
        s["outputs"] = dict(image=image, params=rows_of(block, n, case["bf16"]),
                            first=rows_of(view_of(s["solver"], m, (rows * n,)), n, case["bf16"]),
                            second=rows_of(view_of(s["solver"], v, (rows * n,)), n, case["bf16"]),
                            stats=view_of(s["solver"], stats, (2, n)),
                            absolute=view_of(s["solver"], absolute, (2, n)))
    return s["outputs"]


def run_train(s, case):
    if s["trainer"].train(case["iterations"]) != 0:
        raise RuntimeError("train failed")
    state = s["trainer"].state()
    if s.get("at") != state["params"]:
        s["at"] = state["params"]
        s["outputs"] = rows_of(view_of(s["trainer"], state["params"], (34 * state["count"],)), state["count"], True)
    return s["outputs"]


def run_render(s, case):
    if s["renderer"].render(s["p"].data_ptr(), case["n"], s["cam"], (0, 0, 0), s["image"].data_ptr(), case["sh"]):
        raise RuntimeError("render failed")
    return dict(image=s["image"], **gsn.eval_metrics(s["image"].data_ptr(), s["target"].data_ptr(), case["width"],
                                                     case["height"]))


def run_views(s, case):
    s["mv"].render(s["p"].data_ptr(), case["n"], s["cams"], [x.data_ptr() for x in s["images"]], (0, 0, 0), case["sh"])
    return s["images"]


def run_loss(s, case):
    grad = s["solver"].image_gradients(s["cam"], s["image"].data_ptr(), s["target"].data_ptr())
    return dict(grad=view_of(s["solver"], grad, (case["height"], case["width"], 3)),
                loss=view_of(s["solver"], s["solver"].loss_device(), (4,), "<f8"))


def run_knn(s, case):
    if s["call"](s["points"].data_ptr(), case["n"], s["dist"].data_ptr(), s["near"].data_ptr(),
                 s["workspace"].data_ptr(), None):
        raise RuntimeError("knn failed")
    return dict(dist=s["dist"], near=s["near"])


def run_policy(s, case):
    n, mlp = case["n"], s["mlp"]
    loss = mlp.train(s["f"].data_ptr(), s["labels"].data_ptr(), s["weights"].data_ptr(), n, case["steps"], 1e-3)
    mlp.infer(s["f"].data_ptr(), n, 0.9, s["actions"].data_ptr(), s["probs"].data_ptr())
    return dict(loss=loss, weights=mlp.weights(), actions=s["actions"], probs=s["probs"])


def run_order(s, case):
    gsn.spatial_permutation(s["p"].data_ptr(), case["n"], s["perm"].data_ptr())
    gsn.gather_gaussians(s["block"].data_ptr(), s["out"].data_ptr(), s["perm"].data_ptr(), case["n"], case["bf16"])
    return dict(perm=s["perm"], block=s["out"].view(torch.int32))


RUN = dict(step=run_step, train=run_train, render=run_render, views=run_views, loss=run_loss, knn=run_knn,
           policy=run_policy, order=run_order)


# ------------------------------------------------------------------ what a pass cannot do without
# Blended (pixel, record) pairs per pixel of these scenes, about what a counting render of the 1.2M ring scene
# reports (73); forward and backward FLOP of one pair.
PAIRS, FORWARD, BACKWARD = 60, 16, 46


def work(case):
    kind = case["kind"]
    if kind in ("knn", "policy", "order"):
        n = case["n"]
        if kind == "knn":
            return dict(bytes=n * (12 + 4 + 12), flops=n * 30 * math.log2(max(n, 2)))
        if kind == "policy":
            return dict(bytes=n * (64 + 4 + 4) * case["steps"] + n * (64 + 1 + 16),
                        flops=n * 5376 * 2 * (3 * case["steps"] + 1))
        return dict(bytes=n * ((34 if case["bf16"] else 58) * 8 + 12 + 4), flops=n * 30)
    if kind == "views":
        pixels = int(case["views"] * 1.9e6)
        return dict(bytes=case["views"] * case["n"] * 232 + pixels * 12, flops=pixels * PAIRS * FORWARD)
    pixels = case["width"] * case["height"]
    if kind == "loss":
        return dict(bytes=pixels * 27, flops=pixels * 3 * 2 * 11 * 2 * 8)
    if kind == "render":
        return dict(bytes=case["n"] * 232 + pixels * (12 + 12 + 3), flops=pixels * (PAIRS * FORWARD + 3 * 11 * 20))
    if kind == "train":
        steps, n, rows, touched = case["iterations"], case["points"], 136, 0.9
    else:
        steps, n, rows = case["steps"], case["n"], 136 if case["bf16"] else 232
        touched = 0.6 if case["sparse"] else 1.0  # the visible share of a ring view
    return dict(bytes=steps * (n * rows * (1 + 5 * touched) + n * 16 + pixels * 15),
                flops=steps * pixels * (PAIRS * (FORWARD + BACKWARD) + 3 * 2 * 11 * 2 * 8))


def tolerance(case):
    kind = case["kind"]
    if kind == "order":
        return "exact"
    if kind == "knn":
        # fp32 distances (5e-8 off exact); equal third distances may resolve to another neighbour
        return dict(rel=1e-6, max=1e-5, differ=1e-4)
    if kind == "policy":
        # fp32 sums over the samples (4e-7 off exact); a working weight may round to the other fp16 neighbour
        return dict(rel=1e-5, max=1e-2, differ=1e-3)
    if kind == "loss":
        # hi / lo bf16 products (4e-4 off exact), or fp32 filters (3e-6)
        return dict(rel=2e-3, max=0.05) if case["tensor_core"] else dict(rel=2e-5, max=2e-2)
    if kind in ("render", "views"):
        # fp32 blends (1e-6 to 9e-6 off exact); a value at the 1/255 or 1e-4 threshold may fall on the other side
        return dict(rel=3e-5, max=2e-2)
    if kind == "train":
        # 20 steps of the bf16 form, each one's rounding travelling through the next
        return dict(rel=8e-3, max=0.9)
    # moments off exact by 6e-5 (plain), 2e-4 (24-bit depth order) and 2e-3 (bf16 moments): float-atomic sums, and
    # values at the blend's thresholds, whose flips reach single elements
    return dict(rel=8e-3 if case["bf16"] else 1e-3 if case["fast"] else 3e-4, max=0.9 if case["steps"] > 1 else 0.5)


# ------------------------------------------------------------------ 64-bit restatement
def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return exact_step(case, seed)
    if kind == "render":
        g = generator(seed)
        p = model_of(case["n"], case["sigma"], g).double()
        cam = ring_view(case["width"], case["height"], 0.875 * case["width"], 8.0, int(seed) % 40, 40)
        target = photograph(g, case["height"], case["width"]).double() / 255.0
        with torch.no_grad():
            image = Frame64(p, cam, case["sh"]).blend()
            clamped = image.clamp(0, 1)
            mse = (clamped - target).square().mean().item()
            return dict(image=image, psnr=-10.0 * math.log10(mse), ssim=ssim64(clamped, target).mean().item(),
                        l1=(clamped - target).abs().mean().item(), mse=mse)
    if kind == "views":
        p = model_of(case["n"], case["sigma"], generator(seed)).double()
        with torch.no_grad():
            return [Frame64(p, c, case["sh"]).blend() for c in uneven_views(case, seed)]
    if kind == "loss":
        s = loss_inputs(case, seed)
        grad, values = loss64(s["image"].double(), s["target"])
        return dict(grad=grad, loss=values)
    if kind == "knn":
        points = cloud(case, seed).double()
        dist = []
        for chunk in points.split(max(1, 20_000_000 // case["n"])):
            d = torch.zeros((len(chunk), case["n"]), dtype=torch.float64, device="cuda")
            for a in range(3):
                d += (chunk[:, a, None] - points[None, :, a]).square()
            dist.append(d.topk(4, dim=1, largest=False, sorted=True).values[:, 1:].mean(1))
        return dict(dist=torch.cat(dist), near=None)
    if kind == "policy":
        return exact_policy(case, seed)
    return None


def loss_inputs(case, seed):
    g = generator(seed)
    target = photograph(g, case["height"], case["width"])
    # a render that has come part of the way to its target
    image = (target.float() / 255.0 + normal(g, target.shape, 0.01, 0.05)).clamp(0, 1.2).contiguous()
    return dict(image=image, target=target)


def exact_policy(case, seed):
    f, labels, weights, master = policy_inputs(case, seed)
    f, w, y = f.double(), weights.double() / weights.double().sum(), labels.long()
    p = torch.from_numpy(master).cuda().double()
    m, v, loss = torch.zeros_like(p), torch.zeros_like(p), 0.0

    def logits(half):
        W1, b1, W2, b2, W3, b3 = torch.split(half, [1024, 64, 4096, 64, 256, 4])
        h = torch.relu(f @ W1.view(64, 16).T + b1)
        h = torch.relu(h @ W2.view(64, 64).T + b2)
        return h @ W3.view(4, 64).T + b3

    for k in range(1, case["steps"] + 1):
        half = p.half().double().requires_grad_(True)
        value = (torch.nn.functional.cross_entropy(logits(half), y, reduction="none") * w).sum()
        grad, = torch.autograd.grad(value, half)
        loss = value.item()
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad.square()
        p = p - 1e-3 * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
    with torch.no_grad():
        probs = torch.softmax(logits(p.half().double()), 1)
    return dict(loss=loss, weights=p.cpu().numpy(), actions=None, probs=probs)


def window64(n):
    """The 11-tap Gaussian window (sigma 1.5, zero padding) as a banded matrix."""
    taps = torch.exp(-(torch.arange(11, dtype=torch.float64, device="cuda") - 5).square() / 4.5)
    taps = taps / taps.sum()
    out = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for k in range(11):
        d = torch.full((max(n - abs(k - 5), 0),), taps[k].item(), dtype=torch.float64, device="cuda")
        if len(d):
            out += torch.diag(d, k - 5)
    return out


def ssim64(x, y):
    wv, wh = window64(x.shape[0]), window64(x.shape[1])

    def blur(t):
        return wv @ (t.permute(2, 0, 1) @ wh)

    a, b = blur(x), blur(y)
    aa, bb, ab = blur(x * x) - a * a, blur(y * y) - b * b, blur(x * y) - a * b
    return (2 * a * b + 1e-4) * (2 * ab + 9e-4) / ((a * a + b * b + 1e-4) * (aa + bb + 9e-4))


def loss64(image, target):
    image = image.detach().requires_grad_(True)
    t = target.double() / 255.0
    ssim, l1 = ssim64(image, t).mean(), (image - t).abs().mean()
    loss = 0.8 * l1 + 0.2 * (1 - ssim)
    grad, = torch.autograd.grad(loss, image)
    psnr = -10.0 * torch.log10((image - t).square().mean())
    return grad, torch.stack([loss, l1, ssim, psnr]).detach()


def sh_basis64(d, degree):
    x, y, z = d
    xx, yy, zz = x * x, y * y, z * z
    b = [torch.full_like(x, SH_C0)]
    if degree > 0:
        b += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree > 1:
        b += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
              -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy)]
    if degree > 2:
        b += [-0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
              -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
              -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
              -0.5900435899266435 * x * (xx - 3 * yy)]
    return torch.stack(b)


class Frame64:
    """One view of a model in 64 bits: projection, per-tile lists, blend and its gradients."""

    def __init__(self, p, cam, degree):
        self.p, self.cam = p, cam
        self.w, self.h = cam.width, cam.height
        R = torch.tensor(list(cam.R_c_w), dtype=torch.float64, device="cuda").view(3, 3)
        t = torch.tensor(list(cam.t_c_w), dtype=torch.float64, device="cuda")
        c = R @ p[0:3] + t[:, None]
        z = c[2]
        self.front = (z > cam.near_depth) & (z <= cam.far_depth)
        z = torch.where(self.front, z, torch.ones_like(z))
        w = p[6:9]
        angle = w.square().sum(0).clamp_min(1e-30).sqrt()
        ax = w / angle
        co, si = torch.cos(angle), torch.sin(angle)
        zero = torch.zeros_like(co)
        K = torch.stack([zero, -ax[2], ax[1], ax[2], zero, -ax[0], -ax[1], ax[0], zero]).view(3, 3, -1)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")[:, :, None]
        rot = eye * co + si * K + (1 - co) * (ax[:, None] * ax[None])
        M = torch.einsum("ij,jkn->ikn", R, rot) * torch.exp(p[3:6])[None]
        V = (M[:, None] * M[None]).sum(2)
        lx, ly = 0.65 * self.w / cam.fx, 0.65 * self.h / cam.fy
        nx, ny = c[0] / z, c[1] / z
        jx, jy = nx.clamp(-lx, lx), ny.clamp(-ly, ly)
        J0 = torch.stack([cam.fx / z, zero, -cam.fx * jx / z])
        J1 = torch.stack([zero, cam.fy / z, -cam.fy * jy / z])
        VJ0, VJ1 = (V * J0[None]).sum(1), (V * J1[None]).sum(1)
        a, b, d = (J0 * VJ0).sum(0) + 0.3, (J1 * VJ0).sum(0), (J1 * VJ1).sum(0) + 0.3
        det = a * d - b * b
        u, v = cam.fx * nx + cam.cx, cam.fy * ny + cam.cy
        view = p[0:3] + (R.T @ t)[:, None]
        view = view / view.norm(dim=0, keepdim=True)
        basis = sh_basis64(view, degree)
        k = (degree + 1) ** 2
        rgb = (torch.stack([(basis * p[10 + 16 * ch:10 + 16 * ch + k]).sum(0) for ch in range(3)]) + 0.5).clamp_min(0)
        self.screen = torch.stack([u, v, d / det, -b / det, a / det, torch.sigmoid(p[9]), rgb[0], rgb[1], rgb[2]])
        self.covariance = (a, b, d)
        with torch.no_grad():
            self.lists(u, v, z, a, d, det)

    def lists(self, u, v, z, a, d, det):
        mid = 0.5 * (a + d)
        r = torch.ceil(3 * (mid + (mid * mid - det).clamp_min(0.1).sqrt()).sqrt())
        tx, ty = self.cam.tile_count_x, self.cam.tile_count_y
        x0, x1 = ((u - r) / 16).clamp(0, tx).long(), ((u + r + 15) / 16).clamp(0, tx).long()
        y0, y1 = ((v - r) / 16).clamp(0, ty).long(), ((v + r + 15) / 16).clamp(0, ty).long()
        self.visible = self.front & (det > 0) & (x0 < x1) & (y0 < y1)
        ids = torch.nonzero(self.visible)[:, 0]
        ids = ids[torch.argsort(z[ids].float(), stable=True)]
        wide = (x1 - x0)[ids]
        count = wide * (y1 - y0)[ids]
        first = torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
        k = torch.arange(len(first), device="cuda") - first
        rep = torch.repeat_interleave(ids, count)
        wide = torch.repeat_interleave(wide, count)
        tile = (y0[rep] + k // wide) * tx + x0[rep] + k % wide
        order = torch.argsort(tile.int(), stable=True)
        self.records = rep[order]
        per_tile = torch.bincount(tile, minlength=tx * ty)
        self.begin = torch.cumsum(per_tile, 0) - per_tile
        self.count = per_tile

    def batches(self, carry, backward):
        """Walks groups of tiles through their lists 32 records at a time."""
        tx = self.cam.tile_count_x
        order = torch.argsort(self.count, descending=True)
        lane = torch.arange(256, device="cuda")
        table = torch.cat([self.screen.detach(), torch.zeros((9, 1), dtype=torch.float64, device="cuda")], 1)
        empty = table.shape[1] - 1
        for tiles in order.split(1024):
            px = (tiles % tx * 16)[:, None] + lane % 16
            py = (tiles // tx * 16)[:, None] + lane // 16
            inside = (px < self.w) & (py < self.h)
            pix = torch.where(inside, py * self.w + px, torch.zeros_like(px))
            T = torch.ones_like(px, dtype=torch.float64)
            done = ~inside
            state = carry(pix, inside)
            longest = int(self.count[tiles].max())
            for base in range(0, longest, 32):
                k = base + torch.arange(32, device="cuda")
                real = k[None] < self.count[tiles][:, None]
                ids = torch.where(real, self.records[(self.begin[tiles][:, None] + k).clamp_max(
                    max(len(self.records) - 1, 0))], torch.full_like(real, empty, dtype=torch.long))
                q = table[:, ids]  # 9 x tiles x 32
                dx, dy = q[0][..., None] - px[:, None], q[1][..., None] - py[:, None]
                power = -0.5 * (q[2][..., None] * dx * dx + q[4][..., None] * dy * dy) - q[3][..., None] * dx * dy
                raw = q[5][..., None] * torch.exp(power)
                alpha = raw.clamp_max(0.99)
                alpha = torch.where((alpha < 1.0 / 255.0) | (power > 0) | done[:, None], torch.zeros_like(alpha), alpha)
                after = T[:, None] * torch.cumprod(1 - alpha, 1)
                kept = after >= 1e-4
                alpha = alpha * kept
                through = T[:, None] * torch.cat([torch.ones_like(alpha[:, :1]), torch.cumprod(1 - alpha, 1)], 1)
                backward(state, q, ids, dx, dy, raw, alpha, through[:, :-1])
                T = through[:, -1]
                done = done | ~kept[:, -1]
                if bool(done.all()):
                    break
            state["finish"]()

    def blend(self):
        image = torch.zeros((self.h * self.w, 3), dtype=torch.float64, device="cuda")

        def carry(pix, inside):
            s = dict(C=torch.zeros(pix.shape + (3,), dtype=torch.float64, device="cuda"))
            s["finish"] = lambda: image.index_put_((pix[inside],), s["C"][inside])
            return s

        def add(s, q, ids, dx, dy, raw, alpha, through):
            s["C"] += torch.einsum("tkp,ctk->tpc", alpha * through, q[6:9])

        self.batches(carry, add)
        return image.view(self.h, self.w, 3)

    def gradients(self, image, grad):
        """d loss / d screen values (9 x n) and the sums of |d u|, |d v|."""
        n = self.screen.shape[1]
        out = torch.zeros((11, n + 1), dtype=torch.float64, device="cuda")
        flat, gflat = image.reshape(-1, 3), grad.reshape(-1, 3)

        def carry(pix, inside):
            g = gflat[pix] * inside[..., None]
            S = (g * flat[pix]).sum(-1)
            return dict(g=g, S=S, P=torch.zeros_like(S), finish=lambda: None)

        def add(s, q, ids, dx, dy, raw, alpha, through):
            G = torch.einsum("tpc,ctk->tkp", s["g"], q[6:9])
            weight = alpha * through
            front = s["P"][:, None] + torch.cumsum(weight * G, 1)
            s["P"] = front[:, -1]
            dalpha = (front - weight * G + through * G - s["S"][:, None]) / (1 - alpha)
            common = torch.where((alpha > 0) & (raw < 0.99), dalpha * alpha, torch.zeros_like(alpha))
            du = -common * (q[2][..., None] * dx + q[3][..., None] * dy)
            dv = -common * (q[4][..., None] * dy + q[3][..., None] * dx)
            values = [du.sum(2), dv.sum(2), (-0.5 * common * dx * dx).sum(2), (-common * dx * dy).sum(2),
                      (-0.5 * common * dy * dy).sum(2), common.sum(2) / q[5].clamp_min(1e-300)]
            colour = torch.einsum("tkp,tpc->ctk", weight, s["g"])
            values += [colour[0], colour[1], colour[2], du.abs().sum(2), dv.abs().sum(2)]
            out.index_add_(1, ids.reshape(-1), torch.stack(values).reshape(11, -1))

        self.batches(carry, add)
        return out[:9, :n], out[9:, :n]


def exact_step(case, seed):
    p32, cams, targets = step_inputs(case, seed)
    p = p32.double()
    if case["bf16"]:
        p[10:] = p32[10:].to(torch.bfloat16).double()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    rate = torch.tensor([POSITION_RATE] * 3 + [RATES["scale"]] * 3 + [RATES["rotation"]] * 3 + [RATES["opacity"]] +
                        ([RATES["sh_dc"]] + [RATES["sh_rest"]] * 15) * 3, dtype=torch.float64, device="cuda")[:, None]
    for k in range(1, case["steps"] + 1):
        leaf = p.detach().requires_grad_(True)
        frame = Frame64(leaf, cams[(k - 1) % VIEWS], case["sh"])
        with torch.no_grad():
            image = frame.blend()
        gimage, _ = loss64(image, targets[(k - 1) % VIEWS])
        with torch.no_grad():
            screen, absolute = frame.gradients(image, gimage)
        screen = torch.where(frame.visible, screen, torch.zeros_like(screen))
        # an invisible Gaussian's screen values can be infinite: they take no gradient
        grad, = torch.autograd.grad(frame.screen, leaf, screen)
        grad = torch.where(frame.visible, grad, torch.zeros_like(grad))
        with torch.no_grad():
            m1, v1 = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad.square()
            p1 = p - rate * (m1 / (1 - 0.9 ** k)) / ((v1 / (1 - 0.999 ** k)).sqrt() + 1e-15)
            live = frame.visible if case["sparse"] else torch.ones_like(frame.visible)
            p, m, v = torch.where(live, p1, p), torch.where(live, m1, m), torch.where(live, v1, v)
            half = torch.tensor([[0.5 * case["width"]], [0.5 * case["height"]]], dtype=torch.float64, device="cuda")
            stats = torch.stack([(screen[:2] * half).norm(dim=0), frame.visible.double()])
            absolute = torch.stack([(absolute * half).norm(dim=0), absolute[1]])
        del leaf, frame, grad, screen

    def rows(block):
        return [block[:10], block[10:].view(24, 2, -1).transpose(1, 2)] if case["bf16"] else block

    return dict(image=image, params=rows(p), first=rows(m), second=rows(v), stats=stats, absolute=absolute)
