"""What is timed: the work a program that uses this package has it do, through its public entry points.

    image      NeuralPrimitiveSceneTileCUDA.forward, one frame (precision fp16, bf16 or fp32)
    depth      ...render_rgb_t_no_grad: colour, expected depth and opacity of one frame
    features   ...forward(return_feature=True): one frame with its per-pixel feature map
    query      ...render_feature_map, then FeatureUpsampleDecoder.classify: an open-vocabulary label map
    views      engine.ViewBatchRenderer.render: several views of a scene per call (an evaluation sweep, a video)
    stream     engine.FramePipeline: frames from host rays to host images, several in flight (serving)
    gradients  the backward half of a training step from saved records: primitive_records_reverse (reverse compositing),
               group_records, grouped_weight_gradients
    step       a whole training step: cumodel.render_tiles_training_records, which packs the scene's current weights
               on each call as they change with each step, the loss, and the backward half

Scenes are the seeded distributions of synthetic.make_scene_device: centres uniform in a cube, log-normal scales,
random rotations, Xavier weights that binary16 represents, cameras on a circle of radius 3.
"""
import functools
import math

import numpy as np
import torch

import mlp_splatting_b200  # noqa: F401  (makes the package importable under this name)
from mlp_splatting_b200 import synthetic

THRESHOLD = 5.0e-3      # hit-test threshold of the reference's inference benchmark
RECORDS_PER_PIXEL = 9.5     # records a pixel composites before its transmittance is below 1e-3 (face-on views)
PARAMETERS = ("positions", "log_scales", "quats", "W1", "b1", "W2", "b2", "W3", "b3")


def listed():
    return [
        # the smallest frame: the 2,000-primitive scene that also runs on a CPU; latency of one call
        dict(name="image_2k_128x96", kind="image", n=2_000, W=128, H=96, mu=-3.5, hidden=32, precision="fp16"),
        # the headline frame: an interactive viewer's view of a room-sized scene
        dict(name="image_100k_1200x680", kind="image", n=100_000, W=1200, H=680, mu=-4.2, hidden=32, precision="fp16"),
        # the same frame in the reference's default FP32 numerics
        dict(name="image_fp32_100k_1200x680", kind="image", n=100_000, W=1200, H=680, mu=-4.2, hidden=32, precision="fp32"),
        # depth for a mesh or a point cloud, at an image size that no tile divides
        dict(name="depth_60k_639x477", kind="depth", n=60_000, W=639, H=477, mu=-4.2, hidden=32, precision="fp16"),
        # full-width semantic features of one view
        dict(name="features512_250k_1200x680", kind="features", n=250_000, W=1200, H=680, mu=-4.8, hidden=32,
             precision="fp16", channels=512),
        # low-dimensional features, decoded and queried with 20 text embeddings; an odd image size
        dict(name="query128_120k_957x541", kind="query", n=120_000, W=957, H=541, mu=-4.6, hidden=32, precision="fp16",
             channels=128, classes=20),
        # four views 90 degrees apart of a large scene, in one batch
        dict(name="views4_500k_1200x680", kind="views", n=500_000, W=1200, H=680, mu=-5.2, hidden=32, precision="fp16",
             views=4, step=90.0),
        # the largest: neighbouring views of an orbit, 64-wide layers, more primitives than a frame has pixels to show
        dict(name="views4_1m_hidden64_1920x1080", kind="views", n=1_000_000, W=1920, H=1080, mu=-6.05, hidden=64,
             precision="fp16", views=4, step=11.25),
        # a rendering service: eight requests from pinned host memory to pinned host memory
        dict(name="stream8_100k_1200x680", kind="stream", n=100_000, W=1200, H=680, mu=-4.2, hidden=32, precision="fp16",
             frames=8),
        # a training step on a small training image
        dict(name="step_20k_320x240", kind="step", n=20_000, W=320, H=240, mu=-4.0, hidden=32, precision="fp16"),
        # backward half of a training step, mixed precision, about 90 records per primitive
        dict(name="gradients_50k_800x600", kind="gradients", n=50_000, W=800, H=600, mu=-4.2, hidden=32, precision="fp16"),
        # the smallest backward, in IEEE FP32
        dict(name="gradients_fp32_2k_128x96", kind="gradients", n=2_000, W=128, H=96, mu=-3.5, hidden=32, precision="fp32"),
    ]


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _mu(n, H, most):
    """Mean log-scale at which the densest tile of a face-on view holds about `most` candidates (the capacity is 1,536):
    n / 4 * (tile width + 12 exp(mu))^2, with the tile's width in the scene 27.7 / H.  At most -3.5."""
    return round(min(-3.5, math.log((math.sqrt(4.0 * most / n) - 27.7 / H) / 12.0)), 3)


def draw(rng):
    kind = rng.choice(["image", "image", "image", "depth", "features", "query", "views", "stream", "step", "gradients",
                       "gradients"])
    low, high = {"image": (2_000, 400_000), "depth": (2_000, 250_000), "features": (10_000, 250_000),
                 "query": (10_000, 250_000), "views": (20_000, 500_000), "stream": (2_000, 200_000),
                 "step": (2_000, 40_000), "gradients": (1_000, 50_000)}[kind]
    n = int(_log(rng, low, high))
    # a tile may not see more of the scene than its candidate list holds: large scenes come with large images
    H = int(_log(rng, max(64.0, 1.15 * math.sqrt(n / 2.08)), 600.0 if kind in ("step", "gradients") else 760.0))
    W = int(H * rng.uniform(1.2, 1.8))
    c = dict(kind=kind, n=n, W=W, H=H, mu=_mu(n, H, 700.0 if kind == "views" else 900.0), hidden=32, precision="fp16")
    if kind == "image":
        c["precision"] = rng.choice(["fp16", "fp16", "fp16", "bf16", "fp32"])
        c["hidden"] = rng.choice([32, 32, 32, 64]) if n <= 250_000 else 32
    elif kind == "features":
        c["channels"] = rng.choice([64, 128, 256, 384, 512])
    elif kind == "query":
        c["channels"] = rng.choice([64, 128])
        c["classes"] = rng.randint(5, 100)
    elif kind == "views":
        c["hidden"] = rng.choice([32, 64])
        c["views"] = rng.randint(2, 6)
        c["step"] = rng.choice([90.0, 11.25]) if c["views"] <= 4 else 5.0
    elif kind == "stream":
        c["frames"] = rng.randint(4, 12)
    elif kind == "depth":
        c["precision"] = rng.choice(["fp16", "fp16", "fp32"])
    elif kind == "step":
        c["precision"] = rng.choice(["fp16", "fp32"])
    elif kind == "gradients":
        c["precision"] = rng.choice(["fp16", "fp16", "bf16", "fp32"])
    return c


@functools.lru_cache(maxsize=32)
def _camera(W, H, azimuth):
    return synthetic.make_camera(W, H, azimuth_deg=azimuth)


def _device_camera(case, azimuth=0.0):
    cam = _camera(case["W"], case["H"], azimuth)
    return {k: torch.from_numpy(np.ascontiguousarray(cam[k])).cuda() for k in ("rays_o", "rays_d", "view", "proj")}


def _scene(case, seed, n=None, parts=("geometry", "weights")):
    return synthetic.make_scene_device(case["n"] if n is None else n, seed, torch.device("cuda"), mu=case["mu"],
                                       hidden=case["hidden"], feat_dim=case.get("channels", 0), parts=parts)


def _module(case, seed):
    """The renderer module with the scene's parameters, as after load_state_dict."""
    from mlp_splatting_b200.cumodel import NeuralPrimitiveSceneTileCUDA
    with torch.device("cuda"):
        model = NeuralPrimitiveSceneTileCUDA(num_primitives=case["n"], hidden_dim=case["hidden"], pe_frequencies=6,
                                             feature_dim_low=case.get("channels", 0), precision=case["precision"],
                                             wide_hidden=case["hidden"] > 32)
    scene = _scene(case, seed)
    with torch.no_grad():
        for k in PARAMETERS + (("feat_attr",) if "channels" in case else ()):
            getattr(model, k).copy_(scene.pop(k))
    model.set_image_size(case["W"], case["H"])
    return model


def _packed_image(case, seed, chunk=131_072):
    """A scene that keeps geometry and the packed fp16 weights only; its FP32 weights are drawn and packed slice by slice."""
    from mlp_splatting_b200.engine import PackedScene
    geo = _scene(case, seed, parts=("geometry",))
    images = []
    for a in range(0, case["n"], chunk):
        m = min(chunk, case["n"] - a)
        w = _scene(case, seed + 1 + a, n=m, parts=("weights",))
        part = PackedScene(geo["positions"][a:a + m], geo["log_scales"][a:a + m], geo["quats"][a:a + m], w["W1"], w["b1"], w["W2"],
                           w["b2"], w["W3"], w["b3"], geo["freq"], geo["att"])
        images.append(part.w16)
        del w, part
    image = torch.cat(images)
    return PackedScene.from_packed_image(geo["positions"], geo["log_scales"], geo["quats"], geo["freq"], geo["att"], image,
                                         case["hidden"])


def _record_tensors(case, seed):
    """The 15 tensors of the record entry point, tile lists included."""
    from mlp_splatting_b200.engine import FrameRenderer, PackedScene, normalize_rows
    scene = _scene(case, seed)
    cam = _device_camera(case)
    rays_d = normalize_rows(cam["rays_d"])
    quats = normalize_rows(scene["quats"])
    packed = PackedScene(*(scene[k] for k in PARAMETERS), scene["freq"], scene["att"], pack_f16=False)
    renderer = FrameRenderer(case["W"], case["H"], max_records=0)
    prims, offsets = renderer.bin(packed, cam["view"].cpu().numpy(), cam["proj"].cpu().numpy(), THRESHOLD)
    return [cam["rays_o"], rays_d, scene["positions"], scene["log_scales"], quats, prims.clone(), offsets.clone(), scene["freq"],
            scene["att"], *(scene[k] for k in PARAMETERS[3:])]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("image", "depth", "features", "query"):
        state = dict(kind=kind, model=_module(case, seed), cam=_device_camera(case), size=(case["H"], case["W"]))
        if kind == "query":
            from mlp_splatting_b200.feature_decoder import FeatureUpsampleDecoder
            weights, text = synthetic.make_decoder(case["channels"], 128, 512, case["classes"], seed=seed)
            decoder = FeatureUpsampleDecoder(case["channels"], 512, 128)
            decoder.load_state_dict({k: torch.from_numpy(v) for k, v in weights.items()})
            state.update(decoder=decoder, text=torch.from_numpy(text).cuda())
        return state
    if kind == "views":
        from mlp_splatting_b200.engine import ViewBatchRenderer
        cams = [_camera(case["W"], case["H"], case["step"] * v) for v in range(case["views"])]
        rays = [_device_camera(case, case["step"] * v) for v in range(case["views"])]
        batch = ViewBatchRenderer(case["W"], case["H"], case["views"], max_records=16 * case["views"] * case["W"] * case["H"])
        return dict(kind=kind, scene=_packed_image(case, seed), batch=batch, rays_o=[r["rays_o"] for r in rays],
                    rays_d=[r["rays_d"] for r in rays], view=[c["view"] for c in cams], proj=[c["proj"] for c in cams])
    if kind == "stream":
        from mlp_splatting_b200.engine import FramePipeline
        scene = _packed_image(case, seed)
        frames = []
        for f in range(case["frames"]):     # a camera that moves by a degree per request
            cam = _camera(case["W"], case["H"], float(f))
            P = case["W"] * case["H"]
            frames.append(dict(view=cam["view"], proj=cam["proj"],
                               rays_o=torch.from_numpy(cam["rays_o"][:1].copy()).pin_memory(),     # one origin for all rays
                               rays_d=torch.from_numpy(cam["rays_d"]).pin_memory(),
                               rgb=torch.empty((P, 3), pin_memory=True), alpha=torch.empty((P, 1), pin_memory=True)))
        return dict(kind=kind, pipe=FramePipeline(scene, case["W"], case["H"], depth=case["frames"]), frames=frames)
    tensors = _record_tensors(case, seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    pixels = case["W"] * case["H"]
    target = torch.rand((pixels, 3), generator=g, device="cuda")
    grad_t = torch.randn(pixels, generator=g, device="cuda") * (0.03 / pixels)
    state = dict(kind=kind, n=case["n"], tensors=tensors, size=(case["W"], case["H"]), target=target, grad_t=grad_t,
                 precision={"fp16": "float16", "bf16": "bfloat16", "fp32": "float32"}[case["precision"]])
    if kind == "gradients":
        from mlp_splatting_b200.cumodel import render_tiles_training_records
        state["records"] = render_tiles_training_records(tensors, case["W"], case["H"], 8, THRESHOLD, 1.5, 2.0)
        state["grad_rgb"] = _loss_gradient(state["records"][0], target)
    return state


def _loss_gradient(rgb, target):
    return (rgb - target) * (2.0 / rgb.numel())     # of the mean squared error


def _backward(state, records, grad_rgb):
    from mlp_splatting_b200.primitive_csr import group_records, primitive_records_reverse
    from mlp_splatting_b200.primitive_gemm import grouped_weight_gradients
    _rgb, _alpha, ids, x6, raw, masks, _gates, offsets = records
    log_scales, quats, freq, att, weights = (state["tensors"][3], state["tensors"][4], state["tensors"][7], state["tensors"][8],
                                             state["tensors"][9:15])
    d4, d_positions, d_log_scales, d_quats = primitive_records_reverse(ids, offsets, x6, raw, log_scales, quats, grad_rgb,
                                                                       state["grad_t"])
    csr = group_records(ids, x6, d4, state["n"], masks)
    d_weights = grouped_weight_gradients(csr, freq, att, weights, dtype=getattr(torch, state["precision"]))
    return [d_positions, d_log_scales, d_quats, *d_weights]


def run(state):
    kind = state["kind"]
    if kind in ("image", "depth", "features", "query"):
        model, cam = state["model"], state["cam"]
        kw = dict(score_threshold=THRESHOLD, view_matrix=cam["view"], proj_matrix=cam["proj"])
        if kind == "image":
            return model(cam["rays_o"], cam["rays_d"], **kw)
        if kind == "depth":
            return model.render_rgb_t_no_grad(cam["rays_o"], cam["rays_d"], **kw)
        if kind == "features":
            return model(cam["rays_o"], cam["rays_d"], return_feature=True, **kw)
        feat = model.render_feature_map(cam["rays_o"], cam["rays_d"], **kw).view(*state["size"], -1)
        return feat, state["decoder"].classify(feat, state["text"])
    if kind == "views":
        return state["batch"].render(state["scene"], state["rays_o"], state["rays_d"], THRESHOLD, state["view"], state["proj"])
    if kind == "stream":
        for f in state["frames"]:
            state["pipe"].submit(f["rays_o"], f["rays_d"], THRESHOLD, f["view"], f["proj"], out_rgb_host=f["rgb"],
                                 out_alpha_host=f["alpha"])
        state["pipe"].drain()
        return [(f["rgb"], f["alpha"]) for f in state["frames"]]
    if kind == "gradients":
        return _backward(state, state["records"], state["grad_rgb"])
    from mlp_splatting_b200.cumodel import render_tiles_training_records
    records = render_tiles_training_records(state["tensors"], *state["size"], 8, THRESHOLD, 1.5, 2.0, precision=state["precision"])
    rgb, alpha = records[:2]
    return [rgb, alpha, *_backward(state, records, _loss_gradient(rgb, state["target"]))]


def work(case):
    """Rays, geometry, weights (at the precision the evaluator takes), attributes and records once each, and the outputs;
    the multiply-adds of the MLPs for the records that pixels composite."""
    kind, n, h, P = case["kind"], case["n"], case["hidden"], case["W"] * case["H"]
    macs = 72 * h + h * h + 4 * h
    params = macs + 2 * h + 4
    wide = 4 if case["precision"] == "fp32" else 2
    frames = case.get("views", case.get("frames", 1))
    records = RECORDS_PER_PIXEL * P * frames
    scene = n * (40 + params * wide)
    if kind in ("gradients", "step"):
        # in: ids, x6, raw, masks, offsets, image adjoints, geometry, FP32 weights; out: geometry and weight gradients.
        # Recomputed forward, adjoints of the activations, outer products: three products per weight (the encoding needs none)
        bytes_, flops = P * 24 + n * (28 + 4 * params) + n * (40 + 4 * params), records * 2 * (3 * macs - 72 * h)
        if kind == "gradients":
            return dict(bytes=bytes_ + records * (4 + 24 + 32 + 8), flops=flops)
        return dict(bytes=bytes_ + P * (24 + 16), flops=flops + records * 2 * macs)
    image = {"image": 12, "depth": 20, "features": 12, "query": 8}.get(kind, 16)
    bytes_ = frames * P * (24 + image) + scene
    flops = records * 2 * macs
    if "channels" in case:
        c = case["channels"]
        bytes_ += n * 4 * c * 2 + P * c * 4
        flops += records * 2 * 4 * c
    if kind == "query":
        c = case["channels"]
        bytes_ += 2 * (c * 128 + 9 * 128 * 128 + 128 * case["classes"])
        flops += P * 2 * (c * 128 + 9 * 128 * 128 + 128 * case["classes"])
    return dict(bytes=float(bytes_), flops=float(flops))


def tolerance(case):
    """FP32: order of 32-bit sums, and pixels whose transmittance ends within rounding of the 1e-3 stop.  fp16 / bf16: operands
    and activations rounded to 11 / 8 bits with 32-bit sums, so a last-bit difference of an activation moves an output by
    that much.  Labels may differ where two classes score alike."""
    if case["precision"] == "fp32":
        return {"rel": 2e-5, "max": 1e-2}
    if case["precision"] == "bf16":
        return {"rel": 1e-2, "max": 0.3}
    if case["kind"] == "query":
        return {"rel": 2e-3, "max": 0.05, "differ": 5e-3}
    return {"rel": 2e-3, "max": 0.1 if case["kind"] in ("gradients", "step") else 0.05}
