"""The frame path's kernels at the sizes where their splits and dispatch rules can go wrong: hit masks per window length and
ray arrangement, record placement at the edges of its blocks, sorts of long lists, the FP32 evaluator's row groups, the
reverse pass over record chunks and windows, device-resident cameras."""
import numpy as np
import pytest
import torch

from tests.helpers import WKEYS, oracle_frame, popcount64, small_case

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
THR = 5e-3


@pytest.fixture(autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _t(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV)


def _packed(scene, **kw):
    from mlp_splatting_b200.engine import PackedScene
    return PackedScene(scene["positions"], scene["log_scales"], scene["quats"], *[scene[k] for k in WKEYS], scene["freq"],
                       scene["att"], device=DEV, **kw)


def _rays(kind, cam, scene):
    """Ray arrangements: the camera's, from among the primitives, from inside one of them, one origin per image half, and a
    field of view far beyond the one the lists were made for."""
    ro, rd = cam["rays_o"].copy(), cam["rays_d"].copy()
    if kind == "near":
        ro[:] = ro * 0.2
    elif kind == "inside":
        ro[:] = scene["positions"][0] + np.float32(0.01)
    elif kind == "two origins":
        ro[: len(ro) // 2] += np.float32(0.3)
    elif kind == "wide":
        rd = rd + 6.0 * (rd - rd.mean(0))
    return _t(ro), _t(rd.astype(np.float32))


@pytest.mark.parametrize("kind", ["camera", "near", "inside", "two origins", "wide"])
@pytest.mark.parametrize("n,mu", [(40, -3.0), (120, -3.0), (400, -3.2), (3000, -3.3)])
@pytest.mark.parametrize("thr", [5e-3, 0.3])
def test_one_wave_evaluates_exactly_the_hits(kind, n, mu, thr):
    """A single wave over the whole lists, whose capacity picks the hit kernel of that window length: the records are the
    pairs that the exact test counts, the image does not depend on the kernel."""
    from mlp_splatting_b200.engine import FrameRenderer, normalize_rows
    scene, cam = small_case(n=n, W=61, H=43, mu=mu, seed=n)
    ps = _packed(scene, pack_f16=False)
    r = FrameRenderer(61, 43, device=DEV)
    ro, rd = _rays(kind, cam, scene)
    rd = normalize_rows(rd)
    prims, offs = (t.clone() for t in r.bin(ps, cam["view"], cam["proj"], thr))
    M, longest = int(prims.numel()), int((offs[1:] - offs[:-1]).max())
    r.sort(ps, ro, rd, M)
    hits = int(popcount64(r.hit_masks(ps, ro, rd, thr, M).cpu().numpy().view(np.uint64)).sum())
    images = []
    for cap in [c for c in (32, 64, 128, 1536) if c >= longest]:
        q = FrameRenderer(61, 43, device=DEV, tile_capacity=cap)
        rgb, _ = q.render(ps, ro, rd, thr, precision=0, tile_lists=(prims, offs), rays_normalized=True, waves=[cap])
        assert q.last_stats.records == hits
        images.append(rgb.clone())
    assert images and all(torch.equal(images[0], i) for i in images)
    if kind == "camera":
        assert hits > 0


@pytest.mark.parametrize("n", [1, 2, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("W,H", [(17, 8), (40, 24), (208, 200)])
@pytest.mark.parametrize("precision,tol", [(0, 2e-5), (1, 2e-3)])
def test_frames_at_placement_and_fill_edges(n, W, H, precision, tol):
    """Primitive counts around the placement blocks, from three tiles (short windows per warp) to 650 (long ones)."""
    from mlp_splatting_b200.engine import FrameRenderer
    scene, cam = small_case(n=n, W=W, H=H, mu=-3.6 if n > 2 else -1.5, seed=7 + n)
    f = oracle_frame(scene, cam, THR, precision=0, want_masks=False, capacity=2048)
    ps, r = _packed(scene), FrameRenderer(W, H, device=DEV, tile_capacity=2048)
    rgb, _ = r.render(ps, _t(cam["rays_o"]), _t(cam["rays_d"]), THR, view=cam["view"], proj=cam["proj"], precision=precision)
    np.testing.assert_allclose(rgb.cpu().numpy(), f["render"].rgb, atol=tol)


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("hidden,n,W,H", [(32, 2000, 483, 365), (32, 21_428, 500, 300), (64, 3000, 803, 501), (64, 20_000, 800, 500)])
def test_frames_with_a_direction_table_equal_a_batch_without(precision, hidden, n, W, H):
    """Frames on the table's side of its rule, on the line and with ragged tiles; a batch of views never takes the table."""
    from mlp_splatting_b200 import synthetic
    from mlp_splatting_b200.engine import FrameRenderer, PackedScene, ViewBatchRenderer
    scene = synthetic.make_scene_device(n, 7, torch.device(DEV), mu=-3.5, hidden=hidden)
    ps = PackedScene(scene["positions"], scene["log_scales"], scene["quats"], *[scene[k] for k in WKEYS], scene["freq"],
                     scene["att"], device=DEV, pack_bf16=True)
    cam = synthetic.make_camera(W, H)
    ro, rd = _t(cam["rays_o"]), _t(cam["rays_d"])
    got = FrameRenderer(W, H, device=DEV).render(ps, ro, rd, THR, view=cam["view"], proj=cam["proj"], precision=precision)
    want = ViewBatchRenderer(W, H, 1, device=DEV).render(ps, [ro], [rd], THR, [cam["view"]], [cam["proj"]], precision=precision)[0]
    assert float(want[1].max()) > 0.5
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("n", [257, 512, 513, 1024, 1025, 1500])
@pytest.mark.parametrize("W,H", [(5, 3), (23, 17)])
def test_long_lists_sort_exactly(n, W, H):
    from mlp_splatting_b200.engine import FrameRenderer
    from oracle import oracle as orc
    scene, cam = small_case(n=n, W=W, H=H, mu=-2.0, seed=n)
    ps, r = _packed(scene, pack_f16=False), FrameRenderer(W, H, device=DEV, tile_capacity=2048)
    prims, offs = (t.clone() for t in r.bin(ps, cam["view"], cam["proj"], THR))
    rd = orc.normalize_rows(cam["rays_d"])
    got = r.sort(ps, _t(cam["rays_o"]), _t(rd), int(prims.numel()))
    want = orc.sort_tiles(cam["rays_o"], rd, ps.geom.cpu().numpy()[:n], offs.cpu().numpy(), prims.cpu().numpy(), W, H, 8)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    if W == 5:
        assert int((offs[1:] - offs[:-1]).max()) > 256


@pytest.mark.parametrize("n", [2000, 8191, 8192])
def test_rectangle_corners_count_the_tiles(n):
    """Below and above the rule that sums the corners in shared memory first (8,192 primitives)."""
    from mlp_splatting_b200.engine import FrameRenderer
    scene, cam = small_case(n=n, W=128, H=96, mu=-4.5, seed=n)
    f = oracle_frame(scene, cam, THR, want_masks=False)
    prims, offs = FrameRenderer(128, 96, device=DEV).bin(_packed(scene, pack_f16=False), cam["view"], cam["proj"], THR)
    np.testing.assert_array_equal(offs.cpu().numpy(), f["tile_offsets"])
    np.testing.assert_array_equal(prims.cpu().numpy(), f["tile_prims"])


@pytest.mark.parametrize("hidden", [32, 64])
def test_fp32_evaluator_at_row_group_edges(hidden):
    from mlp_splatting_b200.primitive_gemm import grouped_forward
    from oracle import oracle as orc
    counts = [0, 1, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 0, 300]
    scene, _ = small_case(n=len(counts), seed=5, hidden=hidden)
    ids = np.repeat(np.arange(len(counts), dtype=np.int32), counts)
    x6 = np.random.default_rng(1).normal(0, 0.4, (len(ids), 6)).astype(np.float32)
    offsets = np.concatenate(([0], np.cumsum(counts))).astype(np.int64)
    out = grouped_forward(_t(offsets), _t(x6), _packed(scene, pack_f16=False), dtype=torch.float32)
    want = orc.mlp_eval([scene[k] for k in WKEYS], scene["freq"], scene["att"], ids, x6, precision=0)
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=0, atol=1e-5)


def test_camera_matrices_and_raw_rays_on_the_device():
    """Matrices and rays that are on the device already take the path without host copies: the same bits."""
    from mlp_splatting_b200.engine import FrameRenderer, normalize_rows
    scene, cam = small_case(W=61, H=43)
    ps, ro, rd = _packed(scene), _t(cam["rays_o"]), _t(cam["rays_d"])
    out = []
    for view, proj, rays, unit in ((cam["view"], cam["proj"], normalize_rows(rd), True), (_t(cam["view"]), _t(cam["proj"]), rd, False)):
        r = FrameRenderer(61, 43, device=DEV)
        for _ in range(2):
            rgb, alpha = r.render(ps, ro, rays, THR, view=view, proj=proj, precision=1, rays_normalized=unit)
        out.append((rgb.clone(), alpha.clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1]) and out[0][1].max() > 0.1


def _reverse_reference(ids, offsets, x6, raw, ls, quats, grgb, gt):
    """float64: the recurrence per pixel, then the geometry gradients by autograd of sum (k / decay) decay."""
    raw, grgb, gt = raw.double().cpu().numpy(), grgb.double().cpu().numpy(), gt.double().cpu().numpy().reshape(-1)
    d4, k = np.zeros((len(raw), 4)), np.zeros(len(raw))
    for p in range(len(offsets) - 1):
        behind = gt[p]
        for r in range(int(offsets[p + 1]) - 1, int(offsets[p]) - 1, -1):
            c, sig, tr, al, dec, logit = raw[r, :3], raw[r, 3], raw[r, 4], raw[r, 5], raw[r, 6], raw[r, 7]
            colour = float(grgb[p] @ c)
            g_alpha = tr * (colour - behind)
            behind = behind * (1 - al) + colour * al
            g = g_alpha * np.exp(-sig * dec)
            d4[r, :3] = grgb[p] * tr * al * c * (1 - c)
            d4[r, 3] = g * dec / (1 + np.exp(-logit))
            k[r] = g * dec * sig
    pid = torch.as_tensor(ids).long().cpu()
    d0 = x6[:, 3:].double().cpu()
    shift = torch.zeros(len(ls), 3, dtype=torch.float64, requires_grad=True)
    ls64, q64 = ls.double().cpu().requires_grad_(), quats.double().cpu().requires_grad_()
    w, u = q64[pid, :1], -q64[pid, 1:]
    d = d0 + shift[pid]
    t = 2 * torch.linalg.cross(u, d)
    q = d + w * t + torch.linalg.cross(u, t)
    e = -0.5 * (q * q * torch.exp(-2 * ls64[pid])).sum(1)
    (torch.from_numpy(k) * e).sum().backward()
    return d4, shift.grad, ls64.grad, q64.grad


@pytest.mark.parametrize("n", [1, 40, 1500, 100_000])
@pytest.mark.parametrize("per_pixel", [[0], [1, 0, 2], [3, 30], [40, 7, 0, 90]])
@pytest.mark.parametrize("pixels", [1, 127, 129, 300])
def test_records_reverse_at_chunk_and_window_edges(n, per_pixel, pixels):
    """From no records to several windows of a pixel block and chunks whose primitives overflow the table."""
    from mlp_splatting_b200.primitive_csr import primitive_records_reverse
    counts = np.resize(np.array(per_pixel), pixels)
    offsets = np.concatenate(([0], np.cumsum(counts))).astype(np.int64)
    R = int(offsets[-1])
    g = torch.Generator(device=DEV)
    g.manual_seed(R + n)
    rnd = lambda *s: torch.rand(s, generator=g, device=DEV)
    ids = torch.randint(0, n, (R,), generator=g, device=DEV, dtype=torch.int32)
    x6 = torch.randn((R, 6), generator=g, device=DEV) * 0.3
    raw = rnd(R, 8) * 0.8 + 0.1
    ls, quats = rnd(n, 3) * 0.5 - 0.5, torch.nn.functional.normalize(torch.randn((n, 4), generator=g, device=DEV), dim=1)
    grgb, gt = rnd(pixels, 3) - 0.5, rnd(pixels) - 0.5
    got = primitive_records_reverse(ids, _t(offsets), x6, raw, ls, quats, grgb, gt)
    want = _reverse_reference(ids, offsets, x6, raw, ls, quats, grgb, gt)
    for a, b in zip(got, want):
        b = torch.as_tensor(b)
        assert tuple(a.shape) == tuple(b.shape)
        scale = max(float(b.abs().max()) if b.numel() else 0.0, 1e-3)
        assert float((a.double().cpu() - b).abs().max() if b.numel() else 0.0) < 3e-5 * scale


@pytest.mark.parametrize("case,slots,C", [("ragged", 1, 512), ("ragged", 5, 512), ("ragged", 4, 384), ("tiny", 4, 128)])
def test_feature_channels_per_cta(case, slots, C):
    """Every channel split and stage length of the tensor-core compositing, lists around whole stages included."""
    from mlp_splatting_b200.engine import FrameRenderer
    scene, cam = small_case(**(dict(n=1500, W=61, H=43, mu=-3.2, seed=31, az=140.0) if case == "ragged" else dict(n=700, W=40, H=24)))
    fa = np.random.default_rng(C).normal(0, 0.2, (len(scene["positions"]), slots, C)).astype(np.float16).astype(np.float32)
    scene = dict(scene, feat_attr=fa if slots > 1 else fa[:, 0, :])
    f = oracle_frame(scene, cam, THR, precision=0, feat=True, want_masks=False)
    ps, r = _packed(scene, pack_f16=False, feat_attr=scene["feat_attr"]), FrameRenderer(cam["W"], cam["H"], device=DEV)
    assert ps.feat16 is not None
    r.render(ps, _t(cam["rays_o"]), _t(cam["rays_d"]), THR, view=cam["view"], proj=cam["proj"], precision=0, want_feat=True)
    np.testing.assert_allclose(r.feat.cpu().numpy(), f["render"].feat, rtol=0, atol=2e-5)


@pytest.mark.parametrize("per_tile", [1, 31, 33, 700])
def test_exported_rows_compose_the_image(per_tile):
    """Record export from one candidate to long runs per pixel, against the composited image and itself."""
    from mlp_splatting_b200.engine import FrameRenderer
    scene, cam = small_case(n=per_tile, W=16, H=11, mu=-1.8 if per_tile < 100 else -2.3, seed=per_tile)
    scene["b3"] = scene["b3"].copy()
    scene["b3"][:, 3] = -5.0                 # nearly transparent primitives: long runs of records per pixel
    ps, r = _packed(scene, pack_f16=False), FrameRenderer(16, 11, device=DEV)
    rgb, alpha, ids, x6, raw, masks, gates, offsets = r.render_records(
        ps, _t(cam["rays_o"]), _t(cam["rays_d"]), THR, view=cam["view"], proj=cam["proj"], precision=0, max_hits=4096)
    f = oracle_frame(scene, cam, THR, precision=0, want_masks=False, want_records=True)
    np.testing.assert_allclose(rgb.cpu().numpy(), f["render"].rgb, atol=2e-5)
    pid = torch.repeat_interleave(torch.arange(16 * 11, device=DEV), offsets[1:] - offsets[:-1])
    assert int(offsets[-1]) == len(ids) == len(raw) and bool(((ids >= 0) & (ids < per_tile)).all())
    image = torch.zeros(16 * 11, 3, device=DEV).index_add_(0, pid, raw[:, 4:5] * raw[:, 5:6] * raw[:, :3])
    torch.testing.assert_close(image, rgb, rtol=0, atol=2e-5)
    # transmittance before a record: the product over the pixel's records before it
    log_t = torch.log1p(-raw[:, 5].double())
    before = torch.cumsum(log_t, 0) - log_t
    before = torch.exp(before - torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), torch.cumsum(log_t, 0)])[offsets[:-1]][pid])
    torch.testing.assert_close(before.float(), raw[:, 4], rtol=1e-4, atol=1e-6)
    if per_tile == 700:
        assert int((offsets[1:] - offsets[:-1]).max()) > 40


def test_record_frame_that_outgrows_its_scratch():
    """The count of a frame's records is launched before its status is known; an overflow renders and counts again."""
    from mlp_splatting_b200.engine import FrameRenderer
    scene, cam = small_case(W=61, H=43)
    ps, got = _packed(scene, pack_f16=False), []
    for most in (16_000_000, 1000):
        r = FrameRenderer(61, 43, device=DEV, max_records=most)
        got.append(r.render_records(ps, _t(cam["rays_o"]), _t(cam["rays_d"]), THR, view=cam["view"], proj=cam["proj"], precision=0))
    assert r.max_records > 1000 and len(got[0][2]) > 1000
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_training_records_with_weights_beyond_binary16():
    """The frame is launched before the status of the weight packing is known; weights that do not fit give the FP32 records."""
    from mlp_splatting_b200.cumodel import render_tiles_training_records
    from mlp_splatting_b200.engine import FrameRenderer, normalize_rows
    scene, cam = small_case(W=61, H=43)
    scene["W2"] = scene["W2"].copy()
    scene["W2"][3, 5, 7] = 1.0e6
    ps = _packed(scene, pack_f16=False)
    culled, offs = FrameRenderer(61, 43, device=DEV).bin(ps, cam["view"], cam["proj"], THR)
    tensors = [_t(cam["rays_o"]), normalize_rows(_t(cam["rays_d"])), ps.positions, ps.log_scales, ps.quats_unit, culled, offs,
               ps.freq, ps.att] + [_t(scene[k]) for k in WKEYS]
    half, full = (render_tiles_training_records(tensors, 61, 43, 8, THR, 1.5, 2.0, precision=p) for p in ("float16", "float32"))
    assert len(half[2]) > 1000
    for a, b in zip(half, full):
        assert torch.equal(a, b)


@pytest.mark.parametrize("out_dim,classes,hidden,cin,W,H", [(300, 160, 64, 24, 170, 150), (768, 700, 128, 128, 161, 137), (128, 1, 96, 7, 8, 5000)])
def test_decoder_queues_layer_one_behind_the_last_output_chunk(out_dim, classes, hidden, cin, W, H):
    """Several tiles per CTA with one to six output chunks: the ring of weight blocks wraps at every offset."""
    from mlp_splatting_b200 import synthetic as syn
    from mlp_splatting_b200.feature_decoder import FeatureUpsampleDecoder
    from oracle import oracle as orc
    w, text = syn.make_decoder(cin, hidden, out_dim, classes, seed=W)
    dec = FeatureUpsampleDecoder(cin, out_dim, hidden, device=torch.device(DEV))
    dec.load_state_dict({k: torch.from_numpy(v) for k, v in w.items()})
    x = syn.make_feature_map(W, H, cin, seed=H)
    want = orc.decode_features(x, w, precision=1)
    assert np.abs(dec.decode_hwc(_t(x)).cpu().numpy() - want).max() <= 2e-3
    labels, margin = orc.classify_features(want, text)
    assert not (dec.classify(_t(x), _t(text)).cpu().numpy() != labels)[margin > 2e-3].any()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("views,n,mu,W,H", [(1, 300, -3.0, 17, 9), (2, 8192, -5.0, 129, 95), (8, 40, -2.5, 40, 24), (9, 9000, -5.0, 113, 90),
                                            (17, 500, -3.2, 33, 17)])
def test_batches_at_the_edges_of_a_launch(precision, views, n, mu, W, H):
    """One view, a full launch of eight and one beyond it, raw and normalised rays, against the frames rendered alone (the same
    arithmetic per record, hence equal bits); windows of which the last ones find no live tiles."""
    from mlp_splatting_b200 import synthetic
    from mlp_splatting_b200.engine import FrameRenderer, ViewBatchRenderer, normalize_rows
    scene = synthetic.make_scene(n, 5, mu=mu)
    ps, single = _packed(scene), FrameRenderer(W, H, device=DEV, tile_capacity=2048)
    cams = [synthetic.make_camera(W, H, azimuth_deg=31.0 * v) for v in range(views)]
    ros, rds = [_t(c["rays_o"]) for c in cams], [_t(c["rays_d"]) for c in cams]
    vs, prs = [c["view"] for c in cams], [c["proj"] for c in cams]
    want, pairs, records = [], 0, 0
    for v in range(views):
        rgb, alpha = single.render(ps, ros[v], rds[v], THR, view=vs[v], proj=prs[v], precision=precision, waves=[16, 64, 512, 1024])
        want.append((rgb.clone(), alpha.clone()))
        pairs, records = single.last_stats.pairs, records + single.last_stats.records
    batch = ViewBatchRenderer(W, H, views, device=DEV, tile_capacity=2048)
    for normalized in (False, True):
        got = batch.render(ps, ros, [normalize_rows(d) for d in rds] if normalized else rds, THR, vs, prs, precision=precision,
                           waves=[16, 64, 512, 1024], rays_normalized=normalized)
        for (rgb, alpha), (rgb_w, alpha_w) in zip(got, want):
            assert torch.equal(rgb, rgb_w) and torch.equal(alpha, alpha_w)
        assert batch.last_stats.records == records and batch.last_stats.pairs == pairs      # the pairs are the last view's
    assert records > 0


@pytest.mark.parametrize("n", [257, 512, 513, 1025, 2000])
@pytest.mark.parametrize("depths", ["equal", "outlier", "pairs", "spread"])
def test_long_lists_of_any_depths_sort_exactly(n, depths):
    """Lists whose keys fall into one bucket (all equal, or one far candidate that stretches the range), into few, into all:
    the order is the stable one, and the frame that lists its own long tiles draws what one with given lists draws."""
    from mlp_splatting_b200.engine import FrameRenderer
    from oracle import oracle as orc
    W, H = 23, 17
    scene, cam = small_case(n=n, W=W, H=H, mu=-1.0, seed=n)
    p = scene["positions"]
    if depths != "spread":
        p[:] = p[:1] if depths != "pairs" else p[np.arange(n) // 2]
        scene["quats"][:], scene["log_scales"][:] = scene["quats"][:1], scene["log_scales"][:1]
    if depths == "outlier":
        p[0] += 40.0 * cam["rays_d"].reshape(H, W, 3)[H // 2, W // 2]
    ps, r = _packed(scene), FrameRenderer(W, H, device=DEV, tile_capacity=2048)
    prims, offs = (t.clone() for t in r.bin(ps, cam["view"], cam["proj"], THR))
    rd = orc.normalize_rows(cam["rays_d"])
    got = r.sort(ps, _t(cam["rays_o"]), _t(rd), int(prims.numel()))
    want = orc.sort_tiles(cam["rays_o"], rd, ps.geom.cpu().numpy()[:n], offs.cpu().numpy(), prims.cpu().numpy(), W, H, 8)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert int((offs[1:] - offs[:-1]).max()) > 256
    kw = dict(view=cam["view"], proj=cam["proj"], precision=1)
    given = [t.clone() for t in r.render(ps, _t(cam["rays_o"]), _t(cam["rays_d"]), THR, tile_lists=(prims, offs), **kw)]
    own = r.render(ps, _t(cam["rays_o"]), _t(cam["rays_d"]), THR, **kw)
    assert torch.equal(own[0], given[0]) and torch.equal(own[1], given[1]) and float(own[1].max()) > 0.0


@pytest.mark.parametrize("precision", [0, 1])
def test_deep_stacks_of_large_splats_get_shorter_windows_and_the_same_image(precision):
    """1,500 splats of 0.14 on 200 x 150 pixels: several times as many hits as a pixel composites before it is opaque."""
    from mlp_splatting_b200.engine import FrameRenderer
    scene, cam = small_case(n=1_500, W=200, H=150, mu=-2.0, seed=7)
    ps, ro, rd = _packed(scene), _t(cam["rays_o"]), _t(cam["rays_d"])
    kw = dict(view=cam["view"], proj=cam["proj"], precision=precision)
    want = [t.clone() for t in FrameRenderer(200, 150, device=DEV).render(ps, ro, rd, THR, waves=[16] * 7 + [1536], **kw)]
    r = FrameRenderer(200, 150, device=DEV)
    evaluated = []
    for _ in range(6):
        rgb, alpha = r.render(ps, ro, rd, THR, **kw)
        assert torch.equal(rgb, want[0]) and torch.equal(alpha, want[1])
        evaluated.append(r.last_stats.records)
    assert evaluated[-1] < 0.8 * evaluated[0] and r.last_stats.used <= evaluated[-1]


@pytest.mark.parametrize("n", [257, 520, 1500])
@pytest.mark.parametrize("kind", ["few behind", "many behind", "all behind", "wall", "thick wall"])
def test_long_lists_of_crowded_keys_sort_exactly(n, kind):
    """Keys that crowd into few buckets.  Behind the camera: equal keys sorted by their tie-breaks, and the largest key there is,
    which fits one bucket, does not, or is all that there is.  Walls: up to 128 in a bucket, and beyond."""
    from mlp_splatting_b200.engine import FrameRenderer
    from oracle import oracle as orc
    W, H = 23, 17
    scene, cam = small_case(n=n, W=W, H=H, mu=-1.0, seed=n)
    rng = np.random.default_rng(n)
    rd = orc.normalize_rows(cam["rays_d"])
    d = rd.reshape(H, W, 3)[H // 2, W // 2]
    p, eye = scene["positions"], cam["rays_o"][0]
    order = rng.permutation(n)
    if "behind" in kind:
        p[:] = p[:1]
        scene["quats"][:], scene["log_scales"][:] = scene["quats"][:1], scene["log_scales"][:1]
        m = {"few": 60, "many": n // 2, "all": n}[kind.split()[0]]
        p[order[:m]] = eye - 2.0 * d
    else:
        step = 2e-3 if kind == "wall" else 2e-5
        depth = 2.0 + step * rng.permutation(n).astype(np.float32) / n
        depth[order[: n // 8]] += 6.0
        p[:] = eye + depth[:, None] * d
        scene["quats"][:] = scene["quats"][:1]
        scene["log_scales"][:] = -1.0
    ps, r = _packed(scene), FrameRenderer(W, H, device=DEV, tile_capacity=2048)
    prims = np.tile(rng.permutation(n).astype(np.int32), r.T)           # every tile lists every primitive
    offs = (np.arange(r.T + 1) * n).astype(np.int32)
    r.tile_prims[: prims.size].copy_(_t(prims))
    r.tile_offsets.copy_(_t(offs))
    got, keys = r.sort(ps, _t(cam["rays_o"]), _t(rd), prims.size, want_keys=True)
    want, want_keys = orc.sort_tiles(cam["rays_o"], rd, ps.geom.cpu().numpy()[:n], offs, prims, W, H, 8, want_keys=True)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    np.testing.assert_array_equal(keys.cpu().numpy(), want_keys)
    behind = int((want_keys[:n] == np.float32(1e30)).sum())
    assert behind == (m if "behind" in kind else 0)


@pytest.mark.parametrize("hidden", [32, 64])
@pytest.mark.parametrize("small_groups", [False, True])
def test_overflow_of_layer_two_alone_falls_back_to_fp32(hidden, small_groups):
    """Weights and first activations within binary16, second ones beyond it: only the evaluator's outputs show it.  Once in
    the evaluator of full blocks, once where every work item is a small group."""
    from mlp_splatting_b200.engine import FrameRenderer
    n, W, H, mu = (6_000, 64, 48, -4.6) if small_groups else (300, 64, 48, -3.0)
    scene, cam = small_case(n=n, W=W, H=H, mu=mu, hidden=hidden)
    ro, rd, kw = _t(cam["rays_o"]), _t(cam["rays_d"]), dict(view=cam["view"], proj=cam["proj"])
    r = FrameRenderer(W, H, device=DEV)
    r.render(_packed(scene), ro, rd, THR, precision=1, **kw)
    work = r.last_stats
    assert r.f32_fallbacks == 0 and work.work_total > 0 and (work.work_small == work.work_total) == small_groups
    scene["b1"][:] = 1.0
    scene["W1"][:] *= 0.1
    scene["W2"][:, 0, :] = 3.0e4
    ps = _packed(scene)
    assert ps.has_f16
    rgb = r.render(ps, ro, rd, THR, precision=1, **kw)[0].clone()
    assert r.f32_fallbacks == 1
    assert torch.isfinite(rgb).all() and torch.equal(rgb, r.render(ps, ro, rd, THR, precision=0, **kw)[0])


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_on_an_image_beyond_the_corner_array(precision):
    """More rows of tiles than one CTA's corner array: the views of a batch are binned and sorted one by one, and the binning
    lists the tiles with long lists."""
    from mlp_splatting_b200 import synthetic
    from mlp_splatting_b200.engine import FrameRenderer, ViewBatchRenderer
    W, H, views = 24, 8 * 1025, 3
    scene = synthetic.make_scene(900, 5, mu=-1.6)
    ps = _packed(scene)
    cams = [synthetic.make_camera(W, H, azimuth_deg=31.0 * v) for v in range(views)]
    ros, rds = [_t(c["rays_o"]) for c in cams], [_t(c["rays_d"]) for c in cams]
    vs, prs = [c["view"] for c in cams], [c["proj"] for c in cams]
    single, want = FrameRenderer(W, H, device=DEV, tile_capacity=2048), []
    for v in range(views):
        rgb, alpha = single.render(ps, ros[v], rds[v], THR, view=vs[v], proj=prs[v], precision=precision, tile_pretest=False)
        want.append((rgb.clone(), alpha.clone()))
        assert 256 < single.last_stats.max_tile_len
    batch = ViewBatchRenderer(W, H, views, device=DEV, tile_capacity=2048)
    for _ in range(2):
        got = batch.render(ps, ros, rds, THR, vs, prs, precision=precision)
        assert batch.last_stats.pairs_kept > 0
        for (rgb, alpha), (rgb_w, alpha_w) in zip(got, want):
            assert torch.equal(rgb, rgb_w) and torch.equal(alpha, alpha_w) and float(alpha.max()) > 0.1
