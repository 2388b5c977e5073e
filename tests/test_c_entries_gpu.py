"""The C entry points that the Python layer does not call itself, on torch memory through the ctypes binding."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _at(numel, floats):
    """A float32 array that starts `floats` elements past a 256-byte boundary."""
    return torch.full((numel + 64,), float("nan"), device=DEV)[floats:floats + numel]


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_records_reverse_takes_gradients_of_any_alignment(shift):
    """Against torch autograd's adjoints (tests/golden/backward.npz), with the bound of the test of the Python call."""
    from mlp_splatting_b200 import _lib as L
    fx = np.load(os.path.join(HERE, "golden", "backward.npz"))
    ids, offsets, x6, raw, logs, quats, grgb, gt = (
        torch.from_numpy(np.ascontiguousarray(fx["rev_" + k])).to(DEV)
        for k in ("ids", "offsets", "x6", "raw", "logs", "quats", "grgb", "gt"))
    R, P, n = ids.numel(), grgb.shape[0], logs.shape[0]
    d4 = torch.full((R, 4), float("nan"), device=DEV)
    gp, gs, gq = _at(3 * n, shift), _at(3 * n, shift), _at(4 * n, shift)
    lib = L.load()
    L.check(lib.mlpsp_records_reverse(*(L.ptr(t) for t in (ids, offsets, x6, raw, logs, quats, grgb, gt)), P, R, n,
                                      *(L.ptr(t) for t in (d4, gp, gs, gq)), _stream()), "mlpsp_records_reverse")
    for got, key in ((d4, "rev_d4"), (gp, "rev_gp"), (gs, "rev_gs"), (gq, "rev_gq")):
        want = torch.from_numpy(fx[key]).to(DEV)
        torch.testing.assert_close(got.view(want.shape), want, atol=2e-5 * float(want.abs().max()) + 1e-7, rtol=2e-4)
    # no pixels: zero gradients, and nothing else is read
    L.check(lib.mlpsp_records_reverse(None, L.ptr(offsets), *[None] * 6, 0, 0, n, None, *(L.ptr(t) for t in (gp, gs, gq)),
                                      _stream()), "mlpsp_records_reverse")
    assert all((t == 0).all() for t in (gp, gs, gq))
    # pixels, but no arrays to read or write
    assert lib.mlpsp_records_reverse(None, L.ptr(offsets), *[None] * 6, P, 0, n, None, *(L.ptr(t) for t in (gp, gs, gq)),
                                     _stream()) == -1


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("with_masks", [True, False])
def test_grouped_weight_gradients_over_a_prepared_layout(dtype, with_masks):
    """The same bits as the call that plans its own segments; the caller's partial rows hold the sums of the primitives of
    several segments and nothing else; a layout that does not belong to the offsets gives the flag and no access."""
    from mlp_splatting_b200 import _lib as L
    from mlp_splatting_b200.primitive_csr import PrimitiveCSR
    from mlp_splatting_b200.primitive_gemm import grouped_weight_gradients, prepare_groups
    counts = [0, 1, 64, 65, 0, 129, 700, 3, 0] + [2] * 600         # several blocks of the planning kernel
    n, R, seg = len(counts), sum(counts), 64
    g = torch.Generator(device=DEV)
    g.manual_seed(23)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    w = [rnd(n, 32, 72) * 0.2, rnd(n, 32) * 0.1, rnd(n, 32, 32) * 0.2, rnd(n, 32) * 0.1, rnd(n, 4, 32) * 0.2, rnd(n, 4) * 0.1]
    x6, d3 = rnd(R, 6), rnd(R, 4) * 1e-3
    masks = torch.randint(-2**31, 2**31 - 1, (R, 2), generator=g, device=DEV, dtype=torch.int32) if with_masks else None
    freq = torch.tensor(2.0 ** np.arange(6), device=DEV, dtype=torch.float32)
    att = torch.exp(-0.5 * freq ** 2 * 1e-4)
    csr = PrimitiveCSR(torch.tensor(np.concatenate(([0], np.cumsum(counts))), device=DEV), None, x6, d3, masks)
    layout = prepare_groups(csr, seg)
    scale = 4096.0 if dtype == torch.float16 else 1.0
    want = grouped_weight_gradients(csr, freq, att, w, dtype=dtype, segment_size=seg, loss_scale=scale, groups=layout)
    want = torch.cat([t.flatten(1) for t in want], 1)
    lib = L.load()
    row = int(lib.mlpsp_grouped_gradient_floats())
    sc = L.Scene()
    sc.n, sc.hidden, sc.num_freq = n, 32, 6
    sc.W1, sc.b1, sc.W2, sc.b2, sc.W3, sc.b3 = (L.ptr(t) for t in w)
    sc.freq, sc.att = L.ptr(freq), L.ptr(att)
    precision = {torch.float32: L.PRECISION_F32, torch.float16: L.PRECISION_F16, torch.bfloat16: L.PRECISION_BF16}[dtype]

    def run(prims, starts, offs, G):
        partial = torch.full((max(G, 1), row), float("nan"), device=DEV)
        result = torch.full((n, row), float("nan"), device=DEV)
        flag = torch.full((1,), -1, device=DEV, dtype=torch.int32)
        L.check(lib.mlpsp_grouped_weight_gradients(
            C.byref(sc), *(L.ptr(t) for t in (csr.offsets, x6, d3, masks, prims, starts, offs)), G, seg, precision, scale,
            L.ptr(partial), L.ptr(result), L.ptr(flag), _stream()), "mlpsp_grouped_weight_gradients")
        return partial, result, int(flag)

    prims, starts, offs = layout.primitives, layout.starts, layout.offsets
    G = prims.numel()
    partial, result, flag = run(prims, starts, offs, G)
    assert flag == 0 and torch.equal(result, want)
    several = ((offs[1:] - offs[:-1]) > 1)[prims]
    assert 0 < int(several.sum()) < G
    assert torch.isfinite(partial[several]).all() and partial[~several].isnan().all()
    _partial, result, flag = run(prims, starts, offs, 0)
    assert flag == 0 and (result == 0).all()

    def changed(t, i, v):
        t = t.clone()
        t[i] = v
        return t

    last = int(csr.offsets[-1])
    for bad in ((changed(prims, 3, n), starts, offs), (changed(prims, 3, -1), starts, offs), (changed(prims, 0, 2), starts, offs),
                (prims, changed(starts, 1, last), offs), (prims, changed(starts, 1, -1), offs),
                (prims, starts, changed(offs, n, G + 1)), (prims, starts, changed(offs, 5, -1)), (prims, starts, changed(offs, 6, G))):
        assert run(*bad, G)[2] & 4


@pytest.mark.parametrize("n,R", [(1, 0), (1, 5), (7, 4097), (300, 10_000), (70_000, 50_001)])
def test_group_records_against_a_stable_sort(n, R):
    from mlp_splatting_b200 import _lib as L
    g = torch.Generator(device=DEV)
    g.manual_seed(n + R)
    ids = torch.randint(0, n, (R,), generator=g, device=DEV, dtype=torch.int32)
    offsets = torch.full((n + 1,), -1, device=DEV, dtype=torch.int64)
    order = torch.full((R,), -1, device=DEV, dtype=torch.int64)
    lib = L.load()
    nbytes = int(lib.mlpsp_group_records_scratch_bytes(R, n))
    scratch = torch.empty(nbytes, device=DEV, dtype=torch.uint8)
    call = lambda size: lib.mlpsp_group_records(L.ptr(ids), R, n, L.ptr(offsets), L.ptr(order), L.ptr(scratch), size, _stream())
    assert call(nbytes - 1) == -2            # the scratch is checked
    L.check(call(nbytes), "mlpsp_group_records")
    want = torch.zeros(n + 1, device=DEV, dtype=torch.int64)
    want[1:] = torch.bincount(ids, minlength=n).cumsum(0)
    assert torch.equal(offsets, want) and torch.equal(order, torch.argsort(ids, stable=True))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("W,H", [(128, 96), (61, 43)])
def test_render_frame_gives_the_image_of_the_fused_call(precision, W, H):
    """Unit rays, host matrices and a status block that the caller resets, against the call that does these itself."""
    from mlp_splatting_b200 import _lib as L
    from mlp_splatting_b200.engine import FrameRenderer, PackedScene, normalize_rows
    from tests.helpers import WKEYS, small_case
    scene, cam = small_case(n=2000, W=W, H=H)
    ps = PackedScene(scene["positions"], scene["log_scales"], scene["quats"], *[scene[k] for k in WKEYS], scene["freq"],
                     scene["att"], device=DEV)
    r = FrameRenderer(W, H, device=DEV)
    ro, rd = torch.from_numpy(cam["rays_o"]).to(DEV), torch.from_numpy(cam["rays_d"]).to(DEV)
    args = dict(view=cam["view"], proj=cam["proj"], precision=precision, waves=[32, 32, 64, 128, 256, 1536])
    want = [t.clone() for t in r.render(ps, ro, rd, 5e-3, **args)]
    words = r.status_host.clone()
    assert float(want[1].max()) > 0.5
    unit = normalize_rows(rd)
    f = r._frame(ps, ro, unit, 5e-3, precision, cam["view"], cam["proj"], None, False, False, args["waves"])
    r.rgb.fill_(float("nan"))
    r.alpha.fill_(float("nan"))
    lib = L.load()
    L.check(lib.mlpsp_status_reset(L.ptr(r.status), _stream()), "mlpsp_status_reset")
    L.check(lib.mlpsp_render_frame(C.byref(ps.c), C.byref(f), _stream()), "mlpsp_render_frame")
    assert torch.equal(r.rgb, want[0]) and torch.equal(r.alpha, want[1])
    assert torch.equal(r.status.cpu(), words)


def test_export_records_in_one_call_gives_the_rows_of_the_counted_export():
    from mlp_splatting_b200 import _lib as L
    from mlp_splatting_b200.engine import FrameRenderer, PackedScene
    from tests.helpers import WKEYS, small_case
    scene, cam = small_case(n=1500, W=61, H=43)
    ps = PackedScene(scene["positions"], scene["log_scales"], scene["quats"], *[scene[k] for k in WKEYS], scene["freq"],
                     scene["att"], device=DEV)
    r = FrameRenderer(61, 43, device=DEV)
    ro, rd = torch.from_numpy(cam["rays_o"]).to(DEV), torch.from_numpy(cam["rays_d"]).to(DEV)
    want = r.render_records(ps, ro, rd, 5e-3, view=cam["view"], proj=cam["proj"])[2:]
    R = want[0].numel()
    assert R > 1000
    got = [torch.full_like(t, -7) for t in want]
    f, _ = r._last_frame
    total, worst = C.c_int64(-1), C.c_int32(-1)
    lib = L.load()
    call = lambda room: L.check(lib.mlpsp_export_records(
        C.byref(ps.c), C.byref(f), L.ptr(got[5]), *(L.ptr(t) for t in got[:5]), room, 512, C.byref(total), C.byref(worst),
        _stream()), "mlpsp_export_records")
    call(R - 1)                                   # no room: the count and the offsets only
    assert total.value == R and torch.equal(got[5], want[5]) and all((t == -7).all() for t in got[:5])
    call(R)
    assert total.value == R and worst.value == int((want[5][1:] - want[5][:-1]).max())
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    # a total beyond the frame's records: no row behind the last one is made
    more = [torch.full((R + 1000, *t.shape[1:]), -7, device=DEV, dtype=t.dtype) for t in want[:5]]
    L.check(lib.mlpsp_export_counted_records(C.byref(ps.c), C.byref(f), *(L.ptr(t) for t in more), R + 1000, _stream()),
            "mlpsp_export_counted_records")
    assert all(torch.equal(a[:R], b) and (a[R:] == -7).all() for a, b in zip(more, want))
