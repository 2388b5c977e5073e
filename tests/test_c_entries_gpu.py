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
