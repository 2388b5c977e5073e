"""The backward half's own kernels at the sizes where their splits can go wrong: the grouping sort at the edges of its
blocks, warps and digit passes, and the weight gradients at the edges of their record blocks and segments."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("n", [1, 2, 255, 256, 65_535, 65_536, 200_000])
@pytest.mark.parametrize("R", [0, 1, 31, 33, 4095, 4096, 4097, 70_001])
def test_group_records_is_a_stable_sort_of_the_rows(n, R):
    from mlp_splatting_b200.primitive_csr import group_order, group_records
    g = torch.Generator(device=DEV)
    g.manual_seed(1000 * n + R)
    ids = torch.randint(0, n, (R,), generator=g, device=DEV, dtype=torch.int32)
    x6 = torch.randn((R, 6), generator=g, device=DEV)
    d4 = torch.randn((R, 4), generator=g, device=DEV)
    masks = torch.randint(-2**31, 2**31 - 1, (R, 2), generator=g, device=DEV, dtype=torch.int32)
    order = torch.argsort(ids, stable=True)
    offsets = torch.zeros(n + 1, device=DEV, dtype=torch.int64)
    offsets[1:] = torch.bincount(ids, minlength=n).cumsum(0)
    csr = group_records(ids, x6, d4, n, masks)
    for got, want in ((csr.offsets, offsets), (csr.record_indices, order), (csr.x6, x6[order]), (csr.grad4, d4[order]),
                      (csr.relu_masks, masks[order])):
        assert got.dtype == want.dtype and torch.equal(got, want)
    plain = group_records(ids, x6.double(), d4, n)          # rows of another type take torch's indexing
    assert plain.relu_masks is None and torch.equal(plain.x6, x6.double()[order])
    assert all(torch.equal(a, b) for a, b in zip(group_order(ids, n), (offsets, order)))


@pytest.mark.parametrize("dtype,bound", [(torch.float32, 2e-6), (torch.float16, 1e-2), (torch.bfloat16, 4e-2)])
@pytest.mark.parametrize("with_masks", [True, False])
@pytest.mark.parametrize("segment", [64, 512])
def test_weight_gradients_at_block_and_segment_edges(dtype, bound, with_masks, segment):
    """Against the same sums in float64; counts around 16-row steps, 64- and 128-record blocks and the segments."""
    from mlp_splatting_b200.primitive_csr import PrimitiveCSR
    from mlp_splatting_b200.primitive_gemm import grouped_weight_gradients
    counts = [0, 1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 0, 500, 512, 513, 1030]
    n, R = len(counts), sum(counts)
    g = torch.Generator(device=DEV)
    g.manual_seed(5)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    w = [rnd(n, 32, 72) * 0.2, rnd(n, 32) * 0.1, rnd(n, 32, 32) * 0.2, rnd(n, 32) * 0.1, rnd(n, 4, 32) * 0.2, rnd(n, 4) * 0.1]
    w = [t.half().float() for t in w]
    x6, d3 = rnd(R, 6), rnd(R, 4) * 1e-3
    freq = torch.tensor(2.0 ** np.arange(6) * np.pi, device=DEV, dtype=torch.float32)
    att = torch.exp(-0.5 * freq ** 2 * 1e-4)
    offsets = torch.tensor(np.concatenate(([0], np.cumsum(counts))), device=DEV)
    W1, b1, W2, b2, W3, _b3 = (t.double() for t in w)
    pid = torch.repeat_interleave(torch.arange(n, device=DEV), torch.tensor(counts, device=DEV))
    ph = ((x6[:, :, None] * freq) * att).double().reshape(R, 36)
    e = torch.cat([ph.sin(), ph.cos()], 1)
    a1 = torch.einsum("rhj,rj->rh", W1[pid], e) + b1[pid]
    m1, h1 = a1 > 0, a1.clamp_min(0)
    a2 = torch.einsum("rqh,rh->rq", W2[pid], h1) + b2[pid]
    m2, h2 = a2 > 0, a2.clamp_min(0)
    dd3 = d3.double()
    d2 = torch.einsum("rc,rch->rh", dd3, W3[pid]) * m2
    d1 = torch.einsum("rq,rqh->rh", d2, W2[pid]) * m1
    want = [torch.zeros_like(t).index_add_(0, pid, v) for t, v in
            ((W1, d1[:, :, None] * e[:, None]), (b1, d1), (W2, d2[:, :, None] * h1[:, None]), (b2, d2),
             (W3, dd3[:, :, None] * h2[:, None]), (torch.zeros(n, 4, device=DEV, dtype=torch.float64), dd3))]
    bits = 2 ** torch.arange(32, device=DEV, dtype=torch.int64)
    words = torch.stack([(m1 * bits).sum(1), (m2 * bits).sum(1)], 1)
    masks = torch.where(words >= 2**31, words - 2**32, words).to(torch.int32).contiguous() if with_masks else None
    csr = PrimitiveCSR(offsets, torch.arange(R, device=DEV), x6, d3, masks)
    got = grouped_weight_gradients(csr, freq, att, w, dtype=dtype, segment_size=segment)
    for a, b in zip(got, want):
        assert a.shape == b.shape and torch.isfinite(a).all()
        # without saved masks a rounded activation near zero may take the other sign
        assert float((a.double() - b).norm() / b.norm()) < (bound if with_masks or dtype == torch.float32 else 3 * bound)
        assert (a[0] == 0).all() and (a[11] == 0).all()


def test_records_reverse_refuses_bad_offsets_and_ids():
    from mlp_splatting_b200.primitive_csr import primitive_records_reverse
    R, P, n = 300, 50, 7
    ids = torch.randint(0, n, (R,), device=DEV, dtype=torch.int32)
    offsets = torch.linspace(0, R, P + 1, device=DEV).round().to(torch.int64)
    args = [torch.rand(R, 6, device=DEV), torch.rand(R, 8, device=DEV), torch.zeros(n, 3, device=DEV),
            torch.nn.functional.normalize(torch.randn(n, 4, device=DEV)), torch.rand(P, 3, device=DEV), torch.rand(P, device=DEV)]
    primitive_records_reverse(ids, offsets, *args)
    bad = ids.clone()
    bad[-1] = n
    with pytest.raises(ValueError, match="ids out of range"):
        primitive_records_reverse(bad, offsets, *args)
    for change in ((0, 1), (P, R - 1), (20, int(offsets[22]))):
        off = offsets.clone()
        off[change[0]] = change[1]
        with pytest.raises(ValueError, match="pixel offsets"):
            primitive_records_reverse(ids, off, *args)
    primitive_records_reverse(ids, offsets, *args)          # the next call starts clean


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_weight_gradients_refuse_offsets_that_leave_the_records(dtype):
    """Offsets past the rows, below zero or descending are found before an item or a record is touched; rows behind the last
    offset are nobody's."""
    from mlp_splatting_b200.primitive_csr import PrimitiveCSR
    from mlp_splatting_b200.primitive_gemm import grouped_weight_gradients
    counts = [40, 0, 1, 700, 129, 0, 330]
    n, R, spare = len(counts), sum(counts), 77
    g = torch.Generator(device=DEV)
    g.manual_seed(17)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    w = [rnd(n, 32, 72) * 0.2, rnd(n, 32), rnd(n, 32, 32) * 0.2, rnd(n, 32), rnd(n, 4, 32), rnd(n, 4)]
    freq = torch.tensor(2.0 ** np.arange(6), device=DEV, dtype=torch.float32)
    att = torch.exp(-0.5 * freq ** 2 * 1e-4)
    x6, d3 = rnd(R + spare, 6), rnd(R + spare, 4) * 1e-3
    offsets = torch.tensor(np.concatenate(([0], np.cumsum(counts))), device=DEV)
    run = lambda off, rows: grouped_weight_gradients(PrimitiveCSR(off, None, x6[:rows], d3[:rows]), freq, att, w, dtype=dtype,
                                                     segment_size=64)
    want = run(offsets, R)
    assert all(torch.equal(a, b) for a, b in zip(run(offsets, R + spare), want))
    changed = lambda i, v: torch.cat([offsets[:i], offsets.new_tensor([v]), offsets[i + 1:]])
    for off, rows in ((offsets, R - 1), (offsets, 1), (offsets, 0), (changed(n, R + 10**6), R), (changed(0, -5), R),
                      (changed(4, 10), R), (changed(3, R), R), (changed(3, 2**40), R)):
        with pytest.raises(ValueError, match="CSR offsets"):
            run(off, rows)
    assert all(torch.equal(a, b) for a, b in zip(run(offsets, R), want))          # the next call starts clean


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shifted", [("W1",), ("W2",), ("W1", "b1", "W2", "b2", "W3", "b3")])
def test_weight_gradients_of_weights_at_any_alignment(dtype, shifted):
    """Masters whose first element lies four bytes beyond a 16-byte boundary (a slice of one flat parameter, say): the same
    values through four-byte loads, hence the same bits."""
    from mlp_splatting_b200.primitive_csr import PrimitiveCSR
    from mlp_splatting_b200.primitive_gemm import grouped_weight_gradients
    counts = [0, 1, 63, 200, 128, 700]
    n, R = len(counts), sum(counts)
    g = torch.Generator(device=DEV)
    g.manual_seed(8)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    w = dict(W1=rnd(n, 32, 72) * 0.2, b1=rnd(n, 32) * 0.1, W2=rnd(n, 32, 32) * 0.2, b2=rnd(n, 32) * 0.1, W3=rnd(n, 4, 32) * 0.2,
             b3=rnd(n, 4) * 0.1)
    moved = {}
    for k, t in w.items():
        flat = torch.empty(t.numel() + 1, device=DEV)
        moved[k] = flat[1:].view(t.shape).copy_(t) if k in shifted else t
        assert moved[k].data_ptr() % 16 == (4 if k in shifted else 0) and moved[k].is_contiguous()
    freq = torch.tensor(2.0 ** np.arange(6) * np.pi, device=DEV, dtype=torch.float32)
    att = torch.exp(-0.5 * freq ** 2 * 1e-4)
    offsets = torch.tensor(np.concatenate(([0], np.cumsum(counts))), device=DEV)
    csr = PrimitiveCSR(offsets, torch.arange(R, device=DEV), rnd(R, 6), rnd(R, 4) * 1e-3, None)
    want = grouped_weight_gradients(csr, freq, att, list(w.values()), dtype=dtype)
    got = grouped_weight_gradients(csr, freq, att, list(moved.values()), dtype=dtype)
    for a, b in zip(got, want):
        assert torch.equal(a, b) and float(b.abs().max()) > 0
