"""Attention through a latent on the tensor cores (csrc/latent_attention_mma.cu) where its forms can go wrong."""
import pytest
import torch
from test_logozen_parts_gpu import DEV, _meta, _ops, _plain_rows_attention, g

pytestmark = pytest.mark.gpu
PAGE = 16


def _case(H, C, R, lens, contexts):
    """Rows of one request that all requests of the step read, and queries: (rows, q_abs [T, H, C], q_rot [T, H, R], sink, table)."""
    n = -(-max(contexts) // PAGE) * PAGE
    gen = g(C + R + max(contexts))
    rows = (torch.randn(n, C + R, generator=gen) * 0.5).bfloat16()
    T = sum(lens)
    return (rows, (torch.randn(T, H, C, generator=gen) * 0.3).bfloat16(), (torch.randn(T, H, R, generator=gen) * 0.3).bfloat16(),
            torch.randn(H, generator=gen) + 2.0, torch.arange(n // PAGE, dtype=torch.int32)[None].repeat(len(lens), 1))


def _run(lens, contexts, rows, qa, qr, sink, table, scale, window=None):
    T, H, C = qa.shape
    out = torch.empty(H, T, C, dtype=torch.bfloat16, device=DEV)
    _ops().latent_attention(qa.transpose(0, 1).contiguous().to(DEV), qr.to(DEV), rows.to(DEV), PAGE, table.to(DEV), _meta(lens, contexts),
                            sink.to(DEV), None, out, scale, window=window)
    return out.cpu().transpose(0, 1)


# One key of 700 or 8,500 (of the merge's first and second round of ranges) has an infinite score, all others have -inf: as in a softmax
# written out, inf - inf is what the row shows, and the other heads know nothing of it.  Single tokens, and a portion of three.
@pytest.mark.parametrize("L, key", [(700, 5), (700, 699), (8500, 100), (8500, 8400)])
def test_an_infinite_score_stays_visible(L, key):
    H, C, R, lens, contexts = 4, 64, 8, [1, 3], [L, L]
    rows, qa, qr, sink, table = _case(H, C, R, lens, contexts)
    rows[:, 0] = -1.0
    rows[key, 0] = 1.0
    qa[:, 1, 0] = float("inf")
    got = _run(lens, contexts, rows, qa, qr, sink, table, 0.2).double()
    for t, p in enumerate([L - 1, L - 3, L - 2, L - 1]):
        ref = _plain_rows_attention(qa[t], qr[t], rows, C, 0.2, sink, p)
        assert got[t].isnan().equal(ref.isnan()) and bool(ref[1].isnan().all()) == (key <= p)
        assert torch.allclose(got[t, [0, 2, 3]], ref[[0, 2, 3]], atol=2e-2, rtol=2e-2)


# Beyond 8,192 keys a request has more ranges than the merge has threads; with a window its ranges are counted from the window's first tile.
@pytest.mark.parametrize("C, R", [(64, 8), (128, 32), (264, 24)])
@pytest.mark.parametrize("contexts, window", [([8193], None), ([12000], None), ([12000], 9000), ([12000, 3, 8192, 70], None)])
def test_single_tokens_of_long_requests(C, R, contexts, window):
    H, lens, scale = 3, [1] * len(contexts), 0.3
    rows, qa, qr, sink, table = _case(H, C, R, lens, contexts)
    got = _run(lens, contexts, rows, qa, qr, sink, table, scale, window).double()
    for t, n in enumerate(contexts):
        ref = _plain_rows_attention(qa[t], qr[t], rows[max(0, n - window):] if window else rows, C, scale, sink, n - 1 - max(0, n - window) if window else n - 1)
        assert torch.allclose(got[t], ref, atol=2e-2, rtol=2e-2)


# More ranges than the merge keeps weights of, which the engine's plan never asks for: the ranges beyond are worked out again in every thread.
def test_more_ranges_than_the_merge_keeps():
    H, C, R, n, scale = 2, 8, 8, 70000, 0.5
    rows, qa, qr, sink, table = _case(H, C, R, [1], [n])
    ops, meta = _ops(), _meta([1], [n])
    splits = -(-n // 64)
    assert splits > 1024
    partial = torch.full((1, splits, H, C + 2), float("nan"), device=DEV)
    d = [t.to(DEV) for t in (qa.transpose(0, 1).contiguous(), qr, rows, table, sink)]
    out = torch.empty(H, 1, C, dtype=torch.bfloat16, device=DEV)
    ops._call("me_latent_attention_decode", *(t.data_ptr() for t in d[:4]), table.shape[1], meta.cu_seqlens.data_ptr(), meta.context_lens.data_ptr(),
              1, d[4].data_ptr(), 0, out.data_ptr(), partial.data_ptr(), splits, 64, 1, H, C, R, PAGE, scale, 0, ops._stream())
    ref = _plain_rows_attention(qa[0], qr[0], rows, C, scale, sink, n - 1)
    assert torch.allclose(out.cpu()[:, 0].double(), ref, atol=2e-2, rtol=2e-2)


# The heads' products straight into their columns of [T, H * V] rows: 256 terms of float32 or of bfloat16 values, one rounding of the result.
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T, H, C, V", [(1, 5, 40, 12), (1, 16, 256, 128), (7, 3, 40, 33), (300, 16, 256, 128)])
def test_products_of_heads_into_columns(T, H, C, V, dtype):
    lat = torch.randn(H, T, C, generator=g(T)).to(dtype).to(DEV)
    uv = torch.randn(H, V, C, generator=g(V)).to(dtype).to(DEV)
    rows = torch.full((T, H * V), float("nan"), dtype=dtype, device=DEV)
    _ops().batched_heads_mm(lat, uv.transpose(1, 2), rows.view(T, H, V).transpose(0, 1))
    ref = torch.einsum("htc,hvc->thv", lat.double(), uv.double()).reshape(T, H * V)
    size = torch.einsum("htc,hvc->thv", lat.double().abs(), uv.double().abs()).reshape(T, H * V)
    assert ((rows.double() - ref).abs() <= C * 2.0 ** -24 * size + (2.0 ** -8 * ref.abs() if dtype == torch.bfloat16 else 0)).all()
