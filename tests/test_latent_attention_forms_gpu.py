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
