"""Portions of prompts through a latent on tcgen05 (csrc/latent_attention_tcgen05.cu) against 64 bits: sizes at the edges of its tiles and
blocks, pages of every kind it takes, windows, heads that do not fill a block, cache rows that hold NaN where no key stands.  The kernel rounds
what the mma.sync one rounds (the weights and the result, to bfloat16: 2^-8 of values below 4 in a row of weights that add up to one)."""
import pytest
import torch
from test_logozen_parts_gpu import DEV, _meta, _ops, _plain_rows_attention, g

pytestmark = pytest.mark.gpu


def _tiles(lens, tq):
    D = sum(1 for n in lens if n == 1)
    tiles = [(b, q0) for b in range(D, len(lens)) for q0 in range(0, lens[b], tq)]
    return torch.tensor(tiles or [(0, 0)], dtype=torch.int32, device=DEV), len(tiles)


def _run(lens, contexts, rows, page, table, qa, qr, sink, gate, scale, window, on):
    ops, meta = _ops(), _meta(lens, contexts)
    meta.tile_lists[128] = _tiles(lens, 128)
    meta.error_flag = torch.zeros(4, dtype=torch.int32, device=DEV)
    T, H, C = qa.shape
    out = torch.full((H, T, C), float("nan"), dtype=torch.bfloat16, device=DEV)
    pool, q, table = rows.to(DEV), qa.transpose(0, 1).contiguous().to(DEV), table.to(DEV)
    qr, sink, gate = qr.to(DEV), sink.to(DEV), gate.to(DEV) if gate is not None else None
    assert ops.latent_tcgen05_heads_per_block(q, qr, pool, page, meta, out, scale) > 0
    before, ops.use_latent_tcgen05 = ops.use_latent_tcgen05, on
    try:
        ops.latent_attention(q, qr, pool, page, table, meta, sink, gate, out, scale, window=window)
    finally:
        ops.use_latent_tcgen05 = before
    assert not meta.error_flag.any()
    return out.cpu().transpose(0, 1).double()


@pytest.mark.parametrize("H, C, R, page", [(16, 256, 64, 16), (16, 128, 32, 16), (1, 64, 0, 8), (2, 64, 8, 32), (3, 128, 128, 64), (9, 192, 40, 16),
                                           (5, 256, 24, 128), (40, 64, 64, 16)])
@pytest.mark.parametrize("lens, contexts, window", [([2, 64, 131], [2, 64, 131], None), ([1, 33, 70], [9, 97, 700], None), ([63, 130], [640, 130], 100)])
def test_portions_of_prompts(H, C, R, page, lens, contexts, window):
    gen = g(H + C + R)
    most = -(-max(contexts) // page)
    perm = torch.randperm(most * len(lens) + 3, generator=gen)[:most * len(lens)].view(len(lens), most).int()
    pool = torch.full((int(perm.numel() + 3) * page, C + R), float("nan"), dtype=torch.bfloat16)
    rows = [(torch.randn(n, C + R, generator=gen) * 0.5).bfloat16() for n in contexts]
    for b, n in enumerate(contexts):
        for j in range(n):
            pool[int(perm[b, j // page]) * page + j % page] = rows[b][j]
    T = sum(lens)
    qa, qr = (torch.randn(T, H, C, generator=gen) * 0.4).bfloat16(), (torch.randn(T, H, R, generator=gen) * 0.4).bfloat16()
    qa[T // 2] *= 12.0                                        # rows of a few large weights, whose maximum rises by much between tiles
    sink, gate = torch.randn(H, generator=gen) + 1.0, torch.rand(T, H, generator=gen)
    got = _run(lens, contexts, pool, page, perm, qa, qr, sink, gate, 0.3, window, True)
    old = _run(lens, contexts, pool, page, perm, qa, qr, sink, gate, 0.3, window, False)
    t, err, err_old = 0, 0.0, 0.0
    for b, n in enumerate(lens):
        for i in range(n):
            p = contexts[b] - n + i
            lo = max(0, p - window + 1) if window else 0
            ref = _plain_rows_attention(qa[t], qr[t], rows[b][lo:], C, 0.3, sink, p - lo) * gate[t].double()[:, None]
            assert torch.allclose(got[t], ref, atol=2e-2, rtol=2e-2), f"request {b}, place {p}"
            err, err_old, t = err + float((got[t] - ref).square().sum()), err_old + float((old[t] - ref).square().sum()), t + 1
    assert err <= 1.1 * err_old                               # the same roundings: no further from 64 bits


def test_infinite_scores_and_rows_beside_them():
    """One key has an infinite score for one head, all others -inf: that head shows inf - inf, the others know nothing of it."""
    H, C, R, L, lens = 4, 64, 8, 700, [3]
    gen = g(5)
    rows = (torch.randn(704, C + R, generator=gen) * 0.5).bfloat16()
    qa, qr = (torch.randn(3, H, C, generator=gen) * 0.3).bfloat16(), (torch.randn(3, H, R, generator=gen) * 0.3).bfloat16()
    sink, table = torch.randn(H, generator=gen) + 2.0, torch.arange(44, dtype=torch.int32)[None]
    rows[:, 0] = -1.0
    qa[:, 1, 0] = float("inf")
    for key in (5, 699):
        r = rows.clone()
        r[key, 0] = 1.0
        got = _run(lens, [L], r, 16, table, qa, qr, sink, None, 0.2, None, True)
        for t in range(3):
            ref = _plain_rows_attention(qa[t], qr[t], r, C, 0.2, sink, L - 3 + t)
            assert got[t].isnan().equal(ref.isnan()) and bool(ref[1].isnan().all()) == (key <= L - 3 + t)
            assert torch.allclose(got[t, [0, 2, 3]], ref[[0, 2, 3]], atol=2e-2, rtol=2e-2)
