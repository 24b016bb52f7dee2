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
    # the same roundings: level with the other kernel (0.970 to 1.006 of its sum of squares over these cases; larger batches, 12 seeds: 0.98 to 1.00)
    assert err <= 1.02 * err_old


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


@pytest.mark.parametrize("apart", [True, False])
@pytest.mark.parametrize("C, R, page", [(64, 8, 16), (128, 32, 16), (256, 64, 64)])
def test_warps_that_rescale_at_every_tile_beside_warps_that_never_do(C, R, page, apart):
    """Long contexts, two blocks an SM where the sizes allow it.  With 16 heads a warp holds two tokens of a block's eight: those of one warp
    score higher from tile to tile and the others lower (``apart``), or the other way round, so warps drift apart as far as the barriers let
    them; the last block has one token, and three warps without any.  Repeated launches agree bit for bit.  Weights, their sum and the result
    are rounded to bfloat16, 2^-9 each: below 2^-7 of the terms' magnitudes."""
    H, scale, lens, contexts = 16, 0.25, [1160, 1201], [3000, 4001]
    gen, ops = g(C + R), _ops()
    pages = [-(-n // page) for n in contexts]
    perm = torch.randperm(sum(pages), generator=gen).int()
    table = torch.zeros(2, max(pages), dtype=torch.int32)
    pool = torch.full((sum(pages) * page, C + R), float("nan"), dtype=torch.bfloat16)
    rows = []
    for b, n in enumerate(contexts):
        table[b, :pages[b]] = perm[sum(pages[:b]):sum(pages[:b + 1])]
        rows.append((torch.randn(n, C + R, generator=gen) * 0.5).bfloat16())
        rows[b][:, 0] = (torch.arange(n) // 64).float() / 8         # (exact in bfloat16)
        places = (table[b, :pages[b], None].long() * page + torch.arange(page)).flatten()[:n]
        pool[places] = rows[b]
    T = sum(lens)
    qa, qr = (torch.randn(T, H, C, generator=gen) * 0.02).bfloat16(), (torch.randn(T, H, R, generator=gen) * 0.02).bfloat16()
    local = torch.cat([torch.arange(n) for n in lens])
    qa[:, :, 0] = torch.where(((local // 2) % 4 == 2) == apart, 10.0, -10.0)[:, None].bfloat16()     # 0.3 a tile, against noise of 0.05
    sink = torch.randn(H, generator=gen).to(DEV)
    meta = _meta(lens, contexts)
    meta.error_flag = torch.zeros(4, dtype=torch.int32, device=DEV)
    q, qr, pool, table = qa.transpose(0, 1).contiguous().to(DEV), qr.to(DEV), pool.to(DEV), table.to(DEV)
    first, out = None, torch.empty(H, T, C, dtype=torch.bfloat16, device=DEV)
    assert ops.latent_tcgen05_heads_per_block(q, qr, pool, page, meta, out, scale) == 16
    for _ in range(20):
        out.fill_(float("nan"))
        ops.latent_attention(q, qr, pool, page, table, meta, sink, None, out, scale)
        first = out.clone() if first is None else first
        assert torch.equal(out, first) and not meta.error_flag.any()
    t0 = 0
    for b, n in enumerate(contexts):
        keys = rows[b].to(DEV).double()
        seen = torch.arange(n, device=DEV)[None] <= torch.arange(n - lens[b], n, device=DEV)[:, None]
        for h in range(H):
            s = torch.cat([q[h, t0:t0 + lens[b]], qr[t0:t0 + lens[b], h]], 1).double() @ keys.t() * scale
            s = torch.where(seen, s, -torch.inf)
            m = torch.maximum(s.amax(1, keepdim=True), sink[h].double())
            p = torch.exp(s - m)
            p = p / (p.sum(1, keepdim=True) + torch.exp(sink[h].double() - m))
            err = (first[h, t0:t0 + lens[b]].double() - p @ keys[:, :C]).abs()
            assert bool((err <= 2.0 ** -7 * (p @ keys[:, :C].abs()) + 1e-6).all()), f"request {b}, head {h}"
        t0 += lens[b]


@pytest.mark.parametrize("C, R, lens, contexts, taken", [(256, 64, [40, 64], [40, 64], False), (256, 64, [40, 3], [40, 65], True), (256, 64, [64] * 17, [64] * 17, False),
                                                         (128, 32, [64] * 16, [64] * 16, False), (128, 32, [64] * 16 + [2], [64] * 16 + [2], True)])
def test_steps_of_one_key_tile(C, R, lens, contexts, taken):
    """Steps whose longest context is one key tile keep the mma.sync kernel, of small latents up to 1,024 tokens; the neighbouring sizes do not."""
    H, gen, ops, T = 4, g(C), _ops(), sum(lens)
    meta = _meta(lens, contexts)
    meta.error_flag = torch.zeros(4, dtype=torch.int32, device=DEV)
    pages = -(-max(contexts) // 16)
    table = torch.arange(pages * len(lens), dtype=torch.int32, device=DEV).view(len(lens), pages)
    pool = (torch.randn(pages * 16 * len(lens), C + R, generator=gen) * 0.5).bfloat16().to(DEV)
    q, qr = (torch.randn(H, T, C, generator=gen) * 0.4).bfloat16().to(DEV), (torch.randn(T, H, R, generator=gen) * 0.4).bfloat16().to(DEV)
    sink, out = torch.randn(H, generator=gen).to(DEV), torch.full((H, T, C), float("nan"), dtype=torch.bfloat16, device=DEV)
    meta.tile_lists[32] = _tiles(lens, 32)
    assert (ops.latent_tcgen05_heads_per_block(q, qr, pool, 16, meta, out, 0.3) > 0) == taken
    ops.latent_attention(q, qr, pool, 16, table, meta, sink, None, out, 0.3)
    assert not meta.error_flag.any()
    t = 0
    for b, n in enumerate(lens):
        for i in range(n):
            p = contexts[b] - n + i
            ref = _plain_rows_attention(q[:, t].cpu(), qr[t].cpu(), pool[table[b, 0] * 16:][:p + 1].cpu(), C, 0.3, sink.cpu(), p)
            assert torch.allclose(out[:, t].cpu().double(), ref, atol=2e-2, rtol=2e-2), f"request {b}, place {p}"
            t += 1
