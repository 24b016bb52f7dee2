"""Kernels with a form that takes four neighbouring values at a time, against 64 bits, and beside their general form, which the same
call runs when one of its vectors does not start on 16 bytes (sizes that the form does not take run the general one twice).  Sums are
float32; in any of these orders a sum of W terms is off by a few units in the last place: 32 * 2^-24 relative to the row's scale is
several times that.  bfloat16 results: half a unit of their last place on top."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 32 * 2.0 ** -24


@pytest.fixture(scope="module")
def ops():
    from mini_engine_b200 import ops
    ops.require_extension()
    return ops


def off(t):
    """The same values one element further on: not on 16 bytes."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:].copy_(t.reshape(-1))
    return flat[1:].view(t.shape)


def near(a, b, scale=None):
    """``scale``: of the terms, where results can be small beside them."""
    half = 2.0 ** -8 if a.dtype == torch.bfloat16 else 0.0
    a, b = a.double(), b.double()
    assert not a.isnan().any() and ((a - b).abs() <= TOL * (b.abs().max() if scale is None else scale) + half * b.abs()).all()


class Meta:
    def __init__(self, lengths, contexts):
        cu = [0]
        for n in lengths:
            cu.append(cu[-1] + n)
        self.cu_seqlens = torch.tensor(cu, dtype=torch.int32, device=DEV)
        self.context_lens = torch.tensor(contexts, dtype=torch.int32, device=DEV)
        self.num_reqs = len(lengths)
        self.token_req = torch.repeat_interleave(torch.arange(len(lengths), dtype=torch.int32, device=DEV),
                                                 torch.tensor(lengths, device=DEV)).int()


# a run each up to 1,024 values, two beyond (up to 4,096); threads that hold nothing; beyond the form's reach
@pytest.mark.parametrize("W", [4, 132, 1024, 1028, 2048, 4096, 4100])
@pytest.mark.parametrize("S", [1, 2, 4, 5])
@pytest.mark.parametrize("taps", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("rows", [False, True])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_hc_norm(ops, W, S, taps, rows, dt):
    if rows and taps:
        pytest.skip("the convolution goes with all rows")
    g = torch.Generator(DEV).manual_seed(W + 10 * S + taps)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    T = 5
    x, y, mix, outw, inw, nw = rnd(S, T, W), rnd(T, W), rnd(S, S), rnd(S), rnd(S), rnd(W)
    cw, state = (rnd(W, taps), rnd(9, taps - 1, W)) if taps else (None, None)
    slots = torch.tensor([3, 0, -1, 8, 5], dtype=torch.int32, device=DEV)
    lens = torch.tensor([1, 2, 7, 3, 40], dtype=torch.int32, device=DEV)      # a first token, too few inputs before it, a request without a slot
    picked = torch.tensor([4, 1], dtype=torch.int32, device=DEV) if rows else None
    new = torch.einsum("sr,stw->rtw", mix.double(), x.double()) + outw.double()[:, None, None] * y.double()
    u = torch.einsum("s,stw->tw", inw.double(), new)
    d = u - u.mean(-1, keepdim=True)
    norm = d / torch.sqrt(d.square().mean(-1, keepdim=True) + 1e-5) * nw.double()
    ref, ref_state = norm[[4, 1]] if rows else norm.clone(), state
    if taps:
        ref *= 1 + cw.double()[:, -1]
        ref_state = state.double().clone()
        for t, (slot, length) in enumerate(zip(slots.tolist(), lens.tolist())):
            if slot < 0:
                continue
            before = state[slot].double() * (length - 1 - torch.arange(taps - 1, 0, -1, device=DEV) >= 0)[:, None]
            ref[t] += (before * cw.double()[:, :-1].T).sum(0)
            ref_state[slot] = torch.cat((before[1:], norm[t][None]))
    res = []
    for weight in (nw, off(nw)):
        xs, st = x.clone(), state.clone() if taps else None
        out = torch.full((2 if rows else T, W), float("nan"), device=DEV, dtype=dt)
        ops.hc_norm(xs, update=(y, mix, outw), mix_in=inw, norm_weight=weight, eps=1e-5, out=out, rows=picked,
                    conv=(cw, st, slots, lens) if taps else None)
        res.append((out, xs, st))
        # (the streams' sums can cancel, and what is left stands beside the row's deviation: rounded to the scale of their terms)
        scale = inw.abs().sum() * new.abs().max() / torch.sqrt(d.square().mean(-1).min() + 1e-5) * nw.abs().max()
        near(out, ref, scale * (1 + (cw.abs().sum(1).max() if taps else 0)))
        near(xs, x if rows else new, (S + 1) * new.abs().max())
        if taps:
            near(st, ref_state, scale)
    if dt == torch.float32:
        near(res[0][0], res[1][0])
    near(res[0][1], res[1][1])
    if taps:
        near(res[0][2], res[1][2])


@pytest.mark.parametrize("W", [4, 128, 516, 2048])
@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("add_input", [True, False])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_short_conv(ops, W, taps, add_input, dt):
    # requests that begin and end inside a run of eight tokens, that go on from their state, without a slot, of one token
    g = torch.Generator(DEV).manual_seed(W + taps)
    lengths, contexts = [1, 3, 9, 2, 16, 1], [1, 3, 30, 3, 16, 2]
    m, T = Meta(lengths, contexts), sum(lengths)
    h, w, state = (torch.randn(*s, device=DEV, generator=g) for s in ((T, W), (W, taps), (8, max(taps - 1, 1), W)))
    slots = torch.tensor([2, 7, 0, 5, -1, 4], dtype=torch.int32, device=DEV)
    ref, t0 = [], 0
    for n, c, slot in zip(lengths, contexts, slots.tolist()):
        seen = torch.zeros(taps - 1 + n, W, device=DEV)                  # the inputs before the portion (zero before the first token), then its own
        seen[taps - 1:] = h[t0:t0 + n]
        if slot >= 0 and taps > 1:
            there = min(taps - 1, c - n)
            seen[taps - 1 - there:taps - 1] = state[slot, taps - 1 - there:]
        part = sum(w.double()[:, j] * seen[j:j + n].double() for j in range(taps))
        ref.append(part + h[t0:t0 + n].double() if add_input else part)
        t0 += n
    ref = torch.cat(ref)
    res = []
    for x in (h, off(h)):
        st, out = state.clone(), torch.full((T, W), float("nan"), device=DEV, dtype=dt)
        ops.short_conv(x, w, st if taps > 1 else None, m.token_req, m, slots, out, add_input=add_input)
        res.append((out, st))
        near(out, ref, 3 * ref.abs().max())
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("F", [4, 2048, 2052, 8192, 8196, 16384, 16388])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("to", [torch.float32, torch.bfloat16])
def test_polynorm(ops, F, dt, to):
    g = torch.Generator(DEV).manual_seed(F)
    z = torch.randn(3, F, device=DEV, generator=g)
    coef = torch.tensor([0.7, -0.4, 0.9, 0.1], device=DEV)
    p, (a, b, c, e) = z.to(dt).double(), coef.double()
    unit = lambda t: t / torch.sqrt(t.square().mean(-1, keepdim=True) + 1e-5)
    ref = a * unit(p) + b * unit(p ** 2) + c * unit(p ** 3) + e
    outs = [torch.full((3, F), float("nan"), device=DEV, dtype=to) for _ in range(2)]
    for x, out in zip((z.to(dt), off(z.to(dt))), outs):
        ops.polynorm(x, coef, 1e-5, out)
        near(out, ref)
    if to == torch.float32:
        near(*outs)


# (one value at a time: no vector has to start anywhere)
@pytest.mark.parametrize("H, V", [(1, 4), (5, 128), (8, 132), (8, 256), (3, 512), (2, 516)])
@pytest.mark.parametrize("gate", [None, "sigmoid", "silu"])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_mlstm_out(ops, H, V, gate, shared, dt):
    g = torch.Generator(DEV).manual_seed(H * V)
    T = 3
    o, proj, w = (torch.randn(*s, device=DEV, generator=g) for s in ((T, H * V), (T, H * V + 8), (V if shared else H * V,)))
    x, z = o.double().view(T, H, V), proj[:, 4:4 + H * V].double()
    ref = (x / torch.sqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w.double().view(1 if shared else H, V)).view(T, H * V)
    ref = ref * (1.0 if gate is None else torch.sigmoid(z) * (z if gate == "silu" else 1.0))
    for weight in (w, off(w)):
        out = torch.full((T, H * V), float("nan"), device=DEV, dtype=dt)
        ops.mlstm_out(o, proj, 4, weight, 1e-5, out, H, V, shared_weight=shared, gate=gate)
        near(out, ref)


# The statistics of a row come from sums of pairs, so that the form's results lie no further from 64 bits than the general form's (thousands of
# values: the distances themselves vary by some 0.3%).
@pytest.mark.parametrize("W", [1024, 2048, 4096, 8192, 12288, 16384])
def test_forms_are_as_close_to_64_bits(ops, W):
    g = torch.Generator(DEV).manual_seed(W)
    T, far = 2000, {}
    x, w = torch.randn(1, T, W, device=DEV, generator=g) * 3 + 1, torch.rand(W, device=DEV, generator=g) + 0.5
    coef = torch.tensor([0.7, -0.4, 0.9, 0.1], device=DEV)
    d = x[0].double() - x[0].double().mean(-1, keepdim=True)
    p, unit = x[0].double(), lambda t: t / torch.sqrt(t.square().mean(-1, keepdim=True) + 1e-5)
    a, b, c, e = coef.double()
    refs = {"hc_norm": d / torch.sqrt(d.square().mean(-1, keepdim=True) + 1e-5) * w.double(), "polynorm": a * unit(p) + b * unit(p ** 2) + c * unit(p ** 3) + e}
    for form in ("vectors", "general"):
        out = torch.empty(T, W, device=DEV)
        if W <= 4096:
            ops.hc_norm(x, norm_weight=w if form == "vectors" else off(w), eps=1e-5, out=out)
            far["hc_norm", form] = (out.double() - refs["hc_norm"]).norm()
        ops.polynorm(x[0] if form == "vectors" else off(x[0]), coef, 1e-5, out)
        far["polynorm", form] = (out.double() - refs["polynorm"]).norm()
    for name in refs:
        if (name, "general") in far:
            assert far[name, "vectors"] <= 1.003 * far[name, "general"]


# The sum of a head's squares has one order in all forms: every 32nd value a lane, then a butterfly over the lanes.  Worked out here with numpy
# (fused multiply-adds through 64 bits), the results are the same to the bit.  Heads of one value to beyond the form in registers.
@pytest.mark.parametrize("H, V", [(1, 4), (2, 33), (5, 128), (8, 132), (8, 256), (3, 510), (3, 512), (2, 516)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_mlstm_out_sums_in_one_order(ops, H, V, dt):
    f32 = np.float32
    rng = np.random.default_rng(H * V)
    T = 3
    o, w = rng.standard_normal((T, H * V), dtype=f32), rng.standard_normal(H * V, dtype=f32)
    x = np.zeros((T, H, -(-V // 32) * 32), dtype=f32)
    x[..., :V] = o.reshape(T, H, V)
    s = np.zeros((T, H, 32), dtype=f32)
    for c in range(x.shape[2] // 32):
        v = x[..., 32 * c:32 * c + 32].astype(np.float64)
        s = (v * v + s).astype(f32)
    for step in (16, 8, 4, 2, 1):
        s = s + s[..., np.arange(32) ^ step]
    r = f32(1) / np.sqrt(s[..., :1] / f32(V) + f32(1e-5))
    ref = torch.from_numpy((x[..., :V] * r * w.reshape(H, V)).reshape(T, H * V)).to(dt)
    out = torch.full((T, H * V), float("nan"), device=DEV, dtype=dt)
    o = torch.from_numpy(o).to(DEV)
    ops.mlstm_out(o, o, 0, torch.from_numpy(w).to(DEV), 1e-5, out, H, V, gate=None)
    assert torch.equal(out.cpu(), ref)


def _rotated(x, pos, freq):
    """Neighbouring pairs of the first values of ``x`` [T, (heads,) R] turned by position times frequency, in 64 bits."""
    a = (pos.double()[:, None] * freq).view(len(pos), *[1] * (x.dim() - 2), -1)
    y, n = x.clone(), 2 * len(freq)
    y[..., 0:n:2] = x[..., 0:n:2] * a.cos() - x[..., 1:n:2] * a.sin()
    y[..., 1:n:2] = x[..., 1:n:2] * a.cos() + x[..., 0:n:2] * a.sin()
    return y


@pytest.mark.parametrize("H, D, R, C, rot", [(1, 4, 4, 4, 4), (16, 64, 64, 256, 64), (5, 32, 16, 132, 8), (9, 128, 64, 512, 0), (2, 8, 12, 16, 6)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_latent_prep(ops, H, D, R, C, rot, dt):
    g = torch.Generator(DEV).manual_seed(H + D)
    T = 6
    offsets = {"q": 0, "c": H * (D + R), "g": H * (D + R) + C + R}
    proj = torch.randn(T, (offsets["g"] + H + 3) // 4 * 4, device=DEV, generator=g)
    cw = torch.randn(C, device=DEV, generator=g)
    freq = 10000.0 ** (-torch.arange(rot // 2, dtype=torch.float64, device=DEV) * 2 / max(rot, 1))
    pos = torch.tensor([0, 1, 7, 100, 5000, 12], dtype=torch.int32, device=DEV)
    slots = torch.tensor([0, 5, -1, 15, 16, 31], dtype=torch.int32, device=DEV)
    q, c = proj[:, :H * (D + R)].double().view(T, H, D + R), proj[:, offsets["c"]:offsets["c"] + C].double()
    key = proj[:, offsets["c"] + C:offsets["g"]].double()
    c = c / torch.sqrt(c.square().mean(-1, keepdim=True) + 1e-5) * cw.double()
    rows = torch.cat((c, _rotated(key, pos, freq)), 1)
    ref = (q[..., :D], _rotated(q[..., D:], pos, freq), torch.sigmoid(proj[:, offsets["g"]:offsets["g"] + H].double()))
    res = []
    for weight in (cw, off(cw)):
        pool = torch.zeros(2, 1, 1, 16, C + R, dtype=dt, device=DEV)
        outs = [torch.full(s, float("nan"), dtype=dt, device=DEV) for s in ((T, H, D), (T, H, R))] + [torch.full((T, H), float("nan"), device=DEV)]
        ops.latent_prep(proj, offsets, weight, 1e-5, freq, rot, pos, slots, pool, *outs, H, D, R, C)
        res.append([pool] + outs)
        for got, want in zip(outs, ref):
            near(got, want)
        for t, slot in enumerate(slots.tolist()):
            if slot >= 0:
                near(pool.view(-1, C + R)[slot], rows[t])
    # (bfloat16 results of sums that differ in their last place may round to the neighbour)
    for a, b in zip(*res):
        if dt == torch.float32 or a.dtype == torch.float32:
            near(a, b)
        else:
            assert not a.isnan().any() and ((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + TOL).all()
