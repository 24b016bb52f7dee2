"""The mLSTM recurrence's kernels against 64 bits, for several requests of a step with states of their own.  Queries, keys and sums of keys are
positive, so that no denominator cancels: a score's 256 terms and an output's 130 tokens put at most 400 * 2^-24 = 2.4e-5 of its size on a
weight, and exponents, sums of gates of up to a hundred or so, 100 * 2^-24 = 6e-6 each on both sides; a weight's error joins the output
times the largest value, so outputs and states agree to 1e-4 of their largest entry."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
CAP = 15.0


@pytest.fixture(scope="module")
def ops():
    from mini_engine_b200 import ops
    ops.require_extension()
    return ops


def meta_of(lens, contexts):
    D = sum(n == 1 for n in lens)
    tiles = [(b, q0) for b in range(D, len(lens)) for q0 in range(0, lens[b], 64)]
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return SimpleNamespace(cu_seqlens=ints(cu), context_lens=ints(contexts), num_reqs=len(lens), num_decodes=D,
                           tile_lists={64: (ints(tiles or [(0, 0)]), len(tiles))},
                           workspace=lambda name, shape, dtype: torch.full(shape, float("nan"), dtype=dtype, device=DEV))


def make(H, D, V, lens, slots, seed):
    g = torch.Generator(DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    T, width = sum(lens), 2 * H * D + H * V + 2 * H
    proj = rnd(T, width + 1)[:, :width] if D % 4 else rnd(T, (width + 3) // 4 * 4)
    proj[:, :2 * H * D] = proj[:, :2 * H * D].abs()
    offs = {"q": 0, "k": H * D, "v": 2 * H * D, "i": 2 * H * D + H * V, "f": 2 * H * D + H * V + H}
    proj[T // 3:T // 2 + 1, offs["i"]:offs["i"] + H] += 12               # gates near the cap: the running maximum rises and stays
    return proj, offs, rnd(H), rnd(H) + 3, (rnd(slots, H, D, V), rnd(slots, H, D).abs(), rnd(slots, H).abs())


def reference(proj, offs, bi, bf, state, lens, before, slots, H, D, V):
    p = proj.double()
    S, n, m = (t.double().clone() for t in state)
    part = lambda name, w: p[:, offs[name]:offs[name] + H * w].reshape(-1, H, w)
    q, k, v = part("q", D) * D ** -0.5, part("k", D), part("v", V)
    gi = CAP * torch.tanh((part("i", 1)[..., 0] + bi.double()) / CAP)
    gf = torch.nn.functional.logsigmoid(CAP * torch.tanh((part("f", 1)[..., 0] + bf.double()) / CAP))
    o, t = torch.full((p.shape[0], H, V), 7.0, dtype=torch.float64, device=DEV), 0
    for b, length in enumerate(lens):
        s = slots[b]
        if s >= 0 and before[b] == 0:
            S[s], n[s], m[s] = 0, 0, 0
        for t in range(t, t + length):
            if s < 0:
                continue
            new = torch.maximum(gf[t] + m[s], gi[t])
            fa, fb = torch.exp(gf[t] + m[s] - new), torch.exp(gi[t] - new)
            S[s] = fa[:, None, None] * S[s] + fb[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
            n[s], m[s] = fa[:, None] * n[s] + fb[:, None] * k[t], new
            o[t] = torch.einsum("hdv,hd->hv", S[s], q[t]) / (torch.maximum((n[s] * q[t]).sum(-1).abs(), torch.exp(-new)) + 1e-6)[:, None]
        t += 1
    return o.view(-1, H * V), S, n, m


def check(ops, H, D, V, lens, before, slots, chunks=True):
    proj, offs, bi, bf, state = make(H, D, V, lens, max(slots) + 1, seed=D + V)
    ref = reference(proj, offs, bi, bf, state, lens, before, slots, H, D, V)
    S, n, m = state
    o = torch.full((sum(lens), H * V), 7.0, device=DEV)                   # (rows of a request without a slot are left alone)
    meta = meta_of(lens, [a + b for a, b in zip(before, lens)])
    ops.mlstm_chunks = chunks
    try:
        ops.mlstm_scan(proj, offs, bi, bf, CAP, S, n, m, meta, torch.tensor(slots, dtype=torch.int32, device=DEV), o, H, D, V, D ** -0.5)
    finally:
        ops.mlstm_chunks = True
    for got, want in zip((o, S, n, m), ref):
        assert ((got.double() - want).abs() <= 1e-4 * want.abs().max()).all()


# vector forms (one, two and four tiles of 64 columns, heads beyond 64 and 128 keys) and the form for sizes that are no multiples of four;
# runs of every kind: a rest of two tokens, 63, 64, 65, three runs, nine runs (the walk's groups of loads), a request without a slot
@pytest.mark.parametrize("H, D, V", [(8, 128, 256), (2, 256, 68), (1, 4, 4), (3, 72, 132), (2, 13, 70)])
def test_prompts(ops, H, D, V):
    check(ops, H, D, V, [1, 1, 2, 63, 64, 65, 130, 570, 70], [0, 9, 5, 0, 64, 3, 0, 1, 0], [5, 1, 0, 7, 3, 2, 6, 4, -1])


# token by token: more blocks than the device holds at once, so that some start when others have ended; several tokens a request; heads and values
# beyond the prompt kernels' sizes; one request without a slot
@pytest.mark.parametrize("H, D, V, lens", [(8, 128, 256, [1] * 64), (8, 64, 128, [1] * 3), (4, 72, 130, [1] * 9 + [3, 5, 40]), (2, 300, 1000, [1, 2, 9])])
def test_single_tokens(ops, H, D, V, lens):
    slots = [(b * 3) % len(lens) if len(lens) % 3 else b for b in range(len(lens))]
    slots[1] = -1
    check(ops, H, D, V, lens, [0 if b % 5 == 2 else 7 for b in range(len(lens))], slots, chunks=False)


def test_weights_behind_a_strong_decay(ops):
    """Fifty tokens whose forget gates stand at the cap take the sums of the gates to some -750; 14 tokens without decay then weigh about the
    same.  An output is a sum of 14 terms that weigh, of scores of 4 terms, with weights whose exponents lie within 4: at most 14 + 4 + 4 of
    float32's rounding steps, as many for the sum of the weights, and a few for exponentials and the division."""
    H, D, V, T = 4, 4, 64, 64
    g = torch.Generator(DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    offs = {"q": 0, "k": H * D, "v": 2 * H * D, "i": 2 * H * D + H * V, "f": 2 * H * D + H * V + H}
    proj = rnd(T, offs["f"] + H)
    proj[:, :2 * H * D] = proj[:, :2 * H * D].abs()
    proj[:50, offs["f"]:] -= 200
    proj[50:, offs["f"]:] += 200
    bias = torch.zeros(H, device=DEV)
    state = [torch.zeros(s, device=DEV) for s in ((1, H, D, V), (1, H, D), (1, H))]
    ref = reference(proj, offs, bias, bias, state, [T], [0], [0], H, D, V)[0][50:]
    size = reference(torch.cat((proj[:, :2 * H * D], proj[:, 2 * H * D:offs["i"]].abs(), proj[:, offs["i"]:]), 1), offs, bias, bias, state, [T], [0], [0],
                     H, D, V)[0][50:]
    o = torch.empty(T, H * V, device=DEV)
    ops.mlstm_scan(proj, offs, bias, bias, CAP, *state, meta_of([T], [T]), torch.zeros(1, dtype=torch.int32, device=DEV), o, H, D, V, D ** -0.5)
    assert ((o[50:].double() - ref).abs() <= 64 * 2.0 ** -24 * size).all()


def test_the_workspace_is_made_once(ops):
    """Steps of ever more runs, within an engine's limits, leave the recurrence's workspaces where the first prompt put them."""
    import logozen_models as zoo
    from mini_engine_b200 import LLM
    from mini_engine_b200.cache.manager import CacheHolder
    from mini_engine_b200.engine.model_runner import StepItem
    llm = LLM(zoo.folder("P"), dtype="bfloat16", kvcache_block_size=16, num_kvcache_blocks=64, max_num_seqs=4, max_num_batched_tokens=300,
              max_model_len=400)
    places = set()
    for lens in ([2], [70, 3], [200], [65, 65, 65, 65], [258, 2, 2, 2]):
        items = []
        for n in lens:
            h = CacheHolder()
            assert llm.cache.allocate(h, n)
            items.append(StepItem(h, [i % 97 for i in range(n)], 0, [n - 1]))
        llm.model_runner.step(items)
        for it in items:
            llm.cache.free(it.holder)
        arena = llm.model_runner.ctx._arena
        places.add((arena["mlstm_states"].data_ptr(), arena["mlstm_runs"].data_ptr()))
    assert len(places) == 1
