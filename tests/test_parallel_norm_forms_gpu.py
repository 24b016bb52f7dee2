"""The parallel norm's form for few rows and its general one against 64 bits.  Sums of up to 4,100 float32 terms stay within 32 * 2^-24 of the row's
scale in any of these orders (partial sums of 16 terms, then a tree), results likewise."""
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


# one, two and four runs a thread, threads that hold nothing, beyond the form's reach; few rows and more than four an SM
@pytest.mark.parametrize("W", [4, 260, 512, 1024, 1028, 2048, 4096, 4100])
@pytest.mark.parametrize("n", [1, 3, 700])
@pytest.mark.parametrize("full", [True, False])
def test_parallel_norm(ops, W, n, full):
    g = torch.Generator(DEV).manual_seed(W + n)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x = rnd(n, W) + 0.5
    ya, yb = rnd(n, W).bfloat16(), rnd(n, W).bfloat16()
    va, vb, w1, b1, w2, b2 = (rnd(W) for _ in range(6))
    adds, vectors = ([ya, yb], [va, vb]) if full else ([ya], [])
    new = x.double() + sum(t.double() for t in adds) + sum((t.double() for t in vectors), torch.zeros(W, device=DEV, dtype=torch.float64))
    unit = (new - new.mean(1, keepdim=True)) / torch.sqrt(new.var(1, unbiased=False, keepdim=True) + 1e-5)
    out1, out2 = torch.empty(n, W, device=DEV), torch.empty(n, W, device=DEV)
    norms = [(w1, b1, out1), (w2, b2, out2)] if full else [(w1, None, out1)]
    ops.parallel_norm(x, adds, vectors, 1e-5, norms[0][:2], out1, *((norms[1][:2], out2) if full else ()))
    assert ((x - new).abs() <= TOL * new.abs().max()).all()
    for w, b, out in norms:
        ref = unit * w.double() + (b.double() if b is not None else 0.0)
        assert ((out - ref).abs() <= TOL * unit.abs().max() * (w.abs().max() + 1)).all()


# which form runs is a matter of the number of rows, which a row's result does not show
@pytest.mark.parametrize("W", [4, 260, 1028, 2048, 4096])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_a_row_among_few_and_among_many(ops, W, dt):
    g = torch.Generator(DEV).manual_seed(W)
    x, ya, yb = (torch.randn(700, W, device=DEV, generator=g) for _ in range(3))
    va, w1, b1, w2 = (torch.randn(W, device=DEV, generator=g) for _ in range(4))
    res = []
    for n in (700, 3):
        s, out1, out2 = x[:n].clone(), torch.empty(n, W, device=DEV, dtype=dt), torch.empty(n, W, device=DEV, dtype=dt)
        ops.parallel_norm(s, [ya[:n].bfloat16(), yb[:n].bfloat16()], [va], 1e-5, (w1, b1), out1, (w2, None), out2)
        res.append((s[:3], out1[:3], out2[:3]))
    assert all(torch.equal(a, b) for a, b in zip(*res))
