"""Products of float32 operands (csrc/gemm_f32.cu, the general form of csrc/gemm_simt.cu) against 64 bits.  A sum of K terms in any
order is off by at most K 2^-24 times the sum of their sizes; here the chains have K / 8 terms, with four further additions, and the
general form has one chain of K.  SiLU times up: the factors' bounds, and a few units in the last place for the exponential."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -24


@pytest.fixture(scope="module")
def ops():
    from mini_engine_b200 import ops
    ops.require_extension()
    return ops


def product(ops, x, w, epilogue):
    N = w.shape[0] // (2 if epilogue == "silu_mul" else 1)
    wide = torch.full((x.shape[0], N + 3), 7.0, device=DEV)          # rows further apart than the results are wide
    ops.linear(x, w, wide[:, :N], epilogue)
    assert (wide[:, N:] == 7.0).all()
    return wide[:, :N]


def check(got, x, w, epilogue, terms):
    ref, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    bound = (terms + 4) * U * size
    if epilogue == "silu_mul":
        (g, u), (bg, bu) = ref.chunk(2, 1), bound.chunk(2, 1)
        s = g * torch.sigmoid(g)                                     # silu's slope is below 1.1
        ref, bound = s * u, 1.1 * bg * (u.abs() + bu) + s.abs() * bu + 16 * U * (s * u).abs()
    assert ((got.double() - ref).abs() <= bound + 1e-37).all()


# the rows kernel's forms (4 and 8 rows), the tiles' edges; slices of 1,024 with remainders of one piece
@pytest.mark.parametrize("M", [1, 3, 4, 5, 8, 9, 16, 17, 31, 64, 65, 300])
@pytest.mark.parametrize("N,K", [(5, 4), (100, 12), (64, 64), (40, 1020), (33, 1028), (72, 3080), (520, 5000)])
@pytest.mark.parametrize("epilogue", ["none", "silu_mul"])
def test_float32_products(ops, M, N, K, epilogue):
    g = torch.Generator(DEV).manual_seed(M + N + K)
    x = torch.randn(M, K + 8, device=DEV, generator=g)[:, :K]        # rows further apart than they are long
    w = torch.randn(2 * N if epilogue == "silu_mul" else N, K, device=DEV, generator=g) * K ** -0.5
    got = product(ops, x, w, epilogue)
    check(got, x, w, epilogue, K // 8 + 1)
    one = product(ops, x[M // 2:M // 2 + 1], w, epilogue)            # a row's result does not depend on the rest of the batch
    assert torch.equal(one, got[M // 2:M // 2 + 1])
    flat = torch.empty(w.numel() + 1, device=DEV)                    # a weight that does not start on 16 bytes: the general form
    flat[1:].copy_(w.reshape(-1))
    check(product(ops, x, flat[1:].view(w.shape), epilogue), x, w, epilogue, K)


# tiles of every size by the number of SMs they fill
@pytest.mark.parametrize("M,N", [(5, 9000), (8, 4700), (17, 1024), (200, 1024), (600, 1024), (600, 4096), (33, 9000)])
def test_float32_products_of_many_tiles(ops, M, N):
    g = torch.Generator(DEV).manual_seed(M)
    x, w = torch.randn(M, 192, device=DEV, generator=g), torch.randn(N, 192, device=DEV, generator=g)
    for epilogue in ("none", "silu_mul"):
        got = product(ops, x, w, epilogue)
        check(got, x, w, epilogue, 25)
        assert torch.equal(product(ops, x[5:7], w, epilogue), got[5:7])


# rows whose distance is no multiple of four values: the general form whatever their number
@pytest.mark.parametrize("epilogue", ["none", "silu_mul"])
def test_a_row_alone_among_rows_at_odd_distances(ops, epilogue):
    g = torch.Generator(DEV).manual_seed(1)
    x = torch.randn(7, 1029, device=DEV, generator=g)[:, :1028]
    w = torch.randn(80, 1028, device=DEV, generator=g)
    got = product(ops, x, w, epilogue)
    check(got, x, w, epilogue, 1028)
    for i in (0, 4):                                                 # (row 4 starts on 16 bytes)
        assert torch.equal(product(ops, x[i:i + 1], w, epilogue), got[i:i + 1])


# more rows than tiles of rows fit the grid's y
def test_float32_products_of_very_many_rows(ops):
    g = torch.Generator(DEV).manual_seed(2)
    x, w = torch.randn(65535 * 32 + 1000, 4, device=DEV, generator=g), torch.randn(3, 4, device=DEV, generator=g)
    got = product(ops, x, w, "none")
    check(got, x, w, "none", 1)
    assert torch.equal(product(ops, x[-3:], w, "none"), got[-3:])
