"""32-bit products with long rows, which run on the tensor cores, operands cut in three: against 64-bit and against chains of
multiply-adds, at the edges of tiles, chunks and parts; a row's bits depend on nothing that comes beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


def operands(M, N, K, gated, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + N + K)
    return torch.randn(M, K, device=DEV, generator=g), torch.randn(2 * N if gated else N, K, device=DEV, generator=g) * K ** -0.5, g


# Rows of w that end inside a tile, k's that end inside a chunk, a part and a 16-byte unit, rows of x on both sides of every
# tile of 16, 32 and 64 and of what a cluster shares.
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("N,K", [(5, 768), (64, 769), (130, 1030), (257, 900), (896, 4864), (700, 1024)])
def test_rows_do_not_depend_on_their_batch(N, K, gated):
    x, w, g = operands(530, N, K, gated)
    full = ops().gemm_plain(x, w, gated=gated)
    want = x.double() @ w.double().T
    chain = torch.zeros_like(want, dtype=torch.float32)
    for k in range(K):
        chain.addcmul_(x[:, k, None], w[None, :, k])
    if gated:
        want, chain = (torch.nn.functional.silu(t[:, :N]) * t[:, N:] for t in (want, chain))
    error = lambda t: float((t.double() - want).norm() / want.norm())  # noqa: E731
    assert error(full) <= error(chain) and error(full) < 4e-7
    for rows in (1, 8, 15, 16, 17, 31, 33, 64, 65, 100, 129, 300):
        assert torch.equal(ops().gemm_plain(x[:rows], w, gated=gated), full[:rows]), rows
    assert torch.equal(ops().gemm_plain(x[37:290], w, gated=gated), full[37:290])
    # rows that start anywhere
    wide = torch.empty(530, K + 3, device=DEV)
    wide[:, 2: K + 2] = x
    assert torch.equal(ops().gemm_plain(wide[:, 2: K + 2], w, gated=gated), full)
    out = torch.full((530, N + 5), 7.0, device=DEV)
    ops().gemm_plain(x, w, gated=gated, out=out[:, 1: N + 1])
    assert torch.equal(out[:, 1: N + 1], full) and bool((out[:, 0] == 7).all()) and bool((out[:, N + 1:] == 7).all())
    if not gated:
        bias = torch.randn(N, device=DEV, generator=g)
        assert torch.equal(ops().gemm_plain(x, w, bias), full + bias)
    ops().take_device_errors()


@pytest.mark.parametrize("rows", [4, 70, 600])
def test_infinities_and_numbers_that_the_split_cannot_hold(rows):
    K, N, inf, nan = 800, 200, float("inf"), float("nan")
    x, w, _ = operands(rows, N, K, False)
    x[0, 5], x[1, 7], x[2, 700] = inf, nan, 3.4e38
    w[9, 5], w[10, 3], w[11], w[12, 700] = 0.0, -inf, 0.0, 0.5
    got = ops().gemm_plain(x, w)
    want = x.double() @ w.double().T
    big = want.abs() > 3.4028235e38
    assert torch.equal(got.isnan(), want.isnan()) and bool((got[big].double() == want[big].sign() * inf).all())
    fine = want.isfinite() & ~big
    assert bool(((got.double() - want)[fine].abs() <= 1e-5 * (x.double().abs() @ w.double().abs().T)[fine]).all())
    tiny = ops().gemm_plain(x[2:] * 1e-25, w * 1e-5)
    assert float((tiny.double() - (x[2:] * 1e-25).double() @ (w * 1e-5).double().T)[1:, 13:].abs().max()) <= 1e-35
    ops().take_device_errors()


def former(x, w):
    """x @ w.T by fused multiply-adds as the ordinary units add them up: blocks of 16 k's to four sums in turn, even and odd k's apart."""
    s = torch.zeros(4, 2, x.shape[0], w.shape[0], device=DEV)
    for k in range(x.shape[1]):
        s[k // 16 % 4, k % 2].addcmul_(x[:, k, None], w[None, :, k])
    p = s[:, 0] + s[:, 1]
    return (p[0] + p[1]) + (p[2] + p[3])


@pytest.mark.parametrize("K", [768, 1000, 4864])
@pytest.mark.parametrize("kind", ["normal", "one sign", "eight decades", "one large term", "results of 1e-36", "weights of 1e-39",
                                  "results of 1e28"])
def test_errors_are_no_larger_than_those_of_multiply_adds(K, kind):
    x, w, g = operands(60, 150, K, False, seed=3)
    w = w * K ** 0.5
    u = lambda t: torch.rand(t.shape, device=DEV, generator=g)  # noqa: E731
    if kind == "one sign":
        x, w = u(x) + 0.5, u(w) + 0.5
    elif kind == "eight decades":
        x, w = x * 10 ** (8 * u(x) - 4), w * 10 ** (8 * u(w) - 4)
    elif kind == "one large term":
        x = x * 1e-6
        x[torch.arange(60), torch.randint(K, (60,), device=DEV, generator=g)] = 1.2345678
    elif kind == "results of 1e-36":
        x, w = x * 1e-18, w * 1e-18
    elif kind == "weights of 1e-39":
        x, w = x * 1e17, w * 1e-39
    elif kind == "results of 1e28":
        x, w = x * 1e14, w * 1e14
    want, got, chain = x.double() @ w.double().T, ops().gemm_plain(x, w).double(), former(x, w).double()
    ops().take_device_errors()
    size = x.double().abs() @ w.double().abs().T
    assert (got - want).norm() <= (chain - want).norm()
    # every sum: what a chunk of 32 k's loses at its two steps and, added up, is rounded by; the parts' tree; the small terms
    assert ((got - want).abs() <= (4 + 3 + K / 256) * 2.0 ** -24 * size + 2.0 ** -149).all()


@pytest.mark.parametrize("rows,N,K", [(5, 300, 768), (70, 64, 1030)])
def test_a_row_with_one_entry_gives_back_the_column(rows, N, K):
    _, w, g = operands(rows, N, K, False)
    w[:, 3] *= 1e-30
    at, power = torch.randint(K, (rows,), device=DEV, generator=g), torch.randint(-20, 21, (rows,), device=DEV, generator=g)
    at[:2] = torch.tensor([3, K - 1])
    x = torch.zeros(rows, K, device=DEV)
    x[torch.arange(rows), at] = 2.0 ** power
    assert torch.equal(ops().gemm_plain(x, w), (w[:, at] * 2.0 ** power).T)
    assert bool((ops().gemm_plain(torch.zeros(rows, K, device=DEV), w) == 0).all())
    ops().take_device_errors()
