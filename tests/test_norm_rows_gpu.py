"""Residual add and RMS norm of bfloat16 rows, few and many, at the widths where the launch changes: against 64-bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


@pytest.mark.parametrize("hidden", [4, 128, 132, 896, 1024, 1026, 1032, 1536, 2048, 2056, 4096, 4100, 4104, 8192, 8200])
@pytest.mark.parametrize("rows,parts,delta,picked", [(1, 0, False, False), (8, 9, False, False), (64, 1, True, False), (65, 3, False, True),
                                                     (700, 2, False, False), (7, 0, True, True), (8, 0, False, True),
                                                     (131, 0, True, False), (130, 0, False, True), (1300, 5, True, True)])
def test_add_and_norm(hidden, rows, parts, delta, picked):
    g = torch.Generator(device=DEV).manual_seed(hidden + rows)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    x, w = rand(rows, hidden).bfloat16(), rand(hidden).bfloat16()
    add, partial = rand(rows, hidden).bfloat16() if delta else None, rand(parts, rows, hidden) if parts else None
    pick = torch.randperm(rows, device=DEV, generator=g).to(torch.int32)[: max(1, rows // 2)] if picked else None
    before = x.clone()
    y = ops().add_rmsnorm(x, w, 1e-6, delta=add, partial=partial, rows=pick)
    ops().take_device_errors()
    v = before.double() + (add.double() if delta else 0) + (partial.double().sum(0) if parts else 0)
    if picked:
        assert torch.equal(x, before)
        stream = v[pick.long()]
    else:
        # the stream is rounded once; where 32-bit sums end on the other side of a tie, to the next value
        assert ((x.double() - v).abs() <= 2.0 ** -8 * v.abs() + 1e-6).all()
        stream = x.double()
    want = stream / torch.sqrt((stream * stream).mean(1, keepdim=True) + 1e-6) * w.double()
    # a rounding, of 2^-8 at most, of the result; where the stream is not left behind one of its entry as well, and one of the
    # row's root mean square, which a few rounded entries may make up
    assert ((y.double() - want).abs() <= (3 if picked else 1) * 2.0 ** -8 * want.abs() + 1e-5).all()


@pytest.mark.parametrize("hidden", [8, 896, 1024, 1032, 1536, 2048, 2056])
def test_a_row_has_the_same_bits_in_every_step_of_many_rows(hidden):
    """Whatever their number: 65, around four a multiprocessor, around sixteen."""
    most = 4 * ops().sm_count()
    g = torch.Generator(device=DEV).manual_seed(hidden)
    rows = 4 * most + 7
    x, w = torch.randn(rows, hidden, device=DEV, generator=g).bfloat16(), torch.randn(hidden, device=DEV, generator=g).bfloat16()
    delta = torch.randn(rows, hidden, device=DEV, generator=g).bfloat16()
    few = [(x[a: a + 65].clone(), delta[a: a + 65].contiguous()) for a in range(0, rows - 65, 65)]
    y = ops().add_rmsnorm(x, w, 1e-6, delta=delta)
    for i, (stream, add) in enumerate(few):
        assert torch.equal(ops().add_rmsnorm(stream, w, 1e-6, delta=add), y[65 * i: 65 * i + 65])
        assert torch.equal(stream, x[65 * i: 65 * i + 65])
    for n in (most, most + 1, most + 6):
        assert torch.equal(ops().add_rmsnorm(x[:n].clone(), w, 1e-6), ops().add_rmsnorm(x.clone(), w, 1e-6)[:n])
    ops().take_device_errors()


def test_a_row_out_of_range_is_an_error():
    x, w = torch.zeros(3, 896, device=DEV, dtype=torch.bfloat16), torch.ones(896, device=DEV, dtype=torch.bfloat16)
    ops().add_rmsnorm(x, w, 1e-6, rows=torch.tensor([1, 3], dtype=torch.int32, device=DEV))
    with pytest.raises(ops().KernelError):
        ops().take_device_errors()
