"""Selective scans of states of up to 16 entries: single tokens, portions of a few and of many, and cuts anywhere give the same
bits, with every number of entries, channels that fill no CTA, and rows that start on no 16-byte boundary."""
import pytest
import torch

from test_segments_gpu import DEV, context, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("channels,N,shift", [(40, 16, 0), (33, 16, 1), (24, 12, 0), (37, 7, 0), (64, 8, 0), (21, 4, 0), (19, 1, 2)])
def test_cuts_and_batches_change_no_bit(channels, N, shift, dtype):
    g = torch.Generator(device=DEV).manual_seed(channels + N)
    T = 3 * 32 + 9
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    wide = lambda c: rand(T, c + shift)[:, shift:]  # noqa: E731
    x, dt_pre, z, bc = wide(channels), wide(channels) - 3, wide(channels), wide(2 * N)
    a_log, skip, bias = rand(channels, N).to(dtype), rand(channels).to(dtype), rand(channels).to(dtype)
    start = rand(3, channels, N)

    def walk(cuts, alone=True):
        state, out, at = start.clone(), [], 0
        for n in cuts:
            rows, lens, slots = torch.arange(at, at + n, device=DEV), [n], [1]
            if not alone:      # behind another request's rows and one of padding
                rows, lens, slots = torch.cat([torch.arange(5, device=DEV), rows]), [3, 2, n], [0, -1, 1]
            out.append(ops().selective_scan(x[rows], dt_pre[rows], bc[rows], 0, N, z[rows], a_log, skip, bias, state,
                                            context(lens, slots))[-n:])
            at += n
        assert torch.equal(state[2], start[2])
        return torch.cat(out), state[1]

    whole, last = walk([T])
    for cuts, alone in (([1] * T, True), ([1, 8, 3, 1, 40, 32, 20], True), ([33, 1, 71], False), ([T], False)):
        got, end = walk(cuts, alone)
        assert torch.equal(got, whole) and torch.equal(end, last), cuts
    ops().take_device_errors()
