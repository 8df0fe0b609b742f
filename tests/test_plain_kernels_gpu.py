"""The plain kernels at the edges of their tiles: every variant a size picks, against 64-bit, and rows that do not
depend on the batch they come in."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


# Rows on both sides of every choice (few rows by 2, 4, 8, 16, 32; tiles of 16 and of 32), columns that end inside a
# tile, k's that end inside a load, a part and a stage, rows that are whole 16-byte units or not.
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("N,K", [(5, 3), (33, 20), (70, 65), (130, 132), (900, 72), (257, 300)])
def test_product_rows_do_not_depend_on_their_batch(N, K, gated):
    g = torch.Generator(device=DEV).manual_seed(N + K)
    x = torch.randn(530, K, device=DEV, generator=g)
    w = torch.randn(2 * N if gated else N, K, device=DEV, generator=g)
    full = ops().gemm_plain(x, w, gated=gated)
    want = x.double() @ w.double().T
    if gated:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    # every rounding is at most 2^-24 of a partial sum, of which there are K / 8 in a chain, below |x| |w|; the gate's
    # slope is at most 1.1 and its factors |x| |w|
    size = x.abs().double() @ w.abs().double().T
    size = 2.2 * size[:, :N] * size[:, N:] if gated else size
    assert bool(((full.double() - want).abs() <= (K / 8 + 8) * 2.0 ** -24 * size + 1e-30).all())
    for rows in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 47, 64, 100, 200):
        assert torch.equal(ops().gemm_plain(x[:rows], w, gated=gated), full[:rows]), rows
    bias = torch.randn(w.shape[0], device=DEV, generator=g)
    if not gated:
        assert torch.equal(ops().gemm_plain(x[3:40], w, bias), ops().gemm_plain(x, w, bias)[3:40])


def paged(rng, lens, n_kv, d, page, dtype):
    """(keys, values, block table, keys and values per request); what no request holds is NaN"""
    blocks = [-(-n // page) for n in lens]
    order = rng.permutation(sum(blocks))
    ck = np.full((sum(blocks), n_kv, page, d), np.nan, dtype=np.float32)
    cv, bt, held, at = ck.copy(), -np.ones((len(lens), max(blocks)), dtype=np.int32), [], 0
    for r, n in enumerate(lens):
        bt[r, :blocks[r]] = order[at: at + blocks[r]]
        at += blocks[r]
        k, v = (rng.standard_normal((n, n_kv, d)).astype(np.float32) for _ in range(2))
        for c, src in ((ck, k), (cv, v)):
            for j in range(n):
                c[bt[r, j // page], :, j % page] = src[j]
        held.append((k, v))
    t = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
    return t(ck).to(dtype), t(cv).to(dtype), t(bt), held


ATTENTION = [
    # heads, kv heads, head size, page, window, first positions kept, requests (positions held, new rows)
    (14, 2, 64, 16, 0, 0, [(517, 517), (40, 1), (33, 1), (1, 1)]),
    (7, 1, 128, 16, 0, 0, [(100, 40), (300, 1)]),
    (40, 2, 64, 8, 0, 0, [(70, 5), (64, 64)]),          # more heads to a kv head than a tile has rows
    (3, 3, 20, 4, 0, 0, [(90, 90), (31, 31), (32, 32), (33, 2)]),
    (4, 2, 256, 16, 0, 0, [(150, 60), (65, 1)]),
    (2, 2, 200, 16, 40, 7, [(260, 130), (9, 9)]),
    (6, 2, 8, 16, 33, 70, [(400, 200), (50, 1)]),
    (6, 3, 18, 16, 0, 0, [(70, 33)]),                    # rows of no whole 16-byte units: the block-per-row kernel
    (5, 1, 96, 32, -64, 0, [(200, 150), (129, 1)]),      # chunks
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_q,n_kv,d,page,window,keep,requests", ATTENTION)
def test_attention_rows(n_q, n_kv, d, page, window, keep, requests, dtype):
    rng = np.random.default_rng(d + n_q)
    ck, cv, bt, held = paged(rng, [n for n, _ in requests], n_kv, d, page, dtype)
    pos = np.concatenate([np.arange(n - new, n) for n, new in requests]).astype(np.int32)
    req = np.concatenate([np.full(new, r) for r, (_, new) in enumerate(requests)]).astype(np.int32)
    q = torch.from_numpy(rng.standard_normal((len(pos), n_q * d)).astype(np.float32)).to(DEV).to(dtype)

    def run(rows, single=False):
        rows = np.asarray(rows)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a[rows])).to(DEV)  # noqa: E731
        out = ops().attention_plain(q[torch.from_numpy(rows).to(DEV)], ck, cv, t(req), t(pos), bt, n_q, n_kv, d, window, d ** -0.5,
                                    keep_first=keep, single=single)
        ops().take_device_errors()
        return out

    full = run(np.arange(len(pos)))
    want = np.zeros((len(pos), n_q, d))
    for i, (r, p) in enumerate(zip(req, pos)):
        k, v = (torch.from_numpy(a[: p + 1]).to(dtype).double().numpy() for a in held[r])
        j = np.arange(p + 1)
        first = max(0, p - window + 1) if window > 0 else p // -window * -window if window else 0
        seen = (j >= first) | (j < (keep if window > 0 else 0))
        for h in range(n_q):
            s = (k[seen, h // (n_q // n_kv)] @ q[i, h * d: (h + 1) * d].double().cpu().numpy()) * d ** -0.5
            e = np.exp(s - s.max())
            want[i, h] = e @ v[seen, h // (n_q // n_kv)] / e.sum()
    err = np.linalg.norm(full.double().cpu().numpy().reshape(want.shape) - want) / np.linalg.norm(want)
    assert err < (2e-6 if dtype == torch.float32 else 4e-3)     # roundings of sums; of the result to 8 bits
    # a row alone, in tiles of its own, and in another neighbourhood gives the same bits
    some = [0, len(pos) // 2, len(pos) - 1]
    for i in some:
        assert torch.equal(run([i], single=True)[0], full[i])
    assert torch.equal(run(some), full[torch.tensor(some, device=DEV)])


def test_attention_rows_keep_infinities_and_nans_to_the_rows_that_see_them():
    rng = np.random.default_rng(3)
    n, n_q, n_kv, d = 70, 4, 2, 64
    ck, cv, bt, _ = paged(rng, [n], n_kv, d, 16, torch.float32)
    q = torch.from_numpy(rng.standard_normal((n, n_q * d)).astype(np.float32)).to(DEV)
    t = lambda a: torch.from_numpy(np.asarray(a, dtype=np.int32)).to(DEV)  # noqa: E731
    run = lambda: ops().attention_plain(q, ck, cv, t([0] * n), t(range(n)), bt, n_q, n_kv, d, 0, 0.125)  # noqa: E731
    clean = run()
    page, at = int(bt[0, 40 // 16]), 40 % 16
    cv[page, 0, at, 5], cv[page, 0, at, 9], ck[page, 1, at, 3] = float("nan"), float("inf"), float("nan")
    got = run()
    assert torch.equal(got[:40], clean[:40])
    heads, before = got[40:].view(n - 40, n_q, d), clean[40:].view(n - 40, n_q, d)
    assert bool(heads[:, :2, 5].isnan().all()) and bool((heads[:, :2, 9] == float("inf")).all())
    assert not bool(heads[:, 2:].any())      # a denominator that is no positive number leaves zeros, as the other kernel does
    assert torch.equal(heads[:, :2, 10:], before[:, :2, 10:])


def step_of(requests):
    """(rows' requests, rows' positions, the requests' first rows and the number of all) of requests (held, new)"""
    t = lambda a: torch.from_numpy(np.asarray(a, dtype=np.int32)).to(DEV)  # noqa: E731
    return (t(np.concatenate([np.full(new, r) for r, (_, new) in enumerate(requests)])),
            t(np.concatenate([np.arange(n - new, n) for n, new in requests])), t(np.cumsum([0] + [new for _, new in requests])))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_q,n_kv,d,requests", [
    (2, 2, 64, [(40, 1)] * 3 + [(90, 33)] + [(70, 1)] * 17 + [(20, 16)] + [(65, 2)] * 15),      # tiles of 8 tokens; 37 requests
    (16, 16, 64, [(40, 5)] * 60 + [(130, 70)]),                                                  # of 16
    (6, 3, 128, [(33, 1), (300, 300), (31, 1), (64, 64)]),                                       # of 8 and 4
    (7, 1, 64, [(50, 1), (80, 80), (90, 1)]), (20, 2, 32, [(50, 3), (30, 1), (90, 2)])])         # of one token
def test_requests_in_tiles_of_their_own_change_no_bit(n_q, n_kv, d, requests, dtype):
    rng = np.random.default_rng(n_q * d)
    ck, cv, bt, _ = paged(rng, [n for n, _ in requests], n_kv, d, 16, dtype)
    req, pos, q_start = step_of(requests)
    q = torch.from_numpy(rng.standard_normal((len(pos), n_q * d)).astype(np.float32)).to(DEV).to(dtype)
    run = lambda **k: ops().attention_plain(q, ck, cv, req, pos, bt, n_q, n_kv, d, 0, d ** -0.5, **k)  # noqa: E731
    together = run()
    assert torch.equal(run(out=torch.full_like(together, float("nan")), q_start=q_start, requests=len(requests)), together)
    ops().take_device_errors()


@pytest.mark.parametrize("n_q,n_kv", [(8, 8), (16, 8)])
def test_single_tokens_beside_a_portion_do_not_wait_for_one_another(n_q, n_kv):
    rng, d = np.random.default_rng(1), 64
    singles, portion = [(3000, 1)] * 16, [(64, 64)]
    ck, cv, bt, _ = paged(rng, [n for n, _ in singles + portion], n_kv, d, 16, torch.float32)

    def time_of(requests):
        req, pos, q_start = step_of(requests)
        q = torch.randn(len(pos), n_q * d, device=DEV)
        ctx = SimpleNamespace(row_req=req, row_pos=pos, q_start=q_start, n_requests=len(requests), max_q_len=max(n for _, n in requests),
                              q_lens=[n for _, n in requests])
        run = lambda: ops().attention(q, ck, cv, ctx, SimpleNamespace(block_table=bt), n_q, n_kv, d, 0, 0.125)  # noqa: E731
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            run()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    # one after another the sixteen would take many times what they take as a step of their own
    assert time_of(singles + portion) <= 2.5 * time_of(singles) + time_of(portion)


# tiles of sixteen rows (taken once they fill the multiprocessors twice): every build of them, heads in one tile and in two
WIDE = [
    (16, 8, 128, [(200, 200), (130, 110), (33, 1)]),
    (12, 4, 96, [(300, 280), (120, 119), (40, 1)]),
    (8, 8, 40, [(500, 480), (150, 130), (10, 1)]),
    (8, 8, 200, [(400, 400), (330, 219), (64, 1)]),
    (40, 2, 256, [(90, 70), (60, 20), (33, 1)]),
    (34, 2, 64, [(90, 70), (60, 20), (33, 1)]),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_q,n_kv,d,requests", WIDE)
def test_attention_in_tiles_of_sixteen_rows(n_q, n_kv, d, requests, dtype):
    group, T = n_q // n_kv, sum(new for _, new in requests)
    assert -(-T // max(1, 16 // group)) * -(-group // 16) * n_kv >= 2 * ops().sm_count()
    rng = np.random.default_rng(d)
    ck, cv, bt, held = paged(rng, [n for n, _ in requests], n_kv, d, 16, dtype)
    req, pos, q_start = step_of(requests)
    q = torch.from_numpy(rng.standard_normal((T, n_q * d)).astype(np.float32)).to(DEV).to(dtype)
    run = lambda q, req, pos, **k: ops().attention_plain(q, ck, cv, req, pos, bt, n_q, n_kv, d, 0, d ** -0.5, **k)  # noqa: E731
    full = run(q, req, pos, q_start=q_start, requests=len(requests))
    ops().take_device_errors()
    at, want = 0, []
    for (n, new), (k, v) in zip(requests, held):
        k, v = (torch.from_numpy(a).to(DEV).to(dtype).double().repeat_interleave(group, 1) for a in (k, v))
        scores = torch.einsum("qhd,khd->hqk", q[at: at + new].double().view(new, n_q, d), k) * d ** -0.5
        ahead = torch.arange(n, device=DEV)[None, :] > torch.arange(n - new, n, device=DEV)[:, None]
        want.append(torch.einsum("hqk,khd->qhd", torch.softmax(scores.masked_fill(ahead, -torch.inf), -1), v).reshape(new, -1))
        at += new
    want = torch.cat(want)
    assert float((full.double() - want).norm() / want.norm()) < (2e-6 if dtype == torch.float32 else 4e-3)
    for i in (0, T // 3, T // 2, T - 2, T - 1):      # a row alone, in a tile of eight
        assert torch.equal(run(q[i: i + 1], req[i: i + 1], pos[i: i + 1], single=True)[0], full[i])


@pytest.mark.parametrize("gated", [False, True])
def test_product_of_more_rows_than_a_grid_has_tiles(gated):
    M, N, K = 65534 * 32 + 45, 3, 4
    g = torch.Generator(device=DEV).manual_seed(0)
    x, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(2 * N if gated else N, K, device=DEV, generator=g)
    full = ops().gemm_plain(x, w, gated=gated)
    for a, b in ((0, 500), (65534 * 32 - 300, 65534 * 32), (65534 * 32 - 33, M), (65534 * 32, M)):
        assert torch.equal(full[a:b], ops().gemm_plain(x[a:b], w, gated=gated))
    want = x @ w.T
    if gated:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    assert torch.allclose(full, want, rtol=1e-4, atol=1e-5)      # (every row is there, to 32-bit roundings)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_convolution_of_many_rows(dtype):
    """From 1,500,000 entries on a thread takes eight rows: bit for bit what a thread a row gives, at requests' borders inside
    an eight, with the inputs kept from earlier steps, rows of padding and a last eight that is not full."""
    lens, slots, taps, channels = [1, 2, 3, 8, 5, 700, 16, 1, 400, 4, 300, 1], [7, 0, 2, 9, 1, 3, -1, 4, 8, -1, 5, 6], 4, 1100
    g, T = torch.Generator(device=DEV).manual_seed(4), sum(lens)
    assert T * channels >= 1500000 > T * (channels // 4) and T % 8
    t = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = SimpleNamespace(row_req=t(np.repeat(np.arange(len(lens)), lens).tolist()), q_start=t([0] + np.cumsum(lens).tolist()),
                          state_slot=t(slots), n_requests=len(lens), n_tokens=T, max_q_len=max(lens))
    proj = torch.randn(T, channels + 24, device=DEV, generator=g)
    w, b = (torch.randn(channels, taps, device=DEV, generator=g) * 0.5).to(dtype), torch.randn(channels, device=DEV, generator=g).to(dtype)
    kept = torch.randn(10, taps - 1, channels, device=DEV, generator=g)
    many = kept.clone()
    out, rounded = ops().conv_silu(proj, 8, channels, taps, w, b, many, ctx)
    part = channels // 4
    for c in range(0, channels, part):
        few = kept[:, :, c: c + part].contiguous()
        small, small_rounded = ops().conv_silu(proj, 8 + c, part, taps, w[c: c + part].contiguous(), b[c: c + part].contiguous(), few, ctx)
        assert torch.equal(out[:, c: c + part], small) and torch.equal(rounded[:, c: c + part], small_rounded)
        assert torch.equal(many[:, :, c: c + part], few)
    ops().take_device_errors()
    at = 0
    for n, slot in zip(lens, slots):
        if slot < 0:
            assert not bool(out[at: at + n].any()) and not bool(rounded[at: at + n].any())
        else:
            u = torch.cat([kept[slot], proj[at: at + n, 8: 8 + channels]]).double()
            want = torch.nn.functional.silu(sum(u[j: j + n] * w[:, j].double() for j in range(taps)) + b.double())
            # five roundings of sums of a few units, and the exponential's
            assert float((out[at: at + n].double() - want).abs().max()) < 1e-5
            assert torch.equal(many[slot].double(), u[-(taps - 1):])
        at += n
    ctx.state_slot = t([10] + slots[1:])
    ops().conv_silu(proj, 8, channels, taps, w, b, many.clone(), ctx)
    with pytest.raises(ops().KernelError):
        ops().take_device_errors()
