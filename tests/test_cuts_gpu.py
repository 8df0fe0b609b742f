"""Recurrent mixers over long prompts, whole and in portions: in 32-bit storage the same bits whatever the cut and whoever
shares the step; where rows are walked in segments, nothing but 32-bit roundings."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from test_segments_gpu import DEV, context, ops

pytestmark = pytest.mark.gpu
MIXERS = {
    "selective_scan": dict(inner=40, state=16, dt_rank=8, taps=4),
    "decay_linear_attention": dict(heads=2, dim=16, vdim=20, decay=(0.99, 0.9), eps=1e-6),
    "state_space": dict(heads=4, vdim=12, state=16, groups=2, taps=4, norm_groups=2, eps=1e-6),
    "matrix_memory": dict(heads=3, dim=16, vdim=12, gate_cap=15.0, eps=1e-6, floor=1e-6),
}


def build(kind, seed):
    """(part, a function from lengths, slots and inputs of a step to its outputs, its states)"""
    import llm_inference_lab_b200.models.builder  # noqa: F401  (registers the parts)
    from llm_inference_lab_b200.parts.base import CacheView, lookup
    from llm_inference_lab_b200.parts.spec import CacheParts, PartSpec

    g = torch.Generator(device=DEV).manual_seed(seed)
    spec = PartSpec(kind, dict(hidden=48, **MIXERS[kind]))
    cls = lookup("mixer", kind)
    w = {t.name: torch.randn(t.shape, device=DEV, generator=g) * (0.3 if len(t.shape) > 1 else 0.5) for t in cls.tensors(spec)}
    if "A_log" in w:
        w["A_log"] -= 1.0
    part, need = cls(spec, w, torch.float32, torch.device(DEV)), cls.cache_need(spec)
    needs = need.parts if isinstance(need, CacheParts) else (need,)
    states = [torch.randn((3, *n.shape), device=DEV, generator=g) for n in needs]
    views = [CacheView(n, state=s) for n, s in zip(needs, states)]
    view = CacheView(need, parts=views) if isinstance(need, CacheParts) else views[0]

    def step(lens, slots, x):
        return part.forward(x, context(lens, slots), view)

    return step, states


@pytest.mark.parametrize("kind", list(MIXERS))
def test_32_bit_bits_depend_on_neither_cut_nor_batch(kind):
    T, other = 1100, 700
    x = torch.randn(T + other, 48, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5))
    step, states = build(kind, 1)
    start = [s.clone() for s in states]
    whole, at = step([T], [1], x[:T]), 0
    last = [s[1].clone() for s in states]

    def again():
        for s, b in zip(states, start):
            s.copy_(b)

    again()
    parts = []
    for n in (333, 1, 600, 2, 164):
        parts.append(step([n], [1], x[at: at + n]))
        at += n
    assert torch.equal(torch.cat(parts), whole) and all(torch.equal(s[1], e) for s, e in zip(states, last))
    again()
    both = step([other, T], [2, 1], torch.cat([x[T:], x[:T]]))
    assert torch.equal(both[other:], whole) and all(torch.equal(s[1], e) for s, e in zip(states, last))
    again()
    crowd = step([3] * 200 + [T], [-1] * 200 + [1], torch.cat([x[:600], x[:T]]))
    assert torch.equal(crowd[600:], whole) and all(torch.equal(s[1], e) for s, e in zip(states, last))
    ops().take_device_errors()


def recurrence(name, T):
    """(a walk over rows a .. b of a prompt of T tokens from the states it is given, the states' shapes, the number of
    segments or chunks the whole prompt is cut into)"""
    g = torch.Generator(device=DEV).manual_seed(9)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    if name == "selective_scan":
        C, N = 72, 16
        x, dt_pre, z, bc, a_log, skip, bias = rand(T, C), rand(T, C) - 4, rand(T, C), rand(T, 2 * N), rand(C, N), rand(C), rand(C)
        walk = lambda a, b, s: ops().selective_scan(x[a:b], dt_pre[a:b], bc[a:b], 0, N, z[a:b], a_log, skip, bias, s[0],  # noqa: E731
                                                    context([b - a], [0]))
        n = ops().scan_segments(3, T)
        return walk, [(1, C, N)], n if ops().scan_segments_pay(n, C, N, 1, T) else 1
    H, D, V = 3, 64, 64
    if name == "gated_delta":
        taps, G = 4, 3
        proj, conv = rand(T, 2 * G * D + H * V + 2 * H), rand(2 * G * D + H * V, taps) * 0.5
        a_log, bias, ch = rand(H), rand(H) - 4, 2 * G * D + H * V

        def walk(a, b, s):
            ctx = context([b - a], [0])
            p = proj[a:b].contiguous()
            operands = ops().delta_prepare(p, ch, ch + H, taps, H, G, D, V, conv, a_log, bias, s[1], ctx, D ** -0.5, 1e-6)
            return ops().delta_walk(*operands, s[0], ctx, H, G, D, V, proj=p, kept=s[1])

        return walk, [(1, H, D, V), (1, taps - 1, ch)], ops().delta_walk_segments(H, D, V, T)
    qk, v = rand(T, 2 * H * D), rand(T, H * V)
    gates = torch.stack([rand(T, H) * 2, -torch.nn.functional.softplus(rand(T, H) - 4)], dim=1)      # log scale, log decay
    fixed = torch.tensor([0.999, 0.99, 0.9], device=DEV)

    def walk(a, b, s):
        ctx, how = context([b - a], [0]), dict(a_head=fixed, silu=True)
        if name == "matrix_memory":
            kept = gates[a:b].clone()
            m = ops().memory_stabilize(kept, s[1], ctx)
            how = dict(a_tok=kept[:, 0], s_tok=kept[:, 1])
        o = ops().decay_scan(qk[a:b, : H * D], qk[a:b, H * D:], v[a:b], s[0], ctx, H, H, D, V, **how)
        return o if name != "matrix_memory" else o.view(-1, H, V) * torch.exp(m.clamp(-20, 20))[:, :, None]

    # (chunks of 64 rows)
    return walk, [(1, H, D, V), (1, H)], -(-T // 64) if ops().decay_scan_chunks(H * 2, D, T, H, V, T, 1) else 1


@pytest.mark.parametrize("name", ["selective_scan", "linear_state", "matrix_memory", "gated_delta"])
@pytest.mark.parametrize("T", [700, 2048])
def test_segments_and_cuts_change_roundings_only(name, T):
    walk, shapes, segments = recurrence(name, T)
    assert segments > 1
    zeros = lambda: [torch.zeros(s, device=DEV) for s in shapes]  # noqa: E731
    whole_states, states, parts = zeros(), zeros(), []
    whole = walk(0, T, whole_states)
    for a in range(0, T, 233):      # below every recurrence's first segmented length
        parts.append(walk(a, min(a + 233, T), states))
    ops().take_device_errors()
    for got, want in zip([whole] + whole_states, [torch.cat(parts)] + states):
        # 32-bit roundings over memories of up to a thousand tokens
        assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max()), float((got - want).abs().max() / want.abs().max())
