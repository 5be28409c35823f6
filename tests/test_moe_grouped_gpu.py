"""The grouped products of a mixture of experts on tcgen05 against the same sums in 64 bits."""
from __future__ import annotations

import pytest
import torch

from test_kernels_gpu import DEV, K, randn

pytestmark = pytest.mark.gpu

LOADS = {
    "edges": [0, 1, 15, 16, 17, 63, 64, 65, 0, 127, 129, 255, 256, 257, 300, 2, 513],
    "one": [700] + [0] * 7,
    "small": [3, 40, 0, 16, 33, 64, 1] * 5,
    "middle": [90, 120, 0, 70, 129, 16, 180, 60],
}


@pytest.mark.parametrize("width,ff", [(264, 136), (72, 520), (1024, 256), (8, 8), (128, 384)])
@pytest.mark.parametrize("loads", list(LOADS))
@pytest.mark.parametrize("how", ["silu", "bounded", "squared"])
def test_grouped_products(loads, width, ff, how):
    """Runs at the edges of row tiles of 64, 128 and 256, weight tiles that are not whole, K that is no multiple of 64.  Hidden
    rows, results and their weighted sums are rounded to bf16 (2^-8 of a number at most, each); the fast exponential and
    division are below 2^-18, 32-bit sums below 2^-12 of their terms at these widths: 2^-6 of the terms."""
    counts = LOADS[loads]
    experts, tokens = len(counts), sum(counts)
    order = torch.randperm(tokens, generator=torch.Generator().manual_seed(1))
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts))[order].to(DEV, torch.int32)[:, None].contiguous()
    x = randn(tokens, width, dtype=torch.bfloat16, seed=2)
    up = randn(experts, (1 if how == "squared" else 2) * ff, width, dtype=torch.bfloat16, seed=3, scale=width ** -0.5)
    down = randn(experts, width, ff, dtype=torch.bfloat16, seed=4, scale=ff ** -0.5)
    weights = torch.rand(tokens, 1, generator=torch.Generator().manual_seed(5)).to(DEV) + 0.25
    join = (1.702, 2.0, 1.0) if how == "bounded" else None
    on_input = how == "silu"
    pairs = K().moe_experts(x, ids, weights, up, down, weight_on_input=on_input, path="grouped", join=join,
                            activation="squared_relu" if how == "squared" else None)
    got = K().moe_combine(pairs, tokens, 1).double()
    a = (x.float() * weights).to(torch.bfloat16) if on_input else x
    for e in range(experts):
        mine = (ids[:, 0] == e).nonzero()[:, 0]
        both = a[mine].double() @ up[e].double().T
        if how == "squared":
            hidden = both.clamp(min=0.0) ** 2
        else:
            g, u = both[:, :ff], both[:, ff:]
            if how == "bounded":
                g, u = g.clamp(max=2.0), u.clamp(-2.0, 2.0) + 1.0
            hidden = g * torch.sigmoid(g * (1.702 if how == "bounded" else 1.0)) * u
        factor = 1.0 if on_input else weights[mine].double()
        want, terms = factor * (hidden @ down[e].double().T), factor * (hidden.abs() @ down[e].double().abs().T)
        sums = a[mine].double().abs() @ up[e].double().abs().T
        # what the 32-bit sums of the first product may be off by, through the activation (slope below 2 * the sums)
        terms = terms + factor * 2.0 ** -3 * ((1 + sums) ** 2 if how == "squared" else (1 + sums[:, :ff]) * (1 + sums[:, ff:])).amax(-1, True) * 2.0 ** -9
        assert ((got[mine] - want).abs() <= terms * 2.0 ** -6).all(), e
        if len(mine) and how != "squared":
            assert (got[mine] - want).norm() <= want.norm() * 2.0 ** -7, e
    assert K().read_status() == 0


@pytest.mark.parametrize("loads", ["small", "edges"])
def test_grouped_products_of_several_experts_a_token_and_pairs_without(loads):
    """Three slots a token, some of them of experts that hand the token on; against the way by tiles of 16 rows."""
    experts = len(LOADS[loads])
    tokens, width, ff = 500, 256, 144
    generator = torch.Generator().manual_seed(7)
    ids = torch.stack([torch.randperm(experts + 2, generator=generator)[:3] for _ in range(tokens)]).to(DEV, torch.int32)
    x = randn(tokens, width, dtype=torch.bfloat16, seed=2)
    up = randn(experts, 2 * ff, width, dtype=torch.bfloat16, seed=3, scale=0.06)
    down = randn(experts, width, ff, dtype=torch.bfloat16, seed=4, scale=0.08)
    weights = torch.rand(tokens, 3, generator=generator).to(DEV)
    sums = [K().moe_combine(K().moe_experts(x, ids, weights, up, down, weight_on_input=False, path=path, identity=2), tokens, 3).double()
            for path in ("grouped", "tiles")]
    assert (sums[0] - sums[1]).norm() <= sums[1].norm() * 2.0 ** -7
    assert K().read_status() == 0


def test_grouped_products_in_a_captured_graph():
    """The host learns nothing of the loads: a graph replayed with other choices."""
    tokens, experts, width, ff = 600, 8, 256, 256
    x = randn(tokens, width, dtype=torch.bfloat16, seed=2)
    up = randn(experts, 2 * ff, width, dtype=torch.bfloat16, seed=3, scale=0.06)
    down = randn(experts, width, ff, dtype=torch.bfloat16, seed=4, scale=0.06)
    weights = torch.ones(tokens, 1, device=DEV)
    ids = torch.zeros(tokens, 1, dtype=torch.int32, device=DEV)
    run = lambda: K().moe_combine(K().moe_experts(x, ids, weights, up, down, weight_on_input=False, path="grouped"), tokens, 1)  # noqa: E731
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for seed in (1, 2):
        ids.copy_(torch.randint(0, experts if seed == 1 else 2, (tokens, 1), generator=torch.Generator().manual_seed(seed)))
        graph.replay()
        assert torch.equal(out, run())
    assert K().read_status() == 0


@pytest.mark.parametrize("of", ["up", "down"])
def test_experts_off_16_byte_boundaries_are_still_taken(of):
    """Views of a larger allocation that begin 2 bytes behind a boundary: the results of the same numbers on one (results of two
    ways, each of three roundings to bf16: 2^-7 of the sums)."""
    tokens, experts, width, ff = 300, 6, 128, 64
    x = randn(tokens, width, dtype=torch.bfloat16, seed=2)
    up = randn(experts, 2 * ff, width, dtype=torch.bfloat16, seed=3, scale=0.08)
    down = randn(experts, width, ff, dtype=torch.bfloat16, seed=4, scale=0.1)
    weights = torch.ones(tokens, 2, device=DEV)
    ids = torch.stack([torch.randperm(experts, generator=torch.Generator().manual_seed(i))[:2] for i in range(tokens)]).to(DEV, torch.int32)

    def off(t):
        room = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
        room[1:] = t.flatten()
        return room[1:].view(t.shape)
    want = K().moe_combine(K().moe_experts(x, ids, weights, up, down, weight_on_input=False), tokens, 2).double()
    rows = K().moe_experts(x, ids, weights, off(up) if of == "up" else up, off(down) if of == "down" else down, weight_on_input=False)
    got = K().moe_combine(rows, tokens, 2).double()
    assert (got - want).norm() <= want.norm() * 2.0 ** -7
    assert K().read_status() == 0
