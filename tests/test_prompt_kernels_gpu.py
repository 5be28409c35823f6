"""Kernels chosen by sizes and alignment, at the edges of their tiles, runs and pieces, against their plain statements
(tests/plain_kernels.py) and against the form that takes the same call otherwise."""
from __future__ import annotations

import pytest
import torch

import plain_kernels as P
from test_dutivik_kernels_gpu import F32, _HostBatch, _states
from test_kernels_gpu import DEV, DTYPES, K, randn
from test_pipesun_kernels_gpu import _Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps,heads,kv_heads,dim,vdim", [(4, 4, 2, 128, 128), (3, 2, 1, 32, 200), (2, 3, 3, 4, 8), (4, 2, 2, 64, 300)])
def test_convolution_in_runs(dtype, taps, heads, kv_heads, dim, vdim):
    """Runs of tokens that cross requests, requests that end inside a run, single tokens; and the same tokens in other
    portions: the same bits."""
    channels = 2 * kv_heads * dim + heads * vdim
    b_col, width = channels + heads * vdim, (channels + heads * vdim + 2 * heads + 7) & ~7
    weights = randn(channels, taps, dtype=dtype, seed=13)
    a_log, dt_bias = randn(heads, dtype=dtype, seed=14), randn(heads, dtype=dtype, seed=15)
    sizes = dict(heads=heads, kv_heads=kv_heads, dim=dim, value_dim=vdim, b_col=b_col, a_col=b_col + heads,
                 q_scale=dim ** -0.5, unit_eps=1e-6, state_offset=4)
    floats = 4 + channels * (taps - 1)
    for lens in ([(0, 530), (0, 1), (0, 9)], [(0, 61), (0, 2), (0, 7)], [(0, 1), (0, 1)]):
        batch = _Batch(lens, slots=[2, 0, 3][:len(lens)])
        rows = randn(batch.num_tokens, width, dtype=dtype, seed=17)
        state, host_state = _states(4, floats, seed=16)
        again = state.clone()
        got = K().conv_prepare(rows, weights, state, batch, a_log, dt_bias, **sizes)
        want = P.conv_prepare(rows.cpu(), weights.cpu(), host_state, _HostBatch(batch), a_log.cpu(), dt_bias.cpu(), **sizes)
        torch.testing.assert_close(got.cpu(), want, **F32)
        torch.testing.assert_close(state.cpu(), host_state, rtol=0, atol=0)
        at, parts, first = 0, [], lens[0][1]
        for n in ([first // 3, 1, first - first // 3 - 1] if first > 2 else [first]):
            parts.append(K().conv_prepare(rows[at:at + n], weights, again, _Batch([(at, n)], slots=[2]), a_log, dt_bias, **sizes))
            at += n
        assert torch.equal(torch.cat(parts), got[:first])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,vdim", [(3, 4), (2, 128), (1, 132), (5, 256), (2, 260), (1, 1024), (1, 1028), (1, 4096), (1, 4100)])
@pytest.mark.parametrize("act,weighted", [("silu", True), ("sigmoid", False)])
def test_norm_and_gate_in_pieces(dtype, heads, vdim, act, weighted):
    """Widths around the pieces a thread or a block holds; one entry off the boundary takes the other kernel."""
    tokens = 5
    o = randn(tokens, heads, vdim, dtype=torch.float32, seed=18, scale=4.0)
    weight = randn(vdim, dtype=dtype, seed=20) + 1.0 if weighted else None
    for offset in (8, 1):
        rows = randn(tokens, heads * vdim + 16, dtype=dtype, seed=19)
        gate = rows[:, offset:offset + heads * vdim]
        got = torch.zeros(tokens, heads * vdim + 8, dtype=dtype, device=DEV)
        want = got.cpu().clone()
        K().gated_rms_norm(o, gate, weight, 1e-5, got[:, 8:], 0.7, gate_act=act)
        P.gated_rms_norm(o.cpu(), gate.cpu(), None if weight is None else weight.cpu(), 1e-5, want[:, 8:], 0.7, gate_act=act)
        # the sums differ in order (2^-20 of the result at these widths); bfloat16 results may round the other way
        torch.testing.assert_close(got.cpu(), want, **(F32 if dtype == torch.float32 else dict(rtol=2.0 ** -7, atol=1e-5)))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("experts,gates,width", [(32, 1, 384), (5, 0, 1000), (70, 3, 129), (16, 0, 4096)])
def test_router_logits_have_the_same_bits_in_every_kernel(dtype, experts, gates, width):
    """Few tokens (four a block), many (eight or sixteen a block), and rows that no piece fits."""
    tokens, top = 1700, min(4, experts)
    x = randn(tokens, width, dtype=dtype, seed=1)
    router = randn(experts, width, dtype=torch.float32, seed=2, scale=0.1)
    gate_rows = randn(gates, width, dtype=torch.float32, seed=3, scale=0.1) if gates else None
    bias = randn(experts, dtype=torch.float32, seed=4)

    def route(part):
        return K().moe_route(part, router, top, score="softmax_chosen", gate_rows=gate_rows, bias=bias)
    ids, weights, g = route(x)
    z = x.double() @ router.double().T + bias.double()
    best = z.topk(top, -1).values
    # a logit of `width` products is off by less than width 2^-24 of the terms' magnitudes
    bound = (x.double().abs() @ router.double().abs().T).amax() * width * 2.0 ** -24 + 1e-6
    assert ((z.gather(1, ids.long()) - best).abs() <= 2 * bound).all()
    torch.testing.assert_close(weights.double(), torch.softmax(z.gather(1, ids.long()), -1), rtol=0, atol=float(2 * bound) + 1e-6)
    for rows in (slice(0, 1), slice(3, 8), slice(100, 227), slice(100, 228), slice(0, 600)):
        some = route(x[rows])
        assert torch.equal(some[0], ids[rows]) and torch.equal(some[1], weights[rows])
        assert g is None or torch.equal(some[2], g[rows])
    assert K().read_status() == 0


@pytest.mark.parametrize("ff", [40, 264])
@pytest.mark.parametrize("width", [128, 520])
def test_few_pairs_share_an_experts_pass(width, ff):
    """One to sixteen pairs of one expert, none shared, and pairs without an expert: each pair's row as if it were alone."""
    experts, top = 6, 2
    gate_up = randn(experts, 2 * ff, width, dtype=torch.bfloat16, seed=2, scale=0.2)
    down = randn(experts, width, ff, dtype=torch.bfloat16, seed=3, scale=0.2)
    for choice in ([[3, 3]] * 8, [[0, 1], [2, 3], [4, 5]], [[1, 4], [4, 1], [1, 1], [4, 2], [1, 4]], [[5, 6], [6, 5], [5, 5]]):
        ids = torch.tensor(choice, dtype=torch.int32, device=DEV)
        x = randn(len(choice), width, dtype=torch.bfloat16, seed=1)
        weights = torch.rand(len(choice), top, device=DEV) + 0.5

        def run(part):
            return K().moe_experts(x[part], ids[part].contiguous(), weights[part].contiguous(), gate_up, down,
                                   weight_on_input=True, path="stream", identity=1).rows.view(-1, top, width)
        rows = run(slice(None))
        real = ids < experts
        for t in range(len(choice)):
            assert torch.equal(run(slice(t, t + 1))[0][real[t]], rows[t][real[t]])
        want = P.moe_experts(x, ids.clamp(max=experts - 1), weights, gate_up, down, weight_on_input=True).view(-1, top, width)
        torch.testing.assert_close(rows[real], want[real], rtol=3e-2, atol=0.02 * float(want[real].float().abs().max()))
    assert K().read_status() == 0
