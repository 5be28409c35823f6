"""What is timed when a change is to make the framework faster: the calls a program that serves these models makes, from
the smallest (a tiny model in 32-bit, bound by launches) to the largest (a prompt of 2,048 tokens through one layer).

A case is a dict of plain values.  ``kind`` names the entry point:

* ``layer``:   one Llama decoder layer and the norm behind it, on a batch of prompt portions and decoded tokens;
* ``mixer``:   a mixer of one of the other designs (``design``) with its projections, states or cached rows;
* ``experts``: a mixture of experts (``form``: bounded units and softmax over the chosen logits, or SiLU units and
               sigmoid scores);
* ``head``:    the final norm and the logits;
* ``replay``:  a whole model through ``StepFunction``: prompts, then decode steps, logits of every step.

``prepare`` makes the part with weights of the wanted seed, the inputs and the step's description; ``run`` is one call.
``exact`` states the same arithmetic in 64 bits with plain torch.
"""
from __future__ import annotations

import hashlib
import json
import math
import tempfile
from pathlib import Path

import torch

from kvcore_b200 import CacheConfig, DeviceConfig, KVCoreConfig, LoadConfig, ModelConfig, SchedulerConfig
from kvcore_b200.config.model_spec import PartSpec
from kvcore_b200.config.registry import model_spec_from_config
from kvcore_b200.engine.runner import ModelRunner
from kvcore_b200.engine.step import LayerCache, StepContext, StepEntry
from kvcore_b200.parts.base import BLOCKS, FEED_FORWARDS, LM_HEADS, MIXERS, NORMS, Summed

DEV = "cuda"
PAGE = 16
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
# layer sizes of the benchmark's models: Llama 3.1 8B, Llama 3.2 3B, and the narrow size of its design comparison
SIZES = {
    "8b": dict(width=4096, heads=32, kv_heads=8, dim=128, ff=14336, vocab=128256, factor=8.0),
    "3b": dict(width=3072, heads=24, kv_heads=8, dim=128, ff=8192, vocab=128256, factor=32.0),
    "w2048": dict(width=2048, heads=16, kv_heads=4, dim=128, ff=8192, vocab=32000, factor=8.0),
    "tiny": dict(width=64, heads=4, kv_heads=2, dim=16, ff=128, vocab=256, factor=None),
}
STATEFUL = ("lightning", "gated_linear", "retention", "state_space", "delta")


def listed():
    return [
        # the decode step of a served model: few requests with long contexts, many with short ones
        dict(name="layer decode 8 x 8192", kind="layer", size="8b", dtype="bfloat16", prompts=0, prompt=0, cached=0,
             decodes=8, context=8192),
        dict(name="layer decode 64 x 1024", kind="layer", size="8b", dtype="bfloat16", prompts=0, prompt=0, cached=0,
             decodes=64, context=1024),
        # a whole prompt, and the step of continuous batching: portions of prompts beside decoded tokens
        dict(name="layer prompt 2048", kind="layer", size="8b", dtype="bfloat16", prompts=1, prompt=2048, cached=0,
             decodes=0, context=0),
        dict(name="layer mixed 511 3b", kind="layer", size="3b", dtype="bfloat16", prompts=2, prompt=240, cached=700,
             decodes=31, context=3000),
        # the 32-bit model, prompt beside decodes
        dict(name="layer float32 mixed", kind="layer", size="3b", dtype="float32", prompts=1, prompt=250, cached=0,
             decodes=6, context=1000),
        # recurrent mixers: a prompt (prefill) and a batch of single tokens (decode)
        dict(name="lightning prompt 2048", kind="mixer", design="lightning", size="8b", requests=1, tokens=2048, cached=0),
        dict(name="delta prompts 3 x 517", kind="mixer", design="delta", size="8b", requests=3, tokens=517, cached=0),
        dict(name="state space decode 64", kind="mixer", design="state_space", size="8b", requests=64, tokens=1, cached=0),
        # attention on one cached latent a token, a prompt
        dict(name="latent prompt 2048", kind="mixer", design="latent", size="8b", requests=1, tokens=2048, cached=0),
        # a mixture of experts: a prompt, and a decode step
        dict(name="experts prompt 2048", kind="experts", form="bounded", size="8b", tokens=2048, experts=32, top=4),
        dict(name="experts decode 8", kind="experts", form="bounded", size="w2048", tokens=8, experts=16, top=2),
        # a whole model: the smallest configuration in 32-bit, two requests of 7 and 13 tokens, 8 decoded tokens each
        dict(name="replay tiny float32", kind="replay", size="tiny", layers=2, dtype="float32", lens="7,13", decodes=8),
    ]


def _log(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(("layer", "layer", "layer", "mixer", "mixer", "mixer", "experts", "head", "replay"))
    if kind == "layer":
        dtype = "float32" if rng.random() < 0.2 else "bfloat16"
        size = "w2048" if dtype == "float32" else rng.choice(("8b", "3b", "w2048"))
        form = rng.choice(("decode", "prompt", "mixed"))
        case = dict(kind=kind, size=size, dtype=dtype, prompts=0, prompt=0, cached=0, decodes=0, context=0)
        if form != "decode":
            case.update(prompts=1 if form == "prompt" else rng.randint(1, 3), cached=rng.choice((0, 0, _log(rng, 16, 3000))))
            case["prompt"] = _log(rng, 17, (2048 if form == "prompt" else 512) // (4 if dtype == "float32" else 1)) // case["prompts"] + 1
        if form != "prompt":
            case.update(decodes=_log(rng, 1, 8 if dtype == "float32" else 64))
            case["context"] = _log(rng, 33, 1000 if dtype == "float32" else 65536 // max(8, case["decodes"]))
        return case
    if kind == "mixer":
        case = dict(kind=kind, design=rng.choice(STATEFUL + ("latent", "differential")), size=rng.choice(("8b", "w2048")),
                    cached=0)
        if rng.random() < 0.4:
            case.update(requests=_log(rng, 1, 64), tokens=1)
        else:
            case["requests"] = rng.randint(1, 4)
            case["tokens"] = _log(rng, 5, 2048 // case["requests"])
        if case["design"] not in STATEFUL:
            case["cached"] = _log(rng, 20, 2048) if case["tokens"] == 1 or rng.random() < 0.3 else 0
        return case
    if kind == "experts":
        size, experts, top = rng.choice((("8b", 32, 4), ("w2048", 16, 2)))
        return dict(kind=kind, form=rng.choice(("bounded", "silu")), size=size, tokens=_log(rng, 1, 2048), experts=experts, top=top)
    if kind == "head":
        return dict(kind=kind, size=rng.choice(("8b", "3b", "w2048")), rows=_log(rng, 1, 64))
    size = rng.choice(("tiny", "w2048"))
    lens = ",".join(str(_log(rng, 3, 60 if size == "tiny" else 300)) for _ in range(rng.randint(1, 6)))
    return dict(kind=kind, size=size, layers=rng.randint(1, 3), dtype=rng.choice(("bfloat16", "float32")), lens=lens,
                decodes=rng.randint(3, 12))


# ---- weights and inputs, made from the seed and a name alone ----------------------------------------------------------
def _random(seed, name, shape, std=1.0, mean=0.0):
    number = int.from_bytes(hashlib.sha256(f"{seed}/{name}".encode()).digest()[:7], "little")
    generator = torch.Generator(device=DEV).manual_seed(number)
    return torch.randn(tuple(shape), generator=generator, device=DEV, dtype=torch.float32) * std + mean


def _weight(seed, name, shape):
    """A checkpoint tensor, 32-bit: norms around one, constants of the recurrences as models have them, else N(0, 0.02)."""
    leaf = name.split(".")[-1]
    if name.endswith("norm.weight") or leaf == "norm":
        return _random(seed, name, shape, 0.1, 1.0)
    if leaf == "A_log":
        return torch.log(0.5 + 3.0 * torch.sigmoid(_random(seed, name, shape)))
    if leaf == "dt_bias":
        return _random(seed, name, shape, 1.0, -2.0)
    if leaf == "conv":
        return _random(seed, name, shape, 0.5)
    if name.endswith("a2.b"):
        return _random(seed, name, shape, 1.0, 2.0)
    if leaf in ("lq1", "lk1", "lq2", "lk2"):
        return _random(seed, name, shape, 0.1)
    if leaf in ("sink", "D"):
        return _random(seed, name, shape, 1.0)
    return _random(seed, name, shape, 0.02)


def _fill(part, seed):
    for slot in part.weight_slots():
        slot.dest.copy_(_weight(seed, slot.name, slot.shape).reshape(slot.dest.shape))
    part.finalize_weights()
    return part


def _double(seed, name, shape, dtype):
    """The same tensor as the part holds it, in 64 bits."""
    return _weight(seed, name, shape).to(dtype).double()


# ---- the designs ------------------------------------------------------------------------------------------------------
def _decay(heads):
    return [1.0 - 2.0 ** (-5.0 - 5.0 * h / max(1, heads - 1)) for h in range(heads)]


def _llama(s, layers=1):
    scaling = None if s["factor"] is None else dict(rope_type="llama3", factor=s["factor"], low_freq_factor=1.0,
                                                    high_freq_factor=4.0, original_max_position_embeddings=8192)
    config = dict(architectures=["LlamaForCausalLM"], model_type="llama", vocab_size=s["vocab"], hidden_size=s["width"],
                  intermediate_size=s["ff"], num_hidden_layers=layers, num_attention_heads=s["heads"],
                  num_key_value_heads=s["kv_heads"], head_dim=s["dim"], max_position_embeddings=131072,
                  tie_word_embeddings=False, rms_norm_eps=1e-5, rope_theta=10000.0 if scaling is None else 500000.0,
                  hidden_act="silu")
    return config if scaling is None else dict(config, rope_scaling=scaling)


def _mixer(case):
    """Sizes of a design's mixer at the width of ``size`` and its part, as the benchmark's design comparison has them."""
    s = SIZES[case["size"]]
    half, dim, design = s["heads"] // 2, s["dim"], case["design"]
    common = dict(hidden_size=s["width"], eps=1e-6, name="mix")
    if design == "lightning":
        m = dict(heads=half, dim=dim, vdim=2 * dim, decay=_decay(half))
        return m, PartSpec("lightning_attention", dict(common, num_heads=half, head_dim=dim, value_dim=2 * dim,
                                                       decay=tuple(m["decay"]), q_scale=dim ** -0.5))
    if design == "gated_linear":
        m = dict(heads=half, dim=dim, vdim=2 * dim, tau=8.0, rank=16)
        return m, PartSpec("gated_linear_attention", dict(common, num_heads=half, head_dim=dim, value_dim=2 * dim, tau=8.0,
                                                          decay_rank=16))
    if design == "retention":
        m = dict(heads=half, dim=dim, vdim=2 * dim, decay=_decay(half))
        return m, PartSpec("retention", dict(common, num_heads=half, head_dim=dim, value_dim=2 * dim, decay=tuple(m["decay"]),
                                             position=PartSpec("rope", dict(head_dim=dim, rotary_dim=dim, theta=10000.0))))
    if design == "state_space":
        heads = s["width"] // 64
        m = dict(heads=heads, groups=8, dim=128, vdim=64, taps=4, norm_groups=8)
        return m, PartSpec("selective_state_space", dict(common, num_heads=heads, num_groups=8, state_dim=128, value_dim=64,
                                                         conv_taps=4, norm_groups=8))
    if design == "delta":
        m = dict(heads=half, kv_heads=half // 2, dim=dim, vdim=dim, taps=4)
        return m, PartSpec("gated_delta_rule", dict(common, num_heads=half, num_kv_heads=half // 2, head_dim=dim, value_dim=dim,
                                                    conv_taps=4))
    if design == "latent":
        m = dict(heads=s["heads"], dim=dim, rot=64, vdim=dim, rank=512, scale=(dim + 64) ** -0.5)
        return m, PartSpec("latent_attention", dict(common, num_heads=s["heads"], head_dim=dim, rot_dim=64, value_dim=dim,
                                                    kv_rank=512, scale=m["scale"], rot_base=10000.0, rot_dims=64))
    m = dict(heads=half, kv_heads=s["kv_heads"] // 2, dim=dim, vdim=2 * dim, scale=dim ** -0.5, diff=0.5)
    return m, PartSpec("differential_attention", dict(common, num_heads=half, num_kv_heads=m["kv_heads"], head_dim=dim,
                                                      value_dim=2 * dim, scale=m["scale"], diff=0.5))


# ---- the step's description ---------------------------------------------------------------------------------------------
def _portions(case):
    """(cached, new) tokens of every request, longest portion first; lengths of one case differ as requests' do."""
    if case["kind"] == "mixer":
        n, count = case["tokens"], case["requests"]
        new = [n] * count if n == 1 else [max(1, n - i * n // (3 * count)) for i in range(count)]
        return [(case["cached"] - i * case["cached"] // (2 * count), t) for i, t in enumerate(new)]
    out = [(case["cached"], max(1, case["prompt"] - i * case["prompt"] // 5)) for i in range(case["prompts"])]
    return out + [(case["context"] - i * case["context"] // (4 * case["decodes"]) - 1, 1) for i in range(case["decodes"])]


def _context(portions, seed):
    ctx = StepContext()
    lens, cached = [n for _, n in portions], [c for c, _ in portions]
    totals = [c + n for c, n in portions]
    ctx.num_reqs, ctx.num_tokens, ctx.page_size = len(portions), sum(lens), PAGE
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)
    ints = dict(dtype=torch.int32, device=DEV)
    ctx.query_start, ctx.context_lens = torch.tensor(starts, **ints), torch.tensor(cached, **ints)
    ctx.seq_lens, ctx.state_slots = torch.tensor(totals, **ints), torch.arange(len(portions), **ints)
    ctx.positions = torch.cat([torch.arange(c, c + n, **ints) for c, n in portions])
    ctx.req_index = torch.repeat_interleave(torch.arange(len(portions), **ints), torch.tensor(lens, device=DEV)).to(torch.int32)
    needed = [-(-t // PAGE) for t in totals]
    ctx.table_width = -(-max(needed) // 16) * 16
    order = (_random(seed, "pages", (sum(needed),)).argsort() + 1).to(torch.int32)      # page 0 is nobody's
    table, at = torch.zeros(len(portions), ctx.table_width, **ints), 0
    for row, count in enumerate(needed):
        table[row, :count] = order[at:at + count]
        at += count
    ctx.tables = [table]
    ctx.max_query_len, ctx.max_seq_len = max(lens), max(totals)
    ctx.max_seq_len_bound = ctx.table_width * PAGE
    ctx.decode_only = ctx.max_query_len == 1
    ctx.host_query_lens, ctx.host_context_lens, ctx.host_state_slots = lens, cached, list(range(len(portions)))
    return ctx, sum(needed) + 1


def _rows(case, seed):
    tokens = sum(n for _, n in _portions(case))
    return _random(seed, "x", (tokens, SIZES[case["size"]]["width"]))


def _cache(mixer, pages, requests, dtype, seed):
    spec, state = mixer.cache_spec(), mixer.state_spec()
    planes = () if spec is None else tuple(
        _random(seed, f"plane{i}", (pages, spec.heads, PAGE, spec.width)).to(dtype) for i in range(spec.planes))
    held = None if state is None else _random(seed, "state", (requests, *state.shape), 0.1)
    return LayerCache(0 if planes else None, planes, True, held, PAGE)


def prepare(case, seed):
    size = SIZES[case["size"]]
    kind = case["kind"]
    if kind == "replay":
        return _prepare_replay(case, seed)
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    make = dict(dtype=dtype, device=torch.device(DEV, torch.cuda.current_device()))
    state = dict(kind=kind)
    if kind == "head":
        spec = model_spec_from_config(_llama(size))
        state["norm"] = _fill(NORMS.build(spec.final_norm, **make), seed)
        state["head"] = _fill(LM_HEADS.build(spec.lm_head, **make), seed)
        state["x"] = _random(seed, "x", (case["rows"], size["width"])).to(dtype)
        return state
    if kind == "experts":
        state["part"] = _fill(FEED_FORWARDS.build(_experts(case), **make), seed)
        state["x"] = _random(seed, "x", (case["tokens"], size["width"])).to(dtype)
        return state
    portions = _portions(case)
    state["ctx"], pages = _context(portions, seed)
    state["x"] = _rows(case, seed).to(dtype)
    if kind == "layer":
        spec = model_spec_from_config(_llama(size))
        layer = spec.layers[0]
        state["part"] = _fill(BLOCKS.build(layer.block, layer=layer, **make), seed)
        state["norm"] = _fill(NORMS.build(spec.final_norm, **make), seed)
        mixer = state["part"].mixer
    else:
        mixer = state["part"] = _fill(MIXERS.build(_mixer(case)[1], **make), seed)
    state["cache"] = _cache(mixer, pages, len(portions), dtype, seed)
    return state


def run(state):
    kind = state["kind"]
    if kind == "replay":
        return _run_replay(state)
    if kind == "head":
        return state["head"].forward(state["norm"].forward(state["x"]))
    if kind == "experts":
        return state["part"].forward(state["x"], None)
    ctx, cache = state["ctx"], state["cache"]
    ctx._shared = {}          # what layers share lives for one step
    if kind == "layer":
        h, residual = state["part"].forward(state["x"].clone(), None, ctx, cache)
        if isinstance(h, Summed):
            return dict(out=state["norm"].forward(residual), stream=residual, keys=cache.k, values=cache.v)
        out, residual = state["norm"].forward_residual(h, residual)
        return dict(out=out, stream=residual, keys=cache.k, values=cache.v)
    out = state["part"].forward(state["x"], ctx, cache)
    return dict(out=out, state=cache.state) if cache.state is not None else dict(out=out, cached=cache.planes[0])


# ---- whole calls ----------------------------------------------------------------------------------------------------------
def _token_ids(case, seed):
    lens = [int(n) for n in case["lens"].split(",")]
    vocab = SIZES[case["size"]]["vocab"]
    ids = [_random(seed, f"ids{i}", (n + case["decodes"],)) for i, n in enumerate(lens)]
    return lens, [(torch.sigmoid(t) * vocab).long().clamp(max=vocab - 1).tolist() for t in ids]


def _prepare_replay(case, seed):
    folder = Path(tempfile.mkdtemp(prefix="kvcore_cases_"))
    (folder / "config.json").write_text(json.dumps(_llama(SIZES[case["size"]], case["layers"])))
    lens, ids = _token_ids(case, seed)
    longest = max(lens) + case["decodes"]
    pages = sum(-(-(n + case["decodes"]) // PAGE) for n in lens) + 1
    runner = ModelRunner(KVCoreConfig(
        model_config=ModelConfig(model=str(folder), dtype=case["dtype"], max_model_len=longest),
        load_config=LoadConfig(random_weights=True, seed=0),
        cache_config=CacheConfig(block_size=PAGE, num_gpu_blocks=pages),
        scheduler_config=SchedulerConfig(max_num_seqs=len(lens), max_num_scheduled_tokens=sum(lens)),
        device_config=DeviceConfig(device="cuda:0")))
    _fill(runner.model, seed)
    return dict(kind="replay", runner=runner, lens=lens, ids=ids, decodes=case["decodes"])


def _run_replay(state):
    """All prompts in one step, then one token of every request a step; the logits of every sampled position."""
    step, kv = state["runner"].step_function, state["runner"].kv_manager
    lens, ids, out = state["lens"], state["ids"], []
    for d in range(state["decodes"] + 1):
        entries = []
        for i, n in enumerate(lens):
            tokens = ids[i][:n] if d == 0 else ids[i][n + d - 1:n + d]
            if not kv.allocate_slots(f"r{i}", len(tokens)):
                raise RuntimeError("the pool holds every request")
            entries.append(StepEntry(f"r{i}", tokens, (len(tokens) - 1,)))
        out.append(step.step(entries).clone())      # the next step writes its logits where these are
    for i in range(len(lens)):
        kv.free(f"r{i}")
    return torch.stack(out)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def _pairs(portions):
    return sum(c * n + n * (n + 1) // 2 for c, n in portions)


def work(case):
    s, kind = SIZES[case["size"]], case["kind"]
    e = 4 if case.get("dtype") == "float32" else 2
    w = s["width"]
    layer = (s["heads"] + 2 * s["kv_heads"]) * s["dim"] * w + s["heads"] * s["dim"] * w + 3 * s["ff"] * w
    if kind == "head":
        return dict(bytes=2 * s["vocab"] * w + case["rows"] * (2 * w + 4 * s["vocab"]), flops=2 * case["rows"] * s["vocab"] * w)
    if kind == "experts":
        t, ff = case["tokens"], _expert_width(case)
        used = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** t)      # of a uniform router, on average
        return dict(bytes=used * 6 * ff * w + 4 * case["experts"] * w + 4 * t * w, flops=6 * t * case["top"] * ff * w)
    if kind == "replay":
        lens, d = [int(n) for n in case["lens"].split(",")], case["decodes"]
        model = case["layers"] * layer + s["vocab"] * w
        pairs = sum((n + d) * (n + d + 1) // 2 for n in lens)
        return dict(bytes=e * model * (d + 1) + 4 * (d + 1) * len(lens) * s["vocab"],
                    flops=2 * case["layers"] * layer * sum(n + d for n in lens) + 2 * (d + 1) * len(lens) * s["vocab"] * w
                    + 4 * case["layers"] * s["heads"] * s["dim"] * pairs)
    portions = _portions(case)
    tokens, seen = sum(n for _, n in portions), sum(c + n for c, n in portions)
    if kind == "layer":
        cached = 2 * s["kv_heads"] * s["dim"]
        return dict(bytes=e * (layer + 3 * tokens * w + cached * seen),
                    flops=2 * tokens * layer + 4 * s["heads"] * s["dim"] * _pairs(portions))
    m, design = _mixer(case)[0], case["design"]
    if design == "latent":
        weights = w * (m["heads"] * (m["dim"] + m["rot"] + 2 * m["vdim"]) + m["rank"] + m["rot"])
        up = m["heads"] * m["rank"] * (m["dim"] + m["vdim"])
        each = m["heads"] * (m["dim"] + m["rot"] + m["vdim"])
        return dict(bytes=2 * (weights + up + 2 * tokens * w + (m["rank"] + m["rot"]) * seen),
                    flops=2 * tokens * (weights + up) + 2 * each * _pairs(portions))
    if design == "differential":
        row = m["kv_heads"] * (2 * m["dim"] + m["vdim"])
        weights = w * (m["heads"] * (2 * m["dim"] + m["vdim"]) + row)
        return dict(bytes=2 * (weights + 2 * tokens * w + row * seen),
                    flops=2 * tokens * weights + 4 * m["heads"] * (m["dim"] + m["vdim"]) * _pairs(portions))
    groups = m.get("groups", m.get("kv_heads", m["heads"]))
    values = m["heads"] * m["vdim"]
    weights = w * (2 * groups * m["dim"] + 3 * values)
    matrix = m["heads"] * m["dim"] * m["vdim"]
    return dict(bytes=2 * weights + 4 * tokens * w + 8 * matrix * len(portions), flops=2 * tokens * weights + 4 * matrix * tokens)


def tolerance(case):
    """About four times the distance between the framework's results and the 64-bit ones.  ``max`` is left open where a
    token's choice of experts may fall either way at equal scores."""
    if case.get("dtype") == "float32":
        return {"rel": 8e-6, "max": 1e-4}
    if case["kind"] == "experts":
        return {"rel": 1.6e-2}
    return {"rel": 7e-3 if case["kind"] == "head" else 2e-2, "max": 2e-1}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _frequencies(dim, theta, factor=None, original=8192.0, low=1.0, high=4.0):
    inv = 1.0 / theta ** (torch.arange(0, dim, 2, dtype=torch.float64, device=DEV) / dim)
    if factor is None:
        return inv
    wave = 2.0 * math.pi / inv
    smooth = ((original / wave - low) / (high - low)).clamp(0.0, 1.0)
    return (1.0 - smooth) * inv / factor + smooth * inv


def _turn_halves(x, positions, inv):
    """x [T, heads, D]: entry i with entry i + D/2."""
    angle = (positions.double()[:, None] * inv)[:, None]
    a, b = x.chunk(2, -1)
    c, s = torch.cos(angle), torch.sin(angle)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _turn_neighbours(x, positions, inv):
    angle = (positions.double()[:, None] * inv)[:, None]
    a, b = x[..., 0::2], x[..., 1::2]
    c, s = torch.cos(angle), torch.sin(angle)
    return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)


def _attend(q, k, v, cached, scale, sink=None):
    """q [n, D] behind ``cached`` tokens, k [N, D], v [N, V]."""
    n, total = q.shape[0], k.shape[0]
    score = q @ k.T * scale
    hidden = torch.arange(total, device=DEV)[None] > torch.arange(cached, cached + n, device=DEV)[:, None]
    score = score.masked_fill(hidden, -math.inf)
    top = score.amax(-1, keepdim=True)
    if sink is not None:
        top = top.clamp(min=float(sink))
    p = torch.exp(score - top)
    total_weight = p.sum(-1, keepdim=True)
    if sink is not None:
        total_weight = total_weight + torch.exp(sink - top)
    return p @ v / total_weight


def _seen(plane, table, total):
    """Rows of a request's first ``total`` tokens: plane [pages, heads, PAGE, width] -> [heads, total, width]."""
    pages = table[:-(-total // PAGE)].long()
    return plane[pages].transpose(0, 1).flatten(1, 2)[:, :total]


def _store(plane, ctx, rows):
    """rows [T, heads, width] into the pages of their requests."""
    table = ctx.tables[0][ctx.req_index.long()]
    page = table.gather(1, (ctx.positions.long() // PAGE)[:, None])[:, 0].long()
    plane[page, :, ctx.positions.long() % PAGE] = rows


def _each(ctx):
    at = 0
    for row, (cached, n) in enumerate(zip(ctx.host_context_lens, ctx.host_query_lens)):
        yield row, at, at + n, cached
        at += n


def _llama_layer(s, get, prefix, x, planes, ctx):
    inv = _frequencies(s["dim"], 10000.0 if s["factor"] is None else 500000.0, s["factor"])
    heads, kv, dim, tokens = s["heads"], s["kv_heads"], s["dim"], x.shape[0]
    p = prefix + "self_attn."
    y = _rms(x, 1e-5) * get(prefix + "input_layernorm.weight", (s["width"],))
    project = lambda name, rows: (y @ get(p + name, (rows * dim, s["width"])).T).view(tokens, rows, dim)  # noqa: E731
    q = _turn_halves(project("q_proj.weight", heads), ctx.positions, inv)
    _store(planes[0], ctx, _turn_halves(project("k_proj.weight", kv), ctx.positions, inv))
    _store(planes[1], ctx, project("v_proj.weight", kv))
    mixed = torch.empty(tokens, heads, dim, dtype=torch.float64, device=DEV)
    for row, begin, end, cached in _each(ctx):
        total = cached + end - begin
        k, v = (_seen(plane, ctx.tables[0][row], total) for plane in planes)
        for h in range(heads):
            mixed[begin:end, h] = _attend(q[begin:end, h], k[h * kv // heads], v[h * kv // heads], cached, dim ** -0.5)
    x = x + mixed.flatten(1) @ get(p + "o_proj.weight", (s["width"], heads * dim)).T
    y = _rms(x, 1e-5) * get(prefix + "post_attention_layernorm.weight", (s["width"],))
    gate, up = (y @ get(prefix + f"mlp.{n}_proj.weight", (s["ff"], s["width"])).T for n in ("gate", "up"))
    return x + (_silu(gate) * up) @ get(prefix + "mlp.down_proj.weight", (s["width"], s["ff"])).T


def _scan(q, k, v, decay, state, ctx, beta=None):
    """q, k [T, H, D], v [T, H, V], decay [T, H, D or 1], state [requests, H, V, D]; ``beta [T, H]``: the delta rule."""
    out = torch.empty_like(v)
    for row, begin, end, _ in _each(ctx):
        S = state[row]
        for t in range(begin, end):
            S = S * decay[t][:, None]
            u = v[t] if beta is None else beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None]
            out[t] = (S @ q[t][:, :, None])[..., 0]
        state[row] = S
    return out


def _convolve(u, taps, held, ctx):
    """A causal convolution over each request's tokens; ``held [requests, channels, taps - 1]`` is what came before."""
    out, count = torch.empty_like(u), taps.shape[1]
    for row, begin, end, _ in _each(ctx):
        padded = torch.cat([held[row].T, u[begin:end]])
        out[begin:end] = sum(padded[j:j + end - begin] * taps[:, j] for j in range(count))
        held[row] = padded[padded.shape[0] - (count - 1):].T
    return out


def _exact_mixer(case, seed):
    m, spec = _mixer(case)
    design, w, bf16 = case["design"], SIZES[case["size"]]["width"], torch.bfloat16
    portions = _portions(case)
    ctx, pages = _context(portions, seed)
    x = _rows(case, seed).to(bf16).double()
    tokens, heads, dim, vdim = x.shape[0], m["heads"], m["dim"], m["vdim"]
    get = lambda name, *shape: _double(seed, "mix." + name, shape, bf16)  # noqa: E731
    project = lambda name, rows: x @ get(name, rows, w).T  # noqa: E731
    if design in ("latent", "differential"):
        part = MIXERS.build(spec, dtype=bf16, device=torch.device("meta")).cache_spec()
        plane = _random(seed, "plane0", (pages, 1, PAGE, part.width)).to(bf16).double()
        mixed = torch.empty(tokens, heads, vdim, dtype=torch.float64, device=DEV)
        if design == "latent":
            rank, rot = m["rank"], m["rot"]
            inv = _frequencies(rot, 10000.0)
            q = project("q", heads * (dim + rot)).view(tokens, heads, dim + rot)
            q = torch.cat([q[..., :dim], _turn_neighbours(q[..., dim:], ctx.positions, inv)], -1)
            down = project("dkv", rank + rot)
            latent = _rms(down[:, :rank], 1e-6) * get("dkv.norm", rank)
            turned = _turn_neighbours(down[:, None, rank:], ctx.positions, inv)
            _store(plane, ctx, torch.cat([latent[:, None], turned], -1))
            uk, uv = get("uk", heads * dim, rank).view(heads, dim, rank), get("uv", heads * vdim, rank).view(heads, vdim, rank)
            sink = get("sink", heads)
            for row, begin, end, cached in _each(ctx):
                rows = _seen(plane, ctx.tables[0][row], cached + end - begin)[0]
                for h in range(heads):
                    k = torch.cat([rows[:, :rank] @ uk[h].T, rows[:, rank:]], -1)
                    mixed[begin:end, h] = _attend(q[begin:end, h], k, rows[:, :rank] @ uv[h].T, cached, m["scale"], sink[h])
            out = mixed.flatten(1) * torch.sigmoid(project("g", heads * vdim))
        else:
            kv = m["kv_heads"]
            q = _rms((project("q", 2 * heads * dim) + get("q.b", 2 * heads * dim)).view(tokens, heads, 2, dim), 1e-6) * get("q.norm", dim)
            k = _rms((project("k", 2 * kv * dim) + get("k.b", 2 * kv * dim)).view(tokens, kv, 2, dim), 1e-6) * get("k.norm", dim)
            v = project("v", kv * vdim) + get("v.b", kv * vdim)
            _store(plane, ctx, torch.cat([k.flatten(1), v], -1)[:, None])
            vectors = [get(n, dim) for n in ("lq1", "lk1", "lq2", "lk2")]
            lam = torch.exp(vectors[0] @ vectors[1]) - torch.exp(vectors[2] @ vectors[3]) + m["diff"]
            for row, begin, end, cached in _each(ctx):
                rows = _seen(plane, ctx.tables[0][row], cached + end - begin)[0]
                keys, values = rows[:, :2 * kv * dim].unflatten(1, (kv, 2, dim)), rows[:, 2 * kv * dim:].unflatten(1, (kv, vdim))
                for h in range(heads):
                    g = h * kv // heads
                    a, b = (_attend(q[begin:end, h, n], keys[:, g, n], values[:, g], cached, m["scale"]) for n in range(2))
                    mixed[begin:end, h] = _rms(a - lam * b, 1e-6) * (1.0 - m["diff"])
            out = mixed.flatten(1)
        return dict(out=out @ get("o", w, heads * vdim).T, cached=plane)
    held = MIXERS.build(spec, dtype=bf16, device=torch.device("meta")).state_spec().shape[0]
    state = _random(seed, "state", (len(portions), held), 0.1).double()
    matrix = heads * vdim * dim
    S = state[:, :matrix].view(len(portions), heads, vdim, dim)
    kv = m.get("groups", m.get("kv_heads", heads))
    spread = lambda t, rows, size: t.reshape(tokens, rows, size).repeat_interleave(heads // rows, 1)  # noqa: E731
    if design in ("state_space", "delta"):
        channels = heads * vdim + 2 * kv * dim
        conv = state[:, matrix:matrix + channels * (m["taps"] - 1)]
        conv = (conv.view(len(portions), channels, m["taps"] - 1) if design == "delta"
                else conv.view(len(portions), m["taps"] - 1, channels).transpose(1, 2))
    if design == "state_space":
        inner, f32 = heads * vdim, torch.float32
        z, u, dt = torch.split(project("in", inner + channels + heads), [inner, channels, heads], -1)
        u = _silu(_convolve(u, _double(seed, "mix.conv", (channels, m["taps"]), f32), conv, ctx)
                  + _double(seed, "mix.conv.b", (channels,), f32))
        v, b, c = torch.split(u, [inner, kv * dim, kv * dim], -1)
        dt = torch.nn.functional.softplus(dt + _double(seed, "mix.dt_bias", (heads,), f32), threshold=1e6)
        decay = torch.exp(-torch.exp(_double(seed, "mix.A_log", (heads,), f32)) * dt)
        v = v.view(tokens, heads, vdim)
        o = _scan(spread(c, kv, dim), spread(b, kv, dim), v * dt[..., None], decay[..., None], S, ctx)
        o = (o + _double(seed, "mix.D", (heads,), f32)[:, None] * v).flatten(1) * _silu(z)
        out = _rms(o.view(tokens, m["norm_groups"], -1), 1e-6).flatten(1) * _double(seed, "mix.norm", (inner,), f32)
    elif design == "delta":
        u = torch.cat([project("q", kv * dim), project("k", kv * dim), project("v", heads * vdim)], -1)
        taps = torch.cat([get(n, rows, m["taps"]) for n, rows in (("q.conv", kv * dim), ("k.conv", kv * dim), ("v.conv", heads * vdim))])
        q, k, v = torch.split(_silu(_convolve(u, taps, conv, ctx)), [kv * dim, kv * dim, heads * vdim], -1)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        beta = torch.sigmoid(project("b", heads))
        decay = torch.exp(-torch.exp(get("A_log", heads)) * torch.nn.functional.softplus(project("a", heads) + get("dt_bias", heads)))
        o = _scan(unit(spread(q, kv, dim)) * dim ** -0.5, unit(spread(k, kv, dim)), v.view(tokens, heads, vdim), decay[..., None],
                  S, ctx, beta)
        out = ((_rms(o, 1e-6) * get("norm", vdim)) * _silu(project("g", heads * vdim)).view(tokens, heads, vdim)).flatten(1)
    else:
        q, k, v = project("q", heads * dim), project("k", heads * dim), project("v", heads * vdim)
        gate = project("g", heads * vdim)
        if design == "gated_linear":
            z = project("a1", m["rank"]) @ get("a2", heads * dim, m["rank"]).T + get("a2.b", heads * dim)
            decay = (torch.sigmoid(z) ** (1.0 / m["tau"])).view(tokens, heads, dim)
            q = q * dim ** -0.5
        else:
            decay = torch.tensor(m["decay"], dtype=torch.float32, device=DEV).double()[None, :, None].expand(tokens, heads, 1)
            if design == "lightning":
                q, k, v = _silu(q) * dim ** -0.5, _silu(k), _silu(v)
        q, k = q.view(tokens, heads, dim), k.view(tokens, heads, dim)
        if design == "retention":
            inv = _frequencies(dim, 10000.0)
            q, k = _turn_halves(q, ctx.positions, inv), _turn_halves(k, ctx.positions, inv) * dim ** -0.5
        o = _scan(q, k, v.reshape(tokens, heads, vdim), decay, S, ctx)
        if design == "lightning":
            out = _rms(o.flatten(1), 1e-6) * get("norm", heads * vdim) * torch.sigmoid(gate)
        elif design == "gated_linear":
            out = (_rms(o, 1e-6) * get("norm", vdim)).flatten(1) * _silu(gate)
        else:
            out = _rms(o, 1e-6).flatten(1) * _silu(gate)
    return dict(out=out @ get("o", w, heads * vdim).T, state=state)


def _expert_width(case):
    return SIZES[case["size"]]["ff"] // case["top"]


def _experts(case):
    bounded = case["form"] == "bounded"
    return PartSpec("routed_experts", dict(
        hidden_size=SIZES[case["size"]]["width"], num_experts=case["experts"], top_k=case["top"],
        expert_size=_expert_width(case), name="mlp", weight_on="output", join=(1.702, 7.0, 1.0) if bounded else None,
        score="softmax_chosen" if bounded else "sigmoid", renormalize=not bounded, weight_scale=1.0 if bounded else 2.5))


def _exact_experts(case, seed):
    w, ff = SIZES[case["size"]]["width"], _expert_width(case)
    x = _random(seed, "x", (case["tokens"], w)).to(torch.bfloat16).double()
    z = x @ _double(seed, "mlp.router", (case["experts"], w), torch.float32).T
    values, ids = torch.topk(z, case["top"], -1)
    bounded = case["form"] == "bounded"
    weights = torch.softmax(values, -1) if bounded else torch.sigmoid(values)
    if not bounded:
        weights = 2.5 * weights / weights.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(case["experts"]):
        token, place = (ids == e).nonzero(as_tuple=True)
        if not len(token):
            continue
        get = lambda name, *shape: _double(seed, f"mlp.experts.{e}.{name}_proj.weight", shape, torch.bfloat16)  # noqa: E731,B023
        gate, up = (x[token] @ get(n, ff, w).T for n in ("gate", "up"))
        if bounded:
            gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
            mid = gate * torch.sigmoid(1.702 * gate) * (up + 1.0)
        else:
            mid = _silu(gate) * up
        out[token] += weights[token, place, None] * (mid @ get("down", w, ff).T)
    return out


def _exact_replay(case, seed):
    s, dtype = SIZES[case["size"]], DTYPES[case["dtype"]]
    get = lambda name, shape: _double(seed, name, shape, dtype)  # noqa: E731
    lens, ids = _token_ids(case, seed)
    embed, head = get("model.embed_tokens.weight", (s["vocab"], s["width"])), get("lm_head.weight", (s["vocab"], s["width"]))
    out = torch.empty(case["decodes"] + 1, len(lens), s["vocab"], dtype=torch.float64, device=DEV)
    for i, (n, tokens) in enumerate(zip(lens, ids)):
        ctx, pages = _context([(0, len(tokens))], seed)
        x = embed[torch.tensor(tokens, device=DEV)]
        for layer in range(case["layers"]):
            planes = [torch.zeros(pages, s["kv_heads"], PAGE, s["dim"], dtype=torch.float64, device=DEV) for _ in range(2)]
            x = _llama_layer(s, get, f"model.layers.{layer}.", x, planes, ctx)
        out[:, i] = (_rms(x[n - 1:], 1e-5) * get("model.norm.weight", (s["width"],))) @ head.T
    return out


def exact(case, seed):
    kind, s = case["kind"], SIZES[case["size"]]
    if kind == "mixer":
        return _exact_mixer(case, seed)
    if kind == "experts":
        return _exact_experts(case, seed)
    if kind == "replay":
        return _exact_replay(case, seed)
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    get = lambda name, shape: _double(seed, name, shape, dtype)  # noqa: E731
    if kind == "head":
        x = _random(seed, "x", (case["rows"], s["width"])).to(dtype).double()
        return (_rms(x, 1e-5) * get("model.norm.weight", (s["width"],))) @ get("lm_head.weight", (s["vocab"], s["width"])).T
    ctx, pages = _context(_portions(case), seed)
    planes = [_random(seed, f"plane{i}", (pages, s["kv_heads"], PAGE, s["dim"])).to(dtype).double() for i in range(2)]
    x = _llama_layer(s, get, "model.layers.0.", _rows(case, seed).to(dtype).double(), planes, ctx)
    return dict(out=_rms(x, 1e-5) * get("model.norm.weight", (s["width"],)), stream=x, keys=planes[0], values=planes[1])
