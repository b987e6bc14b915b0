"""The work this framework is used for, as cases with their inputs, one pass each through the public session API, the
bytes and operations a pass cannot do without, and what plain 64-bit arithmetic gives for it.

Kinds of work
  decode   one token of ordinary decoding (a draft model's step, or generation without a draft)
  verify   one verify step: the pending token and k drafts over a session's history, greedy acceptance, KV commit
  batch    one verify step of many sessions of one model in one forward
  prefill  a prompt into an empty history
  rounds   whole draft + verify rounds of a target and a draft model, chained on the device

Models have the shapes of this repository's benchmark configurations (uniform decoders in BF16 and int4 group-128, and
the two designs described layer by layer). Weights are random with the spread of trained ones: linears around 0.02
(1 / sqrt(inputs) in the layered designs; those that write to the residual stream smaller, the deeper the model the
more so), embeddings that the layers add to rather than drown, and a vocabulary head that follows the embedding, so that a
token decides its successor as clearly as in a trained model and drafts are accepted and rejected as the seed says.
Histories of uniform decoders are keys of unit size and values of the size the projections give.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__ as entry

package = entry.load_package()
runtime, synthetic = package.runtime, package.synthetic

SHIFT = 7919        # the head's row (t + SHIFT) mod vocabulary follows embedding row t
GROUP = 128


# ---- the cases ------------------------------------------------------------------------------------------------------

def listed():
    return [
        # The smallest call: one token of the 0.6B draft model, where launches and latency are everything.
        {"name": "decode_qwen3_0.6b", "kind": "decode", "model": "qwen3_0.6b", "context": 311},
        # A BF16 target with a short history and a short draft.
        {"name": "verify_qwen3_1.7b_k4", "kind": "verify", "model": "qwen3_1.7b", "rows": 5, "context": 512},
        # The headline: int4 weights, eight drafts, a history of a few pages.
        {"name": "verify_qwen3_8b_awq_k8", "kind": "verify", "model": "qwen3_8b_awq", "rows": 9, "context": 2048},
        # The same model deep in a long conversation, three drafts.
        {"name": "verify_qwen3_8b_awq_k3_long", "kind": "verify", "model": "qwen3_8b_awq", "rows": 4, "context": 30011},
        # A server's step: 64 conversations of unequal lengths, four drafts each.
        {"name": "batch_qwen2.5_7b_awq_64x5", "kind": "batch", "model": "qwen2.5_7b_awq", "sessions": 64, "rows": 5,
         "shortest": 256, "longest": 8192},
        # A few conversations that share a step.
        {"name": "batch_qwen3_8b_awq_3x5", "kind": "batch", "model": "qwen3_8b_awq", "sessions": 3, "rows": 5,
         "shortest": 700, "longest": 2500},
        # A document as the prompt of the int4 target.
        {"name": "prefill_qwen3_8b_awq_2048", "kind": "prefill", "model": "qwen3_8b_awq", "length": 2048},
        # A question of a few hundred tokens, an odd number of them.
        {"name": "prefill_qwen3_1.7b_333", "kind": "prefill", "model": "qwen3_1.7b", "length": 333},
        # Generation itself: draft and target together, a few rounds between two looks at the tokens.
        {"name": "rounds_8b_awq_with_0.6b_k8", "kind": "rounds", "model": "qwen3_8b_awq", "draft": "qwen3_0.6b", "k": 8,
         "rounds": 3, "context": 1024},
        # The layered designs: a long prompt and single tokens behind a history.
        {"name": "prefill_zofesun_w2048_1500", "kind": "prefill", "model": "zofesun_w2048", "length": 1500},
        {"name": "prefill_gikepel_w2048_2048", "kind": "prefill", "model": "gikepel_w2048", "length": 2048},
        {"name": "decode_gikepel_w1024", "kind": "decode", "model": "gikepel_w1024", "context": 700},
    ]


def draw(rng):
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["decode", "verify", "verify", "batch", "prefill", "prefill", "rounds"])
    if kind == "decode":
        model = rng.choice(["qwen3_0.6b", "qwen3_1.7b", "qwen3_8b_awq", "zofesun_w1024", "gikepel_w1024", "gikepel_w2048"])
        return {"kind": kind, "model": model, "context": spread(33, 2000)}
    if kind == "verify":
        model = rng.choice(["qwen3_0.6b", "qwen3_1.7b", "qwen3_8b_awq", "qwen3_8b_awq", "qwen2.5_7b_awq"])
        return {"kind": kind, "model": model, "rows": rng.randint(2, 16),
                "context": spread(64, 8000 if model == "qwen2.5_7b_awq" else 30000)}
    if kind == "batch":
        model = rng.choice(["qwen3_1.7b", "qwen3_8b_awq", "qwen2.5_7b_awq"])
        longest = spread(512, 8192 if model == "qwen2.5_7b_awq" else 3000)
        return {"kind": kind, "model": model, "sessions": spread(2, 64), "rows": rng.randint(2, 9),
                "shortest": rng.randint(100, 256), "longest": longest}
    if kind == "prefill":
        model = rng.choice(["qwen3_0.6b", "qwen3_1.7b", "qwen3_8b_awq", "qwen2.5_7b_awq", "zofesun_w1024", "zofesun_w2048",
                            "gikepel_w1024", "gikepel_w2048"])
        return {"kind": kind, "model": model, "length": spread(33, 2040)}
    return {"kind": "rounds", "model": rng.choice(["qwen3_8b_awq", "qwen3_1.7b"]), "draft": "qwen3_0.6b",
            "k": rng.randint(2, 8), "rounds": rng.randint(1, 3), "context": spread(64, 3000)}


# ---- models ---------------------------------------------------------------------------------------------------------

UNIFORM = {"qwen3_0.6b": synthetic.qwen3_0_6b, "qwen3_1.7b": synthetic.qwen3_1_7b, "qwen3_8b_awq": synthetic.qwen3_8b_awq,
           "qwen2.5_7b_awq": synthetic.qwen25_7b_awq}
# width, layers, attention heads, key / value heads, linear attention heads, feed-forward width
LAYERED = {"w1024": (1024, 28, 16, 8, 8, 3072), "w2048": (2048, 28, 16, 8, 16, 6144)}


def is_layered(name):
    return name.startswith(("zofesun", "gikepel"))


def shape_of(name, positions):
    if not is_layered(name):
        keep = {} if name == "qwen2.5_7b_awq" else {"max_position_embeddings": positions}
        shape = UNIFORM[name](**keep)
        shape.tied_embeddings = False
        return shape
    design, size = name.split("_")
    width, layers, heads, kv_heads, lin_heads, ff = LAYERED[size]
    if design == "zofesun":
        return synthetic.layered_decoder(width, layers, heads, kv_heads, lin_heads, ff)
    return synthetic.parallel_block_decoder(width, layers, heads, lin_heads, ff)


def generator(seed, *more):
    gen = torch.Generator(device="cuda")
    value = seed + 1
    for m in more:
        value = (value * 1000003 + m + 1) % (1 << 61)
    gen.manual_seed(value)
    return gen


def uniform_weights(shape, seed, wrong=0.0):
    """Tensors of a uniform decoder. `wrong`: share of the tokens whose successor the head gets wrong (a draft model)."""
    gen = generator(seed, 1)
    hidden, ffn, vocab = shape.hidden_size, shape.intermediate_size, shape.vocab_size
    q_width, kv_width = shape.n_heads * shape.head_dim, shape.n_kv_heads * shape.head_dim
    tensors = {}

    def linear(name, out, inp, share=1.0):
        if shape.quant_type != 1:
            t = torch.empty((out, inp), dtype=torch.bfloat16, device="cuda")
            tensors[name] = [(runtime.DENSE, t.normal_(0.0, 0.02 * share, generator=gen))]
            return
        groups = inp // GROUP
        q = torch.randint(-2**31, 2**31 - 1, (out, inp // 8), dtype=torch.int32, device="cuda", generator=gen)
        z = torch.randint(-2**31, 2**31 - 1, (out, (groups + 7) // 8), dtype=torch.int32, device="cuda", generator=gen)
        s = ((torch.rand((out, groups), device="cuda", generator=gen) * 0.003 + 0.0015) * share).to(torch.bfloat16)
        tensors[name] = [(runtime.QWEIGHT, q), (runtime.SCALES, s), (runtime.ZEROS, z)]

    def norm(name, width):
        t = torch.empty(width, device="cuda").normal_(1.0, 0.1, generator=gen).to(torch.bfloat16)
        tensors[name] = [(runtime.DENSE, t)]

    embedding = torch.empty((vocab, hidden), dtype=torch.bfloat16, device="cuda").normal_(0.0, 2.0, generator=gen)
    tensors["token_embeddings.weight"] = [(runtime.DENSE, embedding)]
    head = torch.roll(embedding, SHIFT, 0).mul_(0.015625)
    if wrong:
        bad = (torch.rand(vocab, device="cuda", generator=gen) < wrong).nonzero()[:, 0]
        head[bad] = head[torch.roll(bad, 1)]
    tensors["lm_head"] = [(runtime.DENSE, head)]
    norm("rms_out_w", hidden)
    for i in range(shape.n_layers):
        norm(f"rms_att_w{i}", hidden)
        norm(f"rms_ffn_w{i}", hidden)
        if shape.qk_norm:
            norm(f"q_norm{i}", shape.head_dim)
            norm(f"k_norm{i}", shape.head_dim)
        linear(f"wq{i}", q_width, hidden)
        linear(f"wk{i}", kv_width, hidden)
        linear(f"wv{i}", kv_width, hidden)
        linear(f"wo{i}", hidden, q_width, 0.5)
        linear(f"w_gate{i}", ffn, hidden)
        linear(f"w_up{i}", ffn, hidden)
        linear(f"w_down{i}", hidden, ffn, (2 * shape.n_layers) ** -0.5)
        if shape.qkv_bias:
            for proj, width in (("q", q_width), ("k", kv_width), ("v", kv_width)):
                bias = torch.empty(width, dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=gen)
                tensors[f"layers.{i}.self_attn.{proj}_proj.bias"] = [(runtime.DENSE, bias)]
    return tensors


def weights_of(name, shape, seed, wrong=0.0):
    return synthetic.make_device_layered_model(shape, seed) if is_layered(name) else uniform_weights(shape, seed, wrong)


def prompt_of(seed, length, vocab):
    return np.random.RandomState((seed * 7 + 3) % (1 << 31)).randint(0, vocab, length).astype(np.uint32)


def step_tokens_of(seed, rows, vocab, p=0.2):
    """[pending, drafts]: the successors of the pending token, each replaced by another token with probability p."""
    rng = np.random.RandomState((seed * 13 + 5) % (1 << 31))
    first = int(rng.randint(0, vocab))
    tokens = (first + SHIFT * np.arange(rows)) % vocab
    drawn = rng.randint(0, vocab, rows)
    replaced = rng.random_sample(rows) < p
    replaced[0] = False
    return np.where(replaced, drawn, tokens).astype(np.uint32)


def history_pool(shape, layer, longest, seed):
    """Keys and values of one layer; a session's history is a stretch of its rows. The values have the spread that the
    value projection of a unit-size input has."""
    gen = generator(seed, 2, layer)
    width = shape.n_kv_heads * shape.head_dim
    k = torch.empty((longest, width), dtype=torch.bfloat16, device="cuda").normal_(0.0, 1.0, generator=gen)
    v = torch.empty((longest, width), dtype=torch.bfloat16, device="cuda")
    return k, v.normal_(0.0, 0.02 * math.sqrt(shape.hidden_size), generator=gen)


def batch_lengths(case, seed):
    rng = np.random.RandomState((seed * 17 + 11) % (1 << 31))
    return [int(x) for x in rng.randint(case["shortest"], case["longest"] + 1, case["sessions"])]


# ---- one pass -------------------------------------------------------------------------------------------------------

class DeviceArray:
    """Memory of a session as a tensor, without a copy."""

    def __init__(self, owner, pointer, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape, "typestr": kind, "version": 2}


def logits_tensor(session, pointer, rows, vocab, layered):
    if layered:
        return torch.as_tensor(DeviceArray(session, pointer, (rows, vocab), "<f4"), device="cuda")
    return torch.as_tensor(DeviceArray(session, pointer, (rows, vocab), "<i2"), device="cuda").view(torch.bfloat16)


def prepare(case, seed):
    kind, name = case["kind"], case["model"]
    if kind == "prefill":
        capacity = case["length"] + 16
    elif kind == "batch":
        capacity = case["longest"] + 16
    elif kind == "rounds":
        capacity = case["context"] + case["rounds"] * (case["k"] + 1) + 16
    else:
        capacity = case["context"] + 16
    shape = shape_of(name, capacity)
    model = runtime.Model(shape, weights_of(name, shape, seed))
    state = {"case": case, "model": model, "vocab": shape.vocab_size, "layered": is_layered(name)}
    if kind == "prefill":
        state["session"] = model.new_session(capacity, graph=True)
        state["prompt"] = prompt_of(seed, case["length"], shape.vocab_size)
        return state
    if kind == "rounds":
        draft_shape = shape_of(case["draft"], capacity)
        draft = runtime.Model(draft_shape, uniform_weights(draft_shape, seed + 1, wrong=0.2))
        state["decoder"] = runtime.SpeculativeDecoder(model.new_session(capacity, graph=True),
                                                      draft.new_session(capacity, graph=True), case["k"])
        state["decoder"].prefill(prompt_of(seed, case["context"], shape.vocab_size))
        return state
    if state["layered"]:
        state["session"] = model.new_session(capacity, graph=True)
        state["session"].prefill(prompt_of(seed, case["context"], shape.vocab_size))
        state["tokens"] = step_tokens_of(seed, 1, shape.vocab_size)
        return state
    lengths = batch_lengths(case, seed) if kind == "batch" else [case["context"]]
    sessions = [model.new_session(capacity, graph=True) for _ in lengths]
    steps = [step_tokens_of(seed + 31 * j, case.get("rows", 1), shape.vocab_size) for j in range(len(lengths))]
    longest = max(lengths)
    for layer in range(shape.n_layers):
        k, v = history_pool(shape, layer, longest, seed)
        torch.cuda.synchronize()
        for j, (session, length) in enumerate(zip(sessions, lengths)):
            first = (longest - length) * j // len(lengths)
            session.write_kv(layer, 0, k[first:first + length], v[first:first + length])
    for session, length, step in zip(sessions, lengths, steps):
        session.adopt_history(length, int(step[0]))
    state.update(lengths=lengths, sessions=sessions, session=sessions[0], tokens=steps[0])
    if kind == "batch":
        state["batch"], state["steps"] = runtime.SessionBatch(sessions), np.stack(steps)
    return state


def run(state):
    """One pass; a step goes back to where its history ended first, so that every pass does the same work."""
    case = state["case"]
    kind = case["kind"]
    if kind == "prefill":
        pointer = state["session"].prefill(state["prompt"])
        return {"logits": logits_tensor(state["session"], pointer, 1, state["vocab"], state["layered"])}
    if kind == "rounds":
        decoder = state["decoder"]
        decoder.truncate(1)
        decoder.enqueue(case["rounds"])
        generated = decoder.drain()
        tokens = np.full(case["rounds"] * (case["k"] + 1) + 1, -1, dtype=np.int64)
        tokens[:len(generated)] = generated
        return {"tokens": tokens}
    if kind == "batch":
        for session, length in zip(state["sessions"], state["lengths"]):
            session.truncate(length)
        outputs = state["batch"].verify(state["steps"])
        return {"targets": np.array([out.targets for out in outputs], dtype=np.int64),
                "emitted": np.array([out.emitted for out in outputs], dtype=np.int64)}
    session = state["session"]
    if session.context_size() != case["context"]:
        session.truncate(case["context"])
    if kind == "decode":
        pointer = session.decode(int(state["tokens"][0]))
        return {"logits": logits_tensor(session, pointer, 1, state["vocab"], state["layered"])}
    out = session.verify(state["tokens"])
    return {"logits": logits_tensor(session, session.last_logits_ptr, case["rows"], state["vocab"], False),
            "targets": np.array(out.targets, dtype=np.int64), "emitted": out.emitted}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def layer_costs(shape):
    """[(parameters, cache bytes per token, state bytes read and written, flops per token and per pair of tokens)]"""
    hidden, costs = shape.hidden_size, []
    if not isinstance(shape, runtime.LayeredShape):
        q, kv = shape.n_heads * shape.head_dim, shape.n_kv_heads * shape.head_dim
        params = hidden * (2 * q + 2 * kv) + 3 * hidden * shape.intermediate_size
        return [(params, 4 * kv, 0, 0, 4 * q)] * shape.n_layers
    for layer in shape.layers:
        gated = 2 if shape.block == runtime.BLOCK_PARALLEL else 3
        ff = gated * hidden * (layer.ff or 0)
        if layer.rnn_width is not None:
            costs.append((4 * hidden * layer.rnn_width + ff, 0, 8 * layer.rnn_width, 0, 0))
        elif layer.latent is not None:
            a = layer.latent
            params = hidden * (a.heads * (a.dim + a.rot_dim + 2 * a.vdim) + a.kv_rank + a.rot_dim)
            params += a.heads * (a.dim + a.vdim) * a.kv_rank
            costs.append((params + ff, 2 * (a.kv_rank + a.rot_dim), 0, 0, 2 * a.heads * (a.dim + a.rot_dim + a.vdim)))
        elif layer.state_space is not None:
            m = layer.state_space
            params = hidden * (3 * m.heads * m.vdim + 2 * m.groups * m.state + m.heads)
            costs.append((params + ff, 0, 8 * m.heads * m.state * m.vdim, 4 * m.heads * m.state * m.vdim, 0))
        elif layer.delta is not None:
            m = layer.delta
            keys, values = m.kv_heads * m.dim, m.heads * m.vdim
            params = hidden * (2 * keys + 2 * values + m.decay_rank + m.gate_rank + m.heads)
            params += m.heads * m.dim * m.decay_rank + values * m.gate_rank
            costs.append((params + ff, 0, 8 * m.heads * m.dim * m.vdim, 6 * m.heads * m.dim * m.vdim, 0))
        else:
            a, l = layer.attention, layer.linear
            params = hidden * ((a.heads + a.kv_heads) * (a.dim + a.vdim) + l.heads * (2 * l.dim + 3 * l.vdim))
            costs.append((params + ff, 2 * a.kv_heads * (a.dim + a.vdim), 8 * l.heads * l.dim * l.vdim,
                          4 * l.heads * l.dim * l.vdim, 2 * a.heads * (a.dim + a.vdim)))
    return costs


def forward_work(shape, rows, context, head_rows, sessions=1, histories=None):
    """Bytes and flops of one forward of `rows` tokens per session behind `context` cached ones."""
    quantized = getattr(shape, "quant_type", 0) == 1
    per_weight = 0.5 + 2 / GROUP + 0.5 / GROUP if quantized else 2.0
    histories = [context] * sessions if histories is None else histories
    total = rows * sessions
    moved = flops = 0.0
    for params, cache, state, per_token, per_pair in layer_costs(shape):
        moved += params * per_weight + sum(cache * (h + rows) for h in histories) + state * sessions
        flops += 2.0 * params * total + per_token * total
        flops += per_pair * sum(rows * h + rows * (rows + 1) / 2 for h in histories)
    vocab, hidden = shape.vocab_size, shape.hidden_size
    logit_bytes = 4 if isinstance(shape, runtime.LayeredShape) else 2
    moved += 2.0 * vocab * hidden + logit_bytes * vocab * head_rows + 2.0 * total * hidden
    flops += 2.0 * vocab * hidden * head_rows
    return moved, flops


def work(case):
    kind = case["kind"]
    shape = shape_of(case["model"], 4096)
    if kind == "prefill":
        moved, flops = forward_work(shape, case["length"], 0, 1)
    elif kind == "batch":
        mean = (case["shortest"] + case["longest"]) / 2
        moved, flops = forward_work(shape, case["rows"], 0, case["rows"] * case["sessions"], case["sessions"],
                                    [mean] * case["sessions"])
    elif kind == "rounds":
        draft = shape_of(case["draft"], 4096)
        target_work = forward_work(shape, case["k"] + 1, case["context"], case["k"] + 1)
        draft_work = forward_work(draft, 1, case["context"], 1)
        moved, flops = (case["rounds"] * (t + (case["k"] + 1) * d) for t, d in zip(target_work, draft_work))
    else:
        rows = case.get("rows", 1)
        moved, flops = forward_work(shape, rows, case["context"], rows)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """A BF16 residual stream rounded twice a layer through 28 to 36 layers: the logits are 0.013 to 0.017 off the 64-bit
    ones (0.004 to 0.009 with the FP32 stream of the layered designs). Two correct implementations, whose roundings part
    ways after the first layers, are up to sqrt(2) times that from one another; a fifth is left for other seeds."""
    if is_layered(case["model"]):
        return {"rel": 0.015, "max": 0.15}
    return {"rel": 0.03, "max": 0.25, "differ": 0.005}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------

def as64(tensors, name):
    """A tensor in 64 bits; an int4 linear expanded to [out, in]."""
    items = tensors[name]
    if len(items) == 1:
        return items[0][1].double()
    by_kind = dict(items)
    q, s, z = by_kind[runtime.QWEIGHT], by_kind[runtime.SCALES], by_kind[runtime.ZEROS]
    out, inputs = q.shape[0], q.shape[1] * 8
    groups = inputs // GROUP
    at = torch.arange(8, dtype=torch.int32, device="cuda") * 4
    w = ((q[:, :, None] >> at) & 15).reshape(out, groups, GROUP).double()
    zero = ((z[:, :, None] >> at) & 15).reshape(out, -1)[:, :groups].double()
    return w.sub_(zero[:, :, None]).mul_(s.double()[:, :groups, None]).reshape(out, inputs)


def unit_rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def causal_weights(scores, first, sink=None):
    """Softmax of scores [heads, rows, keys] over keys at or before each row; `sink` adds a term to the denominator."""
    rows, keys = scores.shape[-2:]
    late = torch.arange(keys, device="cuda")[None, :] > first + torch.arange(rows, device="cuda")[:, None]
    scores = scores.masked_fill(late, -math.inf)
    top = scores.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink)
    e = torch.exp(scores - top)
    total = e.sum(-1, keepdim=True)
    return e / (total if sink is None else total + torch.exp(sink - top))


def half_rotation(x, first, dims, base):
    """x [rows, heads, dim]: pairs (i, i + dims / 2) turned."""
    half = dims // 2
    frequency = base ** (-2.0 * torch.arange(half, device="cuda", dtype=torch.float64) / dims)
    angle = (first + torch.arange(x.shape[0], device="cuda", dtype=torch.float64))[:, None] * frequency
    c, s = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def exact_uniform(shape, tensors, tokens, context, history, last_only):
    rows, eps, d = len(tokens), shape.rms_norm_eps, shape.head_dim
    heads, kv = shape.n_heads, shape.n_kv_heads
    x = tensors["token_embeddings.weight"][0][1][torch.as_tensor(tokens.astype(np.int64), device="cuda")].double()
    norm = lambda name: as64(tensors, name)  # noqa: E731
    for i in range(shape.n_layers):
        h = unit_rms(x, eps) * norm(f"rms_att_w{i}")
        parts = []
        for proj in "qkv":
            y = h @ as64(tensors, f"w{proj}{i}").T
            bias = f"layers.{i}.self_attn.{proj}_proj.bias"
            parts.append((y + norm(bias) if bias in tensors else y).reshape(rows, -1, d))
        q, k, v = parts
        if shape.qk_norm:
            q, k = unit_rms(q, eps) * norm(f"q_norm{i}"), unit_rms(k, eps) * norm(f"k_norm{i}")
        q, k = half_rotation(q, context, d, shape.rope_theta), half_rotation(k, context, d, shape.rope_theta)
        if context:
            old_k, old_v = history(i)
            k = torch.cat([old_k.double().reshape(context, kv, d), k])
            v = torch.cat([old_v.double().reshape(context, kv, d), v])
        out = torch.empty((rows, heads, d), dtype=torch.float64, device="cuda")
        for j in range(kv):
            mine = slice(j * heads // kv, (j + 1) * heads // kv)
            scores = q[:, mine].transpose(0, 1) @ k[:, j].T / math.sqrt(d)
            out[:, mine] = (causal_weights(scores, context) @ v[:, j]).transpose(0, 1)
        x = x + out.reshape(rows, -1) @ as64(tensors, f"wo{i}").T
        h = unit_rms(x, eps) * norm(f"rms_ffn_w{i}")
        act = silu(h @ as64(tensors, f"w_gate{i}").T)
        act *= h @ as64(tensors, f"w_up{i}").T
        x = x + act @ as64(tensors, f"w_down{i}").T
    x = x[-1:] if last_only else x
    return (unit_rms(x, eps) * norm("rms_out_w")) @ as64(tensors, "lm_head").T


def exact_zofesun(shape, tensors, tokens):
    w = lambda name: as64(tensors, name)  # noqa: E731
    T, eps = len(tokens), shape.norm_eps

    def tanh_norm(name, x):
        return torch.tanh(w(name + ".alpha").reshape(()) * x) * w(name) + w(name + ".b")

    x = w("embed")[torch.as_tensor(tokens.astype(np.int64), device="cuda")]
    for i, layer in enumerate(shape.layers):
        p = f"l{i}."
        h = tanh_norm(p + "norm1", x)
        if layer.rnn_width is not None:
            gate = torch.sigmoid(h @ w(p + "mix.z").T + w(p + "mix.z.b"))
            u = h @ w(p + "mix.x").T + w(p + "mix.x.b")
            fresh = gate * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
            keep, out = 1.0 - gate, torch.empty_like(fresh)
            state = torch.zeros_like(fresh[0])
            for t in range(T):
                state = torch.addcmul(fresh[t], keep[t], state)
                out[t] = state
            mixed = (out * silu(h @ w(p + "mix.g").T)) @ w(p + "mix.o").T
        else:
            a, l = layer.attention, layer.linear
            left, right = p + "mix.left.", p + "mix.right."
            q = half_rotation((h @ w(left + "q").T).reshape(T, a.heads, a.dim), 0, a.rot_dims, a.rot_base)
            k = half_rotation((h @ w(left + "k").T).reshape(T, a.kv_heads, a.dim), 0, a.rot_dims, a.rot_base)
            v = unit_rms((h @ w(left + "v").T).reshape(T, a.kv_heads, a.vdim), eps)
            sink, out = w(left + "sink"), []
            for n in range(a.heads):
                j = n // (a.heads // a.kv_heads)
                out.append(causal_weights(q[:, n] @ k[:, j].T * a.scale, 0, sink[n]) @ v[:, j])
            mixed = layer.left_scale * (torch.cat(out, -1) @ w(left + "o").T)
            q, k = (silu(h @ w(right + n).T).reshape(T, l.heads, l.dim) for n in "qk")
            v = silu(h @ w(right + "v").T).reshape(T, l.heads, l.vdim)
            age = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None, :]
            out = []
            for n in range(l.heads):  # the sum over earlier tokens, each decayed by its age
                fade = torch.where(age >= 0, float(l.decay[n]) ** age.clamp(min=0).double(), 0.0)
                out.append((q[:, n] @ k[:, n].T * fade) @ v[:, n])
            y = unit_rms(torch.cat(out, -1), eps) * w(right + "norm") * torch.sigmoid(h @ w(right + "g").T)
            mixed = mixed + layer.right_scale * (y @ w(right + "o").T)
        x = x + tanh_norm(p + "norm1b", mixed)
        if layer.ff is not None:
            h = tanh_norm(p + "norm2", x)
            g = (h @ w(p + "mlp.gate").T).clamp(max=layer.limit)
            u = (h @ w(p + "mlp.up").T).clamp(-layer.limit, layer.limit)
            x = x + tanh_norm(p + "norm2b", (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(p + "mlp.down").T)
    return tanh_norm("final.norm", x[-1:]) @ w("head").T


def yarn_frequencies(a):
    i = torch.arange(a.rot_dims // 2, device="cuda", dtype=torch.float64)
    plain = a.rot_base ** (-2.0 * i / a.rot_dims)
    if a.yarn is None:
        return plain, 1.0
    turns = lambda t: a.rot_dims * math.log(a.yarn.original / (2 * math.pi * t)) / (2 * math.log(a.rot_base))  # noqa: E731
    low, high = max(math.floor(turns(a.yarn.fast)), 0), min(math.ceil(turns(a.yarn.slow)), a.rot_dims - 1)
    ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
    return plain / a.yarn.factor * ramp + plain * (1.0 - ramp), 0.1 * math.log(a.yarn.factor) + 1.0


def pair_rotation(x, frequency, length):
    """x [rows, heads, n]: entries (2 i, 2 i + 1) turned and scaled by `length`."""
    angle = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None] * frequency
    c, s = length * torch.cos(angle)[:, None, :], length * torch.sin(angle)[:, None, :]
    dims, out = 2 * len(frequency), x.clone()
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    return out


def convolved(x, kernel, bias=None):
    taps = kernel.shape[1]
    padded = torch.cat([x.new_zeros((taps - 1, x.shape[1])), x])
    out = sum(padded[j:j + len(x)] * kernel[:, j] for j in range(taps))
    return silu(out if bias is None else out + bias)


def exact_gikepel(shape, tensors, tokens):
    w = lambda name: as64(tensors, name)  # noqa: E731
    T, eps, pairs = len(tokens), shape.norm_eps, shape.pairs

    def layer_norm(x, name):
        return unit_rms(x - x.mean(-1, keepdim=True), eps) * w(name)

    ids = torch.as_tensor(tokens.astype(np.int64), device="cuda")
    rows = torch.cat([ids.new_tensor([pairs.buckets]), (ids[:-1] * pairs.mul_prev + ids[1:] * pairs.mul_cur) % pairs.buckets])
    x = tensors["embed"][0][1][ids].double() + tensors["bigram"][0][1][rows].double()
    for i, layer in enumerate(shape.layers):
        p, m = f"l{i}.", f"l{i}.mix."
        h = layer_norm(x, p + "norm1")
        if layer.latent is not None:
            a = layer.latent
            q = (h @ w(m + "q").T).reshape(T, a.heads, a.dim + a.rot_dim)
            down = h @ w(m + "dkv").T
            latent = unit_rms(down[:, :a.kv_rank], eps) * w(m + "dkv.norm")
            frequency, length = yarn_frequencies(a)
            q_turned = pair_rotation(q[..., a.dim:], frequency, length)
            k_turned = pair_rotation(down[:, None, a.kv_rank:], frequency, length)[:, 0]
            up_key, up_value = w(m + "uk").reshape(a.heads, a.dim, -1), w(m + "uv").reshape(a.heads, a.vdim, -1)
            out = []
            for n in range(a.heads):
                scores = (q[:, n, :a.dim] @ (latent @ up_key[n].T).T + q_turned[:, n] @ k_turned.T) * a.scale
                out.append(causal_weights(scores, 0) @ (latent @ up_value[n].T))
            mixed = (torch.cat(out, -1) * torch.sigmoid(h @ w(m + "g").T)) @ w(m + "o").T
        elif layer.state_space is not None:
            s = layer.state_space
            inner, per = s.heads * s.vdim, s.heads // s.groups
            z, mix, dt = torch.split(h @ w(m + "in").T, [inner, inner + 2 * s.groups * s.state, s.heads], 1)
            mix = convolved(mix, w(m + "conv"), w(m + "conv.b"))
            u, b, c = torch.split(mix, [inner, s.groups * s.state, s.groups * s.state], 1)
            u = u.reshape(T, s.heads, s.vdim)
            b, c = (y.reshape(T, s.groups, s.state).repeat_interleave(per, 1) for y in (b, c))
            dt = torch.nn.functional.softplus(dt + w(m + "dt_bias"))
            gone = torch.cumsum(-torch.exp(w(m + "A_log")) * dt, 0)
            out = torch.empty_like(u)
            early = torch.ones((T, T), dtype=torch.bool, device="cuda").tril()
            for n in range(s.heads):  # the sum over earlier tokens, each faded by the decays since
                fade = torch.exp((gone[:, None, n] - gone[None, :, n]).masked_fill(~early, -math.inf))
                out[:, n] = (c[:, n] @ b[:, n].T * fade * dt[None, :, n]) @ u[:, n]
            y = (out + w(m + "D")[:, None] * u).reshape(T, inner) * silu(z)
            y = unit_rms(y.reshape(T, s.norm_groups, -1), eps).reshape(T, inner) * w(m + "norm")
            mixed = y @ w(m + "o").T
        else:
            s = layer.delta
            q, k, v = (convolved(h @ w(m + n).T, w(m + n + ".conv")) for n in "qkv")
            unit = lambda y: y * torch.rsqrt(y.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
            per = s.heads // s.kv_heads
            q = (unit(q.reshape(T, s.kv_heads, s.dim)) * s.dim ** -0.5).repeat_interleave(per, 1)
            k = unit(k.reshape(T, s.kv_heads, s.dim)).repeat_interleave(per, 1)
            v = v.reshape(T, s.heads, s.vdim)
            rate = torch.nn.functional.softplus((h @ w(m + "a1").T) @ w(m + "a2").T + w(m + "dt_bias"))
            keep = torch.exp(-torch.exp(w(m + "A_log"))[None, :, None] * rate.reshape(T, s.heads, s.dim))
            beta = torch.sigmoid(h @ w(m + "b").T)
            state = x.new_zeros((s.heads, s.dim, s.vdim))
            out = torch.empty_like(v)
            for t in range(T):
                state = state * keep[t][:, :, None]
                fresh = beta[t][:, None, None] * (v[t][:, None, :] - k[t][:, None, :] @ state)
                state = torch.baddbmm(state, k[t][:, :, None], fresh)
                out[t] = (q[t][:, None, :] @ state)[:, 0]
            gate = torch.sigmoid((h @ w(m + "g1").T) @ w(m + "g2").T)
            mixed = ((unit_rms(out, eps) * w(m + "norm")).reshape(T, -1) * gate) @ w(m + "o").T
        add = mixed * w(p + "ls1")
        if layer.ff is not None:
            h = layer_norm(x, p + "norm2")
            add = add + (h @ w(p + "mlp.up").T).clamp(min=0).square() @ w(p + "mlp.down").T * w(p + "ls2")
        x = x + add
    logits = layer_norm(x[-1:], "final.norm") @ w("embed").T
    return shape.logit_softcap * torch.tanh(logits / shape.logit_softcap)


def exact(case, seed):
    """The logits of decode, verify and prefill; tokens have no 64-bit value, and batches and rounds give only tokens."""
    kind, name = case["kind"], case["model"]
    if kind in ("batch", "rounds"):
        return None
    context = case.get("context", 0)
    shape = shape_of(name, max(context, case.get("length", 0)) + 16)
    tensors = weights_of(name, shape, seed)
    if is_layered(name):
        tokens = prompt_of(seed, case["length"] if kind == "prefill" else context, shape.vocab_size)
        if kind == "decode":
            tokens = np.concatenate([tokens, step_tokens_of(seed, 1, shape.vocab_size)])
        forward = exact_zofesun if name.startswith("zofesun") else exact_gikepel
        return {"logits": forward(shape, tensors, tokens)}
    if kind == "prefill":
        return {"logits": exact_uniform(shape, tensors, prompt_of(seed, case["length"], shape.vocab_size), 0, None, True)}
    tokens = step_tokens_of(seed, case.get("rows", 1), shape.vocab_size)
    logits = exact_uniform(shape, tensors, tokens, context, lambda i: history_pool(shape, i, context, seed), False)
    return {"logits": logits} if kind == "decode" else {"logits": logits, "targets": None, "emitted": None}
