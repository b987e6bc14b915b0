"""Gate and up projection of a prompt with the gated unit in their launch, where it can go wrong: rows beside the token tiles'
edges, gate and up rows in half a feature tile each and in a tile each, the last of them half empty, one and two token tiles, int4
operands in tensor memory and in shared memory, biases, gates of exactly zero, large ones and very negative ones (each a branch
of the SiLU's). Compared with the 16-rows-at-a-time path, whose
kernels are others, through the second layer's keys and values and the last row's logits: both paths round every operator to
BF16, so values differ by flips of roundings; 0.03 of the largest for the worst and 0.005 for the RMS, and 0.01 for the
logits' RMS, as in test_prompt_prefill_gpu.py. Its limit on the worst logit (0.021 with two layers) does not fit here: the
enlarged gates raise the residual stream and with it the flips (0.006 RMS, 0.023 worst were seen). The 512 logits' errors are
sums of many flips, so close to normal; the worst may be 5.5 times the RMS limit, which normal errors at that limit pass in
one of 50 000 runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quantized", [False, True])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("ffn", [128, 384, 1152])
@pytest.mark.parametrize("rows", [33, 250, 449])
def test_gated_prompt_projection(cuda, package, quantized, bias, ffn, rows):
    compare_paths(cuda, package, quantized, bias, ffn, rows, 512)


# int4, rows, inputs, units -> feature tiles, token tiles, columns, stages of activations, operands and packed weights, operands in
# tensor memory (tests/test_prompt_launched_cpu.py holds the shapes to it)
GATED = [
    (0, 250, 512, 192, (1, 1, 64, 8, 8, 0, 0)),
    (0, 600, 512, 3008, (2, 1, 112, 4, 4, 0, 0)),      # the last pair of tiles has 64 of 128 units
    (0, 270, 1024, 16448, (1, 2, 144, 4, 4, 0, 0)),
    (1, 470, 512, 5120, (1, 2, 240, 3, 2, 2, 0)),      # no columns left for the operands
    (1, 333, 512, 5120, (1, 2, 176, 4, 4, 8, 1)),
    (1, 1000, 512, 2944, (1, 2, 176, 4, 4, 8, 1)),     # the last group of tokens' second tile is ragged
]


@pytest.mark.parametrize("awq,rows,hidden,ffn,block", GATED)
def test_gated_blocks(cuda, package, awq, rows, hidden, ffn, block):
    compare_paths(cuda, package, bool(awq), True, ffn, rows, hidden)


def compare_paths(cuda, package, quantized, bias, ffn, rows, hidden):
    syn = package.synthetic
    capacity = 512 if rows < 512 else 1024
    shape = package.Shape(vocab_size=512, n_layers=2, n_heads=4, n_kv_heads=2, hidden_size=hidden, intermediate_size=ffn,
                          quant_type=int(quantized), max_position_embeddings=capacity)
    tensors = syn.make_model(shape, seed=8, vary_norms=True)
    for layer in range(2):
        part = 1 if quantized else 0  # int4: the scales carry a row's size
        pieces = tensors[f"w_gate{layer}"]
        size = syn.bf16_to_float(pieces[part][1]).copy()
        size[: ffn // 8] = 0.0        # gates of zero, or of the bias alone
        size[ffn // 8: ffn // 4] *= 64.0
        pieces[part] = (pieces[part][0], syn.float_to_bf16(size))
        if bias:
            for i, name in enumerate(("gate", "up")):
                values = np.random.default_rng(9 + i).standard_normal(ffn, dtype=np.float32) * np.float32(0.1)
                tensors[f"layers.{layer}.mlp.{name}_proj.bias"] = [(syn.DENSE, syn.float_to_bf16(values))]
    model = package.Model(shape, tensors)
    wide, narrow = model.new_session(capacity), model.new_session(capacity)
    ids = syn.make_prompt(14, rows, shape.vocab_size)
    wide.prefill(ids)
    narrow.prefill(ids, all_logits=cuda.empty((rows, shape.vocab_size), dtype=cuda.bfloat16, device="cuda"))
    for a, b in zip(wide.read_kv(1), narrow.read_kv(1)):
        fa, fb = syn.bf16_to_float(a)[:rows], syn.bf16_to_float(b)[:rows]
        scale = max(1.0, float(np.abs(fb).max()))
        assert np.abs(fa - fb).max() <= 0.03 * scale
        assert float(np.sqrt(((fa - fb) ** 2).mean())) <= 5e-3 * scale
    got, want = (syn.bf16_to_float(s.read_logits(1))[0] for s in (wide, narrow))
    error, scale = np.abs(got - want), float(np.abs(want).max())
    assert float(np.sqrt((error ** 2).mean())) <= 1e-2 * scale and error.max() <= 5.5e-2 * scale
