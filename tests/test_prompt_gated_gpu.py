"""Gate and up projection of a prompt with the gated unit in their launch, where it can go wrong: features that leave the last
tile half empty or fill only part of one, rows beside the token tiles' edges, one and two token tiles, biases, gates of exactly
zero, large ones and very negative ones (each a branch of the SiLU's). Compared with the 16-rows-at-a-time path, whose
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
    syn = package.synthetic
    shape = package.Shape(vocab_size=512, n_layers=2, n_heads=4, n_kv_heads=2, hidden_size=512, intermediate_size=ffn,
                          quant_type=int(quantized), max_position_embeddings=512)
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
    wide, narrow = model.new_session(512), model.new_session(512)
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
