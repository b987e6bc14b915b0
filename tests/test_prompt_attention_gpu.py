"""The tensor-core prompt attention where it can go wrong: rows at the edges of its tiles of 64 tokens and 128 query rows,
groups that divide 128 (queries by copies) and that do not (queries by loads), blocks of one and of two query tiles, the
second of which may have no or few rows, histories in front of the segment, and leftovers behind it.

The uniform decoder's rows are compared with those of its 16-rows-at-a-time path (another kernel): the second layer's keys
and values have gone through the first layer's attention. Both paths round every operator to BF16, so a value differs by
flips of roundings: 0.03 of the largest for the worst, 0.005 for the RMS, as in test_prompt_prefill_gpu.py. The layered
designs are compared with their restatements in double precision, under their own tests' limits."""
import sys
from pathlib import Path

import numpy as np
import pytest

import gikepel_cases
import layered_cases
from test_gikepel_gpu import check as check_gikepel
from test_layered_gpu import check as check_layered

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import gikepel  # noqa: E402
import hybrid  # noqa: E402

pytestmark = pytest.mark.gpu


def two_layers(package, heads, kv_heads, hidden=256):
    return package.Shape(vocab_size=512, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, hidden_size=hidden,
                         intermediate_size=256, max_position_embeddings=1024)


def assert_same_rows(syn, got, want, begin, end):
    for layer in (0, 1):
        for a, b in zip(got.read_kv(layer), want.read_kv(layer)):
            fa, fb = syn.bf16_to_float(a)[begin:end], syn.bf16_to_float(b)[begin:end]
            scale = max(1.0, float(np.abs(fb).max()))
            assert np.abs(fa - fb).max() <= 0.03 * scale, layer
            assert float(np.sqrt(((fa - fb) ** 2).mean())) <= 5e-3 * scale, layer


@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 2), (6, 2), (8, 2), (14, 2)])
@pytest.mark.parametrize("history,rows", [(0, 33), (0, 64), (0, 65), (0, 129), (1, 63), (63, 65), (64, 64), (70, 130)])
def test_edges_of_tiles(cuda, package, heads, kv_heads, history, rows):
    syn = package.synthetic
    shape = two_layers(package, heads, kv_heads)
    model = package.Model(shape, syn.make_model(shape, seed=3, vary_norms=True))
    ids = syn.make_prompt(11, history + rows, shape.vocab_size)
    wide, narrow = model.new_session(256), model.new_session(256)
    narrow.prefill(ids, all_logits=cuda.empty((len(ids), shape.vocab_size), dtype=cuda.bfloat16, device="cuda"))
    if history:
        for session in (wide, narrow):
            session.prefill(ids[:history], all_logits=cuda.empty((history, shape.vocab_size), dtype=cuda.bfloat16, device="cuda"))
        for at in range(history, len(ids), 16):
            narrow.extend(ids[at:at + 16])
        wide.extend(ids[history:])
    else:
        wide.prefill(ids)
    assert_same_rows(syn, wide, narrow, history, len(ids))


@pytest.mark.parametrize("heads,kv_heads,rows", [(40, 40, 300), (32, 8, 610), (32, 8, 600), (56, 8, 400), (40, 40, 428)])
def test_blocks_of_two_query_tiles(cuda, package, heads, kv_heads, rows):
    """More blocks than half the multiprocessors; the last block's second query tile has 0, 8, 0, 112 and 44 rows."""
    syn = package.synthetic
    shape = two_layers(package, heads, kv_heads)
    model = package.Model(shape, syn.make_model(shape, seed=4, vary_norms=True))
    ids = syn.make_prompt(12, rows, shape.vocab_size)
    wide, narrow = model.new_session(640), model.new_session(640)
    wide.prefill(ids)
    narrow.prefill(ids, all_logits=cuda.empty((rows, shape.vocab_size), dtype=cuda.bfloat16, device="cuda"))
    assert_same_rows(syn, wide, narrow, 0, rows)


@pytest.mark.parametrize("history,rows", [(20, 50), (100, 40)])
def test_leftovers_behind_the_history_do_not_matter(cuda, package, history, rows):
    syn = package.synthetic
    shape = two_layers(package, 4, 2)
    model = package.Model(shape, syn.make_model(shape, seed=5, vary_norms=True))
    ids = syn.make_prompt(13, history + rows, shape.vocab_size)
    clean, dirty = model.new_session(256), model.new_session(256)
    for session in (clean, dirty):
        session.prefill(ids[:history])
    bad = cuda.full((256 - history, 256), float("nan"), dtype=cuda.bfloat16, device="cuda")
    for layer in (0, 1):
        dirty.write_kv(layer, history, bad, bad)
    for session in (clean, dirty):
        session.extend(ids[history:])
    for layer in (0, 1):
        for a, b in zip(clean.read_kv(layer), dirty.read_kv(layer)):
            assert np.array_equal(a[:history + rows], b[:history + rows])


@pytest.mark.parametrize("heads,kv_heads", [(40, 40), (42, 14)])
def test_layered_designs_with_two_query_tiles(cuda, package, heads, kv_heads):
    c = layered_cases.config(64, 64, [layered_cases.parallel((heads, kv_heads, 128, 128, 32, 1e5), (1, 16, 16))])
    weights = layered_cases.random_weights(package, c, 6)
    model = package.Model(*package.checkpoint.admit(c, weights, "zofesun_bf16"))
    ids = layered_cases.tokens(c, 450)
    want = hybrid.HybridOracle(c, weights).forward(ids)
    session = model.new_session(460)
    check_layered(layered_cases.run_portions(session, ids, [300, 150]), want, "bf16")


def test_latent_attention_with_two_query_tiles(cuda, package):
    c = gikepel_cases.config(64, 64, [gikepel_cases.latent(40, 128, 64, 128, 64)])
    weights = gikepel_cases.random_weights(package, c, 7)
    model = package.Model(*package.checkpoint.admit(c, weights, "gikepel_bf16"))
    ids = layered_cases.tokens(c, 450)
    want = gikepel.GikepelOracle(c, weights).forward(ids)
    session = model.new_session(460)
    check_gikepel(layered_cases.run_portions(session, ids, [300, 150]), want, "bf16")


def test_a_weight_that_dominates_is_not_rounded(cuda, package):
    """One token of the first tile of 64, then one of the second that outweighs it by 2^n (1 + 0.9 2^-8): rounded to BF16 and
    summed unrounded, that weight would take 0.9 2^-8 off the row; as the largest weight it is 1. All other tokens' weights
    vanish. Every projection only selects, so the second layer's values are the first layer's attention output after two
    roundings to BF16 (2^-8 / sqrt(3) RMS at most, each), whose mean over the 128 values of a head, weighted with their
    squares, has a standard deviation of 2^-8 sqrt(2/3) sqrt(3/128) at most: 4.9e-4. The limit of 1.9e-3 is four times that;
    the rounded weight's errors start at 0.75 x 3.5e-3 (a fifth of the row is the other token, a twentieth goes into the norm)."""
    syn = package.synthetic
    heads, hidden, history, rows, theta = 8, 2048, 128, 64, 1e7
    half = hidden // 2
    shape = package.Shape(vocab_size=512, n_layers=2, n_heads=heads, n_kv_heads=heads, hidden_size=hidden, intermediate_size=256,
                          qk_norm=False, rope_theta=theta, max_position_embeddings=512)
    tensors = syn.make_model(shape, seed=6)

    def put(name, array):
        tensors[name] = [(syn.DENSE, syn.float_to_bf16(array.astype(np.float32)))]

    embedding = np.zeros((512, hidden))
    embedding[:, :half] = 4.0           # the norm's size; the other half receives the attention's output
    put("token_embeddings.weight", embedding)
    normed = float(syn.bf16_to_float(syn.float_to_bf16(np.array([4 / np.sqrt(8 + 1e-6)], dtype=np.float32)))[0])
    wq = np.zeros((heads, 128, hidden))
    # Three values of a query that rotate by next to nothing (pairs of theta^-0.95 and less a token): coarse, fine, finest.
    wq[:, 63, 0], wq[:, 62, 0], wq[:, 61, 0] = 16.0, 1.0, 2.0 ** -8
    zeros = np.zeros((heads * 128, hidden))
    for layer in range(2):
        put(f"wq{layer}", wq.reshape(heads * 128, hidden))
        put(f"wk{layer}", zeros)
        put(f"wv{layer}", np.concatenate([zeros[:, :half], np.eye(half)], 1))
        put(f"wo{layer}", np.concatenate([np.zeros((half, half)), np.eye(half)], 0))
        put(f"w_gate{layer}", np.zeros((256, hidden)))
        put(f"w_down{layer}", np.zeros((hidden, 256)))
    model = package.Model(shape, tensors)

    def bf16(x):
        return syn.bf16_to_float(syn.float_to_bf16(np.asarray(x, dtype=np.float32))).astype(np.float64)

    unit = normed / np.sqrt(128.0) * np.log2(np.e)     # exponents of two per unit of key value 62
    k, v = np.zeros((history, heads, 128)), np.zeros((history, heads, 128))
    first, second = 10, 100
    k[[first, second], :, 63] = 30.0                   # 86 powers of two above the other tokens
    n = 2 + np.arange(heads) % 6
    wanted = (n + np.log2(1 + 0.9 * 2.0 ** -8)) / unit
    k[second, :, 62] = bf16(wanted)
    k[second, :, 61] = bf16((wanted - k[second, :, 62]) * 2.0 ** 8)
    gap = 2.0 ** ((k[second, :, 62] + k[second, :, 61] * 2.0 ** -8) * unit)
    v[[first, second]] = bf16(np.random.default_rng(7).standard_normal((2, heads, 128)))
    expected = (v[first] + gap[:, None] * v[second]) / (1 + gap[:, None])

    session = model.new_session(256)
    session.prefill([1] * history)
    flat = [syn.float_to_bf16(x.reshape(history, heads * 128).astype(np.float32)) for x in (k, v)]
    session.write_kv(0, 0, *flat)
    session.extend([1] * rows)
    got = syn.bf16_to_float(session.read_kv(1)[1])[history:].reshape(rows, heads, 128).astype(np.float64)
    got *= np.sqrt((16 * half + (expected ** 2).sum()) / hidden + 1e-6)
    share = (got * expected).sum(-1) / (expected ** 2).sum(-1)
    assert np.abs(share - 1).max() <= 1.9e-3, np.abs(share - 1).max(0)


def check_steady(c, weights, ids, got):
    """check_layered at the positions that the model's own conditioning allows it for: where the logits in 64 bits move by no more
    than 0.015 (half the limit) when every weight is changed by up to 2^-8, one rounding to BF16. (Position 221 of the case below
    moves by 0.054, and is 0.050 off with one row at a time as well as with any prompt kernel.) 19 in 20 do."""
    want = hybrid.HybridOracle(c, weights).forward(ids)
    rng = np.random.default_rng(0)
    moved = np.zeros(len(ids))
    for _ in range(3):
        other = {name: (w * (1 + rng.uniform(-1, 1, w.shape) * 2.0 ** -8)).astype(np.float32) for name, w in weights.items()}
        moved = np.maximum(moved, layered_cases.logit_error(hybrid.HybridOracle(c, other).forward(ids), want))
    steady = moved <= 0.015
    assert steady.mean() >= 0.9
    check_layered(got[steady], want[steady], "bf16")


@pytest.mark.parametrize("portions", [[192], [193], [64, 128], [64, 129], [2, 260]])
def test_layered_prompts_on_both_sides_of_the_shortest(cuda, package, portions):
    """Up to 192 tokens keys of 128 values have another kernel. 16 rows at a time behind that, which is a third."""
    c = layered_cases.config(64, 64, [layered_cases.parallel((4, 2, 128, 128, 32, 1e5), (1, 16, 16))])
    weights = layered_cases.random_weights(package, c, 8)
    model = package.Model(*package.checkpoint.admit(c, weights, "zofesun_bf16"))
    ids = layered_cases.tokens(c, sum(portions) + 10)
    check_steady(c, weights, ids, layered_cases.run_portions(model.new_session(320), ids, [*portions, 10]))


@pytest.mark.parametrize("portions", [[384], [385], [128, 256], [128, 257]])
def test_latent_prompts_on_both_sides_of_the_shortest(cuda, package, portions):
    c = gikepel_cases.config(64, 64, [gikepel_cases.latent(4, 128, 64, 128, 64)])
    weights = gikepel_cases.random_weights(package, c, 9)
    model = package.Model(*package.checkpoint.admit(c, weights, "gikepel_bf16"))
    ids = layered_cases.tokens(c, sum(portions) + 10)
    session = model.new_session(420)
    check_gikepel(layered_cases.run_portions(session, ids, [*portions, 10]), gikepel.GikepelOracle(c, weights).forward(ids), "bf16")


@pytest.mark.parametrize("scale", [-0.08, 0.0])
def test_scales_that_turn_or_lose_the_scores_order(cuda, package, scale):
    """Sizes that the tensor-core kernel takes, with scales that it does not: a row's largest score is not its largest exponent."""
    c = layered_cases.config(64, 64, [layered_cases.parallel((4, 2, 128, 128, 32, 1e5), (1, 16, 16))])
    c["layers"][0]["mixer"]["left"]["scale"] = scale
    weights = layered_cases.random_weights(package, c, 8)
    model = package.Model(*package.checkpoint.admit(c, weights, "zofesun_bf16"))
    ids = layered_cases.tokens(c, 270)
    check_steady(c, weights, ids, layered_cases.run_portions(model.new_session(280), ids, [210, 60]))


@pytest.mark.parametrize("rows", [40, 450])
def test_latent_attention_gives_up_with_its_copies_in_flight(cuda, package, rows):
    """As test_bounded_waits_gpu.py has it for uniform decoders: both prompt kernels, the tensor-core one with two query tiles."""
    c = gikepel_cases.config(64, 64, [gikepel_cases.latent(40, 128, 64, 128, 64)])
    weights = gikepel_cases.random_weights(package, c, 7)
    model = package.Model(*package.checkpoint.admit(c, weights, "gikepel_bf16"))
    ids = layered_cases.tokens(c, rows)
    session = model.new_session(460)
    want = session.extend(ids, [rows - 1]).copy()
    for _ in range(2):
        session.reset()
        session.inject_attention_wait_timeout(2000)
        with pytest.raises(RuntimeError, match="bounded wait"):
            session.extend(ids, [rows - 1])
        session.reset()
        assert np.array_equal(session.extend(ids, [rows - 1]), want)
