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


@pytest.mark.parametrize("heads,kv_heads,rows", [(40, 40, 300), (32, 8, 610), (32, 8, 600), (56, 8, 400)])
def test_blocks_of_two_query_tiles(cuda, package, heads, kv_heads, rows):
    """More blocks than half the multiprocessors; the last block's second query tile has 44, 8, 0 and 112 rows."""
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
