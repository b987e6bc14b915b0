"""Bounded waits that run out in the weight-streaming kernels after they have gone round their rings (no fault, trap or
endless loop: the first weight copy's barrier is told to expect 16 bytes more than the copy delivers, with a short poll
limit). 128 heads of queries, keys and values are 2048 tiles of eight features, 13 or 14 a block: more than the ring of twelve
holds, so there is a tile left to refill the failed tile's place with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quant", [0, 1])
def test_a_ring_that_gave_up_is_not_refilled(cuda, package, quant):
    syn = package.synthetic
    shape = package.Shape(vocab_size=512, n_layers=1, n_heads=112, n_kv_heads=8, hidden_size=256, intermediate_size=512,
                          quant_type=quant, max_position_embeddings=256)
    model = package.Model(shape, syn.make_model(shape, seed=3))
    session, sibling = model.new_session(64), model.new_session(64)
    sibling.prefill([4, 5, 6])
    session.prefill([1, 2, 3])
    expected = session.read_logits(1).copy()
    first = session.verify([7, 8, 9])
    session.truncate(3)
    for _ in range(3):
        session.inject_wait_timeout(2000)
        with pytest.raises(RuntimeError, match="bounded wait"):
            session.verify([7, 8, 9])
        assert session.context_size() == 0
        session.prefill([1, 2, 3])
        assert np.array_equal(session.read_logits(1), expected)
        again = session.verify([7, 8, 9])
        assert again.targets == first.targets and again.emitted == first.emitted
        session.truncate(3)
    assert sibling.verify([7, 8]).emitted >= 1


@pytest.mark.parametrize("quant", [0, 1])
def test_prompt_gemm_waits_once_for_what_is_in_flight(cuda, package, quant):
    """After a wait has run out in the prompt GEMM its copies in flight are waited for on barriers that complete with their
    bytes: the failing call takes about one poll limit. Barriers that also need the roles that have left would let the limit
    run out once more per stage, four to eight times. The attention kernel's failing wait, which ends after one limit, gives
    the time of a limit."""
    import time
    syn = package.synthetic
    shape = package.Shape(vocab_size=512, n_layers=1, n_heads=16, n_kv_heads=8, hidden_size=2048, intermediate_size=2048,
                          quant_type=quant, max_position_embeddings=256)
    model = package.Model(shape, syn.make_model(shape, seed=5))
    session = model.new_session(256)
    prompt = syn.make_prompt(3, 200, shape.vocab_size)
    session.prefill(prompt)
    expected = session.read_logits(1).copy()
    polls = 1 << 17

    def failing(arm, call):
        session.prefill(prompt)
        arm(polls)
        begin = time.perf_counter()
        with pytest.raises(RuntimeError, match="bounded wait"):
            call()
        return time.perf_counter() - begin

    limit = failing(session.inject_attention_wait_timeout, lambda: session.verify([7, 8, 9]))
    taken = failing(session.inject_wait_timeout, lambda: session.prefill(prompt))
    assert limit > 0.02
    assert taken < 2.5 * limit, (taken, limit)
    session.prefill(prompt)
    assert np.array_equal(session.read_logits(1), expected)


@pytest.mark.parametrize("heads,kv_heads,rows", [(8, 8, 100), (40, 40, 300), (60, 20, 300)])
def test_prompt_attention_gives_up_with_its_copies_in_flight(cuda, package, heads, kv_heads, rows):
    """The first copy of keys of every block is told to bring 16 bytes more than it does. Blocks of one query tile; of two, whose
    softmax warps take turns; of two whose queries are loaded instead of copied (groups of three). Afterwards the session and the
    same prompt are as before."""
    syn = package.synthetic
    shape = package.Shape(vocab_size=512, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, hidden_size=256, intermediate_size=256,
                          max_position_embeddings=512)
    model = package.Model(shape, syn.make_model(shape, seed=7))
    session = model.new_session(512)
    prompt = syn.make_prompt(4, rows, shape.vocab_size)
    session.prefill(prompt)
    expected = session.read_logits(1).copy()
    for _ in range(2):
        session.inject_attention_wait_timeout(2000)
        with pytest.raises(RuntimeError, match="bounded wait"):
            session.prefill(prompt)
        session.prefill(prompt)
        assert np.array_equal(session.read_logits(1), expected)
    assert session.verify([7, 8]).emitted >= 1   # the hook was the prompt's, not the next step's
