"""A verify step's attention over chunks of one to five tiles, so that its ring of K and V buffers goes round, with a last tile of
every kind: one warp a block (three buffers, K's given back early) and several (four). Compared with the oracle's attention
under the operator tests' limits."""
import pytest

from test_operators_gpu import attention_case, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,heads,kv_heads", [(1, 4, 2), (4, 8, 2), (5, 8, 2), (16, 6, 2)])
@pytest.mark.parametrize("length", [4097, 8192, 8193, 12353, 16447])
def test_chunks_of_several_tiles(cuda, package, oracle, ctx, rows, heads, kv_heads, length):  # noqa: F811
    attention_case(cuda, package, oracle, ctx, rows, heads, kv_heads, length, device_offset=False, seed=length + rows)


@pytest.mark.parametrize("rows,heads,kv_heads", [(1, 8, 8), (16, 8, 8), (9, 16, 8), (16, 16, 8), (11, 4, 1), (10, 14, 2), (16, 14, 2)])
@pytest.mark.parametrize("length", [8192, 12353, 16447])
def test_rings_by_live_blocks(cuda, package, oracle, ctx, rows, heads, kv_heads, length):  # noqa: F811
    """One to seven warps a block; the first four have more live blocks than two an SM where the call knows the length, which gives
    them three or four buffers, and six where it does not. Chunks of two to five tiles. The bits are the same."""
    got = [attention_case(cuda, package, oracle, ctx, rows, heads, kv_heads, length, device_offset=unknown, seed=length + rows)
           for unknown in (False, True)]
    assert (got[0] == got[1]).all()


@pytest.mark.parametrize("rows", [4, 12])
@pytest.mark.parametrize("graph", [False, True])
def test_a_session_whose_history_grows_past_two_blocks_an_sm(cuda, package, rows, graph):
    """296 blocks of 8 KV heads and chunks of 128 tokens are 4736 tokens; the step's ring changes there and back."""
    syn = package.synthetic
    shape = package.Shape(vocab_size=512, n_layers=2, n_heads=16, n_kv_heads=8, hidden_size=256, intermediate_size=256,
                          max_position_embeddings=8192)
    model = package.Model(shape, syn.make_model(shape, seed=3))
    tokens = [int(t) for t in syn.make_prompt(5, rows, shape.vocab_size)]
    gen = cuda.Generator(device="cuda").manual_seed(4)
    k, v = (cuda.randn((8000, 1024), device="cuda", generator=gen).to(cuda.bfloat16) for _ in range(2))

    def session_at(length):
        session = model.new_session(8192, graph=graph)
        for layer in range(2):
            session.write_kv(layer, 0, k, v)
        session.adopt_history(length, tokens[0])
        return session

    def step(session, length):
        session.truncate(length)
        session.verify(tokens)
        return session.read_logits(rows).copy()

    wandering = session_at(8000)
    lengths = [3000, 4735, 7000, 3000, 7000]
    for layer in range(2):        # the step at 3000 replaces rows of the history
        wandering.write_kv(layer, 0, k, v)
    for length in lengths:
        got = step(wandering, length)
        for layer in range(2):
            wandering.write_kv(layer, 0, k, v)
        assert (got == step(session_at(length), length)).all(), length
