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
