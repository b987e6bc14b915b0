"""Rotation, caches and value norms of a prompt's rows, one or four a warp: row counts of every remainder, and rotated halves that go by
fours, by twos and one by one. Compared with the restatement in double precision under the layered designs' limits."""
import sys
from pathlib import Path

import pytest

import layered_cases
from test_layered_gpu import check
from test_prompt_attention_gpu import check_steady

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import hybrid  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,rotated", [(32, 32), (24, 12), (20, 10)])
@pytest.mark.parametrize("rows", [33, 34, 35, 36])
def test_rows_of_every_remainder(cuda, package, dim, rotated, rows):
    c = layered_cases.config(64, 64, [layered_cases.parallel((4, 2, dim, 24, rotated, 1e4), (3, 16, 20))])
    weights = layered_cases.random_weights(package, c, 10)
    model = package.Model(*package.checkpoint.admit(c, weights, "zofesun_bf16"))
    ids = layered_cases.tokens(c, rows + 40)
    want = hybrid.HybridOracle(c, weights).forward(ids)
    check(layered_cases.run_portions(model.new_session(len(ids) + 4), ids, [rows, 40]), want, "bf16")


@pytest.mark.parametrize("dim,rotated,rows", [(32, 32, 947), (32, 32, 948), (24, 12, 949), (20, 10, 950), (32, 24, 951)])
def test_four_rows_a_warp(cuda, package, dim, rotated, rows):
    """20 units: one row a warp up to two waves of warps (18 944 on 148 multiprocessors: 947 rows), four beyond."""
    assert package.operators.prepare_execution_context(0).multiprocessors == 148
    c = layered_cases.config(64, 64, [layered_cases.parallel((4, 2, dim, 24, rotated, 1e4), (4, 16, 20))])
    weights = layered_cases.random_weights(package, c, 10)
    model = package.Model(*package.checkpoint.admit(c, weights, "zofesun_bf16"))
    ids = layered_cases.tokens(c, rows)
    check_steady(c, weights, ids, layered_cases.run_portions(model.new_session(rows + 4), ids, [rows]))
