"""The BF16 weight-streaming kernel at every width of its phases (one, two or four tiles side by side) and under the
shared-memory limits that a caller's context may set, against a product in 64 bits of the same BF16 operands.

Bound: the result is rounded once to BF16 (half an ulp is at most 2^-8 of the value), the products of two BF16 numbers are
exact in FP32 and the FP32 sum of K of them carries at most K 2^-23 of the sum of their magnitudes.

The gated and the argmax epilogues are reached through sessions: the logits of a verify step within the bound that
test_session_gpu.py gives for the staged oracle, the greedy tokens exactly those of the logits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 8 * (148 * 5 + 3)   # five or six tiles a block: no multiple of two or four


@pytest.mark.parametrize("limit_kb", [None, 26, 32, 48, 64, 80, 112])
@pytest.mark.parametrize("k", [256, 512, 768, 1024, 1280, 2048, 2304, 4096, 4352])
def test_linear_under_shared_memory_limits(cuda, package, k, limit_kb):
    torch, ops = cuda, package.operators
    gen = torch.Generator(device="cuda").manual_seed(k)
    w = (torch.randn((N, k), device="cuda", generator=gen) * 0.05).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=gen).to(torch.bfloat16)
    ctx = ops.prepare_execution_context(0)
    if limit_kb is not None:
        ctx.shared_memory_limit = ctypes.c_size_t(limit_kb * 1024)
    for rows in (1, 8, 9, 16):
        x = torch.randn((rows, k), device="cuda", generator=gen).to(torch.bfloat16)
        scratch = torch.empty(ops.linear_scratch_bytes(rows, k, N), dtype=torch.uint8, device="cuda")
        guard = torch.full((rows + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.linear(ctx, x, ops.prepare_dense(w.t(), bias), guard[:rows], scratch)
        torch.cuda.synchronize()
        x64, w64 = x.double(), w.double()
        ref = x64 @ w64.T + bias.double()
        bound = ref.abs() * 2.0 ** -8 + (x64.abs() @ w64.abs().T) * (k * 2.0 ** -23) + 1e-30
        worst = ((guard[:rows].double() - ref).abs() / bound).max().item()
        assert worst <= 1.0, (rows, worst)
        assert (guard[rows] == 7.0).all()


@pytest.mark.parametrize("rows", [1, 5, 12])
@pytest.mark.parametrize("hidden,ffn,vocab", [(512, 3328, 5944), (1024, 2816, 8 * 148 * 3 + 8), (1280, 3840, 5936),
                                              (2048, 2560, 8 * 149), (2304, 1536, 5944)])
def test_gated_and_argmax_epilogues(cuda, package, oracle, hidden, ffn, vocab, rows):
    """Two layers whose gate|up projection (pairs of tiles) and vocabulary head give the blocks odd and even numbers of
    tiles, in phases of four (up to 1024 inputs), two (up to 2048) and one."""
    syn = package.synthetic
    shape = package.Shape(vocab_size=vocab, n_layers=2, n_heads=4, n_kv_heads=2, hidden_size=hidden, intermediate_size=ffn,
                          max_position_embeddings=256)
    tensors = syn.make_model(shape, seed=rows + hidden, vary_norms=True)
    session = package.Model(shape, tensors).new_session(256, graph=True)
    reference = oracle.OracleModel(shape, tensors, capacity=256)
    prompt = syn.make_prompt(hidden, 21, vocab)
    session.prefill(prompt)
    reference.forward(prompt, 1)
    tokens = syn.make_prompt(hidden + 1, rows, vocab)
    out = session.verify(tokens)
    got = syn.bf16_to_float(session.read_logits(rows))
    expected = reference.forward(tokens, 1)
    assert np.abs(got - expected).max() <= 1.5e-2 * np.sqrt(2) * np.abs(expected).max()
    assert list(out.targets) == [int(t) for t in oracle.argmax(got)]
