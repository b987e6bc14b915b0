"""The prompt GEMM where its tiles end, against a product in 64 bits of the same BF16 operands: blocks of one tile over token
counts around the column steps of 16 and the 256 columns of a tile, feature tails, the shortest K and K that no ring divides;
and blocks of two feature or two token tiles (two issuing warps) with every depth of the rings that such blocks get.

Bound: the result is rounded once to BF16 (8 significant bits: half an ulp is at most 2^-8 of the value), the products of
two BF16 numbers are exact in FP32 and the FP32 sum of K of them carries at most K 2^-23 of the sum of their magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [33, 47, 48, 49, 111, 161, 255, 257, 320, 511, 513, 1025]


def compare(torch, out, x, w, bias=None):
    x64, w64 = x.double(), w.double()
    ref = x64 @ w64.T + (0 if bias is None else bias.double())
    bound = ref.abs() * 2.0 ** -8 + (x64.abs() @ w64.abs().T) * (x.shape[1] * 2.0 ** -23) + 1e-30
    worst = ((out.double() - ref).abs() / bound).max().item()
    assert worst <= 1.0, worst


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("nk", [(272, 64), (1040, 448), (3072, 1024)])
def test_dense_tiles(cuda, package, rows, nk):
    torch, ops = cuda, package.operators
    n, k = nk
    gen = torch.Generator(device="cuda").manual_seed(rows * 31 + n)
    x = torch.randn((rows, k), device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.randn((n, k), device="cuda", generator=gen) * 0.05).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda", generator=gen).to(torch.bfloat16)
    ctx = ops.prepare_execution_context(0)
    scratch = torch.empty(ops.linear_scratch_bytes(rows, k, n), dtype=torch.uint8, device="cuda")
    for room in (None, scratch):   # with scratch K may be split over blocks
        guard = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.linear(ctx, x, ops.prepare_dense(w.t(), bias), guard[:rows], room)
        torch.cuda.synchronize()
        compare(torch, guard[:rows], x, w, bias)
        assert (guard[rows] == 7.0).all()


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("nk", [(144, 128), (1040, 896), (2048, 2304)])
def test_awq_tiles(cuda, package, rows, nk):
    torch, ops, syn = cuda, package.operators, package.synthetic
    n, k = nk
    q, s, z = syn.awq_triple(5, f"tiles{n}x{k}", n, k)
    w = torch.from_numpy(np.ascontiguousarray(syn.awq_dequantize(q, s, z, k))).cuda().to(torch.bfloat16)
    gen = torch.Generator(device="cuda").manual_seed(rows * 17 + n)
    x = torch.randn((rows, k), device="cuda", generator=gen).to(torch.bfloat16)
    dq, dz = torch.from_numpy(q).cuda(), torch.from_numpy(z).cuda()   # the prepared weight borrows them
    ds = torch.from_numpy(s.view(np.int16)).cuda().view(torch.bfloat16)
    weight = ops.prepare_awq(dq, ds, dz, 128, k, None)
    ctx = ops.prepare_execution_context(0)
    scratch = torch.empty(ops.linear_scratch_bytes(rows, k, n), dtype=torch.uint8, device="cuda")
    for room in (None, scratch):
        guard = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
        ops.awq_linear(ctx, x, weight, guard[:rows], room)
        torch.cuda.synchronize()
        compare(torch, guard[:rows], x, w)
        assert (guard[rows] == 7.0).all()


# awq, rows, features, inputs, K slices that the scratch has room for -> feature tiles, token tiles, columns, stages of
# activations, weight operands and packed weights, K slices (tests/test_prompt_choice_cpu.py holds the shapes to it; int4 is
# launched with deeper rings where its operands stand in tensor memory: tests/test_prompt_launched_cpu.py). 896 inputs
# are 14 K blocks, which no ring here divides evenly into whole rounds of 3, 4 or 5; every count of rows leaves the last token
# tile ragged, and every width the last feature tile.
BLOCKS = [
    (0, 970, 6256, 896, 0, (1, 2, 176, 3, 3, 0, 1)),
    (0, 1341, 3136, 896, 0, (1, 2, 144, 4, 4, 0, 1)),
    (0, 2083, 2096, 896, 0, (1, 2, 144, 4, 4, 0, 1)),    # the last group of tokens has one tile
    (0, 390, 13520, 896, 0, (2, 1, 208, 3, 3, 0, 1)),
    (0, 194, 19728, 896, 0, (2, 1, 208, 3, 3, 0, 1)),    # the last block of features has one tile
    (0, 103, 19728, 896, 0, (2, 1, 112, 4, 4, 0, 1)),
    (0, 229, 10416, 896, 0, (2, 1, 80, 5, 5, 0, 1)),
    (0, 258, 5216, 6144, 4, (1, 2, 144, 4, 4, 0, 3)),
    (0, 150, 10416, 6144, 4, (2, 1, 160, 4, 4, 0, 3)),
    (1, 453, 13520, 896, 0, (1, 2, 240, 3, 2, 2, 1)),
    (1, 439, 10416, 896, 0, (1, 2, 224, 3, 2, 4, 1)),
    (1, 390, 10416, 896, 0, (1, 2, 208, 3, 3, 3, 1)),
    (1, 292, 10416, 896, 0, (1, 2, 160, 3, 3, 6, 1)),
    (1, 2030, 5216, 896, 0, (1, 2, 160, 3, 3, 6, 1)),    # the last group of tokens has one tile
    (1, 257, 10416, 896, 0, (1, 2, 144, 4, 4, 4, 1)),
    (1, 258, 5216, 6144, 4, (1, 2, 144, 4, 4, 4, 3)),
]


@pytest.mark.parametrize("awq,rows,n,k,slices,block", BLOCKS)
def test_blocks_of_two_tiles(cuda, package, awq, rows, n, k, slices, block):
    torch, ops, syn = cuda, package.operators, package.synthetic
    gen = torch.Generator(device="cuda").manual_seed(rows + n)
    x = torch.randn((rows, k), device="cuda", generator=gen).to(torch.bfloat16)
    ctx = ops.prepare_execution_context(0)
    assert ctx.multiprocessors == 148    # what the blocks above were chosen for
    room = torch.empty(slices * rows * n, dtype=torch.float32, device="cuda") if slices else None
    guard = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    if awq:
        q, s, z = syn.awq_triple(5, f"blocks{n}x{k}", n, k)
        w = torch.from_numpy(np.ascontiguousarray(syn.awq_dequantize(q, s, z, k))).cuda().to(torch.bfloat16)
        held = (torch.from_numpy(q).cuda(), torch.from_numpy(s.view(np.int16)).cuda().view(torch.bfloat16), torch.from_numpy(z).cuda())
        bias = torch.randn(n, device="cuda", generator=gen).to(torch.bfloat16)
        ops.awq_linear(ctx, x, ops.prepare_awq(*held, 128, k, bias), guard[:rows], room)
    else:
        w = (torch.randn((n, k), device="cuda", generator=gen) * 0.05).to(torch.bfloat16)
        bias = torch.randn(n, device="cuda", generator=gen).to(torch.bfloat16)
        ops.linear(ctx, x, ops.prepare_dense(w.t(), bias), guard[:rows], room)
    torch.cuda.synchronize()
    compare(torch, guard[:rows], x, w, bias)
    assert (guard[rows] == 7.0).all()
