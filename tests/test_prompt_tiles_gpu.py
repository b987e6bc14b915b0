"""The prompt GEMM where its tiles end: token counts around the column steps of 16 and the 256 columns of a tile, feature
tails, the shortest K and K that no ring divides, against a product in 64 bits of the same BF16 operands.

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
