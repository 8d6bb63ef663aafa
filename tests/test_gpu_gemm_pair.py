"""Products large enough for the CTA-pair kernel (one split, at least 56 tiles of
256 x 256 and 1792 tile x K-block steps), at the edges of its tiles: one row or
column more than a tile and than half of one, so that a CTA of the pair lies
wholly outside; a single narrow column of tiles; odd widths, whose rows do not
start on 16 bytes; an output that does not; a K that ends inside a block; and
more tiles than the device has pairs, so both accumulators go around. Every
kernel accumulates over K in the same order, so each block of the product
equals the small product of its rows, bit for bit.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("M,N,K", [
    (1793, 2049, 2056), (2177, 2308, 1352), (4097, 4099, 456), (14336, 256, 2056), (14400, 100, 2056),
    (257, 14593, 2056), (5000, 5000, 328)])
def test_pair_products_match_their_blocks(M, N, K, shift):
    import torch
    from optimisation_solver_b200.mlp import gemm_bf16

    tiles = -(-M // 256) * -(-N // 256)
    assert tiles >= 56 and tiles * -(-K // 64) >= 1792
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N + K)
    a, b = (torch.randn((r, K), generator=gen, device="cuda").to(torch.bfloat16) for r in (M, N))
    room = torch.full((M * N + 8,), float("nan"), device="cuda")
    c = room[shift:shift + M * N].view(M, N)
    gemm_bf16(a, b, c)
    step = 640   # blocks of at most nine tiles: another kernel
    for i in range(0, M, step):
        for j in range(0, N, step):
            part = torch.empty((min(step, M - i), min(step, N - j)), device="cuda")
            gemm_bf16(a[i:i + step], b[j:j + step], part)
            assert torch.equal(c[i:i + step, j:j + step], part), (i, j)
    assert torch.isnan(room[:shift]).all() and torch.isnan(room[shift + M * N:]).all()
