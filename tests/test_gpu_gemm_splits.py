"""Products with K splits, on every path they take: partials in scratch (a CTA
for every split of every tile, in one wave with six stages and in several with
three), each tile's splits in turn in one CTA (too many partials, or too few
splits for the waves), and the second when another thread holds the scratch.

The contract is the sum of the splits' products in split order, each product
accumulated over K in order, so the result equals the FP32 sum of one-split
products of the K ranges bit for bit, whatever the path. Sizes: less than a
tile, the edges of tiles, rows that end off a 16-byte boundary, an output that
starts off one, a last split shorter than the others, more splits than
accumulators and than K blocks.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _operands(M, N, K, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return [torch.randn((r, K), generator=gen, device="cuda").to(torch.bfloat16) for r in (M, N)]


def _in_order(a, b, splits):
    """The splits' products by one-split calls, added in FP32."""
    import torch
    from optimisation_solver_b200.mlp import gemm_bf16
    M, K = a.shape
    N = b.shape[0]
    blocks = (K + 63) // 64
    per = -(-blocks // max(1, min(splits, blocks))) * 64
    total = torch.zeros((M, N), device="cuda")
    part = torch.empty((M, N), device="cuda")
    for k in range(0, K, per):
        gemm_bf16(a[:, k:k + per].contiguous(), b[:, k:k + per].contiguous(), part, 1)
        total += part
    return total


SHAPES = [
    (1, 1, 640, 3), (100, 100, 1000, 3), (129, 130, 1032, 40), (4, 129, 2056, 5), (64, 200, 4104, 8), (128, 128, 6400, 100),
    (256, 512, 22000, 18),                     # 144 CTAs: one wave, six stages
    (600, 600, 2000, 8), (1000, 1544, 1032, 3),   # more than a wave of them: three stages
    (1537, 1029, 1544, 3), (640, 1023, 2056, 16),
    (1000, 1544, 2568, 4), (896, 2688, 520, 2),   # too few splits for the waves
    (1664, 2570, 712, 5), (1500, 1500, 2056, 17),   # more partials than the scratch holds
]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("M,N,K,splits", SHAPES)
def test_splits_are_added_in_order(M, N, K, splits, shift):
    import torch
    from optimisation_solver_b200.mlp import gemm_bf16

    a, b = _operands(M, N, K, M + N + K + splits)
    room = torch.full((M * N + 8,), float("nan"), device="cuda")
    c = room[shift:shift + M * N].view(M, N)
    gemm_bf16(a, b, c, splits)
    assert torch.equal(c, _in_order(a, b, splits))
    assert torch.isnan(room[:shift]).all() and torch.isnan(room[shift + M * N:]).all()
    # And it is the product, to the tolerance of test_gpu_mlp.py.
    want = a.double() @ b.double().T
    bound = 1e-5 * (a.double().abs() @ b.double().abs().T).max()
    assert (c.double() - want).abs().max() <= bound


def test_calls_on_threads_share_the_scratch():
    import torch
    from optimisation_solver_b200.mlp import gemm_bf16

    shapes = [(256, 512, 4096, 16), (300, 500, 3072, 8), (129, 257, 5000, 12), (512, 512, 1024, 8)]
    operands = [_operands(M, N, K, M + K) for M, N, K, _ in shapes]
    want = [_in_order(a, b, s[3]) for (a, b), s in zip(operands, shapes)]
    torch.cuda.synchronize()
    wrong = []
    start = threading.Barrier(len(shapes))

    def work(k):
        a, b = operands[k]
        c = torch.empty_like(want[k])
        start.wait(timeout=60)
        for _ in range(100):
            c.fill_(float("nan"))
            gemm_bf16(a, b, c, shapes[k][3])
            if not torch.equal(c, want[k]):
                wrong.append(shapes[k])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, np.unique(wrong, axis=0)
