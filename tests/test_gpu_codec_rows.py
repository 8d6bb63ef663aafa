"""The codec between LP instances and the network over rows of every length
relative to a thread block (shorter than its narrowest, one less and one more
than its widths, several blocks long) and batches that end inside a block: the
formulas of the header against torch, and every row as that row alone gives it,
bit for bit.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,pad", [(1, 1, 5), (4, 3, 0), (20, 11, 0), (20, 12, 3), (100, 27, 0), (200, 54, 1),
                                     (200, 56, 0), (300, 212, 0), (700, 323, 0), (3000, 1100, 7)])
@pytest.mark.parametrize("batch", [1, 7, 33, 300])
def test_rows_match_formulas_and_themselves(n, m, pad, batch):
    import torch
    from optimisation_solver_b200 import native

    L = native.lib()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + m + batch)

    def rand(*shape, dtype=torch.float64):
        return torch.rand(shape, generator=gen, device="cuda", dtype=dtype)

    def p(t):
        return C.c_void_p(t.data_ptr())

    width = n + m + 1 + pad
    f32 = torch.float32
    x, y, w = rand(batch, n), rand(batch, m) - 0.5, rand(batch) + 0.5
    scale, mean, std = rand(n) + 0.5, rand(m, dtype=f32), rand(m, dtype=f32) + 0.5
    wmean, wstd = 0.25, 0.75

    def targets(rows):
        out = torch.full((len(rows), width), float("nan"), device="cuda")
        a, b, c = x[rows].contiguous(), y[rows].contiguous(), w[rows].contiguous()
        inv = 1.0 / std
        assert L.pdlpgpu_encode_targets(p(a), p(b), p(c), len(rows), n, m, width, p(scale), p(mean), p(inv),
                                        C.c_float(wmean), C.c_float(1.0 / wstd), p(out)) == 0
        torch.cuda.synchronize()
        return out

    def decoded(rows):
        a = net[rows].contiguous()
        out = [torch.full((len(rows), k), float("nan"), device="cuda", dtype=torch.float64) for k in (n, m, 1)]
        assert L.pdlpgpu_decode_warmstart(p(a), len(rows), n, m, width, p(scale), p(mean), p(std), C.c_float(wmean),
                                          C.c_float(wstd), *[p(t) for t in out]) == 0
        torch.cuda.synchronize()
        return torch.cat(out, dim=1)

    def features(rows):
        a = x[rows].contiguous()
        out = torch.full((len(rows), n + pad), float("nan"), device="cuda").to(torch.bfloat16)
        assert L.pdlpgpu_encode_features(p(a), len(rows), n, n + pad, p(fmean), p(finv), p(out)) == 0
        torch.cuda.synchronize()
        return out.float()

    net = rand(batch, width, dtype=f32) * 1.5 - 0.25
    fmean, finv = rand(n, dtype=f32), rand(n, dtype=f32) + 0.5
    every = list(range(batch))
    want = {
        targets: torch.cat([(x / scale).float(), (y.float() - mean) / std, ((w.float().log() - wmean) / wstd)[:, None],
                            torch.zeros((batch, pad), device="cuda")], dim=1),
        decoded: torch.cat([net[:, :n].clamp(0, 1).double() * scale, (net[:, n:n + m] * std + mean).double(),
                            (net[:, n + m:n + m + 1] * wstd + wmean).exp().double()], dim=1),
        features: torch.cat([((x.float() - fmean) * finv).to(torch.bfloat16).float(),
                             torch.zeros((batch, pad), device="cuda")], dim=1),
    }
    for call, reference in want.items():
        got = call(every)
        # A few FP32 roundings of values of order one.
        assert torch.allclose(got.double(), reference.double(), rtol=2e-6, atol=2e-6), call.__name__
        for r in {0, batch // 2, batch - 1}:
            assert torch.equal(got[r], call([r])[0]), (call.__name__, r)
