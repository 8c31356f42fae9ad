"""The matmul of CTA pairs (csrc/qmm_pair.cu: more than 128 rows, long K) at the edges of its tiles, against the fp64 gold of the CPU
oracle.  The shapes are ones for which it is the cheaper of the two large-M kernels, with and without room to cut K."""
import numpy as np
import pytest
import torch

from oracle import qmm_ref

pytestmark = pytest.mark.gpu


def _gold(x, packed):
    return qmm_ref.qmm_gold(x.numpy(), packed[0].numpy().view(np.uint32), packed[1].numpy(), packed[2].numpy())


def _check(y, gold, roundings=2):
    # as for the other large-M kernel: every fp16 rounding on the way may go the other way, 2^-10 of the value each (two: the product, and
    # what is added to it; five: gate, up, sigmoid and the two products of SiLU(gate) * up), fp32 sums of up to 18944 products
    err = np.abs(y.cpu().numpy().astype(np.float64) - gold)
    assert np.all(err <= roundings * 2.0 ** -10 * np.abs(gold) + 4e-3), f"max err {err.max()}"


# rows one beyond a tile, tiles of 128 to 224 tokens, ragged weight rows (a last 64-row block of 8, a pair without rows for its odd CTA)
@pytest.mark.parametrize("m,n,k,epilogue", [(129, 1000, 18944, 2), (300, 264, 18944, 2), (400, 136, 18944, 2), (300, 1000, 18944, 0),
                                            (200, 2056, 18944, 1), (257, 2056, 8192, 0), (513, 2056, 640, 2), (513, 2056, 2048, 1)])
def test_pair_epilogues_match_gold(be, cuda, m, n, k, epilogue):
    g = torch.Generator().manual_seed(m + n + epilogue)
    packed = be.quantize.quantize(torch.randn(n, k, generator=g) * 0.02)
    x = torch.randn(m, k, generator=g).half()
    gold = _gold(x, packed)
    q = lambda t: torch.from_numpy(t).half().double().numpy()        # the epilogue's fp16 rounding points
    wt2 = bias = extra = None
    if epilogue == 0:
        bias = (torch.randn(n, generator=g) * 0.02).half().to(cuda)
        gold = gold + bias.double().cpu().numpy()
    elif epilogue == 1:
        extra = torch.randn(m, n, generator=g).half().to(cuda)
        gold = gold + extra.double().cpu().numpy()
    else:
        up = be.quantize.quantize(torch.randn(n, k, generator=g) * 0.02)
        wt2 = be.qmm_kernel.relayout(*(t.to(cuda) for t in up))
        a = q(gold)
        gold = q(a * q(1.0 / (1.0 + np.exp(-a)))) * q(_gold(x, up))
    wt = be.qmm_kernel.relayout(*(t.to(cuda) for t in packed))
    xd = x.to(cuda)
    y = torch.full((m, n), 9.0, dtype=torch.float16, device=cuda)
    lib, p = be._lib.lib(), be._lib.ptr
    for size in sorted({4096, lib.b200_qmm_gemm_workspace_bytes(m, n, k, epilogue)}):       # without and with a cut of K
        ws = torch.zeros(size, dtype=torch.uint8, device=cuda)
        for _ in range(2):
            rc = lib.b200_qmm_gemm(p(xd), p(wt), p(wt2), p(bias), p(extra), p(y), m, n, k, epilogue, p(ws), size, be._lib.stream_ptr(cuda))
            assert rc == 0
        torch.cuda.synchronize()
        assert int(ws[:4096].view(torch.int32).abs().sum()) == 0     # tickets restored, no wait gave up
        _check(y, gold, 5 if epilogue == 2 else 2)


# scales in boxes (K a multiple of 512), by loads of two, by loads of one (an odd storage offset); bias or none
@pytest.mark.parametrize("m,n,k,shift,with_bias", [(203, 2056, 18944, 0, True), (300, 2056, 18816, 0, False), (257, 2056, 18944, 1, True)])
def test_pair_on_quantised_weights_matches_gold(be, cuda, m, n, k, shift, with_bias):
    g = torch.Generator().manual_seed(m + k)
    w, s, b = be.quantize.quantize(torch.randn(n, k, generator=g) * 0.02)
    x = torch.randn(m, k, generator=g).half()
    bias = (torch.randn(n, generator=g) * 0.02).half() if with_bias else None

    def moved(t):
        store = torch.zeros(t.numel() + 8, dtype=t.dtype, device=cuda)
        view = store[shift:shift + t.numel()].view(t.shape)
        view.copy_(t)
        return view

    gold = _gold(x, (w, s, b)) + (0 if bias is None else bias.double().numpy())
    y = be.matmul(x.to(cuda), w.to(cuda), moved(s), moved(b), 64, bias=None if bias is None else bias.to(cuda))[0]
    _check(y, gold)
