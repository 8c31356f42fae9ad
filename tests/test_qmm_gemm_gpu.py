"""The large-M tensor-core matmul (b200_qmm_gemm, and b200_qmm beyond 32 rows) at the edges of its tiles, against the fp64
gold of the CPU oracle; prompt passes that cut the key range against the 32-row passes."""
import numpy as np
import pytest
import torch

from oracle import qmm_ref

pytestmark = pytest.mark.gpu


def _problem(n, k, m, seed):
    g = torch.Generator().manual_seed(seed)
    w = torch.randn(n, k, generator=g) * 0.02
    x = torch.randn(m, k, generator=g).half()
    return w, x, g


def _gold(x, packed):
    return qmm_ref.qmm_gold(x.numpy(), packed[0].numpy().view(np.uint32), packed[1].numpy(), packed[2].numpy())


# one token column, a tile less / more than full, ragged weight rows, one chunk, a K cut across CTAs, several token tiles
SHAPES = [(1, 8, 128), (16, 136, 128), (17, 256, 256), (33, 264, 384), (64, 896, 4864), (65, 128, 2048), (128, 1152, 896),
          (129, 72, 128), (257, 520, 640)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("epilogue", [0, 1, 2])
def test_gemm_epilogues_match_gold(be, cuda, m, n, k, epilogue):
    w, x, g = _problem(n, k, m, 10 * m + n + epilogue)
    packed = be.quantize.quantize(w)
    gold = _gold(x, packed)
    q = lambda t: torch.from_numpy(t).half().double().numpy()        # the epilogue's fp16 rounding points
    wt2 = bias = extra = None
    if epilogue == 0:
        bias = (torch.randn(n, generator=g) * 0.02).half()
        gold = gold + bias.double().numpy()
    elif epilogue == 1:
        extra = torch.randn(m, n, generator=g).half()
        gold = gold + extra.double().numpy()
    else:
        up = be.quantize.quantize(torch.randn(n, k, generator=g) * 0.02)
        wt2 = be.qmm_kernel.relayout(*(t.to(cuda) for t in up))
        a = q(gold)
        gold = q(a * q(1.0 / (1.0 + np.exp(-a)))) * q(_gold(x, up))
    wt = be.qmm_kernel.relayout(*(t.to(cuda) for t in packed))
    y = torch.full((m, n), 9.0, dtype=torch.float16, device=cuda)
    lib, p = be._lib.lib(), be._lib.ptr
    dev = lambda t: None if t is None else t.to(cuda)
    xd, bd, ed = dev(x), dev(bias), dev(extra)
    need = lib.b200_qmm_gemm_workspace_bytes(m, n, k, epilogue)
    for size in {4096, need}:                                        # without and with a cut of K
        ws = torch.zeros(size, dtype=torch.uint8, device=cuda)
        rc = lib.b200_qmm_gemm(p(xd), p(wt), p(wt2), p(bd), p(ed), p(y), m, n, k, epilogue, p(ws), size, be._lib.stream_ptr(cuda))
        assert rc == 0
        torch.cuda.synchronize()
        assert int(ws[:4096].view(torch.int32).abs().sum()) == 0     # tickets restored, no wait gave up
        err = np.abs(y.cpu().numpy().astype(np.float64) - gold)
        assert np.all(err <= 2.0 ** -9 * np.abs(gold) + 4e-3), f"max err {err.max()}"


@pytest.mark.parametrize("m,n,k", [(33, 8, 128), (40, 200, 384), (129, 520, 896), (200, 256, 2048)])
def test_operator_beyond_32_rows_matches_gold(be, cuda, m, n, k):
    w, x, g = _problem(n, k, m, m + n)
    packed = be.quantize.quantize(w)
    bias = (torch.randn(n, generator=g) * 0.02).half()
    args = [t.to(cuda) for t in packed]
    y = be.matmul(x.to(cuda), *args, 64, bias=bias.to(cuda))[0]
    gold = _gold(x, packed) + bias.double().numpy()
    assert np.all(np.abs(y.cpu().numpy().astype(np.float64) - gold) <= 2.0 ** -10 * np.abs(gold) + 2e-3)
    # scales at an odd 2-byte address: the same result through the 32-row kernel
    odd = torch.empty(packed[1].numel() + 1, dtype=torch.float16, device=cuda)[1:].view(packed[1].shape)
    odd.copy_(packed[1])
    y2 = be.matmul(x.to(cuda), args[0], odd, args[2], 64, bias=bias.to(cuda))[0]
    assert torch.allclose(y.float(), y2.float(), rtol=2.0 ** -9, atol=2e-3)


@pytest.mark.parametrize("name,cached,n", [("tiny-qwen2", 700, 33), ("tiny-llama", 1500, 100), ("tiny-llama", 0, 1100)])
def test_prompt_chunk_on_a_filled_cache_matches_the_32_row_passes(be, cuda, name, cached, n):
    """Key range cut across CTAs (few tokens, long cache), and more tokens than one pass takes."""
    m = be.Model.random_init(be.shape_preset(name), 5, cuda, gen_device="cpu").relayout()
    cache = m.make_cache(64 * ((cached + n + 127) // 64))
    g = torch.Generator().manual_seed(3)
    cache.data[:, :, :, :cached] = torch.randn(cache.data[:, :, :, :cached].shape, generator=g).half().to(cuda)
    tokens = torch.randint(0, m.args.vocab_size, (1, n), generator=g)
    cache.offset = cached
    got = m(tokens, cache)[0].float()
    kv = cache.data.clone()
    m.prefill_large_m = False
    cache.offset = cached
    want = m(tokens, cache)[0].float()
    m.check_fused_error()
    assert torch.all((got - want).abs() <= 2.0 ** -6 * want.abs() + 2e-2)
    assert torch.all((kv.float() - cache.data.float()).abs() <= 2.0 ** -6 * cache.data.float().abs() + 2e-2)
