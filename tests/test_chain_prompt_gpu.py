"""Short prompts of small models through the chain's kernels (tiles of 32 tokens side by side), at the edges of those tiles, on an empty
and a filled cache, all logits or the last, against the per-op kernels; and with a workspace that has no room for their scratch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [
    # heads, kv heads, head dim, hidden, intermediate, bias
    (2, 1, 64, 128, 128, "qwen2"),           # one chunk of K, one row tile
    (14, 2, 64, 896, 640, "qwen2"),          # clusters along K, groups of 7
    (8, 2, 128, 1024, 2816, "llama"),        # no bias, head dim 128
]


def _model(be, cuda, heads, kv, hd, hidden, inter, kind):
    args = be.ModelArgs(model_type=kind, hidden_size=hidden, num_hidden_layers=2, intermediate_size=inter, num_attention_heads=heads,
                        num_key_value_heads=kv, head_dim=hd, rms_norm_eps=1e-6, vocab_size=520, tie_word_embeddings=True)
    return be.Model.random_init(args, seed=4, device=cuda, gen_device="cpu").relayout()


def _run(be, m, tokens, off, last, large):
    m.prefill_large_m = m.fused = large
    cache = m.make_cache(64 * ((off + tokens.shape[1] + 63) // 64))
    cache.data[:, :, :, :off] = (0.3 * torch.randn(cache.data[:, :, :, :off].shape, generator=torch.Generator().manual_seed(off))).half().to(tokens.device)
    cache.offset = off
    logits = m(tokens, cache, logits_last_only=last)[0].float()
    assert cache.offset == off + tokens.shape[1]
    return logits, cache.data[:, :, :, :cache.offset].float()


@pytest.mark.parametrize("n,off,last", [(33, 0, False), (63, 700, True), (64, 31, False), (64, 1500, False), (65, 0, True), (97, 64, False), (128, 600, True)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_short_prompt_equals_per_op_kernels(be, cuda, shape, n, off, last):
    m = _model(be, cuda, *shape)
    tokens = torch.randint(0, 520, (n,), generator=torch.Generator().manual_seed(n))[None].to(cuda)
    got, want = (_run(be, m, tokens, off, last, large) for large in (True, False))
    m.prefill_large_m = True
    m.check_fused_error()
    for a, b in zip(got, want):                          # the bound of the chain's own test against the per-op kernels
        assert ((a - b).abs() <= 2.0 ** -6 * b.abs() + 1e-2).all()


def test_without_scratch_the_large_kernels_run(be, cuda):
    m = _model(be, cuda, *SHAPES[1])
    tokens = torch.randint(0, 520, (61,), generator=torch.Generator().manual_seed(1))[None].to(cuda)
    full = _run(be, m, tokens, 100, False, True)
    m._pf_buf["ws"] = torch.zeros(4096, dtype=torch.uint8, device=cuda)      # the tickets and the error word only
    small = _run(be, m, tokens, 100, False, True)
    m.check_fused_error()
    for a, b in zip(small, full):
        assert ((a - b).abs() <= 2.0 ** -6 * b.abs() + 1e-2).all()


@pytest.mark.parametrize("n,off", [(33, 700), (64, 448), (64, 1500)])
def test_attention_over_a_filled_cache_takes_nothing_from_scratch(be, cuda, n, off):
    """It starts while kernels two before it may still run, so mask and committed length come by value: the pass writes none of
    them (the scratch behind rotations and sums of squares stays as it was), and what the scratch held changes no bit."""
    m = _model(be, cuda, *SHAPES[1])
    hidden = m.args.hidden_size
    tokens = torch.randint(0, 520, (n,), generator=torch.Generator().manual_seed(n))[None].to(cuda)
    want = _run(be, m, tokens, off, False, True)
    used = 4096 + n * 64 * 8 + hidden // 32 * ((n + 31) // 32 * 32) * 4
    for fill in (0, 255, 1):
        m._pf_buf["ws"][4096:].fill_(fill)
        got = _run(be, m, tokens, off, False, True)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        m._pf_buf["ws"][4096:].fill_(fill)
        cache = m.make_cache(64 * ((off + n + 63) // 64))
        cache.offset = off
        assert m.can_prefill_large_m()
        m._prefill_large_m(tokens[0].int(), cache, off, None, 0)
        assert (m._pf_buf["ws"][used:] == fill).all()
    m.check_fused_error()
