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


def _ranged(be, cuda, shape, embed, norms, group=None):
    """A model whose embedding (the first 64 columns, or all) and norm weights there are multiplied before the re-layout."""
    heads, kv, hd, hidden, inter, kind = shape
    args = be.ModelArgs(model_type=kind, hidden_size=hidden, num_hidden_layers=2, intermediate_size=inter, num_attention_heads=heads,
                        num_key_value_heads=kv, head_dim=hd, rms_norm_eps=1e-6, vocab_size=520, tie_word_embeddings=False)
    m = be.Model.random_init(args, seed=4, device=cuda, gen_device="cpu")
    cols = slice(None) if group is None else slice(group, group + 1)
    m.embed.scales[:, cols].mul_(embed)
    m.embed.biases[:, cols].mul_(embed)
    for w in [lw[k] for lw in m.layers for k in ("input_norm", "post_norm")]:
        w.view(-1, 64)[cols].mul_(norms)
    return m.relayout()


@pytest.mark.parametrize("n,off", [(33, 0), (61, 700), (128, 64)])
@pytest.mark.parametrize("shape", SHAPES[1:], ids=lambda s: "x".join(map(str, s)))
def test_residual_times_norm_weight_beyond_fp16(be, cuda, shape, n, off):
    """A prompt's activations are normed in fp32: with a group of 64 residuals of 4e3 and more under norm weights of 8 some of
    their products do not fit fp16, what is normed (up to 8 sqrt(hidden)) does."""
    m = _ranged(be, cuda, shape, 2e5, 8.0, group=0)
    first, span = (t[:, 0].float().abs().max() for t in (m.embed.biases, m.embed.scales))      # (a nibble of 0 is the bias)
    assert first + 15 * span < 65504 and 8 * first > 65504
    tokens = torch.randint(0, 520, (n,), generator=torch.Generator().manual_seed(n))[None].to(cuda)
    got, want = (_run(be, m, tokens, off, False, large) for large in (True, False))
    m.prefill_large_m = True
    m.check_fused_error()
    for a, b in zip(got, want):
        assert torch.isfinite(a).all() and ((a - b).abs() <= 2.0 ** -6 * b.abs() + 1e-2).all()


@pytest.mark.parametrize("n,off", [(33, 0), (61, 700), (128, 64)])
def test_residual_times_norm_weight_below_fp16(be, cuda, n, off):
    """Residuals of 1.2e-3 under norm weights of 2^-12: their product, 3e-7, is five steps of fp16's smallest.  Normed it is 2e-4, which both
    paths round alike; keys and values, rms 1e-4 or more, are rounded to steps of 2^-24, a relative 3e-4 in the worst case."""
    m = _ranged(be, cuda, SHAPES[2], 1.0 / 16, 2.0 ** -12)
    tokens = torch.randint(0, 520, (n,), generator=torch.Generator().manual_seed(n))[None].to(cuda)
    got, want = (_run(be, m, tokens, off, False, large)[1][:, :, :, off:] for large in (True, False))
    m.prefill_large_m = True
    m.check_fused_error()
    for i in range(2):
        for j in range(2):
            a, b = got[i, j].double(), want[i, j].double()
            assert b.pow(2).mean().sqrt() > 1e-5 and (a - b).norm() <= 2.0 ** -8 * b.norm()


@pytest.mark.parametrize("tail", [1, 6, 32, 33])
def test_last_tokens_of_a_prompt_longer_than_a_pass(be, cuda, tail):
    """They are a pass of their own, through these kernels behind the rows of the large ones."""
    m = _model(be, cuda, *SHAPES[1])
    tokens = torch.randint(0, 520, (be.llama.PREFILL_ROWS + tail,), generator=torch.Generator().manual_seed(tail))[None].to(cuda)
    got, want = (_run(be, m, tokens, 0, False, large) for large in (True, False))
    m.prefill_large_m = True
    m.check_fused_error()
    for a, b in zip(got, want):
        assert ((a - b).abs() <= 2.0 ** -6 * b.abs() + 1e-2).all()
