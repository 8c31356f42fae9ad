"""Attention on the tensor memory (csrc/flash.cu) at the edges of its boxes, key blocks and clusters, in tree passes and prompt passes,
against the per-op kernels (mma.sync)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [
    # heads, kv heads, head dim
    (7, 1, 64),              # groups of 7: boxes of 63 rows
    (80, 1, 64),             # a group wider than a box
    (9, 3, 128),             # groups of 3, 63 rows of 64
    (16, 1, 128),            # groups of 16: four tokens a box
]


def _model(be, cuda, heads, kv, hd):
    args = be.ModelArgs(model_type="llama", hidden_size=256, num_hidden_layers=2, intermediate_size=128, num_attention_heads=heads,
                        num_key_value_heads=kv, head_dim=hd, rms_norm_eps=1e-6, vocab_size=264, tie_word_embeddings=True)
    if heads * hd % 128:
        args.num_attention_heads = heads = heads + 1 if kv == 1 else heads + kv
    return be.Model.random_init(args, seed=3, device=cuda, gen_device="cpu").relayout()


def _cache(m, cached, room, growing=False):
    cache = m.make_cache(64 * ((cached + room + 63) // 64))
    g = torch.Generator().manual_seed(cached)
    rows = 0.3 * torch.randn(cache.data[:, :, :, :cached].shape, generator=g)
    if growing and cached:                               # keys whose scores leave the maximum of the blocks before far behind
        rows[:, 0] *= torch.linspace(0.0, 60.0, cached)[:, None]
    cache.data[:, :, :, :cached] = rows.half().to(cache.data.device)
    cache.offset = cached
    return cache


def _close(pairs):
    for got, want in pairs:                              # the bound of the chain's own test against the per-op kernels
        assert ((got - want).abs() <= 2.0 ** -6 * want.abs() + 1e-2).all()


@pytest.mark.parametrize("rows,cached,split", [(3, 0, 0), (9, 64, 0), (10, 55, 0), (32, 600, 0), (32, 3000, 0), (17, 700, -1), (17, 700, 99)])
@pytest.mark.parametrize("growing", [False, True])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_tree_pass_equals_per_op_kernels(be, cuda, shape, rows, cached, split, growing):
    m = _model(be, cuda, *shape)
    m.attn_split_blocks = split
    g = torch.Generator().manual_seed(rows)
    tokens = torch.randint(0, 264, (rows,), generator=g)[None]
    tm = torch.eye(rows, dtype=torch.bool)
    for i in range(1, rows):
        tm[i] |= tm[int(torch.randint(0, i, (1,), generator=g))]
    out = []
    for fused in (True, False):
        m.fused = fused
        cache = _cache(m, cached, rows, growing)
        logits = be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, m, cache)[0].float()
        out.append((logits, cache.data[:, :, :, :cached + rows].float()))
    m.check_fused_error()
    _close(zip(*out))


@pytest.mark.parametrize("n,off", [(33, 0), (64, 64), (129, 1), (300, 77), (35, 3000), (500, 1000)])
@pytest.mark.parametrize("growing", [False, True])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_prompt_pass_equals_per_op_kernels(be, cuda, shape, n, off, growing):
    m = _model(be, cuda, *shape)
    tokens = torch.randint(0, 264, (n,), generator=torch.Generator().manual_seed(n))[None].to(cuda)
    out = []
    for large in (True, False):
        m.prefill_large_m = m.fused = large
        cache = _cache(m, off, n, growing)
        out.append((m(tokens, cache)[0].float(), cache.data[:, :, :, :off + n].float()))
    m.prefill_large_m = True
    m.check_fused_error()
    _close(zip(*out))


@pytest.mark.parametrize("cached", [40, 3000, 3070])
@pytest.mark.parametrize("rows", [10, 32])
def test_rows_of_the_pass_are_read_as_just_written(be, cuda, rows, cached):
    """K, V and queries come in by copies that the previous kernel's ordinary stores have to be fenced for, on a long cache behind the blocks
    asked for ahead.  A pass over rows that held another pass's, and the same again over its own: the same bits."""
    m = _model(be, cuda, *SHAPES[2])
    tm = torch.ones(rows, rows, dtype=torch.bool).tril()
    cache = _cache(m, cached, rows)
    g = torch.Generator().manual_seed(cached)

    def run(tokens):
        cache.offset = cached
        return be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, m, cache)[0].clone()

    for _ in range(100):
        tokens = torch.randint(0, 264, (rows,), generator=g)[None]
        assert torch.equal(run(tokens), run(tokens))
    m.check_fused_error()
