"""Cache rows behind the last one a pass sees may hold anything (a cache that was rewound, memory that was never written): no bit of
the results depends on them, in tree passes and prompts, by the kernels for few and for many query rows, at the edges of a key block, with
room behind the last row and with the next head's rows there."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [
    # heads, kv heads, head dim
    (14, 2, 64),
    (8, 2, 128),
]


@pytest.mark.parametrize("n,cached", [(1, 0), (1, 62), (1, 64), (2, 1300), (3, 61), (31, 64), (32, 1999), (33, 0), (40, 600), (61, 66), (130, 0), (150, 43), (129, 700)])
@pytest.mark.parametrize("room", [0, 70])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_rows_behind_the_last_are_not_read(be, cuda, shape, room, n, cached):
    heads, kv, hd = shape
    args = be.ModelArgs(model_type="llama", hidden_size=256, num_hidden_layers=2, intermediate_size=128, num_attention_heads=heads,
                        num_key_value_heads=kv, head_dim=hd, rms_norm_eps=1e-6, vocab_size=264, tie_word_embeddings=True)
    m = be.Model.random_init(args, seed=3, device=cuda, gen_device="cpu").relayout()
    g = torch.Generator().manual_seed(n)
    tokens = torch.randint(0, 264, (1, n), generator=g).to(cuda)
    rows = (0.3 * torch.randn(2, 2, kv, cached, hd, generator=g)).half().to(cuda)

    def run(behind, fused=True):
        m.fused = fused
        cache = m.make_cache(max(64, cached + n + room))
        cache.data.fill_(behind)
        cache.data[:, :, :, :cached] = rows
        cache.offset = cached
        return m(tokens, cache).clone(), cache.data[:, :, :, :cached + n].clone()

    for fused in (True, False):
        want = run(0.0, fused)
        assert all(torch.isfinite(t).all() for t in want)
        for behind in (float("nan"), float("inf"), -65504.0):
            assert all(torch.equal(a, b) for a, b in zip(run(behind, fused), want))
    m.check_fused_error()


@pytest.mark.parametrize("count", [2, 4])
def test_requests_that_share_a_pass(be, cuda, count):
    m = be.Model.random_init(be.shape_preset("tiny-qwen2"), seed=3, device=cuda, gen_device="cpu").relayout()
    g = torch.Generator().manual_seed(count)
    M, lengths = 32 // count, [65, 7, 200, 126][:count]
    fwd = be.llama.FwdInputs(cuda)
    fwd.tokens.copy_(torch.randint(0, 1024, (32,), generator=g))
    fwd.pos.copy_(torch.cat([torch.arange(n, n + M) for n in lengths]))
    fwd.mask.copy_(torch.tensor([(2 << i) - 1 for i in range(M)]).repeat(count))
    fwd.prefix[:count].copy_(torch.tensor(lengths))
    old = (0.3 * torch.randn(1, 1, 1, 1, 200, 64, generator=g)).half().to(cuda)

    def run(behind):
        cache = m.make_batch_cache(256, count)
        cache.data.fill_(behind)
        for r, n in enumerate(lengths):
            cache.data[r, :, :, :, :n] = old[0, ..., :n, :]
        return m.forward_device(32, cache, 0, M, fwd, requests=count).clone()

    want = run(0.0)
    assert torch.isfinite(want).all()
    assert all(torch.equal(run(x), want) for x in (float("nan"), float("inf")))
    m.check_fused_error()
