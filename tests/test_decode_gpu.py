"""The kernel chain of a pass of up to 32 tokens (csrc/decode.cu) at the edges of its tiles, key blocks and clusters, against the
per-op kernels; and the inputs of a pass from a caller's tensors."""
import ctypes
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [
    # heads, kv heads, head dim, hidden, intermediate, vocab
    (2, 1, 64, 128, 128, 1032),          # one chunk of K, a last row tile of 8 rows
    (14, 2, 64, 896, 640, 520),          # groups of 7 heads, seven chunks
    (16, 2, 128, 2048, 2176, 2048),      # groups of 8 heads of 128: up to 256 query rows per kv head
]


def _model(be, cuda, heads, kv, hd, hidden, inter, vocab):
    args = be.ModelArgs(model_type="qwen2", hidden_size=hidden, num_hidden_layers=2, intermediate_size=inter, num_attention_heads=heads,
                        num_key_value_heads=kv, rms_norm_eps=1e-6, vocab_size=vocab, tie_word_embeddings=True)
    assert args.head_dim == hd
    return be.Model.random_init(args, seed=3, device=cuda, gen_device="cpu").relayout()


def _cache(m, cached, seed):
    cache = m.make_cache(64 * ((cached + 32 + 63) // 64))
    g = torch.Generator().manual_seed(seed)
    cache.data[:, :, :, :cached] = (0.3 * torch.randn(cache.data[:, :, :, :cached].shape, generator=g)).half().to(cache.data.device)
    cache.offset = cached
    return cache


def _tree(rows, rng):
    tm = np.eye(rows, dtype=bool)
    for i in range(1, rows):
        tm[i] |= tm[int(rng.integers(0, i))]
    return tm


@pytest.mark.parametrize("rows,cached", [(1, 0), (1, 63), (2, 64), (16, 31), (16, 447), (17, 448), (31, 600), (32, 1500)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_chain_equals_per_op_kernels(be, cuda, shape, rows, cached):
    m = _model(be, cuda, *shape)
    rng = np.random.default_rng(rows + cached)
    tokens = torch.from_numpy(rng.integers(0, shape[-1], rows))[None]
    tm = torch.from_numpy(_tree(rows, rng))
    out = []
    for fused in (True, False):
        m.fused = fused
        assert m.can_fuse() == fused
        cache = _cache(m, cached, 1)
        logits = be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, m, cache)[0].float()
        out.append((logits, cache.data[:, :, :, :cached + rows].float()))
    m.check_fused_error()
    for got, want in zip(*out):
        assert ((got - want).abs() <= 2.0 ** -6 * want.abs() + 1e-2).all()


@pytest.mark.parametrize("rows,cached", [(1, 5), (7, 0), (32, 90)])
def test_pass_inputs_whatever_their_form(be, cuda, rows, cached):
    m = _model(be, cuda, *SHAPES[1])
    rng = np.random.default_rng(rows)
    tokens = torch.from_numpy(rng.integers(0, SHAPES[1][-1], rows))[None]
    tm = torch.from_numpy(_tree(rows, rng))
    pos = tm.sum(1) - 1
    additive = torch.where(tm, 0.0, float("-inf"))
    full = torch.cat([torch.zeros(rows, cached), additive], dim=-1)[None, None]
    cache = _cache(m, cached, 2)
    outs = []
    for call in (lambda c: be.eagle.tree_decoding(tokens, tm, pos, m, c),
                 lambda c: be.eagle.tree_decoding(tokens.to(cuda, torch.int32), additive.half().to(cuda), pos.to(cuda, torch.int32), m, c),
                 lambda c: m(tokens, c, mask=full, position_ids=pos + cached)):
        cache.offset = cached
        outs.append(call(cache))
        assert cache.offset == cached + rows
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    cache.offset = cached
    every = m(tokens, cache)
    cache.offset = cached
    last = m(tokens.to(cuda), cache, logits_last_only=True)
    cache.offset = cached
    explicit = m(tokens, cache, position_ids=cached + torch.arange(rows))
    assert last.shape == (1, 1, SHAPES[1][-1]) and torch.equal(last, every[:, -1:]) and torch.equal(explicit, every)


def test_layer_pointers_from_the_device_table(be, cuda):
    """Without a host copy of the layer table the kernels read it: the same logits, and it stays capturable."""
    m = _model(be, cuda, *SHAPES[1])
    cache = _cache(m, 70, 4)
    m.fwd.tokens.copy_(torch.arange(32))
    m.fwd.pos.copy_(70 + torch.arange(32))
    m.fwd.prefix.fill_(70)
    m.fwd.mask.copy_(torch.tensor([(2 << i) - 1 for i in range(32)]))
    want = m.forward_device(20, cache, 0, 20).clone()
    desc = be._lib.ForwardDesc.from_buffer_copy(m._fused_desc(20, cache, 0, 20, m.fwd, 20, None))
    assert desc.timeline_pitch == be._lib.LAYERS_ON_HOST
    desc.timeline, desc.timeline_pitch = None, 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        be._lib.check(be._lib.lib().b200_forward(ctypes.byref(desc), be._lib.stream_ptr(m.device)), "b200_forward")
    m.logits.zero_()
    graph.replay()
    m.check_fused_error()
    assert torch.equal(m.logits[:20], want)


@pytest.mark.parametrize("rows", [8, 16, 20])
def test_without_a_host_table_the_call_returns_at_once_and_takes_the_table_in_stream_order(be, cuda, rows):
    m, other = _model(be, cuda, *SHAPES[1]), _model(be, cuda, *SHAPES[1])
    for lw in other.layers:
        lw["input_norm"].mul_(0.5)
        lw["post_norm"].neg_()
        lw["qkv"].bias.zero_()
    cache = _cache(m, 70, 4)
    m.fwd.tokens.copy_(torch.arange(32))
    m.fwd.pos.copy_(70 + torch.arange(32))
    m.fwd.prefix.fill_(70)
    m.fwd.mask.copy_(torch.tensor([(2 << i) - 1 for i in range(32)]))
    want = m.forward_device(rows, cache, 0, rows).clone()
    wrong = other.forward_device(rows, cache, 0, rows, m.fwd).clone()
    assert not torch.equal(want, wrong)
    desc = be._lib.ForwardDesc.from_buffer_copy(m._fused_desc(rows, cache, 0, rows, m.fwd, rows, None))
    table, right = other._layer_table.clone(), m._layer_table
    desc.timeline, desc.timeline_pitch, desc.layer_table = None, 0, table.data_ptr()
    m.logits.zero_()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                       # (a tenth of a second, which the call must not wait for)
    table.copy_(right)
    done = torch.cuda.Event()
    be._lib.check(be._lib.lib().b200_forward(ctypes.byref(desc), be._lib.stream_ptr(m.device)), "b200_forward")
    done.record()
    assert not done.query()
    done.synchronize()
    m.check_fused_error()
    assert torch.equal(m.logits[:rows], want)


def test_a_repeated_pass_runs_from_a_graph_on_the_data_of_the_call(be, cuda):
    m = _model(be, cuda, *SHAPES[0])
    keep = m._graphs.KEEP
    cache = _cache(m, 10, 5)
    for i in range(4 * m._graphs.AFTER):                 # (two result addresses in turn)
        cache.offset = 10 + i % 3
        tokens = torch.tensor([[i % 5, 7]])
        got = m(tokens, cache)
        cache.offset = 10 + i % 3
        m.fused = False
        assert ((got - m(tokens, cache)).abs() <= 2e-2).all()
        m.fused = True
    assert any(g for _, g in m._graphs._seen.values())
    caches = [m.make_cache(64 * (1 + i)) for i in range(keep + 2)]       # more passes than graphs are kept for
    for _ in range(m._graphs.AFTER + 2):
        for c in caches:
            c.offset = 0
            m(tokens, c)
    m.check_fused_error()
    assert len(m._graphs._seen) <= keep


def test_every_repetition_of_a_pass_gives_the_same_bits(be, cuda):
    """Thirty thousand passes with a wide head, whose CTAs go round their ring of weight stages many times: a stage given back
    before all of its loads are through shows as wrong logits of a few rows in some of them."""
    args = dataclasses.replace(be.shape_preset("qwen2-0.5b"), num_hidden_layers=1)
    m = be.Model.random_init(args, seed=3, device=cuda).relayout()
    tokens = torch.arange(32, dtype=torch.int32, device=cuda)[None]
    cache = m.make_cache(64)
    want = m(tokens, cache)
    wrong = torch.zeros((), dtype=torch.int64, device=cuda)
    for i in range(30000):
        cache.offset = 0
        wrong += (m(tokens, cache) != want).any()
        if i % 200 == 0:
            torch.cuda.synchronize()                     # (the host stays near)
    assert int(wrong) == 0
    m.check_fused_error()


@pytest.mark.parametrize("count", [5, 50])              # kernel chain (replayed from a graph), prompt path
def test_a_tensor_replaced_between_passes_is_seen_by_the_next(be, cuda, count):
    m = _model(be, cuda, *SHAPES[0])
    other, third = (be.Model.random_init(m.args, seed=seed, device=cuda, gen_device="cpu") for seed in (8, 9))
    o = other.layers[1]["o"]
    rows = be.llama.QLinear(o.weight, o.scales, o.biases)
    other.relayout()
    head = third.relayout().embed
    cache = _cache(m, 10, 5)
    tokens = torch.arange(count)[None]

    def run(fused):
        m.fused = m.prefill_large_m = fused
        cache.offset = 10
        return m(tokens, cache).float()

    steps = [lambda: setattr(m, "norm", other.norm), lambda: setattr(m, "embed", other.embed), lambda: setattr(m, "lm_head", head),
             lambda: m.layers[0].update(input_norm=other.layers[0]["input_norm"]), lambda: m.layers[1].update(post_norm=other.layers[1]["post_norm"]),
             lambda: m.layers[1].update(down=other.layers[1]["down"]), lambda: setattr(m.layers[0]["gate"], "tiled", other.layers[0]["gate"].tiled),
             lambda: setattr(m.layers[0]["qkv"], "bias", None), lambda: m.layers.reverse(),
             lambda: m.layers[0].update(o=rows)]
    before = None
    for step in steps:
        for _ in range(2 * m._graphs.AFTER):
            run(True)
        step()
        junk = [torch.full((1 << 16,), 77.0, dtype=torch.float16, device=cuda) for _ in range(8)]      # (where freed weights were)
        got, want = run(True), run(False)
        assert ((got - want).abs() <= 2.0 ** -6 * want.abs() + 1e-2).all()
        assert before is None or not torch.equal(got, before)
        before = got
        del junk
    m.fused = True
    assert not m.can_fuse()                              # (the last one has no re-laid-out weights: the per-op kernels ran it)
    rows.relayout(keep_rowmajor=True)
    assert m.can_fuse()
    got, want = run(True), run(False)
    assert ((got - want).abs() <= 2.0 ** -6 * want.abs() + 1e-2).all()
    m.check_fused_error()


@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(8, 128), (136, 256), (904, 1152), (2056, 2176), (18432, 1024), (2048, 12288), (2048, 12416)])
def test_matmul_of_the_chain_on_its_own(be, cuda, rows, n, k):
    """The operator on either side of the size where it changes kernels, both weight layouts, with edges of row tiles and clusters."""
    g = torch.Generator(device=cuda).manual_seed(n + k)
    wq, s, b = be.quantize.quantize(torch.randn(n, k, generator=g, device=cuda) * 0.02)
    x = torch.randn(rows, k, generator=g, device=cuda).half()
    bias = torch.randn(n, generator=g, device=cuda).half()
    w = be.quantize.dequantize(wq, s, b).float()
    want = x.float() @ w.T + bias.float()
    for got in (be.qmm_kernel.matmul_tiled(x, be.qmm_kernel.relayout(wq, s, b), n, bias=bias), be.matmul(x, wq, s, b, 64, bias=bias)[0]):
        assert ((got.float() - want).abs() <= 2e-3 * want.abs() + 4e-3).all()
    assert be.qmm_kernel.stream_error(cuda) == 0
