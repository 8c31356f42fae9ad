"""The persistent kernel of a tensor-parallel shard (csrc/forward.cu) on one GPU: a group of two whose second member is the first
again, so that the one launch makes all arrivals of the all-GPU barriers itself and waits for nobody.  In the push form the
second member's partial products stay what the test put there (nothing), in the pull forms they are the first's own (a
o_proj and down_proj of half the size then give the whole).  Either way the shard computes the unsharded model, which the
per-op kernels check."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

AUTO, HIERARCHICAL, PUSH, PULL = 0, 2, 3, 4


def _close(got, want, rel=2.0 ** -6, abs_=2e-2):
    assert torch.isfinite(got).all()
    err = (got.float() - want.float()).abs()
    assert (err <= rel * want.float().abs() + abs_).all(), f"max err {float(err.max())} (scale {float(want.abs().max())})"


class _Pair:
    """A model (per-op kernels) and the shard that computes it."""

    def __init__(self, be, cuda, args, form, seed=5, gen_device="cpu"):
        self.be, self.form = be, form
        self.model = be.Model.random_init(args, seed=seed, device=cuda, gen_device=gen_device)
        self.shard = be.Model.random_init(args, seed=seed, device=cuda, gen_device=gen_device)
        if form in (HIERARCHICAL, PULL):
            for lw in self.shard.layers:
                for k in ("o", "down"):
                    lw[k].scales.mul_(0.5)
                    lw[k].biases.mul_(0.5)
        self.model.relayout()
        self.shard.relayout()
        self.model.fused = False
        lib = be._lib.lib()
        self.buffer = torch.zeros(lib.b200_forward_tp_buffer_bytes(args.hidden_size), dtype=torch.uint8, device=cuda)
        self.shard.tp = be.llama.TensorParallel(0, 2)
        self.shard.tp.peers = [self.buffer.data_ptr()] * 2
        self.shard.tp_two_shot = form
        assert self.shard.can_fuse() and not self.model.can_fuse()

    def caches(self, rows, cached, seed=1):
        out = []
        for m in (self.model, self.shard):
            c = m.make_cache(rows)
            g = torch.Generator().manual_seed(seed)
            c.data[:, :, :, :cached] = (0.3 * torch.randn(c.data[:, :, :, :cached].shape, generator=g)).half().to(c.data.device)
            c.offset = cached
            out.append(c)
        return out

    def check(self):
        self.shard.check_fused_error()


def _tree(rows, rng):
    tm = np.eye(rows, dtype=bool)
    for i in range(1, rows):
        tm[i] |= tm[int(rng.integers(0, i))]
    return torch.from_numpy(tm)


@pytest.mark.parametrize("form", [AUTO, HIERARCHICAL, PUSH, PULL])
@pytest.mark.parametrize("name", ["tiny-qwen2", "tiny-llama"])
def test_shard_kernel_equals_per_op_kernels(be, cuda, name, form):
    """Row counts on both sides of the kernel's variants, short and long caches (one phase of attention or a split and a merge),
    both nibble expansions; passes follow one another in the same exchange buffer and repeat bit for bit."""
    p = _Pair(be, cuda, be.shape_preset(name), form)
    rng = np.random.default_rng(3)
    for rows, cached, split, fast in [(1, 0, 0, True), (8, 63, 0, False), (9, 64, -1, True), (16, 300, 0, True), (17, 300, -1, False),
                                      (24, 447, 3, True), (31, 2200, 0, True), (32, 90, 0, True)]:
        tokens = torch.from_numpy(rng.integers(0, p.model.args.vocab_size, rows))[None]
        tm = _tree(rows, rng)
        p.shard.attn_split_blocks, p.shard.fast_dequant = split, fast
        cm, cs = p.caches(64 * ((cached + rows + 63) // 64), cached)
        want = be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, p.model, cm)[0]
        got = be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, p.shard, cs)[0].clone()
        p.check()
        _close(got, want)
        _close(cs.data, cm.data)
        cs.offset = cached
        assert torch.equal(be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, p.shard, cs)[0], got)
        cs.offset = cached
        one = p.shard(tokens, cs, logits_last_only=True)     # causal, the head on one row
        cm.offset = cached
        _close(one[0], p.model(tokens, cm, logits_last_only=True)[0])
    p.check()


@pytest.mark.parametrize("room", [0, 70])
@pytest.mark.parametrize("name", ["tiny-qwen2", "tiny-llama"])
def test_cache_rows_behind_the_last_do_not_reach_the_results(be, cuda, name, room):
    """They may hold anything, the next head's rows where the cache's are no multiple of a key block among it."""
    p = _Pair(be, cuda, be.shape_preset(name), PUSH)
    for rows, cached, split in [(1, 62, 0), (1, 64, 0), (17, 300, -1), (9, 600, 3), (32, 90, 0)]:
        tokens = torch.randint(0, p.model.args.vocab_size, (1, rows), generator=torch.Generator().manual_seed(rows))
        p.shard.attn_split_blocks = split

        def run(behind):
            _, cache = p.caches(max(64, cached + rows + room), cached)
            cache.data[:, :, :, cached:] = behind
            return p.shard(tokens, cache).clone(), cache.data[:, :, :, :cached + rows].clone()

        want = run(0.0)
        assert all(torch.isfinite(t).all() for t in want)
        for behind in (float("nan"), float("inf"), -65504.0):
            assert all(torch.equal(a, b) for a, b in zip(run(behind), want))
    p.check()


@pytest.mark.parametrize("form", [PUSH, PULL])
@pytest.mark.parametrize("world", [4, 8])
def test_shard_kernel_at_the_shapes_of_a_large_model(be, cuda, world, form):
    """What one of 4 or 8 GPUs multiplies of a 70B-shape layer: narrow and deep matrices, K cut across CTAs."""
    full = be.shape_preset("llama3-70b")
    args = dataclasses.replace(full, num_hidden_layers=2, head_dim=128, num_attention_heads=full.num_attention_heads // world,
                               num_key_value_heads=full.num_key_value_heads // world, intermediate_size=full.intermediate_size // world,
                               vocab_size=full.vocab_size // world)
    p = _Pair(be, cuda, args, form, seed=33, gen_device=cuda)
    rng = np.random.default_rng(world)
    for rows, cached in [(5, 100), (16, 700), (32, 140)]:
        tokens = torch.from_numpy(rng.integers(0, args.vocab_size, rows))[None]
        tm = _tree(rows, rng)
        cm, cs = p.caches(64 * ((cached + rows + 63) // 64), cached)
        want = be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, p.model, cm)[0]
        got = be.eagle.tree_decoding(tokens, tm, tm.sum(1) - 1, p.shard, cs)[0]
        p.check()
        # hidden 8192 with random weights gives logits of magnitude ~10: the absolute term follows their scale
        _close(got, want, abs_=max(2e-2, 2.0 ** -8 * float(want.abs().max())))
        _close(cs.data, cm.data, abs_=max(2e-2, 2.0 ** -8 * float(cm.data.abs().max())))


@pytest.mark.parametrize("name", ["tiny-qwen2", "tiny-llama"])
def test_shard_kernel_adds_the_other_members_products(be, cuda, name):
    """One layer, the push form, and real partial products of a second member in its slots: o_proj's and down_proj's of a shard that
    holds the other half of the heads and of the MLP.  Each half's products come from a launch of its own (the first exchange
    does not depend on the other half, the second only on the first), then both are there and the pass is the whole model's."""
    args = dataclasses.replace(be.shape_preset(name), num_hidden_layers=1, num_key_value_heads=2)
    rows, H = 11, args.hidden_size
    whole = be.Model.random_init(args, seed=4, device=cuda, gen_device="cpu")
    halves = [whole.shard(r, 2, shard_head=False) for r in range(2)]
    for h in halves:
        if h.lm_head is not whole.embed:
            h.lm_head = be.llama.QLinear(whole.lm_head.weight, whole.lm_head.scales, whole.lm_head.biases)
        h.relayout()
    whole.relayout()
    whole.fused = False
    tokens = torch.arange(3, 3 + rows)[None]
    want = whole(tokens, whole.make_cache(64))[0]
    lib = be._lib.lib()
    nbytes = lib.b200_forward_tp_buffer_bytes(H)
    base = 4096 + 2 * 32 * H * 4 + 2 * 32 * H * 2                        # csrc/tp_layout.cuh: the push slots
    buffers = [torch.zeros(nbytes, dtype=torch.uint8, device=cuda) for _ in range(2)]
    slots = [b[base:].view(torch.float32).view(2, 8, 32 * H) for b in buffers]       # [exchange & 1][source rank]
    for r, h in enumerate(halves):
        h.tp.peers = [buffers[r].data_ptr()] * 2
        h.tp_two_shot = PUSH
    got = None
    for known in range(3):                                               # exchanges whose products are there from both
        got = []
        for r, h in enumerate(halves):
            buffers[r][:4096].zero_()
            got.append(h(tokens, h.make_cache(64))[0].clone())
            h.check_fused_error()
        for x in range(min(known + 1, 2)):
            slots[0][x, 1].copy_(slots[1][x, 1])
            slots[1][x, 0].copy_(slots[0][x, 0])
    _close(got[0], want)
    assert torch.equal(got[0], got[1])                                   # added in rank order on both
