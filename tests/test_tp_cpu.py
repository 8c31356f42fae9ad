"""Host logic of the tensor-parallel target on CPU: the shards of Model.shard() tile the unsharded weights
exactly (column-parallel q|k|v, gate, up and head by rows; row-parallel o_proj, down_proj by K columns), and the
vocabulary-parallel greedy argmax over two gloo ranks equals the argmax of the whole row, ties to the lower id."""
import os
import sys

import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


@pytest.mark.parametrize("preset,world", [("tiny-qwen2", 2)])
def test_shards_tile_the_unsharded_weights(be, preset, world):
    args = be.shape_preset(preset)
    full = be.Model.random_init(args, seed=3, device="cpu")
    shards = [full.shard(r, world) for r in range(world)]
    nq, nkv = full.nq, full.nkv
    for li, lw in enumerate(full.layers):
        for name in ("weight", "scales", "biases"):
            whole = getattr(lw["qkv"], name)
            parts = [getattr(s.layers[li]["qkv"], name) for s in shards]
            lq, lkv = nq // world, nkv // world
            assert torch.equal(torch.cat([p[:lq] for p in parts]), whole[:nq])                       # q heads
            assert torch.equal(torch.cat([p[lq:lq + lkv] for p in parts]), whole[nq:nq + nkv])        # k heads
            assert torch.equal(torch.cat([p[lq + lkv:] for p in parts]), whole[nq + nkv:])            # v heads
            for key in ("gate", "up"):                                                                # MLP rows
                assert torch.equal(torch.cat([getattr(s.layers[li][key], name) for s in shards]), getattr(lw[key], name))
            for key in ("o", "down"):                                                                 # K columns
                assert torch.equal(torch.cat([getattr(s.layers[li][key], name) for s in shards], dim=1),
                                   getattr(lw[key], name))
        if lw["qkv"].bias is not None:
            lq, lkv = nq // world, nkv // world
            b = [s.layers[li]["qkv"].bias for s in shards]
            assert torch.equal(torch.cat([x[:lq] for x in b]), lw["qkv"].bias[:nq])
        for s in shards:                                                                              # replicated
            assert s.layers[li]["input_norm"] is lw["input_norm"] and s.layers[li]["post_norm"] is lw["post_norm"]
    assert torch.equal(torch.cat([s.lm_head.weight for s in shards]), full.lm_head.weight)
    assert [s.vocab_offset for s in shards] == [r * args.vocab_size // world for r in range(world)]
    assert all(s.vocab_local == args.vocab_size // world and s.embed is full.embed for s in shards)
    assert all(s.args.num_attention_heads == args.num_attention_heads // world and
               s.args.intermediate_size == args.intermediate_size // world and s.args.head_dim == args.head_dim
               for s in shards)
    assert not shards[0].can_fuse()              # a shard fuses only once the peers' exchange buffers are mapped


def test_shard_refuses_degrees_that_do_not_divide(be):
    args = be.shape_preset("tiny-qwen2")
    full = be.Model.random_init(args, seed=3, device="cpu")
    with pytest.raises(be._lib.B200Error):
        full.shard(0, 3)


def test_layer_pointers_follow_the_layers(be):
    """The native walk over the layers: every pointer, whether any has changed, and what is no layer of re-laid-out weights."""
    import ctypes
    model = be.Model.random_init(be.shape_preset("tiny-qwen2"), seed=3, device="cpu")
    walk, n = be._lib.ops().layer_pointers, len(model.layers)
    table = (ctypes.c_void_p * (8 * (n + 1)))()
    at = ctypes.addressof(table)
    assert walk(model.layers, at) == -1                          # (not re-laid-out)
    for lw in model.layers:
        for k in ("qkv", "o", "gate", "up", "down"):
            lw[k].tiled = torch.zeros(16)
    assert walk(model.layers, at) == 1 and walk(model.layers, at) == 0 and walk(tuple(model.layers), at) == 0
    assert [p or 0 for p in table[:8 * n]] == [0 if t is None else t.data_ptr() for lw in model.layers for t in (
        lw["qkv"].tiled, lw["qkv"].bias, lw["o"].tiled, lw["gate"].tiled, lw["up"].tiled, lw["down"].tiled, lw["input_norm"], lw["post_norm"])]
    model.layers[1]["post_norm"].set_(torch.zeros(8, dtype=torch.float16))      # (the same object, other storage)
    assert walk(model.layers, at) == 1 and walk(model.layers, at) == 0
    model.layers[0]["qkv"].bias = None
    assert walk(model.layers, at) == 1 and table[1] is None
    assert walk(model.layers + [None], at) == -1
    without = [dict(lw) for lw in model.layers]
    del without[1]["down"]
    assert walk(without, at) == -1
    model.layers[0]["up"].tiled = None
    assert walk(model.layers, at) == -1


def test_layer_pointers_say_whether_the_scales_that_were_looked_at_are_there(be):
    """Of the very tensor that stands in the layer, with as many changes as then: one in its place may have its address, and its count."""
    import ctypes
    model = be.Model.random_init(be.shape_preset("tiny-qwen2"), seed=3, device="cpu")
    walk = be._lib.ops().layer_pointers
    table, fast = (ctypes.c_void_p * (8 * len(model.layers)))(), ctypes.c_uint32(7)
    ask = lambda: (walk(model.layers, ctypes.addressof(table), ctypes.addressof(fast)), fast.value)
    assert ask() == (-1, 0)
    for lw in model.layers:
        for k in ("qkv", "o", "gate", "up", "down"):
            lw[k].tiled = torch.zeros(16)
            lw[k]._fast_of = (lw[k].tiled, 0)
    lin = model.layers[1]["down"]
    assert ask() == (1, 1) and ask() == (0, 1) and lin.scales_fast
    lin.tiled.zero_()                                            # (written)
    assert ask() == (0, 0) and not lin.scales_fast
    lin._fast_of = (lin.tiled, 1)
    assert ask() == (0, 1) and lin.scales_fast
    other = be.llama.QLinear(lin.weight, lin.scales, lin.biases)
    other.tiled = lin.tiled[:]                                   # (another tensor: same address, same count)
    model.layers[1]["down"] = other
    assert other.tiled._version == 1 and ask() == (0, 0) and not other.scales_fast
    for of in (None, (), (other.tiled, "1"), (other.tiled,), 1):
        other._fast_of = of
        assert ask() == (0, 0)
    del other._fast_of
    assert ask() == (0, 0)
    other._fast_of = (other.tiled, 1)
    assert ask() == (0, 1)
    with torch.inference_mode():
        other.tiled = torch.zeros(16)
    other._fast_of = (other.tiled, 0)
    assert ask() == (1, 0)


def test_the_timeline_of_a_model_that_is_no_shard_is_refused(be):
    full = be.Model.random_init(be.shape_preset("tiny-qwen2"), seed=3, device="cpu")
    with pytest.raises(be._lib.B200Error, match="shard"):        # (its passes have no device-wide barriers to stamp)
        full.enable_timeline()
    full.enable_timeline(False)


def _rank(rank, world, port, out):
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    import b200_eagle as be
    args = be.shape_preset("tiny-qwen2")
    m = be.Model.random_init(args, seed=3, device="cpu").shard(rank, world)
    V = args.vocab_size
    g = torch.Generator().manual_seed(5)
    got = []
    for case in range(4):
        row = torch.randn(V, generator=g).half()
        if case == 1:                             # the maximum sits in both halves: the lower id wins
            row[7], row[V // 2 + 3] = 9.0, 9.0
        if case == 2:                             # ... and twice inside the upper half only
            row[V // 2 + 5], row[V - 1] = 9.0, 9.0
        want = int(torch.argmax(row.float()))     # first maximum
        mine = row[rank * (V // world):(rank + 1) * (V // world)]
        got.append((m.greedy_token(mine), want))
    if rank == 1:
        out.put(got)
    dist.barrier()
    dist.destroy_process_group()


def test_vocabulary_parallel_greedy_token_over_two_ranks():
    ctx = mp.get_context("spawn")
    out = ctx.Queue()
    port = 29700 + os.getpid() % 200
    procs = [ctx.Process(target=_rank, args=(r, 2, port, out), daemon=True) for r in range(2)]
    for p in procs:
        p.start()
    try:
        got = out.get(timeout=120)
        for p in procs:
            p.join(timeout=60)
            assert p.exitcode == 0
    finally:
        for p in procs:
            if p.is_alive():
                p.kill()
    assert all(a == b for a, b in got), got
