"""A device-side wait that runs out: the kernel ends by itself, the host reads an error status, a reset
restores service.  The waits are made to run out by giving them a short poll limit (``b200_set_wait_limit``) and
a peer that never answers (a second buffer on the same GPU whose flags nobody raises): nothing faults, nothing
hangs, no process dies."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

KEY_FLAGS, KEY_COUNT, KEY_ERR, KEYS, FLAG_STRIDE = 1024, 1536, 1540, 2048, 64      # csrc/tp_layout.cuh


@pytest.fixture()
def short_waits(be, cuda):
    lib = be._lib.lib()
    lib.b200_set_wait_limit(4096)
    yield lib
    lib.b200_set_wait_limit(0)


def _buffers(lib, cuda, hidden):
    nbytes = lib.b200_forward_tp_buffer_bytes(hidden)
    own = torch.zeros(nbytes, dtype=torch.uint8, device=cuda)
    peer = torch.zeros(nbytes, dtype=torch.uint8, device=cuda)
    arr = (ctypes.c_void_p * 8)(own.data_ptr(), peer.data_ptr())
    return nbytes, own, peer, arr


def test_argmax_combine_gives_up_reports_and_recovers(be, cuda, short_waits):
    lib, p = short_waits, be._lib.ptr
    nbytes, own, peer, arr = _buffers(lib, cuda, 256)
    st = be._lib.stream_ptr(cuda)
    mine = (torch.arange(1, 9, dtype=torch.int64, device=cuda) << 32) | 0xFFFFFF00
    keys = mine.clone()
    assert lib.b200_tp_argmax_combine(p(keys), 8, 0, 2, 0, arr, st) == 0
    torch.cuda.synchronize()                                     # returns: the wait ran out after 4096 polls
    assert lib.b200_tp_exchange_error(ctypes.c_void_p(own.data_ptr())) == 1
    assert torch.equal(keys, mine)                               # nothing was combined
    # the host's recovery: zero the buffers, then a combine whose peer does answer (the test plays the peer:
    # its keys in its buffer, its flag in ours) succeeds and the error word stays clear
    assert lib.b200_tp_exchange_reset(ctypes.c_void_p(own.data_ptr()), nbytes) == 0
    assert lib.b200_tp_exchange_reset(ctypes.c_void_p(peer.data_ptr()), nbytes) == 0
    theirs = (torch.tensor([9, 1, 9, 1, 9, 1, 9, 1], dtype=torch.int64, device=cuda) << 32) | 0xFFFFFF00
    peer[KEYS:KEYS + 64].view(torch.int64).copy_(theirs)
    own[KEY_FLAGS + FLAG_STRIDE:KEY_FLAGS + FLAG_STRIDE + 4].view(torch.int32).fill_(1)
    keys = mine.clone()
    assert lib.b200_tp_argmax_combine(p(keys), 8, 0, 2, 0, arr, st) == 0
    torch.cuda.synchronize()
    assert lib.b200_tp_exchange_error(ctypes.c_void_p(own.data_ptr())) == 0
    assert torch.equal(keys, torch.maximum(mine, theirs))
    assert int(own[KEY_COUNT:KEY_COUNT + 4].view(torch.int32)) == 1


def test_forward_all_gpu_barrier_gives_up_and_the_model_recovers(be, cuda, short_waits):
    lib = short_waits
    args = be.shape_preset("tiny-qwen2")
    base = be.Model.random_init(args, seed=11, device=cuda, gen_device="cpu")
    prompt = torch.arange(5, 17, dtype=torch.int32)
    whole = be.Model.random_init(args, seed=11, device=cuda, gen_device="cpu").relayout()
    want = whole(prompt[None], cache=whole.make_cache(128))
    shard = base.shard(0, 2).relayout()
    nbytes, own, peer, arr = _buffers(lib, cuda, args.hidden_size)
    shard.tp.peers, shard.tp.peer_array, shard.tp.nbytes = [own.data_ptr(), peer.data_ptr()], arr, nbytes
    assert shard.can_fuse()
    shard(prompt[None], cache=shard.make_cache(128))             # rank 1 does not exist: its arrivals never come
    torch.cuda.synchronize()                                     # ... and the kernel still ends
    with pytest.raises(be._lib.B200Error, match="code 12"):
        shard.check_fused_error()                                # also clears the kernel's barrier words
    assert lib.b200_tp_exchange_reset(ctypes.c_void_p(own.data_ptr()), nbytes) == 0
    # the GPU and the library stay usable: the unsharded model gives its usual logits
    again = whole(prompt[None], cache=whole.make_cache(128))
    whole.check_fused_error()
    assert torch.equal(again, want)


@pytest.mark.parametrize("heads,kv,hd,inter", [(14, 2, 64, 4864), (16, 2, 128, 2176)])      # down_proj cut over clusters; 256 query rows per kv head
def test_a_wait_of_the_kernel_chain_runs_out_is_reported_and_clears(be, cuda, heads, kv, hd, inter):
    """A poll limit of one: the kernels of a pass start while the ones before them run, so waits for their activations run out.
    The pass ends with its error word set (and, since what it waits for comes, with its result)."""
    lib = be._lib.lib()
    args = be.ModelArgs(model_type="qwen2", hidden_size=heads * hd, num_hidden_layers=3, intermediate_size=inter, num_attention_heads=heads,
                        num_key_value_heads=kv, rms_norm_eps=1e-6, vocab_size=2048)
    model = be.Model.random_init(args, seed=3, device=cuda, gen_device="cpu").relayout()
    cache = model.make_cache(3584)
    tokens = torch.arange(5, 37, dtype=torch.int32, device=cuda)[None]

    def run(rows):
        cache.offset = 3500
        return model(tokens[:, :rows], cache)

    for rows in (32, 8):
        for _ in range(4 * model._graphs.AFTER):
            want = run(rows)
        assert any(g for _, g in model._graphs._seen.values())              # (replayed by now: the limit has to reach such passes too)
        model.check_fused_error()
        try:
            lib.b200_set_wait_limit(1)
            assert torch.equal(run(rows), want)
            with pytest.raises(be._lib.B200Error, match="code 2[1-9]"):
                model.check_fused_error()
        finally:
            lib.b200_set_wait_limit(0)
        for _ in range(3):
            assert torch.equal(run(rows), want)
        model.check_fused_error()                                # clear again, and stays so


def test_a_wait_of_a_prompt_pass_runs_out_is_reported_and_clears(be, cuda):
    """The gate / up matmul of these sizes leaves twenty SMs free, on which the next one starts and waits for it."""
    lib = be._lib.lib()
    args = be.ModelArgs(model_type="llama", hidden_size=2048, num_hidden_layers=2, intermediate_size=2048, num_attention_heads=16,
                        num_key_value_heads=2, rms_norm_eps=1e-5, vocab_size=2048)
    model = be.Model.random_init(args, 5, cuda).relayout()
    cache = model.make_cache(1024)
    tokens = torch.randint(0, args.vocab_size, (1, 1000), generator=torch.Generator().manual_seed(1))

    def run():
        cache.offset = 0
        return model(tokens, cache)

    want = run()
    model.check_fused_error()
    try:
        lib.b200_set_wait_limit(1)
        torch.cuda._sleep(4_000_000)                             # (2 ms in which the host gets ahead: the kernels then follow at once)
        assert torch.equal(run(), want)
        with pytest.raises(be._lib.B200Error, match="b200_prefill"):
            model.check_fused_error()
    finally:
        lib.b200_set_wait_limit(0)
    assert torch.equal(run(), want)
    model.check_fused_error()


@pytest.mark.parametrize("m,n,k,epilogue", [(16, 4096, 512, 0), (100, 2048, 4096, 0), (40, 1024, 2048, 2)])
def test_a_wait_of_a_matmul_runs_out_is_reported_and_clears(be, cuda, m, n, k, epilogue):
    """The matmul starts on free SMs while one of a single long tile still runs, and waits for it before its activations."""
    lib, p, st = be._lib.lib(), be._lib.ptr, be._lib.stream_ptr(cuda)
    g = torch.Generator(device=cuda).manual_seed(m)

    def operands(rows, outs, width):
        w = be.quantize.quantize(torch.randn(outs, width, generator=g, device=cuda) * 0.02)
        ws = torch.zeros(lib.b200_qmm_gemm_workspace_bytes(rows, outs, width, epilogue), dtype=torch.uint8, device=cuda)
        return (torch.randn(rows, width, generator=g, device=cuda).half(), be.qmm_kernel.relayout(*w), be.qmm_kernel.relayout(*w),
                torch.empty(rows, outs, dtype=torch.float16, device=cuda), ws)

    def call(o, shape, epi, room):
        assert lib.b200_qmm_gemm(p(o[0]), p(o[1]), p(o[2]) if epi == 2 else None, None, None, p(o[3]), *shape, epi, p(o[4]), room, st) == 0

    long_, mine = operands(16, 128, 65536), operands(m, n, k)
    call(mine, (m, n, k), epilogue, mine[4].numel())
    want = mine[3].clone()
    error = lambda: int(mine[4][4092:4096].view(torch.int32))
    assert error() == 0
    try:
        lib.b200_set_wait_limit(1)
        call(long_, (16, 128, 65536), 0, 4096)                   # (no cut of K: one CTA)
        call(mine, (m, n, k), epilogue, mine[4].numel())
        assert error() in (1, 2, 3)
    finally:
        lib.b200_set_wait_limit(0)
    assert torch.equal(mine[3], want)
    mine[4][4092:4096].zero_()
    call(mine, (m, n, k), epilogue, mine[4].numel())
    assert torch.equal(mine[3], want)
    assert int(mine[4][:4096].view(torch.int32).abs().sum()) == 0            # tickets restored, no wait ran out
