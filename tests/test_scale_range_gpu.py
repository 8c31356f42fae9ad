"""The short nibble expansion is chosen for weights that `relayout` found to allow it.  Weights that take their place afterwards, as
another tensor or written over the old one, are expanded as they need: with passes launched one by one and with graphs of them.  Where
torch does not count the write, the model is told."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["layer", "head"])
@pytest.mark.parametrize("how", ["replaced", "written"])
def test_weights_that_change_after_relayout(be, cuda, how, which):
    args = be.shape_preset("tiny-qwen2")
    m = be.Model.random_init(args, seed=5, device=cuda, gen_device="cpu")
    lin = m.layers[1]["down"] if which == "layer" else m.lm_head
    packed = [t.clone() for t in (lin.weight, lin.scales, lin.biases)]
    packed[1][3:40] = 0.25                               # beyond the range
    packed[1][41] = 0.0
    wide = be.qmm_kernel.relayout(*packed)
    m.relayout()
    tokens = torch.arange(7, dtype=torch.int32, device=cuda)[None]
    cache = m.make_cache(128)

    def run():
        cache.offset = 0
        return m(tokens, cache).clone()

    for _ in range(2 * m._graphs.AFTER):
        before = run()
    assert m._scales_fast is True
    kept = m.weight_addresses()
    if how == "replaced":
        lin.tiled = wide
    else:
        lin.tiled.copy_(wide)
    got = [run() for _ in range(2 * m._graphs.AFTER)]
    assert m._scales_fast is False and m.weight_addresses() != kept
    m.fast_dequant = False
    want = run()
    m.check_fused_error()
    assert torch.isfinite(want).all() and not torch.equal(want, before)
    assert all(torch.equal(g, want) for g in got)        # the same kernels: the same bits


def test_tiled_scales_reads_the_layout(be, cuda):
    for n, k in ((64, 128), (40, 256), (1000, 896)):
        g = torch.Generator().manual_seed(n)
        w, s, b = (t.to(cuda) for t in be.quantize.quantize(torch.randn(n, k, generator=g)))
        assert torch.equal(be.qmm_kernel.tiled_scales(be.qmm_kernel.relayout(w, s, b), n, k), s)


@pytest.mark.parametrize("which", ["layer", "head"])
def test_weights_written_past_torch(be, cuda, which):
    """Through ``.data``, then ``weights_changed``: passes as such weights need them, and, the old ones written back, as before."""
    args = be.shape_preset("tiny-qwen2")
    m = be.Model.random_init(args, seed=5, device=cuda, gen_device="cpu")
    lin = m.layers[1]["down"] if which == "layer" else m.lm_head
    packed = [t.clone() for t in (lin.weight, lin.scales, lin.biases)]
    packed[1][3:40] = 0.25
    packed[1][41] = 0.0
    wide = be.qmm_kernel.relayout(*packed)
    m.relayout()
    tokens = torch.arange(7, dtype=torch.int32, device=cuda)[None]
    cache = m.make_cache(128)

    def run():
        cache.offset = 0
        return m(tokens, cache).clone()

    old, passes = lin.tiled.clone(), 2 * m._graphs.AFTER
    before = [run() for _ in range(passes)]
    kept = m.weight_addresses()
    version = lin.tiled._version
    lin.tiled.data.copy_(wide)
    assert lin.tiled._version == version                 # (torch has not counted it)
    m.weights_changed()
    got = [run() for _ in range(passes)]
    assert m._scales_fast is False and m.weight_addresses() != kept
    m.fast_dequant = False
    want = run()
    m.fast_dequant = True
    assert torch.isfinite(want).all() and not torch.equal(want, before[0])
    assert all(torch.equal(g, want) for g in got)
    lin.tiled.data.copy_(old)
    m.weights_changed()
    assert all(torch.equal(run(), before[0]) for _ in range(passes)) and m._scales_fast is True and m.weight_addresses() == kept
    m.check_fused_error()


def test_weights_relaid_in_inference_mode(be, cuda):
    """They allow the short expansion like any, and writes are seen there, too."""
    m = be.Model.random_init(be.shape_preset("tiny-qwen2"), seed=5, device=cuda, gen_device="cpu")
    lin = m.layers[1]["down"]
    packed = [t.clone() for t in (lin.weight, lin.scales, lin.biases)]
    packed[1][3:40] = 0.25
    wide = be.qmm_kernel.relayout(*packed)
    tokens = torch.arange(7, dtype=torch.int32, device=cuda)[None]
    cache = m.make_cache(128)

    def run():
        cache.offset = 0
        return m(tokens, cache).clone()

    with torch.inference_mode():
        m.relayout()
        before = run()
        assert m._scales_fast is True
        lin.tiled.copy_(wide)
        got = run()
        assert m._scales_fast is False
    m.fast_dequant = False
    want = run()
    m.check_fused_error()
    assert torch.equal(got, want) and not torch.equal(want, before)


def test_weights_where_freed_ones_were(be, cuda):
    """A layer that is made anew once the old one has been let go can have its addresses: its own scales decide."""
    m = be.Model.random_init(be.shape_preset("tiny-qwen2"), seed=5, device=cuda, gen_device="cpu")
    old = m.layers[1]["down"]
    packed = [t.clone() for t in (old.weight, old.scales, old.biases)]
    packed[1][3:40] = 0.25
    m.relayout()
    tokens = torch.arange(7, dtype=torch.int32, device=cuda)[None]
    cache = m.make_cache(128)

    def run():
        cache.offset = 0
        return m(tokens, cache).clone()

    for _ in range(2 * m._graphs.AFTER):
        before = run()
    assert m._scales_fast is True
    at = old.tiled.data_ptr()
    new = be.llama.QLinear(*packed)
    del m.layers[1]["down"], old
    spare = []
    while True:                                          # (the allocator may have other blocks of this size first)
        new.relayout(keep_rowmajor=True)
        if new.tiled.data_ptr() == at or len(spare) > 1000:
            break
        spare.append(new.tiled)
    assert new.tiled.data_ptr() == at
    m.layers[1]["down"] = new
    got = [run() for _ in range(2 * m._graphs.AFTER)]
    assert m._scales_fast is False
    m.fast_dequant = False
    want = run()
    m.check_fused_error()
    assert not torch.equal(want, before) and all(torch.equal(g, want) for g in got)
