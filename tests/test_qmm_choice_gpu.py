"""Up to 32 rows the matmul kernel with clusters along K (csrc/decode.cu) and the one for many rows share the sizes: both sides of each line
between them, and cluster sizes from none to one chunk a CTA, on both layouts, against the fp64 gold of the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import qmm_ref

pytestmark = pytest.mark.gpu


# two chunks, seven of one each, tokens that do not fill their groups; 2040 and 2048 chunks in 120 and 128 tiles, 2048 and 4096 in 64 tiles and
# the next more; as quantised 1024 chunks and more, without a split, 70 tiles in pairs; ragged last tiles
@pytest.mark.parametrize("n,k", [(128, 256), (896, 896), (264, 1024), (15320, 2176), (16384, 2048), (4096, 8192), (8184, 8192), (8200, 8192), (5120, 5120),
                                 (2056, 8192), (8960, 1536), (2560, 9728), (32000, 1024)])
@pytest.mark.parametrize("m", [1, 13, 32])
def test_both_layouts_match_gold(be, cuda, m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    packed = be.quantize.quantize(torch.randn(n, k, generator=g) * 0.02)
    x = torch.randn(m, k, generator=g).half()
    pick = torch.cat([torch.arange(0, min(n, 300)), torch.arange(max(0, n - 300), n)]).unique()        # the first tiles and the last
    gold = qmm_ref.qmm_gold(x.numpy(), packed[0][pick].numpy().view(np.uint32), packed[1][pick].numpy(), packed[2][pick].numpy())
    dev = [t.to(cuda) for t in packed]
    xd = x.to(cuda)
    for y in (be.matmul(xd, *dev, 64)[0], be.qmm_kernel.matmul_tiled(xd, be.qmm_kernel.relayout(*dev), n)):
        err = np.abs(y.cpu().numpy()[:, pick].astype(np.float64) - gold)
        # an fp16 rounding of the result that may go the other way, 2^-10 of it; 4e-3 as for the other kernels on up to 18944 products in fp32
        assert np.all(err <= 2.0 ** -10 * np.abs(gold) + 4e-3), f"max err {err.max()}"
