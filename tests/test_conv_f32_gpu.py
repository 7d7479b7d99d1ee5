"""The tiled fp32 convolution (lists of 128 rows, blocks of 32) and its dense product against the CPU oracle at the
edges of its tiles: row counts around a block and a tile, widths around the 4-channel pieces, the 16-channel chunks
and the per-block widths, and maps small and dense enough for every cluster size."""
import pytest
import torch

from oracle import conv_oracle as co
from oracle import kmap_oracle as ko
from tests.helpers import cmax_of, random_cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1500])
@pytest.mark.parametrize("cin,cout", [(4, 192), (19, 48), (33, 24), (32, 32), (64, 130), (128, 96), (256, 64)])
def test_tiled_fp32_convolution_equals_the_oracle(n, cin, cout):
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    coords = random_cloud(n + cin, 12, n)
    torch.manual_seed(n)
    feats, w = torch.randn(n, cin), torch.randn(27, cin, cout)
    d2 = ko.build_d2(coords, (3, 3, 3), (1, 1, 1), (0, 0, 0), [0, 0, 0], cmax_of(coords), True)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), (3, 3, 3), (1, 1, 1), (0, 0, 0), [0, 0, 0], cmax_of(coords), True)
    csr = km.csr()
    csr.lists_fp32()  # (with lists at hand a layer of any widths runs on the tiled kernel)
    res, shift = torch.randn(n, cout), torch.randn(cout)
    ep = PF.FusedEpilogue(scale=None, shift=shift.cuda(), residual=res.cuda(), act="relu")
    out = PF.conv_forward(feats.cuda(), w.cuda(), csr, ep)
    ref = torch.relu(co.conv_forward(feats, w, d2) + shift + res)
    assert co.rel_l2(out.cpu(), ref) <= 1e-5
    dense = PF.linear_forward(feats.cuda(), w[0].contiguous().cuda())
    assert co.rel_l2(dense.cpu(), feats @ w[0]) <= 1e-5


@pytest.mark.parametrize("n,cin,cout", [(300, 64, 64), (5000, 48, 128)])
def test_tiled_fp32_in_the_explicit_dataflow(n, cin, cout):
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    coords = random_cloud(n, 24, n)
    torch.manual_seed(n)
    feats, w = torch.randn(n, cin), torch.randn(27, cin, cout)
    d2 = ko.build_d2(coords, (3, 3, 3), (1, 1, 1), (0, 0, 0), [0, 0, 0], cmax_of(coords), True)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), (3, 3, 3), (1, 1, 1), (0, 0, 0), [0, 0, 0], cmax_of(coords), True)
    out = PF.conv_forward_d1(feats.cuda(), w.cuda(), km)
    assert co.rel_l2(out.cpu(), co.conv_forward(feats, w, d2)) <= 1e-5
