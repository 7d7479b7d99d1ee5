"""Tiles shared by a cluster of CTAs at the edges of their rule, against the oracle (GPU)."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from oracle import kmap_oracle as ko
from tests.helpers import cmax_of, launches, surface_cloud

pytestmark = [pytest.mark.gpu, pytest.mark.split_tiles]


# one CTA per SM (widths that are multiples of 32): 33 | 34 tiles have four parts each, 74 | 75 two; with 125 offsets 37 | 38 four and
# 98 | 99 two from two K blocks on
_DEEP = [(1, 64, 64, 3, 4), (127, 96, 96, 3, 4), (129, 128, 160, 3, 4), (3072, 256, 256, 3, 4), (4224, 64, 64, 3, 4), (4225, 64, 64, 3, 1),
         (4224, 96, 32, 3, 4), (4225, 96, 32, 3, 2), (9400, 64, 256, 3, 1), (9472, 192, 48, 3, 2), (9473, 192, 48, 3, 1), (9500, 64, 256, 3, 1),
         (14208, 128, 128, 3, 1), (28416, 64, 64, 3, 1), (56832, 96, 96, 3, 1),
         (4224, 64, 32, 5, 4), (4225, 32, 64, 5, 2), (4736, 96, 48, 5, 4), (4737, 96, 48, 5, 2), (9472, 64, 256, 5, 2), (9473, 64, 32, 5, 1),
         (9473, 160, 32, 5, 2), (12544, 96, 128, 5, 2), (12545, 96, 16, 5, 1)]
# two or three (the others): 24 | 25 tiles eight parts, 444 (296 beyond 128 output channels) CTA slots four and two
_UMMA = [(1, 48, 64, 3, 4), (127, 80, 96, 3, 8), (129, 112, 160, 3, 8), (3072, 208, 256, 3, 8), (3073, 208, 256, 3, 4), (9472, 80, 256, 3, 4),
         (9473, 80, 256, 3, 2), (14208, 144, 128, 3, 4), (14209, 144, 128, 3, 2), (28416, 80, 64, 3, 2), (28417, 80, 64, 3, 1)]


@pytest.mark.parametrize("n,cin,cout,ks,parts", _DEEP + _UMMA)
def test_parts_of_a_tile(n, cin, cout, ks, parts):
    import pcengine_b200 as pce
    from pcengine_b200 import _lib
    from pcengine_b200 import functional as PF
    coords = np.ascontiguousarray(surface_cloud(8, int(n ** 0.5 * 1.2) + 2)[:n])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert _lib.lib.pce_conv_split_parts(n, n, cin, cout, ks ** 3, sms) == parts
    d2 = ko.build_d2(coords, (ks,) * 3, (1,) * 3, (0,) * 3, [0] * 3, cmax_of(coords), True)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), (ks,) * 3, (1,) * 3, (0,) * 3, [0] * 3, cmax_of(coords), True)
    g = torch.Generator().manual_seed(n + cin)
    x, w = torch.randn(n, cin, generator=g).half(), (torch.randn(ks ** 3, cin, cout, generator=g) / (ks ** 3 * cin) ** 0.5).half()
    shift, res = torch.randn(cout, generator=g), torch.randn(n, cout, generator=g).half()
    want = torch.relu(co.conv_forward(x, w, d2) + shift + res.float())
    ep = PF.FusedEpilogue(shift=shift.cuda(), residual=res.cuda(), act="relu")
    outs = [PF.conv_forward(x.cuda(), w.cuda(), km.csr(), ep) for _ in range(2)]
    assert torch.equal(*outs) and co.rel_l2(outs[0].float().cpu(), want) <= 1e-3
    if sms == 148:  # what the library says is what it launches
        xd, wd, tiles = x.cuda(), w.cuda(), -(-n // 128)
        (name, blocks), = launches(lambda: PF.conv_forward(xd, wd, km.csr(), ep))
        assert ("k_conv_deep" if cin % 32 == 0 else "k_conv_umma") in name
        assert blocks == parts * tiles if parts > 1 else blocks <= tiles
    assert PF.device_status() == 0


def test_parts_need_no_scratch():
    """The flag alone splits a small map: the engine allocates the output and nothing else, the sums are those that a call
    with scratch gives, and another association than the whole chain's."""
    import pcengine_b200 as pce
    from pcengine_b200 import _lib
    from pcengine_b200 import functional as PF
    coords = surface_cloud(8, 66)[:3000]
    n, sms = len(coords), torch.cuda.get_device_properties(0).multi_processor_count
    assert _lib.lib.pce_conv_split_parts(n, n, 256, 256, 27, sms) > 1
    assert _lib.lib.pce_conv_split_scratch_wanted(n, n, 256, 256, 27, sms) == 0
    csr = pce.KernelMap(torch.from_numpy(np.ascontiguousarray(coords)).cuda(), (3,) * 3, (1,) * 3, (0,) * 3, [0] * 3, cmax_of(coords), True).csr()
    g = torch.Generator().manual_seed(1)
    x, w = torch.randn(n, 256, generator=g).half().cuda(), (torch.randn(27, 256, 256, generator=g) / 83).half().cuda()
    first = PF.conv_forward(x, w, csr)
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    again = PF.conv_forward(x, w, csr)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before + 1
    lists, packed, scratch = csr.tiles(True, 128, False, 1), PF.packed_weights(w), torch.empty(16, device="cuda")
    out, e = torch.empty_like(first), _lib.Epilogue(split_scratch=scratch.data_ptr(), split_scratch_bytes=64)
    _lib.check(_lib.lib.pce_conv_fwd(x.data_ptr(), n, 256, None, packed.data_ptr(), 27, 256, None, None, None, C.byref(lists), n,
                                     out.data_ptr(), _lib.PCE_F16, C.byref(e), _lib.KERNEL_AUTO, _lib.stream_ptr(x.device)), "pce_conv_fwd")
    PF.SPLIT_TILES = False  # (the test's fixture puts it back)
    whole = PF.conv_forward(x, w, csr)
    assert torch.equal(first, again) and torch.equal(first, out) and not torch.equal(first, whole)
