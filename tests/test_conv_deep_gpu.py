"""The one-CTA-per-SM convolution kernel at the edges of its tiles, rings and widths, against the oracle in fp32 and bit for bit
against the three-CTA kernel (GPU)."""
import numpy as np
import pytest
import torch

from oracle import conv_oracle as co
from oracle import kmap_oracle as ko
from tests.helpers import cmax_of, launches, random_cloud, surface_cloud

pytestmark = pytest.mark.gpu


def _map(coords, ks=3):
    import pcengine_b200 as pce
    d2 = ko.build_d2(coords, (ks,) * 3, (1,) * 3, (0,) * 3, [0] * 3, cmax_of(coords), True)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), (ks,) * 3, (1,) * 3, (0,) * 3, [0] * 3, cmax_of(coords), True)
    return d2, km.csr()


def _both(f):
    """f() by the kernel and, with a ring depth of the other one asked for, by that."""
    from pcengine_b200 import _lib
    a = f()
    _lib.lib.pce_tune(0, 2)
    try:
        return a, f()
    finally:
        _lib.lib.pce_tune(0, 0)


# rings of 9, 8, 7, 6, 5 and 4 stages; K blocks 1, 1 + half, 2, 2 + half, 4; rows at the edges of a tile and of a group of four;
# maps of more tiles than SMs; a dense block (27 offsets a row), sheets, and scattered voxels (most groups without rows)
@pytest.mark.parametrize("kind,n,cin,cout,ks", [
    ("sheet", 1, 64, 16, 3), ("sheet", 3, 64, 64, 3), ("sheet", 127, 96, 96, 3), ("sheet", 128, 128, 128, 3), ("sheet", 129, 64, 160, 3),
    ("block", 1331, 160, 224, 3), ("block", 1331, 256, 256, 3), ("random", 5000, 64, 112, 3), ("random", 5000, 128, 192, 5),
    ("sheet", 129, 32, 32, 3), ("block", 1331, 32, 96, 3), ("sheet", 94720, 32, 32, 3), ("sheet", 94721, 32, 32, 3), ("random", 5000, 32, 64, 5),
    ("sheet", 20001, 96, 64, 3), ("sheet", 40000, 64, 256, 3), ("random", 30000, 64, 64, 5)])
def test_layers(kind, n, cin, cout, ks):
    from pcengine_b200 import functional as PF
    if kind == "sheet":
        coords = surface_cloud(8, int(n ** 0.5 * 1.2) + 2)[:n]
    elif kind == "block":
        side = round(n ** (1 / 3))
        i = np.arange(n)
        coords = np.stack([0 * i, i // side ** 2, i // side % side, i % side], 1).astype(np.int32)
    else:
        coords = random_cloud(7, 40, n, batch=1)[:n]
    coords = np.ascontiguousarray(coords)
    n = len(coords)
    d2, csr = _map(coords, ks)
    g = torch.Generator().manual_seed(n + cin + cout)
    x, w = torch.randn(n, cin, generator=g).half(), (torch.randn(ks ** 3, cin, cout, generator=g) / (ks ** 3 * cin) ** 0.5).half()
    scale, shift, res = 0.5 + torch.rand(cout, generator=g), torch.randn(cout, generator=g), torch.randn(n, cout, generator=g).half()
    plain = co.conv_forward(x, w, d2)
    # fp16 outputs of fp32 sums: half a unit in the last place per value, 2^-11, and less in the 2-norm
    for ep, want in ((None, plain), (dict(scale=scale, shift=shift, act="relu"), torch.relu(plain * scale + shift)),
                     (dict(shift=shift, residual=res, act="leaky"), torch.nn.functional.leaky_relu(plain + shift + res.float(), 0.01))):
        e = PF.FusedEpilogue(**{k: v.cuda() if torch.is_tensor(v) else v for k, v in ep.items()}) if ep else None
        got, other = _both(lambda: PF.conv_forward(x.cuda(), w.cuda(), csr, e))
        assert co.rel_l2(got.float().cpu(), want) <= 5e-4
        assert torch.equal(got, other)
    assert PF.device_status() == 0


@pytest.mark.parametrize("n,cin,cin2,cout", [(129, 64, 32, 64), (3000, 32, 32, 32), (3000, 32, 64, 64), (3000, 96, 96, 96), (3000, 128, 96, 128), (3000, 96, 64, 256), (3000, 64, 160, 64)])
def test_second_operand(n, cin, cin2, cout):
    """Widths of the second operand that are whole K blocks, end in a half block and end in padding."""
    from pcengine_b200 import functional as PF
    coords = np.ascontiguousarray(surface_cloud(9, int(n ** 0.5 * 1.2) + 2)[:n])
    d2, csr = _map(coords)
    g = torch.Generator().manual_seed(n + cin2)
    x, w = torch.randn(n, cin, generator=g).half(), (torch.randn(27, cin, cout, generator=g) / (27 * cin) ** 0.5).half()
    x2, w2 = torch.randn(n, cin2, generator=g).half(), (torch.randn(cin2, cout, generator=g) / cin2 ** 0.5).half()
    ep = PF.FusedEpilogue(extra_feats=x2.cuda(), extra_weight=w2.cuda(), act="relu")
    want = torch.relu(co.conv_forward(x, w, d2) + x2.float() @ w2.float())
    got, other = _both(lambda: PF.conv_forward(x.cuda(), w.cuda(), csr, ep))
    assert co.rel_l2(got.float().cpu(), want) <= 5e-4 and torch.equal(got, other)


@pytest.mark.parametrize("n,cin,cout", [(1, 64, 64), (130, 96, 32), (129, 32, 32), (1000, 128, 256), (20000, 256, 48)])
def test_dense_product_and_column_ranges(n, cin, cout):
    """1x1x1 layers, and a layer that reads and writes column ranges of wider matrices."""
    from pcengine_b200 import functional as PF
    g = torch.Generator().manual_seed(n)
    x, w = torch.randn(n, cin, generator=g).half(), (torch.randn(cin, cout, generator=g) / cin ** 0.5).half()
    got, other = _both(lambda: PF.linear_forward(x.cuda(), w.cuda(), None))
    assert co.rel_l2(got.float().cpu(), x.float() @ w.float()) <= 5e-4 and torch.equal(got, other)
    coords = np.ascontiguousarray(surface_cloud(9, int(n ** 0.5 * 1.2) + 2)[:n])
    d2, csr = _map(coords)
    w3 = (torch.randn(27, cin, cout, generator=g) / (27 * cin) ** 0.5).half()
    wide_in, wide_out = torch.full((n, cin + 24), 9.0).half().cuda(), torch.full((n, cout + 40), 7.0).half().cuda()
    wide_in[:, 8:8 + cin] = x.cuda()
    PF.conv_forward(wide_in[:, 8:8 + cin], w3.cuda(), csr, out=wide_out[:, 16:16 + cout])
    assert co.rel_l2(wide_out[:, 16:16 + cout].float().cpu(), co.conv_forward(x, w3, d2)) <= 5e-4
    assert bool((wide_out[:, :16] == 7).all()) and bool((wide_out[:, 16 + cout:] == 7).all())


def test_values_of_absent_rows_do_not_leak():
    """Infinities and NaN of rows that a tile fetches stay with the rows whose neighbours they are."""
    from pcengine_b200 import functional as PF
    coords = np.ascontiguousarray(random_cloud(3, 30, 4000, batch=1))
    n = len(coords)
    d2, csr = _map(coords)
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(n, 64, generator=g).half(), (torch.randn(27, 64, 64, generator=g) / 41).half()
    x[::97] = float("inf")
    got = PF.conv_forward(x.cuda(), w.cuda(), csr).float().cpu()
    want = co.conv_forward(x, w, d2)
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    ok = torch.isfinite(want).all(1)
    assert co.rel_l2(got[ok], want[ok]) <= 5e-4


# the limits of the rule for 32 input channels: one, three and five tiles per SM, widths, and layers between two levels
@pytest.mark.parametrize("way,n,cout,kernel", [
    ("up", 129, 48, "umma"), ("up", 129, 64, "deep"), ("up", 20000, 64, "umma"), ("up", 20000, 192, "umma"), ("up", 20000, 208, "deep"),
    ("down", 20000, 48, "umma"), ("down", 20000, 64, "deep"), ("down", 40000, 64, "umma"),
    ("same", 30000, 16, "deep"), ("same", 94720, 32, "deep"), ("same", 94721, 32, "umma"), ("same", 94721, 48, "deep")])
def test_narrow_layers_run_on_the_faster_kernel(way, n, cout, kernel):
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    coords = np.ascontiguousarray(surface_cloud(9, int(n ** 0.5 * 1.2) + 2)[:n])
    ks, st, same = (3, 1, True) if way == "same" else (2, 2, False)
    d2 = ko.build_d2(coords, (ks,) * 3, (st,) * 3, (0,) * 3, [0] * 3, cmax_of(coords), same)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), (ks,) * 3, (st,) * 3, (0,) * 3, [0] * 3, d2["cmax_out"], same)
    csr = km.csr(transposed=way == "up")
    g = torch.Generator().manual_seed(n + cout)
    x, w = torch.randn(csr.n_src, 32, generator=g).half(), (torch.randn(ks ** 3, 32, cout, generator=g) / (ks ** 3 * 32) ** 0.5).half()
    xd, wd = x.cuda(), w.cuda()
    got = PF.conv_forward(xd, wd, csr)
    assert co.rel_l2(got.float().cpu(), co.conv_forward(x, w, d2, transposed=way == "up")) <= 5e-4
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        (name, _), = launches(lambda: PF.conv_forward(xd, wd, csr))
        assert "k_conv_" + kernel in name
    assert PF.device_status() == 0
