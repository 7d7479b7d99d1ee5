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
    csr.lists_fp32()
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


def test_tiled_fp32_beyond_65535_row_blocks():
    """More rows than 65535 blocks of 32 (lists) and of 128 (dense product), which the kernel of one thread group per
    row always took.  Bound: two fp32 sums of at most 27 * 28 products in different orders."""
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    n = 65535 * 32 + 33
    lin = torch.randperm(256 * 256 * 64, device="cuda", generator=torch.Generator("cuda").manual_seed(0))[:n]
    coords = torch.stack([0 * lin, lin // (256 * 64), lin // 64 % 256, lin % 64], 1).int().contiguous()
    km = pce.KernelMap(coords, (3, 3, 3), (1, 1, 1), (0, 0, 0), [0, 0, 0], [255, 255, 63], True)
    x, w = torch.randn(n, 28, device="cuda"), torch.randn(27, 28, 28, device="cuda")
    got = PF.conv_forward(x, w, km.csr())
    want = PF.conv_forward(x, w, km.csr(), kernel_choice="simt")
    for part in (slice(0, n // 2), slice(n // 2, n), slice(n - 40, n)):
        assert float((got[part] - want[part]).norm() / want[part].norm()) <= 1e-5
    del got, want
    x = torch.randn(65535 * 128 + 129, 28, device="cuda")
    got = PF.linear_forward(x, w[0].contiguous())
    for part in (slice(0, 1 << 20), slice(len(x) - 140, len(x))):
        want = x[part].double() @ w[0].double()
        assert float((got[part] - want).norm() / want.norm()) <= 1e-5
    whole = x @ w[0]  # (another fp32 order)
    assert float((got - whole).norm() / whole.norm()) <= 1e-5


@pytest.mark.parametrize("ks,stride,transposed,cin,cout", [(3, 1, False, 4, 32), (3, 1, False, 32, 16), (3, 1, False, 64, 8),
                                                           (5, 1, False, 16, 16), (2, 2, False, 32, 16), (2, 2, True, 24, 24),
                                                           (3, 2, False, 32, 16)])
def test_narrow_fp32_layers_do_not_depend_on_what_ran_before(ks, stride, transposed, cin, cout):
    """Fewer than 768 weights per offset: the same bits on a fresh map, on one where a wide layer has left tile lists,
    on one whose rowptr or dense table somebody asked for, and on a planned one with and without a wide layer."""
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    coords = random_cloud(3, 24, 3000)
    subm = stride == 1
    cmax = [c if subm else (c - (ks - 1)) // stride for c in cmax_of(coords)]
    cd = torch.from_numpy(coords).cuda()

    def fresh():
        return pce.KernelMap(cd, (ks,) * 3, (stride,) * 3, (0, 0, 0), [0, 0, 0], cmax, subm)
    n_src = fresh().csr(transposed).n_src
    g = torch.Generator().manual_seed(5)
    x, w = torch.randn(n_src, cin, generator=g).cuda(), torch.randn(ks ** 3, cin, cout, generator=g).cuda()
    first = PF.conv_forward(x, w, fresh().csr(transposed))

    def after_wide(km):
        PF.conv_forward(torch.zeros(n_src, 48, device="cuda"), torch.zeros(ks ** 3, 48, 48, device="cuda"), km.csr(transposed))
    for before in (after_wide, lambda km: km.csr(transposed).rowptr, lambda km: km.map,
                   lambda km: PF.conv_forward(x, w, km.csr(transposed), kernel_choice="simt")):
        km = fresh()
        before(km)
        assert torch.equal(PF.conv_forward(x, w, km.csr(transposed)), first)
    use, wide = (ks, stride, transposed, cin, cout), (ks, stride, transposed, 48, 48)
    down = (2, 2, False, 4, 4) if subm or transposed else use  # (ahead of a transposed use; behind a submanifold one: block form)
    for layers in ([use, down], [use, wide, down]) if subm else ([down, use], [down, use, down, wide]) if transposed else ([use],):
        plan = pce.MapPlan(layers, dtype=torch.float32)
        t = pce.spTensor(torch.zeros(len(coords), 4).cuda(), cd, None, [0, 0, 0], cmax_of(coords), init_tag=["D2"])
        assert plan.begin(t)
        csr = t.planner.fetch(t, next(iter(plan.index)), None).csr(transposed)
        assert torch.equal(PF.conv_forward(x, w, csr), first)
        del t, csr
        plan.close()


@pytest.mark.parametrize("cin,cout", [(4, 8), (16, 16), (48, 32)])
def test_fp32_layers_from_an_empty_level(cin, cout):
    """A cloud in one plane has no coarser level (the bounds leave it no outputs): the layer back up has rows and no
    inputs, and gives its bias."""
    import pcengine_b200 as pce
    coords = random_cloud(4, 12, 200)
    coords[:, 3] = 0
    coords = coords[sorted({tuple(c): i for i, c in enumerate(coords.tolist())}.values())]
    x = pce.spTensor(torch.randn(len(coords), cin).cuda(), torch.from_numpy(coords).cuda(), None, [0, 0, 0], cmax_of(coords), init_tag=["D2"])
    down, up = pce.conv3d(cin, cout, 2, 2).cuda(), pce.conv3d(cout, cin, 2, 2, bias=True, transposed=True).cuda()
    with torch.no_grad():
        y = down(x)
        z = up(y)
    assert y.feats.shape == (0, cout)
    assert torch.equal(z.feats, up.bias.expand(len(coords), cin))


@pytest.mark.parametrize("cin,cout,n", [(28, 28, 60), (28, 28, 400), (32, 32, 400), (64, 130, 400), (33, 24, 300)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_infinities_and_nans_stay_with_the_rows_that_meet_them(cin, cout, n, bad):
    """One weight, then one feature, that is not finite: exactly the outputs whose row has that offset (or that neighbour)
    are touched, as on the kernel of one thread group per row, in whole chains and in chains cut over a cluster."""
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    coords = random_cloud(n, 5 if n < 100 else 12, n)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), (3, 3, 3), (1, 1, 1), (0, 0, 0), [0, 0, 0], cmax_of(coords), True)
    g = torch.Generator().manual_seed(n + cin)
    x, w = torch.randn(n, cin, generator=g), torch.randn(27, cin, cout, generator=g)
    for t in (w.clone().index_put_((torch.tensor(3), torch.tensor(2), torch.tensor(1)), torch.tensor(bad)), w):
        y = x.clone()
        if t is w:
            y[17, 3] = bad
        got = PF.conv_forward(y.cuda(), t.cuda(), km.csr()).cpu()
        want = PF.conv_forward(y.cuda(), t.cuda(), km.csr(), kernel_choice="simt").cpu()
        ok = torch.isfinite(want)
        assert torch.equal(torch.isfinite(got), ok) and 0 < int((~ok).sum()) < ok.numel()
        assert torch.equal(torch.isnan(got), torch.isnan(want))
        assert float((got[ok] - want[ok]).norm() / want[ok].norm()) <= 1e-5
