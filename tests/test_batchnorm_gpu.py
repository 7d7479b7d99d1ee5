"""The one-pass BatchNorm / affine kernel against PyTorch in fp32: channel counts that do and do not divide a 16-byte
piece, element counts that end inside one, the widest constants it stages and the width above that, and rows that do
not start on a 16-byte boundary."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float16, 1e-3), (torch.float32, 1e-6)])
@pytest.mark.parametrize("n,c", [(1, 3), (7, 8), (1000, 19), (4097, 96), (3, 4096), (2, 4100)])
def test_batchnorm_in_one_pass(n, c, dtype, tol):
    import pcengine_b200 as pce
    from pcengine_b200 import functional as PF
    g = torch.Generator().manual_seed(n * c)
    bn = pce.BatchNorm(c)
    for t, lo in ((bn.running_mean, -1.0), (bn.running_var, 0.5), (bn.weight.data, 0.5), (bn.bias.data, -1.0)):
        t.copy_(lo + torch.rand(c, generator=g))
    bn = bn.to(dtype).cuda().eval()
    x = torch.randn(n, c, generator=g).to(dtype).cuda()
    ref = torch.nn.functional.batch_norm(x.float(), bn.running_mean.float(), bn.running_var.float(), bn.weight.float(),
                                         bn.bias.float(), False, 0.0, bn.eps)
    coords = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    y = bn(pce.spTensor(x, coords, coords_max=[0, 0, 0])).feats
    assert y.dtype == dtype and float((y.float() - ref).norm() / ref.norm()) <= tol
    odd = torch.empty(n * c + 1, dtype=dtype, device="cuda")[1:].view(n, c).copy_(x)  # off a 16-byte boundary
    z = bn(pce.spTensor(odd, coords, coords_max=[0, 0, 0])).feats
    assert float((z.float() - ref).norm() / ref.norm()) <= tol
    res = torch.randn(n, c, generator=g).to(dtype).cuda()
    s, t = pce.bn_scale_shift(bn)
    w = PF.scale_shift_act(x, PF.FusedEpilogue(scale=s, shift=t, residual=res, act="leaky"))
    full = torch.nn.functional.leaky_relu(ref + res.float(), 0.01)
    assert float((w.float() - full).norm() / full.norm()) <= tol
