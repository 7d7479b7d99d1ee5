"""Device voxelisation and collation against the host path: point counts around a block's chunk and each number of
points per thread of the cooperative kernel, above what it holds, key widths from none to three full axes, negative
voxels, and more samples than one collation launch takes."""
import numpy as np
import pytest
import torch

from tests.helpers import traced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extent", [(1, 0.0), (511, 1.0), (1024, 3.0), (1025, 400.0), (151552, 30.0), (151553, 3000.0),
                                      (400000, 8.0), (900000, 100.0), (1212417, 20.0)])
def test_device_voxelisation_equals_the_host_path(n, extent):
    import pcengine_b200 as pce
    rng = np.random.default_rng(n)
    pts = ((rng.uniform(size=(n, 3)) - 0.5) * extent).astype(np.float32)
    voxel = float(np.float32(0.125))
    want = pce.sparse_quantize(pts, voxel, return_index=True, return_inverse=True)
    got = pce.sparse_quantize(torch.from_numpy(pts).cuda(), voxel, return_index=True, return_inverse=True)
    assert [t.dtype for t in got] == [torch.int32, torch.int64, torch.int64]
    for a, b in zip(got, want):
        assert np.array_equal(a.cpu().numpy(), b)
    alone = pce.sparse_quantize(torch.from_numpy(pts).cuda(), voxel)
    assert np.array_equal(alone.cpu().numpy(), want[0])


@pytest.mark.parametrize("k,width", [(1, 3), (3, 4), (65, 3), (130, 4)])
def test_device_collation_equals_the_host_path(k, width):
    import pcengine_b200 as pce
    rng = np.random.default_rng(k)
    coords = [torch.from_numpy(rng.integers(-50, 900, (int(rng.integers(0, 400)) + (i == 0), width)).astype(np.int32)) for i in range(k)]

    def batch(dev):
        return pce.sparse_collate([pce.spTensor(torch.full((len(c), 2), float(i)).to(dev), c.to(dev), coords_max=[0, 0, 0])
                                   for i, c in enumerate(coords)])
    a, b = batch("cuda"), batch("cpu")
    assert torch.equal(a.coords.cpu(), b.coords) and torch.equal(a.feats.cpu(), b.feats)
    assert a.coords_max == b.coords_max and a.batchsize == k


@pytest.mark.parametrize("n,kind", [(4097, "one voxel"), (9000, "two voxels"), (70000, "wide"), (100000, "sorted"), (100000, "lines"),
                                    (151552, "one voxel"), (90000, "a third in one voxel"), (100000, "hundred voxels"), (100000, "misjudged")])
def test_voxelisation_by_buckets(n, kind):
    """Voxels of more points than a bucket holds, clouds that miss the buckets (key and index beyond a word, points that no
    sample stands for) and clouds in orders that a sample at equal distances could misjudge."""
    import pcengine_b200 as pce
    rng = np.random.default_rng(n)
    pts = rng.uniform(-40, 40, (n, 3))
    if kind == "one voxel":
        pts = rng.uniform(0.01, 0.11, (n, 3))
    elif kind == "two voxels":
        pts = rng.uniform(0.01, 0.11, (n, 3)) + 0.125 * (np.arange(n) % 2)[:, None]
    elif kind == "wide":
        pts *= 90
    elif kind == "sorted":
        pts = pts[np.lexsort(pts.T[::-1])]
    elif kind == "lines":  # every 98th point, the distance of the samples, lies on one line
        pts[n // 2048::n // 1024, :2] = 0.5
    elif kind == "a third in one voxel":  # (in places all over the cloud)
        pts[rng.permutation(n)[:n // 3]] = 0.06
    elif kind == "hundred voxels":
        pts = rng.uniform(0.01, 0.11, (n, 3)) + 0.125 * rng.integers(0, 100, n)[:, None]
    elif kind == "misjudged":  # every point that the samples are taken from lies in front of all others
        pts[:, 0] = 20 + pts[:, 0] / 4
        pts[(np.arange(1024) * n + n // 2) // 1024, 0] = -30
    pts = pts.astype(np.float32)
    voxel = float(np.float32(0.125))
    want = pce.sparse_quantize(pts, voxel, return_index=True, return_inverse=True)
    got = pce.sparse_quantize(torch.from_numpy(pts).cuda(), voxel, return_index=True, return_inverse=True)
    for a, b in zip(got, want):
        assert np.array_equal(a.cpu().numpy(), b)
    names = [e["name"] for e in traced(lambda: pce.sparse_quantize(torch.from_numpy(pts).cuda(), voxel))]
    assert any("k_voxelise_buckets" in name for name in names)
    assert any("k_voxelise<" in name for name in names) == (kind in ("wide", "misjudged"))
