"""Kernel maps in block form (table of 4x4x4 blocks, row order and tile lists in one launch) against the oracle (GPU)."""
import numpy as np
import pytest
import torch

from oracle import kmap_oracle as ko
from tests.helpers import cmax_of, random_cloud, surface_cloud

pytestmark = pytest.mark.gpu


def _cloud(kind, n):
    if kind == "sheet":
        c = surface_cloud(5, int(n ** 0.5 * 1.2) + 2)[:n]
    elif kind == "alone":  # every voxel in a block of its own: more coarse blocks than their table is sized for
        i = np.arange(n)
        c = np.stack([0 * i, i % 40 * 9, i // 40 % 40 * 9, i // 1600 * 9], 1).astype(np.int32)
    else:
        c = random_cloud(6, 40, n, batch=1)[:n]
        c[:, 1:] -= 17  # negative coordinates
    return np.ascontiguousarray(c), [min(0, int(v)) for v in c[:, 1:].min(0)]


def _expect_lists(csr, nb, kv):
    """The row order is the stable sort by bitmask with the rarest offset on top; the lists hold the order's neighbours."""
    n = nb["n_out"]
    rp = nb["rowptr"].astype(np.int64)
    table = -np.ones((n, kv), np.int64)
    bits = ((nb["mask"][:n, :, None] >> np.arange(32, dtype=np.uint32)) & 1).reshape(n, -1)[:, :kv].astype(bool)
    table[bits] = nb["nbr"][: rp[-1]]  # rows ascending, offsets ascending
    csr.tiles()
    _, order, tile_ptr, stage_kp, stage_nbr = csr._tiles[(True, 128, False, 1)]
    order, tile_ptr = order.cpu().numpy(), tile_ptr.cpu().numpy()
    if kv <= 32:
        rank = np.argsort(np.argsort(bits.sum(0), kind="stable"), kind="stable")
        key = (bits.astype(np.int64) << (kv - 1 - rank)).sum(1)
        assert np.array_equal(order, np.argsort(key, kind="stable"))
    stages = int(tile_ptr[-1])
    stage_kp, stage_nbr = stage_kp.cpu().numpy()[:stages] & 255, stage_nbr.cpu().numpy().reshape(-1, 128)[:stages]
    for t in range((n + 127) // 128):
        rows = order[t * 128: (t + 1) * 128]
        present = np.nonzero((table[rows] >= 0).any(0))[0]
        a, b = tile_ptr[t], tile_ptr[t + 1]
        assert np.array_equal(stage_kp[a:b], present)
        assert np.array_equal(stage_nbr[a:b, : len(rows)], table[rows][:, present].T)
        assert (stage_nbr[a:b, len(rows):] == -1).all()


@pytest.mark.parametrize("kind,n,ks", [("sheet", 1, 3), ("sheet", 127, 3), ("sheet", 128, 5), ("random", 129, 3), ("alone", 4097, 3),
                                       ("random", 6000, (3, 1, 5)), ("sheet", 24576, 3), ("sheet", 24577, 3), ("sheet", 65537, 3)])
def test_submanifold_lists(kind, n, ks):
    import pcengine_b200 as pce
    ks = (ks,) * 3 if isinstance(ks, int) else ks
    coords, cmin = _cloud(kind, n)
    d2 = ko.build_d2(coords, ks, (1, 1, 1), (0, 0, 0), cmin, cmax_of(coords), True)
    nb, kv = ko.neighbour_csr(d2), int(np.prod(ks))
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), ks, (1, 1, 1), (0, 0, 0), cmin, cmax_of(coords), True)
    csr = km.csr()
    starts, nbr = (v.cpu().numpy() for v in csr.row_lists())
    assert np.array_equal(csr.mask.cpu().numpy().view(np.uint32), nb["mask"])
    rp = nb["rowptr"]
    for r in range(0, len(coords), max(1, len(coords) // 500)):
        assert np.array_equal(nbr[starts[r]: starts[r] + rp[r + 1] - rp[r]], nb["nbr"][rp[r]: rp[r + 1]])
    assert km.sizes() == (len(d2["imap"]), d2["qsum"]) and int(csr.pair_count()) == int(rp[-1])
    _expect_lists(csr, nb, kv)


@pytest.mark.parametrize("kind,n,ks", [("sheet", 127, 2), ("random", 3000, 2), ("sheet", 30000, 2), ("alone", 4097, 2), ("random", 2000, 3)])
def test_parents_of_voxels(kind, n, ks):
    import pcengine_b200 as pce
    coords, cmin = _cloud(kind, n)
    args = ((ks,) * 3, (ks,) * 3, (0, 0, 0), cmin)
    d2 = ko.build_d2(coords, *args, cmax_of(coords), False)
    km = pce.KernelMap(torch.from_numpy(coords).cuda(), *args, d2["cmax_out"], False)
    assert np.array_equal(km.out_coords.cpu().numpy(), d2["out_coords"].reshape(-1, 4))
    for transposed in (False, True):
        _expect_lists(km.csr(transposed=transposed), ko.neighbour_csr(d2, transposed=transposed), ks ** 3)


@pytest.mark.parametrize("n,stride", [(1, 1), (511, 1), (4097, 2), (40000, 1)])
def test_gather_scatter_codes(n, stride):
    import pcengine_b200 as pce
    coords, cmin = _cloud("sheet", n)
    args = ((3,) * 3, (stride,) * 3, (0, 0, 0), cmin)
    d2 = ko.build_d2(coords, *args, cmax_of(coords), stride == 1)
    want = ko.build_d1(d2)
    got = pce.KernelMap(torch.from_numpy(coords).cuda(), *args, d2["cmax_out"], stride == 1).d1()
    for name, t in zip(("imap", "icsr", "omap", "ocsr"), got):
        assert np.array_equal(t.cpu().numpy(), want[name])


def test_chain_given_up_while_it_is_built():
    """60 000 voxels with a coarse block each: the coarse tables fill up while other warps still insert, the chain is given
    up and the levels are found one by one.  Planned and lazy passes agree bit for bit, pass after pass."""
    import pcengine_b200 as pce
    coords, cmin = _cloud("alone", 60000)
    cd, x0 = torch.from_numpy(coords).cuda(), torch.randn(len(coords), 16, generator=torch.Generator().manual_seed(2)).half().cuda()
    layers = [(3, 1), (2, 2), (3, 1), (2, 2), (3, 1)]
    torch.manual_seed(3)
    convs = [pce.conv3d(16, 16, k, s).cuda().half() for k, s in layers]
    plan = pce.MapPlan([(k, s, False, 16, 16) for k, s in layers])
    outs = []
    for planned in (False, True, True):
        x = pce.spTensor(x0, cd, None, cmin, cmax_of(coords), init_tag=["D2"] * 5)
        assert plan.begin(x) if planned else True
        with torch.no_grad():
            for conv in convs:
                x = conv(x)
        outs.append((x.feats, x.coords))
    for feats, out_coords in outs[1:]:
        assert torch.equal(feats, outs[0][0]) and torch.equal(torch.as_tensor(out_coords), outs[0][1])
    del x, outs
    plan.close()


def _mix64(k):
    with np.errstate(over="ignore"):
        k = k ^ (k >> np.uint64(33))
        k = k * np.uint64(0xff51afd7ed558ccd)
        k = k ^ (k >> np.uint64(33))
        k = k * np.uint64(0xc4ceb9fe1a85ec53)
        return k ^ (k >> np.uint64(33))


@pytest.mark.parametrize("rows,kv", [(1, 65), (257, 75), (5000, 125), (4096, 128)])
def test_row_order_beyond_64_offsets(rows, kv):
    """The stable sort by (rank of the set of the four rarest offsets, hash of the bitmask): empty rows, rows with fewer
    than four offsets, rows with all of them."""
    from math import comb
    from pcengine_b200.kmap import NeighbourCSR
    rng = np.random.default_rng(rows)
    bits = rng.random((rows, kv)) < rng.choice([0.0, 0.01, 0.05, 0.5, 1.0], (rows, 1))
    words = (kv + 31) // 32
    mask = np.packbits(np.pad(bits, ((0, 0), (0, 32 * words - kv))), axis=1, bitorder="little").view(np.uint32)
    csr = NeighbourCSR(torch.from_numpy(mask.view(np.int32)).cuda(), None, None, rows, rows, kv)
    order = csr.order().cpu().numpy()
    place = kv - 1 - np.argsort(np.argsort(bits.sum(0), kind="stable"), kind="stable")
    permuted = np.zeros((rows, 128), bool)
    permuted[:, place] = bits
    halves = np.packbits(permuted, axis=1, bitorder="little").view(np.uint64)
    hashes = _mix64(halves[:, 0] ^ _mix64(halves[:, 1])) >> np.uint64(32)
    sets = np.zeros(rows, np.uint64)
    for r in range(rows):
        for q, p in enumerate(np.nonzero(permuted[r])[0][::-1][:4]):
            sets[r] += np.uint64(sum(comb(int(p), i) for i in range(5 - q)))
    key = sets * np.uint64(389) + (hashes * np.uint64(389) >> np.uint64(32))
    assert key.max() < 1 << 32 and np.array_equal(order, np.argsort(key, kind="stable"))


@pytest.mark.parametrize("n", [255, 257, 400000])
def test_table_in_one_launch(n):
    """Presence and neighbours of a cloud of fewer voxels than a block's threads, and of more than a resident grid's, against
    sorted keys."""
    import pcengine_b200 as pce
    g = torch.Generator("cuda").manual_seed(n)
    side = 1 << 10
    lin = torch.randperm(side * side, generator=g, device="cuda")[:n]
    x, y = lin // side, lin % side
    coords = torch.stack([lin % 3, x, y, (x + 2 * y) // 16], 1).int().contiguous()
    km = pce.KernelMap(coords, (3,) * 3, (1,) * 3, (0,) * 3, [0] * 3, coords[:, 1:].amax(0).tolist(), True)
    csr = km.csr()
    starts, nbr = csr.row_lists()
    key = lambda c: ((c[:, 0].long() * 2048 + c[:, 1] + 1) * 2048 + c[:, 2] + 1) * 2048 + c[:, 3] + 1
    keys, rows = torch.sort(key(coords))
    at = torch.zeros(n, dtype=torch.long, device="cuda")
    mask = csr.mask[:, 0].long()
    for kp in range(27):
        d = torch.tensor([0, kp // 9 - 1, kp // 3 % 3 - 1, kp % 3 - 1], device="cuda")
        want = key(coords + d)
        i = torch.searchsorted(keys, want).clamp_(max=n - 1)
        found = keys[i] == want
        assert torch.equal((mask >> kp & 1).bool(), found)
        assert torch.equal(nbr[(starts.long() + at)[found]].long(), rows[i[found]])
        at += found
