"""Calls that read sizes back, from threads that come and go (GPU)."""
import re
import threading

import pytest
import torch

from tests.helpers import cmax_of, random_cloud

pytestmark = pytest.mark.gpu


def test_short_threads_leave_nothing_behind():
    """Every thread's pinned words and events go with it: 300 threads of four such calls each leave the process where the
    100 before them did (kept, they were 6.6 KB a thread, 2 MB here), and the results are those of the main thread."""
    import pcengine_b200 as pce
    coords = random_cloud(1, 16, 500)
    cd, pts, cm = torch.from_numpy(coords).cuda(), torch.rand(300, 3, device="cuda"), cmax_of(coords)
    seen = []

    def work():
        voxels = pce.sparse_quantize(pts, 0.1)
        batch = pce.sparse_collate([pce.spTensor(torch.zeros(500, 1, device="cuda"), cd, coords_max=cm)] * 2)
        halves = pce.KernelMap(cd, (2,) * 3, (2,) * 3, (0,) * 3, [0] * 3, [(v - 1) // 2 for v in cm], False)
        strided = pce.KernelMap(cd, (3,) * 3, (2,) * 3, (0,) * 3, [0] * 3, [(v - 2) // 2 for v in cm], False)
        seen.append((len(voxels), batch.coords_max, halves.n_out, strided.n_out))

    def resident():
        return int(re.search(r"VmRSS:\s+(\d+)", open("/proc/self/status").read()).group(1))

    def run(n):
        for _ in range(n):
            t = threading.Thread(target=work)
            t.start()
            t.join()
    work()
    run(100)
    before = resident()
    run(300)
    assert resident() - before < 1000
    assert len(seen) == 401 and all(s == seen[0] for s in seen)
