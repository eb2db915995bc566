"""One workspace serves every sort up to the size it was made for: its size
never falls as the number of pairs grows (the sort takes shorter partitions, so
more descriptors, where it is short), and smaller sorts run in the workspace of
the largest, bit for bit as in their own."""
import ctypes as C

import numpy as np
import pytest

from torpedo_gb300 import _lib as L

# the sizes at which the sort changes its form or its partitions, and a step to either side
EDGES = [1, 4096, 12288, 12289, 65536, 131072, 131073, 200_000, 262_144, 524_288, 524_289, 600_000, 1 << 20,
         2_000_001, 1 << 24, (1 << 31) - 1]


def test_size_never_falls():
    lib = L.load()
    sizes = sorted({max(1, n + d) for n in EDGES for d in (-1, 0, 1) if n + d < 1 << 31})
    got = [int(lib.tpd_sort_workspace_size(n)) for n in sizes]
    falls = [(sizes[i], got[i], sizes[i + 1], got[i + 1]) for i in range(len(got) - 1) if got[i + 1] < got[i]]
    assert not falls, falls


@pytest.mark.gpu
@pytest.mark.parametrize("largest", [200_000, 600_000])
def test_smaller_sorts_in_the_largest_workspace(cuda, largest):
    torch = cuda
    lib = L.load()
    ws = torch.empty(int(lib.tpd_sort_workspace_size(largest)), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(largest)
    for n in sorted({min(n, largest) for n in (1, 12_288, 12_289, 131_072, 131_073, 524_288, 524_289, largest)}):
        keys = rng.integers(0, 1 << 45, size=n, dtype=np.uint64)
        k = torch.from_numpy(keys.view(np.int64)).cuda()
        v = torch.arange(n, dtype=torch.int32, device="cuda")
        ka, va = torch.empty_like(k), torch.empty_like(v)
        alt = C.c_int(0)
        rc = lib.tpd_sort_pairs(k.data_ptr(), v.data_ptr(), ka.data_ptr(), va.data_ptr(), n, 45, ws.data_ptr(),
                                ws.numel(), stream, C.byref(alt))
        assert rc == L.TPD_OK, (n, L.status_string(rc))
        torch.cuda.synchronize()
        assert int(ws[:4].view(torch.int32).item()) == 0
        order = np.argsort(keys, kind="stable")
        np.testing.assert_array_equal((va if alt.value else v).cpu().numpy(), order)
        np.testing.assert_array_equal((ka if alt.value else k).cpu().numpy().view(np.uint64), keys[order])
