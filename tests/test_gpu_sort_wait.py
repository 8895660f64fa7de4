"""The pair sort's look-back when waits give up: no tile publishes its words, so that every thread
counts its digit in all earlier tiles itself. Whole numbers, equal to numpy's stable sort, for one
tile, a few ragged ones and both tile sizes; and sorts recorded into a graph whose kernels the
first call did not run."""
import os
import subprocess
import sys

import numpy as np
import pytest

from non_ficks_diffusion_gb300 import capi

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("n", [1, 2048, 2049, 30001, 500001])
@pytest.mark.parametrize("bits", [(0, 8), (6, 30)])
def test_sort_without_published_words(built_lib, n, bits):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    keys[: n // 3] &= 0xFF00FF00
    vals = rng.integers(-(1 << 31), 1 << 31, n, dtype=np.int64).astype(np.int32)
    kin, vin = torch.from_numpy(keys.view(np.int32)).cuda(), torch.from_numpy(vals).cuda()
    kout, vout = torch.empty_like(kin), torch.empty_like(vin)
    args = (kin.data_ptr(), vin.data_ptr(), kout.data_ptr(), vout.data_ptr(), n) + bits
    assert capi.lib().mpm_selftest_sort_wait(*args, 1, None) == capi.OK
    torch.cuda.synchronize()
    perm = np.argsort((keys >> bits[0]) & ((1 << (bits[1] - bits[0])) - 1), kind="stable")
    assert np.array_equal(kout.cpu().numpy().view(np.uint32), keys[perm])
    assert np.array_equal(vout.cpu().numpy(), vals[perm])
    assert capi.lib().mpm_selftest_sort_wait(*args, 0, None) == capi.BAD_ARG
    assert capi.lib().mpm_selftest_sort_wait(*args, 1001, None) == capi.BAD_ARG


CAPTURE = """
import sys
import numpy as np, torch
from non_ficks_diffusion_gb300 import capi
first, n = int(sys.argv[1]), int(sys.argv[2])
L = capi.lib()
g = np.random.default_rng(0)
def arrays(m):
    k = g.integers(0, 1 << 24, m, dtype=np.int64).astype(np.int32)
    a = torch.from_numpy(k).cuda()
    return k, a, torch.empty_like(a), torch.empty_like(a)
k, a, ko, vo = arrays(first)
assert L.mpm_sort_pairs_noalloc(a.data_ptr(), None, ko.data_ptr(), vo.data_ptr(), first, 0, 24, None) == capi.OK
k, a, ko, vo = arrays(n)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    s = torch.cuda.current_stream().cuda_stream
    assert L.mpm_sort_pairs_noalloc(a.data_ptr(), None, ko.data_ptr(), vo.data_ptr(), n, 0, 24, s) == capi.OK
for _ in range(2):
    graph.replay()
torch.cuda.synchronize()
p = np.argsort(k, kind="stable")
assert np.array_equal(ko.cpu().numpy(), k[p]) and np.array_equal(vo.cpu().numpy(), p)
"""


@pytest.mark.parametrize("first,n", [(600000, 3000), (3000, 600000)])
def test_sort_under_capture(built_lib, first, n):
    pytest.importorskip("torch")
    subprocess.run([sys.executable, "-c", CAPTURE, str(first), str(n)], check=True, timeout=300, cwd=ROOT)
