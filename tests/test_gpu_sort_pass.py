"""The pair sort's one-sweep passes at the edges of its tiles and of its tile sizes, on keys of a
single digit, two digits and random ones: whole numbers, equal to numpy's stable sort."""
import numpy as np
import pytest

from non_ficks_diffusion_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 2047, 2048, 2049, 500000, 500001, (1 << 20) - 1])
@pytest.mark.parametrize("kind", ["one", "two", "random"])
def test_sort_passes_match_numpy(built_lib, n, kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    keys = {"one": np.full(n, 0x5A5A5A, np.uint32), "two": rng.integers(0, 2, n).astype(np.uint32) * 0x0100FF,
            "random": rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)}[kind]
    kin = torch.from_numpy(keys.view(np.int32)).cuda()
    kout, vout = torch.empty_like(kin), torch.empty(n, dtype=torch.int32, device="cuda")
    assert capi.lib().mpm_sort_pairs_noalloc(kin.data_ptr(), None, kout.data_ptr(), vout.data_ptr(), n, 0, 24, None) == capi.OK
    torch.cuda.synchronize()
    perm = np.argsort(keys & 0xFFFFFF, kind="stable")
    assert np.array_equal(kout.cpu().numpy().view(np.uint32), keys[perm])
    assert np.array_equal(vout.cpu().numpy(), perm.astype(np.int32))
