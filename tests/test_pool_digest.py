"""State digests of pools: the digest kernels take 16 bytes of up to eight
pools at a time (equal pools share a sum), single bytes at the tail, for
values that carry out of the low byte and for unaligned pools.  Checked
against a NumPy sum of the same mix."""
import ctypes as C

import numpy as np
import pytest

from toucangpurt_gb300 import capi, sim

pytestmark = pytest.mark.gpu


def _digests(pools):
    i = np.arange(pools.shape[1], dtype=np.uint64) << np.uint64(8)
    with np.errstate(over="ignore"):
        return np.array([sim.mix64(i | p.astype(np.uint64)).sum(dtype=np.uint64) for p in pools], np.uint64)


# tails of 0..15 bytes; 4 MiB and more, where the bits above 2^30 of the mixed
# index change inside a 16-byte vector; 1, 7, 8, 9 and 17 pools
@pytest.mark.parametrize("size", [1, 15, 16, 17, 4099, (1 << 22) + 5])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 17, 130])
@pytest.mark.parametrize("fill", ["equal", "sparse", "nibbles", "bytes"])
@pytest.mark.parametrize("offset", [0, 3])
def test_pool_digests(built, size, n, fill, offset):
    torch = pytest.importorskip("torch")
    if size > 1 << 20 and (n not in (1, 9) or fill == "equal"):
        pytest.skip("the long pool with two pool counts only")
    rng = np.random.default_rng(size + n)
    host = rng.integers(0, 256 if fill == "bytes" else 16, (n, size)).astype(np.uint8)
    if fill == "sparse":  # equal but for a few bytes of every pool, several in one 16-byte piece among them
        host[:] = host[0]
        for k in range(n):
            at = rng.integers(0, size, max(1, size // 40))
            host[k, at] = rng.integers(0, 256, at.size)
            host[k, size // 3:size // 3 + 5] ^= k
    if fill == "equal":
        host[:] = host[0]
        host[n // 2, size // 2] ^= 1
    stride = (size + 15) // 16 * 16 + (16 if offset == 0 else 5)
    dev = torch.zeros(offset + n * stride, dtype=torch.uint8, device="cuda:0")
    for k in range(n):
        dev[offset + k * stride:offset + k * stride + size] = torch.from_numpy(host[k])
    torch.cuda.synchronize()
    got = np.zeros(n, np.uint64)
    capi.check(capi.lib().tgs_pool_digests_noalloc(C.c_void_p(dev.data_ptr() + offset), stride, size, n,
                                                   got.ctypes.data_as(capi.u64p)))
    np.testing.assert_array_equal(got, _digests(host))
