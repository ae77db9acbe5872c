"""Pool digests on both sides of the lines between the kernel that takes a byte a
thread and the one that takes 16 bytes of up to 64 pools: 128 KiB in all, 32 KiB
a pool, 4 MiB in all.  Tails of 0 to 15 bytes, equal, sparsely and wholly
different pools, bytes of 0x80 and above, against a NumPy sum of the same mix."""
import ctypes as C

import numpy as np
import pytest

from tests.test_pool_digest import _digests
from toucangpurt_gb300 import capi

pytestmark = pytest.mark.gpu

K = 1024


@pytest.mark.parametrize("n,size", [
    (1, 128 * K), (1, 128 * K + 1), (1, 128 * K + 31), (2, 64 * K), (2, 64 * K + 15), (5, 32 * K), (5, 32 * K + 1),
    (7, 32 * K + 16), (8, 32 * K + 17), (9, 40 * K + 3), (17, 33 * K), (63, 33 * K + 8), (64, 40 * K), (65, 33 * K + 5),
    (130, 32 * K + 9), (128, 32 * K), (129, 32 * K), (1023, 4 * K), (1025, 4 * K), (1100, 4 * K - 1), (4096, K + 2)])
@pytest.mark.parametrize("fill", ["equal", "sparse", "dense", "bytes"])
def test_both_kernels(built, n, size, fill):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(size + n)
    host = np.repeat(rng.integers(0, 16, (1, size)).astype(np.uint8), n, axis=0)
    if fill == "equal":
        host[n // 2, size // 2] ^= 1
    elif fill == "sparse":
        for k in range(n):
            at = rng.integers(0, size, max(1, size // 100))
            host[k, at] = rng.integers(0, 16, at.size)
            host[k, size - 1] ^= k & 15
    else:
        host = rng.integers(0, 256 if fill == "bytes" else 16, (n, size)).astype(np.uint8)
    stride = (size + 15) // 16 * 16
    dev = torch.zeros((n, stride), dtype=torch.uint8, device="cuda:0")
    dev[:, :size] = torch.from_numpy(host).to("cuda:0")
    torch.cuda.synchronize()
    got = np.zeros(n, np.uint64)
    capi.check(capi.lib().tgs_pool_digests_noalloc(C.c_void_p(dev.data_ptr()), stride, size, n,
                                                   got.ctypes.data_as(capi.u64p)))
    np.testing.assert_array_equal(got, _digests(host))
