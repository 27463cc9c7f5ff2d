"""The sort over the widths of a key range (digits of up to eight bits, or of nine where that saves a pass) and on either side
of the sizes that choose the cluster, against a stable sort on the CPU."""
import numpy as np
import pytest
import torch

from oracle import oracle
from tests.util import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0, 1, 8, 9, 10, 16, 17, 18, 19, 24, 25, 26, 27, 28, 31, 32])
@pytest.mark.parametrize("nseg,n", [(3, 5000), (2, 8 * 4096 + 8)])
def test_key_widths(bits, nseg, n):
    import lampa_b200
    rng = np.random.default_rng(bits)
    k = rng.integers(0, 1 << bits, nseg * n, dtype=np.int64) - (1 << 31)
    for s in range(nseg):                                    # both ends of the range in every segment, and a few ties
        k[s * n] = -(1 << 31)
        k[s * n + 1] = (1 << bits) - 1 - (1 << 31)
        k[s * n + 2 : s * n + 40] = k[s * n + 40 : s * n + 78]
    k = k.astype(np.int32)
    init = np.concatenate([rng.permutation(n) for _ in range(nseg)]).astype(np.int64)
    seg = (np.arange(nseg + 1) * n).astype(np.int64)
    kd = torch.from_numpy(k).cuda()
    np.testing.assert_array_equal(to_np(lampa_b200.segmented_sort(kd, nseg=nseg)), oracle.segsort(k, seg))
    np.testing.assert_array_equal(to_np(lampa_b200.segmented_sort(kd, nseg=nseg, init=torch.from_numpy(init).cuda())), oracle.segsort(k, seg, init=init))


@pytest.mark.parametrize("nseg,n", [(1, 8 * 4096), (1, 8 * 4096 + 1), (1, 200001), (9, 33000), (10, 40000)])
def test_float_keys_and_cluster_sizes(nseg, n):
    import lampa_b200
    rng = np.random.default_rng(n)
    k = (rng.random(nseg * n) * 100 + 1).astype(np.float32)
    k[::1000] = np.inf
    k[1::5000] = -3.0
    np.testing.assert_array_equal(to_np(lampa_b200.segmented_sort(torch.from_numpy(k).cuda(), nseg=nseg)), oracle.segsort(k, (np.arange(nseg + 1) * n).astype(np.int64)))
