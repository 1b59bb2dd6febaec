"""Reads of a batch's fields share one staging buffer, as large as the largest member's."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 8])
def test_reads_of_all_members_from_several_threads(threads):
    import optimizec_b200 as P

    # the smallest member first: the buffer has to be large enough for all from the first read on
    members = [(N, 1e4, 4.0, 0.1, 3 + i) for i, N in enumerate([32, 64, 512, 128, 256, 64, 512, 32])]
    b = P.Batch(members)
    b.init_k4()
    with ThreadPoolExecutor(threads) as pool:
        got = list(pool.map(b.om2, list(range(len(members))) * 4))
    b.close()
    for i, om in enumerate(got):
        N, _, K0, _, seed = members[i % len(members)]
        np.testing.assert_array_equal(om, P.k4_spectrum(N, K0, seed))
