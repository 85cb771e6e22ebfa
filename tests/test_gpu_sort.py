"""Trees over the sizes at which the sorts and scans change form: one CTA, clusters of 2 to 16,
tiles of 2,048 and 4,096, and their remainders; against the oracle's tree (bit-exact lists)."""
import numpy as np
import pytest

import ogx_ic
from helpers import assert_same_tree_arrays, canonical_rank

pytestmark = pytest.mark.gpu


# 1,024 items per CTA up to 8,192, 2,048 up to 32,768, 4,096 up to 65,536, tiles of 2,048 up to
# 606,208, then 4,096
@pytest.mark.parametrize("n", [33, 1023, 1025, 4097, 8192, 8193, 16385, 32767, 32769, 65535, 65536, 65537, 131073, 606209])
def test_tree_matches_the_oracle(ogx, oracle, n):
    rng = np.random.Generator(np.random.PCG64(n))
    pos = rng.standard_normal((n, 3)) * rng.random((n, 1)) ** 3   # clustered, no velocities needed
    ref = oracle.tree(pos, 64)
    with ogx.AdaptiveFMM3D(p=1, threshold=64) as s:
        s.compute_accelerations(pos, np.ones(n))
        got = s.tree()
    assert_same_tree_arrays(ref, got, f"n={n}")


def test_deep_cluster_takes_all_key_levels(ogx, oracle):
    # a clump below level 16: the full 72-bit sort, one and several CTAs
    for n in (3000, 40000, 140000):
        pos, _, _ = ogx_ic.plummer(n, seed=n)
        pos[: n // 3] = 0.3 + 1e-6 * pos[: n // 3]
        ref = oracle.tree(pos, 32)
        with ogx.AdaptiveFMM3D(p=1, threshold=32) as s:
            s.compute_accelerations(pos, np.ones(n))
            got = s.tree()
        assert_same_tree_arrays(ref, got, f"deep n={n}")


# boxes and leaves up to 4,096 in one scan tile, up to 131,072 in the one-launch scan, above
# that in two launches
@pytest.mark.parametrize("n, thr, boxes", [(3001, 1, (4097, 8192)), (40009, 2, (32769, 131072)), (130003, 2, (131073, 400000))])
def test_scans_of_many_boxes(ogx, oracle, n, thr, boxes):
    rng = np.random.Generator(np.random.PCG64(n))
    pos = rng.random((n, 3))
    ref = oracle.tree(pos, thr)
    assert boxes[0] <= len(ref["boxes"]) <= boxes[1]
    with ogx.AdaptiveFMM3D(p=1, threshold=thr) as s:
        s.compute_accelerations(pos, np.ones(n))
        got = s.tree()
    assert_same_tree_arrays(ref, got, f"n={n} thr={thr}")
