"""The n-mer search where its staging in shared memory grows: match capacities
around the default limit of a block (48 KB), above it, and at the most a block
can have (GPU)."""
import numpy as np
import pytest

import mbx_oracle as mo
from mbx_b200 import batch, system as msys, workloads

pytestmark = pytest.mark.gpu

FAR = 400.0   # A: further than any two molecules of the clusters below


def waters(n):
    """n waters at the density of the liquid, without a box."""
    side = int(np.ceil((1.3 * n) ** (1 / 3)))
    ids, xyz, _ = workloads.water_box(side, n, 39.44 * (n / 2048) ** (1 / 3), seed=n)
    return ids, xyz


def all_pairs(n):
    return np.stack(np.triu_indices(n, 1), 1)


# A query with n matches (itself among them) above the capacity makes it
# max(2 x 192, n + 32).  64 bytes of staging per match and 1.2 KB beside it:
# 749 and 750 lie on either side of 48 KB in all, 768 and 769 of 48 KB of
# staging alone
@pytest.mark.parametrize("cap", [749, 750, 760, 768, 769, 1100])
def test_pairs_at_match_capacity(cap):
    n = cap - 32
    ids, xyz = waters(n)
    s = msys.from_arrays(ids, xyz, None, 9.0, 7.0)
    assert np.array_equal(s.GetPairList(2, FAR), all_pairs(n))
    assert np.array_equal(s.GetPairList(2, FAR), all_pairs(n))   # the capacity as it is now


@pytest.mark.parametrize("cap", [749, 750, 768, 769])
def test_batch_at_match_capacity(cap):
    n = cap - 32
    confs = [waters(m) + (None,) for m in (n, 5)]
    far = batch.Batch(confs, FAR, 5.0)
    near = batch.Batch(confs, 9.0, 5.0)   # (no evaluator reaches further)
    e, f = far.energy(2)[0], near.energy(2)[0]
    assert far.ctx.counts(2)[0] == n * (n - 1) // 2 + 10
    assert np.all(np.abs(e - f) <= 1e-10 * np.abs(f))


# trimers: 48 bytes per match; the block's collection of accepted trimers fits
# beside them up to 4656, the matches alone up to 4842
@pytest.mark.parametrize("cap", [4656, 4657, 4842])
def test_trimers_at_match_capacity(cap):
    n = cap - 32
    ids, xyz = waters(n)
    s = msys.from_arrays(ids, xyz, None, FAR, 4.0)
    s.TwoBodyEnergy(False)
    assert s.NmerCounts(2)[0] == n * (n - 1) // 2
    got = s.GetPairList(3, 4.0)
    ref = mo.OracleSystem(ids, xyz, None, 9.0, 4.0)
    want = ref.top.nmers_to_input(ref.nmers(3))
    assert len(want) > 10000 and np.array_equal(got, want)
    # and their energy, from the buckets
    near = msys.from_arrays(ids, xyz, None, 9.0, 4.0)
    e, f = s.ThreeBodyEnergy(True), near.ThreeBodyEnergy(True)
    assert abs(e - f) <= 1e-10 * abs(f)
    assert np.abs(s.GetRealGrads() - near.GetRealGrads()).max() <= 1e-8
