"""Flip-form operators with more groups than one gather launch takes (256): they are
added launch by launch by the general kernels (k_gather_m's records and their ranges
are one launch's).  Against the oracle, through mul_; the project's bars, relative l2
< 1e-12 (ComplexF64, double-float) and < 1e-5 (ComplexF32)."""
import pytest

import qobgpu as Q
from test_gpu_flip import _check, _spins

pytestmark = pytest.mark.gpu


def _low_strings(n, count):
    """sigmax strings on distinct sets of sites, each with site 1 or 2 in it: in ComplexF32,
    where a thread owns four consecutive indices, all of them touch its own bits."""
    sets = []
    for first in (1, 2):
        for l1 in range(1, 6):
            run1 = tuple(range(first, first + l1))
            if l1 == 5:
                sets.append(run1)
            for l2 in range(1, 6 - l1):
                sets += [run1 + tuple(range(b, b + l2)) for b in range(first + l1 + 1, n - l2 + 2)]
    assert len(sets) >= count
    f = Q.Rng(count).uniform(len(sets))
    return _spins(n, [(float(f[i]) - 0.3, tuple((s, "x") for s in sets[i])) for i in range(count)])


@pytest.mark.parametrize("count", [256, 257, 270])
def test_more_groups_than_a_launch_takes(count):
    _check(_low_strings(18, count), 1, "left", 0.3, count)
