"""What a device call derives from its parameters: the C arguments and the
element counts its buffers are checked against, which are kept by the
integer parameters' values."""

import numpy as np
import pytest

from polymage_b200.apps import catalog


def test_counts_follow_the_parameters():
    cp = catalog.build("unsharp")
    sizes = [(5, 7), (64, 33), (5, 7), (np.int32(64), 33), (64.0, 33)]
    for i, (R, C) in enumerate(sizes):
        prm = {'R': R, 'C': C, 'threshold': 0.25 * i, 'weight': -i}
        args, counts = cp._signature(prm)
        want = {'R': R, 'C': C, 'threshold': 0.25 * i, 'weight': -i}
        assert [float(a) for a in args] == [float(want[p.name])
                                            for p in cp.params]
        R, C = int(R), int(C)
        assert counts == [3 * (R + 4) * (C + 4), 3 * R * C]


def test_missing_parameter_is_named_and_the_store_is_bounded():
    cp = catalog.build("harris")
    cp._counts.clear()
    with pytest.raises(KeyError, match="missing parameter C"):
        cp._signature({'R': 10})
    for n in range(cp.COUNTS_KEPT + 10):
        assert cp._signature({'R': n + 1, 'C': 9})[1][0] == (n + 3) * 11
    assert len(cp._counts) <= cp.COUNTS_KEPT
