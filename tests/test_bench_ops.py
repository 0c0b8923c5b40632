"""Lane-operations that bench.py's ALU roofline counts (no GPU)."""
import pytest

import bench


@pytest.mark.parametrize("s", [1, 2, 3, 5])
def test_lane_ops(s):
    n, m, o, k = bench.PARAMS[s]
    macs, own, one = bench.mac_counts(s), bench.lane_ops(s, False), bench.lane_ops(s, True)
    for op in ("keypair", "verify"):  # nothing but products of the key
        assert own[op] == 9 / 32 * macs[op]
        assert one[op] == 0.5 * macs[op]
    elim = m * m * (k * o + 1)
    assert own["sign"] == pytest.approx(9 / 32 * (macs["sign"] - elim) + 0.5 * elim) and one["sign"] == 0.5 * macs["sign"]
    assert 9 / 32 * macs["sign"] < own["sign"] < one["sign"]
