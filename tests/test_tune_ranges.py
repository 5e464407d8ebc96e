"""Ranges of the launch-shape table (host only): one entry for a size, and parity
shapes that hold the instances they are used for."""
import pytest

from cvrp_aco_ocl_b200 import MODE_PARITY, MODE_THROUGHPUT, default_params
from cvrp_aco_ocl_b200.tune import DEFAULT_TABLE, TuneTable

from test_tune import entry


def test_shipped_table_has_one_entry_a_size():
    e = TuneTable.load(DEFAULT_TABLE).entries
    for i, a in enumerate(e):
        for b in e[:i]:
            if (a.mode, a.batch, a.ants) == (b.mode, b.batch, b.ants):
                assert a.n_hi < b.n_lo or b.n_hi < a.n_lo, (a, b)


@pytest.mark.parametrize("n", [3, 71, 708, 709, 1582, 1583, 2501, 4096, 4097, 5000, 8000, 8192])
def test_shipped_parity_shapes_hold_32_nodes_a_thread(n):
    p = default_params(n)
    p.mode, p.n_ants = MODE_PARITY, n
    TuneTable.load(DEFAULT_TABLE).apply(p, n)
    assert p.warps_per_ant > 0 and n <= 32 * 32 * p.warps_per_ant


def test_add_drops_overlapping_ranges_of_the_same_kind():
    t = TuneTable([entry(lo=3, hi=708, ants=50), entry(lo=709, hi=1 << 30, ants=50), entry(lo=709, hi=1 << 30, ants=64),
                   entry(mode=MODE_PARITY, lo=709, hi=1 << 30, ants=50)])
    batch = entry(lo=101, hi=1001, ants=50)
    batch.batch = 1
    t.add(batch)
    assert len(t.entries) == 5
    t.add(entry(lo=709, hi=1582, ants=50, apc=2))
    t.add(entry(lo=1583, hi=1 << 30, ants=50, apc=8))
    assert len(t.entries) == 6
    assert t.lookup(5000, MODE_THROUGHPUT, 50).ants_per_block == 8
    assert t.lookup(700, MODE_THROUGHPUT, 50).n_hi == 708


def test_lookup_leaves_parity_shapes_that_do_not_hold_the_instance():
    t = TuneTable([entry(mode=MODE_PARITY, lo=709, hi=1 << 30, ants=50, apc=1, wpa=4)])
    assert t.lookup(4096, MODE_PARITY, 50).warps_per_ant == 4
    assert t.lookup(4097, MODE_PARITY, 50) is None
