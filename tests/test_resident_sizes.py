"""Which graphs the resident solver is asked to take, by size (no GPU needed):
one block exactly where one block's shared memory holds the graph, whose layout
has a slot for each of the block's 1,024 threads, used or not."""
import ctypes as C

import pytest

import wbpr_gb300 as W

SMEM, THREADS, CLUSTER = 227 * 1024, 1024, 16


def _rule(name, result):
    f = getattr(W.lib(), name)
    f.argtypes, f.restype = [C.c_longlong, C.c_longlong], result
    return f


@pytest.fixture(scope="module")
def rules():
    return _rule("_ZN8wbpr_dev16resident_clusterExx", C.c_int), _rule("_ZN8wbpr_dev18resident_one_blockExx", C.c_bool)


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 200, 1000, 1023, 1024, 1025, 2000, 2049, 4095, 4096, 4097, 9000, 60000, 65536,
                               65537])
def test_one_block_exactly_where_it_fits(rules, n):
    cluster, one_block = rules
    limit = (SMEM - 14 * max(n, THREADS)) // 8  # arcs, but for the control words
    for na in [0, n, 20000, 28400, *range(max(0, limit - 600), max(0, limit + 600), 7), 60000, 65535, 65536]:
        assert (cluster(n, na) == 1) == one_block(n, na), (n, na)
        if one_block(n, na):
            assert 14 * max(THREADS, n) + 8 * na < SMEM and n <= 4096 and na <= 65535


@pytest.mark.parametrize("n", [200, 1000, 5000, 16383, 16384, 40000])
def test_a_block_of_the_cluster_has_a_slot_a_thread(rules, n):
    cluster, _ = rules
    for na in range(0, 700000, 997):
        if cluster(n, na) == CLUSTER:
            assert 14 * max(THREADS, n // CLUSTER) + 8 * na // CLUSTER < SMEM, (n, na)
    assert cluster(n, 100000) == CLUSTER
