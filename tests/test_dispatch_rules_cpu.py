"""Which of two kernels with the same result a call takes, by its sizes alone (csrc/dispatch_rules.h, through b200_rule_query, no GPU):
both sides of every line, at sizes where both kernels were timed."""
import ctypes as C

import pytest

from kubeai_b200._lib import lib

PICKED_ALONE = 0


def rule(which, *v):
    return lib().b200_rule_query(which, (C.c_int32 * len(v))(*v), len(v))


def test_unknown_rules_are_refused():
    assert rule(99, 1) < 0 and rule(PICKED_ALONE, 1, 2) < 0 and lib().b200_rule_query(PICKED_ALONE, None, 4) < 0


# pairs, N, K: experts of 2048 and of 4096, gate and up side by side
@pytest.mark.parametrize("rows,N,K,alone", [(2, 4096, 2048, 0), (16, 2048, 2048, 0), (24, 2048, 2048, 1), (16, 4096, 2048, 1), (2, 8192, 4096, 0), (4, 8192, 4096, 1),
                                            (32, 8192, 4096, 1), (64, 8192, 4096, 1), (64, 64, 64, 0)])
def test_large_streams_of_picked_rows_run_behind_their_predecessor(rows, N, K, alone):
    """Overlapping a product that holds most of an SM as shared memory, 64 pairs of 8192 x 4096 took 5335 us a step against 4222."""
    assert rule(PICKED_ALONE, rows, N, K, 2) == alone
