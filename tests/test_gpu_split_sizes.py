"""The small-batch kernel at its largest lifting sizes, where rows are split over four lanes and, from Zc 144 of BG1 on,
a thread computes its edges' addresses instead of reading them from a table: equal to the pair kernel and the oracle."""

import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import capi
from test_gpu_split import ROWS, test_small_batches_equal_the_pair_kernel as check_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row", range(len(ROWS)))
@pytest.mark.parametrize("bgn,zc,A,E,rv,Qm,n,pad", [
    (1, 128, 2760, 8000, 0, 4, 3, 0),    # the largest with a table
    (1, 144, 3100, 5002, 2, 2, 2, 1),
    (1, 176, 3840, 9000, 0, 6, 5, 0),
    (1, 208, 4352, 6400, 1, 8, 2, 0),    # the largest of BG1
    (2, 176, 1704, 8000, 3, 2, 3, 0),
    (2, 208, 2040, 5200, 0, 4, 2, 2),    # the largest of BG2
])
def test_largest_sizes(oracle, cuda, lib, row, bgn, zc, A, E, rv, Qm, n, pad):
    A = A // 8 * 8
    cfg = (bgn, A, 1, E, rv, Qm, 1 if row == 0 else 0)
    assert capi.gen_ldpc_parameters(capi.make_in_config(*cfg)).Zc == zc
    route = capi.decode_route(cfg, ROWS[row], n, beliefs=True)
    assert route.kernel == capi.ROUTE_SMALL_BATCH and route.lanes == 4
    check_batch(oracle, cuda, lib, row, bgn, A, E, rv, Qm, n, pad)


@pytest.mark.parametrize("bgn,A", [(1, 4568), (1, 8424), (2, 2128), (2, 2480), (2, 3816)])
def test_larger_sizes_run_on_the_pair_kernel(cuda, bgn, A):
    """Above 832 threads the pair kernel is the faster one even for a single block."""
    cfg = (bgn, A, 1, 9600, 0, 2, 0)
    assert capi.gen_ldpc_parameters(capi.make_in_config(*cfg)).Zc >= 224
    for row in ROWS:
        assert capi.decode_route(cfg, row, 1).kernel == capi.ROUTE_PAIR
