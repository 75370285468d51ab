"""Which kernel a uniform batch runs on, and results that depend on it: the arithmetic variant of the fixed-point kernels
follows the decoder row, the tables and whether the call returns beliefs, and every variant equals the oracle."""

import numpy as np
import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import capi, ldpc_decode, set_degree_alpha
from oracle.oracle import dec_cfg, in_config

pytestmark = pytest.mark.gpu

DISTINCT = 5
OPEN_LOW = [1, 6, 22936, 0, 1280, 32767, -20000]   # open maximum, a minimum that sums often reach


def pair_batch(cfg, row, beliefs=False, lib=None):
    """The smallest odd batch of this configuration that runs on the pair kernel."""
    n = 1
    while capi.decode_route(cfg, row, n, beliefs, lib).kernel == capi.ROUTE_SMALL_BATCH:
        n = 2 * n + 1
    lo = (n - 1) // 2
    while lo + 1 < n:   # lo: small-batch kernel (or 0), n: pair kernel
        mid = (lo + n) // 2
        if capi.decode_route(cfg, row, mid, beliefs, lib).kernel == capi.ROUTE_SMALL_BATCH:
            lo = mid
        else:
            n = mid
    return n | 1


def noisy_blocks(oracle, cfg, seed):
    """DISTINCT noisy words of one random codeword: clean to hopeless, one that saturates, one of int16 extremes."""
    E = cfg[3]
    rng = np.random.default_rng(seed)
    rm = oracle.encode(rng.integers(0, 256, cfg[1] // 8, dtype=np.uint8), in_config(*cfg))
    bits = np.unpackbits(rm)[:E].astype(np.float64)
    x = (1 - 2 * bits)[None, :] * 300 + rng.normal(0, rng.uniform(120, 420, size=(DISTINCT, 1)), size=(DISTINCT, E))
    x[0] *= 60
    x[1, :: 7] = rng.choice([-32768, 32767, 0, -1], size=x[1, :: 7].shape)
    return np.clip(np.round(x), -32768, 32767).astype(np.int16)


def repeated(host, n, cuda):
    return torch.from_numpy(host).to(cuda)[torch.arange(n, device=cuda) % host.shape[0]].contiguous()


def check_against_oracle(oracle, cfg, row, host, got):
    for i in range(host.shape[0]):
        es, eb, ei, lq = oracle.decode(np.ascontiguousarray(host[i]), in_config(*cfg), dec_cfg(row))
        same = slice(i, got.status.shape[0], host.shape[0])
        assert (got.status[same] == es).all() and (got.iterations[same] == ei).all(), i
        if ei > 0:
            assert (got.hardbits[same] == torch.from_numpy(eb).to(got.hardbits.device)).all(), i
        if got.app is not None:
            assert (got.app[same] == torch.from_numpy(np.asarray(lq, dtype=np.int16)).to(got.app.device)).all(), i


@pytest.mark.parametrize("row,plain,beliefs", [
    ([1, 8, 22936, 0, 1280, 32767, -32767], capi.ARITH_OPEN_PARITY, capi.ARITH_OPEN),
    ([3, 8, 0, 0, 1280, 32767, -32768], capi.ARITH_OPEN_PARITY, capi.ARITH_OPEN),
    (OPEN_LOW, capi.ARITH_OPEN, capi.ARITH_OPEN),
    ([1, 8, 22936, 0, 1280, 32767, -32766], capi.ARITH_OPEN, capi.ARITH_OPEN),
    ([1, 8, 22936, 1, 1280, 32767, -32767], capi.ARITH_CLAMP, capi.ARITH_CLAMP),
    ([1, 8, 40000, 0, 1280, 32767, -32767], capi.ARITH_CLAMP, capi.ARITH_CLAMP),      # alpha < 0 as int16
    ([1, 8, 22936, 0, 1280, 32766, -32767], capi.ARITH_CLAMP, capi.ARITH_CLAMP),
    ([1, 8, 22936, 0, 1280, -100, 100], capi.ARITH_DEGENERATE, capi.ARITH_DEGENERATE),
])
def test_arithmetic_of_a_decoder_row(cuda, row, plain, beliefs):
    for cfg, n in (((1, 8424, 1, 25344, 0, 8, 0), 1), ((2, 488, 1, 1920, 0, 2, 0), 20000), ((2, 488, 1, 1920, 0, 2, 0), 1)):
        assert capi.decode_route(cfg, row, n).arithmetic == plain
        assert capi.decode_route(cfg, row, n, beliefs=True).arithmetic == beliefs
    if row[0] == 3:
        set_degree_alpha([-1] * 19)
        try:
            assert capi.decode_route((2, 488, 1, 1920, 0, 2, 0), row, 1).arithmetic == capi.ARITH_CLAMP
        finally:
            set_degree_alpha()


@pytest.mark.parametrize("row", [OPEN_LOW, [3, 5, 0, 0, 900, 32767, -3], [1, 6, 22936, 0, 1280, 32767, -32767],
                                 [1, 0, 22936, 0, 1280, 32767, -20000]])
@pytest.mark.parametrize("bgn,A,E,rv,Qm", [(1, 8, 96, 0, 2), (2, 120, 400, 2, 8), (1, 2376, 3600, 1, 4),
                                           (2, 3816, 9600, 0, 8), (1, 8424, 25344, 0, 8)])
def test_open_maximum_without_parity_words(oracle, cuda, row, bgn, A, E, rv, Qm):
    cfg = (bgn, A, 1, E, rv, Qm, 0)
    host = noisy_blocks(oracle, cfg, A + row[1])
    n = max(pair_batch(cfg, row), pair_batch(cfg, row, True))
    llr = repeated(host, n, cuda)
    check_against_oracle(oracle, cfg, row, host, ldpc_decode(llr, cfg, row))
    check_against_oracle(oracle, cfg, row, host, ldpc_decode(llr, cfg, row, return_app=True))
