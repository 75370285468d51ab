"""Which kernel a uniform batch runs on, and results that depend on it: the arithmetic variant of the fixed-point kernels
follows the decoder row, the tables and whether the call returns beliefs, and every variant equals the oracle."""

import ctypes
import os

import numpy as np
import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import capi, ldpc_decode, set_degree_alpha
from deeplearning_5g_ldpc_decoder_b200.build import DEBUG_LIB_PATH, build_library
from deeplearning_5g_ldpc_decoder_b200.decoder import DecodeResult
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


def _sizes(bgn):
    """One (A, crctype) per lifting size of the base graph that a payload reaches."""
    seen = {}
    for A in range(8, (8448 if bgn == 1 else 3840) - 24 + 1, 8):
        for crc in (1, 0):
            p = capi.gen_ldpc_parameters(capi.make_in_config(bgn, A, crc, 960, 0, 2, 0))
            seen.setdefault(int(p.Zc), (A, crc))
    return sorted(seen.items())


def _raw_decode(lib, llr, cfg, row, app):
    p = capi.gen_ldpc_parameters(capi.make_in_config(*cfg), lib)
    n = llr.shape[0]
    bits = torch.zeros((n, (p.B + 7) // 8), dtype=torch.uint8, device=llr.device)
    st, it = (torch.full((n,), -9, dtype=torch.int32, device=llr.device) for _ in range(2))
    bel = torch.zeros((n, p.N + 2 * p.Zc), dtype=torch.int16, device=llr.device) if app else None
    rc = lib.nrldpc_decode_batch(llr.data_ptr(), llr.shape[1], n, ctypes.byref(capi.make_in_config(*cfg)),
                                 ctypes.byref(capi.make_decoder_config(row)), bits.data_ptr(), bits.shape[1], st.data_ptr(),
                                 it.data_ptr(), bel.data_ptr() if app else 0, bel.shape[1] if app else 0, 0, 0,
                                 torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return bits, st, it, bel


def _set_tables(libs, bgn, alpha=None, beta=None):
    for lib in libs:
        assert lib.nrldpc_set_trained_weights(bgn, alpha.ctypes.data if alpha is not None else None,
                                              beta.ctypes.data if beta is not None else None,
                                              alpha.shape[0] if alpha is not None else 0) == 0


@pytest.mark.parametrize("bgn", [1, 2])
def test_every_lifting_size_on_the_pair_kernel(oracle, cuda, lib, bgn):
    """Both row forms of the pair kernel at every lifting size, with groups that end inside a warp and an odd block at
    the end: equal to the oracle, and the same in the bounds-checked library without a violation."""
    if not os.path.exists(DEBUG_LIB_PATH):
        build_library(debug=True)
    dbg = capi.load_library(DEBUG_LIB_PATH)
    rec = (ctypes.c_uint32 * 4)()
    assert dbg.nrldpc_bounds_check_status(rec, 1) == 1
    rows = [[1, 5, 22936, 0, 1280, 32767, -32767], [2, 5, 0, 0, 1280, 20000, -20000], OPEN_LOW,
            [1, 3, 22936, 0, 1280, -100, 100]]
    rng = np.random.default_rng(bgn)
    alpha, beta = (rng.integers(lo, hi, (3, capi.BG_ROWS[bgn])).astype(np.int16) for lo, hi in ((15000, 30000), (0, 30)))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = _sizes(bgn)
    assert len(sizes) >= (51 if bgn == 1 else 45)
    _set_tables((lib, dbg), bgn, alpha, beta)
    oracle.set_trained(bgn, alpha, beta)
    try:
        for k, (zc, (A, crc)) in enumerate(sizes):
            B = A + (16 if crc == 0 else 24)
            cfg = (bgn, A, crc, 2 * ((2 * B + 1) // 2), k % 4, 2, 0)
            host = noisy_blocks(oracle, cfg, zc)
            for row in (rows[0], rows[1 + k % 3]):
                n = pair_batch(cfg, row)
                many = max(n, (2 * sms * -(-160 // zc) + 1) | 1)   # enough groups per CTA for the wide form
                for m in sorted({n, many}):
                    route = capi.decode_route(cfg, row, m)
                    assert route.kernel == capi.ROUTE_PAIR
                    assert route.wide == int(route.groups == 1 or route.groups * zc >= 160)
                    llr = repeated(host, m, cuda)
                    plain = _raw_decode(lib, llr, cfg, row, False)
                    full = _raw_decode(lib, llr, cfg, row, True)
                    for a, b in zip(plain[:3], full[:3]):
                        assert torch.equal(a, b), (cfg, row, m)
                    check_against_oracle(oracle, cfg, row, host, DecodeResult(*full))
                    if m == many and m != n and k % 3:
                        continue
                    for app, ref in ((False, plain), (True, full)):
                        got = _raw_decode(dbg, llr, cfg, row, app)
                        torch.cuda.synchronize()
                        assert all(torch.equal(a, b) for a, b in zip(got[:3 + app], ref[:3 + app])), (cfg, row, m)
                        assert dbg.nrldpc_bounds_check_status(rec, 1) == 1 and list(rec) == [0] * 4, (cfg, row, m, list(rec))
    finally:
        _set_tables((lib, dbg), bgn)
        oracle.set_trained(bgn)


@pytest.mark.parametrize("row", [[4, 5, 22936, 0, 1280, 32767, -32767], [4, 3, 22936, 0, 1280, -100, 100]])
@pytest.mark.parametrize("bgn,A,E,Qm", [(1, 8, 96, 2), (2, 488, 1920, 2), (1, 4352, 8754, 6)])
def test_both_row_forms_of_float_min_sum(oracle, cuda, row, bgn, A, E, Qm):
    """Rows of up to five edges uncompressed where an SM holds many threads, of up to three in smaller batches."""
    cfg = (bgn, A, 1, E, 0, Qm, 0)
    host = noisy_blocks(oracle, cfg, A)
    n = 1
    while not capi.decode_route(cfg, row, n).wide:
        n += max(1, n // 2)
    small = ldpc_decode(repeated(host, DISTINCT, cuda), cfg, row, return_app=True)
    large = ldpc_decode(repeated(host, n, cuda), cfg, row, return_app=True)
    assert not capi.decode_route(cfg, row, DISTINCT).wide
    for i in range(DISTINCT):
        es, eb, ei, lq = oracle.decode(np.ascontiguousarray(host[i]), in_config(*cfg), dec_cfg(row))
        for got in (small, large):
            same = slice(i, got.status.shape[0], DISTINCT)
            assert (got.status[same] == es).all() and (got.iterations[same] == ei).all()
            assert (got.app[same] == torch.from_numpy(lq).to(cuda)).all()
            assert (got.hardbits[same] == torch.from_numpy(eb).to(cuda)).all()
