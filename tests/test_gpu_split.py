"""The small-batch kernel (one code block per CTA, rows split over four lanes) against the pair kernel, reached through
the no-allocation entry point, and against the oracle: statuses, iterations, bits, beliefs and soft buffers are equal."""

import ctypes

import numpy as np
import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import capi, ldpc_decode
from deeplearning_5g_ldpc_decoder_b200.decoder import set_trained_weights
from oracle.oracle import dec_cfg, in_config

pytestmark = pytest.mark.gpu

ROWS = [[1, 8, 22936, 0, 1280, 32767, -32767], [3, 5, 0, 0, 1280, 32767, -32768], [2, 7, 0, 0, 900, 20000, -20000],
        [1, 6, 24000, 40, 1280, 8000, -8000], [1, 4, 65000, 0, 1280, 32767, -32767],
        [1, 3, 22936, 0, 1280, -100, 100], [1, 0, 22936, 0, 1280, 32767, -32767]]


def _pair_kernel(lib, llr, E, cfg, row, harq):
    p = capi.gen_ldpc_parameters(capi.make_in_config(*cfg))
    n, nb, L = llr.shape[0], (p.B + 7) // 8, p.N + 2 * p.Zc
    bits = torch.zeros((n, nb), dtype=torch.uint8, device="cuda")
    st, it = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    app = torch.empty((n, L), dtype=torch.int16, device="cuda")
    rc = lib.nrldpc_decode_batch_noalloc(
        llr.data_ptr(), llr.stride(0), n, ctypes.byref(capi.make_in_config(*cfg)),
        ctypes.byref(capi.make_decoder_config(row)), bits.data_ptr(), nb, st.data_ptr(), it.data_ptr(), app.data_ptr(),
        L, harq.data_ptr() if harq is not None else 0, L if harq is not None else 0,
        torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return bits, st, it, app


@pytest.mark.parametrize("row", range(len(ROWS)))
@pytest.mark.parametrize("bgn,A,E,rv,Qm,n,pad", [
    (1, 8, 96, 0, 2, 3, 0),           # Zc 2: one word per column
    (2, 8, 64, 0, 4, 5, 1),           # odd Zc below 16, rows off the 16-byte grid
    (1, 88, 600, 0, 1, 2, 0),         # Zc 6, repetition
    (2, 120, 400, 2, 8, 7, 0),        # Zc 18 of BG2
    (1, 264, 900, 0, 6, 33, 2),       # Zc 14
    (2, 488, 1920, 0, 2, 64, 0),      # Zc 64: the small-packet batch
    (1, 2376, 3600, 1, 4, 9, 0),      # Zc 112
    (1, 8424, 25344, 0, 8, 3, 0),     # Zc 384: all shared memory in use
    (1, 8424, 65520, 3, 6, 2, 0),     # Zc 384, repetition
    (2, 3816, 9600, 0, 8, 100, 0),    # Zc 384 of BG2
])
def test_small_batches_equal_the_pair_kernel(oracle, cuda, lib, row, bgn, A, E, rv, Qm, n, pad):
    cfg, r = (bgn, A, 1, E, rv, Qm, 1 if row == 0 else 0), ROWS[row]
    rng = np.random.default_rng(A + E + row)
    p = capi.gen_ldpc_parameters(capi.make_in_config(*cfg))
    L = p.N + 2 * p.Zc
    # noisy words of random codewords, with int16 extremes in one block
    rm = oracle.encode(rng.integers(0, 256, A // 8, dtype=np.uint8), in_config(*cfg))
    bits = np.unpackbits(rm)[:E].astype(np.float64)
    x = (1 - 2 * bits)[None, :] * 300 + rng.normal(0, rng.uniform(120, 420, size=(n, 1)), size=(n, E))
    x[0, :: 7] = rng.choice([-32768, 32767, 0, -1], size=x[0, :: 7].shape)
    llr = torch.zeros((n, E + pad), dtype=torch.int16, device=cuda)
    llr[:, :E] = torch.from_numpy(np.clip(np.round(x), -32768, 32767).astype(np.int16)).to(cuda)
    soft = torch.from_numpy(rng.integers(-400, 400, size=(n, L)).astype(np.int16)).to(cuda)
    if r[0] == 2:
        g = np.random.default_rng(1)
        set_trained_weights(bgn, g.integers(15000, 30000, (4, capi.BG_ROWS[bgn])), g.integers(0, 30, (4, capi.BG_ROWS[bgn])))
    try:
        h1, h2 = soft.clone(), soft.clone()
        want = _pair_kernel(lib, llr, E, cfg, r, h1)
        before = capi.kernel_launch_count()
        got = ldpc_decode(llr, cfg, r, return_app=True, harq=h2)
        assert capi.kernel_launch_count() == before + 1
        assert torch.equal(got.status, want[1]) and torch.equal(got.iterations, want[2])
        assert torch.equal(got.app, want[3]) and torch.equal(got.hardbits, want[0])
        assert torch.equal(h1, h2)
    finally:
        if r[0] == 2:
            set_trained_weights(bgn)
    if row == 0 or r[0] == 2:
        return
    host = llr.cpu().numpy()
    for i in range(min(n, 2)):
        es, eb, ei, lq = oracle.decode(np.ascontiguousarray(host[i, :E]), in_config(*cfg), dec_cfg(r))
        assert int(got.status[i]) == es and int(got.iterations[i]) == ei
        assert np.array_equal(got.app[i].cpu().numpy(), lq)


@pytest.mark.parametrize("row", [0, 2, 3, 5])
@pytest.mark.parametrize("bgn,A,E,Qm,per_sm,extra", [
    (1, 488, 1536, 2, 3, 0),          # Zc 24: eight lanes, the last batch of three blocks per SM
    (1, 488, 1536, 2, 4, 0),          # four per SM: only eight lanes fit
    (1, 840, 2400, 4, 2, 0),          # Zc 40: 640 threads on an SM
    (1, 1736, 5000, 4, 0, 5),         # Zc 80: the last size with eight lanes
    (1, 1744, 5000, 4, 1, 1),         # Zc 88 and above, two rounds of one block: pair kernel or four lanes
    (2, 120, 400, 2, 2, 0),           # Zc 24 of BG2: 384 threads, four lanes
    (2, 104, 400, 2, 1, 0),           # eight lanes
    (2, 24, 100, 2, 10, 0),           # four lanes do not fit
])
def test_lane_counts_equal_the_pair_kernel(oracle, cuda, lib, row, bgn, A, E, Qm, per_sm, extra):
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    test_small_batches_equal_the_pair_kernel(oracle, cuda, lib, row, bgn, A, E, 0, Qm, n, 0)
