"""Rows that keep their messages uncompressed (csrc/nrldpc_fixed_row.cuh: row_update_direct) against the compressed
form and the oracle.  The no-allocation entry point has four message words per row, so longer rows stay compressed there,
and with the open maximum a batch that returns beliefs compresses every row with a parity column of its own."""

import numpy as np
import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import capi, ldpc_decode
from deeplearning_5g_ldpc_decoder_b200.decoder import set_trained_weights
from oracle.oracle import dec_cfg, in_config
from test_gpu_split import ROWS, _pair_kernel

pytestmark = pytest.mark.gpu

DISTINCT = 6


@pytest.mark.parametrize("row", range(len(ROWS)))
@pytest.mark.parametrize("bgn,A,E,rv,Qm,many", [
    (1, 8, 96, 0, 2, True),           # Zc 2: 192 groups per CTA
    (2, 120, 400, 2, 8, True),        # Zc 18 of BG2
    (1, 2376, 3600, 1, 4, False),     # Zc 112: three groups per CTA
    (2, 3816, 9600, 0, 8, False),     # Zc 384 of BG2: core rows of 8 and 10 edges
    (1, 8424, 25344, 0, 8, False),    # Zc 384
])
def test_direct_rows_equal_the_compressed_form(oracle, cuda, lib, row, bgn, A, E, rv, Qm, many):
    cfg, r = (bgn, A, 1, E, rv, Qm, 0), ROWS[row]
    # more blocks than the small-batch kernel takes at this lifting size
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 32 * sms + 3 if many else 3 * sms + 1
    rng = np.random.default_rng(A + row)
    rm = oracle.encode(rng.integers(0, 256, A // 8, dtype=np.uint8), in_config(*cfg))
    bits = np.unpackbits(rm)[:E].astype(np.float64)
    x = (1 - 2 * bits)[None, :] * 300 + rng.normal(0, rng.uniform(120, 420, size=(DISTINCT, 1)), size=(DISTINCT, E))
    x[0] *= 60                                                       # sums that leave int16
    x[1, :: 7] = rng.choice([-32768, 32767, 0, -1], size=x[1, :: 7].shape)
    host = np.clip(np.round(x), -32768, 32767).astype(np.int16)
    llr = torch.from_numpy(host).to(cuda)[torch.arange(n, device=cuda) % DISTINCT].contiguous()
    if r[0] == 2:
        g = np.random.default_rng(1)
        set_trained_weights(bgn, g.integers(15000, 30000, (4, capi.BG_ROWS[bgn])), g.integers(0, 30, (4, capi.BG_ROWS[bgn])))
    try:
        want = _pair_kernel(lib, llr, E, cfg, r, None)
        plain, full = ldpc_decode(llr, cfg, r), ldpc_decode(llr, cfg, r, return_app=True)
    finally:
        if r[0] == 2:
            set_trained_weights(bgn)
    for got in (plain, full):
        assert torch.equal(got.hardbits, want[0])
        assert torch.equal(got.status, want[1]) and torch.equal(got.iterations, want[2])
    assert torch.equal(full.app, want[3])
    if r[0] == 2:
        return
    for i in range(DISTINCT if many else 2):
        es, eb, ei, lq = oracle.decode(np.ascontiguousarray(host[i]), in_config(*cfg), dec_cfg(r))
        assert int(plain.status[i]) == es and int(plain.iterations[i]) == ei
        assert np.array_equal(full.app[i].cpu().numpy(), lq)
