"""Float min-sum at ties, zeros, signed zeros and clipped sums, bit for bit against the oracle, in rows that keep their
messages (up to five edges) and rows that compress them."""

import numpy as np
import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import ldpc_decode
from oracle.oracle import dec_cfg, in_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row", [[4, 5, 22936, 0, 1280, 32767, -32767], [4, 3, -22936, 0, 1280, 900, -900],
                                 [4, 4, 26000, 60, 1280, 8000, -3000], [4, 3, 22936, 0, 1280, -100, 100]])
@pytest.mark.parametrize("bgn,A,E,Qm", [(1, 8, 96, 2), (1, 488, 1536, 1), (2, 488, 1920, 2), (1, 4352, 8754, 6),
                                        (2, 3816, 9600, 8)])
def test_float_rows_at_ties_and_clips(oracle, cuda, bgn, A, E, Qm, row):
    cfg = (bgn, A, 1, E, 0, Qm, 0)
    rng = np.random.default_rng(A + row[1])
    host = np.stack([rng.choice([-32768, 32767, 0, -1, 1], E), rng.choice([-128, 128], E), rng.integers(-40, 41, E),
                     rng.integers(-32768, 32768, E)]).astype(np.int16)
    got = ldpc_decode(torch.from_numpy(host).to(cuda), cfg, row, return_app=True)
    for i in range(len(host)):
        es, eb, ei, lq = oracle.decode(np.ascontiguousarray(host[i]), in_config(*cfg), dec_cfg(row))
        assert int(got.status[i]) == es and int(got.iterations[i]) == ei
        assert np.array_equal(got.app[i].cpu().numpy(), lq)
        assert np.array_equal(got.hardbits[i].cpu().numpy(), eb)
