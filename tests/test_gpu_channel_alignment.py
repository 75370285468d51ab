"""The channel's LLR rows at every address a caller can give: the widest stores a row's start allows write the same LLRs
as 16-byte aligned rows do, and nothing outside the row."""

import ctypes

import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import channel_llrs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Qm", [1, 2, 4, 6, 8])
@pytest.mark.parametrize("symbols,n", [(1, 3), (4, 1), (11, 5), (256, 4)])
def test_rows_at_every_alignment(cuda, lib, Qm, symbols, n):
    E = symbols * Qm
    gen = torch.Generator(device=cuda).manual_seed(symbols)
    rm = torch.randint(0, 256, (n, (E + 7) // 8), dtype=torch.uint8, device=cuda, generator=gen)
    want = torch.stack([channel_llrs(rm, E, Qm, -6.0, seed=5)[i] for i in range(n)])
    for shift in range(8):
        for stride in range(E, E + 8):
            buf = torch.full((shift + n * stride + 16,), 77, dtype=torch.int16, device=cuda)
            rc = lib.nrldpc_channel_batch(rm.data_ptr(), rm.shape[1], n, E, Qm, ctypes.c_float(-6.0), 5,
                                          buf.data_ptr() + 2 * shift, stride, 0, torch.cuda.current_stream().cuda_stream)
            assert rc == 0
            rows = buf[shift:shift + n * stride].view(n, stride)
            assert torch.equal(rows[:, :E], want), (shift, stride)
            assert (buf[:shift] == 77).all() and (rows[:, E:] == 77).all() and (buf[shift + n * stride:] == 77).all()
