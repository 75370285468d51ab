"""The tape of the float32 training kernels: its layout does not depend on where it lies, rows with infinities or sums
beyond float32 have the checkpoint form's values and gradients, evaluation keeps no tape, and a batch whose tape does not
fit the device trains with checkpoints."""

import ctypes

import pytest
import torch

from deeplearning_5g_ldpc_decoder_b200 import capi
from deeplearning_5g_ldpc_decoder_b200.train import MinSumUnrolled, NeuralLayeredMinSumDecoder
from test_gpu_train import _checkpoint_form

pytestmark = pytest.mark.gpu


def _inputs(cfg, T, batch, seed):
    p = capi.gen_ldpc_parameters(capi.make_in_config(*cfg))
    n, R = p.N + 2 * p.Zc, capi.BG_ROWS[p.bgn]
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((batch, n), device="cuda", generator=g) * 4 + 3
    a = torch.rand((T, R), device="cuda", generator=g) * 0.4 + 0.5
    b = torch.rand((T, R), device="cuda", generator=g) * 0.1
    gf = torch.randn((batch, n), device="cuda", generator=g)
    gi = torch.randn((T, batch, n), device="cuda", generator=g) * 0.1
    return x, a, b, gf, gi


def _tape_form(lib, cfg, x, a, b, clip, detach, gf, gi, forward_at, backward_at):
    """Forward and backward of the C ABI with the tape that many floats from a 16-byte boundary."""
    c, T, batch = capi.make_in_config(*cfg), a.shape[0], x.shape[0]
    floats = ctypes.c_int64(0)
    assert lib.nrldpc_train_tape_floats(ctypes.byref(c), T, batch, ctypes.byref(floats)) == 0
    tapes = [torch.zeros(floats.value + 4, device="cuda") for _ in range(2)]
    first, second = tapes[0][forward_at:], tapes[1][backward_at:]
    fin, its = torch.empty_like(x), torch.empty((T, *x.shape), device="cuda")
    gx, ga, gb = torch.empty_like(x), torch.zeros_like(a), torch.zeros_like(b)
    s = torch.cuda.current_stream().cuda_stream
    assert lib.nrldpc_train_forward_tape(x.data_ptr(), batch, ctypes.byref(c), T, a.data_ptr(), b.data_ptr(), clip or 0.0,
                                         fin.data_ptr(), its.data_ptr(), first.data_ptr(), s) == 0
    second[:floats.value] = first[:floats.value]
    assert lib.nrldpc_train_backward_tape(x.data_ptr(), batch, ctypes.byref(c), T, a.data_ptr(), b.data_ptr(), clip or 0.0,
                                          int(detach), second.data_ptr(), gf.data_ptr(), gi.data_ptr(), gx.data_ptr(),
                                          ga.data_ptr(), gb.data_ptr(), s) == 0
    return fin, its, gx, ga, gb


@pytest.mark.parametrize("cfg,T,batch,clip", [
    ((2, 488, 1, 1920, 0, 2, 0), 3, 5, None), ((1, 600, 1, 1500, 0, 2, 0), 2, 4, 7.0),   # Zc 64; Zc 30, planes
    ((1, 2440, 1, 7392, 0, 2, 0), 2, 3, 9.0), ((2, 8, 1, 96, 0, 2, 0), 3, 40, None),     # Zc 112; Zc 6
    ((2, 56, 1, 300, 0, 2, 0), 2, 9, None),                                              # Zc 16
])
def test_tape_can_be_moved(cuda, lib, cfg, T, batch, clip):
    inputs = _inputs(cfg, T, batch, T)
    want = _tape_form(lib, cfg, *inputs[:3], clip, False, *inputs[3:], 0, 0)
    for places in ((0, 1), (2, 0), (3, 2), (1, 1)):
        got = _tape_form(lib, cfg, *inputs[:3], clip, False, *inputs[3:], *places)
        for k in range(3):
            assert torch.equal(got[k], want[k]), (places, k)
        for k in (3, 4):   # sums over CTAs in any order
            assert (got[k] - want[k]).abs().max().item() <= 1e-4 * want[k].abs().max().item(), (places, k)


@pytest.mark.parametrize("clip", [None, 11.0])
@pytest.mark.parametrize("detach", [False, True])
@pytest.mark.parametrize("cfg", [(2, 488, 1, 1920, 0, 2, 0), (2, 40, 1, 200, 0, 2, 0), (1, 600, 1, 1500, 0, 2, 0)])
def test_infinite_and_huge_inputs(cuda, lib, cfg, clip, detach):
    """Known bits at +-infinity, a block of nothing else, and magnitudes whose row sum is beyond float32: values and LLR
    gradients equal those of the checkpoint form, infinities and NaN among them."""
    T, batch = 2, 6
    x, a, b, gf, gi = _inputs(cfg, T, batch, 7)
    n = x.shape[1]
    inf = float("inf")
    x[0, ::5], x[1, 3::7] = inf, -inf
    x[2] = torch.where(x[2] < 3, -inf, inf)
    x[3] = x[3] * 2e37
    x[4, : n // 3] = 3e38
    got = _tape_form(lib, cfg, x, a, b, clip, detach, gf, gi, 0, 0)
    want = _checkpoint_form(cfg, x, a, b, clip, detach, gf, gi)
    for k in range(2):
        assert torch.equal(got[k], want[k]) or torch.equal(got[k].nan_to_num(1.5), want[k].nan_to_num(1.5)), k
    g, w = got[2], want[2]
    assert torch.equal(g.isnan(), w.isnan()) and torch.equal(g.isinf(), w.isinf())
    ok = w.isfinite()
    for i in range(batch):   # two summation orders, as with finite inputs
        if ok[i].any():
            scale = w[i][ok[i]].abs().max().item()
            assert (g[i][ok[i]] - w[i][ok[i]]).abs().max().item() <= 1e-4 * scale + 1e-12, i
    for k in (3, 4):
        assert torch.equal(got[k].isnan(), want[k].isnan()), k


@pytest.mark.parametrize("cfg,T,batch,clip", [((2, 488, 1, 1920, 0, 2, 0), 6, 700, None), ((1, 600, 1, 1500, 0, 2, 0), 4, 33, 9.0),
                                              ((2, 40, 1, 200, 0, 2, 0), 3, 5, None), ((1, 2440, 1, 7392, 0, 2, 0), 5, 400, 12.0)])
def test_evaluation_keeps_no_tape(cuda, cfg, T, batch, clip):
    """Under no_grad, and where nothing needs a gradient: the same values, in a fraction of the tape's memory."""
    x = _inputs(cfg, T, batch, 3)[0]
    model = NeuralLayeredMinSumDecoder(cfg, num_iterations=T, alpha_mode="checkpoint", init_beta=0.02, clip_llr=clip).cuda()
    bits, final, its = model(x, return_llr=True, return_iteration_llrs=True)
    floats = ctypes.c_int64(0)
    assert capi.load_library().nrldpc_train_tape_floats(ctypes.byref(capi.make_in_config(*cfg)), T, batch,
                                                        ctypes.byref(floats)) == 0
    with torch.no_grad():
        got = model(x, return_llr=True, return_iteration_llrs=True)
    assert torch.equal(got[0], bits) and torch.equal(got[1], final.detach())
    assert all(torch.equal(a, b.detach()) for a, b in zip(got[2], its))
    model.requires_grad_(False)
    del bits, its, got
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    last = model(x, return_llr=True)[1]
    assert torch.equal(last, final.detach()) and last.grad_fn is None
    outputs = 4 * x.nelement() * 4
    assert torch.cuda.max_memory_allocated() - before < 4 * floats.value // 2 + outputs


def test_checkpoints_where_the_tape_does_not_fit(cuda):
    """A BG1 batch between the checkpoints' size and the tape's trains all the same, with the same values and gradients."""
    cfg, T, batch = (1, 2440, 1, 7392, 0, 2, 0), 10, 400
    x, a, b, gf, gi = _inputs(cfg, T, batch, 5)

    def step():
        leaves = [t.clone().requires_grad_(True) for t in (x, a, b)]
        final, _ = MinSumUnrolled.apply(*leaves, cfg, None, False, False)
        final.backward(gf)
        return (final.detach(), *[t.grad for t in leaves])

    want = step()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    tape = 4 * T * batch * 316 * 112                       # 566 MB; checkpoints take 452 MB
    limit = torch.cuda.memory_reserved() + int(0.92 * tape)
    torch.cuda.set_per_process_memory_fraction(limit / total)
    try:
        got = step()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        torch.cuda.empty_cache()
    assert torch.equal(got[0], want[0])
    for g, w in zip(got[1:], want[1:]):
        assert (g - w).abs().max().item() <= 1e-4 * w.abs().max().item()
