"""What is timed when this package's speed is measured: the calls a user makes, from one code block per call to
full-GPU batches, through the package's public entry points.

kind      entry point                                     stands for
call      cuda_ldpc_5g_decode (C ABI, host buffers)       a BLER harness or a legacy receiver, one block per call
decode    ldpc_decode (CUDA tensors)                      batched receive, algos 0-4, with and without soft buffers
host      ldpc_decode_host (host buffers)                 batched receive whose LLRs and results live in host memory
mixed     mixed.MixedPlan.decode                          a slot's code blocks of many sizes, rates and modulations
tb        tb.TbEngine.decode                              whole transport blocks (segmentation, CRCs, payload gather)
encode    ldpc_encode                                     transmit side, simulation and training data
channel   channel_llrs                                    simulation and training data
train     train.NeuralLayeredMinSumDecoder                learning the min-sum tables: forward, loss, backward

Received LLRs are made the way the framework's own benchmark and tests make them: random payloads, encoded, sent over
QAM and AWGN, demapped to int16.  A noise margin of a few dB above the Shannon limit of the block's spectral efficiency
makes most blocks converge after a few iterations; a negative margin never converges, so every iteration runs.
"""

import ctypes
import math

import numpy as np
import torch

# [algo, max_iterations, alpha, beta, filling_bit_value, max_llr, min_llr]
_ALPHA, _FILL = 22936, 1280


def _row(case):
    return [case["algo"], case["iters"], _ALPHA, 0, _FILL, 32767, -32767]


def listed():
    return [
        # the smallest case of the reference's CUDA decoder test: one BPSK block per call, Zc 24, latency only
        {"name": "call_bg1_zc24", "kind": "call", "bgn": 1, "A": 488, "crc": 1, "E": 1536, "rv": 0, "Qm": 1,
         "algo": 1, "iters": 32, "margin": 4.5},
        # a slot with a few small packets (BG2 Zc64, QPSK): a batch much smaller than the GPU
        {"name": "decode_bg2_zc64_n64", "kind": "decode", "bgn": 2, "A": 488, "crc": 1, "E": 1920, "rv": 0, "Qm": 2,
         "algo": 1, "iters": 10, "margin": 4.0, "n": 64, "harq": False},
        # full-GPU batch of the largest blocks, all iterations executed (the benchmark's workload)
        {"name": "decode_bg1_zc384_n8192", "kind": "decode", "bgn": 1, "A": 8424, "crc": 1, "E": 25344, "rv": 0,
         "Qm": 8, "algo": 1, "iters": 8, "margin": -3.0, "n": 8192, "harq": False},
        # high code rate with the trained tables, soft buffers stored for a retransmission, ragged batch, early exit
        {"name": "decode_trained_harq_n1001", "kind": "decode", "bgn": 1, "A": 8424, "crc": 1, "E": 9600, "rv": 0,
         "Qm": 8, "algo": 2, "iters": 10, "margin": 3.0, "n": 1001, "harq": True},
        # float min-sum at a lifting size that does not fill its thread blocks, with filler bits
        {"name": "decode_float_zc208_n777", "kind": "decode", "bgn": 1, "A": 4352, "crc": 1, "E": 8754, "rv": 0,
         "Qm": 6, "algo": 4, "iters": 10, "margin": 3.5, "n": 777, "harq": False},
        # belief propagation on the largest blocks
        {"name": "decode_bp_zc384_n1024", "kind": "decode", "bgn": 1, "A": 8424, "crc": 1, "E": 25344, "rv": 0,
         "Qm": 8, "algo": 0, "iters": 10, "margin": 4.0, "n": 1024, "harq": False},
        # LLRs that arrive in pinned host memory, results back in host memory
        {"name": "host_bg1_zc384_n2048", "kind": "host", "bgn": 1, "A": 8424, "crc": 1, "E": 25344, "rv": 0, "Qm": 8,
         "algo": 1, "iters": 8, "margin": 3.0, "n": 2048, "pinned": True},
        # code blocks of many users at once
        {"name": "mixed_n2048", "kind": "mixed", "algo": 1, "iters": 10, "margin": 4.5, "n": 2048, "a_max": 8424},
        # transport blocks of one serving batch, several code blocks each
        {"name": "tb_n32", "kind": "tb", "algo": 1, "iters": 10, "margin": 3.5, "n": 32, "a_max": 200000},
        # transmit side: the benchmark's code block
        {"name": "encode_bg1_zc384_n4096", "kind": "encode", "bgn": 1, "A": 8424, "crc": 1, "E": 25344, "rv": 0,
         "Qm": 8, "n": 4096},
        # the simulation channel, 64QAM
        {"name": "channel_qam64_n2048", "kind": "channel", "E": 25344, "Qm": 6, "noise_db": -14.0, "n": 2048},
        # one training step of the learned tables at the benchmark's size
        {"name": "train_bg2_zc64_n4096", "kind": "train", "bgn": 2, "A": 488, "crc": 1, "E": 1920, "Qm": 2, "T": 10,
         "n": 4096, "alpha_mode": "checkpoint", "ebn0_db": 1.5},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_code(rng, qms=(1, 2, 4, 6, 8), rvs=(0,), rate=(0.2, 0.9)):
    bgn = rng.choice((1, 1, 2))
    A = 8 * _log_int(rng, 8, (8424 if bgn == 1 else 3816) // 8)
    Qm = rng.choice(qms)
    B = A + 24
    R = rng.uniform(*rate)
    E = max(Qm, min(65520 // Qm * Qm, int(round(B / R / Qm)) * Qm))
    return {"bgn": bgn, "A": A, "crc": rng.choice((1, 1, 2, 3)), "E": E, "rv": rng.choice(rvs), "Qm": Qm}


def _edges(bgn, A):
    """Lifted edges of one block, about: 316 / 197 base edges times B / (22 or 10) rows."""
    return (316 / 22 if bgn == 1 else 197 / 10) * (A + 24)


def draw(rng):
    """One more case of the ranges the listed ones stand for; no dearer than the dearest of them."""
    kind = rng.choice(("call", "decode", "decode", "decode", "host", "mixed", "tb", "encode", "channel", "train"))
    if kind == "call":
        c = _draw_code(rng, rate=(0.2, 0.7))
        return {"kind": kind, **c, "algo": rng.choice((0, 1, 1, 3, 4)), "iters": rng.choice((8, 20, 32)),
                "margin": round(rng.uniform(2.5, 6.0), 2)}
    if kind in ("decode", "host"):
        algo = rng.choice((0, 1, 1, 1, 2, 3, 4)) if kind == "decode" else rng.choice((1, 1, 2, 4))
        # a repeated rate (more coded bits than the mother code has) now and then
        c = _draw_code(rng, rate=(0.15, 0.92))
        iters = rng.choice((5, 8, 10, 16))
        top = {0: 0.5e9, 4: 2e9}.get(algo, 4e9) / (8 if kind == "host" else 1)   # edges times iterations
        n_max = max(1, min(20000, int(top / (_edges(c["bgn"], c["A"]) * iters))))
        n_max = max(1, min(n_max, int(2e8 / c["E"])))
        n = _log_int(rng, 1, n_max)
        margin = round(rng.uniform(2.5, 5.5), 2) if rng.random() < 0.8 else -3.0
        if algo == 0:
            margin = abs(margin) + 1.0   # belief propagation without convergence is chaotic
        more = {"harq": rng.random() < 0.25} if kind == "decode" else {"pinned": rng.random() < 0.7}
        return {"kind": kind, **c, "algo": algo, "iters": iters, "margin": margin, "n": n, **more}
    if kind == "mixed":
        return {"kind": kind, "algo": rng.choice((1, 1, 2, 3)), "iters": rng.choice((8, 10)),
                "margin": round(rng.uniform(3.5, 5.5), 2), "n": _log_int(rng, 16, 2048),
                "a_max": rng.choice((1000, 3816, 8424))}
    if kind == "tb":
        return {"kind": kind, "algo": 1, "iters": rng.choice((8, 10)), "margin": round(rng.uniform(2.5, 5.0), 2),
                "n": _log_int(rng, 1, 48), "a_max": _log_int(rng, 2000, 200000)}
    if kind == "encode":
        c = _draw_code(rng, rvs=(0, 1, 2, 3))
        return {"kind": kind, **c, "n": _log_int(rng, 1, min(20000, int(1e8 / c["E"])))}
    if kind == "channel":
        Qm = rng.choice((1, 2, 4, 6, 8))
        E = Qm * _log_int(rng, 40, 25344 // Qm)
        return {"kind": kind, "E": E, "Qm": Qm, "noise_db": round(rng.uniform(-25.0, 2.0), 2),
                "n": _log_int(rng, 1, min(20000, int(5e7 / E)))}
    bgn, A, E = rng.choice(((2, 488, 1920), (1, 2440, 7392), (2, 1000, 3000), (1, 600, 1500), (2, 200, 800)))
    T = rng.choice((4, 6, 10))
    n = _log_int(rng, 32, int(2.5e8 / (_edges(bgn, A) * T)))
    return {"kind": "train", "bgn": bgn, "A": A, "crc": 1, "E": E, "Qm": 2, "T": T, "n": n,
            "alpha_mode": rng.choice(("single", "degree", "checkpoint")), "ebn0_db": round(rng.uniform(0.5, 2.0), 2)}


# ------------------------------------------------------------------ inputs


def _in_config(case):
    return (case["bgn"], case["A"], case["crc"], case["E"], case["rv"], case["Qm"], 0)


def _noise_db(B, E, Qm, margin):
    """Noise power (unit-energy symbols) for Es/N0 = Shannon limit of Qm B / E bits per symbol + margin."""
    eta = min(Qm * B / E, Qm - 0.05)
    return -(10.0 * math.log10(2.0 ** eta - 1.0) + margin)


def _payload(n, A, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 256, (n, A // 8), dtype=torch.uint8, device="cuda", generator=g)


def _received(cfg, n, margin, seed):
    """int16 LLRs [n, E] of n random blocks."""
    from deeplearning_5g_ldpc_decoder_b200 import channel_llrs, ldpc_encode

    bgn, A, crc, E, rv, Qm = cfg[:6]
    rm = ldpc_encode(_payload(n, A, seed), cfg)
    return channel_llrs(rm, E, Qm, _noise_db(A + 24, E, Qm, margin), seed=seed * 7919 + 13)


def _block_mix(case):
    """(bgn, A, crctype, E, rv, Qm) of a mixed batch: sizes over their logarithm, every modulation, rates 0.2 to 0.9.
    The composition belongs to the case; payloads and noise come from the seed."""
    rng = np.random.default_rng(case["n"] + case["a_max"])
    out = []
    for _ in range(case["n"]):
        A = 8 * int(round(math.exp(rng.uniform(math.log(3), math.log(case["a_max"] // 8)))))
        bgn = 2 if (A <= 292 or A <= 3816 and rng.random() < 0.4) else 1
        Qm = int(rng.choice((2, 4, 6, 8)))
        E = int(round((A + 24) / rng.uniform(0.2, 0.9) / Qm)) * Qm
        out.append((bgn, A, int(rng.integers(1, 4)), min(E, 65520), 0, Qm))
    return out


def prepare(case, seed):
    import deeplearning_5g_ldpc_decoder_b200 as pkg
    from deeplearning_5g_ldpc_decoder_b200 import capi

    kind = case["kind"]
    if kind == "call":
        llr = _received(_in_config(case), 1, case["margin"], seed).cpu().numpy()[0].copy()
        icfg = capi.make_in_config(*_in_config(case))
        bits = np.zeros((capi.gen_ldpc_parameters(icfg).B + 7) // 8, dtype=np.uint8)
        return {"kind": kind, "lib": capi.load_library(), "llr": llr, "bits": bits, "icfg": icfg,
                "dcfg": capi.make_decoder_config(_row(case))}
    if kind == "decode":
        llr = _received(_in_config(case), case["n"], case["margin"], seed)
        harq = None
        if case["harq"]:
            p = pkg.code_params(_in_config(case))
            harq = torch.zeros((case["n"], p.N + 2 * p.Zc), dtype=torch.int16, device="cuda")
        return {"kind": kind, "llr": llr, "cfg": _in_config(case), "row": _row(case), "harq": harq}
    if kind == "host":
        llr = _received(_in_config(case), case["n"], case["margin"], seed).cpu()
        return {"kind": kind, "llr": llr.pin_memory() if case["pinned"] else llr.numpy().copy(),
                "cfg": _in_config(case), "row": _row(case)}
    if kind == "mixed":
        from deeplearning_5g_ldpc_decoder_b200.mixed import MixedPlan

        cfgs = _block_mix(case)
        llrs = [_received(c + (0,), 1, case["margin"], seed * 100003 + i) for i, c in enumerate(cfgs)]
        plan = MixedPlan(cfgs, _row(case))
        return {"kind": kind, "plan": plan, "arena": plan.pack_llrs(llrs), "out": plan.outputs(),
                "stream": torch.cuda.Stream()}
    if kind == "tb":
        from deeplearning_5g_ldpc_decoder_b200 import tb

        rng = np.random.default_rng(case["n"] + case["a_max"])   # the blocks' sizes belong to the case
        rows, noise, cbs = [], [], 0
        for _ in range(case["n"]):
            A = math.exp(rng.uniform(math.log(200), math.log(case["a_max"])))
            R, Qm = rng.uniform(0.3, 0.88), int(rng.choice((2, 4, 6, 8)))
            bgn = tb.select_bg(int(A), R)
            A = tb.round_tbs(A, bgn)
            G = tb.coded_bits(A, bgn, Qm, R)
            C, _ = tb.code_block_count(A, bgn)
            cbs += C
            rows.append((A, G, Qm, 0, bgn, 0, 0))
            noise.append(_noise_db(R, 1.0, Qm, case["margin"]))
        rng = np.random.default_rng(seed)
        pay = [rng.integers(0, 256, r[0] // 8, dtype=np.uint8) for r in rows]
        tbs, arena, out_bytes = tb.encode_transport_blocks(pay, tb.tb_array(rows), noise, seed=seed)
        return {"kind": kind, "engine": tb.TbEngine(case["n"], cbs, _row(case)), "tbs": tbs, "arena": arena,
                "out": torch.zeros(out_bytes, dtype=torch.uint8, device="cuda")}
    if kind == "encode":
        return {"kind": kind, "info": _payload(case["n"], case["A"], seed), "cfg": _in_config(case)}
    if kind == "channel":
        g = torch.Generator(device="cuda").manual_seed(seed)
        rm = torch.randint(0, 256, (case["n"], (case["E"] + 7) // 8), dtype=torch.uint8, device="cuda", generator=g)
        return {"kind": kind, "rm": rm, "E": case["E"], "Qm": case["Qm"], "noise_db": case["noise_db"], "seed": seed}
    if kind == "train":
        from deeplearning_5g_ldpc_decoder_b200 import train

        model = train.NeuralLayeredMinSumDecoder((case["bgn"], case["A"], case["crc"], case["E"], 0, case["Qm"], 0),
                                                 num_iterations=case["T"], alpha_mode=case["alpha_mode"],
                                                 init_alpha=0.7, init_beta=0.02).cuda()
        noise = train.ebn0_to_noise_power_db(case["ebn0_db"], case["Qm"], model.B, case["E"])
        llr, target = train.make_training_batch(model, case["n"], noise, seed)
        return {"kind": kind, "model": model, "llr": llr, "target": target}
    raise ValueError(kind)


# ------------------------------------------------------------------ one pass


def run(state):
    import deeplearning_5g_ldpc_decoder_b200 as pkg

    kind = state["kind"]
    if kind == "call":
        status = state["lib"].cuda_ldpc_5g_decode(state["llr"].ctypes.data, state["bits"].ctypes.data,
                                                  ctypes.byref(state["icfg"]), ctypes.byref(state["dcfg"]))
        return {"status": int(status), "bits": state["bits"]}
    if kind == "decode":
        r = pkg.ldpc_decode(state["llr"], state["cfg"], state["row"], harq=state["harq"])
        return {"bits": r.hardbits, "status": r.status, "iterations": r.iterations, "harq": state["harq"]}
    if kind == "host":
        bits, status, iters = pkg.ldpc_decode_host(state["llr"], state["cfg"], state["row"])
        return {"bits": bits, "status": status, "iterations": iters}
    if kind == "mixed":
        with torch.cuda.stream(state["stream"]):
            bits, status, iters = state["plan"].decode(state["arena"], out=state["out"])
        return {"bits": bits, "status": status, "iterations": iters}
    if kind == "tb":
        status, iters = state["engine"].decode(state["tbs"], state["arena"], state["out"])
        return {"payload": state["out"], "status": status, "iterations": iters}
    if kind == "encode":
        return pkg.ldpc_encode(state["info"], state["cfg"])
    if kind == "channel":
        return pkg.channel_llrs(state["rm"], state["E"], state["Qm"], state["noise_db"], seed=state["seed"])
    from deeplearning_5g_ldpc_decoder_b200 import train

    model = state["model"]
    model.zero_grad(set_to_none=True)
    _, final = model(state["llr"], return_llr=True)
    loss = train.decoder_loss(final, state["target"], model.B)
    loss.backward()
    return {"loss": loss.detach(), "final": final.detach(), "d_raw_alpha": model.raw_alpha.grad,
            "d_raw_beta": model.raw_beta.grad}


# ------------------------------------------------------------------ what a pass cannot do without


def work(case):
    """Inputs read once, outputs written once; flops: 8 operations per lifted edge and iteration (subtract, magnitude,
    two minima, sign, select, add, clip), counted for every iteration where no block converges and for half of them
    (at most 5) otherwise."""
    kind, n = case["kind"], case.get("n", 1)
    if kind in ("call", "decode", "host"):
        its = case["iters"] if case["margin"] < 0 else min(5.0, case["iters"] / 2)
        B = case["A"] + 24
        by = n * (2 * case["E"] + B / 8 + 8)
        if case.get("harq"):
            by += n * 2 * (68 / 22 if case["bgn"] == 1 else 52 / 10) * B
        return {"bytes": by, "flops": 8 * n * its * _edges(case["bgn"], case["A"])}
    if kind in ("mixed", "tb"):
        mean = (case["a_max"] - 100) / math.log(case["a_max"] / 100)
        return {"bytes": n * mean * 4, "flops": 8 * n * 4 * _edges(1, mean)}
    if kind == "encode":
        return {"bytes": n * (case["A"] + case["E"]) / 8, "flops": n * _edges(case["bgn"], case["A"]) / 8}
    if kind == "channel":
        return {"bytes": n * (case["E"] / 8 + 2 * case["E"]), "flops": n * case["E"] * 10}
    B = case["A"] + 24
    return {"bytes": n * (2 * 4 * (68 / 22 if case["bgn"] == 1 else 52 / 10) * B + 8 * B),
            "flops": 24 * n * case["T"] * _edges(case["bgn"], case["A"])}


# ------------------------------------------------------------------ 64-bit values


def exact(case, seed):
    """Only training computes real numbers; every other path returns whole numbers and bytes.

    The model of the training path (unrolled layered min-sum, alpha * max(u - beta, 0) messages) and its gradients,
    in float64 with torch's own operations and autograd, on the inputs of prepare().  Minimum search and clipping at
    zero make the model piecewise linear: over many iterations float32 rounding lands some blocks on other pieces than
    float64, which hardly moves the LLRs but turns their gradients (16 to 41 % at 10 iterations), so gradients have a
    64-bit value only for few iterations."""
    if case["kind"] != "train":
        return None
    from deeplearning_5g_ldpc_decoder_b200 import capi

    s = prepare(case, seed)
    model, llr_all, target = s["model"], s["llr"].double(), s["target"].double()
    p = capi.gen_ldpc_parameters(capi.make_in_config(*model.in_config))   # the code's tables (data)
    Zc, R, T, n = int(p.Zc), model.num_rows, case["T"], case["n"]
    off = [int(p.HBG_offset_array[r]) for r in range(R + 1)]
    z = torch.arange(Zc, device="cuda")
    cols = [torch.stack([int(p.HBG_array[e]) * Zc + (z + int(p.Vij_array[e]) % Zc) % Zc
                         for e in range(off[r], off[r + 1])], dim=1) for r in range(R)]
    raw_a = model.raw_alpha.detach().double().requires_grad_()
    raw_b = model.raw_beta.detach().double().requires_grad_()
    lo, hi = model.alpha_min, model.alpha_max
    final, loss = [], 0.0
    for i in range(0, n, 512):
        a = (lo + (hi - lo) * torch.sigmoid(raw_a)).clamp(lo, hi)
        b = torch.sigmoid(raw_b).clamp(0.0, 1.0 - 1e-6)
        if model.alpha_mode == "single":
            a = a.reshape(1, 1).expand(T, R)
        elif model.alpha_mode == "degree":
            a = a[model.row_alpha_degree_indices].reshape(1, R).expand(T, R)
        lq = llr_all[i:i + 512]
        msgs = [0.0] * R
        for t in range(T):
            for r in range(R):
                flat, d = cols[r].reshape(-1), cols[r].shape[1]
                rel = lq[:, flat].reshape(-1, Zc, d) - msgs[r]
                sgn = torch.where(rel < 0, -1.0, 1.0).double()
                mag = rel.abs()
                m1, i1 = mag.min(dim=2, keepdim=True)
                first = torch.zeros_like(mag, dtype=torch.bool).scatter_(2, i1, True)
                m2, _ = mag.masked_fill(first, math.inf).min(dim=2, keepdim=True)
                u = torch.where(first, m2, m1)
                msgs[r] = sgn.prod(dim=2, keepdim=True) * sgn * (a[t, r] * torch.clamp(u - b[t, r], min=0.0))
                lq = lq.index_copy(1, flat, (rel + msgs[r]).reshape(-1, Zc * d))
        part = torch.nn.functional.binary_cross_entropy_with_logits(-lq[:, :model.B], target[i:i + 512],
                                                                    reduction="sum") / target.numel()
        part.backward()
        loss += float(part.detach())
        final.append(lq.detach())
    few = T <= 4
    return {"loss": torch.tensor(loss, dtype=torch.float64), "final": torch.cat(final),
            "d_raw_alpha": raw_a.grad if few else None, "d_raw_beta": raw_b.grad if few else None}
