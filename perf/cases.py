"""Workloads of the expert-parallel MoE library on one GPU, through the public `Buffer` API.

Four kinds of call, each as a program makes it:

  train         `teramoe_autograd` and `backward`: one MoE layer of a training step
  forward       `teramoe_forward`: the same layer at inference, decode batches and prefill
  comm          `get_dispatch_layout`, `deepep_dispatch`, `deepep_combine`: the un-fused exchange around a program's own
                expert GEMMs
  low_latency   `low_latency_dispatch`, `low_latency_combine`: the exchange of a decoding server

The layer shapes are those of the benchmark (`bench.py`) and of the tests. `draw` spreads the same parameters over their
ranges. Inputs are synthetic: N(0, 1) activations and gradients, N(0, 0.02) weights, random routing.
"""
import math
import weakref

import torch

import teramoe_b200 as tm

DEV = "cuda"
MAX_TRAIN_FLOPS = 18.0 * 32768 * 8 * 7168 * 2048
MAX_WEIGHTS = 32 * 3 * 2048 * 7168

# One buffer per set of parameters, alive as long as any state uses it: a program constructs its Buffer once and runs every
# step through it.
_buffers = weakref.WeakValueDictionary()


def _train(name, T, H, I, E, K, skew=0.0, **kw):
    case = {"name": name, "kind": "train", "T": T, "H": H, "I": I, "E": E, "K": K, "skew": skew, "idx": "int64", "drop": 0.0,
            "sms": 24, "batch": 2048}
    case.update(kw)
    return case


def _forward(name, T, H, I, E, K, **kw):
    case = _train(name, T, H, I, E, K, **kw)
    case["kind"] = "forward"
    return case


def _comm(name, T, H, E, K, fp8, cached, **kw):
    case = {"name": name, "kind": "comm", "T": T, "H": H, "E": E, "K": K, "skew": 0.0, "idx": "int64", "drop": 0.0, "fp8": fp8,
            "cached": cached}
    case.update(kw)
    return case


def _low_latency(name, T, M, H, E, K, wire, logfmt, hook, **kw):
    case = {"name": name, "kind": "low_latency", "T": T, "M": M, "H": H, "E": E, "K": K, "skew": 0.0, "idx": "int64", "drop": 0.0,
            "wire": wire, "logfmt": logfmt, "hook": hook}
    case.update(kw)
    return case


def listed():
    return [
        # the smallest training step: a debugging model or a micro-batch, where launches and host work decide
        _train("train_tiny", 512, 512, 256, 4, 2),
        # a mid-size layer with the documented schedule arguments: the shape of the accuracy test
        _train("train_medium", 4096, 2048, 2048, 16, 8, sms=48, batch=4096),
        # the layer whose latency is published for the original library, per rank
        _train("train_published", 8192, 2048, 3072, 16, 6),
        # the benchmark's default: a fine-grained large layer, the ordinary production step
        _train("train_large", 8192, 7168, 2048, 32, 8, sms=32),
        # narrow experts: little arithmetic for every row that moves
        _train("train_sparse", 16384, 7168, 512, 32, 8, sms=48, batch=4096),
        # a long step with skewed routing (hottest expert about three times the mean): the largest call
        _train("train_imbalanced", 32768, 7168, 2048, 32, 8, skew=0.65),
        # decoding: a few tokens through the large layer, bound by reading the weights
        _forward("forward_decode", 32, 7168, 2048, 32, 8),
        # prefill of a ragged batch, 32-bit routing indices, some entries without an expert
        _forward("forward_prefill", 3001, 7168, 2048, 32, 8, idx="int32", drop=0.05),
        # the un-fused exchange of a training step, forward and backward: dispatch, combine, then the gradients through the
        # cached layout and the combine that also carries the routing weights' gradients
        _comm("comm_bf16", 4096, 7168, 32, 8, False, True),
        # the exchange of a ragged prefill batch with FP8 rows
        _comm("comm_fp8_ragged", 1003, 7168, 32, 8, True, False),
        # a decoding server's exchange: FP8 rows out, bf16 rows back
        _low_latency("ll_fp8", 128, 128, 7168, 32, 8, "fp8", False, False),
        # the same with packed power-of-two scales, 10-bit rows back and receive hooks, a partly filled batch
        _low_latency("ll_ue8m0_logfmt", 77, 128, 7168, 32, 8, "ue8m0", True, True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_layer(rng, lo, hi):
    """Layer sizes and a token count between lo and hi, within the weights and the work of the largest listed case."""
    while True:
        H = rng.choice((512, 1024, 2048, 4096, 5120, 7168))
        I = rng.choice((256, 512, 768, 1024, 1536, 2048, 3072, 14336))
        E = rng.choice((4, 8, 16, 32, 64))
        K = rng.choice((2, 4, 6, 8))
        T = _log_int(rng, lo, hi)
        if K < E and E * 3 * H * I <= MAX_WEIGHTS and 18.0 * T * K * H * I <= MAX_TRAIN_FLOPS and T * K <= 32768 * 8:
            return T, H, I, E, K


def draw(rng):
    kind = rng.choice(("train", "train", "train", "forward", "forward", "comm", "comm", "low_latency", "low_latency"))
    more = {"idx": rng.choice(("int64", "int32")), "drop": rng.choice((0.0, 0.0, 0.05)), "skew": rng.choice((0.0, 0.0, 0.5))}
    if kind == "train":
        T, H, I, E, K = _draw_layer(rng, 64, 32768)
        case = _train("", T, H, I, E, K, sms=rng.choice((24, 32, 48)), batch=rng.choice((1024, 2048, 4096)), **more)
    elif kind == "forward":
        T, H, I, E, K = _draw_layer(rng, 1, 8192)
        case = _forward("", T, H, I, E, K, **more)
    elif kind == "comm":
        case = _comm("", _log_int(rng, 64, 16384), rng.choice((2048, 4096, 5120, 7168)), rng.choice((8, 32, 64, 256)),
                     rng.choice((2, 4, 6, 8)), rng.random() < 0.5, rng.random() < 0.5, **more)
    else:
        T = _log_int(rng, 1, 512)
        case = _low_latency("", T, max(64, -(-T // 64) * 64), rng.choice((2048, 4096, 5120, 7168)), rng.choice((8, 16, 32, 64)),
                            rng.choice((2, 4, 6, 8)), rng.choice(("bf16", "fp8", "fp8_pow2", "ue8m0")), rng.random() < 0.3,
                            rng.random() < 0.5, **more)
    del case["name"]
    return case


def _buffer(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    buf = _buffers.get(key)
    if buf is None:
        if case["kind"] == "low_latency":
            size = tm.Buffer.get_low_latency_rdma_size_hint(case["M"], case["H"], 1, case["E"])
            buf = tm.Buffer(None, size, low_latency_mode=True)
        else:
            buf = tm.Buffer(None, int(2e9), int(1e9))
        _buffers[key] = buf
    return buf


def _routing(case, gen):
    """Top-k of random logits; `skew` is the exponent of a Zipf-like preference among the experts."""
    T, E, K = case["T"], case["E"], case["K"]
    logits = -torch.log(-torch.log(torch.rand(T, E, device=DEV, generator=gen).clamp(1e-7, 1 - 1e-7)))
    if case["skew"]:
        rank = torch.randperm(E, device=DEV, generator=gen) + 1
        logits -= case["skew"] * torch.log(rank.float())
    top = torch.topk(logits, K, dim=1)
    idx, w = top.indices, torch.softmax(top.values, dim=1).float()
    if case["drop"]:
        gone = torch.rand(T, K, device=DEV, generator=gen) < case["drop"]
        gone[:, 0] = False
        idx = idx.masked_fill(gone, -1)
    return idx.to(torch.int32 if case["idx"] == "int32" else torch.int64).contiguous(), w.contiguous()


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    T, H, E, K = case["T"], case["H"], case["E"], case["K"]
    bf = dict(device=DEV, dtype=torch.bfloat16, generator=gen)
    idx, w = _routing(case, gen)
    s = {"case": case, "buf": _buffer(case), "x": torch.randn(T, H, **bf), "idx": idx, "w": w}
    if case["kind"] in ("train", "forward"):
        I = case["I"]
        s["W_gateup"] = torch.randn(E, 2 * I, H, **bf).mul_(0.02)
        s["W_down"] = torch.randn(E, H, I, **bf).mul_(0.02)
        s["opts"] = {"num_dispatch_sms": case["sms"], "num_combine_sms": case["sms"], "compute_batch_size": case["batch"]}
        if case["kind"] == "train":
            s["go"] = torch.randn(T, H, **bf)
            for leaf in ("x", "w", "W_gateup", "W_down"):
                s[leaf].requires_grad_(True)
    elif case["kind"] == "comm":
        s["y"] = torch.randn(T, H, **bf)                   # the program's expert outputs: one row per received token
        if case["fp8"]:
            s["x"] = tm.low_latency.fp8_quantize(s["x"])
    else:
        # where tokens sit in the packed receive tensor: expert e's rows are the first ones of its M rows
        sent = torch.bincount(idx[idx >= 0].long(), minlength=E)
        row = torch.arange(case["M"], device=DEV)
        s["valid"] = (row.view(1, -1) < sent.view(-1, 1)).flatten().nonzero().flatten()
        s["y"] = torch.randn(E, case["M"], H, **bf).mul_(0.1)      # the program's expert outputs
    return s


def _run_train(s):
    for leaf in ("x", "w", "W_gateup", "W_down"):
        s[leaf].grad = None
    out = s["buf"].teramoe_autograd(s["x"], s["idx"], s["w"], s["W_gateup"], s["W_down"], s["case"]["E"], **s["opts"])
    out.backward(s["go"])
    return out.detach(), s["x"].grad, s["w"].grad, s["W_gateup"].grad, s["W_down"].grad


def _run_forward(s):
    return s["buf"].teramoe_forward(s["x"], s["idx"], s["w"], s["W_gateup"], s["W_down"], s["case"]["E"], **s["opts"])


def _run_comm(s):
    buf, case = s["buf"], s["case"]
    per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(s["idx"], case["E"])
    recv_x, recv_idx, recv_w, counts, handle, _ = buf.deepep_dispatch(
        s["x"], topk_idx=s["idx"], topk_weights=s["w"], num_tokens_per_rank=per_rank, is_token_in_rank=in_rank,
        num_tokens_per_expert=per_expert)
    out, _, _ = buf.deepep_combine(s["y"], handle)
    res = [per_rank, per_expert, in_rank, recv_x, recv_idx, recv_w, torch.tensor(counts), out]
    if case["cached"]:
        grad_rows, *_ = buf.deepep_dispatch(s["y"], handle=handle)
        dx, dw, _ = buf.deepep_combine(grad_rows, handle, topk_weights=recv_w)
        res += [grad_rows, dx, dw]
    return res


def _run_low_latency(s):
    buf, case = s["buf"], s["case"]
    wire = case["wire"]
    recv, count, handle, _, hook = buf.low_latency_dispatch(
        s["x"], s["idx"], case["M"], case["E"], use_fp8=wire != "bf16", round_scale=wire in ("fp8_pow2", "ue8m0"),
        use_ue8m0=wire == "ue8m0", return_recv_hook=case["hook"])
    if hook is not None:
        hook()
    # the expert GEMM reads the rows that hold tokens
    rows, scales = recv if isinstance(recv, tuple) else (recv, None)
    n = case["E"] * case["M"]
    res = [count, rows.view(torch.int32).view(n, -1).index_select(0, s["valid"]).view(rows.dtype)]
    if scales is not None:
        res.append(scales.reshape(n, -1).index_select(0, s["valid"]))
    out, _, hook = buf.low_latency_combine(s["y"], s["idx"], s["w"], handle, use_logfmt=case["logfmt"], return_recv_hook=case["hook"])
    if hook is not None:
        hook()
    return res + [out]


def run(state):
    return {"train": _run_train, "forward": _run_forward, "comm": _run_comm, "low_latency": _run_low_latency}[state["case"]["kind"]](state)


def work(case):
    T, H, E, K = case["T"], case["H"], case["E"], case["K"]
    live = 1.0 - case["drop"] * (K - 1) / K
    rows = T * K * live
    routing = T * K * (8 if case["idx"] == "int64" else 4) + T * K * 4
    if case["kind"] in ("train", "forward"):
        I = case["I"]
        hit = E * (1.0 - (1.0 - live * K / E) ** T)                # experts that any token chose: only their weights are read
        weights = 3.0 * H * I * 2
        if case["kind"] == "forward":
            return {"bytes": 2.0 * T * H * 2 + routing + hit * weights, "flops": 6.0 * rows * H * I}
        return {"bytes": 4.0 * T * H * 2 + routing + T * K * 4 + (hit + E) * weights, "flops": 18.0 * rows * H * I}
    if case["kind"] == "comm":
        row_in = H + H // 128 * 4 if case["fp8"] else 2 * H
        once = 2.0 * T * row_in + 2.0 * T * H * 2 + 2.0 * routing
        return {"bytes": once + (4.0 * T * H * 2 + 2.0 * T * K * 4 if case["cached"] else 0.0), "flops": 0}
    row_out = {"bf16": 2.0 * H, "fp8": H + H / 32, "fp8_pow2": H + H / 32, "ue8m0": H + H / 128}[case["wire"]]
    return {"bytes": 2.0 * T * H + rows * row_out + rows * 2.0 * H + T * H * 2.0 + routing, "flops": 0}


def tolerance(case):
    if case["kind"] == "comm":
        return "exact"          # rows, indices and weights are moved; on one rank the sum over ranks has one term
    return {"rel": 1e-2}        # bf16 results and intermediates; e4m3 rows and their scales, weighted sums rounded to bf16
