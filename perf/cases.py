"""What the performance of this library is measured on: one rank's share of the work a user's program hands to it.

Every case goes through the public entry points (``Buffer`` and ``MoELayer``) on a group of one rank, with inputs drawn on
the GPU from a seed. The kinds of work:

* ``ll``      low-latency dispatch + combine, the communication pair around the experts of a decode step;
* ``normal``  get_dispatch_layout + dispatch + combine, the pair of a prefill or of a training forward pass, or (``cached``)
              the dispatch with a kept handle + combine of the backward pass;
* ``fused`` / ``fp8``  FP8 forward of one MoE layer (prefill): the overlapped pipeline and the step-by-step chain;
* ``decode``  FP8 forward of one MoE layer through the low-latency pair;
* ``train``   BF16 forward and backward of one MoE layer.

Sizes are those of the benchmarks (128 / 4096 tokens, hidden 7168, 256 experts, top-8, expert FFN 7168 -> 2048; training with
8192 tokens, hidden 4096, 64 experts, top-6, FFN 4096 -> 1408), smaller and ragged ones of the same layers, and in ``draw``
what lies between.
"""
import math

import torch

from deepep_efa_b200 import Buffer
from deepep_efa_b200.models.moe import MoEConfig, MoELayer

DEVICE = "cuda"


class SoloComm:
    """The communicator of a job with one rank."""

    def Get_rank(self):
        return 0

    def Get_size(self):
        return 1

    def allgather(self, obj):
        return [obj]


def listed():
    return [
        # one user's decode step, its kernels replayed from a CUDA graph: nothing but latency
        dict(name="ll_1", kind="ll", tokens=1, max_tokens=128, hidden=7168, experts=256, topk=8, wire="fp8", expert_out="symmetric",
             masked=0.0, graph=True),
        # the benchmark's decode batch, expert outputs in symmetric memory (read in place)
        dict(name="ll_128", kind="ll", tokens=128, max_tokens=128, hidden=7168, experts=256, topk=8, wire="fp8", expert_out="symmetric",
             masked=0.0, graph=False),
        # a partly filled batch of a BF16 model with dropped selections, expert outputs in ordinary device memory (pushed)
        dict(name="ll_77_bf16", kind="ll", tokens=77, max_tokens=128, hidden=4096, experts=64, topk=6, wire="bf16", expert_out="device",
             masked=0.05, graph=False),
        # a short prompt: launches, allocations and the one host wait
        dict(name="normal_61", kind="normal", tokens=61, hidden=4096, experts=64, topk=6, wire="bf16", cached=False, bias=0, overlap=False),
        # the benchmark's prefill batch, cast to FP8 on the way, BF16 back
        dict(name="normal_4096_fp8", kind="normal", tokens=4096, hidden=7168, experts=256, topk=8, wire="cast", cached=False, bias=0, overlap=False),
        # gradients of a ragged batch with the forward's handle, on the communication stream, with a residual added
        dict(name="normal_3001_cached", kind="normal", tokens=3001, hidden=4096, experts=64, topk=6, wire="bf16", cached=True, bias=1, overlap=True),
        # prefill through the overlapped FP8 layer, the benchmark's size
        dict(name="fused_4096", kind="fused", tokens=4096, hidden=7168, inter=2048, experts=256, topk=8, skew=0.0, native=True),
        # a ragged prompt through the step-by-step FP8 layer with fp32 block scales
        dict(name="fp8_777", kind="fp8", tokens=777, hidden=4096, inter=1408, experts=64, topk=6, skew=0.0, native=False),
        # decode of the benchmark's layer: streams every expert's weights
        dict(name="decode_128", kind="decode", tokens=128, max_tokens=128, hidden=7168, inter=2048, experts=256, topk=8, skew=0.0,
             native=True, graph=False),
        # decode of a smaller layer with a few live sequences, replayed from a CUDA graph
        dict(name="decode_20", kind="decode", tokens=20, max_tokens=128, hidden=4096, inter=1408, experts=64, topk=6, skew=0.0,
             native=True, graph=True),
        # the benchmark's training step, skewed routing
        dict(name="train_8192", kind="train", tokens=8192, hidden=4096, inter=1408, experts=64, topk=6, skew=1.2),
        # a ragged micro-batch of the same layer
        dict(name="train_999", kind="train", tokens=999, hidden=4096, inter=1408, experts=64, topk=6, skew=0.0),
    ]


def _log_int(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    """One more case of the same ranges: any kind, 1 to 8192 tokens (spread over their logarithm, odd numbers as they come),
    hidden sizes 1024 to 7168, 8 to 256 experts, top-1 to top-8."""
    kind = rng.choice(["ll", "ll", "normal", "normal", "fused", "fp8", "decode", "train"])
    experts = rng.choice([8, 16, 32, 60, 64, 128, 160, 256])
    topk = min(experts, rng.choice([1, 2, 4, 6, 8]))
    if kind == "ll":
        wire = rng.choice(["fp8", "fp8_pow2", "fp8_ue8m0", "bf16"])
        return dict(kind=kind, tokens=_log_int(rng, 1, 128), max_tokens=128, hidden=512 * rng.randint(2, 14) if wire == "fp8_ue8m0" else 128 * rng.randint(8, 56),
                    experts=experts, topk=topk, wire=wire, expert_out=rng.choice(["symmetric", "device"]), masked=rng.choice([0.0, 0.0, 0.02, 0.05]),
                    graph=rng.random() < 0.3)
    if kind == "normal":
        cached = rng.random() < 0.3
        return dict(kind=kind, tokens=_log_int(rng, 16, 8192), hidden=128 * rng.randint(8, 56), experts=experts, topk=topk,
                    wire="bf16" if cached else rng.choice(["bf16", "fp8", "cast"]), cached=cached, bias=rng.choice([0, 0, 1, 2]),
                    overlap=rng.random() < 0.3)
    hidden, inter = 256 * rng.randint(4, 28), 128 * rng.randint(4, 16)
    while experts * hidden * inter > 64 * 7168 * 2048:
        experts //= 2
    topk = min(experts, topk)
    skew = rng.choice([0.0, 0.0, 1.2])
    if kind == "decode":
        return dict(kind=kind, tokens=_log_int(rng, 1, 128), max_tokens=128, hidden=hidden, inter=inter, experts=experts, topk=topk, skew=skew,
                    native=rng.random() < 0.75, graph=rng.random() < 0.3)
    if kind == "train":
        return dict(kind=kind, tokens=_log_int(rng, 64, 4096), hidden=hidden, inter=inter, experts=experts, topk=topk, skew=skew)
    return dict(kind=kind, tokens=_log_int(rng, 64, 7168), hidden=hidden, inter=inter, experts=experts, topk=topk, skew=skew,
                native=rng.random() < 0.75)


# ---------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------
def _routing(case, gen):
    """Top-k expert ids without replacement (uniform, or skewed like 1 / (e + 1)^s) and softmax weights."""
    tokens, experts, topk = case["tokens"], case["experts"], case["topk"]
    u = torch.rand(tokens, experts, generator=gen, device=DEVICE).clamp_(1e-7, 1 - 1e-7)
    scores = -torch.log(-torch.log(u))
    if case.get("skew", 0.0) > 0:
        scores -= case["skew"] * torch.log(torch.arange(1, experts + 1, device=DEVICE, dtype=torch.float32))
    idx = scores.topk(topk, dim=-1).indices
    weights = torch.softmax(torch.randn(tokens, topk, generator=gen, device=DEVICE), dim=-1)
    if case.get("masked", 0.0) > 0:
        idx[torch.rand(tokens, topk, generator=gen, device=DEVICE) < case["masked"]] = -1
    return idx, weights


def _tokens(case, gen):
    return torch.randn(case["tokens"], case["hidden"], generator=gen, device=DEVICE).to(torch.bfloat16)


def _capture(step):
    """Two steps in one CUDA graph: the low-latency buffers alternate between two parities, so a program captures them in pairs."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
        step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            outputs = [step(), step()]
    torch.cuda.current_stream().wait_stream(side)
    return graph, outputs


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind, tokens, hidden, experts, topk = (case[k] for k in ("kind", "tokens", "hidden", "experts", "topk"))
    state = dict(case=case, x=_tokens(case, gen))
    state["idx"], state["weights"] = _routing(case, gen)
    mib = 1 << 20
    # explicitly_destroy: the symmetric memory lives as long as the last tensor in it, so results may outlive the buffer object
    low_latency = Buffer.get_low_latency_rdma_size_hint(case["max_tokens"], hidden, 1, experts) if kind in ("ll", "decode") else 0
    if kind == "ll":
        shape = [experts, case["max_tokens"], hidden]
        buf = Buffer(None, experts * case["max_tokens"] * hidden * 2 + 4 * mib, low_latency, low_latency_mode=True, explicitly_destroy=True,
                     comm=SoloComm())
        # what the experts of this rank wrote: in symmetric memory, or in a tensor of their own
        out = buf.empty_symmetric(shape, torch.bfloat16) if case["expert_out"] == "symmetric" else torch.empty(shape, dtype=torch.bfloat16, device=DEVICE)
        for e in range(experts):
            out[e] = torch.randn(shape[1:], generator=gen, device=DEVICE).to(torch.bfloat16)
        state["expert_out"] = out
    elif kind == "normal":
        buf = Buffer(None, 8 * tokens * hidden * 2 + 16 * tokens * topk * 16 + 64 * mib, explicitly_destroy=True, comm=SoloComm())
        if case["wire"] == "fp8":
            blocks = state["x"].float().view(tokens, -1, 128)
            scales = blocks.abs().amax(dim=2).clamp(min=1e-4) / 448.0
            state["x"] = ((blocks / scales.unsqueeze(2)).view(tokens, hidden).to(torch.float8_e4m3fn), scales)
        state["expert_out"] = buf.empty_symmetric([tokens, hidden], torch.bfloat16)
        state["expert_out"].copy_(_tokens(case, gen))
        bias = [_tokens(case, gen) for _ in range(case["bias"])]
        state["bias"] = None if not bias else bias[0] if len(bias) == 1 else tuple(bias)
        if case["cached"]:
            per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(state["idx"], experts)
            state["handle"] = buf.dispatch(state["x"], num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert,
                                           topk_idx=state["idx"], topk_weights=state["weights"])[4]
    else:
        inter = case["inter"]
        if kind == "fused":
            rows = tokens * min(topk, experts) + experts * 127 + 128
            arena = rows * (hidden + hidden // 128 * 4 + 4) + tokens * topk * hidden * 2
        elif kind == "fp8":
            arena = 2 * tokens * (hidden * 3 + hidden // 32 + topk * 12 + 4)
        elif kind == "train":
            arena = 12 * tokens * (hidden * 2 + topk * 12 + 4)
        else:
            arena = 0
        buf = Buffer(None, arena + 64 * mib, low_latency, low_latency_mode=kind == "decode", explicitly_destroy=True,
                     comm=SoloComm())
        layer = MoELayer(MoEConfig(hidden=hidden, intermediate=inter, num_experts=experts, num_topk=topk, init_std=0.02), buf, seed=seed)
        state["layer"] = layer
        if kind == "train":
            state["x"].requires_grad_(True)
            state["weights"].requires_grad_(True)
            state["grad"] = _tokens(case, gen)
        else:
            layer.prepare_fp8(native_block_scaling=case["native"])
    state["buffer"] = buf
    if case.get("graph"):
        state["graph"], state["outputs"] = _capture(lambda: _RUN[kind](state))
    return state


# ---------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------
def _run_ll(s):
    case, buf = s["case"], s["buffer"]
    wire = case["wire"]
    recv, count, handle, _, _ = buf.low_latency_dispatch(s["x"], s["idx"], case["max_tokens"], case["experts"], use_fp8=wire != "bf16",
                                                         round_scale=wire in ("fp8_pow2", "fp8_ue8m0"), use_ue8m0=wire == "fp8_ue8m0")
    combined, _, _ = buf.low_latency_combine(s["expert_out"], s["idx"], s["weights"], handle)
    return recv, count, handle[0], handle[1], combined


def _run_normal(s):
    case, buf = s["case"], s["buffer"]
    overlap = case["overlap"]
    how = dict(previous_event=Buffer.capture(), async_finish=True, allocate_on_comm_stream=True) if overlap else {}
    if case["cached"]:
        recv, _, _, _, _, event = buf.dispatch(s["x"], handle=s["handle"], **how)
        handle, outputs, recv_weights = s["handle"], [recv], None
    else:
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(s["idx"], case["experts"])
        if overlap:
            how["previous_event"] = Buffer.capture()
        recv, recv_idx, recv_weights, _, handle, event = buf.dispatch(
            s["x"], num_tokens_per_rank=per_rank, is_token_in_rank=in_rank, num_tokens_per_expert=per_expert, topk_idx=s["idx"],
            topk_weights=s["weights"], quantize_fp8=case["wire"] == "cast", **how)
        outputs = [recv, recv_idx, recv_weights, per_expert]
    event.current_stream_wait()
    if overlap:
        how["previous_event"] = Buffer.capture()
    combined, combined_weights, event = buf.combine(s["expert_out"], handle, topk_weights=recv_weights, bias=s["bias"], **how)
    event.current_stream_wait()
    return outputs + [combined, combined_weights]


def _run_fused(s):
    return s["layer"].forward_fused(s["x"], s["idx"], s["weights"])


def _run_fp8(s):
    return s["layer"].forward_fp8(s["x"], s["idx"], s["weights"])


def _run_decode(s):
    return s["layer"].forward_low_latency(s["x"], s["idx"], s["weights"], num_max_tokens=s["case"]["max_tokens"])


def _run_train(s):
    layer, x, weights = s["layer"], s["x"], s["weights"]
    layer.zero_grad(set_to_none=True)
    x.grad = weights.grad = None
    y = layer(x, s["idx"], weights)
    y.backward(s["grad"])
    return y.detach(), x.grad, weights.grad, layer.w13.grad, layer.w2.grad


_RUN = dict(ll=_run_ll, normal=_run_normal, fused=_run_fused, fp8=_run_fp8, decode=_run_decode, train=_run_train)


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["outputs"]
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exactly it is computed
# ---------------------------------------------------------------------------------------------------------
def work(case):
    """Bytes: every input read once and every output written once. Operations: those of the sums and products asked for."""
    kind, tokens, hidden, experts, topk = (case[k] for k in ("kind", "tokens", "hidden", "experts", "topk"))
    row = hidden * 2
    if kind == "ll":
        picks = tokens * topk * (1 - case["masked"])
        wire = dict(bf16=hidden * 2, fp8=hidden + hidden // 32, fp8_pow2=hidden + hidden // 32, fp8_ue8m0=hidden + hidden // 128)[case["wire"]]
        moved = 2 * tokens * row + picks * (wire + 4 + row) + tokens * topk * 12 + experts * 12
        steps = 2 if case["graph"] else 1
        return {"bytes": steps * moved, "flops": steps * 2 * picks * hidden}
    if kind == "normal":
        fp8_row = hidden + hidden // 32
        read = fp8_row if case["wire"] == "fp8" else row
        written = row if case["wire"] == "bf16" else fp8_row
        routing = 0 if case["cached"] else topk * (2 * 12 + 2 * 4)
        return {"bytes": tokens * (read + written + (2 + case["bias"]) * row + routing), "flops": tokens * hidden * max(1, case["bias"])}
    matrix = 3 * hidden * case["inter"]
    flops = 2.0 * tokens * topk * matrix
    if kind == "train":
        return {"bytes": 2 * 3 * experts * matrix + tokens * 4 * row, "flops": 3 * flops}
    # experts that at least one token picks, on average
    share = [(e + 1) ** -case["skew"] for e in range(experts)]
    used = sum(1 - (1 - min(1.0, topk * p / sum(share))) ** tokens for p in share)
    steps = 2 if case.get("graph") else 1
    return {"bytes": steps * (used * matrix + 2 * tokens * row), "flops": steps * flops}


def tolerance(case):
    """Results are BF16, summed in fp32; what travels as FP8 is rounded from the same values. Inside an FP8 layer another order
    of summation now and then rounds an intermediate value to the neighbouring FP8 number."""
    return {"rel": 5e-3} if case["kind"] in ("ll", "normal") else {"rel": 1e-2}
