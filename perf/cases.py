"""Workloads of the MoE block, as a serving program calls it on one GPU.

Two layer shapes, those of bench.py: "120b" (128 experts) and "20b" (32 experts), hidden and intermediate size
2880, four experts per token, MXFP4 expert weights with uniform codes and scale exponents in [-8, -4].  Routing is
uniform, or skewed by a router bias that makes expert popularity follow Zipf(1.2).  Row counts go from one decode
row to a prefill chunk of 8192.  A program loads its layers once and then serves batch after batch from one handle
sized for its largest batch, so the handles are made on first use and shared by all cases of a shape; what a seed
decides is the batch.

Forms of a case:
  forward  normalised rows in device memory -> block output (moe_forward)
  block    residual stream x += MoE(rmsnorm(x) * gain), in place (moe_block)
  host     four batches in pinned host memory through moe_forward_host_submit/_wait, three in flight
  shard    one rank's share of a tensor-parallel group of four on the union of the group's rows: 720 of the 2880
           intermediate features of every expert, partial output
  quantise fp32 expert weights -> MXFP4 codes and scales on the device (checkpoint loading)
"""
import importlib
import math

import numpy as np
import torch

moe = importlib.import_module("gpt-oss_b200")

EXPERTS = {"120b": 128, "20b": 32}
H = D = 2880
K = 4
MAX_ROWS = 8192
ZIPF_S = 1.2
HOST_BATCHES, HOST_IN_FLIGHT = 4, 3
LOGIT_STD = 0.02 * math.sqrt(H)          # rows of unit rms against a router weight ~ N(0, 0.02)

_handles = {}                            # (shape, tp) -> (MoeBlock, layers loaded)


def listed():
    def case(name, form, shape, rows, zipf=False):
        return {"name": name, "form": form, "shape": shape, "rows": rows, "zipf": zipf}
    return [
        # one user's decode step: four experts read, everything else is latency
        case("decode_1", "forward", "120b", 1),
        # a small decode batch: most experts get one or two rows
        case("decode_32", "forward", "120b", 32),
        # the small model at the batch its CPU reference is quoted on
        case("decode_20b_64", "forward", "20b", 64),
        # a decode batch in the calling form of the runtime: norm in front, residual add behind
        case("block_256", "block", "120b", 256),
        # an odd batch with popular and idle experts
        case("block_zipf_777", "block", "120b", 777, zipf=True),
        # the headline batch
        case("decode_1856", "forward", "120b", 1856),
        # the same batch with one expert taking most rows
        case("zipf_1856", "forward", "120b", 1856, zipf=True),
        # the small model's decode batch
        case("block_20b_1536", "block", "20b", 1536),
        # a prefill chunk
        case("prefill_8192", "forward", "120b", 8192),
        # a rank of a four-GPU group at 1856 rows per rank
        case("shard_7424", "shard", "120b", 7424),
        # batches that arrive in and return to host memory
        case("host_1856", "host", "120b", 1856),
        # the MLP1 weights of eight experts of an fp32 checkpoint
        {"name": "quantise_8_experts", "form": "quantise", "values": 8 * 2 * D * H},
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    form = rng.choice(["forward", "forward", "forward", "block", "block", "block", "shard", "host", "quantise"])
    if form == "quantise":
        return {"form": form, "values": log_int(1 << 20, 8 * 2 * D * H)}
    shape = "120b" if form == "shard" else rng.choice(["120b", "120b", "20b"])
    lo, hi = {"shard": (4, 7424), "host": (1, 1856)}.get(form, (1, MAX_ROWS))
    return {"form": form, "shape": shape, "rows": log_int(lo, hi), "zipf": rng.random() < 0.4}


def _bits(t):
    """bf16 tensor -> its bit patterns as a numpy array."""
    return t.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)


def _layer(n_experts, zipf):
    g = torch.Generator(device="cuda")
    g.manual_seed(n_experts)

    def codes(*shape):
        return torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=g).cpu().numpy()

    def scales(*shape):
        return torch.randint(119, 124, shape, dtype=torch.uint8, device="cuda", generator=g).cpu().numpy()

    def normal(*shape):
        return 0.02 * torch.randn(shape, device="cuda", generator=g)
    E = n_experts
    layer = {
        "w1_codes": codes(E, 2 * D, H // 2), "w1_scales": scales(E, 2 * D, H // 32), "b1": _bits(normal(E, 2 * D)),
        "w2_codes": codes(E, H, D // 2), "w2_scales": scales(E, H, D // 32), "b2": _bits(normal(E, H)),
        "router_w": normal(E, H).cpu().numpy(), "router_b": normal(E).cpu().numpy(),
    }
    if zipf:
        layer["router_b"] = moe.synth.zipf_router_bias(E, ZIPF_S)
    return layer


def _handle(shape, tp, zipf):
    """The handle a program of this shape keeps, and the index of its uniform or its skewed layer."""
    if (shape, tp) not in _handles:
        _handles[shape, tp] = (moe.MoeBlock(H, D, EXPERTS[shape], top_k=K, n_layers=2, max_rows=MAX_ROWS, tp_size=tp,
                                            tp_rank=0), set())
    blk, loaded = _handles[shape, tp]
    layer = int(zipf)
    if layer not in loaded:
        blk.load_layer(layer, _layer(EXPERTS[shape], zipf))
        loaded.add(layer)
    return blk, layer


def _normalised(rows, g):
    x = torch.randn((rows, H), device="cuda", generator=g)
    return (x * torch.rsqrt(x.square().mean(dim=1, keepdim=True) + 1e-5)).to(torch.bfloat16)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    form = case["form"]
    if form == "quantise":
        n = case["values"]
        blocks = (n + 31) // 32
        return {"form": form, "n": n, "src": 0.02 * torch.randn(n, device="cuda", generator=g),
                "codes": torch.empty(blocks * 16, dtype=torch.uint8, device="cuda"),
                "scales": torch.empty(blocks, dtype=torch.uint8, device="cuda")}
    blk, layer = _handle(case["shape"], 4 if form == "shard" else 1, case["zipf"])
    rows = case["rows"]
    state = {"form": form, "blk": blk, "layer": layer, "rows": rows}
    if form == "host":
        state["in"] = [_normalised(rows, g).view(torch.int16).cpu().pin_memory() for _ in range(HOST_BATCHES)]
        state["out"] = [torch.empty((rows, H), dtype=torch.int16, pin_memory=True) for _ in range(HOST_BATCHES)]
    elif form == "block":
        # rows of a residual stream: row scales over two decades, a few strong channels
        x = torch.randn((rows, H), device="cuda", generator=g)
        x *= torch.exp(torch.empty((rows, 1), device="cuda").uniform_(math.log(0.2), math.log(20.0), generator=g))
        x[:, torch.randperm(H, device="cuda", generator=g)[:H // 64]] *= 8.0
        state["x0"] = x.to(torch.bfloat16)
        state["x"] = torch.empty_like(state["x0"])
        state["gain"] = (1.0 + 0.25 * torch.randn(H, device="cuda", generator=g)).to(torch.bfloat16)
    else:
        state["t"] = _normalised(rows, g)
        state["out"] = torch.empty_like(state["t"])
    return state


def run(state):
    form = state["form"]
    if form == "quantise":
        moe.quantize_mxfp4(state["src"].data_ptr(), state["n"], state["codes"].data_ptr(), state["scales"].data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        return state["codes"], state["scales"]
    blk, layer, rows = state["blk"], state["layer"], state["rows"]
    if form == "host":
        tickets = []
        for i in range(HOST_BATCHES):
            if i >= HOST_IN_FLIGHT:
                blk.forward_host_wait(tickets[i - HOST_IN_FLIGHT])
            tickets.append(blk.forward_host_submit(layer, state["in"][i].numpy().view(np.uint16),
                                                   state["out"][i].numpy().view(np.uint16)))
        for t in tickets[-HOST_IN_FLIGHT:]:
            blk.forward_host_wait(t)
        return [o.view(torch.bfloat16) for o in state["out"]]
    stream = torch.cuda.current_stream().cuda_stream
    if form == "block":
        state["x"].copy_(state["x0"])    # the attention's output arrives in the residual buffer
        blk.block(layer, state["x"].data_ptr(), state["gain"].data_ptr(), rows, stream=stream)
        return state["x"]
    blk.forward(layer, state["t"].data_ptr(), rows, state["out"].data_ptr(), stream=stream)
    return state["out"]


def _active_experts(n_experts, rows, zipf):
    """Experts that at least one of the rows selects (a fixed sample of the router's logits)."""
    rng = np.random.default_rng(rows)
    logits = rng.normal(0.0, LOGIT_STD, size=(rows, n_experts))
    if zipf:
        logits += moe.synth.zipf_router_bias(n_experts, ZIPF_S)
    return len(np.unique(np.argpartition(logits, -K, axis=1)[:, -K:]))


def work(case):
    if case["form"] == "quantise":
        n = case["values"]
        return {"bytes": 4 * n + (n + 31) // 32 * 17, "flops": 0}
    E, rows, form = EXPERTS[case["shape"]], case["rows"], case["form"]
    inter = D // 4 if form == "shard" else D
    flops = rows * (K * 6 * H * inter + 2 * H * E)
    nbytes = (_active_experts(E, rows, case["zipf"]) * moe.synth.weight_bytes_per_expert(H, inter)
              + rows * H * 4 + E * H * 4 + (2 * H if form == "block" else 0))
    n = HOST_BATCHES if form == "host" else 1
    return {"bytes": n * nbytes, "flops": n * flops}


def tolerance(case):
    if case["form"] == "quantise":
        return "exact"
    # bf16 outputs of two contractions whose intermediate keeps 8 significant bits; the tensor-core and the
    # CUDA-core path of the library differ by 1.6e-3 (largest difference 7.8e-3 of the value or the rms)
    return {"rel": 6.5e-3, "max": 3.2e-2}
