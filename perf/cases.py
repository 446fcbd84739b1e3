"""The workloads that this framework's speed is judged by, each through the entry points a model calls.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones of the same ranges.  ``prepare`` makes
what a program has in hand before the call (streams, carried state, flags, parameters), ``run`` is one pass.
Training cases are one forward and one backward through autograd; inference cases run without gradients;
a decoding pass is one token through all layers of a model's packed state.  Sizes are those of the
benchmark configurations and their neighbours; the value distributions are those of the operators'
producers (``jaxrwkv_b200.synthetic``).
"""
import torch

from jaxrwkv_b200 import rwkv4, rwkv5_2, rwkv6, rwkv7
from jaxrwkv_b200.synthetic import make_wkv6_device_inputs, make_wkv7_device_inputs
from jaxrwkv_b200.time_mixing import time_mixing_seq

N = 64                                                   # head size, fixed by the model family
LORA = {"w": 64, "a": 64, "v": 32, "g": 128}             # inner widths of a layer's low-rank projections
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
STREAMS7 = ("r", "w", "k", "v", "a", "b")


def listed():
    return [
        # a small fp32 evaluation (benchmark configuration 1): launches and one short chain per head
        {"name": "v7-eval-fp32-small", "op": "wkv7-fwd", "dtype": "fp32", "B": 2, "T": 256, "H": 4, "starts": 0.0, "ragged": False},
        # scoring packed documents with a 0.1B model (configuration 2): start flags and ragged lengths
        {"name": "v7-score-packed-0.1B", "op": "wkv7-fwd", "dtype": "bf16", "B": 8, "T": 1024, "H": 12, "starts": 1 / 256, "ragged": True},
        # prefill of one prompt of no particular length with a 2.9B model: few sequences, one long chain
        {"name": "v7-prefill-one-2.9B", "op": "wkv7-fwd", "dtype": "bf16", "B": 1, "T": 1999, "H": 40, "starts": 0.0, "ragged": False},
        # the headline training step of one layer of a 1.5B model (configuration 4's share of one GPU)
        {"name": "v7-train-1.5B", "op": "wkv7-train", "dtype": "bf16", "B": 8, "T": 4096, "H": 32, "starts": 0.0, "ragged": False},
        # training on packed documents: start flags inside the sequences, ragged lengths, a T that no tile divides
        {"name": "v7-train-packed-odd", "op": "wkv7-train", "dtype": "bf16", "B": 6, "T": 2043, "H": 32, "starts": 1 / 512, "ragged": True},
        # fp32 training of a 0.1B model on short sequences (debugging and gradient checks, small experiments)
        {"name": "v7-train-fp32-0.1B", "op": "wkv7-train", "dtype": "fp32", "B": 2, "T": 512, "H": 12, "starts": 0.0, "ragged": False},
        # decoding for one user: one token through the 32 layers of a 2.9B model; launches and host latency
        {"name": "v7-decode-1-2.9B", "op": "wkv7-decode", "dtype": "bf16", "B": 1, "H": 40, "L": 32},
        # decoding for 256 users (configuration 5): the state's traffic
        {"name": "v7-decode-256-2.9B", "op": "wkv7-decode", "dtype": "bf16", "B": 256, "H": 40, "L": 32},
        # a whole RWKV-7 time-mixing layer, forward and backward: shift, projections, elementwise stages, operator
        {"name": "v7-layer-train-1.5B", "op": "layer-train", "dtype": "bf16", "B": 4, "T": 1024, "H": 32},
        # RWKV-6 training (configuration 3)
        {"name": "v6-train", "op": "wkv6-train", "dtype": "bf16", "B": 16, "T": 4096, "H": 32, "starts": 1 / 512, "ragged": False},
        # RWKV-5.2 training, whose decay is one constant per channel
        {"name": "v5.2-train", "op": "wkv5_2-train", "dtype": "bf16", "B": 4, "T": 1024, "H": 32, "starts": 1 / 512, "ragged": False},
        # RWKV-4 training of a 0.1B model
        {"name": "v4-train-0.1B", "op": "wkv4-train", "dtype": "bf16", "B": 8, "T": 1024, "H": 12, "starts": 1 / 512, "ragged": False},
    ]


# op -> (dtypes, B, T, H range, most tokens x heads); None where the operator has no such size
RANGES = {
    "wkv7-fwd": (("bf16", "bf16", "fp32"), (1, 16), (16, 4096), (4, 12, 16, 32, 40), 1 << 19),
    "wkv7-train": (("bf16", "bf16", "bf16", "fp32"), (1, 16), (64, 4096), (4, 12, 16, 32, 40), 1 << 20),
    "wkv7-decode": (("bf16", "bf16", "fp32"), (1, 256), None, (12, 16, 32, 40), 8192),
    "layer-train": (("bf16",), (1, 8), (64, 2048), (12, 16, 32), 1 << 18),
    "wkv6-train": (("bf16",), (1, 16), (64, 4096), (12, 16, 32, 40), 1 << 20),
    "wkv5_2-train": (("bf16",), (1, 8), (64, 2048), (12, 16, 32, 40), 1 << 18),
    "wkv4-train": (("bf16", "fp32"), (1, 16), (64, 4096), (12, 16, 32, 40), 1 << 19),
}
# the operators by how often the listed cases have them
OPS = ("wkv7-fwd",) * 3 + ("wkv7-train",) * 3 + ("wkv7-decode",) * 2 + ("layer-train", "wkv6-train", "wkv5_2-train", "wkv4-train")


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(OPS)
    dtypes, bs, ts, hs, most = RANGES[op]
    case = {"op": op, "dtype": rng.choice(dtypes), "B": _log(rng, *bs), "H": rng.choice(hs)}
    if op == "wkv7-decode":
        case["L"] = rng.randint(12, 32)
        if case["dtype"] == "fp32":
            most //= 2
        case["B"] = max(1, min(case["B"], most * 40 // (case["H"] * case["L"])))
        return case
    if case["dtype"] == "fp32":
        most = most // 8            # fp32 is for short runs
    t = _log(rng, *ts)
    t = max(ts[0], min(t, most // (case["B"] * case["H"])))
    if rng.random() < 0.5:          # half of the lengths are whole tiles, as batches are often cut; half are as they come
        t = max(64, t - t % 64) if t >= 64 else t
    case["T"] = t
    if op != "layer-train":
        case["starts"] = rng.choice((0.0, 1 / 512, 1 / 256))
        case["ragged"] = rng.random() < 0.4
    return case


def _flags(g, case, dev):
    B, T = case["B"], case["T"]
    ns = (torch.rand(B, T, generator=g, device=dev) < case["starts"]).to(torch.uint8)
    length = torch.full((B,), T, dtype=torch.int32, device=dev)
    if case["ragged"]:
        length = torch.randint(T // 2, T + 1, (B,), generator=g, device=dev, dtype=torch.int32)
    return ns, length


def _layer_parameters(g, C, H, dtype, dev):
    """One layer's parameters under the reference's names: matrices ~ N(0, 1/fan_in), mixes in (0, 1)."""
    def rn(*s, scale=1.0, shift=0.0):
        return (scale * torch.randn(*s, generator=g, device=dev) + shift).to(dtype).requires_grad_(True)

    p = {"x_" + c: torch.rand(1, 1, C, generator=g, device=dev).to(dtype).requires_grad_(True) for c in "rwkvag"}
    for name in ("receptance", "key", "value", "output"):
        p[name] = {"weight": rn(C, C, scale=C ** -0.5)}
    for name, inner in LORA.items():
        p[name + "1"] = rn(C, inner, scale=C ** -0.5)
        p[name + "2"] = rn(inner, C, scale=inner ** -0.5)
    for name in ("w0", "a0", "v0"):
        p[name] = rn(1, 1, C, scale=0.5)
    p["k_k"] = rn(1, 1, C, scale=0.1, shift=0.85)
    p["k_a"] = rn(1, 1, C, scale=0.1, shift=1.0)
    p["r_k"] = rn(H, N, scale=0.1)
    p["ln_x"] = {"weight": rn(C, scale=0.1, shift=1.0), "bias": rn(C, scale=0.1)}
    return p


def _tensors(p):
    for name in sorted(p):
        if isinstance(p[name], dict):
            yield from _tensors(p[name])
        else:
            yield p[name]


def prepare(case, seed):
    dev = torch.device("cuda")
    dtype, op, B, H = DTYPES[case["dtype"]], case["op"], case["B"], case["H"]
    g = torch.Generator(device=dev).manual_seed(seed)

    def rn(*s):
        return torch.randn(*s, generator=g, device=dev)

    st = {"case": case}
    if op in ("wkv7-fwd", "wkv7-train"):
        train = op == "wkv7-train"
        x = make_wkv7_device_inputs(B, case["T"], H, N, dtype, dev, seed, p_start=case["starts"], random_length=case["ragged"],
                                    s0_scale=0.1 if train else 0.0, grads=train)
        st.update(x, leaves=[x[n].requires_grad_(train) for n in STREAMS7 + ("s0",)])
    elif op == "wkv7-decode":
        L = case["L"]
        st["state"] = torch.empty(B, L, 2 + N, H * N, dtype=dtype, device=dev)
        for layer in range(L):                       # the states that a prefill left
            st["state"][:, layer] = (0.5 * rn(B, 2 + N, H * N)).to(dtype)
        x = make_wkv7_device_inputs(B, L, H, N, dtype, dev, seed + 1, grads=False)
        st["layers"] = [[x[n][:, layer:layer + 1].contiguous() for n in STREAMS7] for layer in range(L)]
    elif op == "layer-train":
        T, C = case["T"], H * N
        p = st["att"] = _layer_parameters(g, C, H, dtype, dev)
        x, v_first = (rn(B, T, C).to(dtype).requires_grad_(True) for _ in range(2))
        state = (0.1 * rn(B, 1 + N, C)).to(dtype).requires_grad_(True)
        st.update(x=x, v_first=v_first, state=state, leaves=[x, v_first, state] + list(_tensors(p)))
        st["new_starts"], st["length"] = _flags(g, {**case, "starts": 0.0, "ragged": False}, dev)
        st.update(dy=rn(B, T, C).to(dtype), ds=rn(B, 1 + N, C).to(dtype))
    elif op == "wkv6-train":
        x = make_wkv6_device_inputs(B, case["T"], H, N, dtype, dev, seed, p_start=case["starts"])
        st.update(x, leaves=[x[n].requires_grad_(True) for n in ("r", "k", "v", "w", "u", "s0")])
        if case["ragged"]:
            st["length"] = _flags(g, case, dev)[1]
    elif op == "wkv5_2-train":
        shp = (B, case["T"], H, N)
        x = [rn(*shp).to(dtype) for _ in range(3)]
        x += [torch.exp(-torch.exp(-0.5 + 0.5 * rn(H, N, 1))).to(dtype), (0.1 * rn(H, N, 1)).to(dtype), (0.1 * rn(B, H, N, N)).to(dtype)]
        st["leaves"] = [t.requires_grad_(True) for t in x]
        st["new_starts"], st["length"] = _flags(g, case, dev)
        st.update(dy=rn(*shp).to(dtype), ds=rn(B, H, N, N).to(dtype))
    else:
        T, C = case["T"], H * N
        s0 = torch.zeros(B, 3, C, device=dev)
        s0[:, :2] = rn(B, 2, C).abs() + 0.5           # the triple that an earlier segment left
        s0[:, 2] = rn(B, C)
        x = [torch.sigmoid(rn(B, T, C)), rn(B, T, C), rn(B, T, C), -1.0 + 0.5 * rn(C), 0.5 * rn(C), s0]
        st["leaves"] = [t.to(dtype).requires_grad_(True) for t in x]
        st["new_starts"], st["length"] = _flags(g, case, dev)
        st.update(dy=rn(B, T, C).to(dtype), ds=rn(B, 3, C).to(dtype))
    return st


SEAM = {"wkv7-train": rwkv7.CudaRWKV, "wkv6-train": rwkv6.CudaRWKV, "wkv5_2-train": rwkv5_2.CudaRWKV, "wkv4-train": rwkv4.CudaRWKV}


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "wkv7-fwd":
        with torch.no_grad():
            s, y = rwkv7.CudaRWKV.inner_loop(*st["leaves"], st["length"], st["new_starts"])
        return {"y": y, "s": s}
    if op == "wkv7-decode":
        with torch.no_grad():
            ys = [rwkv7.wkv7_step_packed(*streams, st["state"], layer) for layer, streams in enumerate(st["layers"])]
        return {"y": ys, "state": st["state"]}
    if op == "layer-train":
        y, s, _ = time_mixing_seq(st["x"], st["state"], st["v_first"], st["att"], st["length"], st["new_starts"], case["H"], N, 1)
    else:
        s, y = SEAM[op].inner_loop(*st["leaves"], st["length"], st["new_starts"])
    grads = torch.autograd.grad((y, s), st["leaves"], (st["dy"], st["ds"]))
    return {"y": y, "s": s, "grads": grads}


def work(case):
    """Bytes: each input and each output once.  Flops: the token recurrence itself (per token and head, in units
    of N^2: version 7 forward 9 and backward 19, versions 5 and 6 forward 5 and backward 11)."""
    op, B, H = case["op"], case["B"], case["H"]
    e = 2 if case["dtype"] == "bf16" else 4
    state = B * H * N * N * e
    if op == "wkv7-decode":
        return {"bytes": case["L"] * (2 * state + 7 * B * H * N * e), "flops": case["L"] * B * H * 9 * N * N}
    tokens = B * case["T"]
    stream, flags = tokens * H * N * e, tokens + 4 * B
    token_flops = tokens * H * N * N
    if op == "wkv7-fwd":
        return {"bytes": 7 * stream + 2 * state + flags, "flops": 9 * token_flops}
    if op == "wkv7-train":
        return {"bytes": 14 * stream + 4 * state + flags, "flops": 28 * token_flops}
    if op == "wkv6-train":
        return {"bytes": 10 * stream + 4 * state + flags, "flops": 16 * token_flops}
    if op == "wkv5_2-train":
        return {"bytes": 8 * stream + 4 * state + flags, "flops": 16 * token_flops}
    if op == "wkv4-train":
        return {"bytes": 8 * stream + 4 * B * 3 * H * N * e + flags, "flops": 40 * tokens * H * N}
    C, inner = H * N, sum(LORA.values())
    weights = 4 * C * C + 2 * C * inner + 15 * C
    return {"bytes": 6 * stream + 4 * state + 2 * weights * e, "flops": 6 * tokens * (4 * C * C + 2 * C * inner) + 28 * token_flops}


def tolerance(case):
    # bf16: operands and results are rounded to 8 bits and the gradients of the decay are differences of such
    # products (2e-2 is the operators' stated bf16 tolerance); fp32: sums of 64 products along chains of tokens
    if case["dtype"] == "fp32":
        return {"rel": 3e-5}
    # decoding rounds the state once; RWKV-4 and 5.2 training compute in fp32 and round the results
    return {"rel": 1e-2 if case["op"] in ("wkv7-decode", "wkv4-train", "wkv5_2-train") else 2e-2}
