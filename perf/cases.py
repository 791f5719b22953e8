"""The calls whose speed matters to a user of this package, at the sizes they come in.

Each case is one pass through the public entry points: the state of a training rank is compressed, restored, written
to file images, read back, streamed from host memory, analysed, or handed to the Re-Pair estimator.  The values have
the distributions that such state has (weights ~ N(0, 0.02), first moments ~ N(0, 1e-4), second moments lognormal),
so the tables and the compressed sizes are those of real checkpoints.
"""
import math

import numpy as np
import torch

import checkers_b200 as chk
from checkers_b200.repair import apply_grammar, build_grammar
from checkers_b200.streaming import ChunkedHostPipeline, HostTensor

MI = 1 << 20

# What a rank holds per parameter: (prefix of the registered name, torch dtype, dtype tag, distribution).
MIXES = {
    # bf16 weight with fp32 master copy and both Adam moments: 14 bytes per parameter
    "adam": (("", torch.bfloat16, chk.BF16, "weight"), ("master_weights::", torch.float32, chk.F32, "weight"),
             ("optimizer.exp_avg::", torch.float32, chk.F32, "first"),
             ("optimizer.exp_avg_sq::", torch.float32, chk.F32, "second")),
    # the same without master copies: 10 bytes per parameter
    "adam_no_master": (("", torch.bfloat16, chk.BF16, "weight"),
                       ("optimizer.exp_avg::", torch.float32, chk.F32, "first"),
                       ("optimizer.exp_avg_sq::", torch.float32, chk.F32, "second")),
    "fp32": (("", torch.float32, chk.F32, "small"),),
    "bf16": (("", torch.bfloat16, chk.BF16, "weight"),),
    "fp16": (("", torch.float16, chk.F16, "weight"),),
    # 8-bit (quantised) weights and 32-bit counters: no low bytes to split off, every byte goes through the coder
    "int8": (("", torch.int8, chk.I8, "int8"),),
    "int32": (("", torch.int32, chk.I32, "int32"),),
}
# Compressed bytes per byte of such state (low bytes included), for the traffic that a pass cannot do without.
CODED = {"adam": 0.98, "adam_no_master": 0.97, "fp32": 1.0, "bf16": 0.9, "fp16": 0.93, "int8": 0.8, "int32": 0.5}
CODED_V3 = 0.81
FLOATS = (chk.F32, chk.BF16, chk.F16)


def listed():
    return [
        # The smallest call: one tensor encoded in fixed memory, inside a training step where nothing may be allocated.
        {"name": "encode one tensor", "kind": "static", "mix": "bf16", "n": 256 << 10},
        # The trainable part of an adapter: a few dozen small, odd tensors; launches and host work count.
        {"name": "roundtrip adapter", "kind": "roundtrip", "mix": "adam", "layout": "flat", "n": 40_011, "chunk": 4096,
         "version": 2},
        # The 16 Mi element shard in 64 tensors per state: a batch smaller than what the device can hold at once.
        {"name": "roundtrip 192 tensors", "kind": "roundtrip", "mix": "adam_no_master", "layout": "flat", "n": 16 * MI,
         "chunk": 256 << 10, "version": 2},
        # A rank's slice of a large model in 1 Mi element tensors, resident on the device: the largest.
        {"name": "roundtrip shard", "kind": "roundtrip", "mix": "adam", "layout": "flat", "n": 256 * MI, "chunk": MI,
         "version": 2},
        # A whole small model as its module and optimizer name it: uncut parameters from norm gains to an embedding,
        # and the integer tensors that come with it.
        {"name": "roundtrip whole model", "kind": "roundtrip", "mix": "adam_no_master", "layout": "model",
         "hidden": 1024, "layers": 6, "inter": 2816, "vocab": 32000, "version": 2},
        # The smaller container (a table per byte plane).
        {"name": "roundtrip version 3", "kind": "roundtrip", "mix": "adam", "layout": "flat", "n": 48 * MI, "chunk": MI,
         "version": 3},
        # Restore alone, the codec benchmark's tensor: fp32 in 4 MiB chunks.
        {"name": "restore fp32 chunks", "kind": "restore", "mix": "fp32", "layout": "flat", "n": 128 * MI, "chunk": MI,
         "version": 2},
        # Device state to the three file images in host memory.
        {"name": "compress to images", "kind": "save", "mix": "adam", "layout": "flat", "n": 32 * MI, "chunk": MI,
         "shared": False},
        # File images back to the device; odd sizes, so nothing but the first tensor is aligned.
        {"name": "restore from images", "kind": "load", "mix": "adam", "layout": "flat", "n": 32 * MI + 12_345,
         "chunk": 1_000_003},
        # State that lives in host memory, streamed through the device in parts, both directions.
        {"name": "host stream", "kind": "stream", "mix": "adam", "n": 64 * MI, "chunk": MI, "part": 128 * MI,
         "version": 2},
        # Statistics of every tensor and the clusters formed from them.
        {"name": "analyze", "kind": "analyze", "mix": "adam", "layout": "flat", "n": 128 * MI, "chunk": 4 * MI},
        # The Re-Pair estimator on one group: a grammar from its representative, applied to the two other members.
        {"name": "repair group", "kind": "repair", "mix": "fp32", "n": MI, "members": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "roundtrip", "roundtrip", "roundtrip", "restore", "save", "load", "stream", "analyze",
                       "repair"])
    if kind == "static":
        mix = rng.choice(["bf16", "fp32", "fp16", "int8"])
        return {"kind": kind, "mix": mix, "n": _log(rng, 4096, chk.STATIC_MAX_TENSOR_BYTES // _row_bytes(mix))}
    if kind == "repair":
        return {"kind": kind, "mix": rng.choice(["fp32", "bf16"]), "n": _log(rng, 1 << 16, 1 << 22), "members": 3}
    if kind == "stream":
        return {"kind": kind, "mix": rng.choice(["adam", "bf16", "fp32"]), "n": _log(rng, 4 * MI, 64 * MI),
                "chunk": _log(rng, 100_000, 2 * MI), "part": _log(rng, 32 * MI, 256 * MI), "version": rng.choice([2, 2, 3])}
    if kind == "roundtrip" and rng.random() < 0.25:
        hidden = 64 * rng.randint(2, 20)
        return {"kind": kind, "mix": rng.choice(["adam", "adam_no_master", "bf16"]), "layout": "model", "hidden": hidden,
                "layers": rng.randint(1, 8), "inter": 3 * hidden - 64 * rng.randint(0, 2), "vocab": _log(rng, 2000, 32000),
                "version": 2}
    mix = rng.choice(["adam", "adam", "adam_no_master", "fp32", "bf16", "fp16", "int8", "int32"])
    most = 192 * MI if kind in ("roundtrip", "restore") else 64 * MI
    # between a handful and about a thousand tensors per state, none so long that one of them is the whole time
    n = _log(rng, 20_000, most)
    chunk = min(n, max(1000, n // 1500, _log(rng, 4000, 4 * MI)))
    if rng.random() < 0.4:  # tensors of a round size as often as not
        chunk = 1 << max(10, chunk.bit_length() - 1)
        n = max(chunk, n // chunk * chunk)
    c = {"kind": kind, "mix": mix, "layout": "flat", "n": n, "chunk": chunk}
    if kind in ("roundtrip", "restore"):
        c["version"] = rng.choice([2, 2, 2, 3])
    if kind == "save":
        c["shared"] = rng.random() < 0.4
    return c


def _row_bytes(mix):
    return sum(torch.empty(0, dtype=dt).element_size() for _, dt, _, _ in MIXES[mix])


def _pieces(case):
    """(name, offset, elements, is a norm gain) of every tensor of one state, and the length of the flat buffer."""
    out = []
    if case.get("layout") == "model":
        h, i = case["hidden"], case["inter"]
        params = [("embed.weight", case["vocab"] * h, False)]
        for layer in range(case["layers"]):
            p = f"layers.{layer}."
            params += [(p + "q.weight", h * h, False), (p + "k.weight", h * h // 4, False), (p + "v.weight", h * h // 4, False),
                       (p + "o.weight", h * h, False), (p + "gate.weight", i * h, False), (p + "up.weight", i * h, False),
                       (p + "down.weight", i * h, False), (p + "norm1.weight", h, True), (p + "norm2.weight", h, True)]
        params.append(("norm.weight", h, True))
        at = 0
        for name, n, norm in params:  # tensors of their own, each aligned as an allocator aligns it
            out.append((name, at, n, norm))
            at += (n + 255) // 256 * 256
        return out, at
    n, chunk = case["n"], case["chunk"]
    for at in range(0, n, chunk):  # slices of flat buffers, as a sharded optimizer keeps them
        out.append((f"w@{at}", at, min(chunk, n - at), False))
    return out, n


def _values(dist, dtype, n, pieces, g):
    dev = g.device
    if dist == "int8":
        return torch.empty(n, device=dev).normal_(0.0, 20.0, generator=g).clamp_(-127, 127).to(torch.int8)
    if dist == "int32":
        return torch.randint(0, 50_000, (n,), generator=g, device=dev, dtype=torch.int32)
    x = torch.empty(n, dtype=torch.float32, device=dev)
    if dist == "second":
        return x.normal_(-18.0, 2.0, generator=g).exp_()
    x.normal_(0.0, {"weight": 0.02, "first": 1e-4, "small": 1e-3}[dist], generator=g)
    if dist == "weight":
        for _, at, k, norm in pieces:
            if norm:
                x[at:at + k].normal_(1.0, 1e-3, generator=g)
    return x.to(dtype)


def _buffers(case, seed):
    """One flat buffer per state, and (name, state, offset, elements, dtype tag) of every tensor in registration order."""
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    pieces, total = _pieces(case)
    bufs, tensors = [], []
    for _, dtype, _, dist in MIXES[case["mix"]]:
        bufs.append(_values(dist, dtype, total, pieces, g))
    for name, at, n, _ in pieces:
        for k, (prefix, _, tag, _) in enumerate(MIXES[case["mix"]]):
            tensors.append((prefix + name, k, at, n, tag))
    if case.get("layout") == "model":  # counters and a mask that a module keeps beside its parameters
        bufs.append(torch.randint(0, case["vocab"], (4096,), generator=g, device=dev, dtype=torch.int32))
        tensors.append(("positions", len(bufs) - 1, 0, 4096, chk.I32))
        bufs.append(torch.randint(0, 2, (65536,), generator=g, device=dev, dtype=torch.int32).to(torch.int8))
        tensors.append(("mask", len(bufs) - 1, 0, 65536, chk.I8))
    return bufs, tensors


def _pointer(bufs, t):
    return bufs[t[1]].data_ptr() + t[2] * bufs[t[1]].element_size()


def _context(bufs, tensors, version=2):
    ctx = chk.Context(device=torch.cuda.current_device())
    if version != 2:
        ctx.set_option("format_version", version)
    for t in tensors:
        ctx.register_pointer(t[0], _pointer(bufs, t), t[3], t[4])
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    if kind == "static":
        case = dict(case, layout="flat", chunk=case["n"])
        bufs, tensors = _buffers(case, seed)
        n_bytes = bufs[0].numel() * bufs[0].element_size()
        counter = chk.Context(device=torch.cuda.current_device())
        if tensors[0][4] in FLOATS:  # the table counts what the coder sees: the low bytes zeroed
            masked = torch.empty(n_bytes, dtype=torch.uint8, device="cuda")
            low = torch.empty(n_bytes // 2, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            counter.split(bufs[0].data_ptr(), case["n"], tensors[0][4], masked.data_ptr(), low.data_ptr())
        else:
            masked = bufs[0].view(torch.uint8)
            torch.cuda.synchronize()
        hist = counter.byte_histogram(masked.data_ptr(), n_bytes)
        freq, cum, _, _ = chk.normalize_histogram(hist)
        return {"kind": kind, "src": bufs[0], "n": case["n"], "tag": tensors[0][4], "freq": freq, "cum": cum,
                "payload": torch.zeros(n_bytes + 64, dtype=torch.uint8, device="cuda"),
                "headers": torch.zeros(256 * 16, dtype=torch.uint8, device="cuda"),
                "stream": torch.cuda.current_stream().cuda_stream}
    if kind == "repair":
        bufs, _ = _buffers(dict(case, layout="flat", n=case["n"] * case["members"], chunk=case["n"]), seed)
        raw = bufs[0].view(torch.uint8).cpu().numpy().reshape(case["members"], -1)
        size, mantissa = (4, 23) if case["mix"] == "fp32" else (2, 7)
        return {"kind": kind, "raw": [np.ascontiguousarray(r) for r in raw], "size": size, "masked": mantissa}
    if kind == "stream":
        bufs, tensors = _buffers(dict(case, layout="flat"), seed)
        host = [torch.empty(b.numel(), dtype=b.dtype, pin_memory=True) for b in bufs]
        back = [torch.empty(b.numel(), dtype=b.dtype, pin_memory=True) for b in bufs]
        for h, b in zip(host, bufs):
            h.copy_(b)
        pipe = ChunkedHostPipeline([HostTensor(t[0], host[t[1]][t[2]:t[2] + t[3]], t[4]) for t in tensors],
                                   device=torch.cuda.current_device(), chunk_bytes=case["part"], workers=3,
                                   options={"format_version": case["version"]})
        return {"kind": kind, "pipe": pipe, "host": host, "back": back,
                "targets": [back[t[1]][t[2]:t[2] + t[3]] for t in tensors]}
    bufs, tensors = _buffers(case, seed)
    torch.cuda.synchronize()
    state = {"kind": kind, "bufs": bufs, "ctx": None}
    if kind in ("roundtrip", "restore"):
        outs = [torch.zeros_like(b) for b in bufs]
        torch.cuda.synchronize()
        state.update(outs=outs, targets=np.asarray([_pointer(outs, t) for t in tensors], dtype=np.uint64),
                     ctx=_context(bufs, tensors, case["version"]))
        if kind == "restore":
            state["ctx"].compress()
    elif kind == "save":
        state["ctx"] = _context(bufs, tensors)
        state["shared"] = case["shared"]
        coded = sum(t[3] * bufs[t[1]].element_size() * (CODED[case["mix"]] - (0.5 if MIXES[case["mix"]][t[1]][2] in FLOATS else 0))
                    for t in tensors)
        state["end"] = int(0.75 * (4648 * len(tensors) + coded))
        if case["shared"]:  # one table per cluster of similar tensors, kept decodable
            state["ctx"].set_option("repair_tables", 1)
    elif kind == "load":
        writer = _context(bufs, tensors)
        writer.compress(host_images=True)
        images = []
        for k in range(3):
            img = writer.image(k)
            held = torch.empty(img.size, dtype=torch.uint8, pin_memory=True)
            held.numpy()[:] = img
            images.append(held)
        writer.close()
        outs = [torch.zeros_like(b) for b in bufs]
        torch.cuda.synchronize()
        state.update(bufs=None, outs=outs, images=images, ctx=_context(outs, tensors))
    elif kind == "analyze":
        state["ctx"] = _context(bufs, tensors)
        state["count"] = len(tensors)
    return state


def run(state):
    kind = state["kind"]
    if kind == "static":
        size, raw = chk.encode_tensor_static(state["src"].data_ptr(), state["n"], state["tag"], state["freq"], state["cum"],
                                             state["payload"].data_ptr(), state["headers"].data_ptr(), state["stream"])
        return {"payload": state["payload"], "headers": state["headers"], "size": size, "raw": raw}
    if kind == "repair":
        first, *others = state["raw"]
        g = build_grammar(first, state["size"], state["masked"], 50)
        tokens = [apply_grammar(r, state["size"], state["masked"], g["lhs"], g["rhs"]) for r in others]
        return {"lhs": g["lhs"].astype(np.int64), "rhs": g["rhs"].astype(np.int64), "freq": g["freq"].astype(np.int64),
                "tokens": np.asarray([g["tokens"]] + tokens, dtype=np.int64)}
    if kind == "stream":
        pipe = state["pipe"]
        pipe.compress()
        sizes = pipe.summary()
        pipe.restore(state["targets"])
        return {"restored": state["back"], "sizes": sizes}
    ctx = state["ctx"]
    if kind == "roundtrip":
        ctx.compress()
        sizes = ctx.summary()
        ctx.decompress_resident(state["targets"])
        return {"restored": state["outs"], "sizes": sizes}
    if kind == "restore":
        ctx.decompress_resident(state["targets"])
        return {"restored": state["outs"]}
    if kind == "save":
        if state["shared"]:
            ctx.analyze()
        ctx.compress(host_images=True)
        states, mantissa, tables = (torch.from_numpy(ctx.image(k)) for k in range(3))
        # The states image is as long as the values make it: two views of a fixed length, from its start and to its
        # end, are all of it.
        n = min(state["end"], states.numel())
        images = [states[:n], states[states.numel() - n:], mantissa, tables]
        for image in images:
            image.owner = ctx  # the memory is the context's: a view must not outlive it
        return images
    if kind == "load":
        ctx.decompress_images(*[i.numpy() for i in state["images"]])
        return {"restored": state["outs"]}
    ctx.analyze()
    stats = [ctx.tensor_stats(i) for i in range(state["count"])]
    ids, clusters = ctx.cluster_ids()
    return {"histograms": np.stack([s[0] for s in stats]).astype(np.int64), "moments": np.stack([s[1] for s in stats]),
            "minmax": np.stack([s[2] for s in stats]), "fingerprints": np.stack([s[3] for s in stats]), "ids": ids,
            "clusters": clusters}


def work(case):
    if case["kind"] == "repair":
        return {"bytes": case["n"] * _row_bytes(case["mix"]) * case["members"], "flops": 0}
    if case.get("layout") == "model":
        n = sum(p[2] for p in _pieces(case)[0])
    else:
        n = case["n"]
    tensor = n * _row_bytes(case["mix"])
    coded = tensor * (CODED_V3 if case.get("version") == 3 and case["mix"].startswith("adam") else CODED[case["mix"]])
    passes = {"roundtrip": 2, "stream": 2, "analyze": 0}.get(case["kind"], 1)  # directions
    return {"bytes": tensor if passes == 0 else passes * (tensor + coded), "flops": 0}


def tolerance(case):
    """Files, streams and restored tensors are the same bytes whatever computes them; the statistics are summed in a
    fixed order, so they are too."""
    return "exact"
