"""Performance cases: what a user of the prover calls, over the range it is used in.

A case names one public call (or commit + prove, the prover's step), a field, a
configuration and the matrix shapes.  Sizes are those of the 8B and 70B shape
sets, of the serving pool's single matrices, and small ragged collections.

  block_root  Parameters.block_root_noalloc of one PCS block (no allocation)
  commit      Parameters.commit of device weights
  prove       commit + prove of device weights at the benchmark claims
  open        Parameters.open on a commitment that is kept (a serving pool)
  stream      commit_recomputed + prove of page-locked host weights
  claims      Parameters.evaluate_claims at fresh points
  audit       Committed.range_audit
"""
import numpy as np
import torch

import parcomm_b200 as qf
from parcomm_b200 import layout

FIELDS = {"int8": qf.FIELD_F65521, "int16": qf.FIELD_KOALABEAR}
LAYER_8B = "4096x4096,1024x4096*2,4096x4096,14336x4096*2,4096x14336"
EMBED_8B = "128256x4096"


def _case(name, op, dtype, shapes, chunk_log, packed_log):
    case = {"op": op, "dtype": dtype, "shapes": shapes, "chunk_log": chunk_log, "packed_log": packed_log}
    return dict(case, name=name) if name else case


def listed():
    return [
        # A latency-bound loop's block commitment inside its own stream: a 64K-weight block and the largest it takes.
        _case("block_root_2e16", "block_root", "int8", "300x700", 16, 4),
        _case("block_root_2e20", "block_root", "int8", "1024x4096", 20, 4),
        # A server's opening at a fresh point: a small ragged matrix, and one 8B key projection on its own.
        _case("open_ragged_int8", "open", "int8", "300x700", 14, 4),
        _case("open_key_int8", "open", "int8", "1024x4096", 30, 4),
        # A small ragged collection of 16-bit payloads, committed and proven once (wide packing).
        _case("prove_ragged_int16", "prove", "int16", "129x65,513x1027,77x1,1000x333", 16, 6),
        # The attention projections of one 8B layer in 2^24-entry blocks.
        _case("prove_attention_int8", "prove", "int8", "4096x4096*2,1024x4096*2", 24, 4),
        # One 8B layer committed for a pool that opens it later.
        _case("commit_layer_int8", "commit", "int8", LAYER_8B, 28, 4),
        # The whole 8B set in 8 bits: the headline batch.
        _case("prove_8b_int8", "prove", "int8", "%s,(%s)*32,%s" % (EMBED_8B, LAYER_8B, EMBED_8B), 30, 4),
        # Embedding and eight layers of the 8B set in 16 bits.
        _case("prove_layers_int16", "prove", "int16", "%s,(%s)*8" % (EMBED_8B, LAYER_8B), 30, 4),
        # One 8B layer in 16 bits from page-locked host memory, in the recompute mode.
        _case("stream_layer_int16", "stream", "int16", LAYER_8B, 26, 6),
        # A statement's claims at fresh points: four 8B layers.
        _case("claims_layers_int8", "claims", "int8", "(%s)*4" % LAYER_8B, 28, 4),
        # The range audit of one layer's 16-bit payloads.
        _case("audit_layer_int16", "audit", "int16", LAYER_8B, 28, 4),
    ]


def draw(rng):
    op = rng.choice(["block_root", "commit", "prove", "prove", "open", "stream", "claims", "audit"])
    dtype = "int8" if op == "block_root" else rng.choice(["int8", "int16"])
    top = {"block_root": 22, "open": 28, "stream": 28, "audit": 30}.get(op, 31 if dtype == "int8" else 30)
    total = 2 ** rng.uniform(16, top)
    count = 1 if op == "open" and rng.random() < 0.5 else rng.randint(1, 6)
    shapes = []
    for _ in range(count):
        cols = int(2 ** rng.uniform(4, 14)) if rng.random() < 0.5 else 2 ** rng.randint(6, 14)
        shapes.append("%dx%d" % (max(1, int(total / count / cols)), cols))
    shapes = ",".join(shapes)
    logical = layout.buckets(_shapes(shapes))[2].bit_length() - 1
    low = max(12, logical - 6)
    if op == "block_root":
        chunk_log = rng.randint(max(14, low), max(20, low))
        chunk_log = min(20, chunk_log)
    elif op == "stream":
        chunk_log = rng.randint(low, max(low, logical - 1))
    else:
        chunk_log = rng.randint(low, 30)
    packed_log = rng.choice([4, 4, 6]) if logical > 26 else rng.choice([1, 4, 6])
    return _case(None, op, dtype, shapes, chunk_log, packed_log)


def _shapes(text):
    """'128256x4096,(1024x4096*2,4096x14336)*32' -> [(rows, cols), ...]"""
    out, depth, item = [], 0, ""
    for ch in text + ",":
        if ch == "," and depth == 0:
            body, times = item, 1
            if "*" in item and item.rindex("*") > item.rfind(")"):
                body, times = item[:item.rindex("*")], int(item[item.rindex("*") + 1:])
            if body.startswith("("):
                one = _shapes(body[1:-1])
            else:
                rows, cols = body.split("x")
                one = [(int(rows), int(cols))]
            out += one * times
            item = ""
        else:
            depth += (ch == "(") - (ch == ")")
            item += ch
    return out


def _weights(case, seed):
    """Synthetic weights on the GPU in the statement's layout.  8 bits: N(0, 20^2)
    rounded and clipped, every thousandth entry at +-127; 16 bits: the patterns of
    BF16 values of N(0, 0.02^2)."""
    buckets, active, _ = layout.buckets(_shapes(case["shapes"]))
    dtype = torch.int8 if case["dtype"] == "int8" else torch.int16
    out = torch.zeros(active, dtype=dtype, device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    step = 1 << 27
    for at in range(0, active, step):
        part = torch.randn(min(step, active - at), generator=g, device="cuda")
        if dtype == torch.int8:
            part.mul_(20.0).round_().clamp_(-127, 127)
            part[::1000] = part[::1000].sign().mul_(254.0).add_(127.0).clamp_(-127, 127)
        else:
            part = part.mul_(0.02).to(torch.bfloat16).view(torch.int16)
        out[at:at + part.numel()].copy_(part)
        del part
    for b in buckets:  # the padding of buckets that are wider than their matrix
        view = out[b.offset:b.offset + b.rows * b.cols].view(b.rows, b.cols)
        if b.physical_rows < b.rows:
            view[b.physical_rows:].zero_()
        if b.physical_cols < b.cols:
            view[:, b.physical_cols:].zero_()
    torch.cuda.synchronize()
    return out


def _params(case):
    return qf.Parameters(_shapes(case["shapes"]), qf.Config(case["chunk_log"], case["packed_log"]), FIELDS[case["dtype"]])


def _points(params, seed):
    """Fresh uniform points: canonical little-endian coefficients below the field's modulus."""
    rng = np.random.default_rng(seed)
    coords = sum((n - 1).bit_length() for s in params.shapes for n in (s.rows, s.cols))
    if params.field == qf.FIELD_KOALABEAR:
        return rng.integers(0, 2130706433, coords * 4, dtype=np.uint64).astype("<u4").tobytes()
    return rng.integers(0, 65521, coords * 8).astype("<u2").tobytes()


def prepare(case, seed):
    params, weights, op = _params(case), _weights(case, seed), case["op"]
    state = {"op": op, "params": params, "weights": weights}
    points = _points(params, seed)
    if op == "block_root":
        state["block"] = seed % max(1, params.active // (params.logical // params.blocks))
        state["root"] = torch.zeros(32, dtype=torch.uint8, device="cuda")
        state["stream"] = torch.cuda.current_stream().cuda_stream
    elif op in ("open", "claims", "audit"):
        state["committed"] = params.commit(weights, on_device=True)
        state["points"] = points
        if op == "open":
            state["claims"] = params.evaluate_claims(state["committed"], points)
    elif op in ("prove", "stream"):
        committed = params.commit(weights, on_device=True)
        state["claims"] = params.evaluate_claims(committed, params.benchmark_points(committed.roots))
        committed.close()
        if op == "stream":
            host = torch.empty(weights.numel(), dtype=weights.dtype, pin_memory=True)
            host.copy_(weights)
            state["weights"] = host
    return state


def _bytes(data):
    return np.frombuffer(bytes(data), dtype=np.uint8)


def run(state):
    op, params, weights = state["op"], state["params"], state["weights"]
    if op == "block_root":
        params.block_root_noalloc(weights, state["block"], state["root"], state["stream"])
        return state["root"]
    if op == "commit":
        committed = params.commit(weights, on_device=True)
        roots = _bytes(b"".join(committed.roots))
        committed.close()
        return roots
    if op in ("prove", "stream"):
        committed = params.commit(weights, on_device=True) if op == "prove" else params.commit_recomputed(weights, None)
        proof, _ = params.prove(committed, state["claims"])
        out = {"roots": _bytes(b"".join(committed.roots)), "proof": _bytes(proof.to_bytes())}
        committed.close()
        return out
    if op == "open":
        return _bytes(params.open(state["committed"], state["claims"])[0].to_bytes())
    if op == "claims":
        return _bytes(b"".join(c.value for c in params.evaluate_claims(state["committed"], state["points"])))
    audit = state["committed"].range_audit()
    return {"multiplicities": audit.multiplicities.astype(np.int64), "alpha": _bytes(audit.alpha), "lhs": _bytes(audit.lhs),
            "rhs": _bytes(audit.rhs), "holds": audit.holds}


def work(case):
    """Bytes: the weights once, and what a commitment leaves behind (codewords of
    two 16-byte elements and trees of 4 bytes per packed element) where the call
    commits.  The arithmetic is on integers: no floating-point operations."""
    _, active, logical = layout.buckets(_shapes(case["shapes"]))
    entry, lanes = (1, 8) if case["dtype"] == "int8" else (2, 4)
    block = min(logical, 1 << case["chunk_log"])
    if case["op"] == "block_root":
        return {"bytes": block * entry + 32, "flops": 0}
    n = active * entry
    if case["op"] in ("commit", "prove"):
        n += logical // lanes * 36
    if case["op"] == "audit":
        n += 8 << (8 * entry)
    return {"bytes": n, "flops": 0}


def exact(case, seed):
    """The audit's counts; proofs, roots and claims are bytes over finite fields."""
    if case["op"] != "audit":
        return None
    weights = _weights(case, seed)
    half = 128 if case["dtype"] == "int8" else 32768
    counts = sum(torch.bincount(part.to(torch.int64) + half, minlength=2 * half) for part in weights.split(1 << 26))
    return {"multiplicities": counts.cpu().numpy(), "alpha": None, "lhs": None, "rhs": None, "holds": 1}
