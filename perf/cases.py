"""Performance cases of the codec: what a program that stores integer columns on a GPU
has the library do, through the Python entry points (`leco_b200`), at the sizes of the
repository's own configurations and at ragged ones.

Operations (`op`):
  encode         one column of device values -> block images, offsets, directory
  decode         one encoded column -> its values
  lookup         a batch of uniform random lookups into one encoded column
  filter         indices of the values above a threshold, computed on the encoded column
  varlen_store   variable-length segments: partition the column, encode the segments
  varlen_load    bulk decode of a variable-length column
  batch          many columns of mixed type, codec and length: one encode + decode pass

Values come from the seed alone.  u64 columns are sorted piecewise-linear keys (timestamps,
offsets, surrogate keys), u32 columns the same with small slopes, so that they stay below
2^32; the variable-length columns switch between linear, quadratic and flat regimes.
"""
import math

import numpy as np
import torch

import leco_b200 as lc
from leco_b200 import autotune, workloads

CODECS = {"leco": lc.LINEAR, "for": lc.FOR, "delta": lc.DELTA, "poly2": lc.POLY2}
COARSE = 2000        # values per coarse block of the variable-length partitioner
MERGE_BITS = 12      # its merge penalty
LARGEST = 200_000_000


def listed():
    return [
        # bulk scan of a large key column: the decode side of the default benchmark
        {"name": "decode_leco_u64_200m", "op": "decode", "codec": "leco", "bits": 64, "n": 200_000_000, "block": 4096},
        # loading a large key column with the reference's own fit (its streams interchange)
        {"name": "encode_leco_u64_100m", "op": "encode", "codec": "leco", "bits": 64, "n": 100_000_000, "block": 4096,
         "fit": "reference"},
        # the configuration the reference's drivers run: a million sorted u32 keys, blocks of 1000
        {"name": "encode_leco_u32_1m", "op": "encode", "codec": "leco", "bits": 32, "n": 1_000_000, "block": 1000,
         "fit": "reference"},
        # an append of one full block: the smallest write, all latency
        {"name": "encode_leco_u64_block", "op": "encode", "codec": "leco", "bits": 64, "n": 4096, "block": 4096,
         "fit": "reference"},
        # frame of reference on u32 values, a ragged length: dictionary codes, row ids
        {"name": "encode_for_u32_30m", "op": "encode", "codec": "for", "bits": 32, "n": 30_000_019, "block": 4096,
         "fit": "reference"},
        # differences of sorted keys, an odd length in mid-size blocks: posting lists, event times
        {"name": "encode_delta_u64_20m", "op": "encode", "codec": "delta", "bits": 64, "n": 20_000_003, "block": 2048,
         "fit": "reference"},
        {"name": "decode_delta_u64_60m", "op": "decode", "codec": "delta", "bits": 64, "n": 60_000_001, "block": 4096},
        # point reads: an index join's probe side against a column in device memory
        {"name": "lookup_leco_u64_16m", "op": "lookup", "codec": "leco", "bits": 64, "n": 100_000_000, "block": 4096,
         "lookups": 1 << 24},
        # predicate pushdown at half selectivity
        {"name": "filter_leco_u64_100m", "op": "filter", "codec": "leco", "bits": 64, "n": 100_000_000, "block": 4096,
         "keep": 0.5},
        # variable-length columns: written once, read often
        {"name": "varlen_store_10m", "op": "varlen_store", "n": 10_000_000},
        {"name": "varlen_load_50m", "op": "varlen_load", "n": 50_000_000},
        # a table of mixed columns written and read back, with the tuned launch parameters
        {"name": "batch_20_columns", "op": "batch", "columns": 20, "shortest": 64_000, "longest": 4_000_000},
    ]


def _size(rng, lo, hi):
    """Log-uniform, as often a multiple of a round number as not."""
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return n if rng.random() < 0.5 or n < 2000 else n // 1000 * 1000


def draw(rng):
    op = rng.choice(["encode", "encode", "encode", "decode", "decode", "lookup", "filter", "varlen_store", "varlen_load",
                     "batch"])
    if op == "varlen_store":
        return {"op": op, "n": _size(rng, 200_000, 10_000_000)}
    if op == "varlen_load":
        return {"op": op, "n": _size(rng, 200_000, 60_000_000)}
    if op == "batch":
        c = rng.randint(4, 20)
        return {"op": op, "columns": c, "shortest": 1_000 * rng.randint(1, 64), "longest": 500_000 * rng.randint(1, 8)}
    c = {"op": op, "codec": rng.choice(["leco", "leco", "for", "delta", "poly2"]), "bits": rng.choice([32, 64]),
         "block": rng.choice([1000, 1024, 2048, 4096, 4096, 8192])}
    c["n"] = _size(rng, 4_096, 60_000_000 if c["bits"] == 64 else 100_000_000)
    if op == "encode":
        c["fit"] = rng.choice(["reference", "reference", "exact"])
    elif op == "lookup":
        if c["codec"] == "delta":  # a Delta lookup walks its block: few of them
            c["lookups"] = _size(rng, 1_000, 1 << 18)
        else:
            c["lookups"] = _size(rng, 1_000, 1 << 24)
    elif op == "filter":
        c["codec"] = rng.choice(["leco", "for"])  # the two codecs of the reference that have it
        c["keep"] = rng.choice([0.01, 0.1, 0.5, 0.9])
    return c


def _values(n, bits, seed):
    """A sorted column on the GPU, as int64 or int32 holding the unsigned patterns."""
    if bits == 64:
        return workloads.piecewise_linear_u64(n, seed=seed, device="cuda", noise_on="device")
    # slopes up to 2^4 (mean about 5.4): 100M values stay below 2^32
    x = workloads.piecewise_linear_u64(n, seed=seed, device="cuda", mean_seg=20_000.0, max_slope_log2=4.0, sigma=64.0,
                                       noise_on="device")
    return x.to(torch.int32)  # keeps the low 32 bits


def _encode(values, codec, block, fit="reference"):
    mode = lc.FIT_REFERENCE if fit == "reference" else lc.FIT_EXACT
    return lc.encode(values, CODECS[codec], block, mode)


def _batch_lengths(case):
    """The batch's column lengths, codecs, widths and families: part of the case, not of the seed."""
    rng = np.random.default_rng(case["columns"])
    lo, hi = math.log(case["shortest"]), math.log(case["longest"])
    cols = []
    for k in range(case["columns"]):
        n = int(math.exp(rng.uniform(lo, hi)))
        cols.append((n, 4 if rng.random() < 0.5 else 8, workloads.BATCH_FAMILIES[int(rng.integers(4))],
                     (lc.LINEAR, lc.DELTA, lc.FOR)[int(rng.integers(3))]))
    return cols


def prepare(case, seed):
    op = case["op"]
    if op == "encode":
        v = _values(case["n"], case["bits"], seed)
        L, s = lc.lib(), case["bits"] // 8
        codec = CODECS[case["codec"]]
        mode = lc.FIT_REFERENCE if case["fit"] == "reference" else lc.FIT_EXACT
        cap = L.leco_max_payload_bytes(codec, s, case["n"], case["block"])
        wsb = L.leco_encode_workspace_bytes(codec, s, case["n"], case["block"], mode)
        return dict(op=op, values=v, codec=codec, block=case["block"], mode=mode,
                    payload=torch.zeros(cap, dtype=torch.uint8, device="cuda"),
                    workspace=torch.empty(max(wsb, 1), dtype=torch.uint8, device="cuda"))
    if op in ("decode", "lookup", "filter"):
        v = _values(case["n"], case["bits"], seed)
        col = _encode(v, case["codec"], case["block"]).compact()
        s = dict(op=op, col=col)
        if op == "decode":
            s["out"] = torch.empty_like(v)
        elif op == "lookup":
            g = torch.Generator(device="cuda").manual_seed(seed + 7)
            s["idx"] = torch.randint(0, case["n"], (case["lookups"],), generator=g, device="cuda", dtype=torch.int64)
            s["out"] = torch.empty(case["lookups"], dtype=v.dtype, device="cuda")
        else:
            # the threshold lies somewhere near the selectivity asked for
            near = float(np.random.default_rng(seed).uniform(0.98, 1.02))
            at = min(case["n"] - 1, int(case["n"] * (1.0 - case["keep"] * near)))
            s["above"] = int(v[at].item()) & ((1 << case["bits"]) - 1)
            s["zmin"], s["zmax"] = col.zonemap()
            s["out"] = torch.zeros(case["n"] + col.nblocks, dtype=torch.int32, device="cuda")
            s["ws"] = torch.empty(int(lc.lib().leco_filter_workspace_bytes(case["n"], case["block"])), dtype=torch.uint8,
                                  device="cuda")
        return s
    if op in ("varlen_store", "varlen_load"):
        n = case["n"]
        v = workloads.regime_switching_u64(n, seed=seed, device="cuda")
        ws = torch.empty(int(lc.lib().leco_varlen_partition_workspace_bytes(n, n // COARSE)), dtype=torch.uint8, device="cuda")
        if op == "varlen_store":
            return dict(op=op, values=v, coarse=n // COARSE, ws=ws, arena=_arena(n))
        starts = lc.varlen_partition_device(v, n // COARSE, MERGE_BITS, ws=ws)
        col = lc.varlen_encode(v, starts, max_segment_len=_longest(n))
        col.payload = col.payload[: col.nbytes + lc.PAYLOAD_SLACK].clone()
        return dict(op=op, col=col, out=torch.empty_like(v))
    cols = []
    for k, (n, s, family, codec) in enumerate(_batch_lengths(case)):
        x = workloads.families(n, family, s, np.random.default_rng([seed, k]))
        block, group, unroll = autotune.pick(codec, s, n, family)
        cols.append((torch.from_numpy(x.view(np.int32 if s == 4 else np.int64)).cuda(), codec, block, group, unroll))
    b = lc.Batch(cols)
    for c in b.cols:
        c.payload.zero_()
    return dict(op=op, batch=b)


def _arena(n):
    """Where the program keeps stored columns: segment starts, offsets, payload."""
    return (torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n + 1, dtype=torch.int64, device="cuda"),
            torch.zeros(8 * n, dtype=torch.uint8, device="cuda"))


def _longest(n):
    """No segment is longer than a coarse block."""
    return n // (n // COARSE)


def run(state):
    op = state["op"]
    if op == "encode":
        c = lc.encode(state["values"], state["codec"], state["block"], state["mode"], payload=state["payload"],
                      workspace=state["workspace"])
        return [c.payload, c.offsets, c.dir]
    if op == "decode":
        return state["col"].decode(out=state["out"])
    if op == "lookup":
        return state["col"].gather(state["idx"], out=state["out"])
    if op == "filter":
        # the next operator reads the indices and their count on the device
        idx, count = state["col"].filter_range(state["above"], zone_min=state["zmin"], zone_max=state["zmax"],
                                               out=state["out"], ws=state["ws"], sync=False)
        return [idx, count]
    if op == "varlen_store":
        v = state["values"]
        starts = lc.varlen_partition_device(v, state["coarse"], MERGE_BITS, ws=state["ws"])
        col = lc.varlen_encode(v, starts, max_segment_len=_longest(v.numel()))
        kept = [starts, col.offsets, col.payload[: col.nbytes]]
        for place, t in zip(state["arena"], kept):
            place[: t.numel()].copy_(t)
        return list(state["arena"])
    if op == "varlen_load":
        return state["col"].decode(out=state["out"])
    b = state["batch"]
    b.run_graph(3)
    return [t for c in b.cols for t in (c.payload, c.offsets, c.out)]


# Encoded size over raw size, to estimate a column's compressed bytes (the sizes differ by a few
# per cent between seeds, and the decode side's writes or the encode side's reads are the larger part).
RATIO = {("leco", 64): 0.22, ("for", 64): 0.36, ("delta", 64): 0.22, ("poly2", 64): 0.22,
         ("leco", 32): 0.30, ("for", 32): 0.47, ("delta", 32): 0.28, ("poly2", 32): 0.30}
SEGMENTED = 0.18


def work(case):
    op = case["op"]
    flops = 0
    if op in ("varlen_store", "varlen_load"):
        b = 8 * case["n"] * (1 + SEGMENTED)
        flops = 6 * case["n"]  # sums of the fit, prediction
    elif op == "batch":
        raw = sum(n * s for n, s, _, _ in _batch_lengths(case))
        b = 2 * raw * (1 + 0.28)
        flops = 6 * sum(n for n, _, _, _ in _batch_lengths(case))
    else:
        s = case["bits"] // 8
        packed = case["n"] * s * RATIO[(case["codec"], case["bits"])]
        if op == "lookup":
            # index in, value out, and one 32-byte sector of the payload (a dense batch reads it once)
            b = case["lookups"] * (8 + s) + min(packed, 32 * case["lookups"])
        elif op == "filter":
            # the blocks' headers, offsets and zone map; four bytes for each index
            b = case["n"] // case["block"] * 48 + 4 * case["n"] * case["keep"]
        else:
            b = case["n"] * s + packed
            flops = 2 * case["n"] if case["codec"] in ("leco", "poly2") else 0
            if op == "encode":
                flops *= 3
    return {"bytes": float(b), "flops": float(flops)}


def exact(case, seed):
    """Every output is a whole number or a byte: there is no rounding to measure."""
    return None
