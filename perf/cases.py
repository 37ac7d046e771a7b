"""The work that users have this codec do, as cases to time.

A case is a dict of plain values; ``prepare`` makes what a program holds
before the call (fields, streams and buffers on the GPU), ``run`` makes one
pass through the package's public calls and returns what they wrote.  Kinds:

* ``field``: one array at a fixed rate through ``compress`` / ``decompress``
  (``dir``: compress, decompress, or both, one after the other);
* ``mode``: one array in zfp's fixed-accuracy or fixed-precision mode, through
  the same two calls; decompression has the stream alone, no block offsets;
* ``batch``: many arrays of uneven shape, type and rate through
  ``compress_batch`` and ``decompress_batch``;
* ``blocks``: a list of single blocks of a stream, read with
  ``decode_blocks`` and written with ``encode_blocks``.
"""
from __future__ import annotations

import math
import random

import torch

import cuzfp_gb300 as gz
from cuzfp_gb300 import synth

DEV = "cuda"
TYPES = {"f32": (torch.float32, gz.zfp_type.float, 4), "f64": (torch.float64, gz.zfp_type.double, 8),
         "i32": (torch.int32, gz.zfp_type.int32, 4), "i64": (torch.int64, gz.zfp_type.int64, 8)}


def listed() -> list[dict]:
    return [
        # a simulation's state variable, written to and read back from a
        # compressed checkpoint: the headline workload of the benchmark
        {"name": "3d_f64_512_r16_compress", "kind": "field", "type": "f64", "nx": 512, "ny": 512,
         "nz": 512, "rate": 16.0, "dir": "compress", "data": "waves"},
        {"name": "3d_f64_512_r16_decompress", "kind": "field", "type": "f64", "nx": 512, "ny": 512,
         "nz": 512, "rate": 16.0, "dir": "decompress", "data": "waves"},
        # one small tile of a tiled volume, called over and over: latency
        {"name": "3d_f32_64_r16", "kind": "field", "type": "f32", "nx": 64, "ny": 64, "nz": 64,
         "rate": 16.0, "dir": "both", "data": "noisy"},
        # a volume whose edges are no multiple of the block's (ghost cells,
        # scan data): partial blocks and rows that are not aligned
        {"name": "3d_f32_ragged_r8", "kind": "field", "type": "f32", "nx": 383, "ny": 385,
         "nz": 301, "rate": 8.0, "dir": "both", "data": "noisy"},
        # a long recording (a trace, a time series)
        {"name": "1d_f32_walk_r12_compress", "kind": "field", "type": "f32", "nx": (1 << 26) - 3,
         "ny": 0, "nz": 0, "rate": 12.0, "dir": "compress", "data": "walk"},
        {"name": "1d_f32_walk_r12_decompress", "kind": "field", "type": "f32", "nx": (1 << 26) - 3,
         "ny": 0, "nz": 0, "rate": 12.0, "dir": "decompress", "data": "walk"},
        # a map or slice, both ways
        {"name": "2d_f32_r12", "kind": "field", "type": "f32", "nx": 4093, "ny": 4095, "nz": 0,
         "rate": 12.0, "dir": "both", "data": "waves"},
        # detector frames: integer counts
        {"name": "2d_i32_frame_r8", "kind": "field", "type": "i32", "nx": 1920, "ny": 1081, "nz": 0,
         "rate": 8.0, "dir": "both", "data": "noisy"},
        # an error bound instead of a rate; the reader has zfp's stream alone
        {"name": "3d_f64_256_acc1e-6_compress", "kind": "mode", "type": "f64", "nx": 256, "ny": 256,
         "nz": 256, "tolerance": 1e-6, "precision": 0, "dir": "compress", "data": "waves"},
        {"name": "3d_f64_256_acc1e-6_decompress", "kind": "mode", "type": "f64", "nx": 256,
         "ny": 256, "nz": 256, "tolerance": 1e-6, "precision": 0, "dir": "decompress",
         "data": "waves"},
        # the patches of an adaptive mesh in one call each way
        {"name": "batch_96_mixed", "kind": "batch", "arrays": 96, "lo": 17, "hi": 129, "mix": 1},
        # a compressed array's cache misses: scattered blocks fetched and
        # written back
        {"name": "blocks_20000_f64_r16", "kind": "blocks", "type": "f64", "edge": 256, "rate": 16.0,
         "count": 20000},
    ]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["field", "field", "field", "field", "mode", "batch", "blocks"])
    if kind == "batch":
        return {"kind": "batch", "arrays": int(round(math.exp(rng.uniform(math.log(8), math.log(128))))),
                "lo": 17, "hi": rng.randint(48, 129), "mix": rng.randrange(1 << 20)}
    if kind == "blocks":
        return {"kind": "blocks", "type": rng.choice(["f32", "f64"]), "edge": rng.randint(40, 256),
                "rate": float(rng.randint(4, 32)), "count": rng.randint(200, 30000)}
    if kind == "mode":
        dims = rng.choice([2, 3])
        nx, ny, nz = _draw_shape(rng, dims, 1 << 15, 1 << 22)
        t = rng.choice(["f32", "f64", "f64"])
        acc = rng.random() < 0.6
        return {"kind": "mode", "type": t, "nx": nx, "ny": ny, "nz": nz,
                "tolerance": 10.0 ** rng.uniform(-6, -2) if acc else 0.0,
                "precision": 0 if acc else rng.randint(12, 28),
                "dir": rng.choice(["compress", "decompress"]), "data": rng.choice(["waves", "noisy"])}
    dims = rng.choice([1, 2, 3, 3])
    nx, ny, nz = _draw_shape(rng, dims, 1 << 15, 1 << 25)
    rate = rng.choice([float(rng.choice([4, 8, 12, 16, 24, 32])), round(rng.uniform(4, 32), 2)])
    return {"kind": "field", "type": rng.choice(["f32", "f32", "f64", "f64", "i32", "i64"]),
            "nx": nx, "ny": ny, "nz": nz, "rate": rate,
            "dir": rng.choice(["compress", "decompress", "both"]),
            "data": "walk" if dims == 1 else rng.choice(["waves", "noisy"])}


def _draw_shape(rng: random.Random, dims: int, lo: int, hi: int):
    """Edges of a dims-dimensional array of lo .. hi values, not all alike."""
    values = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    edge = values ** (1.0 / dims)
    n = [max(5, int(edge * rng.uniform(0.8, 1.25))) for _ in range(dims)]
    if rng.random() < 0.4:  # rows of whole blocks
        n[0] = max(8, n[0] // 8 * 8)
    return tuple((n + [0, 0])[:3])


# ------------------------------------------------------------------ inputs

def _shape(case):
    """The C-ordered shape of a case's array."""
    return tuple(n for n in (case["nz"], case["ny"], case["nx"]) if n)


def _make(shape, dtype, data, seed):
    """A field: smooth waves, the same with measurement noise, or a walk.
    Integer fields hold such values as counts."""
    if data == "walk":
        x = synth.random_walk_device(shape[0], seed=seed, dtype=torch.float64, device=DEV)
        scale = {torch.int32: 2.0 ** 10, torch.int64: 2.0 ** 30}.get(dtype)
    else:
        x = synth.sinusoids_device(shape, 8 if len(shape) == 2 else 16, 32, seed=seed,
                                   dtype=torch.float64, device=DEV)
        if data == "noisy":
            g = torch.Generator(device=DEV)
            g.manual_seed(seed)
            x += 1e-3 * torch.randn(shape, generator=g, dtype=torch.float64, device=DEV)
        scale = {torch.int32: 2.0 ** 20, torch.int64: 2.0 ** 40}.get(dtype)
    if scale is not None:
        return torch.round(x * scale).to(dtype)
    return x.to(dtype)


def _batch_specs(case):
    """Shape, type and rate of every array of a batch."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["arrays"]):
        n = [int(round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))))
             for _ in range(3)]
        out.append((tuple(n), r.choice(["f32", "f64"]), float(r.choice([4, 8, 16, 32]))))
    return out


def _zfp(case, words=None, field=None):
    """The stream record of a case: its parameters, as a program sets them."""
    t = TYPES[case["type"]][1]
    z = gz.zfp_stream(stream=words)
    if case["kind"] == "mode":
        if case["precision"]:
            gz.zfp_stream_set_precision(z, case["precision"], t)
        else:
            gz.zfp_stream_set_accuracy(z, case["tolerance"], t)
    else:
        gz.stream_set_rate(z, case["rate"], t, len(_shape(case)))
    return z


def _record(case, x):
    t = TYPES[case["type"]][1]
    return gz.zfp_field(type=t, nx=case["nx"], ny=case["ny"], nz=case["nz"], data=x)


def _arena(sizes, dtype):
    """One zeroed buffer and a slice of it per size, 256 bytes aligned."""
    step = 256 // torch.empty((), dtype=dtype).element_size()
    at, n = [], 0
    for s in sizes:
        at.append(n)
        n += -(-s // step) * step
    flat = torch.zeros(max(n, 1), dtype=dtype, device=DEV)
    return flat, [flat[a:a + s] for a, s in zip(at, sizes)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "blocks":
        return _prepare_blocks(case, seed)
    dtype, t, _ = TYPES[case["type"]]
    x = _make(_shape(case), dtype, case["data"], seed)
    z = _zfp(case)
    f = _record(case, x)
    z.stream = torch.zeros(gz.zfp_stream_maximum_size(z, f) // 8, dtype=torch.int64, device=DEV)
    nbytes = 0
    if kind == "field":
        z.stream = z.stream[:gz.stream_size(t, case["nx"], case["ny"], case["nz"], z.maxbits) // 8]
    if case["dir"] == "decompress":
        nbytes = gz.compress(z, f)
        z.stream = z.stream[:nbytes // 8].clone()
        f.data = None
        del x
    if case["dir"] != "compress":
        g = _record(case, torch.empty(_shape(case), dtype=dtype, device=DEV))
    else:
        g = None
    return {"case": case, "zfp": z, "in": f, "out": g}


def _prepare_batch(case, seed):
    specs = _batch_specs(case)
    fields = [_make(s, TYPES[t][0], "noisy", seed + i) for i, (s, t, _) in enumerate(specs)]
    rates = [r for _, _, r in specs]
    words = [w.numel() for w in gz.batch_stream_buffers(fields, rates)]
    flat_words, streams = _arena(words, torch.int64)
    flat, decoded = {}, [None] * len(specs)
    for t in ("f32", "f64"):
        of = [i for i, s in enumerate(specs) if s[1] == t]
        flat[t], parts = _arena([fields[i].numel() for i in of], TYPES[t][0])
        for i, p in zip(of, parts):
            decoded[i] = p.view(specs[i][0])
    return {"case": case, "fields": fields, "rates": rates, "streams": streams, "decoded": decoded,
            "out": {"words": flat_words, "f32": flat["f32"], "f64": flat["f64"]}}


def _prepare_blocks(case, seed):
    dtype, t, _ = TYPES[case["type"]]
    e = case["edge"]
    x = _make((e, e, e), dtype, "noisy", seed)
    words = gz.compress_tensor(x, case["rate"])
    maxbits = int(round(case["rate"] * 64))
    nb = ((e + 3) // 4) ** 3
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    count = min(case["count"], nb)
    idx = torch.randperm(nb, generator=g, device=DEV)[:count].contiguous()
    whole = gz.decode_blocks(words, dtype, 3, maxbits, idx)
    return {"case": case, "words": words, "target": words.clone(), "maxbits": maxbits, "idx": idx,
            "new": (whole * 1.25).contiguous(), "tiles": torch.zeros_like(whole), "field": x}


# --------------------------------------------------------------------- run

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        gz.compress_batch(state["fields"], state["rates"], state["streams"])
        gz.decompress_batch(state["streams"], state["decoded"], state["rates"])
        return state["out"]
    if kind == "blocks":
        gz.decode_blocks(state["words"], state["tiles"].dtype, 3, state["maxbits"], state["idx"],
                         out=state["tiles"])
        gz.encode_blocks(state["new"], 3, state["maxbits"], state["idx"], state["target"])
        return {"tiles": state["tiles"], "words": state["target"]}
    z = state["zfp"]
    out = {}
    if case["dir"] != "decompress":
        out["bytes"] = gz.compress(z, state["in"])
        out["words"] = z.stream  # zeros after the stream's last word
    if case["dir"] != "compress":
        gz.decompress(z, state["out"])
        out["values"] = state["out"].data
    return out


def exact(case, seed):
    """The values that decoded outputs stand for: the field itself, in 64
    bits.  (The codec is lossy by design; streams and integers have no such
    value and have to come out bit for bit.)"""
    kind = case["kind"]
    if kind == "batch":
        specs = _batch_specs(case)
        flat = {}
        for t in ("f32", "f64"):
            of = [i for i, s in enumerate(specs) if s[1] == t]
            whole, parts = _arena([math.prod(specs[i][0]) for i in of], TYPES[t][0])
            for i, p in zip(of, parts):
                p.copy_(_make(specs[i][0], TYPES[t][0], "noisy", seed + i).view(-1))
            flat[t] = whole.double()
        return {"words": None, "f32": flat["f32"], "f64": flat["f64"]}
    if kind == "blocks":
        dtype = TYPES[case["type"]][0]
        e, nb1 = case["edge"], (case["edge"] + 3) // 4
        x = _make((e, e, e), dtype, "noisy", seed).double()
        g = torch.Generator(device=DEV)
        g.manual_seed(seed)
        idx = torch.randperm(nb1 ** 3, generator=g, device=DEV)[:min(case["count"], nb1 ** 3)]
        if e % 4:  # a partial block's padding has no value in the field
            return None
        tiles = x.view(nb1, 4, nb1, 4, nb1, 4).permute(0, 2, 4, 1, 3, 5).reshape(-1, 64)
        return {"tiles": tiles[idx], "words": None}
    if case["dir"] == "compress" or case["type"] in ("i32", "i64"):
        return None
    out = {"values": _make(_shape(case), TYPES[case["type"]][0], case["data"], seed).double()}
    if case["dir"] == "both":
        out["words"] = out["bytes"] = None
    return out


# -------------------------------------------------------------------- work

def _blocks_of(shape):
    return math.prod((n + 3) // 4 for n in shape)


def work(case):
    """Bytes a pass cannot do without: every value and every stream bit read
    or written once.  (Variable-length streams: their length is known only
    after coding; estimated from the bits a value takes.)  No flops: the
    codec's arithmetic is on integers."""
    kind = case["kind"]
    if kind == "batch":
        n = sum(math.prod(s) * TYPES[t][2] + _blocks_of(s) * 8 * r for s, t, r in _batch_specs(case))
        return {"bytes": 2 * int(n), "flops": 0}
    if kind == "blocks":
        count = min(case["count"], ((case["edge"] + 3) // 4) ** 3)
        return {"bytes": int(2 * count * (64 * TYPES[case["type"]][2] + 8 * case["rate"] + 8)),
                "flops": 0}
    shape = _shape(case)
    size = TYPES[case["type"]][2]
    if kind == "mode":
        bits = case["precision"] / 2 if case["precision"] else 1 - 1.1 * math.log10(case["tolerance"])
        stream = math.prod(shape) * bits / 8
    else:
        stream = _blocks_of(shape) * 4 ** len(shape) * case["rate"] / 8
    passes = 2 if case["dir"] == "both" else 1
    return {"bytes": int(passes * (math.prod(shape) * size + stream)), "flops": 0}
