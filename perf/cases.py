"""Performance cases of the create engine, through its public entry points.

The work a user has it do: Reed-Solomon encodes on device buffers (the
accumulator alone), whole device jobs (encode, slice checksums, file hashes,
packet MD5s), batches of jobs in one launch, and the calls on host buffers
(hash seams and the in-memory create).  Shapes come from this repository's
named workloads (``par2rust_b200.workloads``), its tests and its benchmark;
ragged sizes stand beside the round ones.

A case is a dict: ``op`` names the entry point, the rest are its sizes; file
sizes are ``count`` draws, log-uniform in [``lo``, ``hi``], from the seed
``sizes``.
Source bytes are uniform random, as in the named workloads: GF(2^16), MD5 and
CRC32 costs do not depend on the values.
"""
import hashlib
import math
import zlib

import numpy as np
import torch

import par2rust_b200 as p2g


def listed():
    return [
        # latency of one call: a handful of small slices, a few recovery rows
        {"name": "encode_tiny", "op": "encode", "slices": 6, "slice": 4096, "rows": 3, "first": 0, "pad": 0},
        # ordinary small set: 16 MiB in 256 KiB slices, 32 rows
        {"name": "encode_16m", "op": "encode", "slices": 64, "slice": 262144, "rows": 32, "first": 0, "pad": 0},
        # ragged everything: slice not a multiple of 16, odd slice and row counts, a later exponent range
        {"name": "encode_ragged", "op": "encode", "slices": 331, "slice": 100004, "rows": 53, "first": 1021, "pad": 12},
        # the README-sized file of the benchmark: 538 MB, 512 KiB slices, 200 rows
        {"name": "encode_538m", "op": "encode", "slices": 1027, "slice": 524288, "rows": 200, "first": 0, "pad": 0},
        # many rows over short slices
        {"name": "encode_rows", "op": "encode", "slices": 2000, "slice": 32768, "rows": 2000, "first": 0, "pad": 0},
        # whole device job, the 16 MiB workload
        {"name": "job_16m", "op": "job", "count": 1, "lo": 16777216, "hi": 16777216, "sizes": 0,
         "slice": 65536, "rows": 32, "full": False},
        # whole device job, the benchmark's headline file
        {"name": "job_538m", "op": "job", "count": 1, "lo": 538218411, "hi": 538218411, "sizes": 0,
         "slice": 524288, "rows": 200, "full": False},
        # many small files with their whole-file MD5s on the device (source tree, photo folder)
        {"name": "job_files", "op": "job", "count": 400, "lo": 1024, "hi": 1 << 20, "sizes": 7,
         "slice": 20480, "rows": 300, "full": True},
        # a batch of mixed jobs in one launch, drawn as in the 256-job workload
        {"name": "batch_mixed", "op": "batch", "jobs": 48, "sizes": 11},
        # per-slice MD5 and CRC32 of host slices (the scan of one file)
        {"name": "checksums_64m", "op": "checksums", "slices": 512, "slice": 131072},
        # hashes of a folder of small host files
        {"name": "hashes_files", "op": "hashes", "count": 300, "lo": 64, "hi": 1 << 18, "sizes": 13},
        # the in-memory create from host buffers to the finished index and volume files
        {"name": "create_mem", "op": "create", "count": 24, "lo": 4096, "hi": 4 << 20, "sizes": 17,
         "slice": 65536, "rows": 40},
    ]


def draw(rng):
    op = rng.choice(["encode", "encode", "job", "job", "batch", "checksums", "hashes", "create"])
    if op == "encode":
        while True:
            slices, rows = _log(rng, 2, 4000), _log(rng, 1, 2000)
            size = 4 * _log(rng, 256, 1 << 18)
            if slices * rows * (size // 2) <= 5e10 and slices * size <= 1 << 30 and rows * size <= 1 << 29:
                break
        return {"op": op, "slices": slices, "slice": size, "rows": rows, "first": rng.choice([0, 0, _log(rng, 1, 60000)]),
                "pad": (-size) % 16}
    if op == "job":
        n, size = _log(rng, 1, 400), rng.choice([16384, 65536, 262144, 524288, 4 * _log(rng, 1024, 1 << 17)])
        case = {"op": op, "count": n, "lo": 1024, "hi": max(2048, min(64 << 20, (256 << 20) // n)),
                "sizes": rng.randrange(1 << 30), "slice": size}
        slices = sum(-(-x // size) for x in _files(case))
        return dict(case, rows=min(1000, max(1, int(rng.uniform(0.01, 0.20) * slices))), full=n > 64)
    if op == "batch":
        while True:
            case = {"op": op, "jobs": _log(rng, 2, 48), "sizes": rng.randrange(1 << 30)}
            w = work(case)
            if w["flops"] <= 6e11 and w["bytes"] <= 3e9:
                return case
    if op == "checksums":
        size = 4 * _log(rng, 256, 1 << 16)
        return {"op": op, "slices": min(_log(rng, 4, 1024), (64 << 20) // size), "slice": size}
    if op == "hashes":
        return {"op": op, "count": _log(rng, 2, 300), "lo": 64, "hi": 1 << 18, "sizes": rng.randrange(1 << 30)}
    return {"op": op, "count": _log(rng, 1, 24), "lo": 4096, "hi": 4 << 20, "sizes": rng.randrange(1 << 30),
            "slice": 4 * _log(rng, 4096, 1 << 16), "rows": _log(rng, 1, 60)}


def prepare(case, seed):
    op = case["op"]
    if op == "encode":
        stride = case["slice"] + case["pad"]
        src = _slices(case["slices"], case["slice"], stride, seed)
        rec = torch.empty((case["rows"], stride), dtype=torch.uint8, device="cuda")
        return {"op": op, "src": src, "rec": rec, "case": case, "stride": stride}
    if op == "job":
        src, spec = _job_state(_files(case), case["slice"], case["rows"], seed)
        return dict(spec, op=op, src=src, full=case["full"])
    if op == "batch":
        specs = []
        for k, j in enumerate(_job_shapes(case["sizes"], case["jobs"])):
            src, s = _job_state(j["files"], j["slice"], j["rows"], seed * 1000 + k)
            specs.append(p2g.BatchJobSpec(src, s["files"], s["names"], j["slice"], j["rows"], s["bufs"]))
        # one arena per kind of output, each job's buffers a view of it
        kinds = ("recovery", "checksums", "hash16k", "packet_md5", "set_id_device")
        arenas = []
        for kind in kinds:
            sizes = [getattr(s.bufs, kind).numel() for s in specs]
            arena = torch.empty(sum(sizes), dtype=torch.uint8, device="cuda")
            for s, view in zip(specs, arena.split(sizes)):
                setattr(s.bufs, kind, view)
            arenas.append(arena)
        return {"op": op, "specs": specs, "arenas": arenas, "batch": p2g.Batch(specs)}
    if op == "checksums":
        return {"op": op, "src": _bytes(case["slices"] * case["slice"], seed).cpu().numpy(), "slice": case["slice"]}
    data = _host_files(_files(case), seed)
    if op == "hashes":
        return {"op": op, "files": data}
    opts = p2g.CreateOptions(output="set.par2", slice_size=case["slice"], recovery_block_count=case["rows"],
                             volume_scheme=p2g.VolumeScheme.Exponential())
    return {"op": op, "opts": opts, "inputs": list(zip(_names(len(data)), data))}


def run(state):
    op = state["op"]
    if op == "encode":
        c = state["case"]
        p2g.encode_device(state["src"].data_ptr(), state["stride"], c["slices"], c["slice"], c["rows"],
                          state["rec"].data_ptr(), state["stride"], torch.cuda.current_stream().cuda_stream,
                          first_exponent=c["first"])
        return state["rec"][:, :c["slice"]]
    if op == "job":
        b = p2g.run_device_job(state["src"], state["files"], state["names"], state["slice"], state["rows"],
                               state["bufs"], skip_hash_full=not state["full"])
        return _outputs(b, state["rows"], state["slice"], state["full"]) + [np.frombuffer(b.set_id, dtype=np.uint8)]
    if op == "batch":
        state["batch"].launch()
        return state["arenas"]
    if op == "checksums":
        out = p2g.slice_checksums(state["src"], state["slice"])
        return (np.frombuffer(b"".join(c.md5 for c in out), dtype=np.uint8),
                np.array([c.crc32 for c in out], dtype=np.int64))
    if op == "hashes":
        return np.frombuffer(b"".join(a + b for a, b in p2g.file_hashes(state["files"])), dtype=np.uint8)
    return [np.frombuffer(data, dtype=np.uint8) for _, data in p2g.create_in_memory(state["opts"], state["inputs"])]


def work(case):
    """Source read once, outputs written once; a GF multiply-accumulate counts as two operations."""
    op = case["op"]
    if op == "encode":
        return {"bytes": (case["slices"] + case["rows"]) * case["slice"],
                "flops": case["slices"] * case["rows"] * case["slice"]}
    if op in ("job", "create"):
        return _job_work(_files(case), case["slice"], case["rows"])
    if op == "batch":
        parts = [_job_work(j["files"], j["slice"], j["rows"]) for j in _job_shapes(case["sizes"], case["jobs"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if op == "checksums":
        return {"bytes": case["slices"] * (case["slice"] + 20), "flops": 0}
    return {"bytes": sum(_files(case)) + 32 * case["count"], "flops": 0}


def exact(case, seed):
    op = case["op"]
    if op == "encode":
        if case["slices"] * case["rows"] * case["slice"] > 2e9:
            return None
        src = _slices(case["slices"], case["slice"], case["slice"] + case["pad"], seed).cpu().numpy()
        return _encode(src[:, :case["slice"]], case["rows"], case["first"])
    if op == "checksums":
        src = _bytes(case["slices"] * case["slice"], seed).cpu().numpy().reshape(case["slices"], case["slice"])
        return (np.frombuffer(b"".join(hashlib.md5(s).digest() for s in src), dtype=np.uint8),
                np.array([zlib.crc32(s) for s in src], dtype=np.int64))
    if op == "hashes":
        return np.frombuffer(b"".join(hashlib.md5(d).digest() + hashlib.md5(d[:16384]).digest()
                                      for d in _host_files(_files(case), seed)), dtype=np.uint8)
    return None


# ---- sizes ----------------------------------------------------------------
def _log(rng, lo, hi):
    """Log-uniform in [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _files(case):
    if case["lo"] == case["hi"]:
        return [case["lo"]] * case["count"]
    rng = np.random.default_rng(case["sizes"])
    return [int(x) for x in np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))]


def _job_shapes(seed, n):
    """Jobs of 1-16 files, log-uniform in [4 KiB, 64 MiB], with 1-20 % recovery rows."""
    rng = np.random.default_rng(seed)
    jobs = []
    for _ in range(n):
        files = [int(x) for x in np.exp(rng.uniform(math.log(4096), math.log(64 << 20), rng.integers(1, 17)))]
        size = int(rng.choice([16384, 65536, 262144, 1048576]))
        rows = math.ceil(rng.uniform(0.01, 0.20) * sum(-(-x // size) for x in files))
        jobs.append({"files": files, "slice": size, "rows": max(1, rows)})
    return jobs


def _job_work(files, size, rows):
    slices = sum(-(-x // size) for x in files)
    return {"bytes": sum(files) + rows * (size + 16) + 20 * slices + 16 * len(files), "flops": slices * rows * size}


# ---- inputs ---------------------------------------------------------------
def _bytes(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    words = torch.randint(-(1 << 63), (1 << 63) - 1, (-(-n // 8),), dtype=torch.int64, device="cuda", generator=g)
    return words.view(torch.uint8)[:n]


def _slices(count, size, stride, seed):
    """count slices of `size` random bytes, `stride` apart, zeros between them."""
    src = torch.zeros((count, stride), dtype=torch.uint8, device="cuda")
    src[:, :size] = _bytes(count * size, seed).view(count, size)
    return src


def _names(n):
    return [b"dir/file-%04d.bin" % i for i in range(n)]


def _job_state(files, size, rows, seed):
    """A device job's source (files on slice boundaries, zero-padded) and what its call takes."""
    slices = sum(-(-x // size) for x in files)
    src = torch.zeros(slices * size + 16, dtype=torch.uint8, device="cuda")
    data = _bytes(sum(files), seed)
    at = off = 0
    for x in files:
        src[at * size:at * size + x] = data[off:off + x]
        at += -(-x // size)
        off += x
    bufs = p2g.DeviceJobBuffers(slices, len(files), size, rows, src.device)
    return src, {"files": list(files), "names": _names(len(files)), "slice": size, "rows": rows, "bufs": bufs}


def _host_files(files, seed):
    data = _bytes(sum(files), seed).cpu().numpy().tobytes()
    out, off = [], 0
    for x in files:
        out.append(data[off:off + x])
        off += x
    return out


def _outputs(b, rows, size, full):
    rec = b.recovery[:rows * b.rec_stride].view(rows, b.rec_stride)[:, :size]
    return [rec, b.checksums, b.hash16k, b.packet_md5] + ([b.hash_full] if full else [])


# ---- plain GF(2^16) encode ------------------------------------------------
def _encode(src, rows, first):
    """recovery[r] = XOR over s of base_s^(first + r) * source[s], symbols little-endian, polynomial 0x1100B."""
    antilog = np.zeros(65535, dtype=np.int64)
    log = np.zeros(65536, dtype=np.int64)
    v = 1
    for k in range(65535):
        antilog[k], log[v] = v, k
        v <<= 1
        if v & 0x10000:
            v ^= 0x1100B
    bases = [k for k in range(65535) if math.gcd(k, 65535) == 1][:len(src)]
    lo, hi = log[np.arange(1, 256)], log[np.arange(1, 256) << 8]
    table = np.zeros((2, 256), dtype=np.uint16)
    sym = src.view("<u2") if src.flags.c_contiguous else np.ascontiguousarray(src).view("<u2")
    low, high = (sym & 255).astype(np.intp), (sym >> 8).astype(np.intp)
    out = np.zeros((rows, sym.shape[1]), dtype=np.uint16)
    for r in range(rows):
        for s, base in enumerate(bases):
            c = base * (first + r) % 65535
            table[0, 1:] = antilog[(lo + c) % 65535]
            table[1, 1:] = antilog[(hi + c) % 65535]
            out[r] ^= table[0].take(low[s]) ^ table[1].take(high[s])
    return out.view(np.uint8)
