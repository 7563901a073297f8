"""The work that programs have this framework do, as cases that can be timed:
reads of one block, of chunks and of region batches at the qualities archives
are written with, decodes on the device and into host memory, appends with and
without a max-error bound, the LOD pyramid and the deblocking filter.

A case is a dict of plain values; `prepare` makes what a program has in hand
before the call (an archive of seeded synthetic volumes, output buffers, a
plan), `run` makes the call through the public entry points, `work` gives the
bytes that one pass cannot do without. Decoded voxels and archive bytes are
whole numbers; `exact` restates the one path that needs no codec tables.
"""
import ctypes
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "matter-compressor_b200"))

import mcb200  # noqa: E402
import volumes  # noqa: E402

CHUNK = mcb200.CHUNK
# Coded bytes per voxel at a quality, about: what the synthetic volumes give.
RATE = ((0.5, 0.30), (1.0, 0.20), (3.0, 0.06), (6.0, 0.028), (12.0, 0.018), (64.0, 0.006))


def listed():
    return [
        # a viewer or a sparse reader asking for single blocks, one call each, into host memory
        {"name": "block_requests", "kind": "blocks", "q": 6.0, "n": 8},
        # a program written for the CPU library decoding one whole chunk into its own (pageable) memory
        {"name": "chunk_request", "kind": "chunk", "q": 3.0},
        # payloads already on the GPU, decoded without an allocation inside a training step
        {"name": "gpu_blocks", "kind": "noalloc", "q": 3.0, "n": 700},
        # a few chunks in HBM decoded again and again by a plan: a small field of view at a low quality
        {"name": "plan_3_chunks", "kind": "plan", "q": 12.0, "n": 3},
        # the batched decode of a resident archive at the headline quality
        {"name": "plan_64_chunks", "kind": "plan", "q": 6.0, "n": 64},
        # the same at archival quality: long streams, few chunks
        {"name": "plan_q1_12_chunks", "kind": "plan", "q": 1.0, "n": 12},
        # a data loader's batch of crops at unaligned places, the work list built by every call
        {"name": "region_batch", "kind": "regions", "q": 6.0, "n": 64, "dz": 128, "dy": 128, "dx": 128},
        # compressed chunks arriving in pinned host memory, voxels wanted there
        {"name": "host_blobs", "kind": "blobs", "q": 6.0, "n": 16},
        # an archive being written from volumes on the GPU, no max error
        {"name": "append_q6", "kind": "append", "q": 6.0, "tau": 0, "n": 8, "host": False},
        # the "high" preset (q = 1, |error| <= 4) from a scanner's host buffers
        {"name": "append_bounded", "kind": "append", "q": 1.0, "tau": 4, "n": 2, "host": True},
        # every LOD of a volume of no round size
        {"name": "pyramid", "kind": "pyramid", "q": 12.0, "dz": 300, "dy": 450, "dx": 601},
        # decoded volumes deblocked for display (a copy: the decoded voxels are kept)
        {"name": "deblock", "kind": "deblock", "q": 6.0, "n": 16, "dz": 256, "dy": 256, "dx": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["blocks", "chunk", "noalloc", "plan", "plan", "plan", "regions", "regions", "blobs", "append",
                       "append", "pyramid", "deblock"])
    q = round(math.exp(rng.uniform(0.0, math.log(16.0))) * 8) / 8
    if kind == "blocks":
        return {"kind": kind, "q": q, "n": rng.randint(1, 24)}
    if kind == "chunk":
        return {"kind": kind, "q": q}
    if kind == "noalloc":   # within the call's fixed scratch at every quality
        return {"kind": kind, "q": q, "n": _log(rng, 3, 340 if q < 3 else 1000 if q < 6 else 2400)}
    if kind == "plan":
        return {"kind": kind, "q": q, "n": _log(rng, 1, 10 if q < 2 else 24 if q < 6 else 60)}
    if kind == "regions":
        dz, dy, dx = (_log(rng, 9, 200) for _ in range(3))
        return {"kind": kind, "q": max(q, 2.0), "n": max(1, min(_log(rng, 1, 64), 64 * 128 ** 3 // (dz * dy * dx))),
                "dz": dz, "dy": dy, "dx": dx}
    if kind == "blobs":
        return {"kind": kind, "q": q, "n": rng.randint(1, 16)}
    if kind == "append":
        tau = rng.choice([0, 0, 4, 8, 16])
        return {"kind": kind, "q": q, "tau": tau, "n": rng.randint(1, 2 if q < 3 else 7), "host": rng.random() < 0.4}
    if kind == "pyramid":
        dz, dy, dx = (_log(rng, 60, 500) for _ in range(3))
        return {"kind": kind, "q": max(q, 4.0), "dz": dz, "dy": dy, "dx": dx}
    dz, dy, dx = (_log(rng, 20, 600) for _ in range(3))
    return {"kind": kind, "q": q, "n": max(1, min(rng.randint(1, 16), CHUNK * 16 // (dz * dy * dx))), "dz": dz,
            "dy": dy, "dx": dx}


# ------------------------------------------------------------------ inputs
_lib = None


def _library():
    global _lib
    if _lib is None:
        _lib = mcb200.McLib.product()
    return _lib


def _voxels(seed, i, shape=(256, 256, 256)):
    """Volume i of a seed, 30 to 60 % of it air, on the GPU."""
    s = seed % 20011   # the generator hashes in 64 bits
    return volumes.region(s * 101 + i, (0, 0, 256 * i), shape, 0.3 + 0.3 * ((s * 7 + i * 5) % 8) / 7.0,
                          device="cuda").contiguous()


class Shelf:
    """An open archive in a folder of its own, removed with the state."""

    def __init__(self, nx, ny, nz, q):
        self.dir = tempfile.TemporaryDirectory()
        self.path = os.path.join(self.dir.name, "a.mca")
        self.a = _library().open(self.path, nx, ny, nz, q)

    def __del__(self):
        self.a.close()
        self.dir.cleanup()


def _chunks(seed, n, q):
    """An archive of n chunks in a row along x, and their offsets."""
    s = Shelf(256 * n, 256, 256, q)
    for c0 in range(0, n, 8):
        vox = [_voxels(seed, c) for c in range(c0, min(n, c0 + 8))]
        torch.cuda.synchronize()
        at = [(0, 0, c) for c in range(c0, c0 + len(vox))]
        assert s.a.append_chunks(0, at, [v.data_ptr() for v in vox], q, on_device=True) == 0
    return s, [s.a.chunk_offset(0, 0, 0, c) for c in range(n)]


def prepare(case, seed):
    lib, kind, q, n = _library(), case["kind"], case["q"], case.get("n", 1)
    rng = np.random.default_rng(seed)
    st = {"case": case, "lib": lib}
    if kind in ("blocks", "chunk"):
        st["shelf"], offs = _chunks(seed, 1, q)
        st["off"] = offs[0]
        if kind == "blocks":   # blocks of material, anywhere in the chunk
            coded = [b for b in rng.permutation(4096).tolist()
                     if st["shelf"].a.block_blob(offs[0], b >> 8, (b >> 4) & 15, b & 15)]
            st["blocks"] = [(b >> 8, (b >> 4) & 15, b & 15) for b in coded[:n]]
        else:
            st["out"] = np.zeros(CHUNK, np.uint8)
        st["shelf"].a.sync_device()
    elif kind == "noalloc":
        shelf, offs = _chunks(seed, 1, q)
        pay = [shelf.a.block_blob(offs[0], b >> 8, (b >> 4) & 15, b & 15) for b in rng.permutation(4096)[:n].tolist()]
        st["offs"] = np.concatenate([[0], np.cumsum([len(p) for p in pay])]).astype(np.uint64)
        raw = np.frombuffer(b"".join(pay) + bytes(16), np.uint8)
        st["pay"] = torch.from_numpy(raw.copy()).cuda()
        st["out"] = torch.zeros(n, 4096, dtype=torch.uint8, device="cuda")
    elif kind == "plan":
        st["shelf"], offs = _chunks(seed, n, q)
        st["out"] = torch.zeros(n, CHUNK, dtype=torch.uint8, device="cuda")
        st["plan"] = st["shelf"].a.plan_chunks(offs, st["out"].data_ptr())
    elif kind == "regions":
        # crops of a volume of 4 x 2 chunks, from any voxel on
        st["shelf"] = s = Shelf(1024, 512, 256, q)
        at = [(0, y, x) for y in range(2) for x in range(4)]
        vox = [_voxels(seed, c) for c in range(8)]
        torch.cuda.synchronize()
        assert s.a.append_chunks(0, at, [v.data_ptr() for v in vox], q, on_device=True) == 0
        s.a.sync_device()
        size = (case["dz"], case["dy"], case["dx"])
        st["boxes"] = [tuple(int(rng.integers(0, e - d + 1)) for e, d in zip((256, 512, 1024), size)) for _ in range(n)]
        st["out"] = torch.zeros(n, *size, dtype=torch.uint8, device="cuda")
        st["stream"] = torch.cuda.Stream()
    elif kind == "blobs":
        shelf, offs = _chunks(seed, n, q)
        end = int(lib.L.mc_archive_data_len(shelf.a.a))
        data = np.fromfile(shelf.path, np.uint8, count=end)
        with mcb200.Reader(lib, data=data) as r:
            blobs = [np.frombuffer(r.blob(o), np.uint8) for o in offs]
        st["blobs"] = [torch.from_numpy(b.copy()).pin_memory().numpy() for b in blobs]
        st["out"] = torch.zeros(n * CHUNK, dtype=torch.uint8).pin_memory().numpy()
    elif kind == "append":
        st["shelf"], st["next"] = Shelf(256 * 4096, 256, 256, q), 0
        vox = [_voxels(seed, c) for c in range(n)]
        st["vox"] = [v.cpu().numpy() for v in vox] if case["host"] else vox
    elif kind == "pyramid":
        size = (case["dz"], case["dy"], case["dx"])
        st["shelf"] = Shelf(size[2], size[1], size[0], q)
        st["vox"] = _voxels(seed, 0, size)
    elif kind == "deblock":
        st["src"] = _blocky(case, seed)
        st["out"] = torch.zeros_like(st["src"])
        st["stream"] = torch.cuda.Stream()
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return st


def _blocky(case, seed):
    """Volumes as a coarse block codec leaves them: material quantised with an
    offset of its own per 16^3 block, air untouched."""
    size = (case["dz"], case["dy"], case["dx"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    vols = []
    for i in range(case["n"]):
        v = _voxels(seed, i, size).to(torch.int16)
        off = torch.randint(-4, 5, [-(-s // 16) for s in size], generator=g, device="cuda", dtype=torch.int16)
        for d in range(3):
            off = off.repeat_interleave(16, d).narrow(d, 0, size[d])
        vols.append(torch.where(v > 0, (v + off).clamp(1, 255), v).to(torch.uint8))
    return torch.stack(vols)


# ------------------------------------------------------------------ one pass
def _appended(st, before, voxels):
    """The bytes that a call added to the archive's file, as the file's reader
    maps them, in a window of one size for a case (the file is allocated far
    ahead of its end, with zeros), and their number."""
    path, window = st["shelf"].path, int(2.5 * _coded(st["case"]["q"], voxels)) + (1 << 18)
    window = min(window, os.path.getsize(path) - before)
    after = int(st["lib"].L.mc_archive_data_len(st["shelf"].a.a))
    mapped = np.memmap(path, np.uint8, "r", before, (window,))
    mapped.shelf = st["shelf"]   # closing the archive cuts the file at its end
    return mapped, after - before


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "blocks":
        return [st["shelf"].a.decode_block(st["off"], *b) for b in st["blocks"]]
    if kind == "chunk":
        return st["shelf"].a.decode_chunk(st["off"], out=st["out"])
    if kind == "noalloc":
        rc = st["lib"].L.mc_b200_decode_blocks_noalloc(
            ctypes.c_void_p(st["pay"].data_ptr()), ctypes.c_void_p(st["offs"].ctypes.data), case["n"], case["q"],
            ctypes.c_void_p(st["out"].data_ptr()), None)
        assert rc == 0
        return st["out"]
    if kind == "plan":
        st["plan"].launch()
        return st["out"]
    if kind == "regions":
        st["shelf"].a.read_regions_dev(0, st["boxes"], case["dz"], case["dy"], case["dx"], st["out"].data_ptr(),
                                       stream=st["stream"].cuda_stream)
        return st["out"]
    if kind == "blobs":
        return mcb200.decode_chunk_blobs(st["lib"], st["blobs"], out=st["out"])
    if kind == "append":
        a, n, host = st["shelf"].a, case["n"], case["host"]
        before = int(st["lib"].L.mc_archive_data_len(a.a))
        at = [(0, 0, (st["next"] + i) % 4096) for i in range(n)]
        st["next"] += n
        vox = st["vox"] if host else [v.data_ptr() for v in st["vox"]]
        bound = {"ctx_q": case["q"], "ctx_tau": case["tau"]} if case["tau"] else {}
        assert a.append_chunks(0, at, vox, case["q"], on_device=not host, **bound) == 0
        return _appended(st, before, CHUNK * n)
    if kind == "pyramid":
        a = st["shelf"].a
        before = int(st["lib"].L.mc_archive_data_len(a.a))
        rc, levels = a.append_pyramid(st["vox"].data_ptr(), case["dz"], case["dy"], case["dx"], case["q"])
        assert rc == 0
        return _appended(st, before, case["dz"] * case["dy"] * case["dx"]), levels
    with torch.cuda.stream(st["stream"]):
        st["out"].copy_(st["src"])
        st["lib"].deblock_dev(st["out"].data_ptr(), case["n"], st["out"].stride(0), case["dz"], case["dy"], case["dx"],
                              case["q"], st["stream"].cuda_stream)
    return st["out"]


# ------------------------------------------------------------------ bounds
def _coded(q, voxels):
    """Bytes that hold this many voxels at a quality, interpolated over its logarithm."""
    xs = [math.log(r[0]) for r in RATE]
    ys = [math.log(r[1]) for r in RATE]
    return voxels * math.exp(float(np.interp(math.log(q), xs, ys)))


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    size = case.get("dz", 0) * case.get("dy", 0) * case.get("dx", 0)
    vox = {"blocks": 4096 * n, "chunk": CHUNK, "noalloc": 4096 * n, "plan": CHUNK * n, "regions": size * n,
           "blobs": CHUNK * n, "append": CHUNK * n, "pyramid": size, "deblock": size * n}[kind]
    if kind == "deblock":
        return {"bytes": 2.0 * vox, "flops": 0.0}
    if kind == "pyramid":   # each level is read, and written an eighth as large
        return {"bytes": vox * 8 / 7 + vox / 7 + _coded(case["q"], vox * 8 / 7), "flops": 96.0 * 2 * vox}
    # a separable 16-point transform of every voxel: three sums of 16 products
    return {"bytes": vox + _coded(case["q"], vox), "flops": 96.0 * vox}


def exact(case, seed):
    """The deblocked volumes in whole numbers; the codec's own outputs are defined by its tables."""
    if case["kind"] != "deblock":
        return None
    v = _blocky(case, seed).to(torch.int64)
    beta, tc = int(3.0 * case["q"] + 6.0), int(0.5 * case["q"] + 1.0)
    flat = v.view(case["n"], -1)
    total = flat.shape[1]
    z, y, x = (torch.arange(case[d], device="cuda") for d in ("dz", "dy", "dx"))
    lin = (z.view(-1, 1, 1) * case["dy"] + y.view(1, -1, 1)) * case["dx"] + x.view(1, 1, -1)
    for axis, step in ((2, 1), (1, case["dx"]), (0, case["dx"] * case["dy"])):
        edge = torch.arange(16, lin.shape[axis], 16, device="cuda")
        i = lin.index_select(axis, edge).reshape(-1)
        p0, q0, p1 = flat[:, i - step], flat[:, i], flat[:, i - 2 * step]
        past = i + step
        q1 = torch.where(past < total, flat[:, past.clamp(max=total - 1)], torch.zeros_like(q0))
        d = q0 - p0
        pn, qn = torch.where(p1 > 0, p1, p0), torch.where(q1 > 0, q1, q0)
        delta = ((4 * d + (pn - qn) + 4) >> 3).clamp(-tc, tc)
        on = (p0 > 0) & (q0 > 0) & (d.abs() < beta)
        flat[:, i - step] = torch.where(on, (p0 + delta).clamp(1, 255), p0)
        flat[:, i] = torch.where(on, (q0 - delta).clamp(1, 255), q0)
    return v.to(torch.uint8)
