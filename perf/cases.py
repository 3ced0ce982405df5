"""Workloads of the decompressors and encoders, as a program that keeps its data on the GPU calls
them: one call of the public Python front end (the encoders: of the C interface) per pass, with
inputs, metadata and output buffers resident in device memory.

Each case is one file (or one set of files) of the formats this package reads and writes:
  deflate     chunked zlib file, decoded (word-like text, or the raw bytes of an integer column)
  rlev1/2     chunked ORC RLE file of an integer column, decoded
  transposed  the transposed RLE v2 layout, decoded
  encode1/2   an integer column encoded into a chunked ORC RLE file
  batch       independent files of mixed size and codec, decoded by one plan

listed() holds the sizes of this package's own benchmark and tests (scaled down where making the
input would take longer than using it), draw() further cases of the same ranges.
"""
import functools
import math

import numpy as np
import torch

from codag_b200 import api, native

KIB, MIB = 1 << 10, 1 << 20


def listed():
    return [
        # a large text file: thousands of chunks, the throughput end of the Deflate decoder
        dict(name="deflate text 256 MiB", kind="deflate", data="text", bytes=256 * MIB, chunk=128 * KIB, level=6),
        # an ordinary text file: fewer chunks than the GPU has warps
        dict(name="deflate text 8 MiB", kind="deflate", data="text", bytes=8 * MIB, chunk=128 * KIB, level=6),
        # one small request with a ragged tail: the latency of a chunk
        dict(name="deflate text 200 KB", kind="deflate", data="text", bytes=200_001, chunk=128 * KIB, level=6),
        # an integer column compressed as bytes, in the 64 KiB level 9 chunks of the cuDF comparison
        dict(name="deflate column 40 MB", kind="deflate", data="column", bytes=40_000_003, chunk=64 * KIB, level=9),
        # one million 64-bit values, 64 chunks: the small column of the benchmark
        dict(name="rlev1 u64 8 MiB", kind="rlev1", elem=8, values=1 << 20, chunk=128 * KIB),
        # a large 32-bit column whose size is no multiple of the chunk
        dict(name="rlev1 u32 256 MiB", kind="rlev1", elem=4, values=67_108_863, chunk=128 * KIB),
        # the largest column of the benchmark
        dict(name="rlev2 i64 1 GiB", kind="rlev2", elem=8, values=1 << 27, chunk=128 * KIB),
        # a small 16-bit column, odd size
        dict(name="rlev2 u16 3 MB", kind="rlev2", elem=2, values=1_500_001, chunk=128 * KIB),
        # a column in the transposed layout
        dict(name="transposed i64 256 MiB", kind="transposed", elem=8, values=1 << 25, chunk=128 * KIB, read_unit=1),
        # writing a large column ...
        dict(name="encode rlev2 i64 256 MiB", kind="encode2", elem=8, values=1 << 25, chunk=128 * KIB),
        # ... and an ordinary one of odd size
        dict(name="encode rlev1 u32 20 MB", kind="encode1", elem=4, values=5_000_001, chunk=128 * KIB),
        # many files at once: 4 KiB to 1 MiB, Deflate, RLE v1 and RLE v2
        dict(name="batch 2000 files", kind="batch", files=2000, max_bytes=MIB),
    ]


def _between(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(("deflate", "deflate", "deflate", "rlev1", "rlev2", "transposed", "encode1", "encode2", "batch"))
    if kind == "deflate":
        return dict(kind=kind, data=rng.choice(("text", "text", "column")), bytes=_between(rng, 100_000, 256 * MIB),
                    chunk=rng.choice((64 * KIB, 128 * KIB, 128 * KIB)), level=rng.choice((1, 6, 6, 9)))
    if kind == "batch":
        return dict(kind=kind, files=_between(rng, 20, 2000), max_bytes=rng.choice((64 * KIB, 256 * KIB, MIB)))
    elem = rng.choice((1, 2, 4, 8))
    top = {"rlev1": 256 * MIB, "rlev2": 512 * MIB, "transposed": 256 * MIB, "encode1": 256 * MIB, "encode2": 256 * MIB}
    case = dict(kind=kind, elem=elem, values=_between(rng, 200_000, top[kind]) // elem,
                chunk=rng.choice((64 * KIB, 128 * KIB, 128 * KIB)))
    if kind == "transposed":
        case["read_unit"] = rng.choice((1, 2, 4, 8))
    return case


def _dev(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int64) if a.dtype == np.uint64 else a).to("cuda")


def _column(case, seed, values):
    gen = native.gen_rlev1_column if case["kind"] in ("rlev1", "encode1") else native.gen_rlev2_column
    return gen(values, seed, case["elem"])


def _plain_bytes(case, seed, nbytes):
    if case["data"] == "text":
        return native.gen_text(nbytes, seed)
    return native.gen_rlev2_column((nbytes + 3) // 4, seed, 4)[:nbytes]


def _mixed(case, seed):
    """Independent files of mixed codec, sizes log-uniform from 4 KiB (the sizes and codecs belong to
    the case, the contents to the seed): (packed streams, descriptors, output bytes, file sizes)."""
    n, rng = case["files"], np.random.default_rng(case["files"])
    sizes = np.exp(rng.uniform(math.log(4 * KIB), math.log(case["max_bytes"]), n)).astype(np.int64) // 8 * 8
    codec = rng.choice([native.DEFLATE, native.RLEV1, native.RLEV2], size=n, p=[0.4, 0.3, 0.3]).astype(np.uint8)
    elem = np.where(codec == native.DEFLATE, 1, np.where(rng.random(n) < 0.5, 4, 8)).astype(np.uint8)
    src = 16 * MIB
    parts = [native.gen_text(src, seed), native.gen_rlev1_column(src // 4, seed + 1, 4),
             native.gen_rlev1_column(src // 8, seed + 2, 8), native.gen_rlev2_column(src // 4, seed + 3, 4),
             native.gen_rlev2_column(src // 8, seed + 4, 8)]
    which = np.where(codec == native.DEFLATE, 0, np.where(codec == native.RLEV1, 1, 3) + (elem == 8))
    start = which * src + rng.integers(0, src - sizes + 1) // 8 * 8
    comp, descs, out_bytes = native.encode_set(np.concatenate(parts), start, sizes, codec, elem)
    return comp, descs, out_bytes, sizes


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        comp, descs, out_bytes, sizes = _mixed(case, seed)
        return dict(kind=kind, plan=api.BatchPlan(descs), comp=_dev(comp),
                    out=torch.zeros(out_bytes, dtype=torch.uint8, device="cuda"),
                    status=torch.zeros(sizes.size, dtype=torch.int32, device="cuda"))
    s = dict(kind=kind, chunk=case["chunk"], elem=case.get("elem", 1))
    if kind == "deflate":
        raw = _plain_bytes(case, seed, case["bytes"])
        comp, blk, _ = native.encode_deflate(raw, s["chunk"], case["level"], require_no_stored=False)
        off, n = blk[1:], blk.size - 2
    else:
        raw = _column(case, seed, case["values"])
        if kind in ("encode1", "encode2"):
            lib, codec = native.lib(), native.RLEV1 if kind == "encode1" else native.RLEV2
            size = (raw.size, s["chunk"], s["elem"])
            n = int(lib.codag_compress_chunks(raw.size, s["chunk"]))
            s["need"] = int(lib.codag_compress_workspace_bytes(codec, *size))
            s["col"], s["ws"] = _dev(raw), torch.empty(s["need"], dtype=torch.uint8, device="cuda")
            s["out"] = torch.zeros(int(lib.codag_compress_bound(codec, *size)), dtype=torch.uint8, device="cuda")
            s["off"] = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
            s["len"] = torch.zeros(n, dtype=torch.int64, device="cuda")
            s["meta"] = torch.zeros(2, dtype=torch.int64, device="cuda")  # [file bytes, status]
            return s
        if kind == "rlev1":
            blob, blk, ln = native.encode_rlev1(raw, s["chunk"], s["elem"])
            comp = blob[8:]
        elif kind == "rlev2":
            comp, blk, ln = native.encode_rlev2(raw, s["chunk"], s["elem"])
        else:
            s["read_unit"] = case["read_unit"]
            comp, blk, ln = native.encode_rlev2_transposed(raw, s["chunk"], s["elem"], s["read_unit"])
        n = blk.size - 1
        off = blk[:n]
        s["len"] = _dev(ln)
    s["comp"], s["off"] = _dev(comp), _dev(off)
    s["out"] = torch.zeros(raw.size, dtype=torch.uint8, device="cuda")
    s["status"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    return s


def run(s):
    kind = s["kind"]
    if kind == "encode1" or kind == "encode2":
        fn = native.lib().codag_compress_rlev1 if kind == "encode1" else native.lib().codag_compress_rlev2
        out, meta = s["out"], s["meta"]
        native.check(kind, fn(s["col"].data_ptr(), s["col"].numel(), s["chunk"], s["elem"], out.data_ptr(), out.numel(),
                              s["off"].data_ptr(), s["len"].data_ptr(), meta.data_ptr(), meta.data_ptr() + 8,
                              s["ws"].data_ptr(), s["need"], torch.cuda.current_stream().cuda_stream or None))
        return out, s["off"], s["len"], meta
    if kind == "deflate":
        api.decompress_deflate(s["comp"], s["off"], s["chunk"], s["out"], 2, None, s["status"])
    elif kind == "rlev1":
        api.decompress_rlev1(s["comp"], s["off"], s["len"], s["chunk"], s["elem"], s["out"], None, s["status"])
    elif kind == "rlev2":
        api.decompress_rlev2(s["comp"], s["off"], s["len"], s["chunk"], s["elem"], s["out"], None, s["status"])
    elif kind == "transposed":
        api.decompress_rlev2_transposed(s["comp"], s["off"], s["len"], s["chunk"], s["elem"], s["read_unit"], s["out"],
                                        None, s["status"])
    else:
        s["plan"].run(s["comp"], s["out"], s["status"], use_graph=True)
    return s["out"], s["status"]


@functools.lru_cache(maxsize=None)
def _ratio(kind, data, chunk, level, elem, read_unit):
    """Compressed bytes per byte of data of this kind, from a 2 MiB sample."""
    case = dict(kind=kind, data=data, elem=elem)
    if kind == "deflate":
        raw = _plain_bytes(case, 1, 2 * MIB)
        comp = native.encode_deflate(raw, chunk, level, require_no_stored=False)[0]
        return comp.size / raw.size
    raw = _column(case, 1, 2 * MIB // elem)
    if kind == "transposed":
        ln = native.encode_rlev2_transposed(raw, chunk, elem, read_unit)[2]
    else:
        ln = (native.encode_rlev1 if kind in ("rlev1", "encode1") else native.encode_rlev2)(raw, chunk, elem)[2]
    return float(ln.sum()) / raw.size


def work(case):
    """Bytes read once and written once; the paths do integer work only."""
    if case["kind"] == "batch":
        _, descs, _, sizes = _mixed(case, 1)
        return dict(bytes=float(sizes.sum() + descs["comp_len"].sum()), flops=0)
    raw = case["bytes"] if case["kind"] == "deflate" else case["values"] * case["elem"]
    r = _ratio(case["kind"], case.get("data"), case["chunk"], case.get("level"), case.get("elem"), case.get("read_unit"))
    return dict(bytes=raw * (1.0 + r), flops=0)
