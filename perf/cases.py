"""The codec's performance cases: the work that programs using it have it do, through its public calls.

Three ways in, each in both directions (compress, extract):

  host      zc_compress / zc_decompress (CudaCodec.compress_arrays / decompress_arrays): what `zero c` and
            `zero x` call per batch, from host memory to host memory, copies included
  device    zc_compress_device / zc_decompress_device: data that already lives on the GPU, blocks of one size
  files     zc_archive_write_device, and zc_decompress_device over the records: a folder of many files as one
            solid stream, text, LZ-structured and incompressible files side by side

over block sizes 2^16 .. 2^20, the three level classes (1, 2..8, 9) and the data the repository's benchmark
generates: text_mix (words and short repeats, many short matches), lz_mix (literal runs and log-uniform
matches) and random bytes (stored blocks).  Sizes run from one small file to a full encoder launch (1 GiB).

A program opens the codec once and keeps it for all its jobs, so the cases share one per process; its
scratch is sized by the first job that needs it.  Output buffers are cleared when a state is made, so the
bytes after a job's end are the same in every run.
"""
import atexit
import math
import os
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zero-compression_b200"))
import datagen as G  # noqa: E402
import zero_cuda as Z  # noqa: E402

KIB, MIB = 1 << 10, 1 << 20
SLACK = 64  # readable bytes the device calls ask for after their input
PIECE = 16 * MIB  # inputs are generated in pieces of this size, in parallel
# payload bytes per raw byte at block 18, level 5 (files: a third of each), for the bytes a pass must write
RATIO = {"text": 0.197, "lz": 0.169, "random": 1.0, "files": 0.455}


def listed():
    def case(name, path, op, data, size, block_log, level, files=0):
        return dict(name=name, path=path, op=op, data=data, bytes=size, block_log=block_log, level=level, files=files)

    return [
        # one small document through the default host call: a block's latency and the launches count
        case("host text 200 kB compress", "host", "compress", "text", 200_000, 18, 5),
        case("host text 200 kB extract", "host", "extract", "text", 200_000, 18, 5),
        # an ordinary job of `zero c` then `zero x` from page-locked buffers, the end-to-end measure
        case("host lz 256 MiB both ways", "host", "both", "lz", 256 * MIB, 18, 5),
        # the headline workload: one full launch at the default block size and level
        case("lz 1 GiB b18 l5 compress", "device", "compress", "lz", 1024 * MIB, 18, 5),
        case("lz 1 GiB b18 l5 extract", "device", "extract", "lz", 1024 * MIB, 18, 5),
        # the benchmark's text file: few blocks, dense short matches
        case("text 64 MiB b18 l5 compress", "device", "compress", "text", 64 * MIB, 18, 5),
        case("text 64 MiB b18 l5 extract", "device", "extract", "text", 64 * MIB, 18, 5),
        # the strongest setting: largest blocks, deepest chains; extraction is what an archive pays again
        # and again
        case("lz 256 MiB b20 l9 compress", "device", "compress", "lz", 256 * MIB, 20, 9),
        case("lz 512 MiB b20 l9 extract", "device", "extract", "lz", 512 * MIB, 20, 9),
        # the fastest setting: smallest blocks, shallow chains, an odd size whose last block is short
        case("lz 96 MB b16 l1 compress", "device", "compress", "lz", 96_000_001, 16, 1),
        # a folder of 1000 files of 1 KiB .. 1 MiB as one archive: uneven, mixed, a third incompressible
        case("1000 files b18 l5 write", "files", "compress", "files", 0, 18, 5, files=1000),
        case("1000 files b18 l5 extract", "files", "extract", "files", 0, 18, 5, files=1000),
    ]


def draw(rng):
    """A case of the same ranges: any way in, direction, data, block size and level."""
    path = rng.choice(["host", "device", "device", "files"])
    op = rng.choice(["compress", "extract"])
    block_log, level = rng.randint(16, 20), rng.choice([1, 5, 5, 9])
    if path == "files":
        return dict(path=path, op=op, data="files", bytes=0, block_log=block_log, level=level,
                    files=int(math.exp(rng.uniform(math.log(20), math.log(1200)))))
    data = rng.choice(["text", "text", "lz", "lz", "lz", "random"])
    lo, hi = (4 * KIB, 64 * MIB) if path == "host" else (MIB, 96 * MIB if data == "text" else 400 * MIB)
    size = int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1
    return dict(path=path, op=op, data=data, bytes=size, block_log=block_log, level=level, files=0)


# ---------------------------------------------------------------- inputs
_codec = None


def codec():
    global _codec
    if _codec is None:
        _codec = Z.CudaCodec(level=5)
        atexit.register(_codec.close)
    return _codec


def generate(data, size, block_log, seed, out):
    """`size` bytes of one kind into the numpy array `out`, a piece a thread."""
    def piece(k):
        a = out[k * PIECE: min((k + 1) * PIECE, size)]
        s = seed * 1009 + k
        if data == "text":
            G.text_mix(a.size, s, a)
        elif data == "lz":
            G.lz_mix(a.size, block_log, s, a)
        else:
            G.random_bytes(a.size, s, a)
    with ThreadPoolExecutor(16) as ex:
        list(ex.map(piece, range((size + PIECE - 1) // PIECE)))
    return out


def folder(case, seed):
    """The solid stream of a folder's files and their entries: the files' sizes and kinds are the case's, their
    bytes the seed's."""
    sizes, kinds = G.file_plan(case["files"], KIB, MIB, case["files"])
    sizes, kinds = [int(s) for s in sizes], [int(k) for k in kinds]
    at = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    solid = np.empty(int(at[-1]), np.uint8)

    def one(i):
        a = solid[at[i]: at[i + 1]]
        if kinds[i] == 0:
            G.text_mix(a.size, seed * 7919 + i, a)
        elif kinds[i] == 1:
            G.lz_mix(a.size, case["block_log"], seed * 7919 + i, a)
        else:
            G.random_bytes(a.size, seed * 7919 + i, a)
    with ThreadPoolExecutor(16) as ex:
        list(ex.map(one, range(len(sizes))))
    entries = [Z.ArchiveEntry("data", is_dir=True)]
    entries += [Z.ArchiveEntry("data/f%05d.bin" % i, s, 1_700_000_000 + i) for i, s in enumerate(sizes)]
    return solid, entries


def on_gpu(a):
    """Host bytes on the GPU with the readable slack after them."""
    t = torch.zeros(a.size + SLACK, dtype=torch.uint8, device="cuda")
    t[: a.size].copy_(torch.from_numpy(a))
    return t


def blocks(n, block_log):
    B = 1 << block_log
    nb = (n + B - 1) // B
    lens = np.full(nb, B, np.uint32)
    lens[-1] = n - (nb - 1) * B
    offs = np.arange(nb, dtype=np.uint64) * np.uint64(B)
    return nb, torch.from_numpy(offs.view(np.int64)).cuda(), torch.from_numpy(lens.view(np.int32)).cuda()


def compress_buffers(n, nb):
    z = lambda k, t: torch.zeros(k, dtype=t, device="cuda")  # noqa: E731
    return dict(methods=z(nb, torch.uint8), lens=z(nb, torch.int32), crcs=z(nb, torch.int32),
                out=z(n + SLACK, torch.uint8), offs=z(nb, torch.int64), total=z(1, torch.int64))


def compress_on_gpu(case, d_in, i_offs, i_lens, nb, o):
    codec().compress_device(d_in, i_offs, i_lens, nb, case["block_log"], o["methods"], o["lens"], o["crcs"], o["out"],
                            o["offs"], o["total"], stream=torch.cuda.current_stream().cuda_stream,
                            level=case["level"], out_cap=o["out"].numel() - SLACK)


def prepare(case, seed):
    c = dict(case)
    if c["path"] == "host":
        return prepare_host(c, seed)
    if c["path"] == "files":
        solid, entries = folder(c, seed)
        n = solid.size
    else:
        n = c["bytes"]
        solid, entries = generate(c["data"], n, c["block_log"], seed, np.empty(n, np.uint8)), None
    nb, offs, lens = blocks(n, c["block_log"])
    d_in = on_gpu(solid)
    del solid
    s = dict(case=c, nb=nb)
    if c["op"] == "compress" and entries:
        cap = Z.archive_bound(entries, c["block_log"])
        s.update(d_in=d_in, entries=entries, out=torch.zeros(cap, dtype=torch.uint8, device="cuda"),
                 length=torch.zeros(1, dtype=torch.int64, device="cuda"),
                 crcs=torch.zeros(len(entries), dtype=torch.int32, device="cuda"))
        return s
    o = compress_buffers(n, nb)
    if c["op"] == "compress":
        s.update(d_in=d_in, offs=offs, lens=lens, o=o)
        return s
    # extract: the blocks as the codec wrote them
    compress_on_gpu(c, d_in, offs, lens, nb, o)
    kept = int(o["total"].item())
    body = torch.zeros(kept + SLACK, dtype=torch.uint8, device="cuda")
    body[:kept].copy_(o["out"][:kept])
    s.update(body=body, b_offs=o["offs"], b_lens=o["lens"], methods=o["methods"], raw_lens=lens, offs=offs,
             raw=torch.zeros(n, dtype=torch.uint8, device="cuda"),
             crcs=torch.zeros(nb, dtype=torch.int32, device="cuda"),
             err=torch.zeros(nb, dtype=torch.int32, device="cuda"))
    return s


def pinned(n, dtype=np.uint8):
    t = torch.zeros(n * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True)
    return t.numpy().view(dtype)


def prepare_host(c, seed):
    n, B = c["bytes"], 1 << c["block_log"]
    nb = (n + B - 1) // B
    s = dict(case=c, nb=nb)
    # a program keeps the buffers of its batches; one with large jobs keeps them page-locked
    new = pinned if c["op"] == "both" else np.zeros
    s["data"] = generate(c["data"], n, c["block_log"], seed, new(n, np.uint8))
    s["keep"] = (new(nb, np.uint8), new(nb, np.uint32), new(nb, np.uint32), new(n, np.uint8), new(nb, np.uint64))
    if c["op"] == "both":
        s["raw"] = pinned(n)
        s["raw_lens"] = np.array([min(B, n - b * B) for b in range(nb)], np.uint32)
        return s
    if c["op"] == "extract":
        m, lens, _, pay, offs = codec().compress_arrays(s["data"], c["block_log"], c["level"])
        s["blob"], s["lens"], s["raw_lens"] = Z.record_bodies(s["data"], m, lens, pay, offs, c["block_log"])
        s["offs"] = np.concatenate([[0], np.cumsum(s["lens"], dtype=np.uint64)[:-1]]).astype(np.uint64)
        s["methods"] = m.copy()
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    c = s["case"]
    if c["path"] == "host":
        return run_host(s)
    st = torch.cuda.current_stream().cuda_stream
    if c["op"] == "extract":
        codec().decompress_device(s["body"], s["b_offs"], s["b_lens"], s["methods"], s["raw_lens"], s["nb"],
                                  c["block_log"], s["raw"], s["offs"], s["crcs"], s["err"], stream=st)
        return s["raw"], s["crcs"], s["err"]
    if c["path"] == "files":
        codec().archive_write_device(s["d_in"], s["entries"], c["block_log"], s["out"], s["length"], s["crcs"],
                                     stream=st, level=c["level"])
        return s["out"], s["length"], s["crcs"]
    compress_on_gpu(c, s["d_in"], s["offs"], s["lens"], s["nb"], s["o"])
    o = s["o"]
    return o["methods"], o["lens"], o["crcs"], o["out"], o["offs"], o["total"]


def run_host(s):
    c = s["case"]
    if c["op"] == "extract":
        return codec().decompress_arrays(s["blob"], s["offs"], s["lens"], s["methods"], s["raw_lens"])
    m, lens, crcs, pay, offs = codec().compress_arrays(s["data"], c["block_log"], c["level"], out=s["keep"])
    if c["op"] == "compress":
        return m, lens, crcs, pay, offs
    raw, back, err = codec().decompress_arrays(pay, offs, lens, m, s["raw_lens"], out=s["raw"])
    return m, lens, crcs, pay, offs, raw, back, err


def work(case):
    """The raw bytes and the payload bytes, each moved once a direction (byte work: no floating point)."""
    if case["path"] == "files":  # log-uniform sizes in [1 KiB, 1 MiB]: their mean is (hi - lo) / ln(hi / lo)
        raw = case["files"] * (MIB - KIB) / math.log(MIB / KIB)
    else:
        raw = case["bytes"]
    moved = raw * (1 + RATIO[case["data"]])
    return {"bytes": moved * (2 if case["op"] == "both" else 1), "flops": 0}
