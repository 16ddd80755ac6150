"""What users of this package run, at the sizes they run it: the cases a performance check times.

Every case goes through a public entry point:

  decode_batch   gpu.decode_batch on host buffers or on CUDA tensors (the reference's one GPU call)
  encode_batch   gpu.encode_batch on CUDA tensors
  archive        decode.ArchiveDecoder: run() and check() on an archive resident in HBM
  load           decode.load_archive: a file to verified plaintext in HBM, nothing prepared
  tensors        decode.decode_tensors: a few named tensors out of a file
  save           save.save_archive: BF16 weights in HBM to a file

Inputs are weights as checkpoints hold them (BF16 or FP32 from N(0, 0.02), norm vectors of ones,
later checkpoints of a chain a little noise away from the first) and the byte distributions of the
decoder's stress batches, drawn on the GPU from the seed.  Archives are written here, record by
record as the reference's `lmz compress` lays them out: 64 KiB chunks (`--mapped`) or larger plain
ones, and 8 MiB exponent-conditioned chunks (its default).
"""
from __future__ import annotations

import ctypes
import json
import math
import os
import shutil
import struct
import tempfile
import weakref
import zlib

import numpy as np
import torch

from lmz_b200 import archive as fmt, decode, gpu, save

KIB, MIB = 1 << 10, 1 << 20
CHAIN = 3                                  # checkpoints of a delta chain
SMALL_TENSOR = 64 * KIB                    # below this the reference neither deduplicates nor takes differences
COND_ELEMENTS = MIB                        # chunks of this many BF16 elements are exponent-conditioned


def listed():
    return [
        # seven short planes between host buffers: a reader that fetches one block of a file at a time
        dict(name="host batch 7x4KiB", path="decode_batch", where="host", nstr=7, plane=4096, values="exponent"),
        # the shape of the reference's own `verify` throughput batch, host buffers both ways
        dict(name="host batch 512x32KiB", path="decode_batch", where="host", nstr=512, plane=32768, values="skewed"),
        # the batch the reference's GPU numbers are quoted on: 28 577 exponent planes of 32 KiB in device memory
        dict(name="device batch 28577x32KiB", path="decode_batch", where="device", nstr=28577, plane=32768, values="exponent"),
        # coding the exponent planes of a 256 MiB stretch of BF16 weights in device memory
        dict(name="encode 4096x32KiB", path="encode_batch", nstr=4096, plane=32768, values="exponent"),
        # one weight matrix, 117 MB, in 64 KiB chunks: a layer's weights decoded on demand from a compressed copy in HBM
        dict(name="tensor 4096x14336", path="archive", dtype="BF16", layers=0, hidden=4096, ffn=14336, kv=0, chunk=64 * KIB, checksum=True),
        # four decoder layers of an 8B model, 1.7 GB: the throughput case of the 64 KiB layout
        dict(name="4 layers", path="archive", dtype="BF16", layers=4, hidden=4096, ffn=14336, kv=1024, chunk=64 * KIB, checksum=True),
        # the same matrix in the reference's default layout: fourteen 8 MiB exponent-conditioned chunks
        dict(name="tensor, 8MiB chunks", path="archive", dtype="BF16", layers=0, hidden=4096, ffn=14336, kv=0, chunk=8 * MIB, checksum=True),
        # twelve encoder layers in FP32, 0.8 GB
        dict(name="12 layers FP32", path="archive", dtype="F32", layers=12, hidden=1024, ffn=4096, kv=1024, chunk=64 * KIB, checksum=True),
        # three checkpoints of a small model, the later two as differences against the first
        dict(name="delta chain", path="archive", dtype="BF16", delta=True, layers=12, hidden=768, ffn=3072, kv=768, chunk=64 * KIB, checksum=True),
        # loading a two-layer shard (0.87 GB) from the page cache
        dict(name="load 2 layers", path="load", dtype="BF16", layers=2, hidden=4096, ffn=14336, kv=1024, chunk=64 * KIB, checksum=True),
        # one layer's attention weights and norms out of that file
        dict(name="attention tensors", path="tensors", dtype="BF16", layers=2, hidden=4096, ffn=14336, kv=1024, chunk=64 * KIB, checksum=True),
        # saving one layer (0.44 GB)
        dict(name="save 1 layer", path="save", dtype="BF16", layers=1, hidden=4096, ffn=14336, kv=1024, chunk=64 * KIB),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def matrix(lo, hi):
        """Rows and columns of one tensor of about lo .. hi elements."""
        n = log(lo, hi)
        cols = log(63, 14336)
        return dict(layers=0, hidden=max(1, min(n // cols, hi // cols)), ffn=cols, kv=0)

    def model(most, dim):
        """A few layers of at most `most` elements in all, any width."""
        h = log(256, dim)
        c = dict(layers=rng.randint(1, 12), hidden=h, ffn=rng.randint(2 * h, int(3.5 * h)), kv=max(8, h // rng.choice((1, 4, 8))))
        per = 2 * h * h + 2 * c["kv"] * h + 3 * c["ffn"] * h + 2 * h
        c["layers"] = max(1, min(c["layers"], most // per))
        return c

    path = rng.choice(("host", "host", "device", "device", "encode", "archive", "archive", "f32", "default",
                       "delta", "load", "tensors", "save"))
    checksum = rng.random() < 0.8              # the reference's verify_checksums
    chunk = rng.choice((64, 64, 64, 256, 1024)) * KIB
    values = rng.choice(("exponent", "exponent", "skewed", "geometric", "zipf", "uniform"))
    if path == "host":
        plane = log(17, 64 * KIB)
        return dict(path="decode_batch", where="host", nstr=log(1, min(4096, 16 * MIB // plane)), plane=plane, values=values)
    if path == "device":
        plane = log(1 * KIB, 64 * KIB)
        return dict(path="decode_batch", where="device", nstr=log(1, min(28577, 892 * MIB // plane)), plane=plane, values=values)
    if path == "encode":
        plane = log(1 * KIB, 64 * KIB)
        return dict(path="encode_batch", nstr=log(1, min(16384, 128 * MIB // plane)), plane=plane, values=values)
    if path == "archive":
        return dict(path="archive", dtype="BF16", chunk=chunk, checksum=checksum,
                    **(model(870_000_000, 4096) if rng.random() < 0.6 else matrix(1 << 18, 58_000_000)))
    if path == "f32":
        return dict(path="archive", dtype="F32", chunk=64 * KIB, checksum=checksum,
                    **(model(190_000_000, 1024) if rng.random() < 0.6 else matrix(1 << 18, 30_000_000)))
    if path == "default":
        return dict(path="archive", dtype="BF16", chunk=8 * MIB, checksum=checksum, **matrix(1 << 20, 58_000_000))
    if path == "delta":
        return dict(path="archive", dtype="BF16", delta=True, chunk=64 * KIB, checksum=checksum, **model(110_000_000, 768))
    if path == "save":
        return dict(path="save", dtype="BF16", chunk=chunk, **model(218_000_000, 4096))
    return dict(path=path, dtype="BF16", chunk=64 * KIB, checksum=checksum, **model(436_000_000, 4096))


# ------------------------------------------------------------------------------- inputs

def _planes(case, gen):
    """nstr planes of `plane` bytes in device memory."""
    n, values = case["nstr"] * case["plane"], case["values"]

    def uniform():
        return torch.rand(n, generator=gen, device="cuda")

    if values == "exponent":                    # the exponent bytes of N(0, 0.02) BF16 weights
        w = (torch.randn(n, generator=gen, device="cuda") * 0.02).to(torch.bfloat16).view(torch.int16)
        out = (w.to(torch.int32) >> 7) & 0xFF
    elif values == "uniform":
        out = (uniform() * 256).to(torch.int32)
    elif values == "geometric":                 # p = 0.3
        out = torch.log(1 - uniform()).div_(math.log(0.7)).clamp_(0, 255).to(torch.int32)
    else:
        if values == "skewed":                  # a dominant value, sixteen rare ones, one between
            p = np.array([5.0] * 16 + [6.0, 170.0])
            symbols = np.array(list(range(16)) + [0x7F, 0x40])
        else:                                   # zipf, s = 1.1
            p, symbols = 1.0 / np.arange(1, 257) ** 1.1, np.arange(256)
        edges = torch.from_numpy(np.cumsum(p / p.sum())[:-1].astype(np.float32)).cuda()
        out = torch.from_numpy(symbols).cuda()[torch.bucketize(uniform(), edges)]
    return out.to(torch.uint8)


def _shapes(case):
    """[(tensor name, shape)] of one checkpoint file."""
    h, f, kv = case["hidden"], case["ffn"], case["kv"]
    if not case["layers"]:
        return [("weight", (h, f))]
    out = []
    for i in range(case["layers"]):
        for name, shape in (("self_attn.q_proj", (h, h)), ("self_attn.k_proj", (kv, h)), ("self_attn.v_proj", (kv, h)),
                            ("self_attn.o_proj", (h, h)), ("mlp.gate_proj", (f, h)), ("mlp.up_proj", (f, h)),
                            ("mlp.down_proj", (h, f)), ("input_layernorm", (h,)), ("post_attention_layernorm", (h,))):
            out.append((f"model.layers.{i}.{name}.weight", shape))
    return out


def _element(case):
    return 4 if case["dtype"] == "F32" else 2


def _elements(case):
    return sum(math.prod(s) for _n, s in _shapes(case))


def _checkpoint(case, gen, before=None):
    """One safetensors file as (header bytes, its data area on the GPU as uint8)."""
    es = _element(case)
    meta, pos = {}, 0
    for name, shape in _shapes(case):
        meta[name] = {"dtype": case["dtype"], "shape": list(shape), "data_offsets": [pos, pos + es * math.prod(shape)]}
        pos += es * math.prod(shape)
    head = json.dumps(meta, separators=(",", ":")).encode()
    head += b" " * (-(8 + len(head)) % 8)
    n = pos // es
    if before is None:
        w = torch.randn(n, generator=gen, device="cuda") * 0.02
        for m in meta.values():
            if len(m["shape"]) == 1:
                w[m["data_offsets"][0] // es:m["data_offsets"][1] // es] = 1.0
    else:                                       # 30 % of the elements moved a little
        moved = (torch.rand(n, generator=gen, device="cuda") < 0.3) * torch.randn(n, generator=gen, device="cuda") * 1e-4
        for m in meta.values():
            if len(m["shape"]) == 1:
                moved[m["data_offsets"][0] // es:m["data_offsets"][1] // es] = 0.0
        w = before.view(torch.bfloat16).float() + moved
    data = w if es == 4 else w.to(torch.bfloat16)
    return struct.pack("<Q", len(head)) + head, data.view(torch.uint8), meta


# ------------------------------------------------------------------------------ archives

class _Writer:
    """Chunks in file order, each a list of byte ranges of tensors on the GPU."""

    def __init__(self):
        self.pool, self.pool_bytes = [], 0
        self.pieces = []                        # (chunk numbers, places in the chunk, pool offsets, lengths)
        self.records = []                       # (chunk numbers, dst, rlen, crc, codec, esize, flags)
        self.nchunks = 0

    def put(self, t):
        """Offset of a tensor's bytes in the pool the pieces are cut from."""
        at = self.pool_bytes
        self.pool.append(t.reshape(-1).view(torch.uint8))
        self.pool_bytes += self.pool[-1].numel()
        return at

    def piece(self, chunks, place, offsets, lengths):
        chunks = np.asarray(chunks, dtype=np.int64)
        self.pieces.append(tuple(np.broadcast_to(np.asarray(v, dtype=np.int64), chunks.shape)
                                 for v in (chunks, place, offsets, lengths)))

    def record(self, chunks, *fields):
        chunks = np.asarray(chunks, dtype=np.int64)
        self.records.append(tuple(np.broadcast_to(np.asarray(v, dtype=np.int64), chunks.shape) for v in (chunks, *fields)))

    def stored(self, chunk, dst, raw, payload, codec, flags):
        at = self.put(torch.from_numpy(np.frombuffer(payload, dtype=np.uint8).copy()).cuda())
        self.piece([chunk], 0, at, len(payload))
        self.record([chunk], dst, len(raw), zlib.crc32(raw), codec, 1, flags)

    def finish(self, case, members):
        """The archive as one host array."""
        c, place, src, ln = (np.concatenate(col) for col in zip(*self.pieces))
        order = np.lexsort((place, c))
        c, src, ln = c[order], src[order], ln[order]
        at = np.cumsum(ln) - ln
        total = int(ln.sum())
        pool = torch.cat(self.pool)
        body = torch.empty(total, dtype=torch.uint8, device="cuda")
        step = 1 << 14                          # pieces gathered at a time
        for i in range(0, c.size, step):
            lo, hi = int(at[i]), int(at[min(i + step, c.size) - 1] + ln[min(i + step, c.size) - 1])
            shift = torch.from_numpy(src[i:i + step] - at[i:i + step]).cuda()
            idx = torch.repeat_interleave(shift, torch.from_numpy(np.ascontiguousarray(ln[i:i + step])).cuda())
            idx += torch.arange(lo, hi, device="cuda")
            body[lo:hi] = pool[idx]
        rec = np.zeros(self.nchunks, dtype=fmt.RECORD)
        chunks, dst, rlen, crc, codec, esize, flags = (np.concatenate(col) for col in zip(*self.records))
        for name, v in zip(("dst", "rlen", "crc", "codec", "esize", "flags"), (dst, rlen, crc, codec, esize, flags)):
            rec[name][chunks] = v
        rec["clen"] = np.bincount(c, weights=ln, minlength=self.nchunks).astype(np.int64)
        rec["off"] = fmt.HEADER.size + np.cumsum(rec["clen"].astype(np.int64)) - rec["clen"]
        size = sum(m["size"] for m in members)
        manifest = {"version": 1, "tool": "cases", "level": 1, "chunk_size": case["chunk"], "mapped": case["chunk"] == 64 * KIB,
                    "aligned": False, "entropy": "deflate", "checksum": "crc32", "total_size": size, "members": members,
                    "chunks": self.nchunks, "table_raw_len": int(rec.nbytes)}
        table = zlib.compress(rec.tobytes(), 1)
        man = zlib.compress(json.dumps(manifest, separators=(",", ":")).encode(), 1)
        off = fmt.HEADER.size + total
        blob = np.empty(off + len(table) + len(man) + fmt.FOOTER.size, dtype=np.uint8)
        flag = fmt.FLAG_PAGE_MAPPED if manifest["mapped"] else 0
        blob[:fmt.HEADER.size] = np.frombuffer(fmt.HEADER.pack(fmt.MAGIC, 6, flag, size, 0, 0), dtype=np.uint8)
        torch.from_numpy(blob[fmt.HEADER.size:off]).copy_(body)
        tail = table + man + fmt.FOOTER.pack(off, len(table), off + len(table), len(man), fmt.TAIL)
        blob[off:] = np.frombuffer(tail, dtype=np.uint8)
        return blob


def _keep(n):
    return np.maximum(1024, n >> 8)             # what a coded plane has to save


def _crcs(data, chunk):
    """crc32 of every `chunk` bytes of a CUDA tensor."""
    lib = gpu.library()
    host = np.zeros(lib.lmz_gpu_crc_tables(None, 0), dtype=np.uint8)
    lib.lmz_gpu_crc_tables(host.ctypes.data, host.size)
    tables = torch.from_numpy(host).cuda()
    meta = torch.zeros((-(-data.numel() // chunk), 4), dtype=torch.int32, device="cuda")
    rc = lib.lmz_gpu_crc32_chunks_dev(data.data_ptr(), data.numel(), chunk, tables.data_ptr(), meta.data_ptr(),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != gpu.OK:
        raise RuntimeError(gpu.last_error())
    return meta[:, 3].cpu().numpy().view(np.uint32)


def _split(data, es, n):
    """[chunks, planes, n] byte planes of [chunks, es * n] bytes."""
    if es == 4:
        return data.view(-1, n, 4).transpose(1, 2).contiguous()
    w = data.view(torch.int16).to(torch.int32)
    return torch.stack(((w >> 7) & 0xFF, ((w >> 8) & 0x80) | (w & 0x7F)), dim=1).to(torch.uint8)


def _code_plain(w, chunks, dst, crc, data, es, sources=None):
    """Chunks of one length ([m, bytes] on the GPU): byte planes, coded where that pays.  With
    `sources`, the bytes are differences against those places of the output."""
    m, size = data.shape
    n = size // es
    lead = 0 if sources is None else 1
    codec = fmt.CODEC_SPLIT if es == 4 else fmt.CODEC_BF16
    planes = _split(data, es, n)
    streams, offs = gpu.encode_batch(planes.reshape(-1), m * es, n)
    offs = offs.cpu().numpy().reshape(m, es, 2)
    coded = offs[:, :, 1] + _keep(n) < n
    lens = np.where(coded, offs[:, :, 1], n)
    split = coded.any(axis=1) & (lens.sum(axis=1) + 4 * es < size)
    at_streams, at_planes = w.put(streams), w.put(planes)
    at_heads = w.put(torch.from_numpy(np.ascontiguousarray(lens.astype("<u4")).view(np.uint8)).cuda())
    i = np.nonzero(split)[0]
    w.piece(chunks[i], lead, at_heads + i * 4 * es, 4 * es)
    for p in range(es):
        w.piece(chunks[i], lead + 1 + p, np.where(coded[i, p], at_streams + offs[i, p, 0], at_planes + (i * es + p) * n), lens[i, p])
    raw = np.nonzero(~split)[0]
    if raw.size:
        w.piece(chunks[raw], lead, w.put(data) + raw * size, size)
    inner = np.where(split, codec, fmt.CODEC_STORED)
    flags = np.where(split, (coded * (fmt.METHOD_RANS << (2 * np.arange(es)))).sum(axis=1), 0)
    if sources is None:
        w.record(chunks, dst, size, crc, inner, es, flags)
    else:
        head = np.zeros((m, 9), dtype=np.uint8)
        head[:, :8] = np.ascontiguousarray(sources.astype("<u8")).view(np.uint8).reshape(m, 8)
        head[:, 8] = inner
        w.piece(chunks, 0, w.put(torch.from_numpy(head).cuda()) + np.arange(m) * 9, 9)
        w.record(chunks, dst, size, crc, fmt.CODEC_DELTA, es, flags)


def _code_conditioned(w, chunk, dst, crc, data, stream):
    """One exponent-conditioned chunk; `stream` is its coded exponent plane."""
    exp, sm = _split(data.reshape(1, -1), 2, data.numel() // 2)[0]
    hist = torch.bincount(exp, minlength=256).cpu().numpy()
    lut, b, acc = np.zeros(256, dtype=np.int64), 0, 0
    for s in range(256):
        lut[s] = b
        acc += int(hist[s])
        while b + 1 < 8 and acc * 8 >= (b + 1) * exp.numel():
            b += 1
    bucket = torch.from_numpy(lut).cuda()[exp.long()]
    part = sm[torch.argsort(bucket, stable=True)]
    methods, lens, pos = [], [], 0
    for j, cnt in enumerate(torch.bincount(bucket, minlength=8).tolist()):
        seg, method = part[pos:pos + cnt], fmt.METHOD_STORED
        if cnt:
            p = torch.bincount(seg, minlength=256).double() / cnt
            bits = float(-(p * torch.log2(p.clamp_min(1e-12))).sum())
            if cnt * bits / 8 + 548 + int(_keep(cnt)) < cnt:
                seg, method = gpu.encode_batch(seg, 1, cnt)[0], fmt.METHOD_RANS
            w.piece([chunk], 2 + j, w.put(seg), seg.numel())
        methods.append(method)
        lens.append(int(seg.numel()))
        pos += cnt
    head = struct.pack("<BB8BI8I", 8, fmt.METHOD_RANS, *methods, stream.numel(), *lens)
    w.piece([chunk], 0, w.put(torch.from_numpy(np.frombuffer(head, dtype=np.uint8).copy()).cuda()), len(head))
    w.piece([chunk], 1, w.put(stream), stream.numel())
    w.record([chunk], dst, data.numel(), crc, fmt.CODEC_BF16C, 2, 0)


def _regions(meta, start, delta):
    """Runs of a file's data area that are coded alike: (first byte, last, as a difference)."""
    runs = []
    for m in meta.values():
        lo, hi = m["data_offsets"]
        d = delta and hi - lo >= SMALL_TENSOR
        if runs and runs[-1][2] == d:
            runs[-1][1] = hi
        else:
            runs.append([lo, hi, d])
    return runs


def _archive(case, seed):
    """An archive of the case's checkpoint (or chain of them), as one host array."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    es, chunk = _element(case), case["chunk"]
    w, members, base, first, before = _Writer(), [], 0, None, None
    for k in range(CHAIN if case.get("delta") else 1):
        head, data, meta = _checkpoint(case, gen, before)
        for lo in range(0, len(head), chunk):
            raw = head[lo:lo + chunk]
            packed = zlib.compress(raw, 1)
            plain = len(packed) > len(raw) - (len(raw) >> 5) or len(packed) + _keep(len(raw)) >= len(raw)
            w.stored(w.nchunks, base + lo, raw, raw if plain else packed,
                     fmt.CODEC_STORED if plain else fmt.CODEC_ZSTD, 0 if plain else fmt.METHOD_DEFLATE)
            w.nchunks += 1
        for lo, hi, as_delta in _regions(meta, len(head), k > 0):
            crc = _crcs(data[lo:hi], chunk)
            coded = data[lo:hi] ^ first[lo:hi] if as_delta else data[lo:hi]
            nfull, tail = divmod(hi - lo, chunk)
            dst = base + len(head) + lo + np.arange(nfull + 1) * chunk
            src = base0 + lo + np.arange(nfull + 1) * chunk if as_delta else None
            for a, b, size in ((0, nfull, chunk), (nfull, nfull + 1, tail)):
                if a == b or not size:
                    continue
                rows = coded[a * chunk:a * chunk + (b - a) * size].view(b - a, size)
                ids = w.nchunks + np.arange(b - a)
                if es == 2 and size // 2 >= COND_ELEMENTS and not as_delta:
                    exps = _split(rows, 2, size // 2)[:, 0].contiguous()
                    streams, offs = gpu.encode_batch(exps.reshape(-1), b - a, size // 2)
                    for i, (at, ln) in enumerate(offs.view(-1, 2).tolist()):
                        _code_conditioned(w, int(ids[i]), int(dst[a + i]), int(crc[a + i]), rows[i], streams[at:at + ln])
                else:
                    _code_plain(w, ids, dst[a:b], crc[a:b].astype(np.int64), rows, es, None if src is None else src[a:b])
                w.nchunks += b - a
        members.append({"path": f"model-{k}.safetensors" if k else "model.safetensors", "size": len(head) + data.numel(), "dst": base,
                        "kind": "safetensors", "mode": 0o644, "crc": 0,
                        "tensors": {n: {"dtype": m["dtype"], "shape": m["shape"],
                                        "offsets": [len(head) + m["data_offsets"][0], len(head) + m["data_offsets"][1]]}
                                    for n, m in meta.items()}})
        if k == 0:
            first, base0 = data, base + len(head)
        before = data
        base += len(head) + data.numel()
    return w.finish(case, members)


# --------------------------------------------------------------------------- prepare, run

class _Files:
    """A folder of a state's own, in memory where there is room; gone with the state."""

    def __init__(self, need):
        shm = "/dev/shm"
        where = shm if os.path.isdir(shm) and shutil.disk_usage(shm).free > 8 * need else None
        self.folder = tempfile.mkdtemp(prefix="lmz_cases_", dir=where)
        weakref.finalize(self, shutil.rmtree, self.folder, True)

    def path(self, name):
        return os.path.join(self.folder, name)


def prepare(case, seed):
    path = case["path"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st = {"case": case}
    if path in ("decode_batch", "encode_batch"):
        planes = _planes(case, gen)
        if path == "encode_batch":
            room = planes.numel() + case["nstr"] * 1024
            return dict(st, planes=planes, packed=torch.zeros(room, dtype=torch.uint8, device="cuda"))
        streams, offsets = gpu.encode_batch(planes, case["nstr"], case["plane"])
        if case["where"] == "host":
            streams, offsets = streams.cpu().numpy().tobytes(), offsets.cpu().numpy().astype("<u8").tobytes()
        return dict(st, streams=streams, offsets=offsets)
    if path == "save":
        head, data, _meta = _checkpoint(case, gen)
        member = torch.cat((torch.from_numpy(np.frombuffer(head, dtype=np.uint8).copy()).cuda(), data))
        files = _Files(member.numel())
        return dict(st, member=member, files=files, to=files.path("saved.lmz"))
    blob = _archive(case, seed)
    torch.cuda.empty_cache()
    if path == "archive":
        return dict(st, decoder=decode.ArchiveDecoder(blob, checksum=case["checksum"]))
    files = _Files(blob.size)
    blob.tofile(files.path("model.lmz"))
    last = case["layers"] - 1
    names = [n for n, s in _shapes(case) if n.startswith(f"model.layers.{last}.") and ("self_attn" in n or "layernorm" in n)]
    return dict(st, files=files, file=files.path("model.lmz"), names=names)


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "decode_batch":
        out = gpu.decode_batch(state["streams"], state["offsets"], case["nstr"], case["plane"])
        return np.frombuffer(out, dtype=np.uint8) if case["where"] == "host" else out
    if path == "encode_batch":
        # (how many bytes come out depends on the values: they go to a buffer of one size, the program's own)
        streams, offsets = gpu.encode_batch(state["planes"], case["nstr"], case["plane"])
        state["packed"][:streams.numel()].copy_(streams)
        return {"streams": state["packed"], "offsets": offsets}
    if path == "archive":
        out = state["decoder"].run()
        state["decoder"].check()
        return out
    if path == "load":
        return decode.load_archive(state["file"], checksum=case["checksum"])
    if path == "tensors":
        got = decode.decode_tensors(state["file"], state["names"], checksum=case["checksum"])
        return {key[1]: t for key, t in got.items()}
    size = save.save_archive(state["to"], [("model.safetensors", state["member"])], chunk_size=case["chunk"])
    # (a file's length depends on the values: all get one length, by a hole at the end, and come back as a mapping)
    os.truncate(state["to"], state["member"].numel() + MIB)
    return {"size": size, "file": np.memmap(state["to"], dtype=np.uint8, mode="r")}


# Bits a value of each distribution takes when coded, for work().
_BITS = {"exponent": 2.68, "skewed": 2.0, "geometric": 2.94, "zipf": 6.4, "uniform": 8.0}


def work(case):
    """Coded bytes and plain bytes, each once (and a delta's base once more); no floating-point work."""
    if "nstr" in case:
        plain = case["nstr"] * case["plane"]
        coded = case["nstr"] * 548 + plain * _BITS[case["values"]] / 8
        return {"bytes": plain + coded, "flops": 0}
    plain = _elements(case) * _element(case)
    coded = plain * {2: 0.666, 4: 0.84}[_element(case)]
    if case.get("delta"):
        return {"bytes": plain + coded + 2 * (plain * 1.7 + plain), "flops": 0}
    if case["path"] == "tensors":
        h, kv = case["hidden"], case["kv"]
        plain = 2 * (2 * h * h + 2 * kv * h + 2 * h)
        coded = plain * 0.666
    return {"bytes": plain + coded, "flops": 0}


def tolerance(case):
    return "exact"                              # bytes in, bytes out
