"""Write an lmz archive from bytes that are already in HBM.

The reference compresses on the CPU only (lmz/api.py:651-815 `compress`,
lmz/codec.py:914-1009 `encode_chunk`); this is the same work for the layout the GPU path is
quoted on -- BF16 safetensors members cut into small chunks (`lmz compress --mapped`, or any
chunk size below 2 MiB; from there up the reference conditions the sign/mantissa plane on
the exponent, lmz/codec.py:955-969, which this writer does not do) -- with the per-chunk
work on the device:

    split every chunk into its exponent and sign/mantissa planes   lmz/native/lmzcore.c:430-437
    rANS-code every plane with its own histogram                   lmzcore.c:882-979, 1318-1383
    keep a coded plane only where it pays                          lmz/codec.py:385-393, 396-398
    frame the chunk: plane lengths, then the planes                lmz/codec.py:989-1003
    crc32 of the chunk's plaintext                                 lmz/codec.py:931

and the container (records, manifest, footer; lmz/format.py:279-322) and the few bytes of
safetensors header on the host.  The chunk bytes are the reference encoder's: its early
exits for a hopeless plane (a sampled entropy estimate and a cost estimate from the
histogram, lmz/codec.py:356-372) only predict the comparison that is made here on the real
coded length, and for planes of at most 196 608 bytes -- where its sample is the whole
plane -- they never disagree with it.
"""
from __future__ import annotations

import ctypes
import json
import os
import stat
import struct
import zlib

import numpy as np

from . import archive as fmt, gpu

MIN_GAIN_FLOOR = 1024            # lmz/codec.py:396-398: a coded stream must save max(1024, n >> 8) bytes
COND_MIN_BYTES = 2 << 20         # chunks of a mebi-element or more are exponent-conditioned by the reference
BATCH_BYTES = 64 << 20           # BF16 bytes framed per round of kernel launches: small enough that the first
                                 # round is on its way to the file early, the others are coded under its writing
IN_FLIGHT = 4                    # rounds whose payload may be on its way to the file


def _safetensors_layout(head: bytes):
    """(data start, {name: {dtype, shape, offsets}}) of a safetensors file from its first bytes
    (lmz/planner.py:196-237)."""
    if len(head) < 8:
        raise ValueError("not a safetensors file")
    n = struct.unpack_from("<Q", head, 0)[0]
    if n > len(head) - 8:
        raise ValueError("the safetensors header is longer than the bytes given")
    meta = json.loads(bytes(head[8:8 + n]).decode("utf-8"))
    tensors = {k: {"dtype": v["dtype"], "shape": list(v["shape"]),
                   "offsets": [8 + n + v["data_offsets"][0], 8 + n + v["data_offsets"][1]]}
               for k, v in meta.items() if k != "__metadata__"}
    return 8 + n, tensors


def _header_chunk(raw: bytes, level: int = 1):
    """(payload, codec, flags) of a run of container bytes, as the reference codes them when it
    has no zstd (lmz/codec.py:1005-1009 over _encode_stream :373-393): deflate where that saves
    max(1024, n >> 8) bytes, else stored."""
    n = len(raw)
    best = zlib.compress(raw, min(max(level, 1), 9))
    if len(best) > n - (n >> 5) or len(best) + max(MIN_GAIN_FLOOR, n >> 8) >= n:
        return raw, fmt.CODEC_STORED, 0
    return best, fmt.CODEC_ZSTD, fmt.METHOD_DEFLATE


def save_archive(path, members, chunk_size: int = 64 << 10, mapped: bool = True, stats=None):
    """Write `members` = [(member path, CUDA uint8 tensor holding a BF16 safetensors file)] as
    an lmz archive.  Every tensor must be BF16.  Returns the number of bytes written.
    `stats`, a dict, receives `device_s` (the kernels: split + encode + frame + checksum, timed
    with CUDA events) and `payload_bytes`.  The framed payload leaves the device in batches, through
    the page-locked blocks and the threads that loads use (csrc/host_io.inl); what bounds a save is
    the file system's side of that.  An existing file is overwritten in place and cut to length."""
    if chunk_size < (64 << 10) or chunk_size >= COND_MIN_BYTES or chunk_size % 2:
        raise ValueError("chunk_size must be even, at least 64 KiB and below 2 MiB")
    try:
        fd = os.open(path, os.O_RDWR | os.O_CREAT, 0o666)
    except PermissionError:                                  # a file that may be written only: no mapping, then
        fd = os.open(path, os.O_WRONLY | os.O_CREAT, 0o666)
    try:
        # whatever ends this save early, down to the end of the process, must not leave a file that opens:
        # an archive that is overwritten loses its header first, and gets the new one last
        _put(fd, bytes(fmt.HEADER.size), 0)
        try:
            return _write_archive(fd, members, chunk_size, mapped, stats)
        except BaseException:
            _cut(fd, 0)
            raise
    finally:
        os.close(fd)


def _cut(fd, size: int) -> None:
    """Make a file `size` bytes long; a device (os.devnull) has no length."""
    if stat.S_ISREG(os.fstat(fd).st_mode):
        os.ftruncate(fd, size)


class _FileWriter:
    """Device memory -> a file, in the background, from one position to the next.  On a memory-backed
    file system the bytes are stored through a mapping by all threads at once, elsewhere written."""

    def __init__(self, lib, fd, device):
        import torch
        from . import decode
        self.lib, self.fd, self.device = lib, fd, device
        self.stream = torch.cuda.current_stream(device).cuda_stream
        with torch.cuda.device(device):
            self.handle = lib.lmz_gpu_transfer_new(decode.Staging.shared().handle, self.stream)
        if not self.handle:
            raise RuntimeError(gpu.last_error())
        self.pending = []

    def send(self, data, pos: int) -> None:
        import torch
        n = int(data.numel())
        if not n:
            return
        lead = pos & 4095
        at = self.lib.lmz_host_map_file(self.fd, pos - lead, n + lead)
        with torch.cuda.device(self.device):
            r = self.lib.lmz_gpu_transfer_download(self.handle, data.data_ptr(), n, self.fd, at, lead if at else pos, self.stream)
        if r < 0:
            if at:
                self.lib.lmz_host_unmap_file(at, n + lead)
            raise RuntimeError(gpu.last_error())
        self.pending.append((r, data, at, n + lead))
        while len(self.pending) > IN_FLIGHT:
            self._first_done()

    def _first_done(self):
        r, _data, at, n = self.pending.pop(0)
        rc = self.lib.lmz_gpu_transfer_wait(self.handle, r, self.stream)
        if at:
            self.lib.lmz_host_unmap_file(at, n)
        if rc != gpu.OK:
            raise OSError(f"writing the archive failed: {gpu.last_error()}")

    def close(self):
        try:
            while self.pending:
                self._first_done()
        finally:
            handle, self.handle = self.handle, None
            if handle:
                self.lib.lmz_gpu_transfer_free(handle)          # (waits for whatever is still under way)
            for _r, _data, at, n in self.pending:
                if at:
                    self.lib.lmz_host_unmap_file(at, n)


def _put(fd, data: bytes, pos: int) -> int:
    view = memoryview(data)
    while view.nbytes:
        n = os.pwrite(fd, view, pos)
        view, pos = view[n:], pos + n
    return pos


def _write_archive(fd, members, chunk_size, mapped, stats):
    import torch
    lib = gpu.library()
    recs_parts, metas, base = [], [], 0                      # record arrays, in file order
    timed, pos = [], fmt.HEADER.size                         # the header goes in last: it holds the total size
    writers = {}

    def add_records(dst, rlen, crc, codec, esize, flags, clen):
        part = np.zeros(len(dst), dtype=fmt.RECORD)
        part["dst"], part["rlen"], part["crc"], part["codec"] = dst, rlen, crc, codec
        part["esize"], part["flags"], part["clen"] = esize, flags, clen
        recs_parts.append(part)

    try:
        for mpath, data in members:
            if not (type(data).__module__.startswith("torch") and data.is_cuda and data.dtype == torch.uint8):
                raise ValueError("a member must be a CUDA uint8 tensor")
            flat = data.reshape(-1).contiguous()
            size = int(flat.numel())
            head = bytes(flat[:min(size, 8)].cpu().numpy())
            hlen = struct.unpack("<Q", head)[0] if len(head) == 8 else 0
            head = bytes(flat[:min(size, 8 + hlen)].cpu().numpy())
            start, tensors = _safetensors_layout(head)
            if any(t["dtype"] != "BF16" for t in tensors.values()):
                raise ValueError("this writer takes BF16 members only")
            if (size - start) % 2:
                raise ValueError("a BF16 data area has an odd number of bytes")
            # the header: byte chunks of at most chunk_size (lmz/planner.py:582-652)
            for s in range(0, start, chunk_size):
                raw = head[s:min(s + chunk_size, start)]
                payload, codec, flags = _header_chunk(raw)
                add_records([base + s], [len(raw)], [zlib.crc32(raw) & 0xFFFFFFFF], [codec], [1], [flags], [len(payload)])
                pos = _put(fd, payload, pos)
            # the data area: BF16 chunks, framed on the device
            body = flat[start:]
            nbytes = int(body.numel())
            # (in batches: the coder's slots take a little over twice the bytes they code)
            batch = max(1, BATCH_BYTES // chunk_size) * chunk_size
            if data.device not in writers:
                writers[data.device] = _FileWriter(lib, fd, data.device)
            for b0 in range(0, nbytes, batch):
                part = body[b0:min(b0 + batch, nbytes)]
                payload, clen, codec, flags, crc, events = _frame_bf16(lib, part, chunk_size)
                timed.append(events)
                at = np.arange(clen.size, dtype=np.int64) * chunk_size
                add_records(base + start + b0 + at, np.minimum(chunk_size, int(part.numel()) - at), crc, codec,
                            np.full(clen.size, 2), flags, clen)
                writers[data.device].send(payload, pos)           # the chunks' payloads back to back, in record order
                pos += int(payload.numel())
            metas.append({"path": mpath, "size": size, "dst": base, "kind": "safetensors", "mode": 0o644, "crc": 0,
                          "tensors": {k: dict(v) for k, v in tensors.items()}})
            base += size
        recs = np.concatenate(recs_parts) if recs_parts else np.zeros(0, dtype=fmt.RECORD)
        clens = recs["clen"].astype(np.int64)
        recs["off"] = fmt.HEADER.size + np.cumsum(clens) - clens
        off = fmt.HEADER.size + int(clens.sum())
        manifest = {"version": 1, "tool": "lmz-b200 device writer", "level": 1, "chunk_size": chunk_size,
                    "mapped": bool(mapped), "aligned": False, "entropy": "deflate", "checksum": "crc32",
                    "total_size": base, "members": metas, "chunks": int(recs.size), "table_raw_len": int(recs.nbytes)}
        table_c = zlib.compress(recs.tobytes(), 3)
        man_c = zlib.compress(json.dumps(manifest, separators=(",", ":")).encode(), 3)
        end = _put(fd, table_c + man_c + fmt.FOOTER.pack(off, len(table_c), off + len(table_c), len(man_c), fmt.TAIL), off)
    finally:
        errors = []
        for w in writers.values():
            try:
                w.close()
            except Exception as exc:
                errors.append(exc)
    if errors:
        raise errors[0]
    _cut(fd, end)                                            # (the end of a longer file before is a footer, too)
    _put(fd, fmt.HEADER.pack(fmt.MAGIC, 6, fmt.FLAG_PAGE_MAPPED if mapped else 0, base, 0, 0), 0)
    if stats is not None:
        stats.update(device_s=sum(e0.elapsed_time(e1) + e2.elapsed_time(e3) for e0, e1, e2, e3 in timed) / 1e3,
                     payload_bytes=off - fmt.HEADER.size)
    return end


def _frame_bf16(lib, body, chunk_size: int):
    """Chunk payloads of one BF16 data area, on the device: the payload bytes of all chunks back to
    back (a device tensor, written by work on the current stream), per chunk its length, codec id,
    flags and crc32 (host arrays), and the events around the two stretches of kernels."""
    import torch
    dev = body.device
    nbytes = int(body.numel())
    nfull, tail = divmod(nbytes, chunk_size)
    nchunks = nfull + (1 if tail else 0)
    with torch.cuda.device(dev):
        cs = torch.cuda.current_stream(dev).cuda_stream
        e0, e1, e2, e3 = (torch.cuda.Event(enable_timing=True) for _ in range(4))
        e0.record()
        planes = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        lens = torch.zeros(2 * nchunks, dtype=torch.int32, device=dev)
        rc = lib.lmz_gpu_split_bf16_dev(body.data_ptr(), nbytes, chunk_size, planes.data_ptr(), cs)
        if rc != gpu.OK:
            raise RuntimeError(f"plane split failed ({rc}): {gpu.last_error()}")
        # every plane is coded; which coded planes are kept is decided on their lengths
        slot = lib.lmz_gpu_encode_slot_bytes(chunk_size // 2)
        slot_tail = lib.lmz_gpu_encode_slot_bytes(tail // 2) if tail else 0
        slots = torch.empty(2 * nfull * slot + 2 * slot_tail + 512, dtype=torch.uint8, device=dev)
        sbase = (slots.data_ptr() + 511) & ~511
        if nfull:
            rc = lib.lmz_gpu_encode_batch_dev(planes.data_ptr(), 2 * nfull, chunk_size // 2, sbase,
                                              lens.data_ptr(), cs)
        if rc == gpu.OK and tail:
            rc = lib.lmz_gpu_encode_batch_dev(planes.data_ptr() + nfull * chunk_size, 2, tail // 2,
                                              sbase + 2 * nfull * slot, lens.data_ptr() + 8 * nfull, cs)
        if rc != gpu.OK:
            raise RuntimeError(f"plane encode failed ({rc}): {gpu.last_error()}")
        meta = torch.zeros((nchunks, 4), dtype=torch.int32, device=dev)          # clen, codec, flags, crc
        rc = lib.lmz_gpu_frame_bf16_dev(body.data_ptr(), nbytes, chunk_size, lens.data_ptr(), meta.data_ptr(),
                                        None, None, None, None, cs)              # pass 1: sizes and choices
        if rc != gpu.OK:
            raise RuntimeError(f"chunk framing failed ({rc}): {gpu.last_error()}")
        from . import decode
        tabs = decode._crc_tables(lib, dev)
        rc = lib.lmz_gpu_crc32_chunks_dev(body.data_ptr(), nbytes, chunk_size, tabs.data_ptr(),
                                          meta.data_ptr(), cs)
        if rc != gpu.OK:
            raise RuntimeError(f"chunk checksum failed ({rc}): {gpu.last_error()}")
        clen = meta[:, 0].to(torch.int64)
        offs = (torch.cumsum(clen, 0) - clen).contiguous()
        e1.record()
        m = meta.cpu().numpy()                                                   # (the host needs the sizes: a sync)
        total = int(m[:, 0].astype(np.int64).sum())
        out = torch.empty(total + 16, dtype=torch.uint8, device=dev)
        e2.record()
        rc = lib.lmz_gpu_frame_bf16_dev(body.data_ptr(), nbytes, chunk_size, lens.data_ptr(), meta.data_ptr(),
                                        planes.data_ptr(), ctypes.c_void_p(sbase), offs.data_ptr(),
                                        out.data_ptr(), cs)                      # pass 2: the bytes
        if rc != gpu.OK:
            raise RuntimeError(f"chunk framing failed ({rc}): {gpu.last_error()}")
        e3.record()
        return (out[:total], m[:, 0].astype(np.int64), m[:, 1], m[:, 2],
                m[:, 3].astype(np.int64) & 0xFFFFFFFF, (e0, e1, e2, e3))
