"""Whole-archive decode on one GPU.

The reference decodes an archive on CPU threads (lmz/api.py:889-975
`decompress`, :1061-1143 `verify`); this is the same job on the device: the
archive's payload is uploaded once, `ArchiveDecoder.run()` decodes every chunk
into one device buffer laid out like the reference's concatenated output space
(members end to end, lmz/format.py:17-19), and per-chunk crc32 verdicts come
back with it.  PyTorch only owns the device buffers and the stream.
"""
from __future__ import annotations

import ctypes

import numpy as np

from . import _chunks, archive as fmt, gpu, plan as planner
from .archive import CorruptArchive

_ST_NAMES = {1: "bad stream header", 2: "truncated stream",
             4: "lengths disagree with the record", 5: "checksum mismatch"}

_TORCH_DTYPES = {"BF16": "bfloat16", "F16": "float16", "F32": "float32", "F64": "float64",
                 "I8": "int8", "U8": "uint8", "I16": "int16", "I32": "int32", "I64": "int64",
                 "BOOL": "bool"}


class _Arena:
    """Many small device arrays in two allocations: job arrays, which come over in one copy from one
    page-locked block, and work arrays, cleared by one memset."""

    def __init__(self, lib, device):
        self.lib, self.device = lib, device
        self.jobs, self.work = {}, {}
        self.host = self.copied = None

    def job(self, name, arr):
        self.jobs[name] = np.ascontiguousarray(arr).view(np.uint8).reshape(-1)

    def words(self, name, count, kind="int32"):
        self.work[name] = (max(1, int(count)), kind)

    def place(self):
        """{name: tensor} of everything asked for."""
        import torch
        out, at = {}, 0
        spans = {}
        for name, a in self.jobs.items():
            spans[name] = at
            at += (a.size + 255) & ~255
        self.host = gpu.result_memory(self.lib, max(at, 1))
        for name, a in self.jobs.items():
            self.host[spans[name]:spans[name] + a.size] = a
        work = {}
        total = 0
        size = {"int32": 4, "int16": 2, "uint8": 1}
        for name, (count, kind) in self.work.items():
            work[name] = total
            total += (count * size[kind] + 255) & ~255
        dev = torch.empty(max(at, 1) + total, dtype=torch.uint8, device=self.device)
        dev[:at].copy_(torch.from_numpy(self.host[:at]), non_blocking=True)
        self.copied = torch.cuda.Event()
        self.copied.record(torch.cuda.current_stream(self.device))
        dev[at:].zero_()
        for name, a in self.jobs.items():
            out[name] = dev[spans[name]:spans[name] + a.size]
        for name, (count, kind) in self.work.items():
            lo = at + work[name]
            out[name] = dev[lo:lo + count * size[kind]].view(getattr(torch, kind))
        return out

    def arrived(self):
        """Let the host block go, when the copy out of it has ended: whoever gets it next writes to it at
        once, and a decode that is already queued would run on what they write."""
        if self.copied is not None:
            self.copied.synchronize()
        self.host = self.copied = None

    def __del__(self):
        self.arrived()


_tables = {}


def _crc_tables(lib, device):
    """The CRC tables, uploaded once per device."""
    import torch
    key = str(device)
    if key not in _tables:
        n = lib.lmz_gpu_crc_tables(None, 0)
        host = np.zeros(n, dtype=np.uint8)
        lib.lmz_gpu_crc_tables(host.ctypes.data, n)
        _tables[key] = torch.from_numpy(host).to(device)
    return _tables[key]


def _check_layouts(lib):
    """The library's job layouts are the planner's (asked once of each)."""
    if getattr(lib, "layouts_checked", False):
        return
    sizes = (ctypes.c_uint * 5)()
    lib.lmz_gpu_struct_sizes(ctypes.byref(sizes))
    want = (planner.STREAM_JOB.itemsize, planner.CHUNK_JOB.itemsize,
            planner.COND_JOB.itemsize, planner.COND_STATE_BYTES, planner.FUSED_JOB.itemsize)
    if tuple(sizes) != want or lib.lmz_gpu_piece_bytes() != planner.PIECE or \
            lib.lmz_gpu_shared_group() != planner.T_GROUP or \
            lib.lmz_gpu_delta_job_bytes() != planner.DELTA_JOB.itemsize:
        raise RuntimeError("the CUDA library and the planner disagree on job layouts")
    lib.layouts_checked = True


def _payload_source(ar, plan):
    """(bytes, where the plan's payload starts in them): the archive's own, where the payload is a view of
    them and so may be read from its file; the payload itself where the plan was made of another
    mapping or copy of the archive."""
    lo = plan.payload.ctypes.data - ar.blob.ctypes.data
    if 0 <= lo <= ar.blob.size - plan.payload.size:
        return ar.blob, lo
    return np.ascontiguousarray(plan.payload).view(np.ndarray), 0


class ArchiveDecoder:
    """An archive planned and resident on `device`, ready to decode repeatedly.

    `ar` is an `archive.Archive`, a path, or the archive's bytes.  With
    `checksum=False` the per-chunk crc32 is skipped (the reference's
    `verify_checksums=False`).  `payload` may be given as a CUDA uint8 tensor with room
    for `plan.payload`, the plan's host-inflated header chunks and `gpu.pad_bytes()` of
    slack; the caller then brings the payload bytes there itself (`upload`, or copies of
    its own) before `run`.  With `settle=False` the job arrays may still be on their way when the
    constructor returns: `run` must then be on the stream that was current here."""

    def __init__(self, ar, device=None, checksum: bool = True, out=None, plan=None,
                 fuse=True, payload=None, *, settle: bool = True):
        import torch

        lib = gpu.library()
        self.lib = lib
        _check_layouts(lib)
        self.archive = ar if isinstance(ar, fmt.Archive) else fmt.Archive(ar)
        self.plan = p = plan if plan is not None else planner.build_plan(self.archive, fuse=fuse)
        self.device = torch.device(device if device is not None else
                                   f"cuda:{torch.cuda.current_device()}")
        self.checksum = checksum
        d = self.device
        with torch.cuda.device(d):
            pad = gpu.pad_bytes()
            nbytes = p.extras_pos + p.extras.size
            if payload is not None and payload.numel() < nbytes + pad:
                raise ValueError("the payload buffer is smaller than the plan's payload, header chunks and slack")
            self.d_payload = payload if payload is not None else \
                torch.empty(nbytes + pad, dtype=torch.uint8, device=d)
            self.h2d_bytes = int(p.payload.size + p.extras.size)
            self.d_payload[nbytes:nbytes + pad].zero_()
            up = self._start_upload() if payload is None else None      # under the rest of this
            self.d_scratch = torch.empty(max(p.scratch_bytes, 64), dtype=torch.uint8, device=d)
            self.d_out = out if out is not None else \
                torch.empty(p.total + 64, dtype=torch.uint8, device=d)
            if self.d_out.numel() < p.total + 64:
                raise ValueError("the output buffer needs total + 64 bytes")
            ncond, nchunks, npieces = p.cond_jobs.size, p.chunks.size, p.n_pieces
            self._arena = a = _Arena(lib, d)
            for name in ("stream_jobs", "seg_jobs", "fused_jobs", "delta_jobs", "chunks", "piece_chunk",
                         "cond_jobs", "cond_pieces", "extras"):
                a.job("d_" + name, getattr(p, name))
            if p.n_fused_t:
                a.job("d_tables", p.tables)
            a.words("d_cond_state", ncond * planner.COND_STATE_BYTES, "uint8")
            for name, count in (("hist", ncond * 256), ("piece_cnt", npieces * 16 if ncond else 1), ("piece_crc", npieces),
                                ("stream_status", p.stream_jobs.size), ("seg_status", p.seg_jobs.size),
                                ("fused_status", p.fused_jobs.size), ("delta_status", 2 * p.delta_jobs.size),
                                ("delta_order", p.delta_jobs.size + 4), ("chunk_status", nchunks), ("chunk_crc", nchunks),
                                ("any_bad", 1), ("fused_order", p.n_fused + 4)):
                a.words("d_" + name, count)
            a.words("d_piece_wcnt", npieces * 64 if ncond else 1, "int16")
            self.d_tables = None
            for name, t in a.place().items():
                setattr(self, name, t)
            if not p.device_classify:
                self.d_fused_order = None
            if p.extras.size:
                self.d_payload[p.extras_pos:nbytes].copy_(self.d_extras)
            self.d_piece_lcnt = torch.empty(max(1, p.cond_pieces.size * 2048), dtype=torch.int32, device=d)
            self.d_tabs = _crc_tables(lib, d)
            if up is not None:
                self._finish_upload(up)
            if settle:
                torch.cuda.current_stream(d).synchronize()
                self._arena.arrived()
        c = _chunks.DecodePlan()
        c.d_payload, c.d_scratch = self.d_payload.data_ptr(), self.d_scratch.data_ptr()
        c.d_out = self.d_out.data_ptr()
        c.d_stream_jobs, c.d_seg_jobs = self.d_stream_jobs.data_ptr(), self.d_seg_jobs.data_ptr()
        c.d_stream_status, c.d_seg_status = self.d_stream_status.data_ptr(), self.d_seg_status.data_ptr()
        c.d_fused_jobs, c.d_fused_status = self.d_fused_jobs.data_ptr(), self.d_fused_status.data_ptr()
        c.n_fused, c.n_fused_t = p.n_fused, p.n_fused_t
        c.d_delta_jobs, c.d_delta_status = self.d_delta_jobs.data_ptr(), self.d_delta_status.data_ptr()
        c.n_delta, c.n_delta_plain = p.delta_jobs.size, p.n_delta_plain
        c.d_delta_order = self.d_delta_order.data_ptr()
        c.d_tables = self.d_tables.data_ptr() if self.d_tables is not None else None
        c.n_fused_small = p.n_fused_small
        c.n_fused_f32, c.n_fused_f32_small = p.n_fused_f32, p.n_fused_f32_small
        c.d_chunks, c.d_piece_chunk = self.d_chunks.data_ptr(), self.d_piece_chunk.data_ptr()
        c.d_cond_jobs, c.d_cond_state = self.d_cond_jobs.data_ptr(), self.d_cond_state.data_ptr()
        c.d_cond_pieces = self.d_cond_pieces.data_ptr()
        c.d_hist, c.d_piece_cnt = self.d_hist.data_ptr(), self.d_piece_cnt.data_ptr()
        c.d_piece_wcnt = self.d_piece_wcnt.data_ptr()
        c.d_piece_lcnt = self.d_piece_lcnt.data_ptr()
        c.d_piece_crc = self.d_piece_crc.data_ptr() if checksum else None
        c.d_crc_tables = self.d_tabs.data_ptr()
        c.d_chunk_status, c.d_chunk_crc = self.d_chunk_status.data_ptr(), self.d_chunk_crc.data_ptr()
        c.d_any_bad = self.d_any_bad.data_ptr()
        c.d_fused_order = self.d_fused_order.data_ptr() if self.d_fused_order is not None else None
        c.n_stream_jobs, c.n_seg_jobs = p.stream_jobs.size, p.seg_jobs.size
        c.n_chunks, c.n_pieces = p.chunks.size, p.n_pieces
        c.n_cond, c.n_cond_pieces = ncond, p.cond_pieces.size
        for i in range(6):
            c.piece_split[i] = int(p.piece_split[i])
        self._c = c
        self.launches_per_run = 0            # kernels launched by one run(); known after the first

    def upload(self, pinned=None, non_blocking: bool = False):
        """Copy the archive's payload region host -> device (from `pinned`, a host
        uint8 tensor of `plan.payload.size` bytes, if given)."""
        import torch
        n = self.plan.payload.size
        if pinned is not None:
            self.d_payload[:n].copy_(pinned, non_blocking=non_blocking)
            return
        with torch.cuda.device(self.device):
            self._finish_upload(self._start_upload())
            torch.cuda.current_stream(self.device).synchronize()

    def _start_upload(self):
        blob, lo = _payload_source(self.archive, self.plan)
        up = _Uploader(blob, self.device)
        up.send(lo, lo + self.plan.payload.size, self.d_payload)
        return up

    def _finish_upload(self, up):
        up.wait(0)
        up.close()

    def run(self, stream=None, phases: int = 0):
        """Launch the decode on `stream` (default: torch's current). Asynchronous.
        `phases` restricts the launch sequence (bit 0 stream decode, 1 conditioned-chunk
        kernels, 2 finish, 3 verdicts, 4 fused BF16 chunks) so one phase can be timed
        alone; 0 runs all."""
        import torch
        self._c.phases = phases
        with torch.cuda.device(self.device):
            s = stream if stream is not None else torch.cuda.current_stream(self.device)
            rc = self.lib.lmz_gpu_decode_chunks_dev(ctypes.byref(self._c), s.cuda_stream)
        if rc != gpu.OK:
            raise RuntimeError(f"decode launch failed ({rc}): {gpu.last_error()}")
        if not self.launches_per_run and not phases:
            self.launches_per_run = self.lib.lmz_gpu_plan_launches()
        return self.output

    @property
    def output(self):
        """The decoded output space (device uint8 tensor of `total` bytes)."""
        return self.d_out[:self.plan.total]

    def check(self) -> None:
        """Synchronise and raise CorruptArchive if any stream or chunk failed."""
        import torch
        torch.cuda.synchronize(self.device)
        self._arena.arrived()
        if int(self.d_any_bad.item()) == 0:
            return
        p = self.plan
        st = self.d_chunk_status.cpu().numpy()[:p.chunks.size]
        bad = np.nonzero(st)[0]
        if bad.size:
            rec = int(p.chunks["record"][bad[0]])
            raise CorruptArchive(f"chunk {rec} ({bad.size} in all): "
                                 f"{_ST_NAMES.get(int(st[bad[0]]), st[bad[0]])}")
        ss = self.d_stream_status.cpu().numpy()[:p.stream_jobs.size]
        hard = np.nonzero((ss != 0) & (ss != 0x100))[0]
        if hard.size:
            rec = int(p.stream_owner[hard[0]])
            raise CorruptArchive(f"a plane of chunk {rec}: {_ST_NAMES.get(int(ss[hard[0]]), '?')}")
        fs = self.d_fused_status.cpu().numpy()[:p.fused_jobs.size]
        hard = np.nonzero((fs != 0) & (fs != 0x100))[0]
        if hard.size:
            raise CorruptArchive(f"the exponent plane of a bf16 chunk: "
                                 f"{_ST_NAMES.get(int(fs[hard[0]]), '?')}")
        ds = self.d_delta_status.cpu().numpy()[:2 * p.delta_jobs.size]
        hard = np.nonzero((ds != 0) & (ds != 0x100))[0]
        if hard.size:
            raise CorruptArchive(f"a plane of a delta chunk's difference: {_ST_NAMES.get(int(ds[hard[0]]), '?')}")
        raise CorruptArchive("a bucket segment of a conditioned chunk failed to decode")

    def chunk_crcs(self) -> np.ndarray:
        """crc32 of every decoded chunk, in archive record order."""
        p = self.plan
        crc = self.d_chunk_crc.cpu().numpy().view(np.uint32)[:p.chunks.size]
        out = np.zeros(p.chunks.size, dtype=np.uint32)
        out[p.chunks["record"]] = crc
        return out

    def tensors(self):
        """{(member path, tensor name): device tensor view} for safetensors members,
        typed and shaped from the manifest; views into the output buffer."""
        import torch
        out = {}
        for key, (dt, shape, s, e) in self.archive.tensor_index().items():
            name = _TORCH_DTYPES.get(dt)
            raw = self.d_out[s:e]
            if name is None or s % 2:
                out[key] = raw
                continue
            try:
                out[key] = raw.view(getattr(torch, name)).reshape(shape)
            except RuntimeError:
                out[key] = raw
        return out


class PipelinedDecoder:
    """Host-to-HBM decode with the upload overlapped: the archive's chunks are cut
    into `nslices` runs of consecutive payload bytes, each with its own plan, and
    slice i decodes on the compute stream while slice i+1 is still crossing PCIe on
    the copy stream.  All slices write into one output buffer.  Archives with refs
    or deltas (which read other chunks' output) use a single slice.

    `nslices=None` chooses: 8 for archives of small chunks; for chunks of a megabyte or
    more, whose decode time is the latency of one long stream whatever their number,
    one slice per ~1900 such chunks (a slice of fewer costs as much as a full one)."""

    def __init__(self, ar, nslices=None, device=None, checksum: bool = True):
        import torch
        self.archive = ar if isinstance(ar, fmt.Archive) else fmt.Archive(ar)
        r = self.archive.records
        groups = _slice_groups(self.archive, nslices)
        self.device = torch.device(device if device is not None else
                                   f"cuda:{torch.cuda.current_device()}")
        out = torch.empty(self.archive.total + 64, dtype=torch.uint8, device=self.device)
        self.slices, self.ranges = [], []
        for g in groups:
            lo = int(r["off"][g].min())
            hi = int((r["off"][g].astype(np.int64) + r["clen"][g]).max())
            p = planner.build_plan(self.archive, select=g, payload_range=(lo, hi))
            self.slices.append(ArchiveDecoder(self.archive, device=self.device, checksum=checksum,
                                              out=out, plan=p))
            self.ranges.append((lo, hi))
        self.d_out = out
        self.copy_stream = torch.cuda.Stream(self.device)
        self.h2d_bytes = sum(hi - lo for lo, hi in self.ranges)

    @property
    def launches_per_run(self) -> int:
        return sum(s.launches_per_run for s in self.slices)

    def run_from_host(self, pinned, stream=None):
        """`pinned`: a pinned uint8 host tensor over the archive's bytes (offset 0 =
        file start).  Uploads and decodes slice by slice; asynchronous."""
        import torch
        compute = stream if stream is not None else torch.cuda.current_stream(self.device)
        self.copy_stream.wait_stream(compute)
        for dec, (lo, hi) in zip(self.slices, self.ranges):
            with torch.cuda.stream(self.copy_stream):
                dec.upload(pinned[lo:hi], non_blocking=True)
                ev = torch.cuda.Event()
                ev.record(self.copy_stream)
            compute.wait_event(ev)
            dec.run(stream=compute)
        return self.d_out[:self.archive.total]

    def run_from_file(self, stream=None, staging=None):
        """The same from the archive's own bytes wherever they are (a mapped file, the page
        cache, ordinary memory): see `load_archive`, which also plans under the copies."""
        import torch
        compute = stream if stream is not None else torch.cuda.current_stream(self.device)
        up = _Uploader(self.archive.blob, self.device, staging, compute)
        for dec, (lo, hi) in zip(self.slices, self.ranges):
            up.send(lo, hi, dec.d_payload)
        for si, dec in enumerate(self.slices):
            up.wait(si)
            dec.run(stream=compute)
        up.close()
        return self.d_out[:self.archive.total]

    def check(self):
        for dec in self.slices:
            dec.check()


class Staging:
    """Page-locked staging between a file and the device: `depth` blocks of `block` bytes and
    the library's threads that fill and send them (csrc/host_io.inl).  Twelve threads: the copy out
    of the page cache bounds a load, and a dozen reach the host memory's rate."""

    _shared = None

    def __init__(self, block: int = 2 << 20, depth: int = 24, threads: int = 12):
        import weakref
        if threads >= depth:
            raise ValueError("staging needs more buffers than threads")
        lib = gpu.library()
        self.block, self.depth = block, depth
        self.handle = lib.lmz_gpu_staging_new(block, depth, threads)
        if not self.handle:
            raise RuntimeError(gpu.last_error())
        weakref.finalize(self, lib.lmz_gpu_staging_free, self.handle).atexit = False

    @classmethod
    def shared(cls):
        if cls._shared is None:
            cls._shared = cls()
        return cls._shared


class _Uploader:
    """Byte ranges of an archive -> device memory through `Staging`, in the background.

    `send(lo, hi, dst)` queues one range; the staging's threads copy it block by block while
    the caller plans and launches.  `wait(i)` blocks until the i-th range has been issued
    whole and makes `stream` (default: torch's current) wait for its arrival."""

    def __init__(self, blob, device, staging=None, stream=None):
        import torch
        self.blob, self.fd, self.lib = blob, getattr(blob, "fd", -1), gpu.library()
        self.staging = staging if staging is not None else Staging.shared()
        self.stream = stream if stream is not None else torch.cuda.current_stream(device)
        self.device = device
        self.sent_to = []                    # held until the copies have arrived
        with torch.cuda.device(device):
            self.handle = self.lib.lmz_gpu_transfer_new(self.staging.handle, self.stream.cuda_stream)
        if not self.handle:
            raise RuntimeError(gpu.last_error())

    def send(self, lo: int, hi: int, dst) -> int:
        import torch
        self.sent_to.append(dst)
        with torch.cuda.device(self.device):
            r = self.lib.lmz_gpu_transfer_upload(self.handle, self.fd, self.blob.ctypes.data, int(lo), int(hi - lo),
                                                 dst.data_ptr())
        if r < 0:
            raise RuntimeError(gpu.last_error())
        return r

    def wait(self, si: int) -> None:
        if self.lib.lmz_gpu_transfer_wait(self.handle, si, self.stream.cuda_stream) != gpu.OK:
            raise RuntimeError(f"an upload failed: {gpu.last_error()}")

    def close(self) -> None:
        """Return when every range has arrived; the memory sent to must live until then."""
        if self.handle:
            handle, self.handle = self.handle, None
            rc = self.lib.lmz_gpu_transfer_free(handle)
            self.sent_to.clear()
            if rc != gpu.OK:
                raise RuntimeError(f"an upload failed: {gpu.last_error()}")

    def __del__(self):
        if getattr(self, "handle", None):
            self.lib.lmz_gpu_transfer_free(self.handle)


def _slice_groups(ar, nslices):
    """Record indices of an archive cut into runs of consecutive payload bytes of about
    equal size (refs and deltas read other chunks' output: one run then)."""
    r = ar.records
    if nslices is None:
        big = int((r["rlen"] >= (1 << 20)).sum())
        nslices = 8 if big == 0 else max(1, min(8, big // 1900))
    sourced = np.isin(r["codec"], (fmt.CODEC_REF, fmt.CODEC_DELTA)).any()
    order = np.argsort(r["off"], kind="stable")
    nslices = 1 if sourced or r.size < nslices else nslices
    cum = np.cumsum(r["clen"][order].astype(np.int64))
    cuts = np.searchsorted(cum, cum[-1] * np.arange(1, nslices) / nslices) if r.size else []
    return [g for g in np.split(order, cuts) if g.size]


def _upload_cuts(table_off: int, nslices):
    """Where an archive's payload region is cut into ranges that are uploaded (and decoded) one after
    the other: as many as asked for, or one per 192 MiB, at most eight.  (A range is decoded
    under the upload of the next, but a decode has a smallest duration, that of one stream.)"""
    n = nslices if nslices is not None else min(8, -(-table_off // (192 << 20)))
    n = max(1, min(int(n), table_off >> 16))             # (of 64 KiB at least: a range has an event and a wait of its own)
    return [table_off * i // n for i in range(n + 1)]


def load_archive(path, device=None, checksum: bool = True, nslices=None, stats=None, staging=None):
    """File on disk -> verified plaintext in HBM (the load the reference times as "cold
    disk -> VRAM", README.md:79-84).  The upload of the payload region starts before the index is
    read: the library's threads stream it range after range through page-locked staging to the
    device, while this thread reads the index, plans each range's chunks and, as soon as the
    range has been issued, launches their decode behind it; every chunk's verdict is checked at the
    end.  Returns the decoded output space as a device tensor.  `stats`, a dict, receives `open_s`
    (until the upload has been started), `run_s` (everything else), `plan_s` (reading the index and
    planning inside run_s), `h2d_bytes`, `slices`."""
    import time

    import torch
    t0 = time.perf_counter()
    blob = fmt.open_blob(path)
    table_off = fmt.payload_end(blob)
    dev = torch.device(device if device is not None else f"cuda:{torch.cuda.current_device()}")
    with torch.cuda.device(dev):
        compute = torch.cuda.current_stream(dev)
        pad = gpu.pad_bytes()
        # (room behind the payload for header chunks that are inflated on the host)
        room = (1 << 20) + table_off // 256
        payload = torch.empty(table_off + room + pad, dtype=torch.uint8, device=dev)
        cuts = _upload_cuts(table_off, nslices)

        def start():
            up = _Uploader(blob, dev, staging, compute)
            return up, [up.send(lo, hi, payload[lo:]) for lo, hi in zip(cuts, cuts[1:])]

        up, sent = start()
        t1 = time.perf_counter()
        try:
            ar = fmt.Archive(blob)
            ar.check_coverage()
            inflated = planner.inflated_bytes(ar.records)
            if inflated > room:
                up.close()
                payload = torch.empty(table_off + inflated + pad, dtype=torch.uint8, device=dev)
                up, sent = start()
            out = torch.empty(ar.total + 64, dtype=torch.uint8, device=dev)
            decs, plan_s, extras_at, tp = [], 0.0, table_off, t1
            for upto, group in _range_groups(ar, cuts, nslices):
                p = planner.build_plan(ar, select=group, payload_range=(0, table_off), extras_at=extras_at)
                extras_at += p.extras.size
                dec = ArchiveDecoder(ar, device=dev, checksum=checksum, out=out, plan=p, payload=payload, settle=False)
                plan_s += time.perf_counter() - tp
                for si in sent[:upto]:
                    up.wait(si)
                tp = time.perf_counter()
                dec.run(stream=compute)
                decs.append(dec)
        finally:
            up.close()
        for dec in decs:
            dec.check()
        torch.cuda.synchronize(dev)
    if stats is not None:
        stats.update(open_s=t1 - t0, run_s=time.perf_counter() - t1, plan_s=plan_s,
                     h2d_bytes=table_off, slices=len(decs))
    return out[:ar.total]


def _range_groups(ar, cuts, nslices):
    """[(ranges needed, record indices or None for all)]: the chunks each uploaded range completes.
    One group where chunks read other chunks' output, and for chunks of a megabyte or more, whose
    decode time is the latency of one long stream whatever their number, one per ~1900 of them."""
    r, n = ar.records, len(cuts) - 1
    if np.isin(r["codec"], (fmt.CODEC_REF, fmt.CODEC_DELTA)).any():
        n = 1
    elif nslices is None:
        big = int((r["rlen"] >= (1 << 20)).sum())
        n = min(n, max(1, big // 1900)) if big else n
    if n <= 1 or r.size < n:
        return [(len(cuts) - 1, None)]
    end = r["off"].astype(np.int64) + r["clen"]
    step = (len(cuts) - 1) / n
    out, done = [], 0
    for i in range(1, n + 1):
        upto = len(cuts) - 1 if i == n else int(i * step)
        mine = np.nonzero((end > done) & (end <= cuts[upto]))[0] if i < n else np.nonzero(end > done)[0]
        done = cuts[upto]
        if mine.size:
            out.append((upto, mine))
    return out


def decode_tensors(ar, names, device=None, checksum: bool = True):
    """Decode only what the named tensors need.  `names`: (member path, tensor name)
    keys of `Archive.tensor_index()`, or bare tensor names when they are unambiguous.
    Uploads the payload bytes of the chunks that overlap those tensors (and of the
    sources of any ref or delta among them), decodes them into a buffer that spans
    just their part of the output space, verifies, and returns {key: device tensor}."""
    import torch
    from . import multi

    ar = ar if isinstance(ar, fmt.Archive) else fmt.Archive(ar)
    index = ar.tensor_index()
    by_name = {}
    for key in index:
        by_name.setdefault(key[1], []).append(key)
    keys = []
    for n in names:
        if isinstance(n, tuple):
            if n not in index:
                raise KeyError(n)
            keys.append(n)
        else:
            hits = by_name.get(n, [])
            if len(hits) != 1:
                raise KeyError(f"{n!r} names {len(hits)} tensors; give (member path, name)")
            keys.append(hits[0])
    if not keys:
        return {}
    select = multi.cover(ar, [(index[k][2], index[k][3]) for k in keys])
    r = ar.records[select]
    out_lo = int(r["dst"].min()) & ~15                     # keep the output's 16-byte phase
    out_hi = int((r["dst"].astype(np.int64) + r["rlen"]).max())
    pay_lo = int(r["off"].min()) & ~15
    pay_hi = int((r["off"].astype(np.int64) + r["clen"]).max())
    dev = torch.device(device if device is not None else f"cuda:{torch.cuda.current_device()}")
    with torch.cuda.device(dev):
        # only what the chunks hold crosses, to its place in a buffer that spans all of it, while the
        # chunks are planned (gaps below 256 KiB are not worth a range of their own)
        room = pay_hi - pay_lo + planner.inflated_bytes(r) + gpu.pad_bytes()
        payload = torch.empty(room, dtype=torch.uint8, device=dev)
        up = _Uploader(ar.blob, dev)
        order = np.argsort(r["off"], kind="stable")
        lo = r["off"][order].astype(np.int64)
        hi = np.maximum.accumulate(lo + r["clen"][order])
        first = np.concatenate(([True], lo[1:] > hi[:-1] + (256 << 10)))
        last = np.concatenate((first[1:], [True]))
        sent = [up.send(a, b, payload[a - pay_lo:]) for a, b in zip(lo[first].tolist(), hi[last].tolist())]
        try:
            p = planner.build_plan(ar, select=select, payload_range=(pay_lo, pay_hi), out_range=(out_lo, out_hi))
            dec = ArchiveDecoder(ar, device=dev, checksum=checksum, plan=p, payload=payload, settle=False)
            for si in sent:
                up.wait(si)
            dec.run()
        finally:
            up.close()
    dec.check()
    out = {}
    for k in keys:
        dt, shape, s, e = index[k]
        raw = dec.d_out[s - out_lo:e - out_lo]
        name = _TORCH_DTYPES.get(dt)
        if name is not None and (s - out_lo) % 2 == 0:
            try:
                raw = raw.view(getattr(torch, name)).reshape(shape)
            except RuntimeError:
                pass
        out[k] = raw
    return out


def decode_archive(ar, device=None, checksum: bool = True):
    """Decode a whole archive to a device tensor and verify it (the reference's
    `decompress` + `verify`, lmz/api.py:889, :1061, without the files)."""
    dec = ArchiveDecoder(ar, device=device, checksum=checksum)
    dec.run()
    dec.check()
    return dec.output
