"""Seeded inputs shared by the tests."""
import struct

import numpy as np

# translate() tables over uniform bytes: the reference's awkward distributions
# (tests/test_lmz.py:2335-2346 in the reference tree).
SHAPES = {
    "single": bytes([0x5A]) * 256,
    "two": bytes([0x01]) * 128 + bytes([0xFE]) * 128,
    "flat": bytes(range(256)),
    "tail": bytes([0x20]) * 250 + bytes(range(6)),
    "skewed": bytes([0x40]) * 170 + bytes(range(16)) * 5 + bytes([0x7F]) * 6,
}


def lcg_bytes(n: int, seed: int = 0) -> bytes:
    """The reference tests' deterministic byte source (tests/test_lmz.py:44-51)."""
    out, x = bytearray(), seed | 1
    while len(out) < n:
        x = (x * 6364136223846793005 + 1442695040888963407) & ((1 << 64) - 1)
        out += x.to_bytes(8, "little")
    return bytes(out[:n])


def shaped(name: str, n: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    raw = rng.integers(0, 256, n, dtype=np.uint8).tobytes().translate(SHAPES[name])
    return np.frombuffer(raw, dtype=np.uint8)


def distribution(name: str, n: int, seed: int) -> np.ndarray:
    """The eight symbol distributions of the decoder stress configuration."""
    from oracle import synth
    return synth.stress_plane(name, n, seed)


DISTRIBUTIONS = ("uniform", "single", "two", "geometric", "zipf", "exponent", "mantissa",
                 "zero-runs")


def pack_streams(streams):
    offs, pos = bytearray(), 0
    for s in streams:
        offs += struct.pack("<QQ", pos, len(s))
        pos += len(s)
    return b"".join(streams), bytes(offs)


def archive_of(members, chunks):
    """An archive written record by record.  `members`: manifest entries; `chunks`: (payload, rlen, crc,
    codec, esize, flags) in output order."""
    import json
    import zlib

    from oracle import archive as oa
    recs = np.zeros(len(chunks), dtype=oa.RECORD)
    body, dst = bytearray(oa.HEADER.size), 0
    for rec, (payload, rlen, crc, codec, esize, flags) in zip(recs, chunks):
        rec["off"], rec["dst"], rec["clen"], rec["rlen"], rec["crc"] = len(body), dst, len(payload), rlen, crc
        rec["codec"], rec["esize"], rec["flags"] = codec, esize, flags
        body += payload
        dst += rlen
    body[:oa.HEADER.size] = oa.HEADER.pack(oa.MAGIC, 6, 0, dst, 0, 0)
    table = zlib.compress(recs.tobytes(), 3)
    manifest = zlib.compress(json.dumps({"version": 1, "members": members, "chunks": len(chunks), "checksum": "crc32",
                                         "table_raw_len": recs.nbytes, "total_size": dst}).encode(), 3)
    off = len(body)
    return bytes(body) + table + manifest + oa.FOOTER.pack(off, len(table), off + len(table), len(manifest), oa.TAIL)


def deflated_delta(n: int):
    """(archive, plaintext): a member of `n` random bytes and one that differs from it in a few places, the second
    as one delta chunk whose difference is a single deflated stream."""
    import zlib
    rng = np.random.default_rng(n)
    first = rng.integers(0, 256, n, dtype=np.uint8)
    second = first.copy()
    second[rng.integers(0, n, 40)] ^= 0x55
    members = [{"path": p, "size": n, "dst": i * n, "kind": "safetensors", "mode": 0o644, "crc": 0,
                "tensors": {"w": {"dtype": "U8", "shape": [n], "offsets": [0, n]}}} for i, p in enumerate(("a", "b"))]
    diff = struct.pack("<QB", 0, 1) + zlib.compress((first ^ second).tobytes(), 6)
    return archive_of(members, [(first.tobytes(), n, zlib.crc32(first), 0, 1, 0),
                                (diff, n, zlib.crc32(second), 8, 1, 2)]), np.concatenate((first, second))
