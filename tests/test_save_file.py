"""What save_archive does to the file, on the CPU: the device's part is stood in for."""
import os

import pytest

from oracle import archive as oa, synth


@pytest.fixture
def old(tmp_path):
    """An archive that is to be overwritten."""
    path = tmp_path / "a.lmz"
    path.write_bytes(oa.write_archive([("m.safetensors", synth.llama_shard([0], 5, scale=0.125))], mapped=True))
    return path


def test_an_unfinished_overwrite_does_not_open(old, monkeypatch):
    """From the first byte of a save to its last the file is no archive, also if the process ends in between; a
    save that fails leaves it empty."""
    from lmz_b200 import archive, save
    seen = []

    def writer(fd, *rest):
        for reader in (archive.open_blob, archive.Archive):
            with pytest.raises(archive.FormatError):
                archive.payload_end(reader(str(old)))
        seen.append(old.stat().st_size)
        raise KeyboardInterrupt

    monkeypatch.setattr(save, "_write_archive", writer)
    size = old.stat().st_size
    with pytest.raises(KeyboardInterrupt):
        save.save_archive(str(old), [])
    assert seen == [size] and old.stat().st_size == 0


def test_a_shorter_archive_over_a_longer_one(old, monkeypatch):
    """The header comes after everything else, the cut to length included: with the old footer still at the end
    of the file it would be the new header over the old index."""
    from lmz_b200 import archive, gpu, save
    monkeypatch.setattr(gpu, "library", lambda: None)
    put, cut = save._put, os.ftruncate
    order = []
    monkeypatch.setattr(save, "_put", lambda fd, data, pos: order.append("header" if pos == 0 and any(data) else "put") or put(fd, data, pos))
    monkeypatch.setattr(os, "ftruncate", lambda fd, n: order.append("cut") or cut(fd, n))
    before = old.stat().st_size
    n = save.save_archive(str(old), [])
    assert n == old.stat().st_size < before and archive.Archive(str(old)).total == 0
    assert order[-2:] == ["cut", "header"], order


@pytest.mark.parametrize("where", ["a device", "a file that may be written only"])
def test_where_only_writing_goes(old, monkeypatch, where):
    from lmz_b200 import archive, gpu, save
    monkeypatch.setattr(gpu, "library", lambda: None)
    if where == "a device":
        assert save.save_archive(os.devnull, []) > 0
        with pytest.raises(ValueError, match="CUDA"):
            save.save_archive(os.devnull, [("m", None)])
        return
    real = os.open

    def as_its_writer_may(path, flags, *mode):
        if flags & os.O_RDWR:
            raise PermissionError(13, "made to fail")
        return real(path, flags, *mode)

    monkeypatch.setattr(os, "open", as_its_writer_may)
    assert save.save_archive(str(old), []) == old.stat().st_size
    monkeypatch.undo()
    assert archive.Archive(str(old)).total == 0
