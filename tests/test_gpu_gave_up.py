"""The decoder's fill waits for other warps with a limit.  A wait that runs out (the limit lowered to a poll or two
when the context is opened) is the GPU's failure and not damage: a status of its own, ZC_E_DEVICE from the calls, and
the process's other work goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GAVE_UP = 11


@pytest.fixture(scope="module")
def blocks():
    """A block whose lines each need the line before, and one that is stored."""
    import zero_cuda as Z
    r = np.random.default_rng(1)
    data = np.concatenate([np.resize(r.integers(0, 256, 100, dtype=np.uint8), 1 << 18), r.integers(0, 256, 5000, dtype=np.uint8)])
    with Z.CudaCodec(level=5) as codec:
        m, lens, _, pay, offs = codec.compress_arrays(data, 18)
        body, clens, rlens = Z.record_bodies(data, m, lens, pay, offs, 18)
    assert list(m) == [1, 0]
    return data, body, clens, m, rlens


@pytest.fixture()
def hasty(monkeypatch):
    import zero_cuda as Z
    monkeypatch.setenv("ZC_FILL_POLLS", "0")
    with Z.CudaCodec(level=5) as codec:
        monkeypatch.delenv("ZC_FILL_POLLS")
        yield codec


def test_host_call(hasty, blocks):
    import zero_cuda as Z
    data, body, clens, methods, rlens = blocks
    offs = np.array([0, clens[0]])
    with pytest.raises(Z.DeviceError, match="gave up on block 0"):
        hasty.decompress_arrays(body, offs, clens, methods, rlens)
    raw, _, err = hasty.decompress_arrays(body[clens[0]:], [0], clens[1:], methods[1:], rlens[1:])  # (nothing to wait for)
    assert not err.any() and np.array_equal(raw, data[1 << 18:])
    damaged = body.copy()
    damaged[:20] = 255
    with pytest.raises(Z.DataError, match="block 0 damaged"):
        hasty.decompress_arrays(damaged, offs, clens, methods, rlens)
    with Z.CudaCodec(level=5) as codec:
        raw, _, err = codec.decompress_arrays(body, offs, clens, methods, rlens)
    assert not err.any() and np.array_equal(raw, data)


def test_device_call(hasty, blocks):
    import torch
    data, body, clens, methods, rlens = blocks
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, d)).cuda()  # noqa: E731
    raw = torch.zeros(data.size, dtype=torch.uint8, device="cuda")
    err, crc = torch.zeros(2, dtype=torch.int32, device="cuda"), torch.zeros(2, dtype=torch.int32, device="cuda")
    hasty.decompress_device(t(np.append(body, np.zeros(64, np.uint8)), np.uint8), t([0, clens[0]], np.int64),
                            t(clens, np.int32), t(methods, np.uint8), t(rlens, np.int32), 2, 18, raw,
                            t([0, rlens[0]], np.int64), crc, err)
    torch.cuda.synchronize()
    assert err.tolist() == [GAVE_UP, 0]


def test_archive(hasty, blocks):
    import zero_cuda as Z
    data = blocks[0]
    arch = hasty.archive_write(data, [Z.ArchiveEntry("f", data.size)], 18)
    with pytest.raises(Z.DeviceError, match="gave up on block 0"):
        hasty.archive_extract(arch)


def test_server(blocks, monkeypatch):
    import zero_cuda as Z
    data, body, clens, methods, rlens = blocks
    monkeypatch.setenv("ZC_FILL_POLLS", "0")
    server = Z.Server(1 << 30)
    try:
        with pytest.raises(Z.DeviceError):
            server.wait(server.extract(body, clens, methods, rlens, 18))
        stored = server.wait(server.extract(body[clens[0]:], clens[1:], methods[1:], rlens[1:], 18))  # (nothing to wait for)
        assert np.array_equal(stored.raw, data[1 << 18:])
    finally:
        server.close()
