"""Stored Deflate blocks: of every length at which their copy changes its step, at every alignment of their bytes in
the stream and in the output, after and before blocks whose matches reach into them and across them, cut by the
stream's end and by the output's; and what they cost."""
import zlib

import numpy as np
import pytest

from tests.test_deflate_far_distances import _Fixed

SIZES = [0, 1, 2, 3, 4, 5, 7, 8, 9, 31, 127, 1024, 2047, 2048, 2049, 2052, 4095, 4099, 10000, 32767, 40000, 65535]


class _Blocks(_Fixed):
    """Blocks of stored bytes and of fixed codes, the last one empty."""

    def __init__(self):
        super().__init__()
        self.out = ""  # bits so far

    def stored(self, data):
        self.out += "000"
        self.out += "0" * (-len(self.out) % 8)
        n = len(data)
        raw = np.frombuffer(bytes([n & 255, n >> 8, ~n & 255, ~n >> 8 & 255]) + data, np.uint8)
        self.out += "".join(np.unpackbits(raw, bitorder="little").astype(str))
        self.data += data

    def codes(self):  # what was written since as one block
        self.out += "010" + "".join(self.bits) + "0000000"
        self.bits = []

    def stream(self):
        b = self.out + "110" + "0000000"
        b += "0" * (-len(b) % 8)
        return np.packbits(np.frombuffer(b.encode(), np.uint8) - 48, bitorder="little").tobytes(), bytes(self.data)


def _mixed(seed):
    rng = np.random.default_rng(seed)
    f = _Blocks()
    for n in rng.permutation(SIZES).tolist() + [40000]:
        if len(f.data) + n > 250000:
            continue
        f.stored(rng.integers(0, 256, n, dtype=np.uint8).tobytes())
        if rng.random() < 0.7:
            for _ in range(int(rng.integers(1, 12))):
                f.literal(int(rng.integers(0, 256)))
                if len(f.data) > 16385 and rng.random() < 0.6:
                    f.match(int(rng.integers(3, 259)), int(rng.integers(16385, min(len(f.data), 32768) + 1)))
            f.codes()
    return f.stream()


def test_streams_are_deflate():
    for seed in range(6):
        s, data = _mixed(seed)
        assert zlib.decompress(s, -15) == data


def _decode(cuda, native, parts, lens, shift):
    """The streams one after another, `shift` bytes into the buffer, as one batch: (outputs, statuses)."""
    from codag_b200 import api
    comp = np.frombuffer(b"\xFF" * shift + b"".join(parts), np.uint8).copy()
    descs = np.zeros(len(parts), dtype=native.CHUNK_DESC_DTYPE)
    descs["codec"], descs["elem_bytes"], descs["comp_len"], descs["out_len"] = native.DEFLATE, 1, [len(p) for p in parts], lens
    descs["comp_off"] = shift + np.cumsum([0] + [len(p) for p in parts[:-1]])
    descs["out_off"] = np.cumsum([0] + list(lens[:-1])) + 3 * shift
    out = cuda.full((sum(lens) + 3 * shift + 64,), 0x5A, dtype=cuda.uint8, device="cuda")
    st = cuda.full((len(parts),), -1, dtype=cuda.int32, device="cuda")
    plan = api.BatchPlan(descs)
    plan.run(cuda.from_numpy(comp).to("cuda"), out, st)
    got = out.cpu().numpy()
    plan.close()
    assert np.all(got[sum(lens) + 3 * shift:] == 0x5A)
    return [bytes(got[int(d["out_off"]):int(d["out_off"]) + int(d["out_len"])]) for d in descs], st.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("shift", range(16))
def test_blocks(cuda, native, shift):
    made = [_mixed(shift * 4 + k) for k in range(4)]
    got, st = _decode(cuda, native, [m[0] for m in made], [len(m[1]) for m in made], shift)
    assert not st.any()
    for g, (_, data) in zip(got, made):
        assert g == data


@pytest.mark.gpu
def test_cut(cuda, native, oracle):
    """A stream that ends inside a stored block, an output that does, and a length that does not agree with its
    complement."""
    rng = np.random.default_rng(9)
    data = rng.integers(0, 256, 9000, dtype=np.uint8).tobytes()
    f = _Blocks()
    f.stored(data[:3000])
    f.stored(data[3000:])
    s, _ = f.stream()
    bad = bytearray(s)
    bad[3008] ^= 1  # the second block's complement
    parts = [s, s[:-2], s[:-3], s[:8000], s[:3005], s, s, bytes(bad)]
    lens = [9000, 9000, 9000, 9000, 9000, 8999, 3000, 9000]
    got, st = _decode(cuda, native, parts, lens, 1)
    for p, n, g, status in zip(parts, lens, got, st):
        ost, ref = oracle.deflate_chunk(np.frombuffer(p, np.uint8), n, 0)
        assert status == ost, (len(p), n)
        assert ost or g == bytes(ref[:n])
    assert st.tolist() == [0, 2, 2, 2, 2, 2, 2, 2]


@pytest.mark.gpu
def test_cost(cuda, native):
    """64 MiB of stored blocks: within ten times a device copy of as many bytes (as tokens they took 18 times)."""
    from codag_b200 import api
    size, ch = 64 << 20, 131072
    raw = np.random.default_rng(2).integers(0, 256, size, dtype=np.uint8)
    comp, blk, _ = native.encode_deflate(raw, ch, 6, require_no_stored=False)
    d, o = cuda.from_numpy(comp).to("cuda"), cuda.from_numpy(blk[1:].view(np.int64)).to("cuda")
    out, src = cuda.zeros(size, dtype=cuda.uint8, device="cuda"), cuda.from_numpy(raw).to("cuda")
    st = cuda.full((blk.size - 2,), -1, dtype=cuda.int32, device="cuda")
    best = [1e9, 1e9]
    for r in range(12):
        for i, fn in enumerate((lambda: api.decompress_deflate(d, o, ch, out, 2, None, st), lambda: out.copy_(src))):
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            cuda.cuda.synchronize()
            if r >= 2:
                best[i] = min(best[i], a.elapsed_time(b))
            if r == 0 and i == 0:
                assert not st.cpu().numpy().any() and np.array_equal(out.cpu().numpy(), raw)
    assert best[0] < 10 * best[1], best
