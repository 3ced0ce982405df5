"""Deflate matches at every distance from 32513 to 32768, where a source's place in the decoder's 32 KiB
window is one that a byte of the same 256-byte batch takes over.  zlib's compressor stops at 32506, so the
streams are written here, with the fixed codes (RFC 1951 3.2.6)."""
import zlib

import numpy as np
import pytest

LEN_BASE = [3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 15, 17, 19, 23, 27, 31, 35, 43, 51, 59, 67, 83, 99, 115, 131, 163, 195, 227, 258]
LEN_BITS = [0] * 8 + [b for b in range(1, 6) for _ in range(4)] + [0]
CHUNK = 131072


class _Fixed:
    """One block of fixed codes, and the bytes it stands for."""

    def __init__(self):
        self.bits, self.data = [], bytearray()

    def _code(self, v, n):  # Huffman codes, most significant bit first
        self.bits.append(format(v, f"0{n}b"))

    def _extra(self, v, n):  # extra bits, least significant bit first
        if n:
            self.bits.append(format(v, f"0{n}b")[::-1])

    def _symbol(self, s):
        if s < 144:
            self._code(0x30 + s, 8)
        elif s < 256:
            self._code(0x190 + s - 144, 9)
        elif s < 280:
            self._code(s - 256, 7)
        else:
            self._code(0xC0 + s - 280, 8)

    def literal(self, b):
        self._symbol(b)
        self.data.append(b)

    def match(self, length, dist):
        k = 28 if length == 258 else max(i for i in range(28) if LEN_BASE[i] <= length)
        self._symbol(257 + k)
        self._extra(length - LEN_BASE[k], LEN_BITS[k])
        assert 16385 <= dist <= 32768  # distance codes 28 and 29, 13 extra bits
        self._code(28 + (dist >= 24577), 5)
        self._extra((dist - 16385) % 8192, 13)
        for _ in range(length):
            self.data.append(self.data[-dist])

    def stream(self):
        b = "110" + "".join(self.bits) + "0" * 7  # last block, fixed codes; end of block
        b += "0" * (-len(b) % 8)
        body = np.packbits(np.frombuffer(b.encode(), np.uint8) - 48, bitorder="little").tobytes()
        return body, bytes(self.data)


def _far(seed):
    """32 KiB of literals and some, then matches at all these distances: short ones, so that one batch has many
    of them, or of every length, with literals between some of them."""
    rng = np.random.default_rng(seed)
    f = _Fixed()
    for b in rng.integers(0, 256, 32768 + int(rng.integers(0, 300))).tolist():
        f.literal(b)
    longest = [3, 12, 40, 258][seed % 4]
    for d in rng.permutation(np.arange(32513, 32769)).tolist():
        f.match(int(rng.integers(3, longest + 1)), d)
        for b in rng.integers(0, 256, int(rng.integers(0, 3))).tolist():
            f.literal(b)
    return f.stream()


def test_streams_are_deflate(oracle):
    for seed in range(4):
        s, data = _far(seed)
        assert zlib.decompress(s, -15) == data
        st, out = oracle.deflate_chunk(np.frombuffer(s, np.uint8), CHUNK, 0, len(data))
        assert st == 0 and bytes(out[:len(data)]) == data


@pytest.mark.gpu
def test_gpu(cuda, native):
    from codag_b200 import api
    made = [_far(seed) for seed in range(8)]
    cs = api.pack_chunks([np.frombuffer(s, np.uint8) for s, _ in made], [native.DEFLATE] * 8, [1] * 8,
                         [len(d) for _, d in made], 0)
    out = cuda.zeros(cs.out_bytes, dtype=cuda.uint8, device="cuda")
    st = cuda.full((8,), -1, dtype=cuda.int32, device="cuda")
    plan = api.BatchPlan(cs.descs)
    plan.run(cuda.from_numpy(cs.comp).to("cuda"), out, st)
    batch = out.cpu().numpy()
    plan.close()
    assert not st.cpu().numpy().any()
    for (s, data), d in zip(made, cs.descs):
        o, n = int(d["out_off"]), len(data)
        assert bytes(batch[o:o + n]) == data
        rel = cuda.tensor([0, len(s)], dtype=cuda.int64, device="cuda")
        one = cuda.zeros(n, dtype=cuda.uint8, device="cuda")
        st1 = cuda.full((1,), -1, dtype=cuda.int32, device="cuda")
        api.decompress_deflate(cuda.from_numpy(np.frombuffer(s, np.uint8).copy()).to("cuda"), rel, CHUNK, one, 0, n, st1)
        assert st1.item() == 0 and bytes(one.cpu().numpy()) == data
