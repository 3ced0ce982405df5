"""Long Deflate matches that follow one another at one distance, which are expanded together: at every distance where
the repetition changes its step, for every number of matches around the decoder's lists of 480 and its lanes of 15,
alone, after and before other symbols, and ending a chunk; and what they cost."""
import zlib

import numpy as np
import pytest

from tests.test_deflate_far_distances import LEN_BASE, LEN_BITS
from tests.test_deflate_stored import _Blocks, _decode

DIST_BITS = [0, 0] + [b for b in range(14) for _ in range(2)]
DIST_BASE = [1, 2] + [3 + (1 << (c // 2)) - 2 + (c % 2) * (1 << (c // 2 - 1)) for c in range(2, 30)]
DISTANCES = [1, 2, 3, 5, 31, 32, 33, 127, 128, 129, 257, 2047, 2048, 2049, 30719, 30720, 30721, 32700, 32767, 32768]


class _Any(_Blocks):
    def match(self, length, dist):
        k = 28 if length == 258 else max(i for i in range(28) if LEN_BASE[i] <= length)
        self._symbol(257 + k)
        self._extra(length - LEN_BASE[k], LEN_BITS[k])
        c = max(i for i in range(30) if DIST_BASE[i] <= dist)
        self._code(c, 5)
        self._extra(dist - DIST_BASE[c], DIST_BITS[c])
        if dist <= len(self.data):
            p = self.data[len(self.data) - dist:]
            self.data += (p * (length // dist + 1))[:length]


def test_distance_codes():
    assert DIST_BASE == [1, 2, 3, 4, 5, 7, 9, 13, 17, 25, 33, 49, 65, 97, 129, 193, 257, 385, 513, 769, 1025, 1537, 2049, 3073,
                         4097, 6145, 8193, 12289, 16385, 24577]


def _repeats(seed):
    rng = np.random.default_rng(seed)
    f = _Any()
    f.stored(rng.integers(0, 256, 33000, dtype=np.uint8).tobytes())
    for d in rng.permutation(DISTANCES).tolist():
        for _ in range(int(rng.integers(0, 3))):
            f.literal(int(rng.integers(0, 256)))
        for _ in range(int(rng.choice([1, 14, 15, 16, 30, 45, 90, 200]))):
            f.match(258 if rng.random() < 0.9 else int(rng.integers(3, 259)), d)
        if rng.random() < 0.3:
            f.codes()
    f.codes()
    return f.stream()


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(4))
def test_mixed(cuda, native, seed):
    made = [_repeats(4 * seed + k) for k in range(4)]
    for s, data in made:
        assert zlib.decompress(s, -15) == data
    got, st = _decode(cuda, native, [m[0] for m in made], [len(m[1]) for m in made], 3 * seed)
    assert not st.any()
    for g, (_, data) in zip(got, made):
        assert g == data


@pytest.mark.gpu
@pytest.mark.parametrize("dist", [1, 33, 2049, 30721, 32768])
def test_counts(cuda, native, dist):
    """A literal prefix, then nothing but matches of one distance; and one match more than the output holds."""
    made = []
    for count in (2, 14, 15, 16, 29, 31, 479, 480, 481, 482, 495, 500, 959, 961, 1500):
        f = _Any()
        f.stored(np.random.default_rng(count).integers(0, 256, dist, dtype=np.uint8).tobytes())
        for _ in range(count):
            f.match(258, dist)
        f.codes()
        made.append(f.stream())
    lens = [len(d) for _, d in made]
    got, st = _decode(cuda, native, [s for s, _ in made], lens, 1)
    assert not st.any()
    for g, (_, data) in zip(got, made):
        assert g == data
    _, st = _decode(cuda, native, [s for s, _ in made], [n - 258 for n in lens], 1)
    assert np.all(st == 2)


@pytest.mark.gpu
def test_before_the_start(cuda, native):
    """A distance one past the bytes there are is refused."""
    parts, lens = [], []
    for have, dist in ((1, 1), (1, 2), (40, 40), (40, 41), (32767, 32768), (32768, 32768)):
        f = _Any()
        f.stored(b"x" * have)
        for _ in range(100):
            f.match(258, dist)
        f.codes()
        parts.append(f.stream()[0])
        lens.append(have + 25800)
    _, st = _decode(cuda, native, parts, lens, 0)
    assert st.tolist() == [0, 2, 0, 2, 2, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("period", [1, 24])
def test_cost(cuda, native, period):
    """64 MiB of zeros, or of one record, in 128 KiB chunks: within 15 times a device copy of as many bytes (byte by
    byte they took 43 times)."""
    from codag_b200 import api
    size, ch = 64 << 20, 131072
    raw = np.resize(np.arange(period, dtype=np.uint8) * 5, size)
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
    assert best[0] < 15 * best[1], best
