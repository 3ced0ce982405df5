"""Deflate chunks at the edges of the team decoder: streams shorter than a stretch of its 64 pieces, ends
of blocks in every place, matches at and across the 32-byte steps and 256-byte batches in which bytes
are placed, literals whose codes are longer than the look-up table, stored bytes around a token list's
length, and distances up to the window."""
import zlib

import numpy as np
import pytest


def _periodic(rng, n):
    """Repeats with every period from 1 to 40 and around 256, broken by single bytes."""
    parts, size = [], 0
    for period in list(range(1, 41)) + [63, 64, 65, 255, 256, 257, 258, 259]:
        p = rng.integers(0, 256, period, dtype=np.uint8)
        for ln in (3, 31, 32, 33, 255, 256, 257, 258, 259, 600):
            parts += [np.resize(p, ln), rng.integers(0, 256, 1, dtype=np.uint8)]
            size += ln + 1
    return np.resize(np.concatenate(parts), n)


def _skewed(rng, n):
    """Byte frequencies that halve from symbol to symbol: codes of up to 15 bits."""
    p = 0.5 ** np.arange(1, 41)
    return rng.choice(40, n, p=p / p.sum()).astype(np.uint8) * 5


def _far(rng, n):
    """Matches at distances around 32768 and of a few bytes, in noise."""
    a = rng.integers(0, 256, n, dtype=np.uint8)
    for at in range(32768, n - 300, 331):
        d, ln = int(rng.choice([32768, 32767, 32505, 40, 300])), int(rng.integers(3, 259))
        for i in range(ln):
            a[at + i] = a[at + i - d]
    return a


KINDS = {"periodic": _periodic, "skewed": _skewed, "far": _far,
         "zeros": lambda rng, n: np.zeros(n, np.uint8),
         "noise": lambda rng, n: rng.integers(0, 256, n, dtype=np.uint8)}


def _stream(data, level, strategy, every):
    co = zlib.compressobj(level, zlib.DEFLATED, 15, 9, strategy)
    if not every:
        return co.compress(data) + co.flush()
    out = b""
    for i in range(0, len(data), every):  # a block ends, and an empty stored one follows
        out += co.compress(data[i:i + every]) + co.flush(zlib.Z_FULL_FLUSH)
    return out + co.flush()


@pytest.mark.gpu
@pytest.mark.parametrize("size", [1, 31, 33, 256, 511, 513, 3073, 65536, 131072])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_edges(cuda, oracle, kind, size):
    from codag_b200 import api
    rng = np.random.default_rng(size)
    data = KINDS[kind](rng, max(size, 1)).tobytes()[:size]
    parts = [_stream(data, level, strategy, every)
             for level, strategy in ((0, 0), (1, 0), (9, 0), (6, zlib.Z_FIXED), (6, zlib.Z_HUFFMAN_ONLY))
             for every in (0, max(size // 7, 1), max(size // 2 - 1, 1))]
    rel = np.cumsum([0] + [len(p) for p in parts]).astype(np.int64)
    n = len(parts)
    total = n * size - size // 3  # the last chunk is cut
    out = cuda.full((total + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
    st = cuda.full((n,), -1, dtype=cuda.int32, device="cuda")
    comp = cuda.from_numpy(np.frombuffer(b"".join(parts), np.uint8).copy()).to("cuda")
    api.decompress_deflate(comp, cuda.from_numpy(rel).to("cuda"), size, out, 2, total, st)
    got = out.cpu().numpy()
    assert not st.cpu().numpy().any()
    assert np.all(got[total:] == 0xA5), "wrote past out_bytes"
    assert np.array_equal(got[:total], np.resize(np.frombuffer(data, np.uint8), total))
    for i in (0, n - 1):
        ost, ref = oracle.deflate_chunk(np.frombuffer(parts[i], np.uint8), size)
        assert ost == 0 and np.array_equal(ref[:size], np.frombuffer(data, np.uint8))
