"""GPU encoders at the edges of their tiles (3072 values): runs, literal groups and packed headers that
start, end and are cut there, chunks of a few values and chunks one value longer or shorter than a
tile.  The files equal the host producers' byte for byte."""
import numpy as np
import pytest


def _values(rng, n, mode):
    if mode == "runs":  # constant and stepped runs of every length around the headers' limits, off the tile's grid
        parts, size = [], 0
        while size < n:
            ln = int(rng.choice([1, 2, 3, 4, 9, 10, 11, 127, 128, 129, 130, 131, 132, 255, 256, 257, 511, 513, 2047, 2049]))
            parts.append(int(rng.integers(0, 1 << 40)) + np.arange(ln, dtype=np.uint64) * np.uint64(rng.choice([0, 0, 1, 3, 127, 128, 500])))
            size += ln
        return np.concatenate(parts)[:n]
    if mode == "literals":  # no two steps alike, of every width
        return rng.integers(0, 1 << 63, n, dtype=np.uint64) >> rng.integers(0, 63, n, dtype=np.uint64)
    v = rng.integers(0, 200, n, dtype=np.uint64)  # small values with a few large ones: patched headers
    v[rng.random(n) < 0.03] += np.uint64(1 << 33)
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["runs", "literals", "patches"])
@pytest.mark.parametrize("chunk", [1, 2, 3, 129, 2047, 2048, 2049, 3071, 3072, 3073, 6145, 16384])
@pytest.mark.parametrize("codec", [0, 1], ids=["rlev1", "rlev2"])
def test_tile_edges(cuda, native, codec, chunk, mode):
    from codag_b200 import api
    for e in (1, 2, 4, 8):
        n = max(3 * chunk, 5000) + 1  # the last chunk is short
        dt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[e]
        raw = _values(np.random.default_rng(100 * chunk + e), n, mode).astype(dt).view(np.uint8)
        encode = native.encode_rlev1 if codec == native.RLEV1 else native.encode_rlev2
        if codec == native.RLEV1 and chunk == 1:  # refused: a chunk of RLE v1 has two values at least
            with pytest.raises(native.CodagError):
                encode(raw, chunk * e, e)
            with pytest.raises(native.CodagError):
                api.compress_rle(codec, cuda.from_numpy(raw.copy()).to("cuda"), chunk * e, e)
            continue
        want, w_off, w_len = encode(raw, chunk * e, e)
        f, off, ln = api.compress_rle(codec, cuda.from_numpy(raw.copy()).to("cuda"), chunk * e, e)
        assert np.array_equal(ln.cpu().numpy().view(np.uint64), w_len), e
        assert np.array_equal(off.cpu().numpy().view(np.uint64), w_off), e
        assert np.array_equal(f.cpu().numpy(), want), e
