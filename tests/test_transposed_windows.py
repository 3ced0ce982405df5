"""RLE v2 in the transposed layout where the decoder's 16-byte header window and 64-bit bit buffer meet the
end of a substream: chunks of 1 to 70 values a lane, of every header kind the writer emits, for every
element width, with the last chunk short."""
import numpy as np
import pytest

from tests.rlev2_walk import detranspose, interleave_values


@pytest.mark.gpu
@pytest.mark.parametrize("e,ru", [(8, 1), (4, 2), (2, 1), (1, 4)])
@pytest.mark.parametrize("per_lane", [1, 2, 3, 10, 11, 70])
def test_short_substreams(cuda, native, oracle, e, ru, per_lane):
    from codag_b200 import api
    rng = np.random.default_rng(100 * per_lane + e)
    chunk = 32 * per_lane * ru * e
    n = 32 * per_lane * ru * 5 - 7
    dt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[e]
    kinds = [np.full(n, 77, np.uint64), np.arange(n, dtype=np.uint64) * np.uint64(5),
             rng.integers(0, 1 << 63, n, dtype=np.uint64) >> rng.integers(0, 63, n, dtype=np.uint64),
             rng.integers(0, 100, n, dtype=np.uint64) + (rng.random(n) < 0.05).astype(np.uint64) * np.uint64(1 << 40),
             np.cumsum(rng.integers(0, 9, n, dtype=np.uint64))]
    for v in kinds:
        raw = v.astype(dt).view(np.uint8)
        comp, off, ln = native.encode_rlev2_transposed(raw, chunk, e, ru)
        m = off.size - 1
        out = cuda.full((raw.size + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
        st = cuda.full((m,), -1, dtype=cuda.int32, device="cuda")
        t = lambda a: cuda.from_numpy(np.ascontiguousarray(a).astype(np.uint64).view(np.int64)).to("cuda")
        api.decompress_rlev2_transposed(cuda.from_numpy(comp).to("cuda"), t(off[:m]), t(ln), chunk, e, ru, out, raw.size, st)
        got, status = out.cpu().numpy(), st.cpu().numpy()
        assert np.all(got[raw.size:] == 0xA5)
        for c in range(m):
            parts = [oracle.rlev2_chunk(np.frombuffer(s, np.uint8), per_lane * ru * e, e)
                     for s in detranspose(comp[int(off[c]):], ln[32 * c:32 * c + 32])]
            want = np.frombuffer(interleave_values([v.tobytes() for _, v in parts], ru, e), np.uint8)
            size = min(chunk, raw.size - c * chunk)
            assert status[c] == 0 and not any(x for x, _ in parts)
            assert np.array_equal(got[c * chunk:c * chunk + size], want[:size])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [592, 593])
@pytest.mark.parametrize("e,ru", [(8, 1), (2, 4)])
def test_warps_of_a_chunk(cuda, native, oracle, e, ru, n):
    """Both sides of the chunk count up to which four warps share a chunk's substreams; one substream of
    every warp is damaged in some chunk, and only those chunks report it."""
    from codag_b200 import api
    rng = np.random.default_rng(n)
    chunk = 32 * 24 * e
    dt = {2: np.uint16, 8: np.uint64}[e]
    raw = np.cumsum(rng.integers(0, 3, n * 32 * 24 - 11, dtype=np.uint64)).astype(dt)
    raw[::97] = rng.integers(0, 1 << 15, raw[::97].size)
    raw = raw.view(np.uint8)
    comp, off, ln = native.encode_rlev2_transposed(raw, chunk, e, ru)
    ln = ln.copy()
    m = off.size - 1
    bad = {7 + 40 * k: 4 * k + 1 for k in range(8)}  # chunk: its substream whose last byte is missing
    for c, t in bad.items():
        # only where no other substream has a word in that row does the layout of the rest stay as it was
        ln[32 * c + t] -= 1 if int(ln[32 * c + t]) % 4 != 1 else 0
    good = [c for c in range(m) if c not in bad]
    out = cuda.full((raw.size + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
    st = cuda.full((m,), -1, dtype=cuda.int32, device="cuda")
    t64 = lambda a: cuda.from_numpy(np.ascontiguousarray(a).astype(np.uint64).view(np.int64)).to("cuda")
    api.decompress_rlev2_transposed(cuda.from_numpy(comp).to("cuda"), t64(off[:m]), t64(ln), chunk, e, ru, out, raw.size, st)
    got, status = out.cpu().numpy(), st.cpu().numpy()
    assert np.all(got[raw.size:] == 0xA5)
    for c in range(m):
        parts = [oracle.rlev2_chunk(np.frombuffer(s, np.uint8), 24 * e, e)
                 for s in detranspose(comp[int(off[c]):], ln[32 * c:32 * c + 32])]
        fine = not any(x for x, _ in parts)
        assert (status[c] == 0) == fine, c
        assert fine or c in bad
        if c in good:
            want = np.frombuffer(interleave_values([v.tobytes() for _, v in parts], ru, e), np.uint8)
            size = min(chunk, raw.size - c * chunk)
            assert np.array_equal(got[c * chunk:c * chunk + size], want[:size]), c
