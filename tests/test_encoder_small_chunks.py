"""GPU encoders with so many small chunks that each has a CTA of one warp: chunks of a few values, at the edges of its
tile of 256, up to the 2048 values above which, and down to the numbers of chunks below which, the others take them.
The files equal the host producers' byte for byte; and what they cost, as a multiple of a device copy of the column."""
import numpy as np
import pytest

from tests.test_encoder_tile_edges import _values


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["runs", "literals", "patches"])
@pytest.mark.parametrize("chunk", [1, 2, 3, 31, 127, 128, 129, 255, 256, 257, 383, 513, 1000, 2047, 2048, 2049])
@pytest.mark.parametrize("codec", [0, 1], ids=["rlev1", "rlev2"])
def test_chunks(cuda, native, codec, chunk, mode):
    from codag_b200 import api
    if codec == native.RLEV1 and chunk == 1:
        pytest.skip("a chunk of RLE v1 has two values at least")
    chunks = -(-max(297, (6 if codec else 1) * chunk) // 32) * 32
    for e in (1, 2, 4, 8):
        for n in (chunks, chunks - 32):  # on both sides of the rule
            if n * chunk * e > 26 << 20:
                continue
            dt = {1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[e]
            count = n * chunk - chunk // 2  # the last chunk is short
            raw = np.resize(_values(np.random.default_rng(7 * chunk + e), min(count, 300000), mode), count).astype(dt).view(np.uint8)
            want, w_off, w_len = (native.encode_rlev2 if codec else native.encode_rlev1)(raw, chunk * e, e)
            f, off, ln = api.compress_rle(codec, cuda.from_numpy(raw.copy()).to("cuda"), chunk * e, e)
            assert np.array_equal(ln.cpu().numpy().view(np.uint64), w_len), (e, n)
            assert np.array_equal(off.cpu().numpy().view(np.uint64), w_off), (e, n)
            assert np.array_equal(f.cpu().numpy(), want), (e, n)


@pytest.mark.gpu
@pytest.mark.parametrize("codec", [0, 1], ids=["rlev1", "rlev2"])
def test_cost(cuda, native, codec):
    """65536 chunks of 64 values: a CTA of 16 warps for each takes 100 and 160 times as long as a copy."""
    lib, size, chunk = native.lib(), 32 << 20, 512
    raw = np.random.default_rng(1).integers(0, 256, size, dtype=np.uint8)
    n = int(lib.codag_compress_chunks(size, chunk))
    need = int(lib.codag_compress_workspace_bytes(codec, size, chunk, 8))
    col, ws = cuda.from_numpy(raw).to("cuda"), cuda.empty(need, dtype=cuda.uint8, device="cuda")
    out = cuda.zeros(int(lib.codag_compress_bound(codec, size, chunk, 8)), dtype=cuda.uint8, device="cuda")
    off, ln, meta = (cuda.zeros(k, dtype=cuda.int64, device="cuda") for k in (n + 1, n, 2))
    to = cuda.empty_like(col)
    fn = lib.codag_compress_rlev2 if codec else lib.codag_compress_rlev1

    def encode():
        native.check("compress", fn(col.data_ptr(), size, chunk, 8, out.data_ptr(), out.numel(), off.data_ptr(), ln.data_ptr(),
                                    meta.data_ptr(), meta.data_ptr() + 8, ws.data_ptr(), need, None))

    best = [1e9, 1e9]
    for r in range(10):
        for i, call in enumerate((encode, lambda: to.copy_(col))):
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            cuda.cuda.synchronize()
            if r >= 2:
                best[i] = min(best[i], a.elapsed_time(b))
    assert best[0] < 60 * best[1], best
