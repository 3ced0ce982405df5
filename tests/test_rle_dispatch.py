"""RLE chunks on both sides of the rules that give a chunk a warp or a whole CTA: by their number, by the length of
their streams and by their size; and the cost of a choice that leaves one of these out, as a ratio of times taken
in turn with a call that the rules do not reach (an output that is not element aligned, always a warp each)."""
import numpy as np
import pytest

from tests import fuzz_streams as fz


def _call(native, cuda, codec, elem, comp, off, ln, chunk, shift, n):
    from codag_b200 import api
    t = lambda a: cuda.from_numpy(np.ascontiguousarray(a, dtype=np.uint64).view(np.int64)).to("cuda")
    fn = api.decompress_rlev1 if codec == native.RLEV1 else api.decompress_rlev2
    comp, off, ln = cuda.from_numpy(comp).to("cuda"), t(off), t(ln)
    buf = cuda.full((n * chunk + 16,), 0x5A, dtype=cuda.uint8, device="cuda")
    st = cuda.full((n,), -1, dtype=cuda.int32, device="cuda")
    out = buf[shift:shift + n * chunk]

    def run():
        fn(comp, off, ln, chunk, elem, out, n * chunk, st)
        return out, st
    return run


def _best_us(cuda, *calls):
    best = [1e9] * len(calls)
    for r in range(12):
        for i, fn in enumerate(calls):
            a, b = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            a.record()
            fn()
            b.record()
            cuda.cuda.synchronize()
            if r >= 2:
                best[i] = min(best[i], a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [1, 8])
@pytest.mark.parametrize("chunk", [64, 2048])
@pytest.mark.parametrize("n", [900, 901, 1100, 2600, 9000])
def test_rlev1_counts(cuda, native, n, chunk, elem):
    """64 streams, repeated."""
    comp, off, ln, want = fz.chunk_set("rlev1", 64, chunk, elem, n + elem)
    at = np.arange(n) % 64
    out, st = _call(native, cuda, native.RLEV1, elem, comp, off[at], ln[at], chunk, 0, n)()
    assert not st.cpu().numpy().any()
    assert np.array_equal(out.cpu().numpy().reshape(n, chunk), want.reshape(64, chunk)[at])


@pytest.mark.gpu
@pytest.mark.parametrize("n,chunk", [(16384, 2048), (65536, 512)])
def test_rlev1_many_small_chunks(cuda, native, n, chunk):
    """A CTA for each takes twice and 3.5 times as long as the warps of the unaligned call."""
    col = native.gen_rlev1_column(64 * chunk // 8, 3, 8)
    blob, off, ln = native.encode_rlev1(col, chunk, 8)
    at = np.arange(n) % 64
    calls = [_call(native, cuda, native.RLEV1, 8, blob[8:], off[at], ln[at], chunk, shift, n) for shift in (0, 1)]
    out, st = calls[0]()
    assert not st.cpu().numpy().any()
    assert np.array_equal(out.cpu().numpy().reshape(n, chunk), col.reshape(64, chunk)[at])
    aligned, unaligned = _best_us(cuda, *calls)
    assert aligned < 1.25 * unaligned, (aligned, unaligned)
