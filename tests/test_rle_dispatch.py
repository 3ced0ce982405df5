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


def _repeat(value, nb, count):
    """SHORT_REPEAT: 1 + nb bytes, 3 to 10 values."""
    return bytes([((nb - 1) << 3) | (count - 3)]) + value.to_bytes(nb, "big"), [value] * count


def _direct16(rng, count):
    """DIRECT of 16-bit values: 2 + 2 * count bytes."""
    v = rng.integers(0, 65536, count)
    return bytes([0x5E, count - 1]) + v.astype(">u2").tobytes(), v.tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [1, 2, 4, 8])
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_rlev2_stream_length(cuda, native, elem, extra):
    """Streams of 256 bytes, of two bytes a value, and of one byte more and less; of DIRECT groups only, of some
    before another kind, and of another kind first."""
    rng = np.random.default_rng(extra + 5)
    short = [_repeat(int(v), 1, 5) for v in rng.integers(0, 256, 126 + (extra > 0))]
    short.append(_repeat(7, 1, 4) if extra == 0 else _repeat(777, 2, 4))
    short += [_repeat(9, 1, 3)] * (extra == 0)
    level = [_direct16(rng, c) for c in (200, 255, 77)]
    long = [_direct16(rng, 128) for _ in range(10)]
    level.append({-1: _repeat(500, 2, 5), 0: _repeat(50, 1, 4), 1: _repeat(500, 2, 4)}[extra])
    for parts in (short, level, level[::-1], long, long[:7] + [_repeat(5, 1, 3)] + long, [_direct16(rng, 3 + extra)] * 700):
        s, v = b"".join(p[0] for p in parts), sum((p[1] for p in parts), [])
        assert len(parts) >= 10 and parts is not short or len(s) == (256 if parts is short else 2 * len(v)) + extra
        chunk = len(v) * elem
        want = (np.array(v, np.uint64) & np.uint64((1 << 8 * elem) - 1)).astype(f"u{elem}").view(np.uint8)
        comp = np.frombuffer(s * 3, np.uint8).copy()
        out, st = _call(native, cuda, native.RLEV2, elem, comp, np.arange(3) * len(s), np.full(3, len(s)), chunk, 0, 3)()
        assert not st.cpu().numpy().any()
        assert np.array_equal(out.cpu().numpy().reshape(3, chunk), np.tile(want, (3, 1)))


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [4, 8])
def test_rlev2_incompressible(cuda, native, elem):
    """Streams as long as their chunks: a team, which reads every byte as a header, takes 1.5 and 2 times as long as
    a warp."""
    from codag_b200 import api
    chunk, n = 131072, 64
    col = np.random.default_rng(elem).integers(0, 256, n * chunk, dtype=np.uint8)
    comp, off, ln = native.encode_rlev2(col, chunk, elem)
    calls = [_call(native, cuda, native.RLEV2, elem, comp, off[:n], ln, chunk, shift, n) for shift in (0, 1)]
    out, st = calls[0]()
    assert not st.cpu().numpy().any() and np.array_equal(out.cpu().numpy(), col)
    aligned, unaligned = _best_us(cuda, *calls)
    assert aligned < 1.2 * unaligned, (aligned, unaligned)
    d = cuda.from_numpy(comp).to("cuda")
    times = []
    for shift in (0, 1):  # one file each
        cs = np.zeros(n, dtype=native.CHUNK_DESC_DTYPE)
        cs["comp_off"], cs["comp_len"], cs["codec"], cs["elem_bytes"] = off[:n], ln, native.RLEV2, elem
        cs["out_off"], cs["out_len"] = np.arange(n) * chunk + shift, chunk
        plan = api.BatchPlan(cs)
        o = cuda.zeros(n * chunk + 16, dtype=cuda.uint8, device="cuda")
        times.append((plan, lambda plan=plan, o=o: plan.run(d, o, None)))
    aligned, unaligned = _best_us(cuda, times[0][1], times[1][1])
    for plan, _ in times:
        plan.close()
    assert aligned < 1.2 * unaligned, (aligned, unaligned)
