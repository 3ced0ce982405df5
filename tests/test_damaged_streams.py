"""Damaged streams against independent decoders: Deflate chunks on a team, on a warp and by zlib; RLE chunks on a CTA,
on a warp in every launch shape, in a batch and by the oracle.

zlib refuses Deflate code sets that leave codes unused, which the GPU decoders accept; on everything else
they agree, in what they refuse and in the bytes of what they take."""
import zlib

import numpy as np
import pytest

from tests import fuzz_streams as fz
from tests.test_deflate_fuzz import _chunk

CH = 131072


def _by_zlib(s, size):
    """(status or None where zlib refuses a code set, bytes)"""
    d = zlib.decompressobj(-15)
    try:
        out = d.decompress(s, size + 1)
    except zlib.error as e:
        return (None if " set" in str(e) else 2), b""
    return (0 if d.eof and len(out) == size else 2), out


def _damage(rng, s):
    s = bytearray(s)
    kind = int(rng.integers(0, 6))
    if kind < 3:  # a few bytes changed, anywhere or in the first header
        for p in rng.integers(0, len(s) if kind else min(len(s), 80), int(rng.integers(1, 4))):
            s[p] ^= int(rng.integers(1, 256))
    elif kind == 3:  # one bit
        p = int(rng.integers(0, len(s)))
        s[p] ^= 1 << int(rng.integers(0, 8))
    elif kind == 4 and len(s) > 8:  # cut
        s = s[:int(rng.integers(1, len(s)))]
    return bytes(s)


def _plan(cuda, native, streams, codec, elem, sizes):
    from codag_b200 import api
    n = len(streams)
    cs = api.pack_chunks([np.frombuffer(s, np.uint8) for s in streams], [codec] * n, [elem] * n, sizes, 0)
    out = cuda.zeros(cs.out_bytes, dtype=cuda.uint8, device="cuda")
    st = cuda.full((n,), -1, dtype=cuda.int32, device="cuda")
    plan = api.BatchPlan(cs.descs)
    plan.run(cuda.from_numpy(cs.comp).to("cuda"), out, st)
    got = out.cpu().numpy()
    plan.close()
    return st.cpu().numpy(), [got[int(d["out_off"]):int(d["out_off"]) + int(d["out_len"])] for d in cs.descs]


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(6))
def test_deflate_teams(cuda, native, seed):
    rng = np.random.default_rng(1000 + seed)
    text = native.gen_text(4 * CH, seed)
    streams = []
    for c in range(60):
        data = _chunk(rng, c % 3) if c % 2 else text[c % 4 * CH:][:CH]
        co = zlib.compressobj(int(rng.integers(0, 10)), zlib.DEFLATED, -15, int(rng.integers(1, 10)), int(rng.choice([0, 0, 1, 2, 3, 4])))
        streams.append(_damage(rng, co.compress(data.tobytes()) + co.flush()))
    st, got = _plan(cuda, native, streams, native.DEFLATE, 1, [CH] * 60)
    seen = set()
    for s, status, g in zip(streams, st, got):
        want, ref = _by_zlib(s, CH)
        seen.add(want)
        assert status == want or (want is None and status in (0, 2))
        assert want != 0 or bytes(g) == ref
    assert {0, 2} <= seen


@pytest.mark.gpu
@pytest.mark.parametrize("size", [300, 1500, 3000])
def test_deflate_teams_and_warps(cuda, native, size):
    """Few chunks have teams, many of the same a warp each: one status, and the same bytes where it is good."""
    rng = np.random.default_rng(size)
    text, column = native.gen_text(200 * size, 9), native.gen_rlev2_column(200 * size // 4, 9, 4)
    streams = []
    for c in range(400):
        data = (text if c % 2 else column)[c // 2 * size:][:size]
        co = zlib.compressobj(int(rng.integers(0, 10)), zlib.DEFLATED, -15, 9, int(rng.choice([0, 0, 0, 2, 4])))
        streams.append(_damage(rng, co.compress(data.tobytes()) + co.flush()))
    st, got = _plan(cuda, native, streams, native.DEFLATE, 1, [size] * 400)
    st_many, got_many = _plan(cuda, native, streams * 24, native.DEFLATE, 1, [size] * 9600)
    seen = set()
    for i, s in enumerate(streams):
        want, ref = _by_zlib(s, size)
        seen.add(want)
        assert np.all(st_many[i::400] == st[i]), i
        assert st[i] == want or (want is None and st[i] in (0, 2)), i
        if st[i] == 0:
            assert all(np.array_equal(g, got[i]) for g in got_many[i::400]), i
            assert want is None or bytes(got[i]) == ref, i
    assert seen == {0, 2, None}


def _rle_set(codec, elem, cb, seed):
    """64 chunks, half of them damaged: streams, their offsets and lengths."""
    rng = np.random.default_rng(seed)
    comp, off, ln, _ = fz.chunk_set(codec, 64, cb, elem, seed)
    parts = [comp[int(o):int(o + n)].tobytes() for o, n in zip(off, ln)]
    parts = [_damage(rng, p) if i % 2 else p for i, p in enumerate(parts)]
    lens = np.array([len(p) for p in parts], np.uint64)
    offs = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint64)
    return np.frombuffer(b"".join(parts) + b"\0" * 16, np.uint8).copy(), offs, lens


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [1, 2, 4, 8])
@pytest.mark.parametrize("codec", ["rlev1", "rlev2"])
@pytest.mark.parametrize("cb,n", [(2048, 64), (512, 2048), (32768, 64)])
def test_rle(cuda, native, oracle, codec, elem, cb, n):
    """64 chunks have a CTA each, 2048 small ones a warp each in every launch shape."""
    from codag_b200 import api
    cid = native.RLEV1 if codec == "rlev1" else native.RLEV2
    comp, off, ln = _rle_set(codec, elem, cb, 50 * elem + cb + cid)
    ref = np.zeros(64 * cb, np.uint8)
    want = oracle.decode_batch(comp, off, ln, ref, np.arange(64) * cb, [cb] * 64, [cb] * 64, [cid] * 64, [elem] * 64, [0] * 64)
    assert want.any() and not want.all()
    reps = n // 64
    base = np.repeat(np.arange(reps, dtype=np.uint64) * np.uint64(comp.size), 64)
    t = lambda a: cuda.from_numpy(np.ascontiguousarray(a).view(np.int64)).to("cuda")
    d_comp, d_off, d_len = cuda.from_numpy(np.tile(comp, reps)).to("cuda"), t(np.tile(off, reps) + base), t(np.tile(ln, reps))
    fn = api.decompress_rlev1 if cid == native.RLEV1 else api.decompress_rlev2
    shapes = [(w, s, 0) for w in (1, 2, 4, 8) for s in (4, 8)] if n > 64 else [(8, 4, 0)]
    old = native.get_tune(cid)
    try:
        for warps, slots, cta in shapes + [(8, 4, 1)]:
            native.set_tune(cid, warps, slots, old.lut_bits, cta)
            out = cuda.zeros(n * cb, dtype=cuda.uint8, device="cuda")
            st = cuda.full((n,), -1, dtype=cuda.int32, device="cuda")
            fn(d_comp, d_off, d_len, cb, elem, out, n * cb, st)
            got, status = out.cpu().numpy().reshape(n, cb), st.cpu().numpy()
            assert np.array_equal(status, np.tile(want, reps)), (warps, slots, cta)
            good = np.flatnonzero(status == 0)
            assert np.array_equal(got[good], ref.reshape(64, cb)[good % 64]), (warps, slots, cta)
    finally:
        native.set_tune(cid, old.warps_per_cta, old.ring_slots, old.lut_bits, old.cta_per_chunk)
