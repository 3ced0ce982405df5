"""RLE decode on both sides of the chunk count from which RLE v2 chunks are taken in groups of eight
instead of by a CTA each (444 chunks), with a last group that is not full and a last chunk that is
cut, over random streams of every header form, and the statuses of malformed chunks among good ones."""
import numpy as np
import pytest

from tests import fuzz_streams as fz

CODECS = {"rlev1": 0, "rlev2": 1}


def _decode(cuda, codec, comp, off, ln, cb, elem, total):
    from codag_b200 import api
    t = lambda a: cuda.from_numpy(a.astype(np.uint64).view(np.int64)).to("cuda")
    out = cuda.full((total + 64,), 0xA5, dtype=cuda.uint8, device="cuda")
    st = cuda.full((ln.size,), -1, dtype=cuda.int32, device="cuda")
    fn = api.decompress_rlev1 if codec == "rlev1" else api.decompress_rlev2
    fn(cuda.from_numpy(comp).to("cuda"), t(off), t(ln), cb, elem, out, total, st)
    o = out.cpu().numpy()
    assert np.all(o[total:] == 0xA5), "wrote past out_bytes"
    return st.cpu().numpy(), o[:total]


@pytest.mark.gpu
@pytest.mark.parametrize("elem,cb", [(1, 2048), (2, 6002), (4, 4100), (8, 16384), (8, 8)])
@pytest.mark.parametrize("n", [444, 445, 451])
@pytest.mark.parametrize("codec", ["rlev1", "rlev2"])
def test_counts(cuda, codec, n, elem, cb):
    # the streams repeat after 40 chunks: writing them is the slow part
    comp, off, ln, want = fz.chunk_set(codec, 40, cb, elem, seed=7 * n + elem)
    pick = np.arange(n) % 40
    want = want.reshape(40, cb)[pick].reshape(-1)
    total = n * cb - (cb // elem // 3) * elem
    st, out = _decode(cuda, codec, comp, off[pick], ln[pick], cb, elem, total)
    assert not st.any()
    assert np.array_equal(out, want[:total])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [444, 451])
@pytest.mark.parametrize("codec", ["rlev1", "rlev2"])
def test_malformed_among_good(cuda, oracle, codec, n):
    cb, elem = 16384, 8
    comp, off, ln, want = fz.chunk_set(codec, 40, cb, elem, seed=n)
    pick = np.arange(n) % 40
    off, ln = off[pick], ln[pick].copy()
    ln[5] = 0
    ln[17] //= 2
    ln[18] -= 1
    off[30] = comp.size
    st, out = _decode(cuda, codec, comp, off, ln, cb, elem, n * cb)
    bad = np.array([5, 17, 18, 30])
    good = np.setdiff1d(np.arange(n), bad)
    assert np.all(st[bad] == 2) and not st[good].any()
    assert np.array_equal(out.reshape(n, cb)[good], want.reshape(40, cb)[pick][good])
