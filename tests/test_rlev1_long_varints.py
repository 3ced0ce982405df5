"""RLE v1 literals whose varints are padded to 16, 17, 127 and 128 bytes decode, and those of 129, 200 and 3000 bytes
are refused, whichever decoder takes the stream: the CTA per chunk, the warp with its output in a ring, the two
passes with a workspace, and the batch with the stream on a CTA or on a warp."""
import numpy as np
import pytest

from tests.fuzz_streams import uleb

VALUES = 8300  # 64-bit values: more than the 32 KiB up to which a plan gives a file one warp


def _stream(length, values, at):
    """Groups of 100 literals; value `at` is a varint of `length` bytes."""
    s, vals = bytearray(), []
    for i in range(values):
        if i % 100 == 0:
            s.append((-min(100, values - i)) & 0xFF)
        v = 7 * i + 1
        if i == at:
            s += bytes([(v & 0x7F) | 0x80, (v >> 7 & 0x7F) | 0x80, (v >> 14 & 0x7F) | 0x80]) + b"\x80" * (length - 4) + b"\0"
        else:
            s += uleb(v)
        vals.append(v)
    return np.frombuffer(bytes(s), np.uint8).copy(), np.array(vals, np.uint64).view(np.uint8)


def test_oracle_takes_any_length(oracle):
    for length in (16, 128, 200):
        s, want = _stream(length, 900, 333)
        st, out = oracle.rlev1_chunk(s, want.size, 8)
        assert st == 0 and np.array_equal(out, want)


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0, 99, 333])
@pytest.mark.parametrize("length", [16, 17, 127, 128, 129, 200, 3000])
def test_every_decoder_agrees(cuda, native, length, at):
    from codag_b200 import api
    good = length <= 128
    s, want = _stream(length, VALUES, at)
    chunk = want.size
    comp = cuda.from_numpy(s).to("cuda")
    off = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    ln = cuda.tensor([s.size], dtype=cuda.int64, device="cuda")
    for name, shift, ws in (("team", 0, None), ("ring", 3, None), ("two passes", 0, api.AUTO_WORKSPACE)):
        out = cuda.zeros(chunk + 8, dtype=cuda.uint8, device="cuda")[shift:shift + chunk]
        st = cuda.full((1,), -1, dtype=cuda.int32, device="cuda")
        api.decompress_rlev1(comp, off, ln, chunk, 8, out, chunk, st, ws=ws)
        assert st.item() == (0 if good else 2), name
        assert not good or np.array_equal(out.cpu().numpy(), want), name
    for values in (900, VALUES):
        s, want = _stream(length, values, at)
        cs = api.pack_chunks([s], [native.RLEV1], [8], [want.size])
        out = cuda.zeros(cs.out_bytes, dtype=cuda.uint8, device="cuda")
        st = cuda.full((1,), -1, dtype=cuda.int32, device="cuda")
        plan = api.BatchPlan(cs.descs)
        plan.run(cuda.from_numpy(cs.comp).to("cuda"), out, st)
        assert st.item() == (0 if good else 2), values
        assert not good or np.array_equal(out.cpu().numpy()[:want.size], want), values
        plan.close()
