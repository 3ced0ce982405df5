"""Batch plans whose RLE files lie on both sides of the size from which a whole CTA takes one (32 KiB),
with more long RLE v2 files than CTAs (all by single warps) and with few, one much longer file (fewer
CTAs), files of every header form whose outputs are not element aligned, and damaged ones; and the
launch without a plan, where CTAs take every file."""
import numpy as np
import pytest

from tests import fuzz_streams as fz

SIZES = {0: [8, 32768 - 8, 32768, 32768 + 8, 70000], 1: [16, 32760, 32768, 32776, 65536]}


def _set(native, rng, shift, long_v2):
    """Files of RLE v1 and v2 (one of each width and size) and of Deflate: descriptors, streams, outputs."""
    import zlib
    files = []
    for codec, name in ((native.RLEV1, "rlev1"), (native.RLEV2, "rlev2")):
        for e in (1, 2, 4, 8):
            for size in SIZES[codec] + ([40000] * (long_v2 if name == "rlev2" and e == 8 else 0)):
                comp, _, ln, want = fz.chunk_set(name, 1, size // e * e, e, int(rng.integers(1 << 30)))
                files.append((codec, e, 0, comp[:int(ln[0])], want))
    for size in (1, 5000, 70000, 400000):
        d = native.gen_text(size, size)
        files.append((native.DEFLATE, 1, 2, np.frombuffer(zlib.compress(d.tobytes(), 6), np.uint8), d))
    descs = np.zeros(len(files), dtype=native.CHUNK_DESC_DTYPE)
    comp, out, cpos, opos = [], [], 0, shift
    for d, (codec, e, wrapper, s, want) in zip(descs, files):
        d["codec"], d["elem_bytes"], d["wrapper_bytes"] = codec, e, wrapper
        d["comp_off"], d["comp_len"], d["out_off"], d["out_len"] = cpos, s.size, opos, want.size
        pad = -s.size % 16
        comp += [s, np.zeros(pad, np.uint8)]
        cpos += s.size + pad
        opad = -want.size % 256
        out += [want, np.zeros(opad, np.uint8)]
        opos += want.size + opad
    return descs, np.concatenate(comp), np.concatenate([np.zeros(shift, np.uint8)] + out)


@pytest.mark.gpu
@pytest.mark.parametrize("planned", [True, False])
@pytest.mark.parametrize("shift,long_v2", [(0, 0), (0, 460), (3, 0)])
def test_files(cuda, native, shift, long_v2, planned):
    from codag_b200 import api
    rng = np.random.default_rng(10 * shift + long_v2)
    descs, comp, want = _set(native, rng, shift, 0)
    if long_v2:  # the same stream many times
        k = int(np.flatnonzero((descs["codec"] == native.RLEV2) & (descs["out_len"] > 32768))[0])
        more = np.repeat(descs[k:k + 1], long_v2)
        step = -(-int(descs[k]["out_len"]) // 256) * 256
        more["out_off"] = want.size + step * np.arange(long_v2)
        src = want[int(descs[k]["out_off"]):][:int(descs[k]["out_len"])]
        want = np.concatenate([want] + [src, np.zeros(step - src.size, np.uint8)] * long_v2)
        descs = np.concatenate([descs, more])
    descs = descs.copy()
    bad = np.flatnonzero((descs["codec"] != native.DEFLATE) & (descs["comp_len"] > 64))[::7]
    descs["comp_len"][bad] -= 9
    n = descs.size
    d_comp = cuda.from_numpy(comp).to("cuda")
    out = cuda.zeros(want.size, dtype=cuda.uint8, device="cuda")
    st = cuda.full((n,), -1, dtype=cuda.int32, device="cuda")
    if planned:
        plan = api.BatchPlan(descs)
        plan.run(d_comp, out, st)
        cuda.cuda.synchronize()
        plan.close()
    else:
        d_descs = cuda.from_numpy(descs.view(np.uint8).reshape(-1).copy()).to("cuda")
        queue = cuda.zeros(1, dtype=cuda.int32, device="cuda")
        native.check("codag_batch_launch", native.lib().codag_batch_launch(
            d_descs.data_ptr(), None, n, queue.data_ptr(), None, d_comp.data_ptr(), d_comp.numel(), out.data_ptr(),
            out.numel(), st.data_ptr(), cuda.cuda.current_stream().cuda_stream or None))
        cuda.cuda.synchronize()
    status, got = st.cpu().numpy(), out.cpu().numpy()
    good = np.setdiff1d(np.arange(n), bad)
    assert np.all(status[bad] == 2) and not status[good].any()
    for d in descs[good]:
        o, ln = int(d["out_off"]), int(d["out_len"])
        assert np.array_equal(got[o:o + ln], want[o:o + ln]), d
