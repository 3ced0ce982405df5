"""Which RLE streams of a batch have a whole CTA and which a single warp: the cost of a choice that does not look at
the list, as a ratio of two times taken in turn."""
import pytest

V2 = 1


def _us(cuda, a, b):
    """The best times of two calls, taken in turn."""
    best = [1e9, 1e9]
    for r in range(12):
        for i, fn in enumerate((a, b)):
            t0, t1 = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            t0.record()
            fn()
            t1.record()
            cuda.cuda.synchronize()
            if r >= 2:
                best[i] = min(best[i], t0.elapsed_time(t1) * 1e3)
    return best


@pytest.mark.gpu
def test_a_long_file_among_many(cuda, native):
    """An RLE v2 file of 8 MiB has a CTA although 450 others are longer than 32 KiB: as fast as alone, where a warp
    takes 1.35 times as long."""
    from codag_b200 import api
    big = native.gen_rlev2_column(1 << 20, 3, 8)
    small = native.gen_rlev2_column(5000, 4, 8)
    f, _, fl = native.encode_rlev2(big, big.size, 8)
    g, _, gl = native.encode_rlev2(small, small.size, 8)
    one = api.pack_chunks([f[:int(fl[0])]], [V2], [8], [big.size])
    cs = api.pack_chunks([g[:int(gl[0])]] * 450 + [f[:int(fl[0])]], [V2] * 451, [8] * 451, [small.size] * 450 + [big.size])
    plans, calls = [], []
    for c in (one, cs):
        p = api.BatchPlan(c.descs)
        comp, out = cuda.from_numpy(c.comp).to("cuda"), cuda.zeros(c.out_bytes, dtype=cuda.uint8, device="cuda")
        plans.append(p)
        calls.append(lambda p=p, comp=comp, out=out: p.run(comp, out, None))
    alone, among = _us(cuda, *calls)
    for p in plans:
        p.close()
    assert among < 1.2 * alone, (alone, among)
