"""Which streams of a batch have a whole CTA and which a single warp, planned or not: lists in which the two
kinds alternate, stand apart or leave one kind out, in both orders; and the cost of a choice that does not look at
the list, as a ratio of two times taken in turn."""
import numpy as np
import pytest

from tests import fuzz_streams as fz

KIB = 1 << 10


def _files(native, cuda, spec, seed=1):
    """spec: (codec, elem, size) per file; a few streams of each kind, repeated.  (descs, comp, outputs)"""
    from codag_b200 import api
    rng = np.random.default_rng(seed)
    made = {}
    streams, wants = [], []
    for i, (codec, elem, size) in enumerate(spec):
        key = (codec, elem, size, i % 3)
        if key not in made:
            if codec == native.DEFLATE:
                raw = native.gen_text(size, int(rng.integers(1 << 20)))
                made[key] = native.encode_one(codec, raw), raw
            else:
                comp, _, ln, want = fz.chunk_set("rlev1" if codec == native.RLEV1 else "rlev2", 1, size, elem,
                                                 int(rng.integers(1 << 30)))
                made[key] = comp[:int(ln[0])], want
        streams.append(made[key][0])
        wants.append(made[key][1])
    cs = api.pack_chunks(streams, [f[0] for f in spec], [f[1] for f in spec], [f[2] for f in spec])
    return cs, wants


def _launch(native, cuda, descs, order, comp, out, st):
    q = cuda.zeros(1, dtype=cuda.int32, device="cuda")
    d = cuda.from_numpy(descs.view(np.uint8).reshape(-1).copy()).to("cuda")
    o = None if order is None else cuda.from_numpy(order.astype(np.int32)).to("cuda")
    keep = (q, d, o)

    def run():
        native.check("codag_batch_launch", native.lib().codag_batch_launch(
            d.data_ptr(), None if o is None else o.data_ptr(), descs.size, q.data_ptr(), None, comp.data_ptr(),
            comp.numel(), out.data_ptr(), out.numel(), st.data_ptr(), cuda.cuda.current_stream().cuda_stream or None))
        return keep
    return run


V1, V2, DEF = 0, 1, 2
LISTS = {
    "one": [(V2, 8, 512)],
    "warps only": [(V2, 4, 1024)] * 700 + [(V1, 8, 2048)] * 700,
    "teams only": [(DEF, 1, 3000)] * 300 + [(V1, 4, 40000)] * 3,
    "a team at the end": [(V2, 8, 256)] * 5000 + [(DEF, 1, 5000)],
    "a team at the start": [(DEF, 1, 5000)] + [(V2, 8, 256)] * 5000,
    "far apart": ([(DEF, 1, 2000)] + [(V1, 2, 512)] * 1600) * 3,
    "in turn": [(DEF, 1, 2000), (V2, 8, 512), (V1, 4, 33000), (V2, 2, 40000)] * 120,
    "small deflate": [(DEF, 1, 700)] * 9000,
    "small deflate and others": [(DEF, 1, 700)] * 9000 + [(V2, 8, 512), (DEF, 1, 70000), (V1, 4, 33000), (V2, 8, 40000)] * 30,
    "small deflate, too few": [(DEF, 1, 700)] * 100 + [(V1, 8, 512)] * 100,
    "many long v2, one longest": [(V2, 8, 40000)] * 460 + [(V2, 8, 800000)],
}


@pytest.mark.gpu
@pytest.mark.parametrize("base", [0, 1])
@pytest.mark.parametrize("name", sorted(LISTS))
def test_lists(cuda, native, name, base):
    cs, wants = _files(native, cuda, LISTS[name])
    n = cs.descs.size
    comp = cuda.from_numpy(cs.comp).to("cuda")
    rng = np.random.default_rng(n)
    from codag_b200 import api
    for how in ("launch", "launch, any order", "plan", "plan, graph"):
        buf = cuda.full((cs.out_bytes + 8,), 0x5A, dtype=cuda.uint8, device="cuda")
        out = buf[base:base + cs.out_bytes]
        st = cuda.full((n,), -1, dtype=cuda.int32, device="cuda")
        if how.startswith("launch"):
            run = _launch(native, cuda, cs.descs, rng.permutation(n) if "order" in how else None, comp, out, st)
            for _ in range(2):
                run()
            cuda.cuda.synchronize()
        else:
            plan = api.BatchPlan(cs.descs)
            for _ in range(2):
                plan.run(comp, out, st, use_graph="graph" in how)
            cuda.cuda.synchronize()
            plan.close()
        assert not st.cpu().numpy().any(), how
        got = out.cpu().numpy()
        for d, want in zip(cs.descs, wants):
            o = int(d["out_off"])
            assert np.array_equal(got[o:o + want.size], want), (how, d)


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
@pytest.mark.parametrize("count,size", [(2048, 128 * KIB), (20000, 4 * KIB)])
def test_launch_is_as_fast_as_a_plan(cuda, native, count, size):
    """RLE v2 files that a plan gives a warp each; a CTA each takes 2.3 and 4.8 times as long."""
    from codag_b200 import api
    col = native.gen_rlev2_column(size // 8, 3, 8)
    f, _, ln = native.encode_rlev2(col, size, 8)
    cs = api.pack_chunks([f[:int(ln[0])]] * count, [V2] * count, [8] * count, [size] * count)
    comp = cuda.from_numpy(cs.comp).to("cuda")
    out = cuda.zeros(cs.out_bytes, dtype=cuda.uint8, device="cuda")
    st = cuda.full((count,), -1, dtype=cuda.int32, device="cuda")
    plan = api.BatchPlan(cs.descs)
    launched, planned = _us(cuda, _launch(native, cuda, cs.descs, None, comp, out, st), lambda: plan.run(comp, out, st))
    plan.close()
    assert not st.cpu().numpy().any()
    assert launched < 1.5 * planned, (launched, planned)


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


@pytest.mark.gpu
@pytest.mark.parametrize("planned", [True, False])
def test_rlev1_files_of_32_kib(cuda, native, planned):
    """3000 RLE v1 files of exactly 32 KiB take what as many of 33 KiB take; with a warp each, 1.6 times as long."""
    from codag_b200 import api
    calls, keep = [], []
    for size in (32 * KIB, 33 * KIB):
        col = native.gen_rlev1_column(size, 3, 1)
        blob, _, ln = native.encode_rlev1(col, size, 1)
        cs = api.pack_chunks([blob[8:8 + int(ln[0])]] * 3000, [V1] * 3000, [1] * 3000, [size] * 3000)
        comp, out = cuda.from_numpy(cs.comp).to("cuda"), cuda.zeros(cs.out_bytes, dtype=cuda.uint8, device="cuda")
        st = cuda.full((3000,), -1, dtype=cuda.int32, device="cuda")
        if planned:
            plan = api.BatchPlan(cs.descs)
            keep.append(plan)
            calls.append(lambda plan=plan, comp=comp, out=out, st=st: plan.run(comp, out, st))
        else:
            calls.append(_launch(native, cuda, cs.descs, None, comp, out, st))
        calls[-1]()
        assert not st.cpu().numpy().any() and np.array_equal(out.cpu().numpy()[:size], col)
    at, above = _us(cuda, *calls)
    for plan in keep:
        plan.close()
    assert at < 1.2 * above, (at, above)
