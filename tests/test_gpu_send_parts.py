"""A send whose candidates go through in parts (many short reads): the same
results as the device-resident call on the whole batch, at and beside the
sizes where the number of parts changes, as a graph and as stream launches,
and a smaller send after it on the same buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["plain", "batched"])
@pytest.mark.parametrize("n", [799_999, 800_000, 1_200_001, 2_000_003])
def test_send_parts(mg, orc, cuda_ok, tmp_path, path, n):
    ref_size = 2_000_000
    words = mg.make_reference(ref_size, 5)
    w = mg.make_workload(mg.spec(ref_size, 60_000, 6, length_range=(40, 200), rate_range=(0.02, 0.08), cands=11), words)
    cands = np.resize(w["cands"], n)
    cands["position"][1::1000] = ref_size  # no window fits
    p = mg.PATH_PLAIN if path == "plain" else mg.PATH_BATCHED
    fn = tmp_path / "ref.4bits.ref"
    with open(fn, "wb") as f:
        f.write(np.array([len(words), ref_size], dtype=np.uint32).tobytes())
        f.write(words)
    ref, ctx = mg.Reference(words, ref_size), mg.Context(n)
    expect = mg.verify_torch(ctx, ref, w["peq"], w["qinfo"], cands, 0.2, path=p)
    ctx.close()
    ref.close()
    pick = np.random.default_rng(1).choice(n, 3000, replace=False)
    assert np.array_equal(expect[pick], orc.verify(w["peq"], w["qinfo"], cands[pick], words, ref_size, 0.2))
    mg.lib.myersSetMemoryBudget(64 * n + 400 * len(w["peq"]))
    with mg.Buffers(str(fn), 1, 128, 11) as bufs:
        mg.lib.myersSetMemoryBudget(0)
        bufs.set_path(p)
        for graphs in (True, True, False):
            bufs.set_graphs(graphs)
            bufs.views(0)[3][:n] = np.zeros(n, dtype=mg.RES)
            got, st = mg.verify_buffers(bufs, w["peq"], w["qinfo"], cands, 0.2)
            assert st == mg.SUCCESS and np.array_equal(got, expect)
            got, st = mg.verify_buffers(bufs, w["peq"], w["qinfo"], cands[:5000], 0.2)
            assert st == mg.SUCCESS and np.array_equal(got, expect[:5000])
