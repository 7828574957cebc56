"""Sends with empty reads before, between and after others: the results of the
batch without them, and the shapes (launches) that it takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REF = 400_000


@pytest.mark.parametrize("path", ["plain", "batched"])
@pytest.mark.parametrize("lengths", [(100, 1000), (1000,)])
def test_send_with_empty_reads(mg, orc, cuda_ok, tmp_path, path, lengths):
    words = mg.make_reference(REF, 5)
    w = mg.make_workload(mg.spec(REF, 6000, 6, lengths=max(lengths), sub=0.05, ins=0.005, dele=0.005, cands=1), words)
    size = w["qinfo"]["size"]
    for i, m in enumerate(lengths):
        size[i::len(lengths)] = m
    with_empty = w["qinfo"].copy()
    with_empty["size"][[0, 1, 2999, 3001, 5999]] = 0
    some = np.random.default_rng(1).integers(0, 6000, 60_000).astype(w["cands"]["query"].dtype)
    cands = w["cands"][some]
    p = mg.PATH_PLAIN if path == "plain" else mg.PATH_BATCHED
    fn = tmp_path / "ref.4bits.ref"
    with open(fn, "wb") as f:
        f.write(np.array([len(words), REF], dtype=np.uint32).tobytes())
        f.write(words)
    mg.lib.myersSetMemoryBudget(64 * len(cands) + 400 * len(w["peq"]))
    with mg.Buffers(str(fn), 1, 1000, 10) as bufs:
        mg.lib.myersSetMemoryBudget(0)
        bufs.set_path(p)
        full, st = mg.verify_buffers(bufs, w["peq"], w["qinfo"], cands, 0.2)
        assert st == mg.SUCCESS
        launches = mg.lib.myersBufferLastLaunches(bufs.handles[0])
        got, st = mg.verify_buffers(bufs, w["peq"], with_empty, cands, 0.2)
        assert st == mg.SUCCESS
        assert mg.lib.myersBufferLastLaunches(bufs.handles[0]) == launches
    empty = with_empty["size"][cands["query"]] == 0
    assert empty.any() and np.array_equal(got[~empty], full[~empty])
    fits = REF - cands["position"] > 0
    assert (got["column"][empty & fits] == 0).all() and (got["score"][empty & fits] == 0).all()
    pick = np.random.default_rng(2).choice(len(cands), 1500, replace=False)
    assert np.array_equal(got[pick], orc.verify(w["peq"], with_empty, cands[pick], words, REF, 0.2))
