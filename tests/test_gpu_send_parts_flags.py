"""A send in parts launches the kernels of each part, and a candidate that is
refused in the first part is still reported by the receive, which reads the
flags once, after the last part."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REF = 500_000


@pytest.mark.parametrize("path", ["plain", "batched"])
@pytest.mark.parametrize("lengths", [dict(lengths=100, sub=0.04), dict(lengths=[64, 100, 180], length_weights=[1, 1, 1])])
def test_parts_and_flags(mg, cuda_ok, tmp_path, path, lengths):
    words = mg.make_reference(REF, 5)
    w = mg.make_workload(mg.spec(REF, 20_000, 6, cands=11, **lengths), words)
    fn = tmp_path / "ref.4bits.ref"
    with open(fn, "wb") as f:
        f.write(np.array([len(words), REF], dtype=np.uint32).tobytes())
        f.write(words)
    n = 1_640_000
    mg.lib.myersSetMemoryBudget(64 * n + 400 * len(w["peq"]))
    with mg.Buffers(str(fn), 1, 128, 11) as bufs:
        mg.lib.myersSetMemoryBudget(0)
        bufs.set_path(mg.PATH_PLAIN if path == "plain" else mg.PATH_BATCHED)
        launches = {}
        for parts in (1, 2, 3, 4):  # of 410,000 candidates each
            cands = np.resize(w["cands"], 410_000 * parts)
            got, st = mg.verify_buffers(bufs, w["peq"], w["qinfo"], cands, 0.2)
            assert st == mg.SUCCESS
            launches[parts] = bufs.launches()
        assert launches == {p: p * launches[1] for p in launches}
        for bad in (0, 409_999, 410_000, n - 1):
            wrong = cands.copy()
            wrong["query"][bad] = 20_000  # one past the last read
            refused, st = mg.verify_buffers(bufs, w["peq"], w["qinfo"], wrong, 0.2)
            assert st == mg.E_QUERY_TOO_LONG
            assert refused["score"][bad] == mg.NO_RESULT
            assert np.array_equal(np.delete(refused, bad), np.delete(got, bad))
        again, st = mg.verify_buffers(bufs, w["peq"], w["qinfo"], cands, 0.2)
        assert st == mg.SUCCESS and np.array_equal(again, got)
