"""Traceback of results whose end column lies outside the window, up to the
largest column there is (the column after it wraps to 0): reported as
inconsistent, alone in a call, beside ordinary candidates in one warp, and
with scores of both kernels' bands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REF = 200_000


def _check(mg, orc, words, w, cands, results, window):
    ref = mg.Reference(words, REF)
    with mg.Traceback(len(cands), 64 << 20) as tb:
        aln, ops = mg.traceback_torch(tb, ref, w["peq"], w["qinfo"], cands, results, 0.2, 1000, 600, window=window)
    ref.close()
    e_aln, e_ops = orc.traceback(w["peq"], w["qinfo"], cands, results, words, REF, 0.2, 1000, 600,
                                 exact=window == mg.WINDOW_EXACT)
    assert np.array_equal(aln.view(np.uint32), e_aln.view(np.uint32))
    for k in np.nonzero(e_aln["num_ops"] <= 600)[0]:
        n = int(e_aln["num_ops"][k])
        assert np.array_equal(ops[k, :n], e_ops[k, :n]), k
    return e_aln


@pytest.mark.parametrize("m", [1, 40, 300])
@pytest.mark.parametrize("exact", [False, True])
def test_columns_outside_the_window(mg, orc, cuda_ok, m, exact):
    words = mg.make_reference(REF, 3)
    w = mg.make_workload(mg.spec(REF, 45, 4, lengths=m, sub=0.03, ins=0.01, dele=0.01, cands=1), words)
    window = mg.WINDOW_EXACT if exact else mg.WINDOW_ALIGNED
    good = orc.verify(w["peq"], w["qinfo"], w["cands"], words, REF, 0.2, exact=exact)
    span = int(np.float32(m) * np.float32(1.4))
    columns = span if exact else 8 * (span // 8 + (2 if span % 8 else 1))
    for column in (0xFFFFFFFF, 0xFFFFFFFE, 0x7FFFFFFF, columns):
        for score in (0, int(good["score"][0]), m):
            bad = good.copy()
            bad["column"][0], bad["score"][0] = column, score
            aln = _check(mg, orc, words, w, w["cands"][:1], bad[:1], window)
            assert aln["num_ops"][0] == orc.TB_INCONSISTENT
            bad["column"][33] = column
            aln = _check(mg, orc, words, w, w["cands"], bad, window)
            assert (aln["num_ops"][[0, 33]] == orc.TB_INCONSISTENT).all()
            assert (np.delete(aln["num_ops"], [0, 33]) < orc.TB_INCONSISTENT).all()
