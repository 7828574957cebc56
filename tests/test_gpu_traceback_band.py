"""The banded traceback kernel against the oracle's traceback, op for op, at
the sizes where it can go wrong: every width of its window (scores at and
beside multiples of 32), queries that end at, before and after a word, windows
that begin inside the read or end at the reference's end, reads and text with
N, candidates of very different lengths in one warp, and results that do not
follow from the inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REF = 600_000


def _trace(mg, orc, words, w, results, max_score, max_ops, window, scratch=1 << 30):
    ref = mg.Reference(words, REF)
    with mg.Traceback(len(w["cands"]), scratch) as tb:
        aln, ops = mg.traceback_torch(tb, ref, w["peq"], w["qinfo"], w["cands"], results, 0.2, max_score, max_ops,
                                      window=window)
        chunks = tb.chunks()
    ref.close()
    e_aln, e_ops = orc.traceback(w["peq"], w["qinfo"], w["cands"], results, words, REF, 0.2, max_score, max_ops,
                                 exact=window == mg.WINDOW_EXACT)
    assert np.array_equal(aln.view(np.uint32).reshape(-1, 4), e_aln.view(np.uint32).reshape(-1, 4))
    for k in np.nonzero(e_aln["num_ops"] <= max_ops)[0]:
        n = int(e_aln["num_ops"][k])
        assert np.array_equal(ops[k, :n], e_ops[k, :n]), k
    return e_aln, chunks


def _verify(orc, mg, words, w, window):
    return orc.verify(w["peq"], w["qinfo"], w["cands"], words, REF, 0.2, exact=window == mg.WINDOW_EXACT)


# lengths around words; error rates whose scores fall on every window width
@pytest.mark.parametrize("lengths,rate", [(1, 0.0), (31, 0.1), (32, 0.1), (33, 0.1), (96, 0.02), (100, 0.3), (129, 0.25),
                                          (224, 0.4), (481, 0.06), (500, 0.14), (500, 0.27), (1000, 0.02),
                                          (1000, 0.06), (1000, 0.1), (1000, 0.16), (1000, 0.21), (3000, 0.05)])
@pytest.mark.parametrize("exact", [False, True])
def test_band_widths(mg, orc, cuda_ok, lengths, rate, exact):
    words = mg.make_reference(REF, 11, n_frac=0.01)
    w = mg.make_workload(mg.spec(REF, 90, 12, lengths=lengths, sub=rate / 2, ins=rate / 4, dele=rate / 4, cands=2,
                                 indel_mean=1.5), words)
    window = mg.WINDOW_EXACT if exact else mg.WINDOW_ALIGNED
    res = _verify(orc, mg, words, w, window)
    aln, chunks = _trace(mg, orc, words, w, res, 223, 512, window)
    traced = aln["num_ops"] < orc.TB_INCONSISTENT
    assert chunks == (1 if traced.any() else 0)
    if lengths * rate < 150:
        assert traced.sum() >= 60


@pytest.mark.parametrize("bound", [5, 32, 33, 64, 65, 223])
def test_band_mixed_lengths(mg, orc, cuda_ok, bound):
    words = mg.make_reference(REF, 21, n_frac=0.01)
    w = mg.make_workload(mg.spec(REF, 300, 22, length_range=(20, 1500), rate_range=(0.0, 0.12), cands=3), words)
    res = _verify(orc, mg, words, w, mg.WINDOW_ALIGNED)
    aln, _ = _trace(mg, orc, words, w, res, bound, 512, mg.WINDOW_ALIGNED)
    assert (aln["num_ops"] < orc.TB_INCONSISTENT).any()


def test_band_edges(mg, orc, cuda_ok):
    """Windows shifted against the read, so that the alignment starts in column
    0 with the read's first bases alone, or ends at the reference's last base;
    bogus scores and columns; room for few ops; a scratch of few slots."""
    words = mg.make_reference(REF, 31)
    w = mg.make_workload(mg.spec(REF, 120, 32, lengths=400, sub=0.02, ins=0.01, dele=0.01, cands=1), words)
    rng = np.random.default_rng(5)
    w["cands"]["position"] = np.minimum(w["true_pos"] + rng.integers(0, 60, 120).astype(np.uint64), REF - 600)
    w["cands"]["position"][::10] = REF - 561  # the last window that fits
    for window in (mg.WINDOW_ALIGNED, mg.WINDOW_EXACT):
        res = _verify(orc, mg, words, w, window)
        _trace(mg, orc, words, w, res, 200, 512, window)
        bad = res.copy()
        bad["score"][::3] += 1
        bad["score"][1::5] -= 1
        bad["column"][2::7] += 3
        aln, _ = _trace(mg, orc, words, w, bad, 200, 512, window)
        assert (aln["num_ops"] == orc.TB_INCONSISTENT).sum() > 20
        _trace(mg, orc, words, w, res, 200, 3, window)
        _trace(mg, orc, words, w, res, 200, 512, window, scratch=8 << 20)
