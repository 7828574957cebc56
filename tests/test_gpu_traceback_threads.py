"""Tracebacks on two threads, each with its own object and stream, whose bands
call for different amounts of shared memory: every call gives the results that
the oracle has, whatever the other thread launches in between."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REF = 300_000


def test_two_threads_of_different_band_widths(mg, orc, cuda_ok):
    import torch
    words = mg.make_reference(REF, 41)
    ref = mg.Reference(words, REF)
    jobs = []
    # per thread, bands of one width and then another: 3, 7 and 9, 15 words
    for lengths, rates in ((300, (0.01, 0.25)), (1000, (0.1, 0.2))):
        sets = []
        for rate in rates:
            w = mg.make_workload(mg.spec(REF, 120, 42, lengths=lengths, sub=rate / 2, ins=rate / 4, dele=rate / 4,
                                         cands=1), words)
            res = orc.verify(w["peq"], w["qinfo"], w["cands"], words, REF, 0.2)
            sets.append((w, res, orc.traceback(w["peq"], w["qinfo"], w["cands"], res, words, REF, 0.2, 223, 512)))
        jobs.append(sets)
    barrier, failures = threading.Barrier(2), []

    def work(sets):
        try:
            with torch.cuda.stream(torch.cuda.Stream()), mg.Traceback(120, 256 << 20) as tb:
                barrier.wait()
                for i in range(60):
                    w, res, (e_aln, e_ops) = sets[i % 2]
                    aln, ops = mg.traceback_torch(tb, ref, w["peq"], w["qinfo"], w["cands"], res, 0.2, 223, 512)
                    assert np.array_equal(aln.view(np.uint32), e_aln.view(np.uint32))
                    traced = np.nonzero(e_aln["num_ops"] <= 512)[0]
                    assert len(traced) > 0
                    for k in traced:
                        n = int(e_aln["num_ops"][k])
                        assert np.array_equal(ops[k, :n], e_ops[k, :n])
        except BaseException as e:  # noqa: BLE001  (reported by the main thread)
            failures.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ref.close()
    assert not failures, failures
