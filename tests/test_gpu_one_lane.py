"""The word-parallel shapes of every word count from 1 to 32, one lane per
candidate on the plain path and in the persistent kernel: small batches take
lanes of few words and large ones bit-sliced shapes, so one child process turns
both off and runs all of them, against the oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REF = 300_000


def run():
    sys.path[:0] = [os.path.join(ROOT, "myers-gpu_b200"), os.path.join(ROOT, "oracle")]
    import myersgpu as mg
    import oracle as orc
    words = mg.make_reference(REF, 17, n_frac=0.002)
    ref, ctx = mg.Reference(words, REF), mg.Context(4000)
    for w in range(1, 33):
        for lengths in (32 * w - 31, 32 * w - 9, 32 * w):
            # 40 candidates of few reads, 70 of a read each
            for reads, cands in ((4, 10), (70, 1)):
                b = mg.make_workload(mg.spec(REF, reads, w, lengths=lengths, sub=0.05, ins=0.01, dele=0.01, cands=cands), words)
                for window in (mg.WINDOW_ALIGNED, mg.WINDOW_EXACT):
                    full = orc.verify(b["peq"], b["qinfo"], b["cands"], words, REF, 0.2, exact=window == mg.WINDOW_EXACT)
                    for cut in (None, 0.08):
                        expect = full if cut is None else orc.apply_cutoff(full, b["qinfo"], b["cands"], cut)
                        for path in (mg.PATH_PLAIN, mg.PATH_BATCHED):
                            got = mg.verify_torch(ctx, ref, b["peq"], b["qinfo"], b["cands"], 0.2, window=window, path=path,
                                                  min_size=lengths, max_size=lengths, cutoff=cut)
                            assert np.array_equal(got, expect), (lengths, reads, window, cut, path)
                            assert ctx.flags() == 0
    # and all of them in one batch
    b = mg.make_workload(mg.spec(REF, 300, 5, length_range=(1, 1024), rate_range=(0.02, 0.08), cands=5), words)
    for window in (mg.WINDOW_ALIGNED, mg.WINDOW_EXACT):
        full = orc.verify(b["peq"], b["qinfo"], b["cands"], words, REF, 0.2, exact=window == mg.WINDOW_EXACT)
        for path in (mg.PATH_PLAIN, mg.PATH_BATCHED):
            got = mg.verify_torch(ctx, ref, b["peq"], b["qinfo"], b["cands"], 0.2, window=window, path=path, min_size=1,
                                  max_size=1024)
            assert np.array_equal(got, full), (window, path)


@pytest.mark.parametrize("tuned", ["", "0"])
def test_one_lane_shapes(cuda_ok, tuned):
    env = dict(os.environ, MYERS_SLICED="0", MYERS_SMALL_BATCH="0")
    if tuned:
        env["MYERS_AUTOTUNE"] = tuned  # one lane for every word count
    out = subprocess.run([sys.executable, "-c", "import test_gpu_one_lane as t; t.run()"], cwd=os.path.join(ROOT, "tests"),
                         env=env, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
