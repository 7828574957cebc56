"""Reads outside the announced range, beside reads in it: the same candidates are
verified, with the same results and flags, whether a call takes bit-sliced
shapes, lanes of few words or neither. The choice is read once per process, so
each setting runs in a child; its results are compared with those of the
word-parallel shapes, and these with the oracle's."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REF = 200_000
# ranges within a word, of several words, of several bit-sliced shapes, and whose
# word-parallel shape has more rows than their longest read has words
RANGES = [(100, 128), (545, 576), (700, 736), (930, 960), (990, 1000), (1025, 1056), (1025, 1120), (1285, 1300), (1505, 1568)]


def _reads(mg, words, lo, hi):
    """Half of the reads inside the range, a quarter within 200 bases of it, the
    others anywhere up to 1,900 bases, some of them empty."""
    rng = np.random.default_rng(lo)
    w = mg.make_workload(mg.spec(REF, 160, lo, lengths=1900, sub=0.03, ins=0.01, dele=0.01, cands=3), words)
    size = w["qinfo"]["size"]
    size[::2] = rng.integers(lo, hi + 1, 80)
    size[1::4] = rng.integers(max(1, lo - 200), hi + 201, 40)
    size[3::4] = rng.integers(1, 1901, 40)
    size[3::16] = 0
    return w


def run(out):
    sys.path[:0] = [os.path.join(ROOT, "myers-gpu_b200"), os.path.join(ROOT, "oracle")]
    import myersgpu as mg
    import oracle as orc
    words = mg.make_reference(REF, 8)
    ref, ctx = mg.Reference(words, REF), mg.Context(1000)
    found = {}
    for lo, hi in RANGES:
        w = _reads(mg, words, lo, hi)
        full = orc.verify(w["peq"], w["qinfo"], w["cands"], words, REF, 0.2)
        for cut in (None, 0.08):
            expect = full if cut is None else orc.apply_cutoff(full, w["qinfo"], w["cands"], cut)
            for path in (mg.PATH_PLAIN, mg.PATH_BATCHED):
                got = mg.verify_torch(ctx, ref, w["peq"], w["qinfo"], w["cands"], 0.2, path=path, min_size=lo,
                                      max_size=hi, cutoff=cut)
                flags = ctx.flags()
                refused = (got["score"] == mg.NO_RESULT) & (expect["score"] != mg.NO_RESULT)
                if cut is None:
                    assert np.array_equal(got[~refused], expect[~refused]), (lo, hi, path)
                    m = w["qinfo"]["size"][w["cands"]["query"]]
                    assert not refused[((m >= lo) & (m <= hi)) | (m == 0)].any()
                assert (flags != 0) == refused.any(), (lo, hi, path, cut)
                found[f"{lo}-{hi} {path} {cut}"] = got
    np.savez(out, **found)


@pytest.fixture(scope="module")
def results(cuda_ok, tmp_path_factory):
    def child(**env):
        out = str(tmp_path_factory.mktemp("out") / "results.npz")
        env = {k: v for k, v in os.environ.items() if not k.startswith("MYERS_")} | env
        r = subprocess.run([sys.executable, "-c", f"import test_gpu_admitted as t; t.run({out!r})"],
                           cwd=os.path.join(ROOT, "tests"), env=env, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        return np.load(out)
    return child, child(MYERS_SLICED="0", MYERS_SMALL_BATCH="0")


@pytest.mark.parametrize("mode", ["", "1", "2"])
def test_reads_outside_the_range(results, mode):
    child, expect = results
    got = child(**({"MYERS_SLICED": mode} if mode else {}))
    for name in expect.files:
        assert np.array_equal(got[name], expect[name]), (name, int((got[name] != expect[name]).sum()))
