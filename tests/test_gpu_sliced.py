"""The bit-sliced kernels against the oracle, bit for bit, at the sizes where
they can go wrong: the borders of their shapes (rows per lane, lanes per
group, warps per group), lengths that differ within a group, groups that are
not full, text and reads with N, PEQ rows with no base or with several, and
the lengths a caller did not announce. Small batches take the word-parallel
shapes, so each case runs in a child with MYERS_SLICED=1 (read once per
process); 2 and 3 spread the shapes of reads of up to 512 bases over two and
four times the lanes, as batches of many short lengths do."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _with_n(w, rng):
    b = w["peq"]["bitmap"]
    for e in rng.choice(len(b), len(b) // 3, replace=False):
        k = int(rng.integers(4))
        m = np.uint32(rng.integers(1 << 32)) & np.uint32(rng.integers(1 << 32)) & np.bitwise_or.reduce(b[e, :, k])
        b[e, :4, k] &= ~m
        b[e, 4, k] |= m


def _rows_without_base(w, rng):
    b = w["peq"]["bitmap"]
    for e in rng.choice(len(b), max(1, len(b) // 5), replace=False):
        b[e, :, int(rng.integers(4))] &= np.uint32(rng.integers(1 << 32))


def _rows_of_several_bases(w, rng):
    b = w["peq"]["bitmap"]
    for e in rng.choice(len(b), max(1, len(b) // 5), replace=False):
        b[e, int(rng.integers(5)), int(rng.integers(4))] |= np.uint32(rng.integers(1 << 32))


def _windows_out_of_range(w, rng):
    k = rng.choice(len(w["cands"]), len(w["cands"]) // 10, replace=False)
    w["cands"]["position"][k] = rng.integers(0, 1 << 33, len(k))


RAGGED = dict(length_range=(20, 1100), rate_range=(0.02, 0.08), cand_poisson=4.0)
LONG = dict(sub=0.03, ins=0.06, dele=0.03)
# name: (reference bases, its share of N, reads, workload, change, paths, cut-offs, announce the lengths)
CASES = {
    # 9 rows on 8 lanes, 16 / 17 and 24 / 25 rows, 8 / 16 / 32 lanes, one more and one less
    **{f"{m}b": (200_000, 0.001, 7, dict(lengths=m, cands=11), None, (0, 1), (None,), True)
       for m in (65, 72, 100, 128, 129, 192, 193, 255, 256, 257, 400, 512, 513, 777, 1000, 1024)},
    # 2 / 4 / 8 warps, 32 / 34 and 40 rows per lane
    **{f"{m}b": (400_000, 0.001, 5, dict(lengths=m, cands=8, **LONG), None, (0, 1), (None,), True)
       for m in (1025, 2048, 2049, 4097, 8192, 8193, 10240)},
    "mixed": (300_000, 0.001, 200, dict(lengths=[100, 200, 400, 600, 800, 1000], length_weights=[30, 20, 15, 15, 10, 10],
                                        rate_range=(0.02, 0.08), cand_poisson=10.0, cand_cap=64),
              None, (0, 1), (None,), True),
    "ragged": (300_000, 0.05, 200, RAGGED, None, (0, 1), (None,), True),
    "any-length": (300_000, 0.05, 60, RAGGED, None, (0, 1), (None,), False),
    "long-ragged": (1_000_000, 0.01, 40, dict(length_range=(900, 11000), indel_mean=1.5, cand_poisson=4.0, **LONG),
                    None, (0, 1), (None,), True),
    "reads-with-N": (300_000, 0.05, 60, dict(lengths=990, cands=5), _with_n, (0, 1), (None,), True),
    "long-with-N": (1_000_000, 0.05, 20, dict(length_range=(900, 11000), cand_poisson=4.0, **LONG), _with_n, (0, 1),
                    (None,), True),
    "rows-without-base": (300_000, 0.05, 60, RAGGED, _rows_without_base, (0, 1), (None,), True),
    "rows-of-several-bases": (300_000, 0.05, 60, RAGGED, _rows_of_several_bases, (0, 1), (None,), True),
    "long-rows-of-several-bases": (1_000_000, 0.05, 15, dict(length_range=(900, 11000), cand_poisson=4.0, **LONG),
                                   _rows_of_several_bases, (0,), (None,), True),
    "windows-out-of-range": (300_000, 0.001, 200, RAGGED, _windows_out_of_range, (0, 1), (None,), True),
    "cutoff": (300_000, 0.001, 200, dict(lengths=1000, cands=11), None, (0, 1), (0.0, 0.08, 0.2, 1.0), True),
    "cutoff-ragged": (1_000_000, 0.001, 100, dict(length_range=(65, 3000), cand_poisson=4.0, rate_range=(0.02, 0.08)),
                      None, (0, 1), (0.04, 0.2), True),
}


def run(name):
    sys.path[:0] = [os.path.join(ROOT, "myers-gpu_b200"), os.path.join(ROOT, "oracle")]
    import myersgpu as mg
    import oracle as orc
    ref_size, n_frac, reads, kw, change, paths, cutoffs, announce = CASES[name]
    words = mg.make_reference(ref_size, 3, n_frac=n_frac)
    w = mg.make_workload(mg.spec(ref_size, reads, 4, **kw), words)
    if change:
        change(w, np.random.default_rng(7))
    lo, hi = (int(w["qinfo"]["size"].min()), int(w["qinfo"]["size"].max())) if announce else (0, 0)
    ref, ctx = mg.Reference(words, ref_size), mg.Context(len(w["cands"]))
    for window in (mg.WINDOW_ALIGNED, mg.WINDOW_EXACT):
        full = orc.verify(w["peq"], w["qinfo"], w["cands"], words, ref_size, 0.2, exact=window == mg.WINDOW_EXACT)
        for cut in cutoffs:
            expect = full if cut is None else orc.apply_cutoff(full, w["qinfo"], w["cands"], cut)
            for path in paths:
                got = mg.verify_torch(ctx, ref, w["peq"], w["qinfo"], w["cands"], 0.2, window=window, path=path,
                                      min_size=lo, max_size=hi, cutoff=cut)
                assert np.array_equal(got, expect), (name, window, path, cut, int((got != expect).sum()))
                assert ctx.flags() == 0
    ref.close()
    ctx.close()


def run_unannounced():
    """Lengths outside the announced range: the plain path admits what fits the
    rows of the word-parallel shape, the batched path the word counts
    announced; others are flagged."""
    sys.path[:0] = [os.path.join(ROOT, "myers-gpu_b200"), os.path.join(ROOT, "oracle")]
    import myersgpu as mg
    import oracle as orc
    words = mg.make_reference(300_000, 3)
    w = mg.make_workload(mg.spec(300_000, 60, 4, length_range=(80, 1010), rate_range=(0.02, 0.08), cands=5), words)
    w["qinfo"]["size"][::2] = 1000  # half the reads announced; their entries may be too few
    ok = w["qinfo"]["posEntry"].astype(np.int64) + (w["qinfo"]["size"] + 127) // 128 <= len(w["peq"])
    cands = np.ascontiguousarray(w["cands"][ok[w["cands"]["query"]]])
    size = w["qinfo"]["size"][cands["query"]]
    full = orc.verify(w["peq"], w["qinfo"], cands, words, 300_000, 0.2)
    ref, ctx = mg.Reference(words, 300_000), mg.Context(len(cands))
    for path in (mg.PATH_PLAIN, mg.PATH_BATCHED):
        got = mg.verify_torch(ctx, ref, w["peq"], w["qinfo"], cands, 0.2, path=path, min_size=1000, max_size=1000)
        admitted = size <= 1024 if path == mg.PATH_PLAIN else (size + 31) // 32 == 32
        assert np.array_equal(got[admitted], full[admitted])
        assert (got["score"][~admitted] == mg.NO_RESULT).all()
        assert (ctx.flags() != 0) == (not admitted.all())
    ref.close()
    ctx.close()


SPREAD = ["100b", "128b", "129b", "255b", "256b", "257b", "512b", "mixed", "ragged", "rows-without-base", "cutoff-ragged"]


@pytest.mark.parametrize("name,mode", [*((n, "1") for n in [*CASES, "unannounced"]), *((n, "2") for n in SPREAD),
                                       *((n, "3") for n in SPREAD)])
def test_sliced(name, mode, cuda_ok):
    code = f"import test_gpu_sliced as t; t.run_unannounced() if {name!r} == 'unannounced' else t.run({name!r})"
    out = subprocess.run([sys.executable, "-c", code], cwd=os.path.join(ROOT, "tests"),
                         env=dict(os.environ, MYERS_SLICED=mode), capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
