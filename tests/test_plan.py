"""The choice of kernel shapes, on the CPU: plan_dump.cpp prints the plan that a
call would take and the query lengths that it admits."""
import itertools
import json
import os
import random
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "myers-gpu_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
PLAIN, BATCHED = 0, 1


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "plan_dump")
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{CUDA}/include", f"-I{PKG}/csrc", "-o", exe,
                    os.path.join(ROOT, "tests", "plan_dump.cpp"), os.path.join(PKG, "libmyers_b200.so"),
                    f"-Wl,-rpath,{PKG}"], check=True)

    def dump(path, lo, hi, n, reads=0, cut=-1.0, sms=148, entries=0, **env):
        return run([path, lo, hi, n, reads, cut, sms, entries], env)

    def run(args, env):
        env = {k: v for k, v in os.environ.items() if not k.startswith("MYERS_")} | env
        out = subprocess.run([exe, *map(str, args)], env=env, check=True, capture_output=True, text=True)
        return json.loads(out.stdout)

    dump.lengths = lambda n, by_length, lengths: run(["lengths", n, int(by_length), *lengths], {})
    return dump


@pytest.mark.parametrize("words,shape,length", [(32, [32, 8], 1000), (32, [32, 32], 1000), (16, [16, 32], 500),
                                                (40, [32, 32], 1270), (300, [32, 32], 9590)])
def test_bit_sliced_tiles_can_fall_back(plan, tmp_path, words, shape, length):
    """A lone bit-sliced shape admits the lengths of the word-parallel shape that
    it replaces. Its tiles fall back to word-parallel ones of 4,096 rows (16,384 in
    groups of several warps), so a tuned shape of more rows keeps its place."""
    fn = tmp_path / "tuned.json"
    fn.write_text(json.dumps({"plain": {str(words): shape}, "batched": {}, "batched_large": {}}))
    p = plan(PLAIN, length, length, 2_000_000, 100_000, MYERS_AUTOTUNE=str(fn))["plan"]
    if p["sliced"]:
        assert p["admits"][-1][1] <= (4096 if length <= 1024 else 16384)
    assert p["admits"] == [[1, 32 * shape[0] * shape[1]]]


RANGES = [(1, 32), (35, 301), (65, 96), (100, 100), (100, 128), (20, 1000), (545, 576), (640, 640), (700, 736), (900, 1000),
          (930, 960), (940, 950), (961, 1000), (990, 1000), (1000, 1000), (1000, 1100), (1025, 1088), (1040, 1060),
          (1500, 1600), (1505, 1568), (2000, 2048), (5000, 5100), (9000, 9600), (10000, 10200), (1000, 12000), (1, 1), (32750, 32768), (0, 0)]
CALLS = list(itertools.product((PLAIN, BATCHED), RANGES, (100, 3000, 20_000, 120_000, 1_000_000), (1, 11),
                               (-1.0, 0.0, 0.04, 0.2, 1.0)))


@pytest.mark.parametrize("mode", ["", "1", "2", "3"])
def test_admitted_lengths_do_not_depend_on_the_shapes(plan, mode):
    """The lengths that a call verifies, those its range leaves out among them, are
    the same whether it takes bit-sliced shapes, lanes of few words or neither."""
    for path, (lo, hi), n, per_read, cut in random.Random(mode).sample(CALLS, 250):
        got = plan(path, lo, hi, n, n // per_read, cut, **({"MYERS_SLICED": mode} if mode else {}))
        expect = plan(path, lo, hi, n, n // per_read, cut, MYERS_SLICED="0", MYERS_SMALL_BATCH="0")
        for part in expect:
            assert got[part]["admits"] == expect[part]["admits"], (path, lo, hi, n, per_read, cut, part)


@pytest.mark.parametrize("path,key", [(PLAIN, "plain"), (BATCHED, "batched"), (BATCHED, "batched_large")])
def test_named_autotune_file_decides(plan, tmp_path, path, key):
    """A file that MYERS_AUTOTUNE names decides the shapes of its word counts, in
    batches of the sizes that take bit-sliced shapes and lanes of few words else."""
    fn = tmp_path / "tuned.json"
    entries = {str(w): [16, 2] for w in range(17, 33)}
    fn.write_text(json.dumps({"plain": {}, "batched": {}, "batched_large": {}} | {key: entries}))
    other = tmp_path / "other.json"
    other.write_text(json.dumps({"plain": {}, "batched": {}, "batched_large": {}}))
    for n in (2_000_000,) if key != "plain" else (2_000_000, 3000):
        lo, hi = 520, 1000
        assert all(L == 2 and W == 16 for _, L, W in plan(path, lo, hi, n, n // 11, MYERS_AUTOTUNE=str(fn))["plan"]["shapes"])
        # word counts that it leaves out are chosen as without it
        assert plan(path, lo, hi, n, n // 11, MYERS_AUTOTUNE=str(other)) == plan(path, lo, hi, n, n // 11,
                                                                                 MYERS_AUTOTUNE="0")


@pytest.mark.parametrize("lengths", [[100, 200, 0, 1000], [0, 1000, 100], [1000, 1000, 0], [0, 0, 64], [0], [32768, 32769, 1],
                                     [4294967295, 40000, 33], [0, 65, 64, 0, 96, 97], [5] * 40 + [0, 9] + [7] * 33])
@pytest.mark.parametrize("n", [1, 7, 8, 129, 2047, 2048, 5003])
def test_lengths_of_a_send(plan, n, lengths):
    """Empty queries and those that are too long leave no trace in what the shapes
    are chosen from, wherever they stand."""
    there = {(lengths * (n // len(lengths) + 1))[q] for q in range(n)}
    kept = sorted(m for m in there if 1 <= m <= 32768)
    for by_length in (False, True):
        got = plan.lengths(n, by_length, lengths)
        assert [got["lo"], got["hi"]] == ([kept[0], kept[-1]] if kept else [0, 0])
        assert got["words"] == sorted({(m + 31) // 32 for m in kept})
        assert got["marked"] == (kept if by_length else [])


def test_rounds_are_those_of_the_device(plan):
    """Half the multiprocessors take the shapes of twice the candidates."""
    for lo, hi in ((400, 400), (1000, 1000), (3000, 3000), (100, 1000)):
        for n in range(20_000, 400_000, 20_000):
            whole, half = plan(BATCHED, lo, hi, n), plan(BATCHED, lo, hi, n // 2, sms=74)
            if n // 2 >= 150_000 or n < 150_000:  # on one side of the table for large batches
                assert whole["plan"]["sliced"] == half["plan"]["sliced"], (lo, hi, n)


# path, lengths, candidates, reads, PEQ entries (0, 0: a range is announced) and whether bit-sliced shapes are faster
SLICED = [(PLAIN, 66, 66, 660_000, 0, 0, False), (PLAIN, 96, 96, 520_000, 0, 0, False), (PLAIN, 100, 100, 660_000, 0, 0, True),
          (PLAIN, 128, 128, 440_000, 0, 0, False), (PLAIN, 160, 160, 330_000, 0, 0, False),
          (PLAIN, 160, 160, 440_000, 0, 0, True), (PLAIN, 600, 600, 33_000, 0, 0, False),
          (PLAIN, 600, 600, 38_000, 0, 0, True), (PLAIN, 600, 600, 16_500, 0, 0, False), (PLAIN, 600, 600, 24_000, 0, 0, True), (PLAIN, 20, 120, 60_000, 0, 0, False), (PLAIN, 20, 120, 660_000, 0, 0, False),
          (PLAIN, 65, 128, 5_000, 0, 0, False), (PLAIN, 35, 301, 5_000, 0, 0, True), (PLAIN, 35, 301, 300_000, 0, 0, True),
          (PLAIN, 35, 301, 1_300_000, 0, 0, False), (PLAIN, 250, 500, 1_300_000, 0, 0, True),
          (BATCHED, 35, 301, 660_000, 0, 0, False), (BATCHED, 35, 512, 660_000, 0, 0, False),
          (BATCHED, 20, 1000, 120_000, 0, 0, False), (BATCHED, 100, 1000, 110_000, 0, 0, True),
          (BATCHED, 1000, 10_000, 15_000, 0, 0, False), (BATCHED, 3000, 6000, 15_000, 0, 0, True),
          (BATCHED, 1000, 10_000, 100_000, 0, 0, True), (BATCHED, 1000, 12_000, 15_000, 0, 0, False),
          (BATCHED, 0, 0, 50_000, 4545, 4545, False), (BATCHED, 0, 0, 300_000, 27_272, 27_272, False),
          (BATCHED, 0, 0, 110_000, 10_000, 14_000, False), (BATCHED, 0, 0, 110_000, 10_000, 80_000, True)]


@pytest.mark.parametrize("path,lo,hi,n,reads,entries,faster", SLICED)
def test_bit_sliced_where_it_is_faster(plan, path, lo, hi, n, reads, entries, faster):
    assert (plan(path, lo, hi, n, reads, entries=entries)["plan"]["sliced"] > 0) == faster


@pytest.mark.parametrize("m,n,faster", [(760, 3300, True), (760, 7700, False), (760, 9900, True), (760, 16_500, False),
                                        (880, 3300, False), (880, 5500, True), (1000, 3300, False), (1000, 5500, True),
                                        (1000, 7700, False), (400, 5500, True), (400, 7700, False), (400, 9900, True)])
def test_lanes_of_few_words_where_they_are_faster(plan, m, n, faster):
    p = plan(BATCHED, m, m, n)["plan"]
    assert (p["shapes"][0][2] <= 5) == faster


@pytest.mark.parametrize("m,n,faster", [(600, 9000, True), (600, 16_500, False), (560, 16_500, True), (1000, 12_000, True)])
def test_lanes_of_few_words_on_the_plain_path(plan, m, n, faster):
    p = plan(PLAIN, m, m, n)["plan"]
    assert (p["shapes"][0][2] <= 5) == faster


@pytest.mark.parametrize("entries,faster", [(1272 * 8, False), (1272 * 2, True)])
def test_lanes_of_few_words_without_a_range(plan, entries, faster):
    """14K candidates of 1,000 and of 200 bases."""
    p = plan(BATCHED, 0, 0, 14_000, 1272, entries=entries)["plan"]
    assert all(W <= 5 for v, L, W in p["shapes"] if 32 * L * W in range(400, 1024)) == faster


# path, lengths, candidates, reads and whether bit-sliced shapes are faster: beside the lines between both
LINES = [(PLAIN, 565, 565, 28_700, 5737, True), (PLAIN, 565, 565, 31_000, 6200, False), (PLAIN, 600, 600, 37_000, 7400, False),
         (BATCHED, 73, 102, 1_270_000, 115_000, True), (BATCHED, 73, 102, 800_000, 70_000, False),
         (BATCHED, 193, 503, 1_260_000, 115_000, True), (BATCHED, 137, 396, 1_270_000, 317_000, False),
         (BATCHED, 217, 503, 656_000, 656_000, False), (BATCHED, 217, 503, 656_000, 150_000, True),
         (BATCHED, 553, 2544, 35_609, 3200, True), (BATCHED, 203, 1831, 60_330, 5500, True), (BATCHED, 332, 2385, 31_338, 6300, True)]


@pytest.mark.parametrize("path,lo,hi,n,reads,faster", LINES)
def test_bit_sliced_beside_the_lines(plan, path, lo, hi, n, reads, faster):
    entries = reads * (((lo + hi) // 2 + 127) // 128)
    assert (plan(path, lo, hi, n, reads, entries=entries)["plan"]["sliced"] > 0) == faster


@pytest.mark.parametrize("lo,hi,n,faster", [(613, 916, 5176, True), (114, 824, 9583, True), (100, 1000, 9000, True),
                                            (410, 698, 8447, False), (216, 658, 8746, False)])
def test_lanes_of_few_words_for_mixed_lengths(plan, lo, hi, n, faster):
    p = plan(BATCHED, lo, hi, n)["plan"]
    assert all(W <= 5 for v, L, W in p["shapes"]) == faster


def test_bit_sliced_second_pass(plan):
    """The cut-off's second pass: mostly one candidate per read."""
    assert plan(PLAIN, 666, 666, 292_402, 26_582, 0.04, entries=6 * 26_582)["second"]["sliced"] == 1


@pytest.mark.parametrize("cut,n,faster", [(0.08, 22_000_000, True), (0.2, 969_000, True), (0.2, 320_000, False)])
def test_bit_sliced_first_pass(plan, cut, n, faster):
    """The cut-off's first pass on the batched path: prefixes of a few row counts."""
    assert (plan(BATCHED, 100, 1000, n, n // 11, cut, entries=4 * (n // 11))["first"]["sliced"] > 0) == faster
