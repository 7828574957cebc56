"""The device read packer against the oracle's at the sizes where it can go
wrong: reads that end at, before and after word and entry borders, empty
reads, every byte value, every alignment of the ASCII buffer, reads at its
edges, and few or many reads per warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 3, 31, 32, 33, 95, 127, 128, 129, 255, 257, 1000, 4097]


@pytest.mark.parametrize("reads", [1, 7, 33, 20_000, 400_000])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_pack_reads(mg, orc, cuda_ok, reads, shift):
    import torch
    rng = np.random.default_rng(reads + shift)
    top = 4097 if reads < 100 else 300 if reads < 100_000 else 40
    lengths = rng.choice([x for x in EDGES if x <= top], reads).astype(np.uint64)
    letters = np.frombuffer(b"ACGTacgtN", dtype=np.uint8)
    ascii = rng.choice(letters, int(lengths.sum()) + 1)
    ascii[rng.integers(0, len(ascii), len(ascii) // 20)] = rng.integers(0, 256, len(ascii) // 20)
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    ascii = ascii[:int(offsets[-1])]
    entries = ((lengths + 127) // 128).astype(np.uint32)
    qinfo = np.zeros(reads, dtype=mg.QINFO)
    qinfo["size"] = lengths
    qinfo["posEntry"] = np.concatenate([[0], np.cumsum(entries)[:-1]])
    n_e = int(entries.sum())
    buf = torch.zeros(len(ascii) + 8, dtype=torch.uint8, device="cuda")
    buf[shift: shift + len(ascii)] = torch.from_numpy(ascii).cuda()
    d_off = torch.from_numpy(offsets.view(np.uint8)).cuda()
    d_qi = torch.from_numpy(qinfo.view(np.uint8)).cuda()
    out = torch.full((max(1, n_e) * 80,), 0x5A, dtype=torch.uint8, device="cuda")
    ctx = mg.Context(1)
    st = mg.lib.myersPackPEQAsync(ctx.h, buf.data_ptr() + shift, len(ascii), d_off.data_ptr(), d_qi.data_ptr(), reads,
                                  out.data_ptr(), n_e, torch.cuda.current_stream().cuda_stream)
    assert st == mg.SUCCESS
    torch.cuda.synchronize()
    assert ctx.flags() == 0
    ctx.close()
    got = out.cpu().numpy()[: n_e * 80].view(np.uint32).reshape(-1, 20)
    check = range(reads) if reads < 30_000 else rng.choice(reads, 5000, replace=False)
    for r in check:
        if lengths[r]:
            e = int(qinfo["posEntry"][r])
            expect = orc.pack_peq(bytes(ascii[offsets[r]: offsets[r + 1]])).reshape(-1, 20)
            assert np.array_equal(got[e: e + len(expect)], expect), (r, int(lengths[r]))
