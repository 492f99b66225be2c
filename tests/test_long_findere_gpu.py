"""Windows of many s-mers, whose rings of masks or hashes decide how many warps
an SM the tile kernels are compiled for, on both sides of each limit."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu

# s-mers a window, hashes: inserts change at 6 and 16, queries at 8 and 19 (four
# hashes) or 6 and 12.
CASES = [(5, 4), (6, 4), (8, 4), (15, 4), (16, 4), (19, 4), (31, 4), (6, 8), (11, 8), (12, 8)]


@pytest.mark.parametrize("f,h", CASES)
def test_long_findere_matches_oracle(sbf, cuda, oracle_mod, f, h):
    torch = cuda
    rng = np.random.default_rng(f * 100 + h)
    cfg = dict(k=31, s=32 - f, m=16, hashes=h)
    genome = random_dna(rng, 40_000, b"ACGT" * 100 + b"N")
    genome[20_000:20_300] = np.resize(genome[:7], 300)
    query = np.concatenate([genome[5_000:35_000], random_dna(rng, 10_003)])
    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(1 << 22)
    o.insert(words, genome)
    flt = sbf.Filter(1 << 22, **cfg)
    assert flt.kernel_path() == sbf.Filter.KERNELS_RUNTIME_COMPILED
    flt.insert_sequence_async(torch.from_numpy(genome.copy()).cuda())
    np.testing.assert_array_equal(flt.words_host(), words)
    want = o.contains(words, query)
    out = torch.full((want.size,), 7, dtype=torch.uint8, device="cuda")
    flt.contains_sequence_async(torch.from_numpy(query).cuda(), out)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


def test_long_findere_does_not_spill(sbf, cuda):
    """An insert of 16 s-mers a window takes twice as long as one of 4 (with its
    masks spilled from 80 registers a thread, ten times)."""
    torch = cuda
    seq = torch.from_numpy(random_dna(np.random.default_rng(7), 40_000_000)).cuda()

    def best(s):
        flt = sbf.Filter(1 << 31, k=31, s=s, m=16, hashes=4)
        times = []
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            flt.insert_sequence_async(seq)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert best(16) < 4 * best(28)
