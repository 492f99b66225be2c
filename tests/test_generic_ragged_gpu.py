"""Ragged inserts of the kernels with flush rings (proteins with windows of less
than four m-mers, DNA triplets), at the edges of their CTAs of 256 threads
(8192 windows) and over grids of many of them."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu

CASES = [(2, 12, 10, 10, 4), (2, 8, 6, 8, 8), (2, 4, 3, 2, 4), (1, 10, 8, 5, 4), (1, 6, 5, 6, 4)]


@pytest.mark.parametrize("alphabet,k,s,m,h", CASES)
@pytest.mark.parametrize("windows", [1, 8_191, 8_193, 3_700_000])
def test_ragged_insert_matches_oracle(sbf, cuda, oracle_mod, alphabet, k, s, m, h, windows):
    torch = cuda
    rng = np.random.default_rng(windows + k)
    width = 3 if alphabet == sbf.ALPHABET_DNA_TRIPLET else 1
    letters = b"ACGT" * 50 + b"N" if width == 3 else b"ACDEFGHIKLMNPQRSTVWY" * 10 + b"*"
    n = (windows + k - 1) * width
    seq = random_dna(rng, n, letters)
    lens, total = [], 0
    while total < n:  # symbol-aligned records back to back, some shorter than a window
        x = int(rng.choice([k - 1, k, 300, 5_000])) * width
        lens.append(min(x, n - total))
        total += lens[-1]
    ranges = np.stack([np.cumsum(lens) - lens, lens], axis=1).astype(np.int64)
    cfg = dict(k=k, s=s, m=m, hashes=h, alphabet=alphabet)
    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(1 << 22)
    for off, size in ranges:
        o.insert(words, seq[off:off + size])
    f = sbf.Filter(1 << 22, **cfg)
    assert f.kernel_path() == sbf.Filter.KERNELS_RUNTIME_COMPILED
    f.ragged_insert_async(torch.from_numpy(seq.copy()).cuda(), torch.from_numpy(ranges).cuda())
    np.testing.assert_array_equal(f.words_host(), words)
