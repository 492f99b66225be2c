"""The query kernel's run lists and shard pool against the oracle, where the
pool takes one round, several rounds or none, and at the edges of strips
(32 windows), warps (1024) and tiles (8192)."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu

CONFIGS = [
    dict(k=31, s=28, m=16, hashes=4),   # W = 16, F = 4
    dict(k=21, s=19, m=11, hashes=4),   # W = 11, F = 3
    dict(k=31, s=28, m=16, hashes=8),
    dict(k=31, s=28, m=16, hashes=16),
    dict(k=31, s=30, m=21, hashes=4),   # F = 2
    dict(k=31, s=26, m=28, hashes=4),   # W = 4: several rounds, F = 6
    dict(k=31, s=28, m=31, hashes=4),   # W = 1: every window a run
    dict(k=28, s=26, m=6, hashes=12),   # W = 23
    dict(k=5, s=4, m=3, hashes=4),      # W = 3, few m-mers: no pool
]


@pytest.mark.parametrize("cfg", CONFIGS, ids=lambda c: "-".join(map(str, c.values())))
def test_query_matches_oracle(sbf, cuda, oracle_mod, cfg):
    torch = cuda
    k = cfg["k"]
    rng = np.random.default_rng(k * 100 + cfg["m"])
    genome = random_dna(rng, 60_000)
    genome[20_000:21_000] = np.resize(random_dna(rng, 7), 1_000)  # a short period
    genome[30_000:30_500] = ord("A")
    genome[40_000:40_400] = ord("N")
    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(1 << 18)
    o.insert(words, genome)
    f = sbf.Filter(1 << 18, **cfg)
    f.insert_sequence_async(torch.from_numpy(genome).cuda())
    # Invalid bases at every spacing up to twice the window length.
    gaps = random_dna(rng, 20_000)
    at, step = 0, 1
    while at < gaps.size:
        gaps[at] = ord("N")
        at += step
        step = step % (2 * k) + 1
    mixed = np.concatenate([genome[10_000:45_000], random_dna(rng, 20_000), gaps, genome[:5_000]])
    for n in (1, 31, 32, 33, 1023, 1024, 1025, 8191, 8192, 8193, mixed.size - k + 1):
        for shift in (0, 3):
            seq = mixed[shift:][:n + k - 1]
            want = o.contains(words, seq)
            d = torch.zeros(seq.size + 16, dtype=torch.uint8, device="cuda")[shift:][:seq.size]
            d.copy_(torch.from_numpy(seq.copy()))
            out = torch.full((want.size,), 7, dtype=torch.uint8, device="cuda")
            f.contains_sequence_async(d, out)
            bits = torch.full(((want.size + 31) // 32,), -1, dtype=torch.int32, device="cuda")
            f.contains_sequence_bits_async(d, bits)
            np.testing.assert_array_equal(out.cpu().numpy(), want)
            got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")
            np.testing.assert_array_equal(got[:want.size], want)
