"""Filters of a few shards: neighbouring runs of one shard are one run, within
a strip and over the strips of a warp, whatever their minimizers are."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu

CONFIGS = [dict(k=31, s=28, m=16, hashes=4), dict(k=21, s=19, m=11, hashes=4),
           dict(k=5, s=4, m=3, hashes=4), dict(k=31, s=28, m=16, hashes=16)]
IDS = ["-".join(map(str, c.values())) for c in CONFIGS]


@pytest.mark.parametrize("cfg", CONFIGS, ids=IDS)
@pytest.mark.parametrize("shards", [1, 2, 8])
@pytest.mark.parametrize("windows", [33, 3_000, 700_000, 1_900_000])
def test_few_shards_match_oracle(sbf, cuda, oracle_mod, cfg, shards, windows):
    torch = cuda
    rng = np.random.default_rng(windows + shards)
    # Few s-mers, so that a filter of one shard does not fill up; invalid
    # bases end runs within and at the ends of strips.
    seq = np.resize(random_dna(rng, 60), windows + cfg["k"] - 1)
    seq[rng.integers(0, seq.size, seq.size // 200)] = ord("N")
    o = oracle_mod.Oracle(**cfg)
    bits = 256 * shards
    words = o.new_words(bits)
    o.insert(words, seq[:windows // 2 + cfg["k"]])
    f = sbf.Filter(bits, **cfg)
    assert f.num_shards() == shards
    f.insert_sequence_async(torch.from_numpy(seq[:windows // 2 + cfg["k"]].copy()).cuda())
    np.testing.assert_array_equal(f.words_host(), words)
    query = np.where(rng.random(seq.size) < 0.01, random_dna(rng, seq.size), seq)
    out = torch.full((windows,), 7, dtype=torch.uint8, device="cuda")
    f.contains_sequence_async(torch.from_numpy(query).cuda(), out)
    np.testing.assert_array_equal(out.cpu().numpy(), o.contains(words, query))


def test_one_shard_takes_one_update_a_strip(sbf, cuda):
    """With one shard every strip is one run, so the time to insert does not
    depend on how often the minimizer changes: 0.56 runs a window for W = 3
    against 0.12 for W = 16 (compared by minimizers, W = 3 took four times as
    long as W = 16; the updates of one shard follow one another)."""
    torch = cuda
    seq = torch.from_numpy(random_dna(np.random.default_rng(3), 8_000_000)).cuda()

    def best(**cfg):
        f = sbf.Filter(256, **cfg)
        times = []
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            f.insert_sequence_async(seq)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert best(k=5, s=4, m=3, hashes=4) < 2 * best(k=31, s=28, m=16, hashes=4)
