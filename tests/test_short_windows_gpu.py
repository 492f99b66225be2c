"""DNA windows of one and two m-mers, whose strips go through the warp's pool
in parts, and windows of one m-mer that load their shards directly while the
filter has less than 2^20 of them."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu

CONFIGS = [dict(k=31, s=28, m=31, hashes=4), dict(k=31, s=28, m=30, hashes=4),
           dict(k=12, s=11, m=12, hashes=12), dict(k=32, s=20, m=31, hashes=8),
           dict(k=3, s=2, m=2, hashes=4)]
IDS = ["-".join(map(str, c.values())) for c in CONFIGS]


@pytest.mark.parametrize("cfg", CONFIGS, ids=IDS)
@pytest.mark.parametrize("shards", [1, 1 << 10, 1 << 20, 1 << 21])
def test_short_windows_match_oracle(sbf, cuda, oracle_mod, cfg, shards):
    torch = cuda
    k = cfg["k"]
    rng = np.random.default_rng(shards + k + cfg["m"])
    seq = random_dna(rng, 30_000)
    seq[5_000:6_000] = np.resize(seq[:5], 1_000)
    at, step = 9_000, 1
    while at < 14_000:  # invalid bases at every spacing up to 2 k
        seq[at] = ord("N")
        at += step
        step = step % (2 * k) + 1
    seq[20_000:20_500] = ord("A")
    o = oracle_mod.Oracle(**cfg)
    bits = 256 * shards
    f = sbf.Filter(bits, **cfg)
    # 2,000,000 windows run strips of 32 where the launch size counts.
    for n in (1, 8, 33, 255, 1_025, 29_000, 2_000_000) if shards < 1 << 21 else (1_025, 2_000_000):
        part = np.resize(seq, n + k - 1)
        ins = part[:part.size // 2 + k].copy()
        words = o.new_words(bits)
        o.insert(words, ins)
        f.clear()
        f.insert_sequence_async(torch.from_numpy(ins).cuda())
        np.testing.assert_array_equal(f.words_host(), words)
        query = np.where(rng.random(part.size) < 0.02, random_dna(rng, part.size), part)
        want = o.contains(words, query)
        out = torch.full((n + 3,), 7, dtype=torch.uint8, device="cuda")[3:]
        f.contains_sequence_async(torch.from_numpy(query).cuda(), out)
        np.testing.assert_array_equal(out.cpu().numpy(), want)


def test_short_windows_take_one_round(sbf, cuda):
    """In 2 MiB, against windows of 16 m-mers: inserts of two m-mers a window
    take 1.8 times as long and queries of one 2.2 times (in rounds through the
    pool 3.2 and 4.5 times)."""
    torch = cuda
    seq = torch.from_numpy(random_dna(np.random.default_rng(5), 40_000_000)).cuda()
    out = torch.empty(seq.numel(), dtype=torch.uint8, device="cuda")

    def best(m):
        f = sbf.Filter(1 << 24, k=31, s=28, m=m, hashes=4)
        times = {}
        for name, call in (("insert", lambda: f.insert_sequence_async(seq)),
                           ("query", lambda: f.contains_sequence_async(seq, out))):
            for _ in range(6):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                a.record()
                call()
                b.record()
                torch.cuda.synchronize()
                times[name] = min(times.get(name, 1e9), a.elapsed_time(b))
        return times

    long, two, one = best(16), best(30), best(31)
    assert two["insert"] < 2.5 * long["insert"]
    assert one["query"] < 3.3 * long["query"]
