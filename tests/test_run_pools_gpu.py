"""The tile kernels' run lists and slot pools against the oracle, where a pool
takes one round, several rounds or none, and at the edges of strips, warps and
tiles (1024, 2048 and 4096 windows for strips of 8, 16 and 32 windows, which
the launch size selects: on 148 SMs up to 606,207 and 1,818,623 windows)."""
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


LENGTHS = (1, 7, 8, 9, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 60_000, 819_199, 819_200,
           819_201, 1_884_159, 1_884_160, 1_884_161)
IDS = ["-".join(map(str, c.values())) for c in CONFIGS]


def sequences(k, m):
    """A genome with a short period, a homopolymer and a run of N, and a mixed
    sequence that shares parts of it and has invalid bases at every spacing up
    to twice the window length."""
    rng = np.random.default_rng(k * 100 + m)
    genome = random_dna(rng, 60_000)
    genome[20_000:21_000] = np.resize(random_dna(rng, 7), 1_000)
    genome[30_000:30_500] = ord("A")
    genome[40_000:40_400] = ord("N")
    gaps = random_dna(rng, 20_000)
    at, step = 0, 1
    while at < gaps.size:
        gaps[at] = ord("N")
        at += step
        step = step % (2 * k) + 1
    mixed = np.concatenate([genome[10_000:45_000], random_dna(rng, 20_000), gaps, genome[:5_000],
                            random_dna(rng, 47_001)])
    return genome, np.resize(mixed, LENGTHS[-1] + 100)


def on_device(torch, seq, shift):
    d = torch.zeros(seq.size + 16, dtype=torch.uint8, device="cuda")[shift:][:seq.size]
    return d.copy_(torch.from_numpy(seq.copy()))


@pytest.mark.parametrize("cfg", CONFIGS, ids=IDS)
def test_insert_matches_oracle(sbf, cuda, oracle_mod, cfg):
    _, mixed = sequences(cfg["k"], cfg["m"])
    o = oracle_mod.Oracle(**cfg)
    f = sbf.Filter(1 << 18, **cfg)
    for n in LENGTHS:
        for shift in (0, 3) if n < 100_000 else (3,):
            seq = mixed[shift:][:n + cfg["k"] - 1]
            words = o.new_words(1 << 18)
            o.insert(words, seq)
            f.clear()
            f.insert_sequence_async(on_device(cuda, seq, shift))
            np.testing.assert_array_equal(f.words_host(), words)


@pytest.mark.parametrize("cfg", CONFIGS, ids=IDS)
def test_query_matches_oracle(sbf, cuda, oracle_mod, cfg):
    torch = cuda
    k = cfg["k"]
    genome, mixed = sequences(k, cfg["m"])
    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(1 << 18)
    o.insert(words, genome)
    f = sbf.Filter(1 << 18, **cfg)
    f.insert_sequence_async(torch.from_numpy(genome).cuda())
    for n in LENGTHS:
        for shift in (0, 3) if n < 100_000 else (3,):
            seq = mixed[shift:][:n + k - 1]
            want = o.contains(words, seq)
            d = on_device(torch, seq, shift)
            out = torch.full((want.size,), 7, dtype=torch.uint8, device="cuda")
            f.contains_sequence_async(d, out)
            bits = torch.full(((want.size + 31) // 32,), -1, dtype=torch.int32, device="cuda")
            f.contains_sequence_bits_async(d, bits)
            np.testing.assert_array_equal(out.cpu().numpy(), want)
            got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")
            np.testing.assert_array_equal(got[:want.size], want)


PROTEINS = [(12, 10, 6, 4), (12, 12, 6, 8), (12, 8, 4, 16), (12, 5, 9, 4), (7, 6, 7, 4),
            (1, 1, 1, 4)]


@pytest.mark.parametrize("k,s,m,h", PROTEINS)
def test_protein_tiles_match_oracle(sbf, cuda, oracle_mod, k, s, m, h):
    """Proteins in the kernels compiled at run time: every byte value,
    invalid bytes at every spacing up to twice the window length, and the
    edges of strips and tiles."""
    torch = cuda
    rng = np.random.default_rng(k * 100 + m)
    seq = random_dna(rng, 20_000, b"ACDEFGHIKLMNPQRSTVWYacdefghiklmnpqrstvwy")
    at, step = 9_000, 1
    while at < 14_000:
        seq[at] = rng.choice(np.frombuffer(b"*@[`{-\0\xc1", np.uint8))
        at += step
        step = step % (2 * k) + 1
    seq[14_000:16_000] = rng.integers(0, 256, 2_000, dtype=np.uint8)
    seq[17_000:17_500] = np.resize(seq[:5], 500)
    cfg = dict(k=k, s=s, m=m, hashes=h, alphabet=sbf.ALPHABET_PROTEIN)
    o = oracle_mod.Oracle(**cfg)
    f = sbf.Filter(1 << 17, **cfg)
    assert f.kernel_path() == sbf.Filter.KERNELS_RUNTIME_COMPILED
    for n in (1, 31, 32, 33, 1023, 1025, 8191, 8192, 8193, 16_385, 19_900):
        for shift in (0, 3):
            part = seq[shift:][:n + k - 1]
            words = o.new_words(1 << 17)
            o.insert(words, part[:part.size // 2 + k])
            f.clear()
            f.insert_sequence_async(on_device(torch, part[:part.size // 2 + k], shift))
            np.testing.assert_array_equal(f.words_host(), words)
            want = o.contains(words, part)
            d = on_device(torch, part, shift)
            out = torch.full((want.size,), 7, dtype=torch.uint8, device="cuda")
            f.contains_sequence_async(d, out)
            bits = torch.full(((want.size + 31) // 32,), -1, dtype=torch.int32, device="cuda")
            f.contains_sequence_bits_async(d, bits)
            np.testing.assert_array_equal(out.cpu().numpy(), want)
            got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")
            np.testing.assert_array_equal(got[:want.size], want)
