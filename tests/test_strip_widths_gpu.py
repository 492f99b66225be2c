"""Dense and ragged calls against the oracle in each strip width of the tile
kernels, which the launch size selects (on 148 SMs strips of 8 windows below
606,208 windows, of 16 below 1,818,624, then 32), and ragged passes of more
tiles than are resident (888 CTAs), whose CTAs take several tiles each."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu

CONFIGS = [dict(k=31, s=28, m=16, hashes=4), dict(k=21, s=19, m=11, hashes=4),
           dict(k=31, s=28, m=16, hashes=16), dict(k=31, s=30, m=21, hashes=4)]
IDS = ["-".join(map(str, c.values())) for c in CONFIGS]
WINDOWS = [60_001, 819_201, 1_884_161]
BITS = 1 << 22


@pytest.mark.parametrize("cfg", CONFIGS, ids=IDS)
@pytest.mark.parametrize("windows", WINDOWS)
def test_dense_matches_oracle(sbf, cuda, oracle_mod, cfg, windows):
    torch = cuda
    rng = np.random.default_rng(windows + cfg["m"])
    n = windows + cfg["k"] - 1
    seq = random_dna(rng, n)
    other = np.concatenate([seq[:n // 2], random_dna(rng, n - n // 2)])
    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(BITS)
    packed = sbf.pack_dense_sequence(seq)
    o.insert_dense(words, packed, n)
    f = sbf.Filter(BITS, **cfg)
    f.insert_dense_packed_async(torch.from_numpy(packed.view(np.int64)).cuda(), n)
    np.testing.assert_array_equal(f.words_host(), words)
    packed = sbf.pack_dense_sequence(other)
    want = o.contains_dense(words, packed, n)
    d = torch.from_numpy(packed.view(np.int64)).cuda()
    buf = torch.full((windows + 5,), 7, dtype=torch.uint8, device="cuda")
    for shift in (0, 5):  # the output's alignment sets the grid's phase
        f.contains_dense_packed_async(d, n, buf[shift:][:windows])
        np.testing.assert_array_equal(buf[shift:][:windows].cpu().numpy(), want)
    bits = torch.full(((windows + 31) // 32,), -1, dtype=torch.int32, device="cuda")
    f.contains_dense_packed_bits_async(d, n, bits)
    got = np.unpackbits(bits.cpu().numpy().view(np.uint8), bitorder="little")
    np.testing.assert_array_equal(got[:windows], want)
    assert not got[windows:].any()


def records(rng, total, k):
    """Record lengths and gaps of about `total` bytes: reads of uneven length,
    then records of about k bases (more than 128 a tile, several a strip),
    empty ones, and one that spans many tiles."""
    reads = np.clip(rng.lognormal(5.0, 1.0, total // 400), 1, 30_000).astype(np.int64)
    tiny = rng.integers(k - 3, k + 3, total // (4 * k))
    some = rng.integers(0, 4, 2_000)
    lens = np.concatenate([reads, [40_000], tiny, some])
    lens = np.concatenate([lens, np.full(max(1, (total - int(lens.sum())) // 1_000), 999)])
    gaps = np.where(rng.random(lens.size) < 0.3, rng.integers(1, 20, lens.size), 0)
    return lens, gaps


@pytest.mark.parametrize("cfg", CONFIGS[:2], ids=IDS[:2])
@pytest.mark.parametrize("total", [200_000, 1_000_000, 2_200_000, 4_600_000])
def test_ragged_matches_oracle(sbf, cuda, oracle_mod, cfg, total):
    torch = cuda
    k = cfg["k"]
    rng = np.random.default_rng(total + k)
    lens, gaps = records(rng, total, k)
    offs = np.cumsum(lens + gaps) - lens
    seq = random_dna(rng, int(offs[-1] + lens[-1]) + 7, b"ACGT" * 60 + b"N")
    w_of = np.maximum(lens - k + 1, 0)

    def joined(pick):
        """The picked records, each followed by an N, and where they start."""
        size = lens[pick] + 1
        start = np.cumsum(size) - size
        out = np.full(int(size.sum()), ord("N"), np.uint8)
        rid = np.repeat(np.arange(pick.size), lens[pick])
        rel = np.arange(rid.size) - np.repeat(np.cumsum(lens[pick]) - lens[pick], lens[pick])
        out[start[rid] + rel] = seq[offs[pick][rid] + rel]
        return out, start

    def windows(start, counts):
        """Positions start[r] + 0 .. counts[r] - 1 of all records in turn."""
        rid = np.repeat(np.arange(counts.size), counts)
        rel = np.arange(rid.size) - np.repeat(np.cumsum(counts) - counts, counts)
        return start[rid] + rel, rid

    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(BITS)
    half = np.arange(0, lens.size, 2)
    part, _ = joined(half)
    o.insert(words, part)
    every, start = joined(np.arange(lens.size))
    at, rid = windows(start, w_of)
    hit = o.contains(words, every)[at]
    up = every & 0xDF
    bad = np.concatenate([[0], np.cumsum(~np.isin(up, np.frombuffer(b"ACGT", np.uint8)))])
    ok = bad[at + k] == bad[at]
    want_valid = np.bincount(rid, ok, lens.size).astype(np.int64)
    want_pos = np.bincount(rid, hit, lens.size).astype(np.int64)

    def ranges(pick):
        return torch.from_numpy(np.stack([offs[pick], lens[pick]], axis=1)).cuda()

    d = torch.from_numpy(np.concatenate([np.zeros(3, np.uint8), seq])).cuda()[3:]
    f = sbf.Filter(BITS, **cfg)
    total_windows = torch.zeros(2, dtype=torch.int64, device="cuda")
    f.ragged_insert_async(d, ranges(half), total_windows)
    np.testing.assert_array_equal(f.words_host(), words)
    assert int(total_windows[0]) == int(want_valid[half].sum())
    n = lens.size
    valid = torch.full((n,), 99, dtype=torch.int64, device="cuda")
    positive = torch.full((n,), 99, dtype=torch.int64, device="cuda")
    out = torch.full((seq.size - k + 1,), 7, dtype=torch.uint8, device="cuda")
    f.ragged_contains_counts_async(d, ranges(np.arange(n)), valid, positive, out)
    np.testing.assert_array_equal(valid.cpu().numpy(), want_valid)
    np.testing.assert_array_equal(positive.cpu().numpy(), want_pos)
    want = np.zeros(seq.size - k + 1, np.uint8)
    want[windows(offs, w_of)[0]] = hit
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    out.fill_(7)
    f.ragged_contains_async(d, ranges(np.arange(n)), out)
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("k,s,m,h", [(6, 5, 3, 4), (7, 5, 3, 8)])
def test_short_protein_windows_match_oracle(sbf, cuda, oracle_mod, k, s, m, h):
    """Windows of 4 and 5 short m-mers load their shards without a pool."""
    torch = cuda
    rng = np.random.default_rng(k)
    seq = random_dna(rng, 20_000, b"ACDEFGHIKLMNPQRSTVWYacdefghiklmnpqrstvwy" * 3 + b"*@[`{")
    cfg = dict(k=k, s=s, m=m, hashes=h, alphabet=sbf.ALPHABET_PROTEIN)
    o = oracle_mod.Oracle(**cfg)
    words = o.new_words(1 << 17)
    o.insert(words, seq[:3_000])
    f = sbf.Filter(1 << 17, **cfg)
    assert f.kernel_path() == sbf.Filter.KERNELS_RUNTIME_COMPILED
    f.insert_sequence_async(torch.from_numpy(seq[:3_000].copy()).cuda())
    np.testing.assert_array_equal(f.words_host(), words)
    for n in (1, 33, 4_095, 4_097, 19_000):
        part = seq[:n + k - 1]
        want = o.contains(words, part)
        out = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
        f.contains_sequence_async(torch.from_numpy(part.copy()).cuda(), out)
        np.testing.assert_array_equal(out.cpu().numpy(), want)
