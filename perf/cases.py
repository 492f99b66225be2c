"""Performance cases of the Super Bloom filter engine.

Each case is one call of the device-buffer API on inputs that are already on
the GPU: inserts and queries of plain, 2-bit dense and ragged sequences, from
one gene to a whole genome.  Sizes and value distributions follow the
benchmark's workloads (bench.py, workloads/synthetic.py).
"""
import math

import numpy as np
import torch

import cusbf_b200 as sbf

BASE = {"k": 31, "s": 28, "m": 16, "hashes": 4, "alphabet": sbf.ALPHABET_DNA}
K21 = {"k": 21, "s": 19, "m": 11, "hashes": 4, "alphabet": sbf.ALPHABET_DNA}
PROTEIN = {"k": 12, "s": 10, "m": 6, "hashes": 4, "alphabet": sbf.ALPHABET_PROTEIN}
# The other configurations that the library compiles in and the benchmark runs.
OTHERS = [K21, dict(BASE, s=30), dict(BASE, s=31), dict(BASE, m=21), dict(BASE, hashes=8), PROTEIN]


def listed():
    """The listed cases.  `genome` is the number of symbols that the filter is
    built from, `reads` the number of reads of a query (0: it takes the
    genome's first `query` symbols), `shift` the byte offset of the input in
    its buffer."""
    return [
        # One gene goes into a small index: a single launch, all latency.
        dict(BASE, name="insert_gene", op="insert", genome=3_217, log2_bits=20, shift=0),
        # A handful of reads against a bacterial index: the smallest query.
        dict(BASE, name="query_64_reads", op="query", genome=200_000, log2_bits=23, reads=64,
             read_len=150, shift=0),
        # A bacterial chromosome with an index that stays in L2.
        dict(BASE, name="insert_2mbp", op="insert", genome=2_000_000, log2_bits=28, shift=0),
        # A bacterial assembly looked up in it, half of it in the index.
        dict(BASE, name="query_4mbp", op="query", genome=2_000_000, log2_bits=28, reads=0,
             query=4_000_000, shift=0),
        # A small animal genome with runs of N, index twice the L2; the
        # sequence starts at an odd address (it follows a header).
        dict(BASE, name="insert_100mbp", op="insert", genome=100_286_401, log2_bits=31, shift=7),
        # A human-sized genome into an 8 GiB index: the largest build.
        dict(BASE, name="insert_3gbp", op="insert", genome=3_100_000_000, log2_bits=36, shift=0),
        # A sequencing run of short reads, joined by N, against that index.
        dict(BASE, name="query_10m_reads", op="query", genome=3_100_000_000, log2_bits=36,
             reads=10_000_000, read_len=150, shift=0),
        # Contigs of an assembly as one ragged batch.
        dict(BASE, name="ragged_insert_contigs", op="ragged_insert", genome=200_000_000,
             log2_bits=32, median=5_000, sigma=1.18, shift=0),
        # Reads of uneven length as one ragged batch, with per-read counts.
        dict(BASE, name="ragged_query_reads", op="ragged_query", genome=200_000_000, log2_bits=32,
             reads=2_000_000, median=150, sigma=1.0, shift=0),
        # 2-bit input and one result bit per window: the compact wire format.
        dict(BASE, name="dense_query_bits", op="dense_query_bits", genome=100_000_000,
             log2_bits=31, reads=0, query=256_000_000, shift=0),
        # Shorter k-mers (k = 21), as used on noisy reads.
        dict(K21, name="query_k21_1m_reads", op="query", genome=100_000_000, log2_bits=31,
             reads=1_000_003, read_len=150, shift=0),
        # A protein database screened with peptide 12-mers.
        dict(PROTEIN, name="protein_query", op="query", genome=16_000_000, log2_bits=29, reads=0,
             query=64_000_000, shift=0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bits_for(genome):
    """The benchmark's density: 16 to 32 bits per k-mer, a power of two."""
    return max(18, math.ceil(math.log2(genome * 16)))


def draw(rng):
    """One more case: any of the operations, sizes over the listed range."""
    cfg = dict(BASE) if rng.random() < 0.6 else dict(rng.choice(OTHERS))
    op = rng.choice(["insert", "insert", "query", "query", "query_bits", "dense_insert",
                     "dense_query_bits", "ragged_insert", "ragged_query"])
    big = 100_000_000 if cfg["alphabet"] == sbf.ALPHABET_PROTEIN else 1_000_000_000
    c = dict(cfg, op=op, shift=rng.randrange(0, 32) if not op.startswith("dense") else 0)
    if op in ("insert", "dense_insert"):
        c["genome"] = _log_uniform(rng, 2_000, big)
    elif op == "ragged_insert":
        c["genome"] = _log_uniform(rng, 20_000, min(big, 400_000_000))
        c.update(median=rng.choice([300, 1_000, 5_000]), sigma=round(rng.uniform(0.5, 1.2), 2))
    else:
        c["genome"] = _log_uniform(rng, 100_000, min(big, 400_000_000))
        if op == "ragged_query":
            c.update(reads=_log_uniform(rng, 50, 2_000_000), median=rng.choice([100, 150, 250]),
                     sigma=round(rng.uniform(0.0, 1.0), 2))
        elif rng.random() < 0.5 and op != "dense_query_bits":
            c.update(reads=_log_uniform(rng, 20, 5_000_000), read_len=rng.choice([100, 150, 251]))
        else:
            c.update(reads=0, query=_log_uniform(rng, 2_000, min(big, 600_000_000)))
    c["log2_bits"] = _bits_for(c["genome"])
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

_SEG = 2048
_STEP = 1 << 26


def _letters(alphabet, gc):
    """256 letters that a random byte is mapped through."""
    if alphabet == sbf.ALPHABET_PROTEIN:
        a = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
        return a[np.arange(256) * len(a) // 256].copy()
    c = int(round(256 * gc / 2))
    a = int(round(256 * (1 - gc) / 2))
    return np.frombuffer(b"A" * a + b"C" * c + b"G" * c + b"T" * (256 - a - 2 * c),
                         np.uint8).copy()


def _random(n, lut, gen):
    return lut[torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=gen).long()]


def _mutate(x, lut, rate, gen):
    """Substitutes symbols at `rate` (a number or a column of rates)."""
    hit = torch.rand(x.shape, device="cuda", generator=gen) < rate
    return torch.where(hit, _random(x.numel(), lut, gen).view(x.shape), x)


def _genome(n, alphabet, seed, shift=0):
    """`n` symbols: background letters, half interspersed diverged repeats, 4%
    tandem repeats and short runs of N (a letter outside the alphabet for
    proteins), `shift` bytes into a fresh buffer."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lut = torch.from_numpy(_letters(alphabet, 0.41)).cuda()
    gap = ord("*") if alphabet == sbf.ALPHABET_PROTEIN else ord("N")
    units = _random(2000 * _SEG, lut, gen).view(2000, _SEG)
    out = torch.empty(n + shift, dtype=torch.uint8, device="cuda")[shift:]
    col = torch.arange(_SEG, device="cuda")
    for i in range(0, n, _STEP):
        m = min(_STEP, n - i)
        rows = (m + _SEG - 1) // _SEG
        blk = _random(rows * _SEG, lut, gen).view(rows, _SEG)
        kind = torch.rand(rows, device="cuda", generator=gen)
        rep = (kind < 0.5).nonzero().flatten()
        which = torch.randint(0, 2000, (rep.numel(),), device="cuda", generator=gen)
        rate = 0.05 + 0.15 * torch.rand((rep.numel(), 1), device="cuda", generator=gen)
        blk[rep] = _mutate(units[which], lut, rate, gen)
        tan = ((kind >= 0.5) & (kind < 0.54)).nonzero().flatten()
        period = torch.randint(2, 201, (tan.numel(), 1), device="cuda", generator=gen)
        blk[tan] = torch.gather(blk[tan], 1, col[None, :] % period)
        runs = ((kind >= 0.54) & (kind < 0.542)).nonzero().flatten()
        length = torch.randint(10, 1001, (runs.numel(), 1), device="cuda", generator=gen)
        blk[runs] = torch.where(col[None, :] < length, gap, blk[runs])
        out[i:i + m] = blk.view(-1)[:m]
    return out


def _reads(genome, case, seed):
    """Reads of one length joined by N: half of them from the genome with 1%
    substitutions, half random."""
    n, length = case["reads"], case["read_len"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lut = torch.from_numpy(_letters(case["alphabet"], 0.5)).cuda()
    gap = ord("*") if case["alphabet"] == sbf.ALPHABET_PROTEIN else ord("N")
    buf = torch.empty(n * (length + 1) + case["shift"], dtype=torch.uint8, device="cuda")
    out = buf[case["shift"]:].view(n, length + 1)
    out[:, length] = gap
    col = torch.arange(length, device="cuda")
    for i in range(0, n, 1 << 20):
        m = min(1 << 20, n - i)
        start = torch.randint(0, genome.numel() - length, (m, 1), device="cuda", generator=gen)
        src = _mutate(genome[start + col[None, :]], lut, 0.01, gen)
        own = torch.rand((m, 1), device="cuda", generator=gen) < 0.5
        out[i:i + m, :length] = torch.where(own, src, _random(m * length, lut, gen).view(m, length))
    return buf[case["shift"]:][:n * (length + 1) - 1]


def _lengths(case, count, seed):
    """Record lengths: the case's own set, in an order that the seed gives."""
    x = np.random.default_rng(count).lognormal(math.log(case["median"]), case["sigma"], size=count)
    x = np.clip(np.round(x), 20, 200 * case["median"]).astype(np.int64)
    return np.random.default_rng(seed).permutation(x)


def _ranges(lengths):
    off = np.concatenate([[0], np.cumsum(lengths)[:-1]])
    return torch.from_numpy(np.stack([off, lengths], axis=1)).cuda()


def _ragged_reads(genome, case, seed):
    """Reads of uneven length, back to back: 60% from the genome with 0.5%
    substitutions, the rest random."""
    lens = np.minimum(_lengths(case, case["reads"], seed), genome.numel() - 1)
    ranges = _ranges(lens)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    lut = torch.from_numpy(_letters(case["alphabet"], 0.41)).cuda()
    n, total = lens.size, int(lens.sum())
    own = torch.rand(n, device="cuda", generator=gen) < 0.6
    start = (torch.rand(n, device="cuda", generator=gen, dtype=torch.float64) *
             (genome.numel() - ranges[:, 1])).long()
    out = torch.empty(total + case["shift"], dtype=torch.uint8, device="cuda")[case["shift"]:]
    ends = np.cumsum(lens)
    i = 0
    while i < n:
        j = min(n, max(i + 1, int(np.searchsorted(ends, ends[i] + _STEP))))
        a, b = int(ends[i] - lens[i]), int(ends[j - 1])
        rid = torch.repeat_interleave(torch.arange(i, j, device="cuda"), ranges[i:j, 1])
        rel = torch.arange(a, b, device="cuda") - ranges[rid, 0]
        src = _mutate(genome[start[rid] + rel], lut, 0.005, gen)
        out[a:b] = torch.where(own[rid], src, _random(b - a, lut, gen))
        i = j
    return out, ranges


def _query_sequence(genome, case, seed):
    if case["reads"]:
        return _reads(genome, case, seed)
    # A sequence that shares its first half with the genome.
    n, shift = case["query"], case["shift"]
    out = _genome(n, case["alphabet"], seed, shift)
    m = min(n // 2, genome.numel())
    out[:m] = genome[:m]
    return out


def _pack(seq, alphabet):
    """Dense words of device symbols: 32 DNA or 12 protein symbols per word."""
    words = torch.empty(sbf.Filter.dense_packed_word_count(seq.numel(), alphabet),
                        dtype=torch.int64, device="cuda")
    sbf.pack_dense_sequence_device(seq, seq.numel(), words, alphabet=alphabet)
    return words


def prepare(case, seed):
    op = case["op"]
    cfg = {x: case[x] for x in ("k", "s", "m", "hashes", "alphabet")}
    f = sbf.Filter(1 << case["log2_bits"], **cfg)
    plain_insert = op == "insert"
    genome = _genome(case["genome"], case["alphabet"], 2 * seed,
                     case["shift"] if plain_insert or op == "ragged_insert" else 0)
    words = f.words().view(torch.int64)
    words.filter = f  # the tensor aliases the filter's memory: it keeps the filter alive
    st = {"op": op, "filter": f, "words": words}
    if op == "insert":
        st["seq"] = genome
    elif op == "dense_insert":
        st["seq"], st["symbols"] = _pack(genome, case["alphabet"]), genome.numel()
    elif op == "ragged_insert":
        lens = _lengths(case, 2 * case["genome"] // case["median"] + 1, seed)
        lens = lens[:max(1, int(np.searchsorted(np.cumsum(lens), case["genome"], side="right")))]
        lens[0] = min(int(lens[0]), case["genome"])
        st["ranges"] = _ranges(lens)
        st["seq"] = genome[:int(lens.sum())]
    else:
        f.insert_sequence_async(genome)
        if op == "ragged_query":
            st["seq"], st["ranges"] = _ragged_reads(genome, case, 2 * seed + 1)
            n = st["ranges"].shape[0]
            st["valid"] = torch.empty(n, dtype=torch.int64, device="cuda")
            st["positive"] = torch.empty(n, dtype=torch.int64, device="cuda")
            symbols = st["seq"].numel()
        else:
            seq = _query_sequence(genome, case, 2 * seed + 1)
            symbols = st["symbols"] = seq.numel()
            st["seq"] = _pack(seq, case["alphabet"]) if op == "dense_query_bits" else seq
        n = max(symbols - case["k"] + 1, 1)
        if op.endswith("bits"):
            st["out"] = torch.empty((n + 31) // 32, dtype=torch.int32, device="cuda")
        else:
            st["out"] = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    f, op = st["filter"], st["op"]
    if op == "insert":
        return {"kmers": f.insert_sequence_async(st["seq"]), "words": st["words"]}
    if op == "dense_insert":
        return {"kmers": f.insert_dense_packed_async(st["seq"], st["symbols"]),
                "words": st["words"]}
    if op == "ragged_insert":
        f.ragged_insert_async(st["seq"], st["ranges"])
        return {"words": st["words"]}
    if op == "ragged_query":
        f.ragged_contains_counts_async(st["seq"], st["ranges"], st["valid"], st["positive"],
                                       st["out"])
        return {"hits": st["out"], "valid": st["valid"], "positive": st["positive"]}
    if op == "query":
        f.contains_sequence_async(st["seq"], st["out"])
    elif op == "query_bits":
        f.contains_sequence_bits_async(st["seq"], st["out"])
    else:
        f.contains_dense_packed_bits_async(st["seq"], st["symbols"], st["out"])
    return {"hits": st["out"]}


def work(case):
    """Bytes of one pass: the input once, the output once, and one 32-byte
    shard per super-k-mer run (2 runs per W + 1 windows of random sequence),
    read by queries, read and written by inserts; a filter smaller than that
    is read, or read and written, once."""
    op = case["op"]
    if op in ("insert", "dense_insert", "ragged_insert"):
        n = case["genome"]
    elif op == "ragged_query":
        n = case["reads"] * case["median"] * math.exp(case["sigma"] ** 2 / 2)
    else:
        n = case["reads"] * (case["read_len"] + 1) if case["reads"] else case["query"]
    bits = 5 if case["alphabet"] == sbf.ALPHABET_PROTEIN else 2
    inp = n / (64 // bits) * 8 if op.startswith("dense") else n
    shards = min(32 * 2 * n / (case["k"] - case["m"] + 2), 2.0 ** case["log2_bits"] / 8)
    if "insert" in op:
        return {"bytes": inp + 2 * shards, "flops": 0}
    return {"bytes": inp + shards + (n / 8 if op.endswith("bits") else n), "flops": 0}
