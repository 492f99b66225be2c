"""Run records at the edges of tiles (4096 windows, a CTA each), and of windows
short enough that a tile's runs overflow the CTA's log of 768 records: applied
to an empty filter they give the oracle's words."""
import numpy as np
import pytest

from conftest import random_dna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg", [dict(k=31, s=28, m=16, hashes=4), dict(k=21, s=19, m=11, hashes=4),
                                 dict(k=5, s=4, m=3, hashes=4), dict(k=3, s=2, m=2, hashes=4)],
                         ids=["k31", "k21", "k5", "k3"])
def test_emitted_runs_build_the_filter(sbf, cuda, oracle_mod, cfg):
    torch = cuda
    k = cfg["k"]
    rng = np.random.default_rng(k)
    seq = random_dna(rng, 300_000, b"ACGT" * 100 + b"N")
    o = oracle_mod.Oracle(**cfg)
    bad = np.concatenate([[0], np.cumsum(seq == ord("N"))])
    f = sbf.Filter(1 << 18, **cfg)
    for n in (1, 31, 4_095, 4_096, 4_097, 250_000):
        part = seq[:n + k - 1]
        words = o.new_words(1 << 18)
        o.insert(words, part)
        shards, masks, valid = f.emit_runs(torch.from_numpy(part.copy()).cuda())
        assert valid == int((bad[k:n + k] == bad[:n]).sum())
        f.clear()
        f.apply_runs(shards, masks, 0, f.num_shards())
        f.synchronize()
        np.testing.assert_array_equal(f.words_host(), words)
