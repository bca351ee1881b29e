"""The per-step ion lists at the sizes where their builders change course:
ladders around one and two 32-prefix chunks, longer ones (recomputed per
pass), lists around the 1,024-entry staging buffers, rows around the ends of
a bit word, every charge level.  FP32 search over the lists against the
oracle, bit for bit (the canonical order makes list and scores one)."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 6, 16, 17, 31, 32, 33, 34, 50, 63, 64, 65, 66, 96, 97, 130]


def _database(seed, longest=130):
    rng = np.random.default_rng(seed)
    letters = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWYUBZX", np.uint8)
    seq = letters[rng.integers(0, len(letters), size=4000)].astype(np.uint8)
    tc, tn = [], []
    for k, n in enumerate([n for n in LENGTHS * 2 if n <= longest]):
        a = int(rng.integers(0, 4000 - 140))
        tc.append(a)
        tn.append(a + n)
    mt = np.zeros(26, np.float32)
    for c, m in synth.MONO.items():
        mt[ord(c) - 65] = m
    mt[ord("U") - 65], mt[ord("B") - 65], mt[ord("Z") - 65], mt[ord("X") - 65] = 150.04344, 114.53494, 128.55059, 0.25
    r = np.array([mt[seq[a:b] - 65].astype(np.float64).sum() + (0.0 if i % 3 else 57.0)
                  for i, (a, b) in enumerate(zip(tc, tn))], np.float32)
    return seq, r, np.array(tc, np.uint32), np.array(tn, np.uint32), mt


def _spectra(seed, charge, top_mz):
    """Six spectra of one charge whose rows end near top_mz."""
    rng = np.random.default_rng(seed)
    mz, it, off = [], [], [0]
    for k in range(6):
        m = np.sort(np.append(rng.uniform(60.0, top_mz, size=300 - 40 * k), top_mz + 7.0 * k))
        mz.append(m.astype(np.float32))
        it.append(rng.lognormal(0.0, 1.0, size=len(m)).astype(np.float32))
        off.append(off[-1] + len(m))
    pcr = np.full(6, (top_mz + 200.0) / charge, np.float32)
    return synth.Spectra(np.concatenate(mz), np.concatenate(it), np.array(off, np.int64), pcr,
                         np.full(6, charge, np.float32), np.full(6, 1e5, np.float32))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("top_mz", [330.0, 1013.0, 2000.0, 4085.0, 7990.0])
def test_lists_at_their_edges(gpulib, oracle, top_mz, precision):
    import hfx_gb300
    seq, r, tc, tn, mt = _database(int(top_mz))
    eng = hfx_gb300.Engine(0)
    eng.upload_db(seq, r, tc, tn, mt)
    rs, tcs, tns, idx, _ = eng.db_export()
    parts = [_spectra(10 * c + 1, c, top_mz) for c in (1, 2, 3, 4, 5)]
    off = np.concatenate([[0], np.cumsum(np.concatenate([np.diff(p.off) for p in parts]))]).astype(np.int64)
    sp = synth.Spectra(*(np.concatenate([getattr(p, f) for p in parts]) for f in ("mz", "it")), off,
                       *(np.concatenate([getattr(p, f) for p in parts]) for f in ("pcr", "z", "tol")))
    res = eng.search(sp, hfx_gb300.default_params(top_n=32, batch_mode=1, precision=precision, rescore_k=64))
    sc, _, key, pep, nc = oracle.search(oracle.pack_ions(seq), mt, rs, tcs, tns, idx, sp, topn=32)
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key, key)
    assert np.array_equal(res.score.view(np.uint32), sc.view(np.uint32))
    eng.close()


@pytest.mark.parametrize("custom", [0, 1])
@pytest.mark.parametrize("width", [0.02, 0.0137])
def test_long_row_lists_at_their_edges(gpulib, oracle, width, custom):
    """Rows beyond 8,192 bins: peptides around 1,024 and 2,048 keys (10 keys a
    prefix and charge) and up to 4,000, both ion widths."""
    import hfx_gb300
    seq, r, tc, tn, mt = _database(5, longest=100)
    eng = hfx_gb300.Engine(0)
    eng.upload_db(seq, r, tc, tn, mt)
    rs, tcs, tns, idx, _ = eng.db_export()
    parts = [_spectra(10 * c + 1, c, 1200.0) for c in (1, 2, 3, 4, 5)]
    off = np.concatenate([[0], np.cumsum(np.concatenate([np.diff(p.off) for p in parts]))]).astype(np.int64)
    sp = synth.Spectra(*(np.concatenate([getattr(p, f) for p in parts]) for f in ("mz", "it")), off,
                       *(np.concatenate([getattr(p, f) for p in parts]) for f in ("pcr", "z", "tol")))
    p = hfx_gb300.default_params(top_n=32, batch_mode=1, bin_width=width, custom_bin_width=1, ion_bins_custom=custom)
    res = eng.search(sp, p)
    sc, _, key, pep, nc = oracle.search(oracle.pack_ions(seq), mt, rs, tcs, tns, idx, sp, topn=32, bw=width,
                                        custom_bw=True, ion_bw=width if custom else 0.0)
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key, key)
    assert np.array_equal(res.score.view(np.uint32), sc.view(np.uint32))
    eng.close()


@pytest.mark.parametrize("lengths", [[1], [16], [9, 16, 16], [16, 17, 3, 33, 12]])
def test_short_ladders_share_a_warp(gpulib, oracle, lengths):
    """Ladders of up to 16 prefixes are built two a warp: odd counts (the last
    one alone), neighbours that need different levels, 16 against 17."""
    import hfx_gb300
    seq, _, _, _, mt = _database(3)
    tc = np.array([40 * i for i in range(len(lengths))], np.uint32)
    tn = tc + np.array(lengths, np.uint32)
    r = np.array([mt[seq[a:b] - 65].astype(np.float64).sum() for a, b in zip(tc, tn)], np.float32)
    eng = hfx_gb300.Engine(0)
    eng.upload_db(seq, r, tc, tn, mt)
    rs, tcs, tns, idx, _ = eng.db_export()
    parts = [_spectra(20 * c + 1, c, 1500.0) for c in (2, 3, 5)]
    off = np.concatenate([[0], np.cumsum(np.concatenate([np.diff(p.off) for p in parts]))]).astype(np.int64)
    sp = synth.Spectra(*(np.concatenate([getattr(p, f) for p in parts]) for f in ("mz", "it")), off,
                       *(np.concatenate([getattr(p, f) for p in parts]) for f in ("pcr", "z", "tol")))
    # charge 2 reaches every peptide; 3 and 5 only those around their own mass
    sp.tol[6:] = 300.0
    res = eng.search(sp, hfx_gb300.default_params(top_n=8, batch_mode=1))
    sc, _, key, pep, nc = oracle.search(oracle.pack_ions(seq), mt, rs, tcs, tns, idx, sp, topn=8)
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key, key)
    assert np.array_equal(res.score.view(np.uint32), sc.view(np.uint32))
    eng.close()
