"""Scores that are no numbers (candidates with an ion in an infinite intensity's
bin).  The per-spectrum path keeps its insertion order over warps, blocks and
lists, restated here; the batched paths name no candidate twice."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
NONE = (-np.inf, 2 ** 64 - 1)


def insert(entries, new, k):
    at = sum(1 for e in entries if e[0] > new[0] or (e[0] == new[0] and e[1] < new[1]))
    if at < k:
        entries[:] = (entries[:at] + [new] + entries[at:])[:k]


def fold(lists, k):
    out = [NONE] * k
    for entries in lists:
        for e in entries:
            if e[1] != NONE[1]:
                insert(out, e, k)
    return out


@pytest.fixture(scope="module")
def search(gpulib, oracle):
    import hfx_gb300
    prot = synth.proteins(300, seed=8)
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    sp = synth.spectra(prot, 40, seed=31, charge_p={2: 0.6, 3: 0.4}, npeaks=(40, 120))
    sp.tol[:] = 20.0
    for s in range(40):
        sp.it[sp.off[s] + (s * 7) % (sp.off[s + 1] - sp.off[s])] = np.inf
    # of the first ones, the bins that all peptides ending in K or R touch
    for s in range(10):
        sp.mz[sp.off[s]] = 147.1 if s % 2 else 175.1
        sp.it[sp.off[s]] = np.inf
    yield eng, prot, sp
    eng.close()


@pytest.mark.parametrize("top_n", [1, 10, 32])
def test_per_spectrum_order(search, oracle, top_n):
    import hfx_gb300
    eng, prot, sp = search
    r, tc, tn, idx, mt = eng.db_export()
    ions = oracle.pack_ions(prot.seq)
    d = torch.device("cuda:0")
    dev = {k: torch.from_numpy(getattr(sp, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
    p = hfx_gb300.default_params(top_n=top_n)
    stride = 8192
    rows = torch.empty((len(sp), stride), device=d)
    lens = torch.empty(len(sp), dtype=torch.int32, device=d)
    eng.preprocess(dev, p, stride, rows, lens=lens)
    rows, lens = rows.cpu().numpy(), lens.cpu().numpy()
    res = eng.search(sp, p)
    seen = 0
    for s in range(len(sp)):
        m = np.float32(oracle.ms2_mass(sp.pcr[s], sp.z[s]))
        b, e = oracle.windows(r[idx], [m - np.float32(20)], [m + np.float32(20)])
        b, e = int(b[0]), int(e[0])
        scores = []
        for pos in range(b, e):
            q = idx[pos]
            bins, lvl = oracle.ion_bins(ions, mt, tc[q], tn[q], r[q], int(sp.z[s]) - 1, int(lens[s]))
            scores.append(oracle.score32(bins, lvl, rows[s]))
        seen += int(np.isnan(scores).any() and not np.isnan(scores).all())
        blocks = min((e - b + 31) // 32, 304)
        parts = []
        for blk in range(blocks):
            warps = []
            for w in range(8):
                mine = range(blk * 8 + w, e - b, blocks * 8)
                warps.append(fold([[(scores[i], b + i) for i in mine]], top_n))
            parts.append(fold(warps, top_n))
        want = fold(parts, top_n)
        assert np.array_equal(res.key[s], np.array([k for _, k in want], np.uint64)), s
        assert np.array_equal(res.score[s], np.array([v for v, _ in want], np.float32), equal_nan=True), s
    assert seen > 5


@pytest.mark.parametrize("kept", [(0, 0), (1, 32), (1, 64)])
def test_finite_results_stay(search, oracle, kept):
    """Batched: spectra without a bin that a candidate touches keep their results."""
    import hfx_gb300
    eng, prot, sp = search
    sub = sp.subset(np.arange(10, 40))
    for s in range(0, 30, 2):
        sub.it[sub.off[s]:sub.off[s + 1]] = np.minimum(sub.it[sub.off[s]:sub.off[s + 1]], 1e6)
    r, tc, tn, idx, mt = eng.db_export()
    sc, _, key, _, _ = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sub.subset(np.arange(0, 30, 2)),
                                     topn=10)
    res = eng.search(sub, hfx_gb300.default_params(top_n=10, batch_mode=1, precision=kept[0], rescore_k=kept[1]))
    assert np.array_equal(res.key[::2], key)
    assert np.array_equal(res.score[::2].view(np.uint32), sc.view(np.uint32))
