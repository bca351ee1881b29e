"""Rows of more bins than a 22-bit or a 28-bit bin number holds (custom widths of
0.0003 and 0.000005 Da): the ions' bins are the correctly rounded quotients up to
the row's end.  Against the ions in NumPy's FP32 and the oracle's scores of their
lists, bit for bit."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

f32 = np.float32
H, H2O, NH3, CO = f32(1.0078246), f32(18.01056), f32(17.02655), f32(27.9949)


def ladder(ions, mt, tc, tn):
    """Prefix masses as the warp scans sum them: 32 residues at a time."""
    out, carry = [], f32(0)
    for c in range(tc, tn, 32):
        n = min(32, tn - c)
        v = np.zeros(32, f32)
        v[:n] = mt[ions[c:c + n] & 31]
        v[0] += carry
        for d in (1, 2, 4, 8, 16):
            v[d:] = v[d:] + v[:-d]
        out.append(v[:n])
        carry = v[n - 1]
    return np.concatenate(out) if out else np.zeros(0, f32)


def fragment_mz(b, y, z):
    """m/z of the b- and y-ions and of the 10s (a, b - H2O, b - NH3, y - NH3)."""
    z, hc = f32(z), H * f32(z)
    mb, my = (b + hc) / z, ((y + H2O) + hc) / z
    return mb, my, [((b - CO) + hc) / z, mb - H2O / z, mb - NH3 / z, my - NH3 / z]


def ion_list(ions, mt, tc, tn, r, charges, width, nbins):
    b = ladder(ions, mt, tc, tn)
    y = f32(r) - b
    level = {}
    for z in range(1, charges + 1):
        mb, my, tens = fragment_mz(b, y, z)
        for x in tens:
            for k in np.rint(x / width).astype(np.int64):
                level[k] = max(level.get(k, 0), 1)
        for x in (mb, my):
            for k in np.rint(x / width).astype(np.int64):
                for j, v in ((-1, 2), (0, 3), (1, 2)):
                    level[k + j] = max(level.get(k + j, 0), v)
    keys = np.array(sorted(k for k in level if 0 <= k < nbins), np.int64)
    return keys, np.array([level[k] for k in keys], np.uint8)


def sparse_row(mz, width, nbins):
    """The nonzero bins of a row whose peaks lie more than 151 bins apart, all of
    one intensity: 50 - 50 / 150 at a peak, -50 / 150 beside it."""
    x = {}
    for p in mz:
        k = int(np.rint(f32(p) / width))
        for j in range(max(0, k - 75), min(nbins, k + 76)):
            x[j] = f32(0) - f32(50) / f32(150)
        x[k] = f32(50) - f32(50) / f32(150)
    return x


@pytest.mark.parametrize("width", [0.0003, 5e-6])
@pytest.mark.parametrize("precision", [0, 1])
def test_bins_beyond_22_and_28_bits(gpulib, oracle, width, precision):
    import hfx_gb300
    width = f32(width)
    prot = synth.proteins(3, seed=6)
    eng = hfx_gb300.Engine(0)
    try:
        eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
        r, tc, tn, idx, mt = eng.db_export()
        mt = np.concatenate([mt, np.zeros(6, f32)]).astype(f32)
        ions = oracle.pack_ions(prot.seq)
        order = [p for p in idx if 2500 < r[p] < 3500]
        # peaks: ions of a few peptides, far apart
        mz = []
        for p in order[:6]:
            b = ladder(ions, mt, tc[p], tn[p])
            for z in (1, 2):
                mb, my, _ = fragment_mz(b, f32(r[p]) - b, z)
                mz += [float(m) for m in np.concatenate([mb, my]) if 900 < m < 1990]
        mz = np.array([m for i, m in enumerate(sorted(mz)) if i % 3 == 0], f32)
        mz = mz[np.concatenate([[True], np.diff(mz) > 0.2])]
        mz = np.append(mz, f32(2000.0))
        sp = synth.Spectra(mz, np.full(len(mz), 4.0, f32), np.array([0, len(mz)], np.int64), np.array([1500.0], f32),
                           np.array([3.0], f32), np.array([1e5], f32))
        nbins = 75 + int(np.ceil(f32(2000.0) / width))
        assert nbins > (1 << 22 if width > 1e-5 else 1 << 28)
        row = sparse_row(mz[:-1], width, nbins)  # (the last peak lies past the ten regions)
        p = hfx_gb300.default_params(top_n=10, precision=precision, rescore_k=50 if precision else 0, batch_mode=1,
                                     bin_width=float(width), custom_bin_width=1, ion_bins_custom=1,
                                     remove_precursor_peak=0, max_len=2 ** 30 - 1)
        res = eng.search(sp, p)
        scores = []
        for q in idx:
            keys, lvl = ion_list(ions, mt, tc[q], tn[q], r[q], 2, width, nbins)
            x = np.array([row.get(k, f32(0)) for k in keys], f32)
            scores.append(oracle.score32(np.arange(len(keys), dtype=np.uint32), lvl, x) if len(keys) else 0.0)
        scores = np.array(scores, f32)
        best = np.lexsort((np.arange(len(idx)), -scores))[:10]
        assert scores[best[0]] > 5000
        assert np.array_equal(res.key[0], best.astype(np.uint64))
        assert np.array_equal(res.score[0].view(np.uint32), scores[best].view(np.uint32))
    finally:
        eng.close()
