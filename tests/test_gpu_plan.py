"""Batch planning at the sizes where it changes course: one block's sort up to
1,024 spectra, mass buckets beyond; charge classes of one spectrum and of many,
equal masses, spectra without a row.  Against the oracle, bit for bit."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def search(gpulib, oracle):
    import hfx_gb300
    prot = synth.proteins(300, seed=8)
    sp = synth.spectra(prot, 1100, seed=12, charge_p={1: 0.02, 2: 0.5, 3: 0.4, 4: 0.08}, npeaks=(20, 60))
    sp.pcr[100:400] = sp.pcr[100]            # many spectra of one mass per charge
    sp.z[5::97] = 9.0                        # no plain ions
    sp.tol[3::7] = 0.4                       # narrow windows, a class apart
    sp.it[sp.off[17]:sp.off[18]] = 0.0
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    r, tc, tn, idx, mt = eng.db_export()
    ref = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sp, topn=5)
    yield eng, sp, ref
    eng.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 1021, 1023, 1024, 1025, 1100])
def test_sorted_and_bucketed(search, n, precision):
    import hfx_gb300
    eng, sp, (sc, _, key, pep, nc) = search
    res = eng.search(sp.subset(np.arange(n)), hfx_gb300.default_params(top_n=5, batch_mode=1, precision=precision,
                                                                       rescore_k=32 if precision else 0))
    assert np.array_equal(res.ncand, nc[:n])
    assert np.array_equal(res.key, key[:n])
    assert np.array_equal(res.score.view(np.uint32), sc[:n].view(np.uint32))
