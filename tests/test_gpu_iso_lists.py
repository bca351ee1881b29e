"""The isoform-list scorer where its pipeline starves or its groups change:
items of a few positions, the default group and every explicit one, FP32 in
the canonical order and BF16/FP16 with FP32 rescoring, against the oracle bit
for bit."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

MA, MA_MASS = b"MSTY", [15.995, 79.966, 79.966, 79.966]


@pytest.fixture(scope="module")
def search(gpulib, oracle):
    import hfx_gb300
    prot = synth.proteins(3000, seed=4)
    sp = synth.spectra(prot, 61, seed=9, charge_p={1: 0.1, 2: 0.4, 3: 0.3, 4: 0.2}, npeaks=(50, 400))
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    eng.set_mods(MA.decode(), MA_MASS, 4, False)
    r, tc, tn, idx, mt = eng.db_export()
    ref = oracle.search(oracle.pack_ions(prot.seq, MA), mt, r, tc, tn, idx, sp, topn=10, ma=MA, ma_mass=MA_MASS,
                        max_ma=4)
    yield eng, sp, ref
    eng.close()


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("G", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("chunk", [0, 3, 40])
def test_items_and_groups(search, chunk, G, precision):
    import hfx_gb300
    eng, sp, (sc, _, key, pep, nc) = search
    res = eng.search(sp, hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, group_size=G, chunk=chunk,
                                                  rescore_k=32 if precision else 0))
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key, key)
    assert np.array_equal(res.score.view(np.uint32), sc.view(np.uint32))
    assert np.array_equal(res.pep, pep)
