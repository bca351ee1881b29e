"""Which batches have tensor-core blocks: 32 pairs per candidate of the union, so
31 spectra of one class have none, 32 with all candidates have one, and classes
of fewer spectra have none beside each other.  The results are the oracle's."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(gpulib):
    import hfx_gb300
    prot = synth.proteins(400, seed=3)
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    yield eng, prot
    eng.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("charges,launches", [({2: 31}, 1), ({2: 32}, 2), ({2: 33}, 2), ({2: 160}, 2),
                                              ({2: 20, 3: 20, 4: 20, 5: 20}, 1), ({2: 31, 3: 33}, 2)])
def test_blocks(engine, oracle, precision, charges, launches):
    import hfx_gb300
    eng, prot = engine
    n = sum(charges.values())
    sp = synth.spectra(prot, n, seed=n, charge_p={2: 1.0}, npeaks=(50, 200))
    sp.z[:] = np.repeat(list(charges), list(charges.values()))
    sp.tol[:] = 1e5
    r, tc, tn, idx, mt = eng.db_export()
    eng.set_profiling(True)
    eng.stage_stats()
    res = eng.search(sp, hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, rescore_k=32))
    seen = eng.stage_stats()["score"][1]
    eng.set_profiling(False)
    assert seen == launches
    sc, _, key, _, nc = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sp, topn=10)
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key, key)
    assert np.array_equal(res.score.view(np.uint32), sc.view(np.uint32))


@pytest.mark.parametrize("precision,top_n,rescore_k,launches", [
    (1, 16, 32, 2), (1, 17, 32, 1), (1, 16, 10, 1), (2, 10, 20, 2), (2, 10, 19, 1), (0, 16, 0, 2), (0, 17, 0, 1)])
def test_candidates_to_spare(engine, precision, top_n, rescore_k, launches):
    """The tensor cores choose candidates only where twice the results are kept."""
    import hfx_gb300
    eng, prot = engine
    sp = synth.spectra(prot, 64, seed=64, charge_p={2: 1.0}, npeaks=(50, 200))
    sp.tol[:] = 1e5
    eng.set_profiling(True)
    eng.stage_stats()
    eng.search(sp, hfx_gb300.default_params(top_n=top_n, batch_mode=1, precision=precision, rescore_k=rescore_k))
    seen = eng.stage_stats()["score"][1]
    eng.set_profiling(False)
    assert seen == launches
