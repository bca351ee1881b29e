"""The tensor-core scorer's bounded waits: a list's lock that nobody gives back
runs out (and with it the pipeline's waits of the CTA that wants it), the search
reports HFX_ERR_TIMEOUT, and the context searches on.  And its long items:
several passes of 512 candidates, the last one short, windows that begin and end
in different passes."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_lock_wait_runs_out(gpulib, monkeypatch, precision):
    import hfx_gb300
    prot = synth.proteins(400, seed=3)
    eng = hfx_gb300.Engine(0)
    try:
        eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
        sp = synth.spectra(prot, 200, seed=5, charge_p={2: 1.0}, npeaks=(50, 400))
        sp.tol[:] = 1e5
        p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision)
        ref = eng.search(sp, p)
        monkeypatch.setenv("HFX_TEST_HOLD_LOCK", "1")
        with pytest.raises(hfx_gb300.HfxError) as ei:
            eng.search(sp, p)
        assert ei.value.code == hfx_gb300.HFX_ERR_TIMEOUT
        monkeypatch.delenv("HFX_TEST_HOLD_LOCK")
        again = eng.search(sp, p)
        assert np.array_equal(again.key, ref.key)
        assert np.array_equal(again.score.view(np.uint32), ref.score.view(np.uint32))
    finally:
        eng.close()


@pytest.fixture(scope="module")
def long_items(gpulib, oracle):
    """2,400 spectra over some 180,000 candidates: 19 blocks, items of three passes."""
    import hfx_gb300
    prot = synth.proteins(2500, seed=3)
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    r, tc, tn, idx, mt = eng.db_export()
    sp = synth.spectra(prot, 2400, seed=9, charge_p={2: 1.0}, npeaks=(50, 200))
    rng = np.random.default_rng(2)
    # the lighter half all candidates or some, the heavier half unions of its own per block
    light = (sp.pcr < np.median(sp.pcr)) & (rng.random(2400) < 0.5)
    sp.tol[:] = np.where(light, 1e5, rng.uniform(1500.0, 2500.0, 2400)).astype(np.float32)
    some = np.sort(rng.choice(2400, 60, replace=False))
    ref = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sp.subset(some), topn=10)
    assert len(r) * 19 // (12 * 152) // 512 >= 3
    yield eng, sp, some, ref
    eng.close()


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_items_of_several_passes(long_items, precision):
    import hfx_gb300
    eng, sp, some, (sc, _, key, _, nc) = long_items
    eng.set_profiling(True)
    eng.stage_stats()
    res = eng.search(sp, hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, rescore_k=32))
    launches = eng.stage_stats()["score"][1]
    eng.set_profiling(False)
    assert launches == 2
    assert np.array_equal(res.ncand[some], nc)
    assert np.array_equal(res.key[some], key)
    assert np.array_equal(np.ascontiguousarray(res.score[some]).view(np.uint32), sc.view(np.uint32))
