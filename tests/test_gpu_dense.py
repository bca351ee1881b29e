"""Wide windows on the tensor cores: blocks of up to 128 spectra
whose windows share most of their candidates.  The screening scores choose the
candidates that FP32 rescoring orders, so the top-10 and its FP32 scores are the
oracle's: partial blocks, windows that begin and end inside a 512-candidate
pass, rows around a 128-bin chunk, every charge, groups of several sizes, graph
replays, spectra with an infinite intensity (left to the list scorer)."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def open_search(gpulib):
    import hfx_gb300
    prot = synth.proteins(400, seed=3)
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    sp = synth.spectra(prot, 400, seed=77, charge_p={1: 0.1, 2: 0.5, 3: 0.3, 4: 0.1}, npeaks=(50, 400))
    yield eng, prot, sp
    eng.close()


def _check(oracle, eng, prot, sp, params, tol, ppm=False):
    sp.tol[:] = tol
    r, tc, tn, idx, mt = eng.db_export()
    res = eng.search(sp, params)
    sc, _, key, pep, nc = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sp, topn=params.top_n)
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key, key)
    assert np.array_equal(res.score.view(np.uint32), sc.view(np.uint32))


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("n,tol", [(400, 1e5), (400, 900.0), (257, 600.0), (17, 1e5), (128, 1500.0)])
def test_wide_windows(open_search, oracle, precision, n, tol):
    import hfx_gb300
    eng, prot, sp = open_search
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, rescore_k=32)
    eng.set_profiling(True)
    eng.stage_stats()
    _check(oracle, eng, prot, sp.subset(np.arange(n)), p, tol)
    launches = eng.stage_stats()["score"][1]
    eng.set_profiling(False)
    # 17 spectra of four charge classes stay below 16 per block: the list scorer's alone
    assert launches == (2 if n > 17 else 1)


@pytest.mark.parametrize("precision,G", [(1, 1), (1, 4), (1, 8), (1, 16), (0, 1), (0, 8)])
def test_group_sizes(open_search, oracle, precision, G):
    import hfx_gb300
    eng, prot, sp = open_search
    p = hfx_gb300.default_params(top_n=5, batch_mode=1, precision=precision, rescore_k=20, group_size=G)
    _check(oracle, eng, prot, sp.subset(np.arange(300)), p, 1200.0)


@pytest.mark.parametrize("top_n", [1, 16, 17])
def test_fp32_results(open_search, oracle, top_n):
    """FP32 rows: up to 16 results are chosen on the tensor cores and rescored,
    more are list-scored."""
    import hfx_gb300
    eng, prot, sp = open_search
    p = hfx_gb300.default_params(top_n=top_n, batch_mode=1, precision=0)
    eng.set_profiling(True)
    eng.stage_stats()
    _check(oracle, eng, prot, sp.subset(np.arange(200)), p, 1e5)
    launches = eng.stage_stats()["score"][1]
    eng.set_profiling(False)
    assert launches == (2 if top_n <= 16 else 1)


def test_mixed_windows(open_search, oracle):
    """Narrow and wide windows in one batch: list-scored groups and dense blocks."""
    import hfx_gb300
    eng, prot, sp = open_search
    tol = np.where(np.arange(400) % 3 == 0, 1e5, 2.0).astype(np.float32)
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=1, rescore_k=32)
    _check(oracle, eng, prot, sp.subset(np.arange(400)), p, tol)


def test_infinite_intensity_keeps_its_neighbours(open_search, oracle):
    """An infinite intensity makes its row NaN: its block is list-scored, the
    others' results stay the oracle's."""
    import hfx_gb300
    eng, prot, sp = open_search
    sub = sp.subset(np.arange(300))
    bad = 41
    sub.it[sub.off[bad] + 3] = np.inf
    sub.tol[:] = 1e5
    r, tc, tn, idx, mt = eng.db_export()
    res = eng.search(sub, hfx_gb300.default_params(top_n=10, batch_mode=1, precision=1, rescore_k=32))
    sc, _, key, _, nc = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sub, topn=10)
    ok = np.arange(300) != bad
    assert np.array_equal(res.ncand, nc)
    assert np.array_equal(res.key[ok], key[ok])
    assert np.array_equal(res.score[ok].view(np.uint32), sc[ok].view(np.uint32))


def test_graph_replay(open_search, oracle):
    """A replay of another batch in the same buffers, and one with more dense
    blocks than the capture had (planned again)."""
    import hfx_gb300
    eng, prot, sp = open_search
    r, tc, tn, idx, mt = eng.db_export()
    sub = sp.subset(np.arange(384))
    d = torch.device("cuda:0")
    dev = {k: torch.from_numpy(getattr(sub, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
    out = dict(score=torch.empty((384, 10), device=d), key=torch.empty((384, 10), dtype=torch.int64, device=d),
               pep=torch.empty((384, 10), dtype=torch.int32, device=d))
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=1, rescore_k=32, use_graph=1)
    for tol in (2.0, 2.0, 900.0, 900.0, 1e5, 700.0):
        sub.tol[:] = tol
        dev["tol"].copy_(torch.from_numpy(sub.tol))
        torch.cuda.synchronize()
        eng.search_device(dev, p, out)
        sc, _, key, _, _ = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sub, topn=10)
        assert np.array_equal(out["key"].cpu().numpy().view(np.uint64), key), tol
        assert np.array_equal(out["score"].cpu().numpy().view(np.uint32), sc.view(np.uint32)), tol
