"""Searches under a workspace limit: what helps speed alone (tensor-core tiles and
queues, more and smaller work items, lists of work) is left out where it does
not fit, and the results stay the same."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu


def _engine(prot, mods=False):
    import hfx_gb300
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    if mods:
        eng.set_mods("MSTY", [15.995, 79.966, 79.966, 79.966], 3, False)
    return eng


def _used(prot, run, mods=False):
    eng = _engine(prot, mods)
    try:
        eng.set_workspace_limit(0)
        ref = run(eng)
        return eng.set_workspace_limit(0), ref, eng.mod_counters() if mods else None
    finally:
        eng.close()


def _same(a, b, n=None):
    assert np.array_equal(a.ncand, b.ncand)
    assert np.array_equal(a.key[:, :n], b.key[:, :n])
    assert np.array_equal(np.ascontiguousarray(a.score[:, :n]).view(np.uint32),
                          np.ascontiguousarray(b.score[:, :n]).view(np.uint32))


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("graph", [0, 1])
def test_open_windows_in_the_list_scorers_room(gpulib, precision, graph):
    """17 FP32 results, or 33 candidates kept for rescoring, are list-scored; the
    same windows with 16 (32) have to run in that room."""
    import hfx_gb300
    prot = synth.proteins(400, seed=3)
    sp = synth.spectra(prot, 400, seed=77, charge_p={2: 1.0}, npeaks=(50, 400))
    sp.tol[:] = 1e5

    def params(more):
        if precision == 0:
            return hfx_gb300.default_params(top_n=16 + more, batch_mode=1, precision=0, use_graph=graph)
        return hfx_gb300.default_params(top_n=10, rescore_k=32 + more, batch_mode=1, precision=precision,
                                        use_graph=graph)
    used, ref, _ = _used(prot, lambda e: e.search(sp, params(1)))
    eng = _engine(prot)
    try:
        eng.set_workspace_limit(used)
        res = eng.search(sp, params(0))
        _same(res, ref, 10)
        assert np.array_equal(eng.search(sp, params(0)).key, res.key)
        assert eng.set_workspace_limit(0) <= used
        assert np.array_equal(eng.search(sp, params(0)).key, res.key)   # and without the limit
    finally:
        eng.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_isoform_lists_without_lists_of_work(gpulib, precision):
    """The isoforms' lists of work take 16 bytes a record beside the lists: half of
    that less has to do."""
    import hfx_gb300
    prot = synth.proteins(400, seed=3)
    sp = synth.spectra(prot, 120, seed=7, charge_p={2: 0.7, 3: 0.3}, npeaks=(50, 400))
    sp.tol[:] = 3.0
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, search_mods=1)

    def run(eng):
        eng.set_profiling(True)
        eng.mod_counters()
        return eng.search(sp, p)
    used, ref, c = _used(prot, run, mods=True)
    records = c["isoforms"]
    assert records > 10000
    eng = _engine(prot, mods=True)
    try:
        eng.set_workspace_limit(used - 8 * records)
        _same(eng.search(sp, p), ref)
    finally:
        eng.close()


def test_list_search_takes_no_more_than_its_lists(gpulib):
    """Lists, their lengths and two coverage arrays, and under 1.5 MB for the rest."""
    import hfx_gb300
    prot = synth.proteins(2500, seed=3)
    sp = synth.spectra(prot, 4, seed=7, charge_p={2: 0.7, 3: 0.3}, npeaks=(50, 100))
    sp.tol[:] = 0.05
    eng = _engine(prot)
    try:
        r, tc, tn, idx, mt = eng.db_export()
        units = int(((10 * (tn.astype(np.int64) - tc) + 7) & ~7).sum())
        room = 20 * units + (2 * 16 + 8) * len(r) + 1_500_000
        eng.set_workspace_limit(room)
        eng.search(sp, hfx_gb300.default_params(top_n=10, batch_mode=1, precision=0))
    finally:
        eng.close()


@pytest.mark.parametrize("mods", [0, 1])
def test_evalues_in_the_least_room(gpulib, mods):
    """E-values under a limit below what the search holds without one, and the room
    is not found before its last workspaces."""
    import hfx_gb300
    torch = pytest.importorskip("torch")
    prot = synth.proteins(400, seed=3)
    n = 60
    sp = synth.spectra(prot, n, seed=7, charge_p={2: 0.7, 3: 0.3}, npeaks=(50, 400))
    d = torch.device("cuda:0")
    dev = {k: torch.from_numpy(getattr(sp, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=1, search_mods=mods)

    def run(eng):
        out = dict(score=torch.empty((n, 10), device=d), key=torch.empty((n, 10), dtype=torch.int64, device=d),
                   pep=torch.empty((n, 10), dtype=torch.int32, device=d),
                   ncand=torch.empty(n, dtype=torch.int64, device=d),
                   ev=torch.empty((n, 10), dtype=torch.float64, device=d),
                   fit=torch.empty((n, 3), dtype=torch.float64, device=d))
        eng.search_evalues(dev, p, out)
        return {k: v.cpu().numpy().copy() for k, v in out.items()}
    used, ref, _ = _used(prot, run, mods=bool(mods))
    eng = _engine(prot, mods=bool(mods))
    try:
        eng.set_workspace_limit(used - 200_000)   # part lists of the few groups' items
        res = run(eng)
        for k in ref:
            assert np.array_equal(res[k].view(np.uint8), ref[k].view(np.uint8)), k
    finally:
        eng.close()
