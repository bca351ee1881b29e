"""A graph's kernels hold the addresses of the workspaces: after an eager search
of the same context that needs larger ones, the next graph search captures anew
and returns the oracle's results."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision", [0, 1])
def test_eager_search_between_replays(gpulib, oracle, precision):
    import hfx_gb300
    prot = synth.proteins(400, seed=3)
    eng = hfx_gb300.Engine(0)
    try:
        eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
        r, tc, tn, idx, mt = eng.db_export()
        sp = synth.spectra(prot, 300, seed=5, charge_p={2: 0.7, 3: 0.3}, npeaks=(50, 400))
        n = 96
        sub = sp.subset(np.arange(n))
        sub.tol[:] = 20.0
        sc, _, key, _, _ = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sub, topn=10)
        d = torch.device("cuda:0")
        dev = {k: torch.from_numpy(getattr(sub, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
        out = dict(score=torch.empty((n, 10), device=d), key=torch.empty((n, 10), dtype=torch.int64, device=d),
                   pep=torch.empty((n, 10), dtype=torch.int32, device=d))
        p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, use_graph=1)
        eager = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision)

        def graph_search():
            """Eager launches of a graph search: none when it is replayed."""
            eng.stage_stats()
            eng.search_device(dev, p, out)
            assert np.array_equal(out["key"].cpu().numpy().view(np.uint64), key)
            assert np.array_equal(out["score"].cpu().numpy().view(np.uint32), sc.view(np.uint32))
            return eng.stage_stats()["windows"][1]

        assert graph_search() > 0       # captured
        assert graph_search() == 0      # replayed
        eng.search(sub, eager)          # the same workspaces
        assert graph_search() == 0
        sp.tol[:] = 1e5
        eng.search(sp, eager)           # larger ones
        assert graph_search() > 0
        assert graph_search() == 0
    finally:
        eng.close()
