"""Graph replays of batches whose windows change: a few groups are cut into more
work items the wider their windows are, and groups may be list-scored in one
batch and on the tensor cores in the next.  Neither makes the search capture
anew each time, and the results are the oracle's."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def replayed(gpulib, oracle):
    import hfx_gb300
    prot = synth.proteins(1500, seed=3)
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    r, tc, tn, idx, mt = eng.db_export()
    n = 512
    sp = synth.spectra(prot, n, seed=5, charge_p={2: 1.0}, npeaks=(50, 400))
    sp.pcr[:] = np.repeat(sp.pcr[::8], 8)   # groups of one mass: their windows are as wide as the tolerance
    d = torch.device("cuda:0")
    dev = {k: torch.from_numpy(getattr(sp, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
    out = dict(score=torch.empty((n, 10), device=d), key=torch.empty((n, 10), dtype=torch.int64, device=d),
               pep=torch.empty((n, 10), dtype=torch.int32, device=d))
    some = np.arange(0, n, 16)

    def search(p, tol):
        """Eager launches of a graph search with these windows: none when it is replayed."""
        sp.tol[:] = tol
        dev["tol"].copy_(torch.from_numpy(sp.tol))
        torch.cuda.synchronize()
        eng.stage_stats()
        eng.search_device(dev, p, out)
        sub = sp.subset(some)
        sc, _, key, _, _ = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sub, topn=10)
        assert np.array_equal(out["key"].cpu().numpy().view(np.uint64)[some], key)
        assert np.array_equal(np.ascontiguousarray(out["score"].cpu().numpy()[some]).view(np.uint32),
                              sc.view(np.uint32))
        return eng.stage_stats()["windows"][1]

    yield search
    eng.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_wider_windows_are_replayed(replayed, precision):
    import hfx_gb300
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, use_graph=1)
    assert replayed(p, 2.0) > 0
    for tol in (2.0, 5.0, 8.0):
        assert replayed(p, tol) == 0, tol


@pytest.mark.parametrize("precision", [0, 1])
def test_kinds_of_windows_alternate(replayed, precision):
    import hfx_gb300
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=precision, use_graph=1)
    # every spectrum all candidates (dense blocks), or windows too narrow for them
    for tol in (1e5, 60.0, 1e5):
        replayed(p, tol)
    for tol in (60.0, 1e5, 60.0, 1e5):
        assert replayed(p, tol) == 0, tol
