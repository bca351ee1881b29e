"""FP32 graph replays that alternate between a batch whose open windows have ties
(scored by the list scorer) and one that has none and more work items: a capture
that has met ties stays with the list scorer, so neither captures anew for ever."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_batches_with_and_without_ties(gpulib, oracle):
    import hfx_gb300
    prot = synth.proteins(1500, seed=3)
    eng = hfx_gb300.Engine(0)
    try:
        eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
        r, tc, tn, idx, mt = eng.db_export()
        n = 512
        sp = synth.spectra(prot, n, seed=5, charge_p={2: 1.0}, npeaks=(50, 400))
        d = torch.device("cuda:0")
        dev = {k: torch.from_numpy(getattr(sp, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
        out = dict(score=torch.empty((n, 10), device=d), key=torch.empty((n, 10), dtype=torch.int64, device=d),
                   pep=torch.empty((n, 10), dtype=torch.int32, device=d))
        p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=0, use_graph=1)
        some = np.arange(0, n, 32)
        peaks, pcr = sp.it.copy(), sp.pcr.copy()
        captures = []
        for turn in range(8):
            ties = turn % 2 == 0
            sp.it[:] = 0.0 if ties else peaks
            sp.tol[:] = 80.0 if ties else 1e5
            sp.pcr[:] = 700.0 if ties else pcr     # few candidates, all in common
            for k in ("it", "tol", "pcr"):
                dev[k].copy_(torch.from_numpy(getattr(sp, k)))
            torch.cuda.synchronize()
            eng.stage_stats()
            eng.search_device(dev, p, out)
            captures.append(eng.stage_stats()["windows"][1] > 0)
            sc, _, key, _, _ = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, sp.subset(some), topn=10)
            assert np.array_equal(out["key"].cpu().numpy().view(np.uint64)[some], key), turn
            assert np.array_equal(np.ascontiguousarray(out["score"].cpu().numpy()[some]).view(np.uint32),
                                  sc.view(np.uint32)), turn
        assert captures[0] and not any(captures[4:]), captures
    finally:
        eng.close()
