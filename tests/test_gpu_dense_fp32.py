"""FP32 searches of wide windows: the results are those of scoring every pair in
FP32 also where many candidates tie to within rounding (spectra of a few peaks),
so that the 32 best by the tensor cores' scores do not hold the FP32 winners.
Against the oracle, bit for bit; alone, beside ordinary spectra, in graphs."""
import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def few_peaks(n, seed):
    """Spectra of one to three peaks and a last one at 200 to 350 m/z; the first has
    hundreds of candidates tied for the first place."""
    rng = np.random.default_rng(seed)
    mz, it, off = [101.57652837, 200.0], [1.0, 2.0], [0, 2]
    for _ in range(n - 1):
        last = rng.uniform(200.0, 350.0)
        k = int(rng.integers(1, 4))
        mz += sorted(rng.uniform(90.0, last - 5.0, k)) + [last]
        it += list(rng.integers(1, 10, k + 1).astype(float))
        off.append(len(mz))
    pcr = np.where(np.arange(n) == 0, 600.0, rng.uniform(400.0, 900.0, n))
    return synth.Spectra(np.array(mz, np.float32), np.array(it, np.float32), np.array(off, np.int64),
                         pcr.astype(np.float32), np.full(n, 2.0, np.float32), np.full(n, 500.0, np.float32))


def join(a, b):
    return synth.Spectra(*[np.concatenate([getattr(a, k), getattr(b, k)]) if k != "off"
                           else np.concatenate([a.off, b.off[1:] + a.off[-1]])
                           for k in ("mz", "it", "off", "pcr", "z", "tol")])


@pytest.fixture(scope="module")
def search(gpulib, oracle):
    import hfx_gb300
    prot = synth.proteins(2500, seed=3)
    eng = hfx_gb300.Engine(0)
    eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
    r, tc, tn, idx, mt = eng.db_export()
    sparse = few_peaks(150, 4)
    plain = synth.spectra(prot, 250, seed=9, charge_p={2: 1.0}, npeaks=(50, 400))
    plain.tol[:] = 500.0
    both = join(sparse, plain)
    ref = oracle.search(oracle.pack_ions(prot.seq), mt, r, tc, tn, idx, both, topn=16)
    yield eng, both, ref
    eng.close()


def _same(res, ref, n, top_n):
    sc, _, key, _, nc = ref
    assert np.array_equal(res.ncand, nc[:n])
    assert np.array_equal(res.key, key[:n, :top_n])
    assert np.array_equal(res.score.view(np.uint32), sc[:n, :top_n].view(np.uint32))


@pytest.mark.parametrize("n", [150, 400])
@pytest.mark.parametrize("top_n", [1, 10, 16])
def test_tied_candidates(search, n, top_n):
    import hfx_gb300
    eng, sp, ref = search
    p = hfx_gb300.default_params(top_n=top_n, batch_mode=1, precision=0)
    eng.set_profiling(True)
    eng.stage_stats()
    _same(eng.search(sp.subset(np.arange(n)), p), ref, n, top_n)
    st = eng.stage_stats()
    eng.set_profiling(False)
    assert st["score"][1] == 2     # list-scored groups and tensor-core blocks
    assert st["rescore"][1] > 4    # and a second plan for the ties


def test_graph(search):
    """A graph made of a batch with ties, and one of ordinary spectra that then
    meets ties."""
    import hfx_gb300
    eng, sp, (sc, _, key, _, _) = search
    d = torch.device("cuda:0")
    n = 100
    p = hfx_gb300.default_params(top_n=10, batch_mode=1, precision=0, use_graph=1)
    for order in ((0, 0, 150, 0), (150, 150, 0, 150)):
        dev = None
        for first in order:
            sub = sp.subset(np.arange(first, first + n))
            new = {k: torch.from_numpy(getattr(sub, k).copy()).to(d) for k in ("mz", "it", "off", "pcr", "z", "tol")}
            if dev is None:   # the buffers of every batch: room for the longest
                dev = {k: torch.zeros(401 * n, dtype=v.dtype, device=d) if k in ("mz", "it") else v.clone()
                       for k, v in new.items()}
                out = dict(score=torch.empty((n, 10), device=d),
                           key=torch.empty((n, 10), dtype=torch.int64, device=d),
                           pep=torch.empty((n, 10), dtype=torch.int32, device=d))
            for k, v in new.items():
                dev[k][:len(v)].copy_(v)
            torch.cuda.synchronize()
            eng.search_device(dev, p, out)
            at = slice(first, first + n)
            assert np.array_equal(out["key"].cpu().numpy().view(np.uint64), key[at, :10]), (order, first)
            assert np.array_equal(out["score"].cpu().numpy().view(np.uint32),
                                  np.ascontiguousarray(sc[at, :10]).view(np.uint32)), (order, first)
