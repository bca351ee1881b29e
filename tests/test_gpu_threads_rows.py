"""Two contexts searched by two threads, one with short rows and one with rows
that need more shared memory: the kernels' shared-memory limit is common to both."""
import threading

import numpy as np
import pytest

from hfx_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_rows_of_two_lengths(gpulib, mode):
    import hfx_gb300
    prot = synth.proteins(60, seed=3)
    sp = synth.spectra(prot, 4, seed=7, charge_p={2: 0.7, 3: 0.3}, npeaks=(50, 100))
    sp.tol[:] = 1.0
    failed, want = [], {}

    def run(width):
        try:
            eng = hfx_gb300.Engine(0)
            eng.build_db(prot.seq, prot.seg, static_add=synth.static_mods(), **synth.DIGEST)
            p = hfx_gb300.default_params(top_n=5, batch_mode=mode, precision=0, search_mods=0, bin_width=width)
            first = eng.search(sp, p)
            start.wait(60)
            for _ in range(4000):
                assert np.array_equal(eng.search(sp, p).key, first.key)
            eng.close()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            failed.append(e)
            start.abort()

    start = threading.Barrier(2)
    ts = [threading.Thread(target=run, args=(w,)) for w in (1.0005079, 0.25)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed
