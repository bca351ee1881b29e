"""XCorr rows at the sizes where their builder changes course: lists of nonzero
bins that leave room for the window sums or not, rows whose ends and windows
cut the list, strides that take 16-byte stores or not.  Bit for bit against the
oracle; the BF16 and FP16 copies are the rounded FP32 row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _row(rng, length, npk):
    """A spectrum of about `npk` 1 Da bins whose row has about `length` bins."""
    top = length - 75
    bins = np.sort(rng.choice(np.arange(1, top), size=min(npk, top - 1), replace=False)) if npk else np.zeros(0, int)
    # edges of the row and of the windows, and the peak that sets the row's length
    edge = [b for b in (0, 74, 75, 76, 150, 151, 152, top - 2, top - 1) if 0 <= b < top and npk > 9]
    mz = np.unique(np.concatenate([bins, edge, [top]])).astype(np.float32)
    it = rng.lognormal(0.0, 2.0, size=len(mz)).astype(np.float32)
    it[rng.random(len(mz)) < 0.05] = 0.0
    return mz, it


def _with_infinity(oracle, mz, it, pcr, z, length):
    """One infinite intensity: its region's other bins become 0, its own (when
    the row normalises it) is no number and no part of a window's sum."""
    k = len(mz) // 2
    it = it.copy()
    sel = (length - 75) // 10
    region = np.minimum(10, mz.astype(int) // sel)
    without = np.where(region == region[k], 0.0, it).astype(np.float32)
    want = oracle.preprocess(mz, without, pcr, z, bw=1.0, custom_bw=True, remove_pcr=False)
    it[k] = np.inf
    return it, want, (int(mz[k]) if mz[k] < sel * 10 else -1)


@pytest.mark.parametrize("infinite", [0, 1])
@pytest.mark.parametrize("stride", [520, 1001, 2048, 4096])
def test_rows_at_their_edges(gpulib, oracle, stride, infinite):
    torch = pytest.importorskip("torch")
    import hfx_gb300
    rng = np.random.default_rng(stride)
    specs = []
    for length in (86, 95, 151, 152, 227, 256, 257, stride - 8, stride - 1, stride):
        # 2 / 7 of the stride is where the sums no longer fit beside the list
        for npk in (0, 1, 12, 2 * stride // 7 - 2, 2 * stride // 7 + 40, stride):
            specs.append(_row(rng, length, npk))
    pcr = np.array([(m[-1] + 500.0) / 2 for m, _ in specs], np.float32)
    z = np.full(len(specs), 2.0, np.float32)
    wants, nans = [], []
    for i, (m, it) in enumerate(specs):
        x = oracle.preprocess(m, it, pcr[i], z[i], bw=1.0, custom_bw=True, remove_pcr=False)
        nans.append(-1)
        if infinite and x is not None:
            it, x, nans[i] = _with_infinity(oracle, m, it, pcr[i], z[i], len(x))
            specs[i] = (m, it)
        wants.append(x)
    off = np.concatenate([[0], np.cumsum([len(m) for m, _ in specs])]).astype(np.int64)
    p = hfx_gb300.default_params(bin_width=1.0, custom_bin_width=1, remove_precursor_peak=0)
    eng = hfx_gb300.Engine(0)
    dev = {k: torch.from_numpy(v).cuda() for k, v in
           dict(mz=np.concatenate([m for m, _ in specs]), it=np.concatenate([i for _, i in specs]), off=off, pcr=pcr,
                z=z).items()}
    n = len(specs)
    rows = torch.full((n, stride), 7.0, device="cuda")
    rbf = torch.full((n, stride), 7.0, dtype=torch.bfloat16, device="cuda")
    rh = torch.full((n, stride), 7.0, dtype=torch.float16, device="cuda")
    eng.preprocess(dev, p, stride, rows, rbf, rh)
    torch.cuda.synchronize()
    for i, x in enumerate(wants):
        want = np.zeros(stride, np.float32)
        if x is not None and len(x) <= stride:
            want[:len(x)] = x
        got = rows[i].cpu().numpy()
        if nans[i] >= 0:
            assert np.isnan(got[nans[i]]), i
            got[nans[i]] = want[nans[i]]
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), i
        keep = ~rows[i].isnan()
        assert torch.equal(rbf[i][keep], rows[i][keep].bfloat16())
        assert torch.equal(rh[i][keep], rows[i][keep].half())
    eng.close()


@pytest.mark.parametrize("npk", [1, 2, 511, 512, 513, 1100])
def test_sparse_rows_by_peaks(gpulib, oracle, npk):
    """0.02 Da rows: the forms for up to 512 peaks and for more, peaks alone, in
    crowds (many to a window) and at the row's ends."""
    torch = pytest.importorskip("torch")
    import hfx_gb300
    rng = np.random.default_rng(npk)
    mz = np.sort(np.concatenate([rng.uniform(0.0, 1400.0, npk - npk // 2 - 1), rng.uniform(700.0, 706.0, npk // 2),
                                 [1400.0]]))[:npk].astype(np.float32)
    it = rng.lognormal(0.0, 2.0, size=npk).astype(np.float32)
    pcr, z = np.array([900.0], np.float32), np.array([2.0], np.float32)
    x = oracle.preprocess(mz, it, pcr[0], z[0], bw=0.02, custom_bw=True, remove_pcr=False)
    stride = 16 * ((len(x) + 15) // 16 if x is not None else 1)
    stride = max(stride, 16 * 4000)
    dev = dict(mz=mz, it=it, off=np.array([0, npk], np.int64), pcr=pcr, z=z)
    dev = {k: torch.from_numpy(v).cuda() for k, v in dev.items()}
    eng = hfx_gb300.Engine(0)
    rows = torch.full((1, stride), 7.0, device="cuda")
    rbf = torch.full((1, stride), 7.0, dtype=torch.bfloat16, device="cuda")
    eng.preprocess(dev, hfx_gb300.default_params(bin_width=0.02, custom_bin_width=1, remove_precursor_peak=0), stride,
                   rows, rbf)
    torch.cuda.synchronize()
    want = np.zeros(stride, np.float32)
    if x is not None:
        want[:len(x)] = x
    assert np.array_equal(rows[0].cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert torch.equal(rbf[0], rows[0].bfloat16())
    eng.close()
