"""matchms ParentMassMatch / PrecursorMzMatch / IntersectMz on the device
(csrc/metadata_match.cu) against the oracle restatement
(oracle/matchms_other_restated.py): bit-exact."""
import numpy as np
import pytest

from conftest import Spectrum
from oracle import matchms_other_restated as other

pytestmark = pytest.mark.gpu


def _dev():
    import torch

    return torch.device("cuda", torch.cuda.current_device())


def _masses(n, rng):
    v = rng.uniform(100.0, 1000.0, n)
    v[::7] = np.round(v[::7], 1)  # repeated and near-equal values
    return v


@pytest.mark.parametrize("n_q", [512, 517])  # 512: 16-byte row stores; 517: per-byte
@pytest.mark.parametrize("ppm", [False, True])
def test_mass_match_kernel(cuda_device, n_q, ppm):
    import torch

    from cudams import kernels

    rng = np.random.default_rng(n_q + ppm)
    r = _masses(300, rng)
    q = _masses(n_q, rng)
    tol = 20.0 if ppm else 0.125
    # pairs exactly at the tolerance and one float64 step beyond it
    q[0], q[1] = r[0] + 0.125, np.nextafter(r[0] + 0.125, np.inf)
    q[2] = r[1] * (1 + 2e-5)
    r[5] = np.nan
    got = kernels.mass_match_matrix(torch.from_numpy(r).to(_dev()),
                                    torch.from_numpy(q).to(_dev()), tol, ppm).cpu().numpy()
    want = other.mass_match(r, q, tol, ppm)
    np.testing.assert_array_equal(got.astype(bool), want)
    assert set(np.unique(got)) <= {0, 1}
    assert want.any() and not want.all()


def _spectra_mz(n, rng, pool):
    out = []
    for i in range(n):
        k = int(rng.integers(0, 60))
        mz = np.sort(rng.choice(pool, size=k, replace=True))  # repeats on purpose
        out.append(mz)
    out[3] = np.zeros(0)
    out[4] = np.sort(rng.choice(pool, size=5000, replace=True))  # past the shared-memory stage
    return out


def _csr(lists):
    import torch

    off = np.zeros(len(lists) + 1, dtype=np.int64)
    off[1:] = np.cumsum([len(a) for a in lists])
    mz = np.concatenate(lists) if lists else np.zeros(0)
    return (torch.from_numpy(mz.astype(np.float64)).to(_dev()),
            torch.from_numpy(off).to(_dev()))


@pytest.mark.parametrize("scaling", [1.0, 0.3])
def test_intersect_mz_kernel(cuda_device, scaling):
    from cudams import kernels

    rng = np.random.default_rng(7)
    pool = rng.uniform(50.0, 500.0, 400)
    a = _spectra_mz(70, rng, pool)
    b = _spectra_mz(300, rng, pool)
    got = kernels.intersect_mz_matrix(*_csr(a), *_csr(b), scaling,
                                      check_errors=True).cpu().numpy()
    want = other.intersect_mz(a, b, scaling)
    np.testing.assert_array_equal(got.view(np.uint64), want.view(np.uint64))
    assert (want > 0).any() and (want == 0).any()


def test_intersect_mz_bad_offsets(cuda_device):
    import torch

    from cudams import _native, kernels

    mz = torch.arange(10, dtype=torch.float64, device=_dev())
    bad = torch.tensor([0, 6, 3], dtype=torch.int64, device=_dev())  # decreasing
    good = torch.tensor([0, 4], dtype=torch.int64, device=_dev())
    with pytest.raises(_native.NativeError, match="offsets"):
        kernels.intersect_mz_matrix(mz, bad, mz, good, check_errors=True)


def _spectra(n, rng):
    pool = rng.uniform(50.0, 500.0, 200)
    out = []
    for i in range(n):
        mz = np.sort(rng.choice(pool, size=int(rng.integers(1, 30)), replace=False))
        out.append(Spectrum(mz, np.ones_like(mz),
                            {"precursor_mz": float(rng.uniform(300, 310)),
                             "parent_mass": float(np.round(rng.uniform(299, 301), 2))}))
    return out


def test_classes(cuda_device):
    from cudams.similarity import CudaIntersectMz, CudaParentMassMatch, CudaPrecursorMzMatch

    rng = np.random.default_rng(3)
    refs, qrys = _spectra(40, rng), _spectra(57, rng)
    pm = [s.get("parent_mass") for s in refs], [s.get("parent_mass") for s in qrys]
    pz = [s.get("precursor_mz") for s in refs], [s.get("precursor_mz") for s in qrys]
    mzs = [s.peaks.mz for s in refs], [s.peaks.mz for s in qrys]

    got = CudaParentMassMatch(0.5).matrix(refs, qrys)
    assert got.dtype == bool
    np.testing.assert_array_equal(got, other.mass_match(*pm, 0.5))
    np.testing.assert_array_equal(CudaPrecursorMzMatch(2.0).matrix(refs, qrys),
                                  other.mass_match(*pz, 2.0))
    np.testing.assert_array_equal(CudaPrecursorMzMatch(5000.0, "ppm").matrix(refs, qrys),
                                  other.mass_match(*pz, 5000.0, ppm=True))
    ix = CudaIntersectMz(0.5).matrix(refs, qrys)
    np.testing.assert_array_equal(ix.view(np.uint64),
                                  other.intersect_mz(*mzs, 0.5).view(np.uint64))
    assert CudaIntersectMz().pair(refs[0], refs[0]) == 1.0
    assert CudaParentMassMatch(0.0).pair(refs[1], refs[1]) is True

    # sparse output holds exactly the nonzero scores; symmetric equals full
    sp = CudaParentMassMatch(0.5).matrix(refs, qrys, array_type="sparse")
    np.testing.assert_array_equal(sp.to_array().astype(bool), other.mass_match(*pm, 0.5))
    sym = CudaIntersectMz().matrix(refs, refs, is_symmetric=True)
    np.testing.assert_array_equal(sym, sym.T)
    np.testing.assert_array_equal(sym, other.intersect_mz(mzs[0], mzs[0]))


@pytest.mark.parametrize("n_q", [31, 511, 512, 513, 1040, 2051])
@pytest.mark.parametrize("ppm,tol", [(False, 0.1), (False, 0.0), (False, 300.0), (False, 1e301),
                                     (True, 10.0), (True, 0.0), (True, 4e5), (True, 3e6)])
def test_mass_match_bounds(cuda_device, n_q, ppm, tol):
    """Row bounds against the definition: values at the tolerance and a few float64
    steps around it, negative, zero, infinite, NaN and extreme values, at the edges of
    a warp's 512 columns, rows of every alignment."""
    import torch

    from cudams import kernels

    rng = np.random.default_rng(n_q)
    r = rng.uniform(100.0, 1000.0, 67)
    r[3:12] = [np.nan, np.inf, -np.inf, 0.0, -250.0, 1e-300, 1e200, 1e301, -1e301]
    q = rng.uniform(50.0, 1200.0, n_q)
    at = rng.integers(12, 67, n_q)
    with np.errstate(all="ignore"):
        edge = r[at] * ((1 + 0.5e-6 * tol) / (1 - 0.5e-6 * tol)) if ppm else r[at] + tol
    step = rng.integers(-3, 4, n_q)
    for _ in range(3):
        edge = np.where(step > 0, np.nextafter(edge, np.inf),
                        np.where(step < 0, np.nextafter(edge, -np.inf), edge))
        step -= np.sign(step)
    q = np.where(rng.random(n_q) < 0.5, edge, q)
    q[5:16] = [np.nan, np.inf, -np.inf, 0.0, -400.0, -1e-3, 1e-300, 1e200, 1e301, -1e301, r[20]]
    got = kernels.mass_match_matrix(torch.from_numpy(r).to(_dev()),
                                    torch.from_numpy(q).to(_dev()), tol, ppm).cpu().numpy()
    with np.errstate(all="ignore"):  # the oracle's expressions on whole rows (0 / 0 is NaN)
        d = np.abs(r[:, None] - q[None, :])
        mean = (r[:, None] + q[None, :]) / 2
        want = d / mean * 1e6 <= tol if ppm else d <= tol
    np.testing.assert_array_equal(got.astype(bool), want)


@pytest.mark.parametrize("scaling", [1.0, -2.5])
@pytest.mark.parametrize("n_q", [1, 2047, 2049, 9216, 9217])
def test_intersect_mz_tiles(cuda_device, n_q, scaling):
    """Query tile edges, a value that every query has, references of more values than
    a CTA has threads, empty spectra on both sides, rows of both alignments."""
    from cudams import kernels

    rng = np.random.default_rng(n_q)
    pool = np.concatenate([[100.25], rng.uniform(101.0, 500.0, 3000)])
    b = [np.sort(np.concatenate([[100.25], rng.choice(pool, size=int(rng.integers(0, 6)))]))
         for _ in range(n_q)]
    if n_q > 3:
        b[n_q - 2] = np.zeros(0)
    a = [np.sort(rng.choice(pool, size=k, replace=False)) for k in (1, 40, 511, 513, 1100)]
    a += [np.zeros(0), np.array([100.25]), np.array([100.25, 100.25, 900.0])]
    got = kernels.intersect_mz_matrix(*_csr(a), *_csr(b), scaling,
                                      check_errors=True).cpu().numpy()
    want = other.intersect_mz(a, b, scaling)
    np.testing.assert_array_equal(got.view(np.uint64), want.view(np.uint64))


def test_mass_match_medium_cost(cuda_device):
    """A result of 64 MB takes at most 1.6 times a plain fill of it: a warp's columns
    are loaded for enough rows."""
    import torch

    from cudams import kernels

    rng = np.random.default_rng(61)
    r, q = (torch.from_numpy(rng.uniform(100.0, 1000.0, n)).to(_dev()) for n in (8000, 8192))
    out = torch.empty((8000, 8192), dtype=torch.uint8, device=_dev())

    def ms(f):
        best = float("inf")
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(8):
                f()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    fill = ms(lambda: out.fill_(1))
    assert ms(lambda: kernels.mass_match_matrix(r, q, 0.1, out=out)) < 1.6 * fill


@pytest.mark.parametrize("entry", ["python", "c"])
def test_intersect_mz_workspace_is_given_back(cuda_device, entry):
    """Nothing of a call's index (80 MB here) stays outside torch's allocator."""
    import torch

    from cudams import _native, kernels
    from cudams._native import ptr, stream_handle

    rng = np.random.default_rng(71)
    a = _csr([np.sort(rng.uniform(50.0, 900.0, 40)) for _ in range(3)])
    off = torch.arange(0, 3_000_001, 3000, dtype=torch.int64, device=_dev())
    mz = torch.from_numpy(np.sort(rng.uniform(50.0, 900.0, (1000, 3000)), axis=1).ravel()).to(_dev())
    out = torch.empty((3, 1000), dtype=torch.float64, device=_dev())

    def call(q_mz, q_off):
        if entry == "python":
            kernels.intersect_mz_matrix(*a, q_mz, q_off, out=out[:, :q_off.shape[0] - 1])
            return
        s = torch.cuda.current_stream(_dev())
        rc = _native.load().cms_intersect_mz(
            ptr(a[0]), ptr(a[1]), 3, a[0].shape[0], ptr(q_mz), ptr(q_off), q_off.shape[0] - 1,
            q_mz.shape[0], 1.0, ptr(out), 1000, ptr(None), stream_handle(s))
        assert rc == _native.CMS_OK, _native.last_error()

    call(mz[:3000], off[:2])  # the module is loaded
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info(_dev())[0]
    call(mz, off)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert before - torch.cuda.mem_get_info(_dev())[0] < 16 << 20


def test_intersect_mz_streams_and_capture(cuda_device):
    """Calls on a stream of their own, overlapping on two, and captured in a graph."""
    import torch

    from cudams import kernels

    rng = np.random.default_rng(72)
    pool = np.round(rng.uniform(50.0, 900.0, 4000), 2)
    sets = [[np.unique(rng.choice(pool, 60)) for _ in range(n)] for n in (300, 290, 310)]
    r, q1, q2 = (_csr(s) for s in sets)
    want = [other.intersect_mz(sets[0], s).view(np.uint64) for s in sets[1:]]
    streams = [torch.cuda.Stream(_dev()) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(3):
        got = [kernels.intersect_mz_matrix(*r, *q, stream=s, out=torch.empty(
            (300, q[1].shape[0] - 1), dtype=torch.float64, device=_dev()))
            for q, s in zip((q1, q2), streams)]
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g.cpu().numpy().view(np.uint64), w)
    out = torch.zeros((300, 290), dtype=torch.float64, device=_dev())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kernels.intersect_mz_matrix(*r, *q1, out=out)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want[0])


def test_mass_match_wide_tolerance_cost(cuda_device):
    """A ppm tolerance past the float32 bounds costs a division a pair, at most twice
    what the widest tolerance inside them takes."""
    import torch

    from cudams import kernels

    rng = np.random.default_rng(62)
    r, q = (torch.from_numpy(rng.uniform(100.0, 1000.0, n)).to(_dev()) for n in (8000, 8192))
    out = torch.empty((8000, 8192), dtype=torch.uint8, device=_dev())

    def ms(tolerance):
        best = float("inf")
        for _ in range(6):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            kernels.mass_match_matrix(r, q, tolerance, True, out=out)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert ms(6e5) < 2 * ms(4e5)


@pytest.mark.parametrize("tol", [5e5, np.nextafter(5e5, 1e6), 1.9e6, 2e6, 2.1e6, -1.0, np.inf])
@pytest.mark.parametrize("n_q", [512, 777])
def test_mass_match_outside_the_bounds(cuda_device, n_q, tol):
    import torch

    from cudams import kernels

    rng = np.random.default_rng(63)
    r, q = rng.uniform(-100.0, 1000.0, 70), rng.uniform(-100.0, 1000.0, n_q)
    q[:3] = [np.nan, np.inf, 0.0]
    got = kernels.mass_match_matrix(torch.from_numpy(r).to(_dev()),
                                    torch.from_numpy(q).to(_dev()), tol, True).cpu().numpy()
    with np.errstate(all="ignore"):
        want = (np.abs(r[:, None] - q[None, :]) / ((r[:, None] + q[None, :]) / 2) * 1e6) <= tol
    np.testing.assert_array_equal(got.astype(bool), want)
