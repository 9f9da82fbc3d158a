"""The dense solve and inverse on matrices inside larger ones (lda > n), at the edges of the 64-wide
tiles, with the result written over the matrix, and from two threads on two streams. The
elimination pads a copy to whole tiles: nothing outside the n x n block is read or written. The
matrices are M M^T + n I (condition below 10), so both are within 1e-12 of numpy's."""
import ctypes as C
import importlib
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return importlib.import_module("torch")


def _spd(n):
    rng = np.random.default_rng(n)
    m = rng.normal(size=(n, n))
    return m @ m.T + n * np.eye(n), rng.normal(size=n)


def _inside(torch, a, lda):
    """a in the first columns of an n x lda device matrix of NaNs."""
    d = torch.full((a.shape[0], lda), float("nan"), dtype=torch.float64, device="cuda")
    d[:, :a.shape[0]] = torch.from_numpy(a).cuda()
    return d


def _p(t):
    return C.c_void_p(t.data_ptr())


def _solve(pkg, n, a, lda, b, x, stream=None):
    pkg.abi.check(pkg.abi.lib().gslam_gj_solve(n, _p(a), lda, _p(b), _p(x), stream, None))


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 129, 200])
@pytest.mark.parametrize("pad", [0, 1, 37])
def test_solve_and_inverse_with_a_leading_dimension(pkg, torch, n, pad):
    a, b = _spd(n)
    lda = n + pad
    da, db = _inside(torch, a, lda), torch.from_numpy(b).cuda()
    x = torch.full((n + 2,), float("nan"), dtype=torch.float64, device="cuda")
    _solve(pkg, n, da, lda, db, x[1:])
    got, ref = x.cpu().numpy(), np.linalg.solve(a, b)
    assert np.linalg.norm(got[1:-1] - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.isnan(got[0]) and np.isnan(got[-1])
    kept = da.cpu().numpy()
    assert np.array_equal(kept[:, :n], a) and np.isnan(kept[:, n:]).all()
    pkg.abi.check(pkg.abi.lib().gslam_gj_inverse(n, _p(da), lda, None, None))
    inv, ref = da.cpu().numpy(), np.linalg.inv(a)
    assert np.linalg.norm(inv[:, :n] - ref) <= 1e-12 * np.linalg.norm(ref)
    assert np.isnan(inv[:, n:]).all()


def test_result_over_the_matrix(pkg, torch):
    n = 100
    a, b = _spd(n)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    _solve(pkg, n, da, n, db, da[3])
    ref = np.linalg.solve(a, b)
    assert np.linalg.norm(da[3].cpu().numpy() - ref) <= 1e-12 * np.linalg.norm(ref)


def test_two_threads_on_two_streams(pkg, torch):
    sizes, out, failed = (190, 330), {}, []
    systems = {n: _spd(n) for n in sizes}

    def work(n):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                a, b = (torch.from_numpy(v).cuda() for v in systems[n])
                x = torch.empty_like(b)
                s.synchronize()
                for _ in range(10):
                    _solve(pkg, n, a, n, b, x, C.c_void_p(s.cuda_stream))
                    out.setdefault(n, []).append(x.cpu().numpy())
        except Exception as e:  # noqa: BLE001 (handed to the test's thread)
            failed.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for n in sizes:
        ref = np.linalg.solve(*systems[n])
        for x in out[n]:
            assert np.array_equal(x, out[n][0])
            assert np.linalg.norm(x - ref) <= 1e-12 * np.linalg.norm(ref)
