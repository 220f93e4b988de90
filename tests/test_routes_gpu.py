"""Float64 routes against one another at small sizes, with the few-pairs kernel off (SIGK_NO_PAIR_WAVE=1): it takes such
calls before the route under test.  A call's launches show which route ran: the few-pairs kernel is one launch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
RTOL64 = 1e-9


@pytest.fixture(scope="module")
def sig():
    import sigpde_b200.torch as s
    return s


@pytest.fixture(autouse=True)
def no_few_pairs_kernel(monkeypatch):
    monkeypatch.setenv("SIGK_NO_PAIR_WAVE", "1")


def cuda(a, dtype=torch.float64):
    return torch.tensor(np.asarray(a), dtype=dtype, device="cuda")


def launches(fn):
    from sigpde_b200 import _lib
    n = _lib.launch_count()
    out = fn()
    return out.double().cpu().numpy(), _lib.launch_count() - n


def check(calls, oracle_values, switch, monkeypatch, fewest):
    """Each call on its default route and with `switch`: bitwise the same, in at least `fewest` launches either way."""
    default = [launches(c) for c in calls]
    monkeypatch.setenv(switch, "1")
    other = [launches(c) for c in calls]
    monkeypatch.delenv(switch)
    for (a, na), (b, nb) in zip(default, other):
        assert na >= fewest[0] and nb >= fewest[1]
        np.testing.assert_array_equal(a, b)
    for (a, _), want in zip(default, oracle_values):
        np.testing.assert_allclose(a, want, rtol=RTOL64)


@pytest.mark.parametrize("nx,ny,lx,ly,d,order", [
    (5, 7, 40, 50, 3, 0), (3, 9, 33, 33, 1, 1), (6, 6, 100, 70, 8, 2), (3, 4, 40, 36, 4, 3), (2, 3, 20, 40, 2, 4),
    (2, 2, 10, 35, 2, 5), (7, 5, 128, 130, 8, 2), (3, 2, 60, 64, 5, 1), (2, 1, 60, 64, 5, 1), (4, 3, 40, 40, 32, 0),
    (5, 3, 300, 40, 2, 0), (3, 3, 513, 36, 1, 0), (61, 53, 20, 36, 3, 1)])
def test_two_entries_a_lane(sig, oracle, nx, ny, lx, ly, d, order, monkeypatch):
    """The two-entry Gram wavefront against one entry a lane: odd and even numbers of y paths, 16 coarse rows a lane."""
    x, y = oracle.brownian(nx, lx, d, 61 + order), oracle.brownian(ny, ly, d, 62 + order)
    X, Y = cuda(x), cuda(y)
    sx, sy = cuda(np.linspace(0.6, 1.4, nx)), cuda(np.linspace(1.2, 0.8, ny))
    k = sig.SigPDE(sig.kernels.LinearKernel(), order)
    calls = [lambda: k.gram(X, Y), lambda: k.gram(X, Y, sx, sy), lambda: k.gram(X.float(), Y.float())]
    check(calls, [oracle.gram(x, y, order)], "SIGK_NO_DUAL_F64", monkeypatch, (2, 2))


@pytest.mark.parametrize("nx,ny,length,d,order", [(9, 7, 40, 16, 1), (6, 11, 33, 24, 0), (5, 4, 70, 32, 2),
                                                  (13, 1, 20, 17, 3), (6, 6, 12, 16, 4), (5, 4, 300, 24, 1)])
@pytest.mark.parametrize("switch,fewest", [("SIGK_NO_DGEMM_PIPE", (3, 3)), ("SIGK_NO_DGEMM_INC", (3, 2))])
def test_wide_paths_matrix(sig, oracle, nx, ny, length, d, order, switch, fewest, monkeypatch):
    """The float64 increment matrix: from the pipelined GEMM against one tile a CTA, and against increments formed in the
    wavefront."""
    x, y = oracle.brownian(nx, length, d, 71 + d), oracle.brownian(ny, length + 5, d, 72 + d)
    X, Y, s = cuda(x), cuda(y), cuda(np.linspace(0.7, 1.3, nx))
    k = sig.SigPDE(sig.kernels.LinearKernel(1.3), order)
    calls = [lambda: k.gram(X), lambda: k.gram(X, None, s)]
    want = [oracle.gram(x * np.sqrt(1.3), None, order)]
    check(calls, want, switch, monkeypatch, fewest)
    a, na = launches(lambda: k.gram(X, Y))  # orders 2 and 3 may take the register kernel: no matrix there
    monkeypatch.setenv(switch, "1")
    b, _ = launches(lambda: k.gram(X, Y))
    assert na >= 2
    np.testing.assert_array_equal(a, b)
    np.testing.assert_allclose(a, oracle.gram(x * np.sqrt(1.3), y * np.sqrt(1.3), order), rtol=RTOL64)


@pytest.mark.parametrize("nx,lx,ly,d,order,chunk_mb", [
    (40, 200, 150, 8, 0, ""), (30, 150, 200, 13, 0, ""), (40, 120, 90, 12, 1, ""), (30, 140, 120, 15, 2, ""),
    (100, 70, 60, 12, 0, "64"), (97, 70, 60, 12, 0, "49"), (90, 140, 60, 9, 0, "190"), (83, 90, 70, 11, 1, "90"),
    (70, 200, 100, 12, 2, "720")])
def test_narrow_paths_matrix(sig, oracle, nx, lx, ly, d, order, chunk_mb, monkeypatch):
    """Below d = 16: the matrix in one chunk, and in several (equal ones, or a symmetric Gram's by its own columns),
    against the wavefront's own increments."""
    from sigpde_b200 import _lib
    x, y = oracle.brownian(nx, lx, d, 81 + d), oracle.brownian(nx + 3, ly, d, 82 + d)
    X, Y = cuda(x), cuda(y)
    k = sig.SigPDE(sig.kernels.LinearKernel(), order)
    if chunk_mb:
        monkeypatch.setenv("SIGK_TC_CHUNK_MB", chunk_mb)
    lib, calls = _lib.lib(), [lambda: k.gram(X, Y), lambda: k.gram(X)]
    matrix = [lib.sigk_workspace_size(*a) > lib.sigk_workspace_min_size(*a)
              for a in ((1, nx, nx + 3, lx, ly, d, order, 1, 0), (2, nx, nx, lx, lx, d, order, 1, 0))]
    assert any(matrix)
    got = [launches(c) for c in calls]
    if chunk_mb:  # differences, then a GEMM and a wavefront a chunk
        assert any(m and n >= 5 for m, (_, n) in zip(matrix, got))
    monkeypatch.setenv("SIGK_NO_DGEMM_INC", "1")
    want = [launches(c) for c in calls]
    for (a, _), (b, nb) in zip(got, want):
        assert nb == 2
        np.testing.assert_array_equal(a, b)
    np.testing.assert_allclose(got[0][0][:3, :4], oracle.gram(x[:3], y[:4], order), rtol=RTOL64)
