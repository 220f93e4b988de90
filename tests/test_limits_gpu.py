"""Calls at the limits of the number range, of memory and of path length, on a GPU."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sig():
    import sigpde_b200.torch as s
    return s


def cuda(a, dtype=torch.float64):
    return torch.tensor(np.asarray(a), dtype=dtype, device="cuda")


def host(t):
    return t.double().cpu().numpy()


@pytest.mark.parametrize("lx,ly", [(2, 2), (2, 5), (3, 2), (40, 37), (70, 34)])
@pytest.mark.parametrize("order", [0, 1, 3])
@pytest.mark.parametrize("where", ["overflow", "last", "first", "nan"])
def test_few_pairs_infinite_increments(sig, oracle, lx, ly, order, where, monkeypatch):
    """Increments that overflow, or that an infinite or NaN point makes, give the general kernels' values
    (a single infinite cell stays infinite)."""
    x, y = oracle.brownian(3, lx, 1, 5 + lx), oracle.brownian(3, ly, 1, 6 + ly)
    if where == "overflow":
        x, y = x * 1e200, y * 1e200
    else:
        x[1, 0 if where == "first" else -1, 0] = np.nan if where == "nan" else np.inf
    X, Y = cuda(x), cuda(y)
    k = sig.SigPDE(sig.kernels.LinearKernel(), order)
    got = [host(v) for v in (k.gram(X, Y), k.gram(X), k.pairwise(X, Y))]
    monkeypatch.setenv("SIGK_NO_PAIR_WAVE", "1")
    want = [host(v) for v in (k.gram(X, Y), k.gram(X), k.pairwise(X, Y))]
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    if (lx, ly, order, where) == (2, 2, 0, "overflow"):
        assert np.isinf(want[0]).any()


def _narrow(oracle):
    """A Gram whose increment matrix takes over 1 GiB and whose differences take a few MB."""
    x, y = oracle.brownian(256, 200, 8, 11), oracle.brownian(200, 200, 8, 12)
    return cuda(x, torch.float32), cuda(y, torch.float32)


def test_narrow_gram_runs_in_the_memory_that_is_left(sig, oracle):
    """A process limited to less than the matrix: the fused kernels, with the same values."""
    X, Y = _narrow(oracle)
    k = sig.SigPDE(sig.kernels.LinearKernel(), 0)
    want = [k.gram(X, Y), k.gram(X)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (256 << 20)) / total)
        torch.cuda.reset_peak_memory_stats()
        got = [k.gram(X, Y), k.gram(X)]
        torch.cuda.synchronize()
        assert torch.cuda.max_memory_allocated() < 512 << 20
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("budget_mb", [64, 16384])
def test_server_admits_narrow_grams_with_their_least_workspace(sig, oracle, budget_mb):
    """Requests whose matrix exceeds the server's budget run, together, with the fused kernels."""
    from sigpde_b200 import serving
    X, Y = _narrow(oracle)
    want = host(sig.SigPDE(sig.kernels.LinearKernel(), 0).gram(X, Y))
    req = serving.GramRequest(x=X.cpu(), y=Y.cpu(), order=0)
    least = serving.footprint_bytes(req, lean=True)
    assert least < 32 << 20 < 1 << 30 < serving.footprint_bytes(req)
    server = serving.GramServer(hbm_budget_bytes=budget_mb << 20, max_inflight=4)
    with server:
        handles = [server.submit(serving.GramRequest(x=X.cpu(), y=Y.cpu(), order=0)) for _ in range(4)]
        for h in handles:
            np.testing.assert_array_equal(h.wait(60).double().numpy(), want)
    assert server.peak_bytes <= budget_mb << 20
    if budget_mb == 64:
        assert server.peak_inflight >= 2


@pytest.mark.parametrize("op,dim", [("gram", 8), ("gram", 12), ("sym", 8)])
def test_narrow_grams_take_a_16_byte_aligned_workspace(sig, oracle, op, dim, monkeypatch):
    """The C entry points accept 16-byte alignment wherever the fused kernels serve, whatever the size given."""
    from sigpde_b200 import _lib
    monkeypatch.setenv("SIGK_NO_PAIR_WAVE", "1")
    lib, n, L = _lib.lib(), 40, 200
    X = cuda(oracle.brownian(n, L, dim, 21), torch.float32)
    stream = torch.cuda.current_stream().cuda_stream
    outs = []
    for shift in (0, 16, 128):
        size = lib.sigk_workspace_size(2 if op == "sym" else 1, n, n, L, L, dim, 0, 0, 0)
        assert size > lib.sigk_workspace_min_size(2 if op == "sym" else 1, n, n, L, L, dim, 0, 0, 0)
        ws = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
        out = torch.full((n, n), float("nan"), device="cuda")
        if op == "sym":
            st = lib.sigk_gram_sym(X.data_ptr(), n, L, dim, 0, 0, 1.0, None, out.data_ptr(), 0, ws.data_ptr() + shift,
                                   size, stream)
        else:
            st = lib.sigk_gram(X.data_ptr(), X.data_ptr(), n, n, L, L, dim, 0, 0, 1.0, None, None, out.data_ptr(), 0,
                               ws.data_ptr() + shift, size, stream)
        assert st == 0, _lib.last_error()
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("n,L,d,order", [(5, 10, 3, 0), (3, 33, 4, 1), (4, 79, 5, 1), (3, 80, 5, 1), (3, 130, 2, 0),
                                         (2, 66, 40, 2), (2, 70, 2, 4), (3, 40, 130, 1), (2, 40, 3, 6), (2, 301, 4, 3)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("given", [False, True])
def test_normalization_one_path_a_warp(sig, oracle, n, L, d, order, dtype, given, monkeypatch):
    """A path a warp (SIGK_NORM_WARP=1) and a path a CTA (0): the same scales bit for bit, from a tile in shared memory,
    from the differences and from the caller's increments, at the edges of bands and of the staged dimensions."""
    class Increments:  # the linear kernel as a static kernel the device does not know
        def pairwise(self, x, y):
            return x @ y.transpose(1, 2)

    x = oracle.brownian(n, L, d, 31 + L, scale=np.linspace(0.8, 3.0, n) / np.sqrt(d))
    X = cuda(x, dtype)
    rk = sig.RobustSigPDE(Increments() if given else sig.kernels.LinearKernel(), order)
    got = []
    for route in ("1", "0"):
        monkeypatch.setenv("SIGK_NORM_WARP", route)
        got.append(host(rk.normalization(X)))
    np.testing.assert_array_equal(got[0], got[1])
    tol = dict(rtol=1e-6, atol=1e-9) if dtype == torch.float64 and not given else dict(rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(got[0], oracle.normalization(host(X), order), **tol)


@pytest.mark.parametrize("n,L,d,order", [(8, 1100, 3, 2), (8, 260, 2, 4), (17, 2061, 2, 0), (150, 1500, 2, 0),
                                         (2600, 20, 3, 1)])
def test_normalization_of_long_paths_and_many(sig, oracle, n, L, d, order, monkeypatch):
    """Thousands of points, more bands than warps a CTA, more tiles than the workspace holds, many short paths: the
    default route within the oracle's bound, and the other one the same."""
    x = oracle.brownian(n, L, d, 41 + L, scale=np.linspace(0.8, 2.5, n))
    X = cuda(x)
    rk = sig.RobustSigPDE(sig.kernels.LinearKernel(), order)
    lam = host(rk.normalization(X))
    idx = np.unique(np.linspace(0, n - 1, 3).astype(int))
    np.testing.assert_allclose(lam[idx], oracle.normalization(x[idx], order), rtol=1e-6, atol=1e-9)
    for route in ("1", "0"):
        monkeypatch.setenv("SIGK_NORM_WARP", route)
        np.testing.assert_array_equal(host(rk.normalization(X)), lam)


@pytest.mark.parametrize("op", ["pairwise", "gram"])
def test_gradient_with_a_graph_reaches_the_scales(sig, oracle, op, monkeypatch):
    """create_graph on a static kernel's gradient: what depends on the scales outside the solver keeps its graph, as
    with torch's own second difference."""
    from sigpde_b200.torch import kernel
    x, y = oracle.brownian(4, 12, 3, 51), oracle.brownian(4, 10, 3, 52)
    k = sig.SigPDE(sig.kernels.RBFKernel(1.0), 1)

    def second():
        X, Y = cuda(x).requires_grad_(), cuda(y).requires_grad_()
        s = cuda(np.linspace(0.7, 1.3, 4)).requires_grad_()
        v = k.pairwise(X, Y, s, s) if op == "pairwise" else k.gram(X, Y, s, s)
        gx, gy = torch.autograd.grad(v.sum(), (X, Y), create_graph=True)
        return torch.autograd.grad((gx ** 2).sum() + (gy ** 2).sum(), (s, X, Y))

    got = second()
    monkeypatch.setattr(kernel, "_takes_second_diff", lambda G, dim: False)
    for a, b in zip(got, second()):
        np.testing.assert_allclose(host(a), host(b), rtol=1e-9, atol=1e-12)
