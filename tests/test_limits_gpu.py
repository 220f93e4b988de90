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
