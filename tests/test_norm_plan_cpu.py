"""Workspace of the robust normalisation (sigk_workspace_size): paths of any length are accepted, and beyond the tiles of
resident CTAs (1 GiB together) nothing grows with the square of the length."""
import pytest

NORMALIZE, F32, FP64 = 3, 0, 0


@pytest.mark.parametrize("n,L,d,order", [(16, 100000, 2, 0), (1, 20000, 3, 0), (16, 50000, 2, 3), (4, 15000, 8, 1),
                                         (512, 4000, 3, 0), (1000, 3000, 4, 0), (64, 2500, 3, 1), (24, 1100, 3, 2)])
@pytest.mark.parametrize("given", [False, True])
def test_workspace_of_long_paths(n, L, d, order, given):
    from sigpde_b200 import _lib
    got = _lib.lib().sigk_workspace_size(NORMALIZE, n, n, L, L, 0 if given else d, order, F32, FP64)
    differences = 0 if given else n * (L - 1) * d * 8
    rows = 8 * 4 * 148 * (((L - 1) << order) + 64) * 8  # one boundary row a resident warp, on the largest device
    assert got <= max(1 << 30, rows) + rows + differences + (1 << 20)
    if (L - 1) ** 2 * 8 > 1 << 30:
        assert got <= rows + differences + (1 << 20)
