"""Route and workspace of float64 Grams of narrow paths (d < 16), as sigk_workspace_size shows them: the increment
matrix is an option there, beside the fused kernels that need the path differences alone."""
import pytest

GRAM, SYM, F32, FP64 = 1, 2, 0, 0


@pytest.fixture(scope="module")
def lib():
    from sigpde_b200 import _lib
    return _lib.lib()


def sizes(lib, monkeypatch, op, nx, ny, lx, ly, d, order):
    """Workspace of the default route and of the fused one."""
    default = lib.sigk_workspace_size(op, nx, ny, lx, ly, d, order, F32, FP64)
    monkeypatch.setenv("SIGK_NO_DGEMM_INC", "1")
    fused = lib.sigk_workspace_size(op, nx, ny, lx, ly, d, order, F32, FP64)
    monkeypatch.delenv("SIGK_NO_DGEMM_INC")
    return default, fused


@pytest.mark.parametrize("op,nx,ny,lx,ly,d,order", [
    (SYM, 47, 47, 1786, 1786, 11, 1), (SYM, 25, 25, 2212, 2212, 9, 0), (SYM, 63, 63, 1307, 1307, 12, 0),
    (SYM, 34, 34, 1364, 1364, 9, 1), (SYM, 26, 26, 1099, 1099, 10, 0), (SYM, 128, 128, 500, 500, 9, 1),
    (GRAM, 110, 14, 1229, 1344, 10, 0), (GRAM, 20, 226, 1092, 1414, 10, 1), (GRAM, 11, 210, 895, 567, 14, 2),
    (GRAM, 64, 64, 1000, 1000, 8, 2), (GRAM, 16, 16, 2000, 2000, 8, 0)])
def test_no_matrix_in_chunks_of_few_pairs(lib, monkeypatch, op, nx, ny, lx, ly, d, order):
    """Long paths, whose matrix comes in chunks of a few pairs each: the fused kernels (1.1 to 6.4 times faster)."""
    default, fused = sizes(lib, monkeypatch, op, nx, ny, lx, ly, d, order)
    assert default == fused


@pytest.mark.parametrize("op,nx,ny,lx,ly,d,order", [
    (GRAM, 24, 12, 765, 580, 8, 0), (SYM, 24, 24, 537, 537, 8, 0), (SYM, 11, 11, 690, 690, 9, 0),
    (GRAM, 34, 34, 153, 173, 8, 2), (SYM, 81, 81, 128, 128, 8, 3), (GRAM, 40, 40, 150, 167, 8, 3),
    (SYM, 120, 120, 200, 200, 8, 2), (GRAM, 90, 90, 300, 317, 8, 2),
    (SYM, 266, 266, 442, 442, 6, 0), (GRAM, 93, 114, 377, 420, 5, 0), (GRAM, 38, 22, 371, 310, 3, 0),
    (GRAM, 37, 24, 554, 605, 8, 0), (GRAM, 27, 36, 625, 608, 8, 0), (SYM, 178, 178, 399, 399, 5, 0)])
def test_no_matrix_where_it_measured_slower(lib, monkeypatch, op, nx, ny, lx, ly, d, order):
    """Several bands with few pairs, few dimensions at orders 2 and 3, chunks that fill the device once at most."""
    default, fused = sizes(lib, monkeypatch, op, nx, ny, lx, ly, d, order)
    assert default == fused


@pytest.mark.parametrize("op,nx,ny,lx,ly,d,order", [
    (GRAM, 256, 256, 200, 200, 8, 0), (GRAM, 128, 128, 120, 120, 12, 1), (GRAM, 1000, 1000, 128, 128, 12, 1),
    (GRAM, 80, 80, 300, 300, 8, 1), (SYM, 300, 300, 200, 200, 10, 0), (GRAM, 100, 90, 180, 200, 9, 2),
    (SYM, 120, 120, 250, 250, 11, 3)])
def test_matrix_where_chunks_hold_enough_pairs(lib, monkeypatch, op, nx, ny, lx, ly, d, order):
    default, fused = sizes(lib, monkeypatch, op, nx, ny, lx, ly, d, order)
    assert default > fused


@pytest.mark.parametrize("op,nx,ny,lx,ly,d,order", [
    (GRAM, 256, 256, 200, 200, 8, 0), (GRAM, 1000, 1000, 128, 128, 12, 1), (SYM, 300, 300, 200, 200, 10, 0),
    (GRAM, 80, 80, 300, 300, 8, 1), (GRAM, 400, 333, 256, 200, 15, 1), (SYM, 2000, 2000, 60, 60, 15, 1),
    (GRAM, 64, 64, 1000, 1000, 8, 2)])
def test_matrix_stays_an_option_of_bounded_size(lib, monkeypatch, op, nx, ny, lx, ly, d, order):
    """At most 3 GiB beside the differences; the least workspace is the fused route's."""
    default, fused = sizes(lib, monkeypatch, op, nx, ny, lx, ly, d, order)
    assert default <= (3 << 30) + 2 * fused + 1024
    assert lib.sigk_workspace_min_size(op, nx, ny, lx, ly, d, order, F32, FP64) == fused


def test_least_workspace_of_other_calls_is_the_whole(lib):
    for op in (0, 1, 2, 3):
        for prec in (0, 1, 2, 3):
            for d in (0, 4, 16, 40):
                full = lib.sigk_workspace_size(op, 20, 20, 30, 30, d, 1, F32, prec)
                assert lib.sigk_workspace_min_size(op, 20, 20, 30, 30, d, 1, F32, prec) == full
