"""A context's eigen-solver workspace is allocated once, for its largest batch; smaller batches (the last of a k shard,
of the C3 representatives or of a group) run in it."""
import ctypes as C

import pytest


def _need(lib, n, iu, batch, mixed):
    out = (C.c_int64 * 5)()
    assert lib.forge_selftest_eig_workspace(C.c_int64(n), C.c_int64(iu), C.c_int64(batch), C.c_int(mixed), out) == 0
    return list(out)


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("n,iu", [(28, 24), (76, 48), (364, 192), (364, 364), (513, 256), (676, 348), (1324, 672),
                                  (1324, 1324), (5044, 2532), (11908, 5964)])
def test_workspace_serves_every_smaller_batch(lib, n, iu, mixed):
    last = 0
    for batch in range(1, 400):
        need, g, groom, w, wroom = _need(lib, n, iu, batch, mixed)
        assert need >= last, batch
        assert g <= groom and w <= wroom, batch
        last = need


@pytest.mark.parametrize("n", [3268, 5044, 11908])
def test_mixed_workspace_holds_nothing_of_the_fp64_path(lib, n):
    """All pairs of one matrix: Z, the factors and pivots (41 n^2 bytes), the FP32 matrix (8), two planes' pairs (16),
    and panels and partial products that fall off as 1 / n."""
    assert _need(lib, n, n, 1, 1)[0] <= (65 + 36000 / n) * n * n
