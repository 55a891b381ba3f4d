"""The engine of every transform length (pk_plan_read: from the extent alone, no device): its radices make up the length
and are ones that the engine's kernels have, and its tile fits shared memory."""
import ctypes as C
import json
import math

import pytest

from petakit5d_b200 import _lib

# radices with a register butterfly in the in-place engine, and those of the mixed-radix engine's stages
IN_PLACE = {2, 3, 4, 5, 8, 16}
MIXED = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16, 17, 19, 23, 29, 31}
MIXED_FIRST = {r for r in MIXED if r % 2}   # a first stage takes an odd radix


def plan(ny, nx, nz):
    buf = C.create_string_buffer(4096)
    n = _lib.lib.pk_plan_read(_lib.i64x3((ny, nx, nz)), buf, len(buf))
    assert n > 0, _lib.last_error()
    return json.loads(buf.value)


def largest_prime(n):
    p, f = 1, 2
    while n > 1:
        while n % f == 0:
            n, p = n // f, f
        f += 1
    return p


def check(axis, n, sums):
    assert axis["n"] == n
    r, e = axis["radices"], axis["engine"]
    assert math.prod(r) == n
    assert axis["lines"] >= 1
    assert axis["smem"] <= 227 * 1024
    if e == "mixed":
        assert not sums and largest_prime(n) <= 31
        assert set(r) <= MIXED and r[0] in MIXED_FIRST
    elif e == "sums":
        # four columns a thread; lengths with a register radix on tiles of at most 4096 points
        assert largest_prime(n) > 31 and n <= 2048 and axis["lines"] % 4 == 0
        if set(r) & IN_PLACE:
            assert axis["lines"] >= 8 and axis["lines"] * n <= 4096
    elif e == "plain":
        assert axis["lines"] * n <= 4096
    else:
        assert e == "plan"


def complex_len(ny):
    return ny if ny % 2 else ny // 2


def test_every_row_length():
    for ny in range(1, 8193):
        if ny % 2 and ny > 4096:
            continue
        n = complex_len(ny)
        axes = plan(ny, 64, 64)
        check(axes[0], n, axes[0]["engine"] in ("sums", "plain") and largest_prime(n) > 31)


def test_every_column_length():
    for n in range(1, 4097):
        axes = plan(64, n, 64)
        check(axes[1], n, largest_prime(n) > 31)
        assert plan(64, 64, n)[2] == axes[1]


# a prime factor above 31 beside a register radix, too long for eight lines of the sums' tile
@pytest.mark.parametrize("ny", [515, 519, 531, 543, 549, 555, 565, 573, 579, 999, 1028, 1030, 1036, 1110, 1332, 2220, 2452])
def test_long_rows_beside_a_register_radix(ny):
    assert plan(ny, 64, 64)[0]["engine"] == "plain"


def test_one_engine_for_a_volume():
    # a large prime on any axis keeps the sums on the others that have no plan
    assert [a["engine"] for a in plan(90, 40, 27)] == ["mixed", "mixed", "mixed"]
    assert [a["engine"] for a in plan(90, 40, 37)] == ["plain", "plain", "sums"]
    assert [a["engine"] for a in plan(74, 40, 27)] == ["sums", "plain", "plain"]
    assert [a["engine"] for a in plan(512, 37, 256)] == ["plan", "sums", "plan"]


def test_few_lines_beside_a_large_prime():
    # a tile's missing lines cost as much as others: fewer lines a tile where there are few, the plain engine (which has
    # tiles of what there is) where they are fewer still
    assert [plan(ny, 126, 233)[2]["engine"] for ny in (3, 400)] == ["plain", "sums"]
    assert plan(6, 467, 60)[1]["lines"] == 4 and plan(300, 467, 60)[1]["lines"] == 8
    assert plan(101, 1, 1)[0]["engine"] == "plain" and plan(101, 100, 1)[0]["engine"] == "sums"


def test_refused_extents():
    for dims in ((0, 1, 1), (1, 4097, 1), (8194, 1, 1), (4097, 1, 1)):
        assert _lib.lib.pk_plan_read(_lib.i64x3(dims), None, 0) < 0
