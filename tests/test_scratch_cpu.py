"""What a call allocates when the device is nearly full (scratch.h): the rows of
wide roots take what is left beside the buffers that a search needs, and are
given back where those do not fit."""
import itertools

import pytest

import emulate

GIB = 1 << 30
LIMIT, RESERVE = 32 * GIB, GIB


def numbers(*args):
    rc, out, err = emulate.run("scratch", *args)
    assert rc == 0, err
    return [int(x) for x in out.split()]


SIZES = (0, 64 << 20, 3 * GIB, 33 * GIB)


@pytest.mark.parametrize("want,held,others", list(itertools.product(SIZES[1:], SIZES[:3], SIZES)))
def test_rows_take_what_is_left(want, held, others):
    for free, needed in itertools.product((0, 512 << 20, 4 * GIB, 150 * GIB), (0, 2 * GIB)):
        got, = numbers("grant", want, held, others, free, needed)
        assert got >= held
        if got > held:  # it grows: within the bound of the handle, beside what is needed
            assert got <= want and got + others <= LIMIT
            assert got + needed + RESERVE <= free + held
        if others == 0 and held <= want <= LIMIT and want + needed + RESERVE <= free + held:
            assert got == want


@pytest.mark.parametrize("limit,held,needs,expect", [
    (1000, 0, (400, 500), (0, 1, 0, 900)),      # it fits
    (1000, 200, (400, 300), (0, 1, 200, 700)),  # beside the rows too
    (1000, 200, (400, 500), (0, 2, 0, 900)),    # only without them
    (1000, 900, (400,), (0, 2, 0, 400)),
    (1000, 0, (400, 700), (12, 1, 0, 400)),     # never
    (1000, 200, (400, 700), (12, 2, 0, 400)),
])
def test_rows_go_before_a_call_fails(limit, held, needs, expect):
    assert tuple(numbers("run", limit, held, *needs)) == expect
