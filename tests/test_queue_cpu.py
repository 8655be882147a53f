"""The task ring (queue.cuh) on the CPU: what it hands out when nobody takes,
over many laps, and the waits that must end."""
import emulate


def ring(mode):
    rc, out, err = emulate.run("queue", mode, timeout=60)
    assert rc == 0, err
    return [int(x) for x in out.split()]


def test_a_full_ring_refuses_before_it_hands_out_a_position():
    accepted, positions = ring("full")
    assert accepted == positions
    assert 32 <= accepted < 64  # less than a lap ahead of the takers


def test_many_laps():
    pushed, taken, err = ring("laps")
    assert err == 0
    # two donors' tasks, three words each: x, x + 1, x + 2
    assert pushed == 2000 and taken == sum(3 * (3 * i) + 3 for i in range(2000))


def test_a_taker_leaves_a_slot_that_is_never_given_back():
    assert ring("stale") == [0]


def test_a_donor_s_wait_for_its_slot_is_bounded_and_reported():
    assert ring("held") == [0, 1]
