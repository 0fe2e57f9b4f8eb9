"""Model-checks the symmetric-memory schedules (KV slots, slabs, dK/dV accumulators, decode inbox)
over every interleaving the barriers allow, and checks that the checker notices broken variants."""
from pathlib import Path

import pytest

from ringattention_b200.parallel import protocol as P


@pytest.mark.parametrize("n", [2, 3])
def test_forward_schedule_is_race_free(n):
    progs = [P.ring_forward_program(r, n, calls=3) for r in range(n)]
    assert P.check_schedule(progs) is None


def test_forward_without_double_buffering_races():
    progs = [P.ring_forward_program(r, 2, calls=2, double_buffer=False) for r in range(2)]
    assert "stage" in (P.check_schedule(progs) or "")


def test_forward_without_barrier_races():
    progs = [P.ring_forward_program(r, 2, calls=1, barrier=False) for r in range(2)]
    assert P.check_schedule(progs) is not None


@pytest.mark.parametrize("n", [2, 3])
def test_backward_schedule_is_race_free(n):
    progs = [P.ring_backward_program(r, n, calls=2) for r in range(n)]
    assert P.check_schedule(progs) is None


def test_backward_needs_its_second_barrier():
    progs = [P.ring_backward_program(r, 2, calls=1, second_barrier=False) for r in range(2)]
    assert "cast" in (P.check_schedule(progs) or "") or "acc" in (P.check_schedule(progs) or "")


@pytest.mark.parametrize("n", [2, 3])
def test_decode_inbox_is_race_free(n):
    progs = [P.decode_program(r, n, calls=3) for r in range(n)]
    assert P.check_schedule(progs) is None


def test_decode_single_buffer_races():
    progs = [P.decode_program(r, 2, calls=2, double_buffer=False) for r in range(2)]
    assert P.check_schedule(progs) is not None


@pytest.mark.parametrize("n", [2, 3])
def test_fsdp_weight_gather_is_race_free(n):
    from ringattention_b200.parallel.protocol import check_schedule, fsdp_program

    assert check_schedule([fsdp_program(r, n, steps=2) for r in range(n)]) is None


def test_fsdp_needs_the_collectives_around_the_update():
    from ringattention_b200.parallel.protocol import check_schedule, fsdp_program

    # without the sync after the optimizer a peer's next step may read a shard that is being rewritten
    assert check_schedule([fsdp_program(r, 2, steps=2, sync_after_update=False) for r in range(2)]) is not None
    # without the gradient collective a rank may rewrite its shard while a slower peer still reads it
    assert check_schedule([fsdp_program(r, 2, steps=1, reduce_before_update=False) for r in range(2)]) is not None


@pytest.mark.parametrize("n,rows", [(2, 2), (3, 2), (2, 3)])
def test_row_exchange_with_two_slots_is_race_free(n, rows):
    assert P.check_row_exchange(n, rows, launches=4) is None


def test_row_exchange_with_one_slot_overwrites_unmerged_rows():
    assert "overwrites" in (P.check_row_exchange(2, 2, launches=2, slots=1) or "")


def _arrivals_after_exit(fills, stages, tail):
    """A CTA pair's `empty` ring as the CTA that does not issue sees it: the issuer's commits arrive at its barriers as late as they may, that
    is when a wait asks for them. Counts those that are still under way when the CTA leaves; the waits are the kernel's, by parity."""
    done, issued = [0] * stages, [0] * stages  # completed phases of each barrier; commits issued for it

    def wait(stage, parity):  # returns once the phase of that parity is complete: the current phase has the other one
        while done[stage] % 2 == parity:
            assert done[stage] < issued[stage], "waits for a commit that nobody issues"
            done[stage] += 1

    stage = phase = 0
    for f in range(fills + (stages if tail else 0)):
        wait(stage, phase ^ 1)
        if f < fills:
            issued[stage] += 1  # filled, multiplied, committed
        stage, phase = (0, phase ^ 1) if stage + 1 == stages else (stage + 1, phase)
    return sum(issued) - sum(done)


@pytest.mark.parametrize("stages", [6, 8])
def test_no_commit_reaches_a_cta_of_a_pair_that_has_left(stages):
    for fills in range(0, 4 * stages):
        assert _arrivals_after_exit(fills, stages, tail=True) == 0
        assert _arrivals_after_exit(fills, stages, tail=False) == min(fills, stages)
    src = (Path(__file__).parent.parent / "ringattention_b200/csrc/gemm_pair.cuh").read_text()
    assert "const int steps = more ? num_kb : STAGES;" in src  # the pass behind the last tile waits and fills nothing
