"""The solve kernel's rounds, launches and tiles, on the CPU: the library's own
rules (vsc_solver_plan with a given number of SMs asks no device)."""
import pytest

SMS = 152
INT_MAX = 2**31 - 1


@pytest.mark.parametrize("form", ["exact", "fma"])
@pytest.mark.parametrize("w,h", [(1, 1), (640, 360), (854, 480), (1920, 1080), (3840, 2160), (16384, 16384),
                                 (46340, 46340)])
@pytest.mark.parametrize("iters", [1, 150, 113_905, 13_800_000, INT_MAX])
def test_a_launchs_tickets_are_counted_in_32_bits(vsc, form, w, h, iters):
    """A launch numbers its tiles x rounds with a 32-bit counter that every CTA
    runs one past the end: whatever the call's steps, a launch holds far
    fewer, and its rounds add up to the solve's."""
    p = vsc.solver_plan(w, h, iters, form, sms=SMS)
    assert p.steps * (p.rounds - 1) < iters <= p.steps * p.rounds
    assert 1 <= p.rounds_per_launch <= p.rounds
    if p.planes:
        assert p.tiles * p.rounds_per_launch <= max(2**20, p.tiles) < 2**31 - 2 * SMS
    if iters == 150 and w <= 3840 and p.planes:
        assert p.rounds_per_launch == p.rounds  # ordinary solves are one launch


def test_plan_rejects_what_no_solve_takes(vsc):
    for args in [(0, 8, 1), (8, -1, 1), (8, 8, -1), (2**30, 2**30, 1)]:
        with pytest.raises(vsc.VscError):
            vsc.solver_plan(*args, sms=SMS)
    with pytest.raises(vsc.VscError):
        vsc.solver_plan(64, 64, 8, workspace_bytes=64 * 64 * 12 * 4 - 4, sms=SMS)
    assert vsc.solver_plan(64, 64, 0, sms=SMS).rounds == 0
