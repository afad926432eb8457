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


SIZES = [(1, 1), (5, 200), (64, 36), (240, 135), (426, 240), (427, 240), (640, 360), (720, 404), (800, 450), (854, 480),
         (856, 480), (960, 540), (1279, 719), (1920, 1080), (3840, 2160)]


def _fields(p):
    return [getattr(p, f) for f, _ in p._fields_]


@pytest.mark.parametrize("form", ["exact", "fma"])
@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("iters", [8, 20, 150])
def test_full_workspace_is_as_good_as_none(vsc, form, w, h, iters):
    """A workspace of the full size takes the path of the library's own."""
    full = vsc.consist_out_workspace_size(w, h, form, full=True)
    assert full >= vsc.consist_out_workspace_size(w, h, form)
    assert _fields(vsc.solver_plan(w, h, iters, form, full, SMS)) == _fields(vsc.solver_plan(w, h, iters, form, 0, SMS))


def test_full_workspace_size_of_no_image(vsc):
    assert vsc.consist_out_workspace_size(0, 10, full=True) == 0
    assert vsc.load().vsc_consist_out_full_workspace_size(8, 8, 2) == 0


@pytest.mark.parametrize("w,h,null_steps,small_steps", [(640, 360, 16, 12), (320, 180, 16, 12), (64, 36, 16, 16), (960, 540, 8, 8),
                                                        (856, 480, 12, 8)])
def test_a_smaller_workspace_gets_the_longest_rounds_it_has_counters_for(vsc, w, h, null_steps, small_steps):
    """FMA form, 150 steps: the documented workspace has counters for the 8-step
    tiles, rounded up to 64, which may be enough for 12-step or 16-step ones."""
    assert vsc.solver_plan(w, h, 150, "fma", 0, SMS).steps == null_steps
    p = vsc.solver_plan(w, h, 150, "fma", vsc.consist_out_workspace_size(w, h, "fma"), SMS)
    assert p.planes and p.steps == small_steps


@pytest.mark.parametrize("w,h,first_on_planes", [(960, 540, 1), (1280, 720, 4), (1600, 900, 1), (1760, 990, 7),
                                                 (1920, 1080, 7), (2560, 1440, 7), (1921, 1080, 1)])
def test_a_few_exact_steps_of_a_large_image_stay_on_interleaved_images(vsc, w, h, first_on_planes):
    """They do not pay for the planes (widths that are a multiple of 4: the
    interleaved kernels with plain loads are slower at any step count)."""
    assert [vsc.solver_plan(w, h, k, "exact", 0, SMS).planes for k in range(1, 12)] == [
        int(k >= first_on_planes) for k in range(1, 12)]
    assert all(vsc.solver_plan(w, h, k, "fma", 0, SMS).planes for k in range(1, 12))
