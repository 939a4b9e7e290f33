"""A case that moves to another context (mt_case_transfer) steps there as one
that never moved, alone and bit for bit, whether its old context still works or
is gone: no stream or event of that context is used any more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(which):
    from mortontrie_amr_b200.case import df_sphere_case, sphere_case
    if which == "df":
        return df_sphere_case(radius=3, max_level=1, re=60.0, oscillating=True, period=100)
    return sphere_case(coarse=(36, 20, 24), max_level=2, refine=[((7, 4, 5), (21, 17, 19)), ((17, 12, 13), (39, 31, 35))],
                       center=(14, 11, 12), radius=2.5, re=40.0)


def _state(mgr):
    return [a for l in range(mgr.L + 1) for a in mgr.populations(l) + mgr.macros(l)] + [mgr.force()]


@pytest.mark.parametrize("source", ["destroyed", "in use"])
@pytest.mark.parametrize("schedule", ["phases", "fused"])
@pytest.mark.parametrize("before", [0, 1])
@pytest.mark.parametrize("which", ["sphere", "df"])
def test_moved_case_steps_alone(source, schedule, before, which):
    """before: coarse steps taken on the old context."""
    from mortontrie_amr_b200.lbm import Context, LBM_Manager
    case = _case(which)
    old, new = Context(0), Context(0)
    mgr = LBM_Manager(old, case, "f64")
    mgr.prepare()
    mgr.fluidSimulate(before)
    mgr.transfer(new)
    if source == "destroyed":
        old.close()
    else:
        other = LBM_Manager(old, _case("sphere"), "f16", schedule="fused")
        other.fluidSimulate(2)
    mgr.set_schedule(schedule)
    mgr.fluidSimulate(3)
    if schedule == "phases":
        mgr.LBMkernel(0)
    still = LBM_Manager(new, case, "f64")
    still.prepare()
    still.fluidSimulate(before)
    still.set_schedule(schedule)
    still.fluidSimulate(3)
    if schedule == "phases":
        still.LBMkernel(0)
    for a, b in zip(_state(mgr), _state(still)):
        assert np.array_equal(a, b)
    new.close()
    old.close()
