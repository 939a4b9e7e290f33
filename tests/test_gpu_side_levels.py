"""A level's own work beside its finer levels' substeps, one explosion for
both substeps, and the launches that the phase order merges, where the order
matters: interface options changed on the way, and sets that overlap."""
import numpy as np
import pytest
from helpers import TAG_BC

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from mortontrie_amr_b200.lbm import Context
    c = Context(0)
    yield c
    c.close()


def _sphere(levels=2):
    from mortontrie_amr_b200.case import sphere_case
    return sphere_case(coarse=(36, 20, 24), max_level=levels, refine=[((7, 4, 5), (21, 17, 19)),
                                                                      ((17, 12, 13), (39, 31, 35))][:levels],
                       center=(14, 11, 12), radius=2.5, re=40.0)


def _oracle_equal(mgr, oc, levels):
    for l in levels:
        f, fcol = mgr.populations(l)
        g = oc.get(l)
        keep = (g["tags"] & TAG_BC) == 0
        assert np.array_equal(f[:, keep], g["f"][:, keep]), l
        assert np.array_equal(fcol, g["fcol"]), l


@pytest.mark.parametrize("schedule", ["phases", "fused"])
@pytest.mark.parametrize("order", [("reference", "hold", "reference"), ("hold", "extrap", "hold")])
def test_interface_option_changed_between_steps(ctx, schedule, order):
    """FP64, bit for bit against the oracle taking the same options."""
    import oracle as O
    from mortontrie_amr_b200.lbm import LBM_Manager
    case = _sphere()
    mgr = LBM_Manager(ctx, case, schedule=schedule, interface_time=order[0])
    oc = O.OracleCase(case)
    for mode in order:
        mgr.set_interface_time(mode)
        oc.set_interface_time(mode)
        mgr.fluidSimulate(2)
        oc.step(2)
    ctx.synchronize()
    _oracle_equal(mgr, oc, range(case.max_level + 1))
    mgr.close()


def test_cells_in_both_overlaps(ctx):
    """Cells that are overlap_F2C and overlap_C2F at once keep the reference's
    order, collision first and copy last."""
    import oracle as O
    from mortontrie_amr_b200.lbm import LBM_Manager
    case = _sphere()
    d = case.mesh.levels[1]
    d["overlap_C2F"] = np.sort(np.concatenate([d["overlap_C2F"], d["overlap_F2C"][::7]]))
    mgr = LBM_Manager(ctx, case)
    oc = O.OracleCase(case)
    mgr.fluidSimulate(3)
    oc.step(3)
    ctx.synchronize()
    _oracle_equal(mgr, oc, range(case.max_level + 1))
    mgr.close()


@pytest.mark.parametrize("schedule", ["phases", "fused"])
@pytest.mark.parametrize("markers", [1, 6, 199, 201])
def test_marker_counts(ctx, schedule, markers):
    """Direct forcing by few and odd numbers of markers (a warp each, four to a
    block): FP64 bit for bit, the body force to the order of its sum."""
    from helpers import run_oracle
    from mortontrie_amr_b200.case import df_sphere_case
    from mortontrie_amr_b200.lbm import LBM_Manager
    case = df_sphere_case(radius=2, max_level=1, re=50.0, oscillating=True, period=60)
    m = case.mesh.markers
    m.ref, m.dv = np.ascontiguousarray(m.ref[:, :markers]), np.ascontiguousarray(m.dv[:markers])
    mgr = LBM_Manager(ctx, case, schedule=schedule)
    mgr.fluidSimulate(5)
    ctx.synchronize()
    oc = run_oracle(case, 5)
    _oracle_equal(mgr, oc, range(case.max_level + 1))
    fg, fo = mgr.force(), oc.force()
    assert fg[3] == fo[3] == 10
    assert np.abs(fg[:3] - fo[:3]).max() <= 1e-12 * np.abs(fo[:3]).max()
    mgr.close()


def _sets_moved(what):
    """The nested sphere with some written children of level 1 taken out of
    overlap_C2F: collided like any cell (lat_f), or also sources of level 2's
    explosion (overlap_F2C, their children copied on level 2)."""
    case = _sphere()
    one, two = case.mesh.levels[1], case.mesh.levels[2]
    some = one["overlap_C2F"][::37]
    one["overlap_C2F"] = np.setdiff1d(one["overlap_C2F"], some)
    to = "lat_f" if what == "collided" else "overlap_F2C"
    one[to] = np.sort(np.concatenate([one[to], some]))
    if what == "sources":
        children = (some[:, None] + np.arange(8, dtype=np.uint64)).ravel()
        two["overlap_C2F"] = np.sort(np.concatenate([two["overlap_C2F"], children]))
    return case


@pytest.mark.parametrize("what", ["collided", "sources"])
@pytest.mark.parametrize("itime", ["reference", "hold", "extrap"])
@pytest.mark.parametrize("schedule", ["phases", "fused", "fused_lists"])
def test_exploded_cells_outside_the_copied_overlap(ctx, what, itime, schedule):
    """FP64, bit for bit against the oracle: children that the explosion writes
    and that something else than the copy writes too keep the order of a level's
    own work and both explosions of a held parent state."""
    import oracle as O
    from mortontrie_amr_b200.lbm import LBM_Manager
    case = _sets_moved(what)
    mgr = LBM_Manager(ctx, case, schedule=schedule, interface_time=itime)
    oc = O.OracleCase(case)
    oc.set_interface_time(itime)
    for n in (1, 2):
        mgr.fluidSimulate(n)
        oc.step(n)
        ctx.synchronize()
        _oracle_equal(mgr, oc, range(case.max_level + 1))
    mgr.close()


def test_interface_option_changed_while_steps_run(ctx):
    """The brick tables that an option drops stay with the steps still running:
    memory that another context takes meanwhile is not theirs."""
    from mortontrie_amr_b200.case import cavity_case
    from mortontrie_amr_b200.lbm import Context, LBM_Manager
    case = cavity_case(q=19, coarse=(32, 32, 32), max_level=2, re=100.0)
    want = LBM_Manager(ctx, case, schedule="fused", scaling="standard", interface_time="hold")
    got = LBM_Manager(ctx, case, schedule="fused", scaling="standard", interface_time="hold")
    other = Context(0)
    for mode in ("extrap", "hold"):
        for m in (want, got):
            m.fluidSimulate(30)
            if m is want:
                ctx.synchronize()
            m.set_interface_time(mode)
            if m is got:
                for _ in range(3):
                    x = LBM_Manager(other, case, "f16", schedule="fused")
                    x.fluidSimulate(1)
                    x.close()
    for l in range(case.max_level + 1):
        for a, b in zip(want.populations(l), got.populations(l)):
            assert np.isfinite(a).all() and np.array_equal(a, b), l
    want.close()
    got.close()
    other.close()


def test_force_of_a_step_that_failed(ctx):
    """mt_lbm_kernel that stops half way (extrapolated explosion without saved
    sources, in the second substep): the force of its first substep counts, now
    and not with some later call."""
    from mortontrie_amr_b200.lbm import LBM_Manager, MTError
    case = _sphere(1)
    mgr = LBM_Manager(ctx, case, interface_time="extrap")
    with pytest.raises(MTError, match="MT_ERR_STATE"):
        mgr.LBMkernel(0)
    f = mgr.force()
    assert f[3] == 1 and f[0] != 0
    mgr.reset_force()
    mgr.set_interface_time("hold")
    mgr.LBMkernel(0)
    assert mgr.force()[3] == 2
    mgr.close()
