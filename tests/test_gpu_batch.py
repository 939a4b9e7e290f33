"""Batches of independent multi-level cases (mt_batch_*): every member of a
batch ends each coarse step in the state it reaches stepped alone, whatever
the mix (models, levels, boundaries, brick or list levels), membership
changes and buffer parities."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from mortontrie_amr_b200.lbm import Context
    c = Context(0)
    yield c
    c.close()


def _mix():
    from mortontrie_amr_b200.case import cavity_case, df_sphere_case, nested_sphere_case, sphere_case
    return [
        sphere_case(coarse=(32, 16, 16), refine=[((6, 4, 4), (18, 12, 12))], center=(12, 8, 8), radius=2.0),
        nested_sphere_case(coarse=(48, 24, 24), max_level=2, center=(16, 12, 12), radius=2.0, half_widths=(4.0, 2.5),
                           re=50.0),
        cavity_case(q=19, coarse=(24, 24, 24), max_level=1, re=100.0),
        cavity_case(q=27, collision="Cumulant", coarse=(24, 24, 24), max_level=2, re=60.0),
        # periodic extent 18 is not a multiple of 4: level 0 runs from cell lists
        sphere_case(coarse=(30, 18, 18), refine=[((6, 5, 5), (18, 13, 13))], center=(12, 9, 9), radius=2.0),
        # direct-forcing oscillating sphere (Lagrangian markers)
        df_sphere_case(radius=3, max_level=2, re=60.0, oscillating=True, period=100),
    ]


def _state(mgr):
    out = []
    for l in range(mgr.L + 1):
        f, fcol = mgr.populations(l)
        rho, u = mgr.macros(l)
        out.append((f, fcol, rho, u))
    return out, mgr.force()


def _assert_same(a, b, exact=True):
    (sa, fa), (sb, fb) = a, b
    for la, lb in zip(sa, sb):
        for x, y in zip(la, lb):
            if exact:
                assert np.array_equal(x, y), float(np.nanmax(np.abs(x - y)))
            else:
                np.testing.assert_allclose(x, y, rtol=1e-6, atol=1e-7)
    if exact:
        assert np.array_equal(fa, fb)
    else:
        np.testing.assert_allclose(fa, fb, rtol=1e-6, atol=1e-9)


@pytest.mark.parametrize("storage", ["f64", "f16"])
def test_batch_members_equal_alone(ctx, storage):
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    cases = _mix()
    alone = [LBM_Manager(ctx, c, storage, schedule="fused") for c in cases]
    members = [LBM_Manager(ctx, c, storage) for c in cases]
    batch = Batch(ctx, members)
    assert len(batch) == len(cases)
    for m in alone:
        m.fluidSimulate(5)
    batch.step(2)
    batch.step(3)
    ctx.synchronize()
    for a, m in zip(alone, members):
        _assert_same(_state(a), _state(m), exact=(storage == "f64"))
    batch.close()


def test_batch_matches_phase_schedule_fp64(ctx):
    """FP64 members equal the reference's phase order stepped alone."""
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    cases = _mix()[:4]
    ref = [LBM_Manager(ctx, c, "f64") for c in cases]
    members = [LBM_Manager(ctx, c, "f64") for c in cases]
    batch = Batch(ctx, members)
    for m in ref:
        m.fluidSimulate(4)
    batch.step(4)
    ctx.synchronize()
    for a, m in zip(ref, members):
        _assert_same(_state(a), _state(m))
    batch.close()


def test_batch_membership_and_parity(ctx):
    """Members join at different coarse-step parities and leave mid-run; the
    others carry on unaffected; a member cannot be stepped on its own."""
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager, MTError
    cases = _mix()
    alone = [LBM_Manager(ctx, c, "f64", schedule="fused") for c in cases[:3]]
    m = [LBM_Manager(ctx, c, "f64", schedule="fused") for c in cases[:3]]
    m[1].fluidSimulate(1)           # odd parity before joining
    alone[1].fluidSimulate(1)
    batch = Batch(ctx, [m[0], m[1]])
    batch.step(3)
    for a in alone[:2]:
        a.fluidSimulate(3)
    with pytest.raises(MTError, match="MT_ERR_STATE"):
        m[0].fluidSimulate(1)
    batch.add(m[2])
    batch.step(2)
    for a in alone:
        a.fluidSimulate(2)
    batch.remove(m[0])
    batch.step(1)
    for a in alone[1:]:
        a.fluidSimulate(1)
    m[0].fluidSimulate(1)           # alone again
    alone[0].fluidSimulate(1)
    ctx.synchronize()
    for a, x in zip(alone, m):
        _assert_same(_state(a), _state(x))
    batch.close()


@pytest.mark.parametrize("storage", ["f64", "f16"])
def test_large_member_runs_its_own_pass(ctx, storage):
    """A member whose level holds 8192 bricks or more (here both levels of a
    96^3 cavity: 706,536 and 1,729,792 cells) runs its own brick pass beside
    the batched pass of the small members; every member still equals itself
    stepped alone."""
    from mortontrie_amr_b200.case import cavity_case
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    cases = [cavity_case(q=19, coarse=(96, 96, 96), max_level=1, re=100.0, mesh="device")] + _mix()[:2]
    alone = [LBM_Manager(ctx, c, storage, schedule="fused") for c in cases]
    members = [LBM_Manager(ctx, c, storage) for c in cases]
    assert members[0].size(0) >= 8192 * 64
    batch = Batch(ctx, members)
    for m in alone:
        m.fluidSimulate(3)
    batch.step(3)
    ctx.synchronize()
    for a, m in zip(alone, members):
        _assert_same(_state(a), _state(m), exact=(storage == "f64"))
    batch.close()
    for m in alone + members:
        m.close()


@pytest.mark.parametrize("with_levels", [False, True])
def test_single_level_direct_forcing_member(ctx, with_levels):
    """A direct-forcing sphere without refinement steps in a batch, by itself
    and after members with levels, as alone."""
    from mortontrie_amr_b200.case import df_sphere_case
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    cases = (_mix()[:2] if with_levels else []) + [
        df_sphere_case(radius=3, max_level=0, re=40.0, oscillating=True, period=100)]
    alone = [LBM_Manager(ctx, c, "f64", schedule="fused") for c in cases]
    members = [LBM_Manager(ctx, c, "f64") for c in cases]
    batch = Batch(ctx, members)
    for m in alone:
        m.fluidSimulate(3)
    batch.step(3)
    ctx.synchronize()
    for a, m in zip(alone, members):
        _assert_same(_state(a), _state(m))
    batch.close()


def test_members_sharing_branches(ctx):
    """More members than branches, of 0 to 2 levels: those that share a branch
    follow one another on its streams, each as it steps alone."""
    from mortontrie_amr_b200.case import cavity_case, df_sphere_case
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    kinds = [df_sphere_case(radius=3, max_level=0, re=40.0, oscillating=True, period=100),
             cavity_case(q=19, coarse=(16, 16, 16), max_level=1, re=100.0),
             cavity_case(q=27, collision="Cumulant", coarse=(24, 24, 24), max_level=2, re=60.0),
             cavity_case(q=19, coarse=(16, 16, 20), max_level=1, re=80.0), _mix()[5]]
    alone = [LBM_Manager(ctx, c, "f64", schedule="fused") for c in kinds]
    for m in alone:
        m.fluidSimulate(3)
    want = [_state(m) for m in alone]
    members = [LBM_Manager(ctx, kinds[(3 * i) % 5], "f64") for i in range(39)]
    batch = Batch(ctx, members)
    batch.step(3)
    ctx.synchronize()
    for i, m in enumerate(members):
        _assert_same(want[(3 * i) % 5], _state(m))
    batch.close()
    for m in alone + members:
        m.close()


def _pass_forms(batch):
    """The forms of the brick passes that two steps of the batch (one graph) launch."""
    import re
    import torch
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        batch.step(2)
        batch.ctx.synchronize()
    if not any("mt::k_" in e.name for e in p.events()):
        pytest.skip("no kernel trace on this machine")
    names = [e.name for e in p.events() if "k_brick_step" in e.name]
    return {int(re.search(r"k_brick_step<\d+, \w+, \d+, (\d+)>", n).group(1)) for n in names}


def test_tuned_member_steps_in_its_new_forms(ctx):
    """The tuner's choice reaches a batch that has captured its step before."""
    from mortontrie_amr_b200.case import sphere_case
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    case = sphere_case(coarse=(128, 64, 64), refine=[((36, 24, 24), (60, 40, 40))], center=(48, 32, 32), radius=3.0,
                       mesh="device")
    m = LBM_Manager(ctx, case, "f16", schedule="fused")
    m.set_brick_forms([1, 1])  # cell by cell, never the fastest on levels of this size
    batch = Batch(ctx, [m])
    batch.step(2)
    assert _pass_forms(batch) == {1}
    v, _ = m.tune_bricks()
    assert _pass_forms(batch) == set(v[v >= 0].tolist())
    batch.close()
    m.close()


@pytest.mark.parametrize("what", ["scaling", "face", "schedule"])
def test_member_changed_between_batch_steps(ctx, what):
    """What a captured step bakes in, changed on a member, reaches the batch."""
    from mortontrie_amr_b200.case import cavity_case
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    case = cavity_case(q=19, coarse=(24, 24, 24), max_level=1, re=100.0)

    def change(m):
        if what == "scaling":
            m.set_interface_scaling("standard")
        elif what == "face":
            m.set_face_velocity(5, (0.02, 0.01, 0.0))
        else:
            m.set_schedule("fused_lists")

    alone, member, plain = (LBM_Manager(ctx, case, "f64", schedule="fused") for _ in range(3))
    batch = Batch(ctx, [member, plain])
    alone.fluidSimulate(2)
    batch.step(2)
    change(alone)
    change(member)
    alone.fluidSimulate(2)
    batch.step(2)
    ctx.synchronize()
    _assert_same(_state(alone), _state(member))
    if what != "schedule":
        assert not np.array_equal(member.populations(1)[0], plain.populations(1)[0])
    batch.close()
    for m in (alone, member, plain):
        m.close()


@pytest.mark.parametrize("storage", ["f64", "f16"])
@pytest.mark.parametrize("counts", [(3, 3, 2), (1, 4, 1, 2), (2, 1, 5), (4, 3, 2, 2, 1, 3)])
def test_step_counts_of_any_parity(ctx, storage, counts):
    """Two steps in one graph and single ones, from either buffer parity."""
    from mortontrie_amr_b200.lbm import Batch, LBM_Manager
    # (FP16: the flows that stay finite)
    cases = [_mix()[k] for k in ((0, 2, 4, 5) if storage == "f64" else (2, 3))]
    alone = [LBM_Manager(ctx, c, storage, schedule="fused") for c in cases]
    members = [LBM_Manager(ctx, c, storage) for c in cases]
    batch = Batch(ctx, members)
    for n in counts:
        batch.step(n)
        for m in alone:
            m.fluidSimulate(n)
        ctx.synchronize()
        for a, m in zip(alone, members):
            _assert_same(_state(a), _state(m))
    batch.close()
    for m in alone + members:
        m.close()
