"""The fused pass over 4x4x4 bricks (pairs of cells, slots of absent cells)
against the pass over cell lists and the neighbour table, which knows
nothing of bricks: the same arithmetic from two independent ways of finding
and moving the populations, so the states agree bit for bit (a cell's
collision is a fixed sequence of rounded operations, whatever the kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from mortontrie_amr_b200.lbm import Context
    c = Context(0)
    yield c
    c.close()


def _case(which, conv):
    from mortontrie_amr_b200.case import cavity_case, df_sphere_case, sphere_case
    if which == "q19":      # boxes off the brick grid on both levels, periodic sides
        return sphere_case(coarse=(36, 20, 24), max_level=2, refine=[((7, 4, 5), (21, 17, 19)), ((17, 12, 13), (39, 31, 35))],
                           center=(14, 11, 12), radius=2.5, re=40.0, stream_convention=conv)
    if which == "q27":
        return sphere_case(q=27, collision="Cumulant", coarse=(36, 20, 24), max_level=1, refine=[((7, 4, 5), (21, 17, 19))],
                           center=(14, 11, 12), radius=2.5, re=40.0, stream_convention=conv)
    if which == "q27_lbgk":
        return sphere_case(q=27, collision="LBGK", coarse=(36, 20, 24), max_level=1, refine=[((7, 4, 5), (21, 17, 19))],
                           center=(14, 11, 12), radius=2.5, re=40.0, stream_convention=conv)
    if which == "cavity":   # odd extents, walls on every face
        return cavity_case(q=19, coarse=(25, 22, 27), max_level=1, re=60.0)
    return df_sphere_case(radius=3, max_level=1, re=50.0, oscillating=True, period=60)


@pytest.mark.parametrize("which,conv", [("q19", "reference"), ("q19", "textbook"), ("q27", "reference"),
                                        ("q27", "textbook"), ("q27_lbgk", "reference"), ("cavity", "reference"),
                                        ("df", "reference")])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "f64"])
def test_brick_pass_equals_list_pass(ctx, which, conv, storage):
    from mortontrie_amr_b200.lbm import LBM_Manager
    case = _case(which, conv)
    runs = []
    for schedule, form in (("fused", 0), ("fused_lists", 0), ("fused", 3 if storage == "f64" else 1)):
        m = LBM_Manager(ctx, case, storage, schedule=schedule, scaling="standard", interface_time="hold")
        m.set_brick_forms([form] * (case.max_level + 1))
        m.fluidSimulate(5)
        runs.append(m)
    ctx.synchronize()
    a = runs[0]
    for b in runs[1:]:
        for l in range(case.max_level + 1):
            fa, ca = a.populations(l)
            fb, cb = b.populations(l)
            assert np.isfinite(fa).all() and np.array_equal(fa, fb) and np.array_equal(ca, cb), l
            for x, y in zip(a.macros(l), b.macros(l)):
                assert np.array_equal(x, y), l
        assert np.array_equal(a.force(), b.force())
    for m in runs:
        m.close()


def test_cells_outside_slots(ctx):
    """A level of scattered cells (most slots of most bricks empty): keys, tags,
    find and the neighbour table by position in key order."""
    from mortontrie_amr_b200.case import cavity_case
    from mortontrie_amr_b200.lbm import LBM_Manager
    case = cavity_case(q=27, collision="Cumulant", coarse=(25, 22, 27), max_level=1, re=60.0)
    m = LBM_Manager(ctx, case, "f16")
    for l in range(2):
        want = case.mesh.all_keys(l)
        keys, tags = m.keys(l)
        assert m.size(l) == want.size and np.array_equal(keys, want) and (tags != 0).all()
        assert np.array_equal(m.find(l, want), np.arange(want.size))
        absent = np.setdiff1d(np.arange(int(want.max()) + 2, dtype=np.uint64), want)[:4096]
        assert (m.find(l, absent) == -1).all()
        nb = m.neighbors(l)
        assert nb.max() < want.size and nb.min() == -1
        j = nb[0]  # +x links: the key's x advances by one cell
        from mortontrie_amr_b200.lattice import morton_decode
        xyz = np.stack(morton_decode(want)).astype(np.int64)
        ok = j >= 0
        d = xyz[:, j[ok]] - xyz[:, ok]
        assert (d[0] == 1 << (1 - l)).all() and (d[1:] == 0).all()
    m.close()


def test_macros_of_an_infinite_population_f64(ctx):
    """calculateMacros multiplies every population by its direction, zero
    components included: an infinite one leaves no component finite."""
    from mortontrie_amr_b200.lattice import directions
    from mortontrie_amr_b200.lbm import LBM_Manager
    m = LBM_Manager(ctx, _case("q19", "reference"))
    f, fcol = m.populations(1)
    cells = np.flatnonzero(m.keys(1)[1] & 1)[5::41]
    for j, c in enumerate(cells):
        f[j % 19, c] = (np.inf, -np.inf)[j % 2]
    m.set_populations(1, f, fcol)
    m.calculateMacros(1)
    rho, u = m.macros(1)
    with np.errstate(invalid="ignore"):
        e = np.array(directions(19)[:3], float).T
        r, v = f[0, cells].copy(), np.zeros((3, cells.size))
        for k in range(1, 19):
            r += f[k, cells]
            v += e[k][:, None] * f[k, cells]
        v /= r
    assert np.array_equal(rho[cells], r) and np.array_equal(u[:, cells], v, equal_nan=True)
    assert np.isnan(v).all(axis=0).sum() >= cells.size * 17 // 19
    m.close()


@pytest.mark.parametrize("which", ["q19", "q27_lbgk", "df"])
def test_macros_of_overflowed_16_bit_populations(ctx, which):
    """Collisions that overflow FP16 storage: the fused passes write the macros
    that the phase order's calculateMacros gives, NaN in the same places."""
    from mortontrie_amr_b200.lbm import LBM_Manager
    got = []
    for schedule in ("phases", "fused", "fused_lists"):
        m = LBM_Manager(ctx, _case(which, "reference"), "f16", schedule=schedule)
        f, fcol = m.populations(0)
        for c in np.flatnonzero(m.keys(0)[1] & 1)[3::29]:
            f[[1, 7, 9, 11, 13], c] = 6e4  # 7/18 of their sum goes on in direction 1
        m.set_populations(0, f, fcol)
        m.fluidSimulate(1)
        got.append(m.macros(0) + m.populations(0))
        m.close()
    assert np.isinf(got[0][2]).any() and np.isnan(got[0][1]).any()
    for other in got[1:]:
        for a, b in zip(got[0][:3], other[:3]):
            assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b))
