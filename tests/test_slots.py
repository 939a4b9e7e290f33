"""estimate_slots bounds the slots (64 per 4x4x4 brick in use) a level takes on
the device, from the specification alone."""
import numpy as np
import pytest

from mortontrie_amr_b200.case import cavity_case, df_sphere_case, sphere_case
from mortontrie_amr_b200.mesh import Octree, estimate_slots


@pytest.mark.parametrize("make", [
    lambda: sphere_case(),
    lambda: cavity_case(coarse=(45, 37, 41), max_level=2),
    lambda: df_sphere_case(radius=4, max_level=2, oscillating=True),
    lambda: df_sphere_case(radius=3, max_level=2, octree=Octree(2.0, 4)),
])
def test_estimate_slots_bounds_the_bricks(make):
    m = make().mesh
    L = m.spec.max_level
    real = [64 * np.unique(m.all_keys(l) >> np.uint64(3 * (L - l) + 6)).size for l in range(L + 1)]
    est = estimate_slots(m.spec)
    assert len(est) == L + 1
    for r, e in zip(real, est):
        assert r <= e <= 1.1 * r


def test_slots_of_a_mesh_are_counted_once_for_its_copies():
    """A request's mesh is its template's with other markers: the count of its
    bricks is the template's, and sets of other sizes are counted anew."""
    import dataclasses
    mesh = sphere_case().mesh
    L = mesh.spec.max_level
    count = lambda m: [64 * np.unique(m.all_keys(l) >> np.uint64(3 * (L - l) + 6)).size for l in range(L + 1)]  # noqa: E731
    copy = dataclasses.replace(mesh, markers=None)
    assert copy.n_slots() == count(mesh)
    assert mesh.n_slots() is copy.n_slots()
    levels = [dict(d) for d in mesh.levels]
    levels[L]["lat_f"] = levels[L]["lat_f"][:1000]
    less = dataclasses.replace(mesh, levels=levels)
    assert less.n_slots() == count(less) and mesh.n_slots() == count(mesh)
