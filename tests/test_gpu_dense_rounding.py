"""The dense path's reduced storages keep their rounding: post-collision
populations of a 4^3 cube after six steps, equal bit for bit to those that the
one-cell-per-thread kernels gave (golden/dense_reduced_rounding.npz, keys
q_collision_storage_stream), whichever kernel a model and storage runs."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "dense_reduced_rounding.npz")


@pytest.fixture(scope="module")
def ctx():
    from mortontrie_amr_b200.lbm import Context
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("q,collision", [(19, "LBGK"), (27, "LBGK"), (27, "Cumulant")])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("conv", ["reference", "textbook"])
def test_dense_reduced_storages_keep_their_rounding(ctx, q, collision, storage, conv):
    from mortontrie_amr_b200.case import uniform_box_case
    from mortontrie_amr_b200.lbm import DenseCase
    n = 4
    d = DenseCase(ctx, uniform_box_case(q=q, n=(n,) * 3, collision=collision, nu=0.02, stream_convention=conv), storage)
    rng = np.random.default_rng(q)
    d.init_fields(1 + 0.02 * rng.uniform(-1, 1, n ** 3), *(0.05 * rng.uniform(-1, 1, (3, n ** 3))))
    d.step(6)
    got = d.populations()[1]
    d.close()
    want = np.load(GOLDEN)[f"{q}_{collision}_{storage}_{conv}"]
    assert np.array_equal(got, want), float(np.abs(got - want).max())
