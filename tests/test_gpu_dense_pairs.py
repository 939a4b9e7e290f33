"""The dense cumulant pass on pairs of cells (FP32, FP16, BF16) against the FP64
dense kernel, from the smallest cubes (an x neighbour pair is the pair
itself at 2^3) up, both stream conventions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 3
# half a unit in the last place of the stored deviation per step, and of the
# FP32 arithmetic on populations of up to 0.3 (about 60 operations deep); four
# times that covers the moments' share between directions
ULP = {"f32": 2.0 ** -24, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}


@pytest.mark.parametrize("n", [2, 4, 8, 32])
@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("conv", ["reference", "textbook"])
def test_dense_cumulant_pairs_close_to_f64(n, storage, conv):
    from mortontrie_amr_b200.case import uniform_box_case
    from mortontrie_amr_b200.lattice import weights
    from mortontrie_amr_b200.lbm import Context, DenseCase
    ctx = Context(0)
    rng = np.random.default_rng(n)
    rho = 1.0 + 0.01 * rng.uniform(-1, 1, n ** 3)
    u = 0.03 * rng.uniform(-1, 1, (3, n ** 3))
    case = uniform_box_case(q=27, n=(n, n, n), nu=0.02, collision="Cumulant", stream_convention=conv)
    got = []
    for st in ("f64", storage):
        d = DenseCase(ctx, case, st)
        d.init_fields(rho, *u)
        d.step(STEPS)
        got.append(d.populations())
        d.close()
    w = weights(27)[:, None]
    for a, b in zip(*got):
        dev = np.abs(a - w).max()
        tol = 4.0 * STEPS * (dev * ULP[storage] + 60 * 0.3 * 2.0 ** -24)
        assert np.isfinite(b).all() and np.abs(a - b).max() <= tol, (float(np.abs(a - b).max()), tol)
    ctx.close()


def test_large_fields_into_pageable_and_pinned_memory():
    """A result large enough for the staged copy arrives the same in ordinary
    arrays and in page-locked ones."""
    import torch
    from mortontrie_amr_b200.case import uniform_box_case
    from mortontrie_amr_b200.lbm import Context, DenseCase
    ctx = Context(0)
    n = 128
    rng = np.random.default_rng(1)
    d = DenseCase(ctx, uniform_box_case(q=19, n=(n, n, n), nu=0.02), "f32")
    d.init_fields(1.0 + 0.01 * rng.uniform(-1, 1, n ** 3), *(0.03 * rng.uniform(-1, 1, (3, n ** 3))))
    d.step(2)
    pinned = torch.empty(4, n ** 3, dtype=torch.float64, pin_memory=True)
    d.macros_ptr(pinned[0].data_ptr(), pinned[1].data_ptr())
    for _ in range(2):  # the staging's first use and its reuse
        rho, u = d.macros()
        assert np.array_equal(rho, pinned[0].numpy()) and np.array_equal(u, pinned[1:].numpy())
    d.close()
    ctx.close()
