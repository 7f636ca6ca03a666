"""The FP32 dual-energy sync where the magnetic energy cancels nearly all of the
total energy (plasma beta of 1e-6).  The internal energy that the step stores is
etot - |B|^2 / (2 rho) of the stored fields, and what float-float arithmetic with
IEEE divisions loses of it is bounded."""
import numpy as np
import pytest
import torch

from mhdvlct import block as B

pytestmark = pytest.mark.gpu


def test_internal_energy_of_magnetically_dominated_cells():
    # at rest, and over a time so short that no flux changes a value: the stored
    # fields are the sync's inputs and its results
    rng = np.random.default_rng(3)
    meth = B.EnzoMethodMHDVlct(riemann_solver="hlle", reconstruct_method="nn",
                               dual_energy=True, dual_energy_eta=1e-12)
    n, g = 48, 3
    m = n + 2 * g
    bfx = rng.uniform(0.5, 2.0, (m, m, m + 1)).astype(np.float32)
    bx = np.float32(0.5) * (bfx[:, :, :-1] + bfx[:, :, 1:])
    rho = rng.uniform(0.5, 2.0, bx.shape).astype(np.float32)
    nte = bx.astype(np.float64) ** 2 / (2 * rho.astype(np.float64))
    blk = B.Block((n, n, n), g, (1.0, 1.0, 1.0), dual_energy=True, dtype=torch.float32)
    blk.load_numpy({
        "density": rho, "bfield_x": bx, "bfieldi_x": bfx,
        "total_energy": nte * (1 + rng.integers(3, 8, bx.shape) * 2.0 ** -23),
        "internal_energy": np.full(bx.shape, 1e-10)})
    meth.compute(blk, 1e-30)
    torch.cuda.synchronize()
    f = {k: v[g:-g, g:-g, g:-g].astype(np.float64) for k, v in blk.to_numpy().items()
         if not k.startswith("bfieldi")}
    for k in ("bfield_y", "bfield_z", "velocity_x", "velocity_y", "velocity_z"):
        assert np.abs(f[k]).max() < 1e-20, k
    nte = f["bfield_x"] ** 2 / (2 * f["density"])
    exact = f["total_energy"] - nte
    # cells that certainly took their internal energy from the total energy: the
    # advected one, 1e-10, leaves a total energy within half an ulp of nte
    took = exact >= 2.0 ** -22 * nte
    assert took.mean() > 0.3
    # one rounding of the difference, and the quotient's three: of the leading
    # quotient's remainder plus the low part, at most 2^-23 of the numerator, and
    # of that over rho
    bound = 2.0 ** -24 * exact + 2.0 ** -46 * nte * (1 + 2.0 ** -20)
    worst = (np.abs(f["internal_energy"] - exact) / bound)[took]
    assert (worst <= 1).all(), (worst.max(), (worst > 1).mean())
