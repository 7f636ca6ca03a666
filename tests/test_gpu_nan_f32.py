"""FP32 HLLE steps of states with NaN densities: next to such a cell the density
fluxes are NaN and the edge EMFs finite, with the upwind weight 1/2 for those
faces; the face B there is the FP64 step's (the oracle's bit for bit) within FP32's
error.  (With NN: HLLD's flux is NaN in all components there, and the FP32 PLM
limiter takes no slope from a NaN where the FP64 one does.)"""
import numpy as np
import pytest
import torch

from mhdvlct import block as B, ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_face_b_next_to_nan_densities(seed):
    n = (14, 11, 13)
    s, w = ic.smooth_block(n, 3, seed=seed)
    rng = np.random.default_rng(seed)
    # rough velocities: the four EMFs that the weights choose from are far apart
    for k in "xyz":
        s["velocity_" + k] = s["velocity_" + k] + 0.5 * rng.standard_normal(s["density"].shape)
    s["total_energy"] = s["total_energy"] + 2.0
    for _ in range(3):
        z, y, x = (int(rng.integers(5, 5 + m - 4)) for m in (n[2], n[1], n[0]))
        s["density"][z, y, x] = np.nan
    meth = B.EnzoMethodMHDVlct(riemann_solver="hlle", reconstruct_method="nn")
    out = []
    for dtype in (torch.float32, torch.float64):
        blk = B.Block(n, 3, w, dtype=dtype)
        blk.load_numpy(s)
        meth.compute(blk, 5e-3)
        torch.cuda.synchronize()
        out.append(blk.to_numpy())
    for k in ("bfieldi_x", "bfieldi_y", "bfieldi_z"):
        a, r = out[0][k].astype(np.float64), out[1][k]
        assert np.array_equal(np.isfinite(a), np.isfinite(r)), k
        ok = np.isfinite(r)
        assert np.abs(a - r)[ok].max() <= 1e-5 * np.abs(r[ok]).max(), k
