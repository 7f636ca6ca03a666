"""Blocks whose fields just fit the no-allocation step's 8 MiB of scratch are
taken however finely their stages are cut, and step like any other."""
import ctypes

import numpy as np
import pytest
import torch

from mhdvlct import block as B, capi, ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,n,npass", [
    ("hlld", (30, 58, 24), 0), ("hllc", (58, 30, 24), 0), ("hlld", (154, 55, 1), 0),
    ("hllc", (156, 19, 11), 0), ("hlld", (20, 147, 7), 2), ("hllc", (17, 144, 9), 2)])
def test_fields_that_just_fit_are_taken(solver, n, npass):
    mhd = solver != "hllc"
    state, w = ic.smooth_block(n, 3, seed=12, mhd=mhd)
    rng = np.random.default_rng(4)
    for k in range(npass):
        state[f"passive_{k}"] = state["density"] * (0.2 + 0.6 * rng.random(state["density"].shape))
    meth = B.EnzoMethodMHDVlct(mhd_choice="constrained_transport" if mhd else "no_bfield",
                               riemann_solver=solver)
    a, b = (B.Block(n, 3, w, mhd=mhd, npassive=npass) for _ in range(2))
    a.load_numpy(state)
    b.load_numpy(state)
    meth.compute(a, 1e-3)
    v = b.view()
    rc = capi.lib().mhdvlct_block_step_noalloc(meth.handle, ctypes.byref(v), 1e-3, None)
    assert rc == capi.MHD_OK, capi.lib().mhdvlct_last_error_string(meth.handle)
    torch.cuda.synchronize()
    x, y = a.to_numpy(), b.to_numpy()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
