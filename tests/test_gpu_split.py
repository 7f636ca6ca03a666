"""The FP64 stages as sequences of kernels over whole blocks (vlct_split.cuh),
at the sizes where their cutting of the work can go wrong: lines of faces that
leave a remainder, blocks of one cell, a block cut into z-slabs, a batch of
more blocks than share the workspace; and states that are not finite.  The
results are the oracle's (or another cutting's) bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as O
from mhdvlct import block as B, capi, ic
from helpers import oracle_block, oracle_params
from test_gpu_batch import Batch

pytestmark = pytest.mark.gpu


def _method(solver, recon, de=False):
    return B.EnzoMethodMHDVlct(
        mhd_choice="no_bfield" if solver == "hllc" else "constrained_transport",
        riemann_solver=solver, reconstruct_method=recon, dual_energy=de)


def _cycle_equals_oracle(state, n, w, solver, recon, de, dt=None):
    mhd = solver != "hllc"
    meth = _method(solver, recon, de)
    blk = B.Block(n, 3, w, mhd=mhd, dual_energy=de)
    blk.load_numpy(state)
    ob = oracle_block(state, n, 3, w, mhd=mhd, de=de)
    prm = oracle_params(solver, recon, de=de, courant=meth.courant)
    if dt is None:
        dt = O.timestep(prm, ob)
        assert meth.timestep(blk) == dt
    O.fill_ghosts_periodic(ob)
    meth.fill_ghosts_periodic(blk)
    O.step(prm, ob, dt)
    meth.compute(blk, dt)
    torch.cuda.synchronize()
    got = blk.to_numpy()
    for k, a in got.items():
        assert np.array_equal(a, ob.f[ic.ORACLE_NAME[k]], equal_nan=True), k


@pytest.mark.parametrize("n,solver,recon,de", [
    ((3, 3, 3), "hlld", "plm", False),        # the smallest a periodic block can be
    ((3, 5, 40), "hlle", "plm_athena", True),  # lines of very different lengths
    ((33, 9, 17), "hlld", "plm", False),      # remainders along every axis
    ((41, 4, 7), "hllc", "plm", True),
    ((16, 13, 29), "hllc", "nn", False),
    ((120, 118, 92), "hlld", "plm", False),   # 126 x 124 x 98 cells: two z-slabs
])
def test_cutting_equals_oracle(n, solver, recon, de):
    state, w = ic.smooth_block(n, 3, seed=11, mhd=solver != "hllc", dual_energy=de)
    _cycle_equals_oracle(state, n, w, solver, recon, de)


@pytest.mark.parametrize("solver,recon,de", [
    ("hlld", "plm", False), ("hlld", "nn", True), ("hllc", "plm", True),
    ("hlle", "plm_athena", False)])
def test_not_finite_and_zero_values_equal_oracle(solver, recon, de):
    # the sign tests, minima and side selections on bit patterns, where the
    # comparisons they stand for see NaN, infinities and zeros of both signs
    n = (10, 9, 11)
    mhd = solver != "hllc"
    state, w = ic.smooth_block(n, 3, seed=5, mhd=mhd, dual_energy=de)
    rng = np.random.default_rng(9)
    for k, bad in (("velocity_y", np.nan), ("total_energy", np.inf), ("velocity_x", -np.inf),
                   ("density", 0.0), ("velocity_z", -0.0), ("total_energy", -1.0)):
        z, y, x = (int(rng.integers(4, 4 + m - 2)) for m in (n[2], n[1], n[0]))
        state[k][z, y, x] = bad
    state["velocity_z"][:, :, 8:] = -0.0
    if mhd:
        state["bfieldi_x"][:, :5, :] = 0.0  # B_x = +-0 on a plane of faces
        state["bfieldi_x"][:, :4, :] = -0.0
        state["bfieldi_z"][5, 5, 5] = np.nan
    _cycle_equals_oracle(state, n, w, solver, recon, de, dt=1e-3)


def test_groups_of_a_large_batch_equal_single_blocks():
    # 30 blocks of 38^3 cells and 40 of 11 x 17 x 23: more than one group, the
    # last one of mixed sizes
    meth = _method("hlld", "plm")
    dims = [(32, 32, 32)] * 30 + [(5, 11, 17)] * 40
    states = [ic.smooth_block(n, 3, seed=i % 5)[0] for i, n in enumerate(dims)]
    widths = [(1.0 / 32,) * 3] * len(dims)
    bt = Batch(meth, dims, widths)
    for i, s in enumerate(states):
        bt.upload(i, s)
    dts = (ctypes.c_double * len(dims))(*[1e-3 + 1e-5 * i for i in range(len(dims))])
    capi.check(capi.lib().mhdvlct_batch_step(bt.h, dts, None), meth.handle, "step")
    for i in (0, 4, 22, 23, 24, 29, 30, 69):
        blk = B.Block(dims[i], 3, widths[i])
        blk.load_numpy(states[i])
        meth.compute(blk, dts[i])
        torch.cuda.synchronize()
        got, ref = bt.download(i), blk.to_numpy()
        act = (slice(3, -3),) * 3
        for k in ("density", "velocity_x", "velocity_y", "velocity_z", "total_energy",
                  "bfield_x", "bfield_y", "bfield_z", "bfieldi_x", "bfieldi_y", "bfieldi_z"):
            assert np.array_equal(got[k][act], ref[k][act]), (i, k)
