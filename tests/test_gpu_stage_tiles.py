"""The fused stage kernel gives every cell the same value whatever tile and
z-chunk it falls into: FP32 states after two batched steps, bit for bit, at
tiles from one column to the largest the kernel holds, against its default; and
the FP64 instantiation (the no-allocation step runs it) against the split
kernels on blocks whose columns do not fill their tiles."""
import ctypes

import numpy as np
import pytest
import torch

from mhdvlct import block as B, capi, ic
from test_gpu_batch import Batch, ctypes_cuda_memcpy

pytestmark = pytest.mark.gpu


def _method(solver, recon, de=False):
    return B.EnzoMethodMHDVlct(
        mhd_choice="no_bfield" if solver == "hllc" else "constrained_transport",
        riemann_solver=solver, reconstruct_method=recon, dual_energy=de)


def _run(meth, dims, states, widths, tile, npassive=0, gravity=False):
    bt = Batch(meth, dims, widths, dtype=capi.MHD_DTYPE_F32, npassive=npassive, gravity=gravity)
    for i, s in enumerate(states):
        bt.upload(i, s)
        v = bt.view(i)
        if v.internal_energy:  # not among the fields Batch handles
            ctypes_cuda_memcpy(v.internal_energy, np.ascontiguousarray(
                s["internal_energy"], dtype=np.float32), to_device=True)
    L = capi.lib()
    if tile is not None:
        for stage in (0, 1):
            capi.check(L.mhdvlct_batch_set_stage_tile(bt.h, stage, *tile, 256), meth.handle, "tile")
    # two steps without a refresh between them: a block of fewer cells than
    # ghosts cannot be refreshed from itself in parallel
    dts = (ctypes.c_double * len(dims))(*[2e-3 + 1e-4 * i for i in range(len(dims))])
    for _ in range(2):
        capi.check(L.mhdvlct_batch_step(bt.h, dts, None), meth.handle, "step")
    return [bt.download(i) for i in range(len(dims))]


@pytest.mark.parametrize("solver,recon,de,npass,gravity", [
    ("hlld", "plm", False, 0, False), ("hlld", "nn", True, 0, False),
    ("hlle", "plm_athena", True, 2, True), ("hllc", "plm", False, 1, False),
    ("hllc", "nn", True, 0, True)])
def test_tiles_do_not_change_results(solver, recon, de, npass, gravity):
    meth = _method(solver, recon, de)
    # windows of 46, 13 and 3 columns; blocks of one and of five cells a side
    dims = [(42, 11, 9), (9, 42, 7), (1, 5, 30)]
    states, widths = [], []
    rng = np.random.default_rng(3)
    for i, n in enumerate(dims):
        s, _ = ic.smooth_block(n, 3, seed=40 + i, mhd=solver != "hllc", dual_energy=de)
        shp = s["density"].shape
        for k in range(npass):
            s[f"passive_{k}"] = s["density"] * (0.2 + 0.6 * rng.random(shp))
        if gravity:
            for k in ("acceleration_x", "acceleration_y", "acceleration_z"):
                s[k] = 0.3 * (rng.random(shp) - 0.5)
        states.append(s)
        widths.append((0.05, 0.05, 0.05))
    ref = _run(meth, dims, states, widths, None, npass, gravity)
    for tile in ((1, 1, 1), (2, 3, 5), (40, 4, 0), (4, 40, 3), (14, 14, 0), (40, 40, 2)):
        got = _run(meth, dims, states, widths, tile, npass, gravity)
        for i, (a, b) in enumerate(zip(got, ref)):
            for k in a:
                assert np.array_equal(a[k], b[k], equal_nan=True), (tile, i, k)
                assert np.isfinite(b[k]).all(), (i, k)


@pytest.mark.parametrize("n,solver,recon,de", [
    ((31, 5, 6), "hlld", "plm", True), ((4, 29, 5), "hlle", "plm_athena", False),
    ((3, 4, 33), "hllc", "plm", True), ((16, 15, 14), "hlld", "nn", False)])
def test_fp64_fused_equals_split(n, solver, recon, de):
    meth = _method(solver, recon, de)
    mhd = solver != "hllc"
    state, w = ic.smooth_block(n, 3, seed=8, mhd=mhd, dual_energy=de)
    a, b = (B.Block(n, 3, w, mhd=mhd, dual_energy=de) for _ in range(2))
    a.load_numpy(state)
    b.load_numpy(state)
    dt = meth.timestep(a)
    assert meth.timestep(b) == dt
    meth.compute(a, dt)
    v = b.view()
    capi.check(capi.lib().mhdvlct_block_step_noalloc(
        meth.handle, ctypes.byref(v), dt, torch.cuda.current_stream().cuda_stream),
        meth.handle, "noalloc")
    torch.cuda.synchronize()
    fa, fb = a.to_numpy(), b.to_numpy()
    for k in fa:
        assert np.array_equal(fa[k], fb[k]), k
