"""The FP64 stages as the fused kernel, which a batch or a handle runs where the
split kernels' workspace cannot be had: tiles and z-chunks pulled from the
launch's queue, gravity and passive scalars, stored boundary fluxes with flux
correction, and the host-state run by groups of blocks.  The results are the
split kernels' bit for bit, and where a cheap oracle run exists the oracle's."""
import ctypes
import json

import numpy as np
import pytest
import torch

from oracle import oracle as O
from mhdvlct import block as B, capi, ic
from helpers import oracle_block, oracle_params
from test_flux_correct_oracle import smr_blocks
from test_gpu_batch import (KEYS, Batch, ctypes_cuda_memcpy, ctypes_cuda_memcpy_raw)
from test_gpu_flux_correct_mesh import NAMES, ONAMES

pytestmark = pytest.mark.gpu
FORMS = ("split", "fused")


def _method(form, solver="hlld", recon="plm", de=False, **kw):
    meth = B.EnzoMethodMHDVlct(
        mhd_choice="no_bfield" if solver == "hllc" else "constrained_transport",
        riemann_solver=solver, reconstruct_method=recon, dual_energy=de, **kw)
    L = capi.lib()
    assert L.mhdvlct_internal_use_split(meth.handle, int(form == "split")) == capi.MHD_OK
    return meth


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("tile", [None, (14, 14, 0), (16, 8, 5), (5, 3, 1)])
def test_tiles_and_chunks_equal_oracle(form, tile):
    meth = _method(form)
    n = (26, 20, 40)
    s, w = ic.smooth_block(n, 3, seed=404)
    bt = Batch(meth, [n], [w])
    bt.upload(0, s)
    L = capi.lib()
    for stage in (0, 1) if tile else ():
        capi.check(L.mhdvlct_batch_set_stage_tile(bt.h, stage, *tile, 0), meth.handle, "tile")
    capi.check(L.mhdvlct_batch_run(bt.h, 2, 0, None, None), meth.handle, "run")
    ob = oracle_block(s, n, 3, w)
    prm = oracle_params(courant=meth.courant)
    for _ in range(2):
        dt = O.timestep(prm, ob)
        O.fill_ghosts_periodic(ob)
        O.step(prm, ob, dt)
    got = bt.download(0)
    act = (slice(3, -3),) * 3
    for k in KEYS:
        assert np.array_equal(got[k][act], ob.f[ic.ORACLE_NAME[k]][act]), k


@pytest.mark.parametrize("solver,recon,de", [
    ("hlld", "plm", True), ("hlle", "nn", False), ("hllc", "plm_athena", True)])
def test_gravity_and_scalars_of_uneven_blocks(solver, recon, de):
    dims, npass = [(17, 9, 12), (5, 33, 8), (8, 8, 8)], 2
    rng = np.random.default_rng(6)
    states, widths = [], []
    for i, n in enumerate(dims):
        s, w = ic.smooth_block(n, 3, seed=i, mhd=solver != "hllc", dual_energy=de)
        shp = s["density"].shape
        for k in range(npass):
            s[f"passive_{k}"] = s["density"] * (0.2 + 0.6 * rng.random(shp))
        for k in "xyz":
            s[f"acceleration_{k}"] = rng.random(shp) - 0.5
        states.append(s)
        widths.append(w)
    dts = (ctypes.c_double * 3)(2e-3, 1e-3, 3e-3)
    out = []
    for form in FORMS:
        meth = _method(form, solver, recon, de)
        bt = Batch(meth, dims, widths, npassive=npass, gravity=True)
        for i, s in enumerate(states):
            bt.upload(i, s)
            v = bt.view(i)
            if v.internal_energy:  # not among the fields Batch handles
                ctypes_cuda_memcpy(v.internal_energy,
                                   np.ascontiguousarray(s["internal_energy"]), to_device=True)
        capi.check(capi.lib().mhdvlct_batch_step(bt.h, dts, None), meth.handle, "step")
        out.append([bt.download(i) for i in range(3)])
    for i in range(3):
        for k, a in out[0][i].items():
            b = out[1][i][k][3:-3, 3:-3, 3:-3]
            assert np.isfinite(b).all(), (i, k)
            assert np.array_equal(a[3:-3, 3:-3, 3:-3], b), (i, k)


@pytest.mark.parametrize("form", FORMS)
def test_flux_correction_equals_oracle(form):
    n, g, cycles = 8, 4, 2
    mesh, oblocks, _ = smr_blocks(n, g)
    meth = _method(form, "hllc", courant=0.4)
    prm = O.params(riemann=O.HLLC, recon=O.PLM, mhd=False, courant=0.4)
    L = capi.lib()
    bt = Batch(meth, [(n,) * 3] * len(oblocks), [ob.widths for ob in oblocks], ghost=g)
    for i, ob in enumerate(oblocks):
        bt.upload(i, {k: ob.f[o] for k, o in zip(NAMES, ONAMES)})
    farr, nf = mesh.face_array()
    cons = capi.MHD_CONSERVATIVE_DEFAULT
    capi.check(L.mhdvlct_batch_set_refresh_faces(bt.h, farr, nf, cons), meth.handle, "faces")
    capi.check(L.mhdvlct_batch_set_flux_correction(bt.h, 0b11111, farr, nf, cons),
               meth.handle, "flux correction")
    capi.check(L.mhdvlct_batch_refresh(bt.h, None), meth.handle, "refresh")
    capi.check(L.mhdvlct_batch_run(bt.h, cycles, 0, None, None), meth.handle, "run")
    faces = mesh.face_ints()
    slots = [{0: b.f["rho"], 1: b.f["vx"], 2: b.f["vy"], 3: b.f["vz"], 4: b.f["etot"],
              9: b.f["pressure"]} for b in oblocks]
    fields = [{q: b.f[k] for q, k in enumerate(ONAMES)} for b in oblocks]
    O.refresh_faces(slots, (n,) * 3, (g,) * 3, faces, cons)
    for _ in range(cycles):
        dt = min(O.timestep(prm, b) for b in oblocks)
        O.refresh_faces(slots, (n,) * 3, (g,) * 3, faces, cons)
        fl = [O.step_fc(prm, b, dt) for b in oblocks]
        O.flux_correct(fields, fl, (n,) * 3, (g,) * 3, faces, cons)
    for i, ob in enumerate(oblocks):
        got = bt.download(i)
        for k, o in zip(NAMES, ONAMES):
            assert np.array_equal(got[k], ob.f[o]), (i, k)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("ngroups", [1, 3])
def test_run_host_equals_device_run(form, ngroups):
    nb, g, n = 2, 3, 12
    blocks, w = ic.turbulent_box(N=nb * n, nb=nb, g=g, seed=5, mach=1.5)
    nbr = ic.brick_neighbors(nb)
    L = capi.lib()
    meth = _method(form)
    runs = []
    for _ in range(2):
        bt = Batch(meth, [(n, n, n)] * 8, [w] * 8)
        capi.check(L.mhdvlct_batch_set_neighbors(
            bt.h, (ctypes.c_int * nbr.size)(*nbr.ravel().tolist())))
        for i, s in enumerate(blocks):
            bt.upload(i, s)
        runs.append(bt)
    dev, hst = runs
    capi.check(L.mhdvlct_batch_run(dev.h, 2, 0, None, None), meth.handle, "run")
    segp, segb, nseg = (ctypes.c_void_p * 2)(), (ctypes.c_size_t * 2)(), ctypes.c_int()

    def state(bt):
        torch.cuda.synchronize()
        capi.check(L.mhdvlct_batch_state_segments(bt.h, segp, segb, 2, ctypes.byref(nseg)))
        out = torch.empty(sum(segb[k] for k in range(nseg.value)), dtype=torch.uint8,
                          pin_memory=True)
        off = 0
        for k in range(nseg.value):
            ctypes_cuda_memcpy_raw(out.data_ptr() + off, segp[k], segb[k], to_device=False)
            off += segb[k]
        return out

    host = state(hst)
    capi.check(L.mhdvlct_batch_run_host(hst.h, host.data_ptr(), host.numel(), 2, ngroups, None,
                                        None), meth.handle, "run_host")
    torch.cuda.synchronize()
    assert torch.equal(host, state(dev))


def test_block_step_with_stored_fluxes():
    n, g = (12, 9, 10), 4
    s, w = ic.smooth_block(n, g, seed=8, mhd=False, dual_energy=True)
    out = []
    for form in FORMS:
        meth = _method(form, "hllc", de=True)
        blk = B.Block(n, g, w, mhd=False, dual_energy=True)
        blk.load_numpy(s)
        bufs = B.FluxBuffers(blk, (0, 1, 2, 3, 4, 5))
        meth.compute_store_fluxes(blk, 1e-3, buffers=bufs)
        torch.cuda.synchronize()
        out.append((blk.to_numpy(), {k: t.cpu().numpy() for k, t in bufs.arrays.items()}))
    for a, b in zip(*out):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("n", [(380, 350, 14), (410, 400, 9)])
def test_wide_planes(n):
    # the widest planes that the split stages take, in slabs of five planes, and
    # wider ones
    out = []
    for form in FORMS:
        meth = _method(form)
        blk = B.Block(n, 3, (1.0 / 64,) * 3)
        g = torch.Generator(device="cuda")
        g.manual_seed(2)
        for k, t in blk.fields.items():
            r = torch.rand(t.shape, generator=g, dtype=t.dtype, device="cuda")
            t.copy_({"density": 1.0, "total_energy": 4.0}.get(k, 0.0) + 0.3 * r)
        meth.compute(blk, 1e-3)
        torch.cuda.synchronize()
        out.append(blk.fields)
    for k in out[0]:
        assert torch.isfinite(out[0][k]).all(), k
        assert torch.equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("dtype,form,says", [
    (capi.MHD_DTYPE_F64, "split", "split"), (capi.MHD_DTYPE_F64, "fused", "fused"),
    (capi.MHD_DTYPE_F32, "split", "fused")])
def test_autotuner_reports_what_runs(dtype, form, says):
    meth = _method(form)
    n = (12, 10, 9)
    s, w = ic.smooth_block(n, 3, seed=2)
    bt = Batch(meth, [n], [w], dtype=dtype)
    bt.upload(0, s)
    buf = ctypes.create_string_buffer(4096)
    capi.check(capi.lib().mhdvlct_batch_autotune(bt.h, 1, buf, 4096, None), meth.handle, "autotune")
    got = json.loads(buf.value.decode())["12x10x9"]
    for k in ("stage1", "stage2"):
        assert got[k]["form"] == says, got
        tile = got[k]["tile_x"], got[k]["tile_y"]
        if says == "split":
            assert tile == (0, 0) and got[k]["zchunk"] == 0 and got[k]["threads"] == 128, got
        else:
            assert min(tile) >= 1 and (tile[0] + 2) * (tile[1] + 2) <= got[k]["threads"], got
