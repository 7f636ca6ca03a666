"""The cell-centred B of the layer around the region that the final stage
updates: after a step it is the mean of the block's own faces, exactly, on every
cell that is at least S cells from the edge of the block, whatever tiles the
stage was cut into; and the FP64 no-allocation step (fused kernel, ring kernel)
leaves the same fields, ghosts included, as the split kernels."""
import ctypes

import numpy as np
import pytest
import torch

from mhdvlct import block as B, capi, ic

pytestmark = pytest.mark.gpu


def _block(n, dtype, seed):
    s, w = ic.smooth_block(n, 3, seed=seed, mhd=True)
    b = B.Block(n, 3, w, dtype=dtype)
    b.load_numpy(s)
    return b


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("recon,stale", [("plm", 2), ("nn", 1)])
@pytest.mark.parametrize("n", [(1, 1, 1), (3, 17, 5), (42, 9, 11), (33, 34, 16)])
def test_centred_b_is_the_mean_of_the_faces(dtype, recon, stale, n):
    meth = B.EnzoMethodMHDVlct(reconstruct_method=recon)
    b = _block(n, dtype, 31)
    meth.compute(b, 1e-3)
    torch.cuda.synchronize()
    f = b.to_numpy()
    half = np.float32(0.5) if dtype == torch.float32 else 0.5
    for k, name in enumerate("xyz"):
        face = f[f"bfieldi_{name}"]
        ax = 2 - k
        lo = np.take(face, range(face.shape[ax] - 1), ax)
        hi = np.take(face, range(1, face.shape[ax]), ax)
        in_ = tuple(slice(stale, m - stale) for m in f["density"].shape)
        assert np.array_equal(f[f"bfield_{name}"][in_], (half * (lo + hi))[in_]), name


@pytest.mark.parametrize("n", [(1, 1, 1), (3, 17, 5), (24, 9, 11)])
def test_no_alloc_step_leaves_the_same_fields(n):
    meth = B.EnzoMethodMHDVlct()
    a, b = _block(n, torch.float64, 32), _block(n, torch.float64, 32)
    meth.compute(a, 1e-3)
    v = b.view()
    capi.check(capi.lib().mhdvlct_block_step_noalloc(meth.handle, ctypes.byref(v), 1e-3, None),
               meth.handle, "no-alloc step")
    torch.cuda.synchronize()
    x, y = a.to_numpy(), b.to_numpy()
    for k in x:
        assert np.array_equal(x[k], y[k]), k
