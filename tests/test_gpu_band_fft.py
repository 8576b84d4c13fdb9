"""Band-pruned transforms (cg_fft_band.cu) against cuFFT's full 2-D transform
(CG_FFT_PRUNE=0) through both directions: lengths of every radix, FP32 and FP64,
data in a narrow band (columns, and rows of 8192 cells, as two half-length
transforms), over most of the grid (where FP32 columns of 4096 and 8192 cells take the
other kernels) and around its edge (whole columns, periodic windows), non-square
images."""
import os

import numpy as np
import pytest

from cugridder_b200 import Plan, synth
from cugridder_b200.synth import rel_l2

from tests.gpu_helpers import to_dev

pytestmark = pytest.mark.gpu


def _run(torch, d, img, precision, prune):
    cdt, rdt = (np.complex128, np.float64) if precision == "fp64" else (np.complex64, np.float32)
    tdt = torch.complex128 if precision == "fp64" else torch.complex64
    os.environ["CG_FFT_PRUNE"] = prune
    try:
        p = Plan(d["nx"], d["ny"], d["fov"], 1e-4, precision=precision)
    finally:
        del os.environ["CG_FFT_PRUNE"]
    uvw, wgt = to_dev(torch, d["uvw"]), to_dev(torch, d["wgt"], rdt)
    dirty = torch.zeros((d["nx"], d["ny"]), dtype=tdt, device="cuda")
    vis = torch.zeros(d["uvw"].shape[0], dtype=tdt, device="cuda")
    p.ms2dirty(uvw, d["freq"], to_dev(torch, d["vis"], cdt), wgt, dirty)
    p.dirty2ms(uvw, d["freq"], to_dev(torch, img, cdt), wgt, vis)
    torch.cuda.synchronize()
    info = p.info()
    p.close()
    return dirty.cpu().numpy(), vis.cpu().numpy(), info


# image sizes whose grids (twice as long) and half grids take radices 2 to 16
@pytest.mark.parametrize("nx,ny", [(32, 64), (48, 40), (50, 90), (54, 162), (96, 80), (108, 150), (128, 250),
                                   (270, 192), (450, 512), (1250, 60), (60, 4096), (4096, 60), (2048, 64)])
@pytest.mark.parametrize("reach", [0.3, 0.8, 1.2])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_matches_full_transform(torch_cuda, nx, ny, reach, precision):
    d = synth.wrap_case(3000, nx, ny, 2.0, seed=nx + ny, reach=reach, w_frac=0.05)
    img = synth.random_image(nx, ny, seed=1)
    a = _run(torch_cuda, d, img, precision, "1")
    b = _run(torch_cuda, d, img, precision, "0")
    assert a[2]["nf1"] >= 2 * ny and a[2]["nf2"] >= 2 * nx
    # rounding of a transform of n points: some log2(n) units in the last place
    tol = 1e-14 if precision == "fp64" else 2e-6
    assert rel_l2(a[0], b[0]) < tol
    assert rel_l2(a[1], b[1]) < tol


def test_tables_count_as_workspace(torch_cuda):
    """The first dirty2ms after an ms2dirty on the same uvw needs nothing new but the
    forward transforms' tables; the plan reports them."""
    d = synth.wrap_case(3000, 96, 80, 2.0, seed=2, reach=0.3, w_frac=0.05)
    p = Plan(96, 80, 2.0, 1e-9, precision="fp64")
    uvw, wgt = to_dev(torch_cuda, d["uvw"]), to_dev(torch_cuda, d["wgt"])
    dirty = torch_cuda.zeros((96, 80), dtype=torch_cuda.complex128, device="cuda")
    vis = to_dev(torch_cuda, d["vis"])
    p.ms2dirty(uvw, d["freq"], vis, wgt, dirty)
    before, info = p.info()["workspace_bytes"], p.info()
    p.dirty2ms(uvw, d["freq"], dirty, wgt, vis)
    torch_cuda.cuda.synchronize()
    # e^{2 pi i x / L} alone: 16 bytes a cell of each axis
    assert p.info()["workspace_bytes"] - before >= 16 * (info["nf1"] + info["nf2"])
    p.close()
