"""Gridding with lane-owned columns (cg_grid_own.cu) against the oracle's
spreading (the reference's conv_3d_outputdriven_t1, conv.cu:522-627, restated),
where its shapes change: every width (one or two cells a lane, odd and even numbers
of planes in registers), the ES and the learned kernel, short axes and axes that are no
multiple of a hive or a tile, more planes than one item holds, split tiles, strips of
tiles, and more rows in a tile than its shared memory has slots for."""
import numpy as np
import pytest

from cugridder_b200 import Plan, _lib, synth
from cugridder_b200.synth import rel_l2

from tests.gpu_helpers import payload, plan_ms2dirty, to_dev

pytestmark = pytest.mark.gpu


def _grid(torch, oracle, d, precision, eps, kernel=None):
    cdt, rdt = (np.complex128, np.float64) if precision == "fp64" else (np.complex64, np.float32)
    p = Plan(d["nx"], d["ny"], d["fov"], eps, precision=precision)
    if kernel is not None:
        p.set_kernel("poly", kernel.W, kernel.horner)
    dirty = torch.zeros((d["nx"], d["ny"]), dtype=torch.complex128 if precision == "fp64" else torch.complex64,
                        device="cuda")
    p.set_stop_stage(2)
    p.ms2dirty(to_dev(torch, d["uvw"]), d["freq"], to_dev(torch, d["vis"], cdt), to_dev(torch, d["wgt"], rdt), dirty)
    torch.cuda.synchronize()
    info = p.info()
    got = p.copy_buffer(_lib.CG_BUF_GRID)
    p.close()
    if kernel is not None:  # the kernel's width sets the geometry (nw) too
        oracle.set_kernel("poly", kernel.W, kernel.horner)
    try:
        o = oracle.setup(d["uvw"], d["nx"], d["ny"], d["fov"], d["freq"], eps,
                         eps_floor=1.1e-16 if precision == "fp64" else 6e-8)
        return got, oracle.grid(o, oracle.grid_coords(o, d["uvw"]), payload(d, o)), info
    finally:
        if kernel is not None:
            oracle.set_kernel("es")


# FP64 1e-12 as in the other gridding tests.  FP32: a tap is the product of three
# values exp(beta sqrt(1 - t^2)), beta = 2.3 W, whose arguments are rounded to 2^-24
# of up to beta, so each is off by up to beta 2^-24 and some units of rounding:
# 3 (beta + 8) 2^-24.
@pytest.mark.parametrize("precision,eps,W", [("fp64", 5e-1, 2), ("fp64", 5e-2, 3), ("fp64", 5e-8, 9), ("fp64", 5e-9, 10),
                                             ("fp64", 5e-10, 11), ("fp64", 5e-12, 13), ("fp64", 5e-15, 16),
                                             ("fp32", 5e-1, 2), ("fp32", 5e-2, 3), ("fp32", 6e-8, 9)])
def test_widths_with_wrap(torch_cuda, oracle, precision, eps, W):
    d = synth.wrap_case(6000, 50, 72, 3.0, seed=W)
    got, ref, info = _grid(torch_cuda, oracle, d, precision, eps)
    assert info["kw"] == W
    assert rel_l2(got, ref) < (1e-12 if precision == "fp64" else 3 * (2.3 * W + 8) * 2.0 ** -24)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("eps", [1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
def test_widths_at_the_centre(torch_cuda, oracle, precision, tol, eps):
    """W = 4..8 on the 256^2 case (rows near the grid centre)."""
    d = synth.make("ms2dirty_256_fp64", seed=23, nrow=30000)
    got, ref, info = _grid(torch_cuda, oracle, d, precision, eps)
    assert 4 <= info["kw"] <= 8
    assert rel_l2(got, ref) < tol


@pytest.mark.parametrize("W", [5, 6, 8])
def test_learned_kernel(torch_cuda, oracle, W):
    from cugridder_b200.learn import available_widths, load_kernel

    if W not in available_widths():
        pytest.skip("no learned kernel of width %d" % W)
    d = synth.wrap_case(20000, 128, 128, 2.0, seed=W)
    got, ref, info = _grid(torch_cuda, oracle, d, "fp32", 1e-5, kernel=load_kernel(W))
    assert info["kw"] == W
    assert rel_l2(got, ref) < 2e-6


@pytest.mark.parametrize("strip", ["0", "1"])
@pytest.mark.parametrize("precision,eps,tol", [("fp64", 1e-5, 1e-12), ("fp64", 1e-6, 1e-12), ("fp64", 1e-9, 1e-12),
                                              ("fp32", 1e-3, 2e-6), ("fp32", 1e-6, 2e-6)])
@pytest.mark.parametrize("shape", [(96, 160), (122, 96), (8, 32), (50, 8)])
def test_tiles_and_strips(torch_cuda, oracle, monkeypatch, strip, precision, eps, tol, shape):
    """Rows over the whole band and past it, tiles one at a time and in strips of four:
    axes of whole tiles (192 x 320), of 250 cells (a partial last tile and hive), of 16
    or 20 cells (a tile next to its own image), a strip that its rows fill and tiles
    that hold more than a chunk."""
    monkeypatch.setenv("CG_GRID_STRIP", strip)
    d = synth.wrap_case(2500, shape[0], shape[1], 3.0, seed=sum(shape))
    d["uvw"][:500, :2] *= 0.05
    got, ref, _ = _grid(torch_cuda, oracle, d, precision, eps)
    assert rel_l2(got, ref) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 2e-5)])
def test_end_to_end(torch_cuda, oracle, precision, tol):
    d = synth.wrap_case(30000, 128, 96, 3.0, seed=77)
    _, dirty, st = plan_ms2dirty(torch_cuda, d, precision, 1e-6)
    assert st == 0
    ref, _ = oracle.ms2dirty(d["uvw"], d["vis"], d["wgt"], 128, 96, d["fov"], d["freq"], 1e-6)
    assert rel_l2(dirty, ref) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("split_rows", [None, "300", "1"])
@pytest.mark.parametrize("strip", ["0", "1"])
def test_plane_batches(torch_cuda, oracle, monkeypatch, precision, tol, split_rows, strip):
    """More than 48 planes: an item holds a batch of them, the last batch fewer; whole,
    with the heavy tiles of a batch as chunks, and with every tile that has rows."""
    if split_rows is not None:
        monkeypatch.setenv("CG_SPLIT_ROWS", split_rows)
    monkeypatch.setenv("CG_GRID_STRIP", strip)
    d = synth.wrap_case(8000, 48, 48, 8.0, seed=3, w_frac=23.0)
    d["uvw"][:3000, :2] *= 0.1
    got, ref, info = _grid(torch_cuda, oracle, d, precision, 1e-5)
    assert info["nw"] > 48 and info["nw"] % -(-info["nw"] // 48)  # nw = 100: batches of 34, 34 and 32
    assert rel_l2(got, ref) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("split", ["0", "1"])
def test_every_candidate_reaches_the_tile(torch_cuda, oracle, monkeypatch, precision, tol, split):
    """All rows within a few cells of the centre of a tile: every candidate of a
    chunk reaches it, more than it has row slots."""
    monkeypatch.setenv("CG_SPLIT", split)
    d = synth.wrap_case(20000, 64, 64, 3.0, seed=5, reach=0.04, w_frac=0.3)
    pix = np.deg2rad(3.0) / 64
    d["uvw"][:, :2] += 8.0 / (128 * pix) * synth.C_LIGHT / d["freq"]  # 8 cells on: the middle of a tile
    got, ref, _ = _grid(torch_cuda, oracle, d, precision, 1e-5)
    assert rel_l2(got, ref) < tol


@pytest.mark.parametrize("eps,W", [(5e-8, 9), (5e-9, 10)])
@pytest.mark.parametrize("shape", [(8, 32), (32, 8), (8, 8)])
def test_short_axes(torch_cuda, oracle, shape, eps, W):
    """Axes of 18 and 20 cells: a tile of 16 and one of 2 or 4, so that the first
    tile's halo goes round the grid both ways (6 hive rows at 18)."""
    d = synth.wrap_case(3000, shape[0], shape[1], 3.0, seed=W)
    got, ref, info = _grid(torch_cuda, oracle, d, "fp64", eps)
    assert info["kw"] == W and 2 * W in (info["nf1"], info["nf2"])
    assert rel_l2(got, ref) < 1e-12
