"""Binning at the row counts where its sort changes shape: one row, the edges of
a tile, the count up to which tiles hold 2048 rows, the counters up to which one block
scans them (32 tiles of 4096 rows); grids on both sides of the hive count up to
which offsets come from a search."""
import numpy as np
import pytest

from cugridder_b200 import Plan, _lib, synth

from tests.gpu_helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 1500])
@pytest.mark.parametrize("nrow", [1, 2047, 2048, 2049, 40960, 40961, 131072, 131073])
def test_stable_order_and_offsets(torch_cuda, nrow, n):
    torch = torch_cuda
    d = synth.wrap_case(nrow, n, n, 3.0, seed=nrow % 97)
    p = Plan(n, n, 3.0, 1e-4, precision="fp32")
    p.set_stop_stage(1)
    p.ms2dirty(to_dev(torch, d["uvw"]), d["freq"], to_dev(torch, d["vis"], np.complex64), None,
               torch.zeros((n, n), dtype=torch.complex64, device="cuda"))
    torch.cuda.synchronize()
    perm, keys = p.copy_buffer(_lib.CG_BUF_PERM), p.copy_buffer(_lib.CG_BUF_SORTED_KEYS)
    hs, nh = p.copy_buffer(_lib.CG_BUF_HIVE_START), p.info()["nhive"]
    p.close()
    row_keys = np.empty(nrow, np.int64)
    row_keys[perm] = keys  # also: perm is a permutation
    assert np.array_equal(np.sort(perm), np.arange(nrow))
    assert np.array_equal(perm, np.argsort(row_keys, kind="stable"))
    assert np.array_equal(hs, np.searchsorted(keys, 64 * np.arange(np.prod(nh) + 1, dtype=np.int64)))
