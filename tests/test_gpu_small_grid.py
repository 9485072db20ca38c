"""The no-allocation photon grid against numpy's stable sort, at the sizes where its kernels change their path:
cells of 1, 2, 32, 64, 128, 256 and 257 photons, a cell with more photons than a slot's word has room for their
rank, slot counts around a block's and a bitmap row's, grids around the scan's tile, odd alignments, no photon."""
import ctypes as C

import numpy as np
import pytest

import rustracer_gb300 as rt
from rustracer_gb300 import _abi as A

pytestmark = pytest.mark.gpu

# (slots, cells along x, y, z, photons put into chosen cells: (cell, count), byte offset of meta)
CASES = [
    (0, (3, 1, 1), [], 0),
    (1, (1, 1, 1), [(0, 1)], 0),
    (1023, (8, 8, 8), [(0, 32), (1, 33), (7, 64), (8, 65), (511, 128)], 4),
    (1025, (13, 11, 15), [(5, 256), (2144, 257)], 0),
    (32_769, (16, 16, 8), [(2047, 16_381), (3, 2)], 0),
    (40_000, (17, 11, 11), [(11, 16_382), (2056, 16_383)], 4),
    (100_003, (2, 2, 2), [(6, 70_000)], 0),
    ((1 << 20) - 1, (64, 64, 64), [(262_143, 20_000), (0, 300)], 0),
    (1 << 20, (64, 64, 64), [(77, 1 << 20)], 0),
]


@pytest.mark.parametrize("slots,dims,crowds,offset", CASES)
def test_small_grid_is_a_stable_sort_by_cell(gpu, slots, dims, crowds, offset):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(slots + dims[0])
    cells = dims[0] * dims[1] * dims[2]
    gp = A.GridParams()
    gp.grid_x, gp.grid_y, gp.grid_z, gp.num_cells, gp.photon_slots, gp.cell_size = *dims, cells, slots, 1.0
    # every slot a cell, in random order; a fifth of the others empty
    cell = rng.integers(0, cells, slots)
    power = np.where(rng.random(slots) < 0.2, 0.0, 1.0).astype(np.float32)
    free = rng.permutation(slots)
    for c, n in crowds:
        take, free = free[:n], free[n:]
        cell[take], power[take] = c, 1.0
    ph = rng.random((slots, 16), np.float32)
    ph[:, 4] = power
    ph[:, 0] = cell % dims[0] + 0.5
    ph[:, 1] = cell // dims[0] % dims[1] + 0.5
    ph[:, 2] = cell // (dims[0] * dims[1]) + 0.5
    kept = np.flatnonzero(power > 0)
    order = kept[np.argsort(cell[kept], kind="stable")]
    counts = np.bincount(cell[kept], minlength=cells)

    dev = torch.device("cuda")
    d_ph = torch.from_numpy(ph).to(dev)
    d_counts = torch.full((cells,), -1, dtype=torch.int32, device=dev)
    d_meta = torch.full((2 * cells + 2,), -1, dtype=torch.int32, device=dev)
    d_sorted = torch.full((max(slots, 1), 16), -1.0, device=dev)
    for _ in range(2):  # the second call finds what the first left in the scratch
        A.check("noalloc", A.load().rt_stage_photon_grid_noalloc(
            C.c_void_p(d_ph.data_ptr()), C.byref(gp), C.c_void_p(d_counts.data_ptr()),
            C.c_void_p(d_meta.data_ptr() + offset), C.c_void_p(d_sorted.data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
        assert np.array_equal(d_counts.cpu().numpy(), counts)
        meta = d_meta.cpu().numpy()[offset // 4: offset // 4 + 2 * cells].reshape(-1, 2)
        assert np.array_equal(meta[:, 1], counts)
        assert np.array_equal(meta[:, 0], np.cumsum(counts) - counts)
        out = d_sorted.cpu().numpy()
        assert np.array_equal(out[: len(order)], ph[order])
        assert (out[len(order):] == -1.0).all()
    assert A.load().rt_scan_timeouts() == 0
