"""The quantizers that also clear maxima refuse memory for them that they read or write otherwise, before anything is launched."""
import pytest
import torch

MB = 1 << 20


def _rms(L, clear, n):      # 130 x 1024, KE 64
    return L.arcq_rmsnorm_quantize_x_clear(MB, 2 * MB, 1e-5, 3 * MB, 130, 1024, 64, 4 * MB, 5 * MB, clear, n, None)


def _grouped(L, clear, n, row_map=4 * MB):      # three runs of 1024 channels, 512 rows
    return L.arcq_quantize_x_grouped_amax_clear(MB, row_map, 5 * MB, 6 * MB, 7 * MB, 3, 512, 1024, 64, 16, 8 * MB, 9 * MB, 10 * MB, clear, n, None)


# (extents: x, gain, order, codes, two scale tiles of 17 atoms)
RMS = [(MB, 130 * 2048), (2 * MB, 2048), (3 * MB, 2048), (4 * MB, 130 * 544), (5 * MB, 2 * 17 * 512)]
# (row map, maxima, orders, run table, codes, four scale tiles, scales)
GROUPED = [(4 * MB, 2048), (5 * MB, 12), (6 * MB, 6144), (7 * MB, 24), (8 * MB, 512 * 544), (9 * MB, 4 * 17 * 512), (10 * MB, 12)]


@pytest.mark.parametrize("n", [1, 3, 64])
def test_overlaps_are_refused(n):
    from arcquant_b200 import _lib

    L = _lib.load()
    for call, extents in ((_rms, RMS), (_grouped, GROUPED)):
        for at, size in extents:
            for clear in (at - 4 * n + 4, at, at + (size - 4) // 4 * 4):
                assert call(L, clear, n) == _lib.ERR_OVERLAP, (call.__name__, hex(clear))
    assert _grouped(L, MB + 512 * 2048 - 4, n, row_map=None) == _lib.ERR_OVERLAP
    assert b"overlap" in L.arcq_status_string(_lib.ERR_OVERLAP)


@pytest.mark.skipif(torch.cuda.is_available(), reason="the addresses are made up: only without a device does nothing run")
@pytest.mark.parametrize("n", [1, 3, 64])
def test_neighbours_are_not(n):
    from arcquant_b200 import _lib

    L = _lib.load()
    for call, extents in ((_rms, RMS), (_grouped, GROUPED)):
        for at, size in extents:
            for clear in (at - 4 * n, at + size):
                assert call(L, clear, n) == _lib.ERR_CUDA, (call.__name__, hex(clear))
    assert _grouped(L, MB, n) == _lib.ERR_CUDA                       # (x behind a row map: its extent is not known)
    assert _rms(L, None, 0) == _lib.ERR_CUDA
