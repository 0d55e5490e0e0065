"""The range partition's workspace, on the host: the size reserved for a window
serves every shorter window, which is what the windowed join's last window and
a caller with one workspace for batches of uneven size rely on."""
import ctypes

import pytest


def _bytes(gj, m, bits, sms):
    reserved, used = ctypes.c_size_t(0), ctypes.c_size_t(0)
    assert gj.lib().gj_debug_partition_bytes(m, bits, sms, ctypes.byref(reserved), ctypes.byref(used)) == 0
    return reserved.value, used.value


@pytest.mark.parametrize("sms", [1, 7, 152, 160])
@pytest.mark.parametrize("bits", [1, 5, 8, 9, 11, 12])
def test_workspace_serves_shorter_windows(gj, bits, sms):
    # every whole and ragged tile count around the sizes where a chunk takes
    # one more tile and where the tile size changes, and spread beyond them
    edge = 2 * sms * 8192
    sizes = {1, 4095, 4096, 4097, 8192, 8193, edge - 1, edge, edge + 1}
    for k in range(1, 9):
        for tile in (4096, 8192):
            sizes |= {k * 2 * sms * tile + d for d in (-tile, -1, 0, 1, tile, tile + 1)}
    m = 4096
    while m < 1 << 32:
        sizes |= {m, m + 1, m + m // 3}
        m += m // 2
    sizes = sorted(s for s in sizes if 0 < s < 1 << 32)
    most = 0
    for m in sizes:
        reserved, used = _bytes(gj, m, bits, sms)
        most = max(most, used)  # by this window or a shorter one
        assert reserved >= most, (m, reserved, most)


@pytest.mark.parametrize("window,last", [(1_500_000, 1_200_000), (1_300_000, 1_200_000), (5_000_000, 4_900_000),
                                         (10_000_000, 9_950_000)])
@pytest.mark.parametrize("bits", [5, 8, 11])
def test_workspace_serves_the_last_window(gj, window, last, bits):
    assert _bytes(gj, window, bits, 152)[0] >= _bytes(gj, last, bits, 152)[1]
