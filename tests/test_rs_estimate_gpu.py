"""The RadixSpline's position estimate against exact rational arithmetic over
its segments: no fewer bits than the double slope and product it stands for."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from test_lookup_gpu import column, from_dev_u32, to_dev

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "drop_in", "rs_estimate.cu")


def build(tmpdir):
    import gpujoin_gb300
    from gpujoin_gb300 import build as gbuild

    gpujoin_gb300.lib()
    out = os.path.join(str(tmpdir), "librsest.so")
    libdir = os.path.dirname(gpujoin_gb300.LIB_PATH)
    r = subprocess.run([gbuild.nvcc(), *gbuild.ARCH, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                        os.path.join(ROOT, "include"), SRC, "-o", out, "-L", libdir, "-lgpujoin", "-Xlinker", "-rpath",
                        "-Xlinker", libdir], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(out)


def test_estimate_compiles(tmp_path, gj):
    assert build(tmp_path).rs_estimates is not None


@pytest.mark.gpu
@pytest.mark.parametrize("max_error", [0, 4, 32])
@pytest.mark.parametrize("case", ["uniform", "wide", "dense", "runs", "two"])
def test_estimate_is_the_segment_line_rounded_down(tmp_path, orc, gj, cuda, case, max_error):
    import torch

    rng = np.random.default_rng(len(case))
    if case == "two":
        col = np.array([3, (1 << 64) - 2], dtype=np.uint64)  # one segment over nearly all keys
    elif case == "dense":
        col = np.arange(1000, 1000 + 70_001, dtype=np.uint64)
    elif case == "runs":
        starts = np.sort(rng.choice(1 << 40, size=300, replace=False).astype(np.uint64)) << np.uint64(20)
        col = np.unique(np.concatenate([s + np.arange(200, dtype=np.uint64) * np.uint64(5) for s in starts]))
    else:
        col = column(rng, 70_001, upper=1 << (63 if case == "wide" else 40))
    _, sx, sy, _ = orc.RadixSpline(col, 18, max_error).arrays()
    keys = np.concatenate([rng.integers(col[0], col[-1], 20_000, dtype=np.uint64), col[rng.integers(0, len(col), 20_000)],
                           sx[1:] - np.uint64(1), sx + np.uint64(1)])
    keys = np.unique(keys[(keys > col[0]) & (keys < col[-1])])
    ix = gj.make_index("radix_spline", rs_max_error=max_error).construct(None, to_dev(torch, col))
    lib = build(tmp_path)
    lib.rs_estimates.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_void_p]
    est = torch.empty(len(keys), dtype=torch.int32, device="cuda")
    rate = torch.empty(len(keys), dtype=torch.float32, device="cuda")
    d_keys = to_dev(torch, keys)
    assert lib.rs_estimates(ix.handle, d_keys.data_ptr(), len(keys), est.data_ptr(), rate.data_ptr()) == 0
    got, rates = from_dev_u32(est), rate.cpu().numpy()
    at = np.searchsorted(sx, keys, side="left")
    step = max(1, len(keys) // 4000)
    for i in range(0, len(keys), step):
        x0, x1, y0, y1 = (int(sx[at[i] - 1]), int(sx[at[i]]), int(sy[at[i] - 1]), int(sy[at[i]]))
        slope = Fraction(y1 - y0, x1 - x0)
        lost = y0 + slope * (int(keys[i]) - x0) - int(got[i])
        # rounded down to a whole position from a value less than 2^-30 low
        assert 0 <= lost < 1 + Fraction(1, 1 << 30), (i, float(lost))
        assert abs(rates[i] - float(slope) * 0.25) <= float(slope) * 0.25 * 2.0**-23  # one float rounding
