"""Copy plan of the 8- and 4-byte staged kernels, checked on the CPU.

The library lists the bulk copies of every tile with the line_runs code the
kernels run (imexlb_debug_line_plan, host build).  Every copy must be 16-byte
aligned at both ends and in size and stay inside its population's plane and
its slot; and where a cell reads its slot, the slot must hold the value the
cell pulls (or, beyond a y / z wall, its own opposite population).
"""
import ctypes

import numpy as np
import pytest

from imexlb_b200 import api

E = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
              (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1),
              (0, 1, -1), (0, -1, 1), (1, 1, 1), (-1, -1, -1), (1, -1, 1), (-1, 1, -1), (1, 1, -1), (-1, -1, 1),
              (1, -1, -1), (-1, 1, 1)])
BB = [int(np.where((E == -e).all(1))[0][0]) for e in E]

CAVITY = [(4, 2, 2), (16, 3, 4), (32, 32, 4), (36, 20, 5), (64, 9, 3), (128, 7, 3), (150, 13, 3), (160, 17, 2),
          (300, 5, 3), (1026, 3, 2)]
SPHERE = [(48, 32, 4), (96, 40, 5), (205, 33, 3), (384, 12, 3), (512, 9, 3), (768, 6, 2)]


def line_plan(n, wrap, elem):
    fn = api.load_library().imexlb_debug_line_plan
    fn.restype = ctypes.c_int64
    fn.argtypes = [ctypes.c_int] * 5 + [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64]
    geo = np.zeros(8, dtype=np.int32)
    dummy = np.zeros((1, 6), dtype=np.int32)
    count = fn(*n, wrap, elem, geo.ctypes.data, dummy.ctypes.data, 0)
    if count < 0:
        return None
    runs = np.zeros((count, 6), dtype=np.int32)
    assert fn(*n, wrap, elem, geo.ctypes.data, runs.ctypes.data, count) == count
    return geo.tolist(), runs


@pytest.mark.parametrize("elem", [8, 4])
@pytest.mark.parametrize("n,wrap", [(n, 0) for n in CAVITY] + [(n, 1) for n in SPHERE])
def test_slots_hold_what_cells_pull(n, wrap, elem):
    nx, ny, nz = n
    got = line_plan(n, wrap, elem)
    assert got is not None
    (P, nty, C, G, slot, base, sz, sq), runs = got
    assert P >= nx and C * elem == 2048 and G * elem == 16 and slot == C + 2 * G and nty == -(-P * ny // C)
    assert ((runs[:, 3:] * elem) % 16 == 0).all()
    assert (runs[:, 4] >= 0).all() and (runs[:, 4] + runs[:, 5] <= slot).all()
    assert (runs[:, 3] >= base).all() and (runs[:, 3] + runs[:, 5] <= base + sz * nz).all() and sz * nz <= sq
    start = np.searchsorted(runs[:, 0], np.arange(nty * nz + 1))
    for t in range(nty * nz):
        k, e0 = t // nty, (t % nty) * C
        held = np.full((27, slot), -1, dtype=np.int64)
        for _, q, pop, src, dst, ln in runs[start[t]:start[t + 1]].tolist():
            assert (held[q, dst:dst + ln] == -1).all(), "two copies write one place"
            held[q, dst:dst + ln] = pop * np.int64(1 << 40) + np.arange(src, src + ln)
        e = np.arange(e0, min(e0 + C, P * ny))
        e = e[e % P < nx]
        j, x, at = e // P, e % P, G + (e - e0)
        for q in range(27):
            ex, ey, ez = E[q].tolist()
            sx, sy, sk = x - ex, j - ey, k - ez
            if wrap:
                sx = np.where(sx >= nx, nx - 1, sx)
                want = q * np.int64(1 << 40) + base + (sk % nz) * sz + (sy % ny) * P + sx
                read = at - np.where((x == nx - 1) & (ex < 0), 0, ex)
                check = sx >= 0  # the inlet takes the inflow's equilibrium
            else:
                out = (sy < 0) | (sy >= ny) | (sk < 0) | (sk >= nz)
                own = BB[q] * np.int64(1 << 40) + base + k * sz + e
                want = np.where(out, own, q * np.int64(1 << 40) + base + sk * sz + sy * P + sx)
                read = at - np.where(out, 0, ex)
                check = out | ((sx >= 0) & (sx < nx))  # x walls: loaded apart
            assert (held[q, read[check]] == want[check]).all()
