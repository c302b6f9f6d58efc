"""GPU: one lattice, several step kernels, the same bits.

The form a step takes depends on the lattice's size, storage and row width
(imexlb_debug_step_form); every form's cells go through the same arithmetic.

* Cavities start at rest and one step carries a value one cell, so after s steps
  a cell more than s away from the y walls equals the middle of a smaller cavity
  of the same rows, and below the lid's reach everything is still at rest.  Every
  cell of a large cavity is compared with the small one, whose step runs in
  blocks across row ends.
* Spheres and vortices are compared with an engine of one instance, whose
  register kernels share nothing with the staged ones but the arithmetic.

EXACT FP64, FP32 and the pair kernels name every rounding, so their bits are
equal.  FAST FP64 leaves the contraction of multiply and add to the compiler,
kernel by kernel: each of the 27 populations, of magnitude 8/27 at most around
rest, may differ by a rounding (2^-53) or two a step, so u, v, w, p after s steps
by s 27 2^-52.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ITEMS, ROWS, LINE, STAGED, BOX = range(5)
S = 6


@pytest.fixture(scope="module")
def api():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from imexlb_b200 import api as a

    return a


def form(api, case, storage, arith, n):
    return api.load_library().imexlb_debug_step_form(api.CASES[case], api.STORAGES[storage], api.ARITHS[arith], *n)


def run(api, case, n, storage, arith, steps=S, **kw):
    with api.LBM(case, *n, 0.07, 1.0, 0.05, bc="standard", storage=storage, arith=arith, **kw) as lbm:
        lbm.step(steps)
        return lbm.fields()


def same(got, want, storage, arith, what):
    if storage == "f64" and arith == "fast":
        assert np.abs(got - want).max() <= S * 27 * 2.0**-52, what
    else:
        assert np.array_equal(got, want), what


# (the last tile of a plane: full, some cells, most of one; planes of less than a
# tile; several tiles a row; padded rows; one row a warp; half a warp of pairs)
@pytest.mark.parametrize("n,storage,arith,want", [
    ((128, 84, 90), "f64", "fast", LINE), ((151, 97, 66), "f64", "fast", LINE), ((112, 2, 4300), "f64", "fast", LINE),
    ((272, 57, 62), "f64", "fast", LINE), ((600, 41, 40), "f64", "fast", LINE), ((80, 75, 77), "f32", "fast", LINE),
    ((112, 4, 1010), "f32", "fast", LINE), ((64, 129, 64), "f32", "fast", LINE), ((1030, 22, 20), "f32", "fast", LINE),
    ((100, 71, 68), "f32", "fast", LINE), ((26, 130, 160), "f32", "fast", LINE), ((18, 130, 120), "f32", "fast", BOX),
    ((20, 64, 64), "f32", "fast", BOX), ((27, 130, 120), "f32", "fast", BOX), ((17, 150, 90), "f64", "fast", BOX),
    ((27, 111, 80), "f64", "exact", BOX), ((31, 100, 90), "f64", "exact", BOX), ((64, 70, 60), "f64", "exact", ROWS),
    ((100, 80, 70), "f64", "exact", ITEMS)])
def test_large_cavity_equals_a_small_one(api, n, storage, arith, want):
    nx, ny, nz = n
    assert form(api, "cavity", storage, arith, n) == want
    # (as odd or even as ny: the FP32 one-cell kernel takes rows in pairs, an odd last one alone)
    small = (nx, min(ny, 2 * S + 3 + (ny + 1) % 2), 2 * S + 3)
    a = run(api, "cavity", small, storage, arith, lid_u=0.05)
    b = run(api, "cavity", n, storage, arith, lid_u=0.05)
    assert form(api, "cavity", storage, arith, small) in (ITEMS, ROWS)
    rows = np.array([j if j <= S + 1 else max(S + 1, small[1] - (ny - j)) for j in range(ny)]) if ny > small[1] else \
        np.arange(ny)
    planes = np.array([max(0, small[2] - (nz - k)) for k in range(nz)])
    planes = np.where(planes <= S + 1, np.where(np.arange(nz) <= S + 1, np.arange(nz), S + 1), planes)
    assert small[2] - 1 in planes
    for k in "uvwp":
        same(b[k], a[k][planes][:, rows], storage, arith, k)


@pytest.mark.parametrize("n,storage,arith,want", [
    ((130, 61, 58), "f64", "exact", LINE), ((130, 61, 58), "f64", "fast", LINE), ((96, 6, 850), "f64", "exact", LINE),
    ((130, 61, 58), "f32", "fast", LINE), ((206, 51, 47), "f32", "fast", LINE), ((128, 9, 400), "f32", "fast", LINE),
    ((303, 40, 38), "f64", "fast", LINE), ((768, 33, 20), "f32", "fast", LINE)])
@pytest.mark.parametrize("body", ["middle", "across y and z"])
def test_sphere_equals_an_engine_instance(api, n, storage, arith, want, body):
    assert form(api, "sphere", storage, arith, n) == want
    kw = dict(inlet_u=0.05, sphere_d=5.0)
    kw["sphere_c"] = (30.3, n[1] / 2, n[2] / 2) if body == "middle" else (30.3, 0.4, n[2] - 0.7)
    got = run(api, "sphere", n, storage, arith, **kw)
    with api.LBM("sphere", *n, 0.07, 1.0, 0.05, bc="standard", storage=storage, arith=arith, **kw) as lbm:
        for _ in range(S):
            lbm.step(1)  # every step sums its drag: the register kernel
        single = lbm.fields()
    want_f = engine(api, "sphere", n, storage, arith, **kw)
    for k in "uvwp":
        same(got[k], want_f[k], storage, arith, k)
        same(single[k], got[k], storage, arith, k)


@pytest.mark.parametrize("n,storage,arith,want", [
    ((18, 130, 120), "f32", "fast", BOX), ((9, 200, 200), "f32", "fast", BOX), ((41, 150, 140), "f32", "fast", BOX),
    ((110, 130, 40), "f32", "fast", BOX), ((17, 150, 90), "f64", "exact", BOX), ((24, 130, 70), "f64", "fast", BOX),
    ((55, 91, 41), "f64", "fast", BOX), ((125, 91, 80), "f16", "fast", BOX), ((55, 130, 121), "bf16", "fast", BOX),
    ((41, 31, 33), "f32", "fast", ITEMS)])
def test_vortex_equals_an_engine_instance(api, n, storage, arith, want):
    assert form(api, "tgv", storage, arith, n) == want
    got, want_f = run(api, "tgv", n, storage, arith), engine(api, "tgv", n, storage, arith)
    for k in "uvwp":
        same(got[k], want_f[k], storage, arith, k)


def engine(api, case, n, storage, arith, **kw):
    d = api.instance_desc(case, *n, 0.07, 1.0, 0.05, **kw)
    with api.Engine(storage=storage, arith=arith, budget_bytes=api.instance_bytes(storage, d) + (64 << 20),
                    max_instances=1) as eng:
        slot = eng.add(d)
        eng.step(S)
        return eng.fields(slot)


PAIRS = [(("cavity", (128, 84, 90), "f64"), ("sphere", (206, 50, 47), "f32")),
         (("tgv", (128, 128, 112), "f16"), ("cavity", (80, 75, 77), "f32")),
         (("sphere", (256, 90, 84), "bf16"), ("cavity", (128, 96, 100), "f16"))]


@pytest.mark.parametrize("pair", PAIRS)
def test_two_lattices_at_once_on_two_streams(api, pair):
    """Neither grid is wholly resident then; nothing waits for a block that is not there."""
    import torch

    want = [run(api, c, n, st, "fast", steps=200) for c, n, st in pair]
    got = [None, None]
    streams = [torch.cuda.Stream() for _ in pair]

    def work(i):
        c, n, st = pair[i]
        got[i] = run(api, c, n, st, "fast", steps=200, stream=streams[i].cuda_stream)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, w in zip(got, want):
        for k in "uvwp":
            assert np.array_equal(g[k], w[k]), k


@pytest.mark.parametrize("case,n,storage", [("cavity", (32, 32, 32), "f64"), ("cavity", (128, 84, 90), "f64"),
                                            ("sphere", (206, 50, 47), "f32"), ("tgv", (128, 128, 112), "f16"),
                                            ("tgv", (18, 130, 120), "f32")])
def test_captured_steps_replay(api, case, n, storage):
    import torch

    kw = dict(bc="standard", storage=storage, arith="fast")
    side = torch.cuda.Stream()
    with api.LBM(case, *n, 0.07, 1.0, 0.05, stream=side.cuda_stream, **kw) as lbm:
        lbm.step(2)
        lbm.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            lbm.step(2)
        with torch.cuda.stream(side):
            for _ in range(3):
                g.replay()
        side.synchronize()
        got = lbm.fields()
        del g
    with api.LBM(case, *n, 0.07, 1.0, 0.05, **kw) as lbm:
        lbm.step(8)
        want = lbm.fields()
    for k in "uvwp":
        assert np.array_equal(got[k], want[k]), k
