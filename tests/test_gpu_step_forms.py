"""GPU: the forms a single-lattice step takes by size, at their edges.

A step runs in blocks across rows, by rows, staged in shared memory (8- and
4-byte formats, from 450,000 cells on), or staged with tiles handed out by
tickets (2-byte vortex and sphere).  FP64 EXACT has to equal the CPU
specification bit for bit in each; the 2-byte forms have to equal an engine
instance of the same lattice, whose kernels deal out their tiles in equal
shares.  FP32 is compared with FP64: one step rounds every population twice
to 2^-24 of at most 8/27 around rest, so after n steps the fields are within
n 27 2^-23 of FP64 absolutely (u, v, w, p are sums of the 27).
"""
import numpy as np
import pytest

from oracle.bindings import OracleStd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from imexlb_b200 import api as a

    return a


# odd rows with padding, a plane of less than a tile's line, a last tile of a
# few cells, one row a block, several blocks a row
FORMS = [("cavity", (77, 75, 79)), ("cavity", (96, 64, 75)), ("cavity", (600, 31, 25)), ("cavity", (64, 33, 20)),
         ("cavity", (33, 128, 110)), ("sphere", (130, 61, 58)), ("sphere", (303, 40, 38)), ("cavity", (5, 7, 9))]


@pytest.mark.parametrize("case,n", FORMS)
def test_exact_equals_the_specification(api, case, n):
    kw = dict(lid_u=0.05) if case == "cavity" else dict(inlet_u=0.05, sphere_d=9.0, sphere_c=(n[0] - 20.0, 2.0, 7.5))
    o = OracleStd(case, *n, 0.07, 1.0, 0.05, **kw)
    with api.LBM(case, *n, 0.07, 1.0, 0.05, bc="standard", storage="f64", arith="exact", **kw) as lbm:
        for steps in (1, 4):
            o.step(steps)
            lbm.step(steps)
            got = lbm.fields()
            for name, want in zip("uvwp", o.moments()):
                assert np.array_equal(got[name], want), name


@pytest.mark.parametrize("case,n", [("cavity", (80, 75, 77)), ("cavity", (78, 81, 75)), ("sphere", (130, 61, 58)),
                                    ("sphere", (206, 50, 47))])
def test_fp32_follows_fp64(api, case, n):
    steps = 6
    f = {}
    for st in ("f64", "f32"):
        with api.LBM(case, *n, 0.07, 1.0, 0.05, bc="standard", storage=st, arith="fast") as lbm:
            lbm.step(steps)
            f[st] = lbm.fields()
    for k in "uvwp":
        assert np.abs(f["f32"][k] - f["f64"][k]).max() <= steps * 27 * 2.0**-23, k


@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("case,n", [("tgv", (128, 128, 112)), ("tgv", (90, 121, 230)), ("sphere", (256, 90, 84)),
                                    ("sphere", (512, 62, 60))])
def test_two_byte_tickets_equal_equal_shares(api, case, n, storage):
    with api.LBM(case, *n, 0.07, 1.0, 0.05, bc="standard", storage=storage) as lbm:
        lbm.step(7)
        want = lbm.fields()
    d = api.instance_desc(case, *n, 0.07, 1.0, 0.05)
    with api.Engine(storage=storage, budget_bytes=api.instance_bytes(storage, d) + (64 << 20), max_instances=1) as eng:
        slot = eng.add(d)
        eng.step(7)
        got = eng.fields(slot)
    for k in "uvwp":
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("storage", ["f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("case,n", [("cavity", (24, 20, 18)), ("cavity", (65, 40, 18)), ("sphere", (96, 32, 36))])
def test_queued_steps_equal_steps_waited_for(api, case, n, storage):
    with api.LBM(case, *n, 0.3, 1.0, 0.05, bc="reference", storage=storage, arith="fast") as lbm:
        for _ in range(30):
            lbm.step(1)
            lbm.synchronize()
        want = lbm.fields()
        lbm.Initialize()
        lbm.step(30)
        got = lbm.fields()
    for k in "uvwp":
        assert np.array_equal(got[k], want[k], equal_nan=True), k


def test_face_layers_of_a_tall_cavity(api):
    """Per-link reference cavities of almost as many planes as a grid has
    rows: three steps of a column that starts at rest are the same at either
    end as in a short one, and the same between."""
    f = []
    for nz in (40, 64000):
        with api.LBM("cavity", 2, 2, nz, 0.3, 1.0, 0.05, bc="reference-links", storage="f64") as lbm:
            lbm.step(3)
            f.append(lbm.fields())
    for k in "uvwp":
        short, tall = f[0][k], f[1][k]
        assert np.array_equal(tall[:20], short[:20]) and np.array_equal(tall[-20:], short[-20:]), k
        assert (tall[20:-20] == short[20]).all(), k
