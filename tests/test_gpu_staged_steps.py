"""GPU: the staged step kernels that draw their tiles by ticket.

line_kernel (FP64 FAST and FP32 cavities, FP64 and FP32 sphere channels, from
some size on) and the 2-byte vortex and sphere channel (from six tiles a block on).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from imexlb_b200 import api as a

    return a


@pytest.mark.parametrize("case,n,storage", [("cavity", (113, 97, 90), "f64"), ("sphere", (130, 61, 58), "f64"),
                                            ("cavity", (80, 75, 77), "f32"), ("sphere", (206, 50, 47), "f32"),
                                            ("tgv", (128, 128, 112), "f16"), ("sphere", (256, 90, 84), "bf16")])
def test_wait_limit_gives_up_and_the_lattice_recovers(api, case, n, storage):
    """With a 1 ns bound blocks give up, let their copies in flight land and
    the next synchronising call reports it; re-initialised with the default
    bound the lattice runs bit for bit like a fresh one, so that the tile
    counters are back at zero."""
    kw = dict(bc="standard", storage=storage, arith="fast")
    with api.LBM(case, *n, 0.07, 1.0, 0.05, **kw) as lbm:
        lbm.step(2)
        lbm.set_wait_limit(1e-9)
        lbm.step(3)
        with pytest.raises(api.ImexlbError) as err:
            lbm.synchronize()
        assert err.value.code == 2 and "gave up waiting" in str(err.value)
        lbm.set_wait_limit(1.0)
        lbm.Initialize()
        lbm.step(9)
        got = lbm.fields()
    with api.LBM(case, *n, 0.07, 1.0, 0.05, **kw) as fresh:
        fresh.step(9)
        want = fresh.fields()
    for k in "uvwp":
        assert np.array_equal(got[k], want[k]), k
