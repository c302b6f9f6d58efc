"""GPU: lattices on streams of their own and on a second device."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imexlb_b200", "csrc")


@pytest.fixture(scope="module")
def api():
    import torch

    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for gpu tests")
    from imexlb_b200 import api as a

    return a


# The legacy stream is not ordered with a lattice's own stream: a clear queued
# on it may land after the lattice's steps, or between them.
@pytest.mark.parametrize("name", ["lattice.cu", "engine.cu"])
def test_device_memory_is_cleared_on_its_owners_stream(name):
    with open(os.path.join(CSRC, name)) as fh:
        assert not re.findall(r"\bcudaMemset\(", fh.read())


# Nor is a copy on it, which from pageable memory may return before its last
# bytes have landed: a lattice's first gather once read a part of its plan that
# was not there yet, and with it an address outside its buffers.
@pytest.mark.parametrize("name", ["lattice.cu", "engine.cu"])
def test_tables_are_uploaded_on_their_owners_stream(name):
    with open(os.path.join(CSRC, name)) as fh:
        assert not re.findall(r"\bcudaMemcpy\(", fh.read())


# reference boundaries: ghost plan, inlet profile, face codes; standard sphere: mask and links
@pytest.mark.gpu
@pytest.mark.parametrize("case,n,bc,storage", [("cavity", (96, 100, 90), "reference", "f32"),
                                               ("cavity", (48, 50, 40), "reference-links", "f64"),
                                               ("sphere", (128, 40, 36), "reference", "f64"),
                                               ("sphere", (128, 40, 36), "standard", "f64")])
def test_tables_are_there_for_the_first_step(api, case, n, bc, storage):
    import torch

    side = torch.cuda.Stream()
    kw = dict(bc=bc, storage=storage, arith="fast")
    with api.LBM(case, *n, 0.3, 1.0, 0.05, **kw) as lbm:
        lbm.step(4)
        want = lbm.fields()
    for _ in range(5):
        torch.cuda._sleep(int(2e7))  # about 10 ms of the legacy stream
        with api.LBM(case, *n, 0.3, 1.0, 0.05, stream=side.cuda_stream, **kw) as lbm:
            lbm.step(4)
            got = lbm.fields()
        for k in "uvwp":
            assert np.array_equal(got[k], want[k], equal_nan=True), k


# FP64 and FP32 staged and the 2-byte vortex: tile counters; the 2-byte cavity:
# the error word
@pytest.mark.gpu
@pytest.mark.parametrize("case,n,storage", [("cavity", (80, 75, 77), "f64"), ("cavity", (80, 75, 77), "f32"),
                                            ("tgv", (128, 128, 112), "f16"), ("cavity", (64, 40, 48), "f16")])
def test_create_beside_work_on_the_legacy_stream(api, case, n, storage):
    import torch

    kw = dict(bc="standard", storage=storage, arith="fast")
    with api.LBM(case, *n, 0.07, 1.0, 0.05, **kw) as lbm:
        lbm.step(6)
        want = lbm.fields()
    # used memory for the next lattice: the pool keeps what this one leaves
    with api.LBM("tgv", 160, 144, 150, 0.07, 1.0, 0.05, bc="standard", storage="f64", arith="fast") as big:
        big.step(1)
        big.synchronize()
    side = torch.cuda.Stream()
    torch.cuda._sleep(int(5e8))  # about a quarter of a second of the legacy stream
    with api.LBM(case, *n, 0.07, 1.0, 0.05, stream=side.cuda_stream, **kw) as lbm:
        lbm.step(6)
        got = lbm.fields()
    torch.cuda.synchronize()
    for k in "uvwp":
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.gpu
@pytest.mark.parametrize("case,storage", [("cavity", "f64"), ("cavity", "f32"), ("sphere", "f32"), ("tgv", "f16"),
                                          ("cavity", "f16")])
def test_a_second_device_steps_like_the_first(case, storage):
    import torch

    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices")
    got = []
    for dev in (0, 1):
        with torch.cuda.device(dev), api.LBM(case, 128, 96, 100, 0.07, 1.0, 0.05, bc="standard", storage=storage,
                                             arith="fast") as lbm:
            lbm.step(4)
            got.append(lbm.fields())
    for k in "uvwp":
        assert np.array_equal(got[0][k], got[1][k]), k
