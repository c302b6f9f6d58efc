"""Which kernel form a standard lattice's step takes, checked on the CPU.

The rules are the library's own (imexlb_debug_step_form); the sizes are those
at which a form was measured slower than the one it had replaced, and some on
either side of each line.
"""
import pytest

from imexlb_b200 import api

ITEMS, ROWS, LINE, STAGED, BOX = range(5)


def form(case, storage, arith, n):
    return api.load_library().imexlb_debug_step_form(api.CASES[case], api.STORAGES[storage], api.ARITHS[arith], *n)


# EXACT cavities: their arithmetic sets the pace, staging costs
@pytest.mark.parametrize("n,want", [((100, 70, 70), ITEMS), ((112, 80, 60), ITEMS), ((16, 2, 15000), ITEMS),
                                    ((112, 7, 640), ITEMS), ((240, 240, 240), ITEMS), ((64, 64, 64), ROWS),
                                    ((128, 128, 128), ROWS), ((156, 156, 156), ITEMS)])
def test_exact_cavity_is_not_staged(n, want):
    assert form("cavity", "f64", "exact", n) == want


# FP64 FAST cavities: from 950,000 cells on
@pytest.mark.parametrize("n,want", [((96, 96, 96), ITEMS), ((100, 70, 70), ITEMS), ((112, 112, 80), LINE),
                                    ((151, 133, 117), LINE), ((128, 128, 128), LINE)])
def test_fp64_cavity_is_staged_from_its_size_on(n, want):
    assert form("cavity", "f64", "fast", n) == want


# planes that would leave their last tile mostly empty: cavities keep the registers
@pytest.mark.parametrize("storage,n,want", [("f64", (16, 2, 60000), ITEMS), ("f64", (32, 4, 8000), ITEMS),
                                            ("f64", (64, 12, 1400), LINE), ("f32", (96, 6, 850), ITEMS),
                                            ("f32", (64, 12, 640), ITEMS), ("f32", (112, 7, 640), LINE),
                                            ("f32", (160, 144, 150), LINE), ("f32", (160, 144, 19), ITEMS)])
def test_cavity_tiles_are_mostly_full(storage, n, want):
    assert form("cavity", storage, "fast", n) == want


@pytest.mark.parametrize("storage,n,want", [("f64", (130, 61, 58), LINE), ("f32", (130, 61, 58), LINE),
                                            ("f32", (206, 50, 47), LINE), ("f64", (96, 6, 850), LINE),
                                            ("f32", (131, 61, 58), ITEMS), ("f64", (128, 40, 40), ITEMS),
                                            ("f16", (256, 64, 64), STAGED), ("f16", (257, 64, 64), ITEMS)])
def test_sphere(storage, n, want):
    assert form("sphere", storage, "exact", n) == want


@pytest.mark.parametrize("storage,n,want", [("f64", (128, 128, 128), ITEMS), ("f32", (128, 128, 128), ITEMS),
                                            ("f16", (128, 128, 128), STAGED)])
def test_vortex(storage, n, want):
    assert form("tgv", storage, "fast", n) == want


# rows that are not whole sectors, of a lattice too large for the L2: one row a
# warp (a half warp of pairs), where they mostly fill it
@pytest.mark.parametrize("case,storage,arith,n,want",
                         [("tgv", "f64", "fast", (17, 180, 170), BOX), ("tgv", "f64", "fast", (24, 130, 120), BOX),
                          ("tgv", "f64", "exact", (24, 130, 120), ITEMS), ("tgv", "f64", "exact", (31, 130, 120), BOX),
                          ("tgv", "f64", "fast", (36, 130, 120), ITEMS), ("tgv", "f64", "fast", (55, 130, 120), BOX),
                          ("tgv", "f64", "fast", (20, 90, 90), ITEMS), ("tgv", "f64", "fast", (25, 25, 25), ITEMS),
                          ("cavity", "f64", "exact", (31, 130, 120), BOX), ("cavity", "f64", "fast", (17, 180, 170), BOX),
                          ("cavity", "f64", "fast", (20, 180, 170), ITEMS), ("cavity", "f64", "fast", (38, 130, 120), ITEMS),
                          ("tgv", "f32", "exact", (18, 130, 120), BOX), ("tgv", "f32", "exact", (9, 200, 200), BOX),
                          ("tgv", "f32", "exact", (24, 130, 120), ITEMS), ("tgv", "f32", "exact", (41, 150, 140), BOX),
                          ("tgv", "f32", "exact", (77, 130, 120), ITEMS), ("tgv", "f32", "exact", (35, 64, 64), ITEMS),
                          ("cavity", "f32", "exact", (20, 64, 64), BOX), ("cavity", "f32", "exact", (34, 130, 120), ITEMS),
                          ("tgv", "f16", "exact", (125, 130, 120), BOX), ("tgv", "f16", "exact", (101, 108, 47), ITEMS),
                          ("cavity", "f16", "exact", (41, 130, 120), ITEMS), ("sphere", "f64", "fast", (31, 130, 60), ITEMS)])
def test_rows_apart(case, storage, arith, n, want):
    assert form(case, storage, arith, n) == want
