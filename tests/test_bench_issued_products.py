"""bench.fx_issued_products, the slice products that the bench reports as issued, against
the rule it states and against the slices that the contexts take."""
import pytest

import bench
from codyfortran_gb300 import spec as S


class _Sys:
    def __init__(self, n):
        self.nG = n


@pytest.mark.parametrize("precision,n,want", [("mixed_fx6", 501, 21), ("mixed_fx6", 1024, 21), ("mixed_fx6", 1025, 15),
                                              ("mixed_fx6", 2001, 15), ("mixed_fx", 501, 15), ("mixed_fx", 2801, 15)])
def test_issued_slice_products(precision, n, want):
    assert bench.fx_issued_products(precision, [_Sys(n), _Sys(100)]) == want


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed_fx", "mixed_fx6"])
@pytest.mark.parametrize("n_el", [40, 204, 205])
def test_the_contexts_slices(precision, n_el):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(n_el, 6, 2)
    e = Engine(sp, precision)
    L = e.contraction_slices()
    e.close()
    assert L * (L + 1) // 2 == bench.fx_issued_products(precision, [e])
