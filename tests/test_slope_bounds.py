"""The errors stated beside the reciprocal estimate (2^-43, with the hardware's
FP32 estimate 2 ulp off) and the van Leer slope in FP32 pairs (2^-42), in units
of 2^-53: tighter than the bound that the slopes need (2^-38)."""
import ctypes as C

import pytest

from fargo_thorin_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_exponent,seed", [(1.0, 31), (40.0, 32), (300.0, 33)])
def test_slope_division_within_its_stated_error(max_exponent, seed):
    ulp = C.c_ulonglong()
    _lib.check(_lib.load().thorin_selftest_slope_division(1 << 26, seed, max_exponent, C.byref(ulp)), "slope_division")
    print("slope division: max", ulp.value, "ulp")
    assert ulp.value <= 1024 + 1                          # and the product's rounding


@pytest.mark.parametrize("max_exponent,seed", [(0.5, 34), (20.0, 35), (29.9, 36), (32.0, 37), (200.0, 38)])
def test_van_leer_slope_within_its_stated_error(max_exponent, seed):
    ulp, q = C.c_ulonglong(), C.c_ulonglong()
    _lib.check(_lib.load().thorin_selftest_vl_slope(1 << 26, seed, max_exponent, C.byref(ulp), C.byref(q)), "vl_slope")
    print("slope: max", ulp.value, "ulp")
    assert ulp.value <= 2048 + 2                          # and the reference's two roundings


@pytest.mark.parametrize("max_exponent,max_weight,seed", [(0.5, 1.05, 41), (20.0, 1.05, 42), (29.9, 2.0, 43),
                                                          (32.0, 4.0, 44), (200.0, 64.0, 45)])
def test_weighted_slope_within_its_stated_error(max_exponent, max_weight, seed):
    """The radial step's slope: w enters as an FP32 pair (2^-48)."""
    ulp = C.c_ulonglong()
    _lib.check(_lib.load().thorin_selftest_vl_slope_weighted(1 << 26, seed, max_exponent, max_weight, C.byref(ulp)),
               "vl_slope_weighted")
    print("weighted slope: max", ulp.value, "ulp")
    assert ulp.value <= 2048 + 3                          # and the reference's three roundings
