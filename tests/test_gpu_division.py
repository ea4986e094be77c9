"""The kernels divide with a reciprocal estimate, one Newton-Raphson step and
Markstein's correction instead of the IEEE divide sequence.  This checks the
routine against CUDA's IEEE division on the GPU over random operands: at
most one ulp apart, and in practice identical."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_exponent,seed", [(40.0, 1), (300.0, 2), (1000.0, 3)])
def test_division_matches_ieee(max_exponent, seed):
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    n = 1 << 26
    mis, ulp = C.c_ulonglong(), C.c_ulonglong()
    _lib.check(lib.thorin_selftest_division(n, seed, max_exponent, C.byref(mis), C.byref(ulp)), "selftest_division")
    assert ulp.value <= 1
    assert mis.value <= n // 1000000


@pytest.mark.parametrize("max_exponent,seed", [(40.0, 4), (300.0, 5)])
def test_slope_division_bound(max_exponent, seed):
    """The van Leer slopes' division (no Markstein correction) stays within
    2^14 ulp of IEEE division, a relative error below 2^-38 (measured on
    GB300: 8696 ulp at most in 2^26 quotients)."""
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    ulp = C.c_ulonglong()
    _lib.check(lib.thorin_selftest_slope_division(1 << 26, seed, max_exponent, C.byref(ulp)),
               "selftest_slope_division")
    print("slope division: max", ulp.value, "ulp")
    assert ulp.value <= 16384


@pytest.mark.parametrize("span,max_exponent,seed", [(0.01, 1.0, 20), (1.0, 40.0, 21), (50.0, 200.0, 22),
                                                     (599.0, 300.0, 23), (700.0, 600.0, 24)])
def test_exp_and_power_match_cuda(span, max_exponent, seed):
    """The exponential by table is within one ulp of exp, as CUDA's is: at
    most 2 ulp apart.  x^(-3/2) is within 2 ulp and 1 / (x sqrt(x)) has three
    roundings (2 ulp): at most 4 ulp apart."""
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    ue, up = C.c_ulonglong(), C.c_ulonglong()
    _lib.check(lib.thorin_selftest_exp(1 << 26, seed, span, max_exponent, C.byref(ue), C.byref(up)), "selftest_exp")
    print("exp:", ue.value, "ulp; x^-3/2:", up.value)
    assert ue.value <= 2
    assert up.value <= 4


@pytest.mark.parametrize("max_exponent,seed", [(0.5, 9), (20.0, 10), (29.9, 11), (32.0, 12), (200.0, 13)])
def test_van_leer_slope_bound(max_exponent, seed):
    """The slope a b / (a + b) in FP32 pairs keeps the bound of the slopes'
    division, 2^14 ulp, on both sides of its range (operands 2^60 apart) and
    for both signs; the density's quotient r / (r + 1e-20) within 2 ulp."""
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    ulp, q = C.c_ulonglong(), C.c_ulonglong()
    _lib.check(lib.thorin_selftest_vl_slope(1 << 26, seed, max_exponent, C.byref(ulp), C.byref(q)),
               "selftest_vl_slope")
    print("slope: max", ulp.value, "ulp; quotient:", q.value)
    assert ulp.value <= 16384
    assert q.value <= 2


@pytest.mark.parametrize("max_exponent,seed", [(40.0, 6), (300.0, 7), (1000.0, 8)])
def test_square_roots_match_ieee(max_exponent, seed):
    """sqrt_fast is Markstein-corrected like the division: at most one ulp
    from sqrt, in practice identical."""
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    n = 1 << 26
    mis, ulp = C.c_ulonglong(), C.c_ulonglong()
    _lib.check(lib.thorin_selftest_sqrt(n, seed, max_exponent, C.byref(mis), C.byref(ulp)), "selftest_sqrt")
    assert ulp.value <= 1
    assert mis.value <= n // 1000000


def test_graph_conditional_nodes():
    """The SOR sweep loop is a WHILE graph node whose condition the last
    sweep's completion step clears; this checks the mechanism in bounded
    form first (IF nodes), then a WHILE node of five runs."""
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    a, b, w = C.c_int(), C.c_int(), C.c_int()
    _lib.check(lib.thorin_selftest_graph_conditional(C.byref(a), C.byref(b), C.byref(w)),
               "selftest_graph_conditional")
    assert (a.value, b.value, w.value) == (0, 1, 5)


def test_graph_nested_conditional_nodes():
    """A WHILE node inside a WHILE node's body (the substep loop around the
    SOR sweep loop of a whole-DT graph), bounded: 3 outer runs of 4 inner."""
    from fargo_thorin_gb300 import _lib
    lib = _lib.load()
    o, i = C.c_int(), C.c_int()
    _lib.check(lib.thorin_selftest_graph_nested(C.byref(o), C.byref(i)), "selftest_graph_nested")
    assert (o.value, i.value) == (3, 12)
