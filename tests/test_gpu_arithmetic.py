"""Device checks of the arithmetic the iteration kernels use in place of a
slower call: the same bits over the range they use it in."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [20261205, 7])
def test_disc_factor_equals_clamped_rhypotf(seed):
    """min(1, rhypotf(a, b)), which the reference's dual projection applies
    (pdflow_cudalib.cu:813-887), on 2^28 random pairs a seed."""
    from pdflow import _lib
    bad = ctypes.c_ulonglong(1)
    assert _lib.load().pdflow_check_disc_factor(1 << 28, seed, ctypes.byref(bad)) == 0
    assert bad.value == 0


@pytest.mark.parametrize("seed", [31, 20261206])
def test_reciprocal_division_equals_ieee_over_its_whole_range(seed):
    """div_rcp over the range the shrinkage takes it in: numerators to 2^60 over
    any denominator, to 2^90 where the quotient stays below 2^31, and a1 of / den
    with |of| at the threshold, on 2^28 random pairs a seed."""
    from pdflow import _lib
    bad = ctypes.c_ulonglong(1)
    assert _lib.load().pdflow_check_div_rcp(1 << 28, seed, ctypes.byref(bad)) == 0
    assert bad.value == 0
