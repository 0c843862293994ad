"""The SUPG kernels' inverse square root (rsqrt_nr) against extended-precision
values on the host, across the points 1e-37 and 1e37 where it goes over to
CUDA's own operations.  Bars: inside, half an ulp for the result's rounding and
half for that of e (an absolute 2^-53, halved by the step), the cut series
below 2^-8 ulp; outside, half an ulp each for the division and (as the root's
relative rounding, at most one ulp) the square root: 1.5."""
import numpy as np
import pytest

from femorph_b200 import api

pytestmark = pytest.mark.gpu


def test_rsqrt_within_ulps():
    rng = np.random.default_rng(11)
    x = [10.0 ** rng.uniform(-40, 40, 300000), rng.uniform(0.25, 4.0, 100000), 10.0 ** rng.uniform(-12, 6, 100000)]
    for edge in (1e-37, 1e37):
        x.append(edge * (1 + np.linspace(-1e-6, 1e-6, 41)))
        x.append(np.array([np.nextafter(edge, 0), edge, np.nextafter(edge, np.inf)]))
    x.append(np.array([1.0, 2.0, 3.0, 4.0, 0.25, 1e-300, 1e300, 5e-324]))
    x = np.concatenate(x)
    out = np.zeros(x.size)
    api.check(api.lib().fm_math_check_rsqrt(x.ctypes.data, x.size, out.ctypes.data))
    exact = 1 / np.sqrt(x.astype(np.longdouble))
    ulps = np.asarray(np.abs(out - exact) / np.spacing(np.asarray(exact, np.float64)), np.float64)
    inside = (x > 1e-37) & (x < 1e37)
    print(f"[math] rsqrt_nr max ulps {ulps[inside].max():.3f} inside, {ulps[~inside].max():.3f} outside")
    assert ulps[inside].max() <= 1.0 + 2.0 ** -8
    assert ulps[~inside].max() <= 1.5


def test_rsqrt_of_special_values():
    x = np.array([0.0, np.inf, np.nan, -1.0])
    out = np.zeros(4)
    api.check(api.lib().fm_math_check_rsqrt(x.ctypes.data, 4, out.ctypes.data))
    assert out[0] == np.inf and out[1] == 0.0 and np.isnan(out[2:]).all()
