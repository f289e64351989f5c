"""The monitors' sums over the nodes are formed to FP64's accuracy and rounded
to REAL*4 once.  VREF = SQRT(2 sum |W|^2 / (IM JM KM)) of fields whose sum
falls on a tie of two REAL*4 values, which a part 2^-52 of it decides; spans
more than the range of one value's digits; or is not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vref(w):
    """VREF of a step that starts with W = (w, 0, 0), w (KM, JM, IM)."""
    from mgpu import case, common_setup, lib
    cd = common_setup.build_common(case.small_nozzle())
    p = lib.Problem(cd)
    z = np.zeros(cd.arrays["RO"].shape, np.float32)
    for n, a in (("RO", z + np.float32(1)), ("ROVX", w.astype(np.float32)), ("ROVR", z), ("RORVT", z), ("WT", z)):
        p.set(n, a)
    return np.float32(p.step(force_end=True, check=False).vref)


def _expected(total, n):
    return np.sqrt(np.float32(total) * (np.float32(2.0) / np.float32(n)))


@pytest.fixture(scope="module")
def shape():
    from mgpu import case, common_setup
    return common_setup.build_common(case.small_nozzle()).arrays["RO"].shape


@pytest.mark.parametrize("where", [(0, 1, 2, 3), (0, 40, 80, 200), (0, 300, 700, 1500), (1500, 3, 900, 0)])
def test_a_tie_is_decided_by_its_last_part(shape, where):
    n = int(np.prod(shape))
    # a^2 an even whole number of 24 bits, such that VREF tells it from a^2 + 1
    a = next(a for a in range(2898, 4096, 2) if _expected(a * a, n) != _expected(a * a + 1, n))
    w = np.zeros(shape, np.float32)
    inner = w[:, 1:, :].reshape(-1)                      # |W| counts from J = 2; a copy, put back below
    inner[list(where)] = a, 0.5, 0.5, 2.0 ** -14         # a^2 + 1/2 + 2^-28
    w[:, 1:, :] = inner.reshape(w[:, 1:, :].shape)
    assert _vref(w) == _expected(a * a + 1, n)


@pytest.mark.parametrize("span", [0, 4, 20, 40])
def test_sums_of_any_spread(shape, span):
    rng = np.random.default_rng(span)
    w = (rng.standard_normal(shape) * 2.0 ** rng.uniform(-span, min(span, 20), shape)).astype(np.float32)
    e = (w[:, 1:, :] * w[:, 1:, :]).astype(np.float64)
    assert _vref(w) == _expected(np.sum(np.sort(e.ravel())), w.size)


@pytest.mark.parametrize("bad", [np.inf, 1e25, np.nan])
def test_what_is_not_finite_stays_so(shape, bad):
    w = np.ones(shape, np.float32)
    w[2, 11, 3] = bad
    v = _vref(w)
    assert np.isnan(v) if np.isnan(bad) else v == np.inf
