"""The process-wide context after other tests have set its schedule: the calls
that go through it run the default one again.  The first test does what tests
that try schedules do; the second one follows it."""
import ctypes

import pytest

from tests.conftest import random_seeds

pytestmark = pytest.mark.gpu

cu = pytest.importorskip("integer_delauney_b200._delauney_cuda")
from integer_delauney_b200 import _capi  # noqa: E402


def _direct_runs():
    out = (ctypes.c_int64 * 3)()
    _capi.check(_capi.load().idl_selftest_counts(_capi.context_for(0).handle, out, 3))
    return out[0]


def test_a_schedule_is_left_behind():
    _capi.context_for(0).set_schedule(3)
    before = _direct_runs()
    cu.triangulate(200, 150, random_seeds(200, 150, 100, 1))
    assert _direct_runs() == before


def test_the_next_test_runs_the_default_schedule():
    before = _direct_runs()
    cu.triangulate(200, 150, random_seeds(200, 150, 100, 1))
    assert _direct_runs() == before + 1
