"""Tests that compare with the reference's own build (tests/refimpl.py) skip
where that library is absent, instead of failing to load it."""
import os

import pytest

REF_SO = os.path.join(os.path.dirname(os.path.abspath(__file__)), "oracle", "_ref",
                      "libfmm2d_ref.so")


def _skip_without_reference(outcome):
    e = outcome.excinfo[1] if outcome.excinfo else None
    if isinstance(e, OSError) and REF_SO in str(e) and not os.path.exists(REF_SO):
        outcome.force_exception(pytest.skip.Exception("reference build absent"))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_setup(item):
    _skip_without_reference((yield))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    _skip_without_reference((yield))
