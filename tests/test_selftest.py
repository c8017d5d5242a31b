"""Device self-checks of arithmetic that restates IEEE operations with other instructions, and of the autotuner's
timing."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_projection_factor_equals_ieee_sqrt_and_reciprocal_everywhere(cuda):
    """The FGP projection's 1 / sqrt(x), from approximate hardware results refined with FMAs, equals
    RN(1 / RN(sqrt(x))) -- the reference's 1.0f / std::sqrt(x) -- for every float in [1, 2^126)."""
    from qoraholo_b200 import capi

    mismatches, first = capi.selftest_rcp_sqrt()
    assert mismatches == 0, f"{mismatches} mismatches, first at x bits {first:#010x}"


def test_the_autotuner_times_the_device_and_not_the_host(cuda):
    """A kernel of 100 us behind 60 us of host work is faster than one of 130 us: a solve queues its launches, so
    the host's work runs while the kernel before does."""
    from qoraholo_b200 import capi

    assert capi.selftest_autotune() == 1
