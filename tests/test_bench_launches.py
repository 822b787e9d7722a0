"""The bench's count of its own launches: by the kernel that runs, not by the
flux alone."""
import pytest

import bench


@pytest.mark.parametrize("flux,variant,per_step,per_call", [("Linde", 0, 2, 1), ("Linde", 1, 4, 0), ("HLLD", 2, 4, 0),
                                                            ("Rusanov", 3, 4, 0), ("Roe", 0, 4, 0)])
def test_own_launches(flux, variant, per_step, per_call):
    assert bench.own_launches(flux, variant, 30) == 30 * per_step + per_call
