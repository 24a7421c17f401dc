"""Both sides of the size from which pageable inputs are staged (28 MB), as test_staging_gpu compares them."""
import pytest

import test_staging_gpu

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("n", [28 * MB // 24, 28 * MB // 24 + 1, 29 * MB // 24 + 1])
def test_both_sides(n):
    test_staging_gpu.test_pageable_equals_page_locked(n)
