"""Inputs in pageable memory of four megabytes and more are staged through a ring of sixteen
page-locked megabytes: the same bits as from page-locked memory, on both sides of the size where it
begins, at whole and ragged pieces, beyond the ring's length and with callers on several threads."""
import os
import threading

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("n", [4 * MB // 24, 4 * MB // 24 + 1, 16 * MB // 24 + 1, 2 * MB, 2 * MB + 3])
def test_pageable_equals_page_locked(n):
    import torch
    import agama_b200
    from agama_b200 import _native
    pot = agama_b200.Potential(file=os.path.join(GOLDEN, "cfg2.coef"))
    lib, ptr = _native.lib(), _native.ptr
    x = np.random.default_rng(n).standard_normal((n, 3)) * 3
    locked = torch.from_numpy(x).pin_memory()
    want = np.empty(n)
    _native.check(lib.agama_evalPotentialMany(pot.handle, n, ptr(locked.numpy()), 0.0, ptr(want), None, None))
    got = [np.empty(n) for _ in range(3)]
    status = [None] * 3

    def call(k):
        status[k] = lib.agama_evalPotentialMany(pot.handle, n, ptr(x), 0.0, ptr(got[k]), None, None)

    threads = [threading.Thread(target=call, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert status == [0] * 3
    for g in got:
        assert np.array_equal(g, want)
