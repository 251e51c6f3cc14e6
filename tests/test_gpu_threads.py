"""GPU: distinct handles used from different host threads at the same time,
as the library's threading contract allows."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def long_rows(seed, m, k, count):
    """`count` rows of 300 entries among rows of two: a skewed matrix."""
    rng = np.random.default_rng(seed)
    A = np.zeros((m, k), dtype=np.float32)
    for i in range(m):
        cnt = 300 if i % (m // count) == 0 else 2
        A[i, rng.choice(k, size=cnt, replace=False)] = rng.standard_normal(cnt).astype(np.float32)
    return A


def repeat(h, B, want, passes, errors):
    import torch
    try:
        s = torch.cuda.Stream()
        C = torch.empty_like(want)
        for _ in range(passes):
            h.spdm(B, C, stream=s)
        s.synchronize()
        if not torch.equal(C, want):
            errors.append("another result")
    except Exception as e:  # the other thread's result is checked all the same
        errors.append(repr(e))


def at_once(native, jobs, passes=4000, **params):
    """Each (A, B) by a thread of its own, multiplied again and again."""
    import torch
    work = []
    for A, B in jobs:
        h = native.GcooHandle(torch.from_numpy(A).cuda(), **params).build()
        dB = torch.from_numpy(B).cuda()
        work.append((h, dB, h.spdm(dB)))
    torch.cuda.synchronize()
    errors = []
    threads = [threading.Thread(target=repeat, args=(*w, passes, errors)) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:3]
    assert all(h.device_status() == 0 for h, _, _ in work)


def test_long_rows_of_two_handles(native):
    """One long row takes all of an SM's shared memory, many share it."""
    rng = np.random.default_rng(1)
    few, many = long_rows(2, 64, 2000, 1), long_rows(3, 4800, 2000, 400)
    B = rng.standard_normal((2000, 64)).astype(np.float32)
    at_once(native, 2 * [(few, B), (many, B)], passes=8000)


def test_panels_of_two_handles(native):
    """One warp per CTA (n = 128) beside four (n = 512)."""
    rng = np.random.default_rng(4)
    A = np.repeat(rng.standard_normal((2, 256)), 16, axis=0).astype(np.float32)
    jobs = [(A, rng.standard_normal((256, n)).astype(np.float32)) for n in (128, 512)]
    at_once(native, jobs, fp32_order="groups")
