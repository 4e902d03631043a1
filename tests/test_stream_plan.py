"""The layout of the direction streams (host side of the stream transport), without a
device: positions and groups for random task levels and upwind counts, over narrow and
wide levels, several parts and ragged sizes."""
import ctypes

import numpy as np
import pytest

from subsweep_gb300 import _native

GROUP = 32  # tasks of a group


def _plan(level, up, np_, n, d, parts):
    f = _native.load_gpu().sw_host_stream_plan
    f.restype = ctypes.c_int64
    f.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_uint32] * 3 + [ctypes.c_void_p, ctypes.c_uint32] + \
        [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64]
    order = np.zeros(n * d, np.uint32)
    plan = np.zeros((n * d, 5), np.int64)
    k = f(level.ctypes.data, up.ctypes.data, np_, n, d, parts.ctypes.data, len(parts) - 1, order.ctypes.data,
          plan.ctypes.data, plan.shape[0])
    assert 0 < k <= plan.shape[0]
    return order, plan[:k]


@pytest.mark.parametrize("n,parts,depth", [(1, [0, 1], 1), (33, [0, 33], 33), (700, [0, 300, 700], 5),
                                           (5000, [0, 5000], 3), (5001, [0, 1, 4100, 5001], 200)])
def test_stream_plan(n, parts, depth):
    rng = np.random.default_rng(n)
    d = 3
    np_ = (n + 31) // 32 * 32
    level = np.full(np_ * d, 0xffff, np.uint16)
    up = np.full(np_ * d, 0xff, np.uint8)
    for k in range(d):  # levels contiguous from 0 in every stream
        for a, b in zip(parts[:-1], parts[1:]):
            m = min(depth, b - a)
            level[k * np_ + a:k * np_ + b] = rng.permutation(np.concatenate([np.arange(m), rng.integers(0, m, b - a - m)]))
            up[k * np_ + a:k * np_ + b] = rng.integers(0, 64, b - a)
    order, plan = _plan(level, up, np_, n, d, np.array(parts, np.uint32))
    assert np.array_equal(np.sort(order), np.concatenate([np.arange(n) + k * np_ for k in range(d)]))
    at, stream = 0, -1
    for s, pos, need, tasks, slots in plan:
        if s != stream:  # a new stream: one direction and part, its groups counted from 0
            stream, groups, lv, before = s, 0, -1, 0
            direction, part = divmod(s, len(parts) - 1)
            assert at == direction * n + parts[part]
        assert pos == at and 0 < tasks <= GROUP
        t = order[at:at + tasks]
        assert np.all(t // np_ == direction) and np.all(level[t] == level[t[0]])
        if level[t[0]] != lv:  # a new level: after every group of the levels before it
            assert level[t[0]] == lv + 1
            lv, before = lv + 1, groups
        assert need == before
        assert slots == (int(up[t].max()) + 3) // 4 * 4 and np.all(np.diff(up[t].astype(int)) >= 0)
        at, groups = at + tasks, groups + 1
    assert at == n * d
