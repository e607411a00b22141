"""Heat smoothing with neighbour lists on either side of what a thread keeps in registers.

Lists of 0 to 13 neighbours, and more points than the launch has threads: the
result equals, bit for bit, the same float64 sums in list order.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _lists(n, rng):
    degree = rng.integers(0, 14, size=n) if n > 1 else np.zeros(1, dtype=np.int64)
    offsets = np.concatenate(([0], np.cumsum(degree))).astype(np.int32)
    return degree, offsets, rng.integers(0, n, size=int(offsets[-1])).astype(np.int32)


def _device(array):
    return torch.as_tensor(array, device="cuda")


@pytest.mark.parametrize("n", [1, 257, 700_000])
def test_geometry(native_library, n):
    rng = np.random.default_rng(n)
    degree, offsets, neighbours = _lists(n, rng)
    points = rng.normal(size=(n, 3)).astype(np.float32)
    want = points.copy()
    for _ in range(3):
        total = np.zeros((n, 3))
        for k in range(int(degree.max(initial=0))):
            has = degree > k
            total[has] = total[has] + want[neighbours[offsets[:-1][has] + k]].astype(np.float64)
        want = ((want.astype(np.float64) + total / 3.0) / (1.0 + degree / 3.0)[:, None]).astype(np.float32)
    v, off, nbr = _device(points), _device(offsets), _device(neighbours if neighbours.size else np.zeros(1, np.int32))
    out = torch.empty_like(v)
    scratch = torch.empty(12 * n + 4096, dtype=torch.uint8, device="cuda")
    assert native_library.csg_feature_smooth_geometry(n, off.data_ptr(), nbr.data_ptr(), v.data_ptr(), 3, out.data_ptr(),
                                                      scratch.data_ptr(), scratch.numel(), 0) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("n", [1, 257, 300_000])
def test_values(native_library, n):
    """Two series of different lengths; coincident points, so that every weight is exactly 1."""

    import ctypes

    rng = np.random.default_rng(n + 1)
    degree, offsets, neighbours = _lists(n, rng)
    values = rng.normal(size=n)
    counts = (3, 1)
    want = []
    for count in counts:
        field = values.copy()
        for _ in range(count):
            total = np.zeros(n)
            for k in range(int(degree.max(initial=0))):
                has = degree > k
                total[has] = total[has] + field[neighbours[offsets[:-1][has] + k]]
            field = (field + total) / (1.0 + degree)
        want.append(field)
    v, off, nbr = _device(values), _device(offsets), _device(neighbours if neighbours.size else np.zeros(1, np.int32))
    geometry = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    out = torch.empty(2, n, dtype=torch.float64, device="cuda")
    scratch = torch.empty(16 * 2 * (neighbours.size + 3 * n) + (1 << 20), dtype=torch.uint8, device="cuda")
    sigmas, iterations = (ctypes.c_double * 2)(1.0, 2.0), (ctypes.c_int32 * 2)(*counts)
    assert native_library.csg_feature_smooth_values(
        n, off.data_ptr(), nbr.data_ptr(), int(neighbours.size), 1, geometry.data_ptr(), v.data_ptr(), 2,
        ctypes.addressof(sigmas), ctypes.addressof(iterations), 0, out.data_ptr(), scratch.data_ptr(), scratch.numel(), 0) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), np.stack(want))


@pytest.mark.parametrize("n, series", [(120_000, 1), (45_000, 3), (110_000, 2), (660_000, 2)])
def test_values_of_more_points_than_threads(native_library, n, series):
    """Launches of more points than threads that keep lists: just more, twice as many, and more than eleven times."""

    import ctypes

    rng = np.random.default_rng(n + series)
    degree, offsets, neighbours = _lists(n, rng)
    values = rng.normal(size=n)
    want = []
    for count in range(1, series + 1):
        field = values.copy()
        for _ in range(count):
            total = np.zeros(n)
            for k in range(int(degree.max(initial=0))):
                has = degree > k
                total[has] = total[has] + field[neighbours[offsets[:-1][has] + k]]
            field = (field + total) / (1.0 + degree)
        want.append(field)
    v, off, nbr = _device(values), _device(offsets), _device(neighbours)
    geometry = torch.zeros(n, 3, dtype=torch.float64, device="cuda")  # coincident points: every weight is exactly 1
    out = torch.empty(series, n, dtype=torch.float64, device="cuda")
    scratch = torch.empty(16 * series * (neighbours.size + 3 * n) + (1 << 20), dtype=torch.uint8, device="cuda")
    sigmas, iterations = (ctypes.c_double * series)(*[1.0] * series), (ctypes.c_int32 * series)(*range(1, series + 1))
    assert native_library.csg_feature_smooth_values(
        n, off.data_ptr(), nbr.data_ptr(), int(neighbours.size), 1, geometry.data_ptr(), v.data_ptr(), series,
        ctypes.addressof(sigmas), ctypes.addressof(iterations), 0, out.data_ptr(), scratch.data_ptr(), scratch.numel(), 0) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), np.stack(want))
