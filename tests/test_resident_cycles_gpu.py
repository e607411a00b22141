"""Resident V-cycles and V-cycle legs against the separate relaxation, residual and transfer kernels.

Every point sees the operations of the separate kernels in their order, so a solve
must equal, bit for bit, the same V-cycles composed of those kernels: at grids on
either side of each size rule, slabs of unequal rows, batches that change the
cluster size, and systems whose quotients need the plain division.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PARAMS = (1.0, 1.0, 0.3, 0.0, 1e-3)


def _levels(nx, ny):
    sizes = [(nx, ny)]
    while sizes[-1] != (1, 1):
        sizes.append(((sizes[-1][0] + 1) // 2, (sizes[-1][1] + 1) // 2))
    return sizes


def _problem(nx, ny, batch, dtype, kind):
    generator = torch.Generator(device="cuda").manual_seed(1000 * nx + ny)
    hess = 0.5 + 0.1 * torch.rand(batch, 3, ny, nx, dtype=dtype, device="cuda", generator=generator)
    hess[:, 2] *= 0.1
    rhs = torch.randn(batch, 2, ny, nx, dtype=dtype, device="cuda", generator=generator)
    start = torch.randn(batch, 2, ny, nx, dtype=dtype, device="cuda", generator=generator)
    if kind == "division":  # zero numerators, and determinants outside the reciprocal's range
        start.zero_()
        rhs[..., ::3, :] = 0
        hess[:, :2, ny // 2 :] *= 1e70 if dtype == torch.float64 else 1e15
    return hess, rhs, start


def _params(level, full):
    sx, sy, mu, lam, ident = PARAMS
    return (ctypes.c_double * 5)(sx * level[0] / full[0], sy * level[1] / full[1], mu, lam, ident)


def _separate(lib, code, hess, rhs, start, cycles, nit):
    batch, _, ny, nx = hess.shape
    sizes = _levels(nx, ny)
    systems = [hess]
    for (snx, sny), (tnx, tny) in zip(sizes, sizes[1:]):
        coarse = torch.empty(batch, 3, tny, tnx, dtype=hess.dtype, device="cuda")
        assert lib.csg_dartel_resize(code, 3 * batch, snx, sny, systems[-1].data_ptr(), tnx, tny, coarse.data_ptr(), 0, 0) == 0
        systems.append(coarse)

    def relax(level, b, u):
        w, h = sizes[level]
        assert lib.csg_dartel_relax(code, batch, w, h, systems[level].data_ptr(), b.data_ptr(), _params(sizes[level], sizes[0]),
                                    nit, u.data_ptr(), 0) == 0

    def cycle(level, b, u):
        w, h = sizes[level]
        relax(level, b, u)
        if level + 1 == len(sizes):
            return
        applied, coarse_b = torch.empty_like(u), torch.empty(batch, 2, *sizes[level + 1][::-1], dtype=u.dtype, device="cuda")
        assert lib.csg_dartel_membrane_apply(code, batch, w, h, systems[level].data_ptr(), u.data_ptr(),
                                             _params(sizes[level], sizes[0]), applied.data_ptr(), 0) == 0
        left = b - applied
        cw, ch = sizes[level + 1]
        assert lib.csg_dartel_resize(code, 2 * batch, w, h, left.data_ptr(), cw, ch, coarse_b.data_ptr(), 0, 0) == 0
        coarse_u = torch.zeros_like(coarse_b)
        cycle(level + 1, coarse_b, coarse_u)
        assert lib.csg_dartel_resize(code, 2 * batch, cw, ch, coarse_u.data_ptr(), w, h, u.data_ptr(), 1, 0) == 0
        relax(level, b, u)

    u = start.clone()
    for _ in range(cycles):
        cycle(0, rhs, u)
    return u


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize(
    "nx, ny, batch, cycles, nit, kind",
    [
        (1, 1, 2, 2, 1, "plain"),
        (2, 1, 1, 1, 3, "plain"),
        (8, 5, 3, 2, 2, "division"),
        (32, 16, 2, 3, 3, "plain"),  # the largest grid of one CTA
        (32, 17, 1, 2, 3, "division"),  # two CTAs, unequal rows
        (2, 300, 1, 2, 1, "plain"),
        (1, 300, 1, 1, 2, "plain"),  # too many rows for one unit per thread
        (64, 32, 1, 2, 3, "division"),
        (64, 33, 3, 2, 1, "plain"),  # transfers that read other CTAs' rows
        (64, 32, 40, 2, 2, "plain"),  # fewer CTAs per grid; float32 two to an SM
        (128, 65, 1, 1, 2, "plain"),
        (256, 100, 1, 2, 1, "plain"),
        (256, 128, 2, 2, 3, "division"),  # the largest resident grid
        (256, 128, 10, 1, 1, "plain"),
        (512, 64, 1, 1, 2, "plain"),
        (256, 130, 1, 1, 1, "plain"),  # the first level as two legs of tiles
        (512, 256, 1, 1, 3, "division"),
        (512, 131, 2, 2, 6, "plain"),  # the widest halo
        (64, 601, 2, 1, 2, "plain"),  # tiles of whole rows
        (2, 17000, 1, 1, 1, "plain"),
        (512, 100, 1, 1, 7, "plain"),  # the first level in separate launches
    ],
)
def test_resident_cycles_equal_the_separate_kernels(native_library, dtype, nx, ny, batch, cycles, nit, kind):
    lib = native_library
    code = 1 if dtype == torch.float64 else 0
    hess, rhs, start = _problem(nx, ny, batch, dtype, kind)
    scratch = torch.empty(lib.csg_dartel_scratch_bytes(code, batch, nx, ny), dtype=torch.uint8, device="cuda")
    u = start.clone()
    assert lib.csg_dartel_fmg(code, batch, nx, ny, hess.data_ptr(), rhs.data_ptr(), _params((nx, ny), (nx, ny)), cycles, nit,
                              u.data_ptr(), 1, 1, scratch.data_ptr(), scratch.numel(), 0) == 0
    torch.cuda.synchronize()
    assert torch.isfinite(u).all()
    assert torch.equal(u, _separate(lib, code, hess, rhs, start, cycles, nit))


@pytest.mark.parametrize(
    "dtype, nx, ny, batch, nit, legs",
    [
        (torch.float64, 512, 256, 1, 3, True),
        (torch.float64, 512, 256, 4, 3, True),
        (torch.float64, 512, 256, 8, 5, False),  # many tiles, a point updated four times
        (torch.float32, 512, 256, 8, 5, True),
        (torch.float64, 512, 256, 1, 6, True),
        (torch.float64, 512, 256, 1, 8, False),  # tiles of 12 x 6
        (torch.float32, 512, 256, 1, 9, False),
        (torch.float64, 512, 100, 1, 9, False),
        (torch.float64, 512, 100, 1, 10, False),  # halos that leave nothing
        (torch.float64, 16, 4096, 1, 9, True),  # whole rows
    ],
)
def test_fine_levels_take_the_cheaper_form(native_library, dtype, nx, ny, batch, nit, legs):
    """The first level, above the resident ones, as two launches or as separate ones, with equal results."""

    lib = native_library
    code = 1 if dtype == torch.float64 else 0
    hess, rhs, start = _problem(nx, ny, batch, dtype, "plain")
    scratch = torch.empty(lib.csg_dartel_scratch_bytes(code, batch, nx, ny), dtype=torch.uint8, device="cuda")
    launches = []
    for cycles in (0, 1):
        u = start.clone()
        before = lib.csg_kernel_launches()
        assert lib.csg_dartel_fmg(code, batch, nx, ny, hess.data_ptr(), rhs.data_ptr(), _params((nx, ny), (nx, ny)), cycles, nit,
                                  u.data_ptr(), 1, 1, scratch.data_ptr(), scratch.numel(), 0) == 0
        launches.append(lib.csg_kernel_launches() - before)
    torch.cuda.synchronize()
    # two legs, or the half-sweeps of both ways, residual, restriction and prolongation; and the resident cycle
    assert launches[1] - launches[0] == (2 if legs else 4 * nit + 3) + 1
    assert torch.equal(u, _separate(lib, code, hess, rhs, start, 1, nit))


@pytest.mark.parametrize(
    "dtype, nx, ny, batch, nit, resident",
    [
        (torch.float64, 256, 128, 7, 3, True),  # one wave of clusters of 16
        (torch.float64, 256, 128, 8, 3, True),
        (torch.float64, 256, 128, 64, 3, False),
        (torch.float64, 256, 113, 32, 1, False),
        (torch.float32, 256, 128, 14, 3, True),
        (torch.float32, 256, 128, 32, 3, False),
        (torch.float32, 64, 33, 32, 2, True),
        (torch.float32, 64, 33, 600, 2, False),
        (torch.float64, 32, 17, 74, 1, True),
        (torch.float64, 32, 17, 600, 1, False),
        (torch.float64, 32, 16, 600, 3, True),  # one CTA per grid
        (torch.float64, 8, 4, 4096, 1, True),
        (torch.float64, 512, 256, 16, 2, False),
    ],
)
def test_batches_of_several_waves(native_library, dtype, nx, ny, batch, nit, resident):
    """V-cycles of batches on either side of where resident clusters take too many waves: one launch, or
    finer levels above the resident ones, with the separate kernels' results."""

    lib = native_library
    code = 1 if dtype == torch.float64 else 0
    hess, rhs, start = _problem(nx, ny, batch, dtype, "plain")
    scratch = torch.empty(lib.csg_dartel_scratch_bytes(code, batch, nx, ny), dtype=torch.uint8, device="cuda")
    launches = []
    for cycles in (0, 2):
        u = start.clone()
        before = lib.csg_kernel_launches()
        assert lib.csg_dartel_fmg(code, batch, nx, ny, hess.data_ptr(), rhs.data_ptr(), _params((nx, ny), (nx, ny)), cycles, nit,
                                  u.data_ptr(), 1, 1, scratch.data_ptr(), scratch.numel(), 0) == 0
        launches.append(lib.csg_kernel_launches() - before)
    torch.cuda.synchronize()
    assert (launches[1] - launches[0] == 1) == resident
    assert torch.equal(u, _separate(lib, code, hess, rhs, start, 2, nit))


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize(
    "nx, ny, batch, silent",
    [(64, 32, 1, 0), (64, 32, 3, 3), (64, 33, 40, 1), (128, 65, 2, 8), (256, 128, 1, 15), (256, 128, 2, 0), (512, 256, 1, 7)],
)
def test_waits_that_run_out_report_it(native_library, dtype, nx, ny, batch, silent):
    """A CTA that sends no edge rows: its neighbours' waits run out, every kernel returns, all rows of all maps are
    NaN and the status word tells; the next solve on the same scratch is whole again."""

    lib = native_library
    code = 1 if dtype == torch.float64 else 0
    hess, rhs, start = _problem(nx, ny, batch, dtype, "plain")
    params = _params((nx, ny), (nx, ny))
    scratch = torch.empty(lib.csg_dartel_scratch_bytes(code, batch, nx, ny), dtype=torch.uint8, device="cuda")

    def status():
        word = ctypes.c_int(1)
        assert lib.csg_read_status(scratch.data_ptr(), 0, ctypes.addressof(word), 0) == 0
        return word.value

    def solve(timeout, rank):
        u = start.clone()
        assert lib.csg_selftest_exchange_timeout(code, batch, nx, ny, hess.data_ptr(), rhs.data_ptr(), params, 2, 2,
                                                 u.data_ptr(), scratch.data_ptr(), scratch.numel(), timeout, rank, 0) == 0
        return u

    lost = solve(0.005, silent)
    assert status() == -3  # CSG_ERR_TIMEOUT
    assert torch.isnan(lost).all()
    whole = solve(2.0, -1)
    assert status() == 0
    u = start.clone()
    assert lib.csg_dartel_fmg(code, batch, nx, ny, hess.data_ptr(), rhs.data_ptr(), params, 2, 2, u.data_ptr(), 1, 1,
                              scratch.data_ptr(), scratch.numel(), 0) == 0
    assert status() == 0
    assert torch.isfinite(u).all() and torch.equal(u, whole)


def test_a_lost_solve_raises():
    """The Python layer turns a solve's status word into an error, and a solve's own is zero."""

    from cat_surface_gpu_b200.surface_warp import check_solve, solve_dartel_maps

    sheets = torch.rand(2, 1, 16, 32, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(0))
    for graph in (False, True):
        result = solve_dartel_maps(sheets[0], sheets[1], loop=2, its=1, cuda_graph=graph)
        check_solve(result.status)
        with pytest.raises(RuntimeError, match="ran out"):
            check_solve(result.status - 3)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nx, ny", [(4, 65536), (16, 70000), (8, 100001)])
def test_legs_of_very_tall_grids(native_library, dtype, nx, ny):
    """Grids of so many rows that the products of row numbers pass 32 bits."""

    lib = native_library
    code = 1 if dtype == torch.float64 else 0
    hess, rhs, start = _problem(nx, ny, 1, dtype, "plain")
    scratch = torch.empty(lib.csg_dartel_scratch_bytes(code, 1, nx, ny), dtype=torch.uint8, device="cuda")
    u = start.clone()
    assert lib.csg_dartel_fmg(code, 1, nx, ny, hess.data_ptr(), rhs.data_ptr(), _params((nx, ny), (nx, ny)), 1, 3, u.data_ptr(),
                              1, 1, scratch.data_ptr(), scratch.numel(), 0) == 0
    torch.cuda.synchronize()
    assert torch.equal(u, _separate(lib, code, hess, rhs, start, 1, 3))


def _operands(kind, count, rng):
    """(numerators [2, count], first diagonal entries [count]): exponents and mantissas of the point systems."""

    def mantissa(shape):
        special = np.array([1.0, 2.0 - 2.0**-52, 1.0 + 2.0**-52, 1.5, 2.0 - 2.0**-51])  # power of two, all ones, ...
        m = 1.0 + rng.random(shape)
        return np.where(rng.random(shape) < 0.3, rng.choice(special, shape), m) * rng.choice([-1.0, 1.0], shape)

    if kind == "inside":
        ea, ed = rng.integers(-500, 500, (2, count)), rng.integers(-400, 401, count)
    elif kind == "edges":  # of the windows in which the reciprocal is used, on both sides
        ea = rng.choice([-502, -501, -500, -499, 498, 499, 500, 501], (2, count))
        ed = rng.choice([-402, -401, -400, -399, 398, 399, 400, 401], count)
    else:
        ea, ed = rng.integers(-1073, 1024, (2, count)), rng.integers(-1073, 1024, count)
    det = np.ldexp(mantissa(count), ed)
    first = det / 1.0000000001  # the determinant's rounding takes it back to det, or next to it
    for near in (np.nextafter(first, 0.0), np.nextafter(first, 2.0 * first)):
        first = np.where((first * 1.0000000001 != det) & (near * 1.0000000001 == det), near, first)
    numerators = np.ldexp(mantissa((2, count)), ea)
    if kind == "outside":
        numerators[:, ::97] = 0.0
        first[::89] = 0.0
    return numerators, first


@pytest.mark.parametrize("kind", ["inside", "edges", "outside"])
def test_quotients_equal_the_division(native_library, kind):
    """Point systems of one point without weights: the resident cycle's quotients by the kept reciprocal against
    csg_dartel_relax's divisions, bit for bit."""

    lib = native_library
    batch, rng = 65535, np.random.default_rng(len(kind))
    params = (ctypes.c_double * 5)(1.0, 1.0, 0.0, 0.0, 0.0)
    scratch = torch.empty(lib.csg_dartel_scratch_bytes(1, batch, 1, 1), dtype=torch.uint8, device="cuda")
    hits = 0
    with np.errstate(over="ignore", under="ignore"):
        for _ in range(16):
            numerators, first = _operands(kind, batch, rng)
            # det = first * 1 * 1.0000000001; quotients numerators[0] / det and (first * numerators[1]) / det
            hess = torch.as_tensor(np.stack((first, np.ones(batch), np.zeros(batch)), 1), device="cuda").contiguous()
            rhs = torch.as_tensor(np.ascontiguousarray(numerators.T), device="cuda")
            plain, kept = torch.zeros_like(rhs), torch.zeros_like(rhs)
            assert lib.csg_dartel_relax(1, batch, 1, 1, hess.data_ptr(), rhs.data_ptr(), params, 1, plain.data_ptr(), 0) == 0
            assert lib.csg_dartel_fmg(1, batch, 1, 1, hess.data_ptr(), rhs.data_ptr(), params, 1, 1, kept.data_ptr(), 1, 1,
                                      scratch.data_ptr(), scratch.numel(), 0) == 0
            torch.cuda.synchronize()
            same = (plain.view(torch.int64) == kept.view(torch.int64)) | (plain.isnan() & kept.isnan())
            assert bool(same.all()), (rhs[~same.all(1)][:3], hess[~same.all(1)][:3])
            det = first * 1.0000000001
            hits += int(np.count_nonzero(np.frexp(np.abs(det))[0] == 1.0 - 2.0**-53))
    assert hits > 1000  # divisors of all ones were among them
