"""The dataflow sweeps' published words at the sizes where their paths change.

Meshes whose vertices have more ring members or more faces than a group has
lanes, projection periods that take each form of the epoch test, and every
lane count: all bit-identical to the oracle's sequential restatement.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from cat_surface_gpu_b200 import synthetic
from oracle import areal as oracle

pytestmark = pytest.mark.gpu


def _mesh(kind):
    """(vertices, faces): closed, with an apex of nine faces, or with faces listed more than once."""

    vertices, faces = synthetic.folded_icosphere(2, seed=5)
    if kind == "apex":  # a vertex of nine faces (ten ring members): a fan over a nine-sided hole
        angle = 2 * np.pi * np.arange(9) / 9
        rim = np.stack((np.cos(angle), np.sin(angle), 0.1 * np.sin(3 * angle)), 1)
        vertices = np.concatenate(([[0.1, 0.0, 1.0], [0.0, 0.1, -1.0]], rim)) * 40.0
        turn = np.arange(9)
        up = np.stack((np.zeros(9), 2 + turn, 2 + (turn + 1) % 9), 1)
        down = np.stack((np.ones(9), 2 + (turn + 1) % 9, 2 + turn), 1)
        faces = np.concatenate((up, down))
    elif kind == "repeated":  # nine faces round vertices with seven ring members
        at = int(np.bincount(faces.reshape(-1)).argmax())
        faces = np.concatenate((faces, faces[(faces == at).any(axis=1)][:3]))
    return np.asarray(vertices, dtype=np.float32), np.ascontiguousarray(faces, dtype=np.int32)


@pytest.mark.parametrize("kind", ["closed", "apex", "repeated"])
@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("arithmetic", ["cat", "fp32"])
@pytest.mark.parametrize("project_every", [0, 1, 2, 7, 2**27])
def test_sweeps_equal_the_oracle(native_library, kind, lanes, arithmetic, project_every):
    from cat_surface_gpu_b200.gifti import GiftiMesh
    from cat_surface_gpu_b200.surf2sphere import Surf2SphereTopology, run_areal_smoothing_cuda

    vertices, faces = _mesh(kind)
    radius = float(np.sqrt(np.max(np.sum(vertices.astype(np.float64) ** 2, axis=1))))
    topology = Surf2SphereTopology.plan_only(GiftiMesh(vertices, faces))
    launch = {"n_ctas": 3, "threads_per_cta": 64, "lanes_per_vertex": lanes}
    got, _ = run_areal_smoothing_cuda(vertices, faces, topology, iterations=35, project_every=project_every,
                                      radius=radius, arithmetic=arithmetic, launch=launch)
    want = oracle.areal_sweeps(vertices, faces, iterations=35, project_every=project_every, radius=radius,
                               arithmetic=arithmetic)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("kind", ["closed", "apex"])
@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("stop_at", [1, 2, 3])
def test_stage_passes_equal_the_oracle(native_library, kind, lanes, stop_at):
    """Rings of at most and of more members than lanes, through smoothing, inflation and selected passes."""

    from cat_surface_gpu_b200.gifti import GiftiMesh
    from cat_surface_gpu_b200.surf2sphere import Surf2SphereTopology, run_surf2sphere_preprocess_cuda
    from oracle import preprocess as oracle_pre

    vertices, faces = _mesh(kind)
    topology = Surf2SphereTopology.plan_only(GiftiMesh(vertices, faces))
    launch = {"n_ctas": 3, "threads_per_cta": 64, "lanes_per_vertex": lanes}
    got, _ = run_surf2sphere_preprocess_cuda(vertices, faces, topology, stop_at=stop_at, desired_surface_area=1.0,
                                             launch=launch)
    want = oracle_pre.preprocess(vertices, faces, stop_at=stop_at)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n, seed", [(60, 0), (150, 1), (300, 3)])  # rings of at most eight members, and of nine
@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("batch", [1, 3])
def test_depth_sor_equals_the_oracle(native_library, n, seed, lanes, batch):
    from cat_surface_gpu_b200.rotation_feature import DepthTopology, depth_potential
    from oracle import depth as oracle_depth

    vertices, faces = synthetic.folded_hull(n, seed)
    surfaces = np.stack([vertices * np.float32(1.0 + 0.25 * b) for b in range(batch)])
    topology = DepthTopology.build(faces, n, torch.device("cuda:0"))
    groups = oracle_depth.colour_groups(faces, n)
    launch = {"n_ctas": 3, "threads_per_cta": 64, "lanes_per_row": lanes}
    for sweeps in (1, 40):
        got, _, residual = depth_potential(torch.as_tensor(surfaces, device="cuda:0"), topology, max_iter=sweeps,
                                           launch=launch)
        for b in range(batch):
            want, _, want_residual = oracle_depth.System(surfaces[b], faces).sor(groups, sweeps)
            np.testing.assert_array_equal(got[b].cpu().numpy(), want)
            assert residual[b] == want_residual


@pytest.mark.parametrize("n", [60, 96])  # 96 vertices: the vectors that the words lie over leave no gap
@pytest.mark.parametrize("batch", [1, 2])
def test_depth_scratch_needs_the_alignment_of_a_double(native_library, monkeypatch, n, batch):
    """Scratch of just the size asked for, 8 bytes off a multiple of 16: the same values."""

    from cat_surface_gpu_b200 import rotation_feature

    vertices, faces = synthetic.folded_hull(n, 2)
    surfaces = torch.as_tensor(np.stack([vertices * np.float32(1.0 + 0.25 * b) for b in range(batch)]), device="cuda:0")
    topology = rotation_feature.DepthTopology.build(faces, n, torch.device("cuda:0"))
    empty = torch.empty

    def off_by_eight(*size, dtype=None, **options):
        if dtype is torch.uint8:
            return empty(size[0] + 8, dtype=dtype, **options)[8:]
        return empty(*size, dtype=dtype, **options)

    want = rotation_feature.depth_potential(surfaces, topology, max_iter=25)
    monkeypatch.setattr(rotation_feature.torch, "empty", off_by_eight)
    got = rotation_feature.depth_potential(surfaces, topology, max_iter=25)
    assert torch.equal(got[0], want[0]) and got[1:] == want[1:]


def _tube(sides, rows):
    """(vertices, faces) of a long closed tube, numbered along it: thousands of dependency levels, two vertices of
    ``sides`` faces."""

    angle = 2 * np.pi * np.arange(sides) / sides
    z = 0.05 * (np.arange(rows) - (rows - 1) / 2)
    radius = 30 + 0.1 * (np.arange(rows) % 7)
    rings = np.stack((radius[:, None] * np.cos(angle), radius[:, None] * np.sin(angle), np.repeat(z[:, None], sides, 1)), -1)
    vertices = np.concatenate((rings.reshape(-1, 3), [[0, 0, z[0] - 5], [0, 0, z[-1] + 5]]))
    here, there = np.arange(sides), (np.arange(sides) + 1) % sides
    low, high = np.stack((here, there, here + sides), 1), np.stack((there, there + sides, here + sides), 1)
    walls = (np.concatenate((low, high))[None] + sides * np.arange(rows - 1)[:, None, None]).reshape(-1, 3)
    n, top = sides * rows, sides * (rows - 1)
    ends = np.concatenate((np.stack((np.full(sides, n), there, here), 1),
                           np.stack((np.full(sides, n + 1), top + here, top + there), 1)))
    return vertices.astype(np.float32), np.concatenate((walls, ends)).astype(np.int32)


# Launches whose shared memory the 8-byte words' layout just held for two CTAs to an SM.
@pytest.mark.parametrize("arithmetic", ["cat", "fp32"])
def test_sweeps_of_two_large_ctas_to_an_sm(native_library, arithmetic):
    from cat_surface_gpu_b200.autotune import sm_count
    from cat_surface_gpu_b200.gifti import GiftiMesh
    from cat_surface_gpu_b200.surf2sphere import Surf2SphereTopology, run_areal_smoothing_cuda

    vertices, faces = _tube(9, 4080)
    topology = Surf2SphereTopology.plan_only(GiftiMesh(vertices, faces))
    launch = {"n_ctas": 2 * sm_count(), "threads_per_cta": 512, "lanes_per_vertex": 8}
    got, _ = run_areal_smoothing_cuda(vertices, faces, topology, iterations=4, project_every=2, radius=60.0,
                                      arithmetic=arithmetic, launch=launch)
    np.testing.assert_array_equal(got, oracle.areal_sweeps(vertices, faces, iterations=4, project_every=2, radius=60.0,
                                                           arithmetic=arithmetic))


def test_stage_passes_of_two_large_ctas_to_an_sm(native_library):
    from cat_surface_gpu_b200.autotune import sm_count
    from cat_surface_gpu_b200.gifti import GiftiMesh
    from cat_surface_gpu_b200.surf2sphere import Surf2SphereTopology, run_surf2sphere_preprocess_cuda
    from oracle import preprocess as oracle_pre

    vertices, faces = _tube(16, 4480)
    topology = Surf2SphereTopology.plan_only(GiftiMesh(vertices, faces))
    launch = {"n_ctas": 2 * sm_count(), "threads_per_cta": 512, "lanes_per_vertex": 16}
    got, _ = run_surf2sphere_preprocess_cuda(vertices, faces, topology, stop_at=1, desired_surface_area=1.0, launch=launch)
    np.testing.assert_array_equal(got, oracle_pre.preprocess(vertices, faces, stop_at=1))


def test_depth_sor_of_two_large_ctas_to_an_sm(native_library):
    from cat_surface_gpu_b200.autotune import sm_count
    from cat_surface_gpu_b200.rotation_feature import DepthTopology, depth_potential
    from cat_surface_gpu_b200.surface_stencil import resampling_sphere

    points, faces = resampling_sphere(4)
    n = points.shape[0]
    topology = DepthTopology.build(faces, n, torch.device("cuda:0"))
    surfaces = torch.as_tensor(np.stack([points * (40.0 + b) for b in range(64)]).astype(np.float32), device="cuda:0")
    launch = {"n_ctas": 2 * sm_count(), "threads_per_cta": 512, "lanes_per_row": 4}
    got, _, _ = depth_potential(surfaces, topology, max_iter=20, launch=launch)
    for b in (0, 63):
        want, _, _ = depth_potential(surfaces[b], topology, max_iter=20)
        assert torch.equal(got[b], want[0])
