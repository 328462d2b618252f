"""Device assembly in slices of equal list length (gpu_elastic.cu) against the host assembly: the same bits, on
meshes whose lists are of every length the slices pad, end or leave empty."""
import numpy as np
import pytest

from fem_gb300 import lina, problems
from tests.conftest import gpu_available


def fan(spokes):
    """A hub with `spokes` triangles around it: lists of 1, 2 and `spokes` contributions."""
    t = 2 * np.pi * np.arange(spokes) / spokes
    xy = np.concatenate([[[0.0, 0.0]], np.stack([np.cos(t), np.sin(t)], axis=1)])
    k = np.arange(spokes)
    return xy, np.stack([np.zeros(spokes, int), 1 + k, 1 + (k + 1) % spokes], axis=1).astype(np.int32)


MESHES = {
    "triangle": lambda: (np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]]), np.array([[0, 1, 2]], np.int32)),
    "free_node": lambda: (np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0], [5.0, 5.0]]), np.array([[0, 1, 2]], np.int32)),
    "fan5": lambda: fan(5),
    "fan40": lambda: fan(40),
    "grid5": lambda: problems.elastic_mesh(5)[:2],
    "grid34": lambda: problems.elastic_mesh(34)[:2],
    "delaunay": lambda: problems.delaunay_mesh(900, 4),
}


@pytest.mark.gpu
@pytest.mark.skipif(not gpu_available(), reason="no CUDA device")
@pytest.mark.parametrize("kind", [lina.P1_LAPLACE, lina.P1_ELASTIC])
@pytest.mark.parametrize("mesh", MESHES)
def test_device_assembly_equals_host(mesh, kind):
    xy, tri = MESHES[mesh]()
    fixed = np.array([0], np.int32)
    p1 = lina.P1Assembly(kind, xy, tri, nu=0.3, fixed_dof=fixed, fixed_val=[0.25])
    rng = np.random.default_rng(1)
    for coef in (rng.uniform(0.5, 2.0, len(tri)), -np.exp(rng.standard_normal(len(tri)))):
        p1.assemble(coef)
        ref = lina.p1_assemble_host(kind, xy, tri, coef, nu=0.3, fixed_dof=fixed, fixed_val=[0.25])
        for a, b in zip(p1.system(), ref):
            assert np.array_equal(a, b) and np.array_equal(np.signbit(a), np.signbit(b))
