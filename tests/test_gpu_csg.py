"""FP64 intersections of CSG shapes (the hits kept are those on the node's
border, which FP32 settles for points far from the other operand's surface)
against the CPU oracle's: identical hit counts and times within 1e-12 of the
ray's crossing time.  Rays aim at random points of the shape's box, along the
axes among them, and start far away, inside, on a surface and next to the
operands' common edges."""

import numpy as np
import pytest
import torch

from acc_gb300 import engine
from acc_gb300.components.samples.homogeneous_single_scatterer import factory
from acc_gb300.geometry import (Block, Cylinder, Difference, Intersection,
                                Sphere, Union)
from acc_gb300.kernels import IsotropicKernel
from acc_gb300.memory import HostBinder

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    torch.cuda.init()
    yield


OPERANDS = {
    "hollow": (Cylinder(0.02, 0.06), Cylinder(0.01, 0.07)),
    # the caps of both cylinders coincide: every cap hit is uncertain
    "flush": (Cylinder(0.02, 0.06), Cylinder(0.01, 0.06)),
    "spheres": (Sphere(0.03), Sphere(0.029999)),
    "mixed": (Block(0.04, 0.05, 0.06), Cylinder(0.022, 0.055)),
    "ball_in_box": (Sphere(0.03), Block(0.05, 0.05, 0.05)),
}


def _rays(n, seed):
    r = np.random.default_rng(seed)
    target = r.uniform(-0.035, 0.035, (n, 3))
    v = r.normal(size=(n, 3))
    v[: n // 8] = np.eye(3)[r.integers(0, 3, n // 8)]
    v *= (r.uniform(300.0, 4000.0, n) / np.linalg.norm(v, axis=1))[:, None]
    back = r.choice([0.0, 1e-5, 0.01, 2.0], n) / 1000.0
    x = target - v * back[:, None]
    # on the radius of a cylinder or sphere
    k = slice(n // 2, n // 2 + n // 8)
    x[k, :2] *= (0.02 / np.linalg.norm(x[k, :2], axis=1))[:, None]
    return np.concatenate([x, v], axis=1)


@pytest.mark.parametrize("op", [Difference, Union, Intersection])
@pytest.mark.parametrize("name", list(OPERANDS))
def test_fp64_csg_hits_match_the_oracle(name, op):
    from oracle import binding as O
    comp = factory(op(*OPERANDS[name]), IsotropicKernel(1.0, 1.0))("s")
    rays = _rays(4001, 12)
    ts, cnt = engine.intersect(comp, rays)
    c = comp.to_struct(HostBinder())
    for i, ray in enumerate(rays):
        ref = np.asarray(O.intersect(c, ray), dtype=float).reshape(-1)
        assert cnt[i] == len(ref), (i, ray)
        scale = 0.1 / np.linalg.norm(ray[3:]) + np.abs(ref).max(initial=0.0)
        assert np.abs(ts[i, :len(ref)] - ref).max(initial=0.0) <= 1e-12 * scale


@pytest.mark.parametrize("name", ["hollow", "thin", "spheres"])
@pytest.mark.parametrize("op", [Difference, Union, Intersection])
@pytest.mark.parametrize("far", [20.0, 50.0, 200.0, 500.0])
def test_fp64_csg_hits_of_distant_rays_match_the_oracle(name, op, far):
    """Rays from `far` metres: a cylinder's side hits miss their surface by up
    to 4 u far^2 / R there, so from some 20 m on some of them are off the
    border to within 1e-10, and are left out as the reference leaves them
    out."""
    from oracle import binding as O
    shapes = dict(OPERANDS, thin=(Cylinder(0.004, 0.06), Cylinder(0.002, 0.07)))
    comp = factory(op(*shapes[name]), IsotropicKernel(1.0, 1.0))("s")
    rays = _rays(2001, 13)
    v = rays[:, 3:]
    rays[:, :3] -= v * (far / np.linalg.norm(v, axis=1))[:, None]
    ts, cnt = engine.intersect(comp, rays)
    c = comp.to_struct(HostBinder())
    for i, ray in enumerate(rays):
        ref = np.asarray(O.intersect(c, ray), dtype=float).reshape(-1)
        assert cnt[i] == len(ref), (i, ray)
        scale = np.abs(ref).max(initial=0.0)
        assert np.abs(ts[i, :len(ref)] - ref).max(initial=0.0) <= 1e-12 * scale
