"""A minimal instrument and geometer.

Restates what mcvine.instrument() / mcni.Instrument provide to the
reference's run_script (acc/run_script.py:141-162): a list of components,
each with a position and orientation, absolute or relative to an earlier
component, and the offset/rotation pairs that take a neutron from one
component's frame to the next one's (r' = R (r - o), v' = R v;
acc/neutron.py:18-23).

Orientation (rx, ry, rz) in degrees uses the McStas rotation convention
(rotate about x, then y, then z; the matrix maps parent-frame coordinates to
the rotated frame's).  The reference's own test
(tests/test_coord_transform_among_comps.py:25-57) pins the single-axis cases.
"""

import math

import numpy as np


def rotation_matrix(orientation):
    """Parent-frame -> local-frame coordinate matrix for (rx, ry, rz) deg."""
    rx, ry, rz = (math.radians(float(a)) for a in orientation)
    cx, sx = math.cos(rx), math.sin(rx)
    cy, sy = math.cos(ry), math.sin(ry)
    cz, sz = math.cos(rz), math.sin(rz)
    return np.array([
        [cy * cz, sx * sy * cz + cx * sz, sx * sz - cx * sy * cz],
        [-cy * sz, cx * cz - sx * sy * sz, sx * cz + cx * sy * sz],
        [sy, -sx * cy, cx * cy],
    ])


class Geometer:
    def __init__(self):
        self._abs = {}

    def register(self, comp, position, orientation, relative_to):
        M_rel = rotation_matrix(orientation)
        p = np.asarray(position, dtype=float)
        if relative_to is None:
            P, M = p, M_rel
        else:
            Pr, Mr = self._abs[id(relative_to)]
            P = Pr + Mr.T @ p
            M = M_rel @ Mr
        self._abs[id(comp)] = (P, M)

    def position(self, comp):
        return self._abs[id(comp)][0]

    def rotation(self, comp):
        return self._abs[id(comp)][1]

    def orientation(self, comp):
        return self.rotation(comp)


class Instrument:
    """Ordered components with placements (mcni.Instrument stand-in)."""

    def __init__(self, name="instrument"):
        self.name = name
        self.components = []
        self.geometer = Geometer()

    def append(self, component, position=(0, 0, 0), orientation=(0, 0, 0),
               relativeTo=None):
        if relativeTo is not None and not any(
                relativeTo is c for c in self.components):
            raise ValueError("relativeTo must be a component already appended")
        self.components.append(component)
        self.geometer.register(component, position, orientation, relativeTo)
        return component

    def __repr__(self):
        names = ", ".join(getattr(c, "name", "?") for c in self.components)
        return f"Instrument({names})"


def instrument(name="instrument"):
    return Instrument(name)


def _hop(a, b, off, rot):
    """Into off and rot, what takes a neutron from frame a to frame b (each a
    position and a rotation)."""
    np.matmul(a[1], b[0] - a[0], out=off)
    np.matmul(b[1], a[1].T, out=rot)
    return off, rot


def relative_transform(geometer, a, b):
    """(offset, rotmat) taking a neutron from a's frame to b's frame."""
    return _hop((geometer.position(a), geometer.rotation(a)),
                (geometer.position(b), geometer.rotation(b)),
                np.empty(3), np.empty((3, 3)))


def calcTransformations(instrument):
    """Offsets (n-1, 3) and rotation matrices (n-1, 3, 3) between
    consecutive components (acc/run_script.py:141-162)."""
    comps = instrument.components
    n = max(len(comps) - 1, 0)
    offs, rots = np.empty((n, 3)), np.empty((n, 3, 3))
    if n:  # (a component without a neighbour need not have been placed)
        g = instrument.geometer
        placed = [(g.position(c), g.rotation(c)) for c in comps]
        for i in range(n):
            _hop(placed[i], placed[i + 1], offs[i], rots[i])
    return offs, rots


def applyTransformation(position, velocity, rotmat, offset):
    """r' = R (r - o), v' = R v on NumPy 3-vectors, in place
    (acc/neutron.py:18-23)."""
    r = rotmat @ (np.asarray(position, dtype=float) - offset)
    v = rotmat @ np.asarray(velocity, dtype=float)
    position[:] = r
    velocity[:] = v
