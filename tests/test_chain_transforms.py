"""The hop transforms that engine.build_chain takes: a 3-vector and a 3x3
matrix per hop, the matrix also flat, both also longer (the first three and
nine elements count); anything shorter is refused."""

import numpy as np
import pytest

from acc_gb300 import _native as nat
from acc_gb300.components.optics.arm import Arm
from acc_gb300.engine import build_chain, chain_for_instrument
from acc_gb300.instrument import (calcTransformations, instrument,
                                  relative_transform)
from acc_gb300.memory import HostBinder

ROT = np.arange(1.0, 10.0).reshape(3, 3)
OFF = np.array([0.5, -1.0, 2.0])


def _hop(off, rot):
    ch = build_chain([Arm("a"), Arm("b")], [off], [rot], HostBinder())
    return (list(ch.off[1]), list(ch.foff[1]), list(ch.rot[1]),
            list(ch.frot[1]), ch.comp[1].flags & nat.FLAG_IDENTITY_ROT)


@pytest.mark.parametrize("off,rot", [
    (OFF, ROT), (OFF.tolist(), ROT.tolist()), (OFF, ROT.reshape(9)),
    (OFF, ROT.reshape(1, 9)), (np.append(OFF, 7.0), np.arange(1.0, 17.0)),
    (OFF.astype(np.float32), np.asfortranarray(ROT)),
], ids=["plain", "lists", "flat", "row", "longer", "other_layouts"])
def test_accepted_forms(off, rot):
    want = list(OFF), list(ROT.reshape(9))
    assert _hop(off, rot) == (want[0], want[0], want[1], want[1], 0)


def test_identity_is_flagged():
    assert _hop(OFF, np.eye(3))[4] == nat.FLAG_IDENTITY_ROT
    assert _hop(OFF, np.eye(3).reshape(9))[2] == list(np.eye(3).reshape(9))


@pytest.mark.parametrize("off,rot", [
    (5.0, ROT), ([5.0], ROT), (OFF.reshape(3, 1), ROT), (OFF[:2], ROT),
    (OFF, 3.0), (OFF, ROT[:2]),
], ids=["scalar", "one", "column", "two", "number", "two_rows"])
def test_refused_forms(off, rot):
    with pytest.raises((ValueError, IndexError, TypeError)):
        _hop(off, rot)


def test_hops_of_an_instrument_are_the_relative_transforms():
    ins = instrument("turned")
    for k in range(3):
        ins.append(Arm(f"a{k}"), position=(0.1 * k, -0.2, 1.0 * k),
                   orientation=(10.0 * k, 5.0, -20.0 * k))
    offs, rots = calcTransformations(ins)
    assert offs.shape == (2, 3) and rots.shape == (2, 3, 3)
    for i in range(2):
        off, rot = relative_transform(ins.geometer, *ins.components[i:i + 2])
        np.testing.assert_array_equal(offs[i], off)
        np.testing.assert_array_equal(rots[i], rot)


def test_a_single_component_needs_no_place():
    ins = instrument("single")
    ins.components.append(Arm("a"))
    assert calcTransformations(ins)[0].shape == (0, 3)
    assert chain_for_instrument(ins, HostBinder()).ncomp == 1
