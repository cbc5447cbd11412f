"""The wave kernels (chains with guides: fronts, bounces and tails of full
warps, csrc/wave.cuh) against the one-neutron-per-thread kernels (launch
variant "thread") on the same streams.

FP64: the same operations in the same order on every neutron that reaches a
tally, so identical counts and sums within 1e-12 (the order of additions
differs).  That also checks the FP32 screen of the FP64 front: it may drop
only neutrons that end at the first guide's opening or first reflection.
FP32: the kernels may contract different multiply-adds, which moves a
coordinate within an ulp of a bin edge: at most 1e-5 of the entries (or two)
move, sums within 1e-6.
"""

import numpy as np
import pytest
import torch

from acc_gb300 import engine, instruments
from acc_gb300.components.monitors.energy_monitor import Energy_monitor
from acc_gb300.components.monitors.psd_monitor import PSD_monitor
from acc_gb300.components.optics.guide import Guide
from acc_gb300.components.optics.slit import Slit
from acc_gb300.components.samples.homogeneous_single_scatterer import factory
from acc_gb300.components.sources.source_simple import Source_simple
from acc_gb300.geometry import Sphere
from acc_gb300.instrument import instrument
from acc_gb300.kernels import IsotropicKernel
from helpers import gpu_tallies

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    torch.cuda.init()
    yield


def _psd(name):
    return PSD_monitor(name, xmin=-0.04, xmax=0.04, ymin=-0.04, ymax=0.04,
                       nx=40, ny=40, filename=name + ".h5")


def _chain(source, guides, between=None, tail=True, offset=(0.0, 0.0)):
    """source -> guides 1 mm apart (`between`: components after the first)
    -> PSD and energy monitor, or nothing after the last guide."""
    ins = instrument("wave")
    src = dict(radius=0.05, dist=1.0, xw=0.05, yh=0.05, E0=52.5, dE=47.5)
    if source.get("Lambda0"):
        src.pop("E0"), src.pop("dE")
        src.update(E0=0, dE=0)
    src.update(source)
    ins.append(Source_simple("src", **src), position=(0, 0, 0))
    z = src["dist"]
    for i, (w1, w2, length) in enumerate(guides):
        ins.append(Guide(f"g{i}", w1=w1, h1=w1, w2=w2, h2=w2, l=length,
                         **instruments.COATING),
                   position=(offset[0], offset[1], z))
        z += length + 1e-3
        if i == 0:
            for c in between or ():
                ins.append(c, position=(0, 0, z))
                z += 0.05
    if tail:
        ins.append(_psd("psd"), position=(0, 0, z))
        ins.append(Energy_monitor("e", xmin=-0.04, xmax=0.04, ymin=-0.04,
                                  ymax=0.04, Emin=0.0, Emax=100.0, nchan=50,
                                  filename="e.h5"), position=(0, 0, z))
    return ins


STRAIGHT = (0.05, 0.05, 4.0)
CHAINS = {
    "guide_chain": instruments.guide_chain,
    # the first guide tapers: both walls of a pair may be ahead at once
    "taper_first": lambda: _chain({}, [(0.05, 0.01, 3.0), (0.02, 0.02, 2.0)]),
    "widening": lambda: _chain({}, [(0.03, 0.06, 3.0)]),
    # most neutrons survive the first reflection: nothing to screen
    "slow": lambda: _chain(dict(Lambda0=15.0, dLambda=4.0), [STRAIGHT] * 2),
    "rectangle_offset": lambda: _chain(
        dict(radius=0, width=0.02, height=0.06, dist=2.0, xw=0.08, yh=0.03),
        [STRAIGHT], offset=(0.004, -0.01)),
    "wide_source": lambda: _chain(dict(radius=0.3, xw=0.2, yh=0.2),
                                  [STRAIGHT]),
    # components between the guides: a monitor, a slit, a sample that draws
    "between": lambda: _chain(
        {}, [STRAIGHT, (0.06, 0.04, 2.0)],
        between=[_psd("mid"), Slit("slit", width=0.045, height=0.045),
                 factory(Sphere(0.02), IsotropicKernel(5.0, 20.0))("s")]),
    "three_guides": lambda: _chain({}, [(0.05, 0.05, 1.0)] * 3),
    "no_tail": lambda: _chain({}, [STRAIGHT], between=[], tail=False),
    "powder": lambda: instruments.powder_banked(ntubes=4, npixels=8, ntof=25),
}
COUNTS = [1, 31, 33, 2047, 300_001]


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("name", list(CHAINS))
def test_wave_kernel_equals_thread_kernel(name, n):
    for ft in ("float64", "float32"):
        a, b = CHAINS[name](), CHAINS[name]()
        sa = engine.run_instrument(a, n, seed=77, first=5, floattype=ft)
        sb = engine.run_instrument(b, n, seed=77, first=5, floattype=ft,
                                   variant="thread")
        assert sa.processed == sb.processed == n
        assert sa.nonfinite == sb.nonfinite
        for ta, tb in zip(gpu_tallies(a).values(), gpu_tallies(b).values()):
            if ft == "float64":
                np.testing.assert_array_equal(ta[0], tb[0])
                np.testing.assert_allclose(ta[1:], tb[1:], rtol=1e-12,
                                           atol=1e-300)
            else:
                moved = np.abs(ta[0] - tb[0]).sum() / 2
                assert moved <= max(2, 1e-5 * tb[0].sum())
                if n == COUNTS[-1]:
                    assert ta[1].sum() == pytest.approx(tb[1].sum(), rel=1e-6)
    if n == COUNTS[-1] and name != "no_tail":
        assert tb[0].sum() > 0


@pytest.mark.parametrize("variant", ["regen", "regen_noqueue"])
def test_wave_kernel_variants_and_launch_shapes(variant):
    """Launch variant 3 runs the tail without waiting for a warp of neutrons;
    a single small block takes every neutron."""
    out = []
    for v, tpb, blocks in (("thread", None, None), (variant, None, None),
                           (variant, 32, 1)):
        ins = instruments.guide_chain()
        engine.run_instrument(ins, 20_011, seed=3, floattype="float64",
                              variant=v, threads_per_block=tpb, blocks=blocks)
        out.append(list(gpu_tallies(ins).values()))
    for o in out[1:]:
        for ta, tb in zip(o, out[0]):
            np.testing.assert_array_equal(ta[0], tb[0])
            np.testing.assert_allclose(ta[1:], tb[1:], rtol=1e-12,
                                       atol=1e-300)
