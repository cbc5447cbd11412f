"""Guide chains away from the usual coatings, sources and launches: the wave
kernels (csrc/wave.cuh) against the one-neutron-per-thread kernels and the
CPU oracle on the same streams.

FP64: every neutron goes through the same rounded operations in each of the
three, so the counts are equal; sums agree within 1e-12 between the kernels
(order of additions) and 1e-9 with the oracle, or 1e-12 of the fullest bin (the
tanh of two libraries in the reflectivity: 1 - tanh keeps an absolute error).
"""

import ctypes
import math
import threading

import numpy as np
import pytest
import torch

from acc_gb300 import _native as nat
from acc_gb300 import engine, instruments
from acc_gb300.components.monitors.energy_monitor import Energy_monitor
from acc_gb300.components.monitors.psd_monitor import PSD_monitor
from acc_gb300.components.optics.guide import Guide
from acc_gb300.components.sources.source_simple import Source_simple
from acc_gb300.instrument import instrument
from helpers import gpu_tallies, oracle_run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _engine(engine_lib):
    torch.cuda.init()
    yield


def _chain(source=None, guide=None, orientation=(0, 0, 0), bins=40):
    """Disc source -> one guide 1 m away -> PSD and energy monitor."""
    src = dict(radius=0.05, dist=1.0, xw=0.05, yh=0.05, E0=52.5, dE=47.5)
    src.update(source or {})
    g = dict(w1=0.05, h1=0.05, w2=0.05, h2=0.05, l=4.0, R0=0.99, Qc=0.0219,
             alpha=3.0, m=3.0, W=0.003)
    g.update(guide or {})
    ins = instrument("edges")
    ins.append(Source_simple("src", **src), position=(0, 0, 0))
    ins.append(Guide("g", **g), position=(0, 0, 1.0), orientation=orientation)
    z = 1.0 + g["l"] + 1e-3
    ins.append(PSD_monitor("psd", xmin=-0.04, xmax=0.04, ymin=-0.04,
                           ymax=0.04, nx=bins, ny=bins, filename="p.h5"),
               position=(0, 0, z))
    ins.append(Energy_monitor("e", xmin=-0.04, xmax=0.04, ymin=-0.04,
                              ymax=0.04, Emin=0.0, Emax=100.0, nchan=50,
                              filename="e.h5"), position=(0, 0, z))
    return ins


def _agree(build, n, first=5):
    """Wave, thread and oracle FP64 runs of one stream agree; returns the
    number of neutrons in the first monitor."""
    a, b, c = build(), build(), build()
    sa = engine.run_instrument(a, n, seed=77, first=first,
                               floattype="float64")
    sb = engine.run_instrument(b, n, seed=77, first=first,
                               floattype="float64", variant="thread")
    ref, stats, _, _ = oracle_run(c, n, seed=77, first=first)
    assert sa.processed == sb.processed == stats["processed"] == n
    assert sa.nonfinite == sb.nonfinite
    for ta, tb, tc in zip(gpu_tallies(a).values(), gpu_tallies(b).values(),
                          ref.values()):
        np.testing.assert_array_equal(ta[0], tb[0])
        np.testing.assert_array_equal(ta[0], tc[0])
        np.testing.assert_allclose(ta[1:], tb[1:], rtol=1e-12, atol=1e-300)
        for x, y in zip(ta[1:], tc[1:]):
            np.testing.assert_allclose(x, y, rtol=1e-9,
                                       atol=1e-12 * y.max(initial=0.0))
    return int(next(iter(ref.values()))[0].sum())


# a mirror edge without width (and with one whose reciprocal overflows), of
# unbounded width, without and with unbounded reach
@pytest.mark.parametrize("coating", [
    dict(W=0.0), dict(W=0.0, m=1.5, alpha=6.07), dict(W=1e-310),
    dict(W=math.inf), dict(m=0.0), dict(m=math.inf), dict(m=1e200),
], ids=str)
def test_fp64_wave_kernel_divides_by_any_edge_width(coating):
    assert _agree(lambda: _chain(guide=coating), 20_001) > 100


# a first guide turned against the source (no screening), and one that
# converges so much that slow neutrons have both walls of a pair ahead
@pytest.mark.parametrize("kw", [
    dict(orientation=(0, 0, 30)), dict(orientation=(0.2, -0.1, 0)),
    dict(source=dict(E0=1.0, dE=0.99), guide=dict(w2=0.01, h2=0.01, l=0.3)),
    dict(source=dict(E0=10.0, dE=9.999), guide=dict(w2=0.02, h2=0.06)),
], ids=str)
def test_fp64_wave_kernel_turned_and_converging_guides(kw):
    assert _agree(lambda: _chain(**kw), 20_001) > 50


def test_fp64_source_divides_unbounded_speeds():
    """A speed that is not finite divides like any other: the components of
    the velocity are infinite with the signs of the flight, as the oracle's."""
    def build():
        ins = instrument("fast")
        ins.append(Source_simple("src", radius=0.05, dist=1.0, xw=0.05,
                                 yh=0.05, E0=math.inf, dE=0.0))
        return ins

    out, _ = engine.replay(engine.chain_for_instrument(build()), 101, seed=3,
                           floattype="float64")
    _, _, ref, _ = oracle_run(build(), 101, seed=3, record=True)
    assert np.isinf(ref[:, 3:6]).all()
    np.testing.assert_array_equal(out.cpu().numpy()[:, 3:6], ref[:, 3:6])


# Neutrons (stream 77) of a band that reaches down to almost nothing, whose
# first reflection is 0.05-0.4% below the mirror's reach: in FP32 the energy
# (wavelength) of the band's low end loses up to a percent, which puts the
# same reflection beyond it.
@pytest.mark.parametrize("first", [1156146778, 1165478551, 1251578636,
                                   1303006222, 1309909697, 1319045109])
def test_fp64_screen_keeps_the_low_end_of_an_energy_band(first):
    band = dict(E0=52.5, dE=52.49999)
    coat = dict(Qc=1e-3, m=1.0, W=1e-5)
    assert _agree(lambda: _chain(source=band, guide=coat), 1, first) == 1


def test_fp64_screen_keeps_the_low_end_of_a_wavelength_band():
    band = dict(E0=0, dE=0, Lambda0=10.0, dLambda=9.99999)
    coat = dict(Qc=200.0, m=1.0, W=0.1, alpha=0.0)
    assert _agree(lambda: _chain(source=band, guide=coat), 1, 330837591) == 1


def _strip_float_copies(ch):
    """The chain without the float copies that the FP32 kernels read."""
    for k in range(ch.ncomp):
        c = ch.comp[k]
        for j in range(len(c.fp)):
            c.fp[j] = 0.0
        for j in range(9):
            ch.frot[k][j] = 0.0
        for j in range(3):
            ch.foff[k][j] = 0.0


def _runs(name):
    """Ways to run an instrument's chain in FP64, with the float copies or
    without: the fused run, a replay, one batched variant."""
    def fused(ch, ins):
        engine.run_chain(ch, 3000, seed=9, floattype="float64")
        return list(gpu_tallies(ins).values())

    def replay(ch, ins):
        out, _ = engine.replay(ch, 3000, seed=9, floattype="float64")
        return [out.cpu().numpy()[:, 9][None]]

    def batched(ch, ins):
        arr, cnt, sd = engine._batch_arrays([ch], [3000], [9])
        st = nat.mcv_status()
        nat.check(nat.lib().mcv_run_batched(
            nat.context().handle, arr, 1, cnt, sd, 64, None,
            nat.current_stream_handle(), ctypes.byref(st)), st)
        return list(gpu_tallies(ins).values())

    runs = [fused]
    if name != "ms_hollow_cylinder":
        runs.append(replay)
        if name != "tapered_guide_chain":
            runs.append(batched)
    return runs


@pytest.mark.parametrize("name", ["guide_chain", "ms_hollow_cylinder",
                                  "tapered_guide_chain", "sqe_hollow_cylinder"])
def test_fp64_kernels_read_the_double_parameters_only(name):
    """fp, frot, foff and a segmented guide's ftable belong to the FP32
    kernels: an FP64 run does not depend on them."""
    wide = torch.full((4096,), 1e3, dtype=torch.float32, device="cuda")
    for run in _runs(name):
        out = []
        for strip in (False, True):
            ins = getattr(instruments, name)()
            ch = engine.chain_for_instrument(ins)
            if strip:
                _strip_float_copies(ch)
                for k in range(ch.ncomp):
                    c = ch.comp[k]
                    if c.opcode == nat.OP_GUIDE_TAPERING:
                        assert c.table_len <= wide.numel()
                        c.ftable = wide.data_ptr()
            out.append(run(ch, ins))
        for a, b in zip(*out):
            assert a[0].max() > 0
            np.testing.assert_array_equal(a[0], b[0])
            np.testing.assert_allclose(a[1:], b[1:], rtol=1e-12, atol=1e-300)


def test_launches_of_different_block_sizes_from_two_threads():
    """The shared memory that a kernel is allowed is a property of the kernel,
    shared by every thread of the process: launches of another block size do
    not take it away between a thread's request and its launch."""
    errors = []

    def work(tpb):
        try:
            ctx = nat.Context(torch.cuda.current_device())
            ch = engine.chain_for_instrument(_chain())
            L = nat.mcv_launch()
            L.threads_per_block = tpb
            st = nat.mcv_status()
            for i in range(3000):
                nat.check(nat.lib().mcv_run_chain(
                    ctx.handle, ctypes.byref(ch), 32, 0, i, 64,
                    ctypes.byref(L), None, ctypes.byref(st)), st)
        except Exception as e:  # reported by the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(t,)) for t in (256, 160)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_a_named_grid_keeps_full_blocks():
    """A launch that names its blocks but not their size has blocks of 256
    threads: one block takes as long as one block of 256 (median of 9; with
    the 32 threads that spread few neutrons over every SM, it took 3.7 times
    as long)."""
    ch = engine.chain_for_instrument(instruments.sphere_theta_tof())

    def us(**kw):
        times = []
        for i in range(11):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            engine.run_chain(ch, 2048, seed=i, floattype="float64", blocks=1,
                             sync=False, **kw)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times[2:]))

    assert us() < 1.5 * us(threads_per_block=256)
    engine.read_status()


# around the sizes of a warp and of a queue
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 2047])
def test_fp32_wave_kernel_loses_no_neutron(n):
    """FP32 wave and thread kernels round a neutron's path in different
    places, which moves entries between neighbouring bins: each monitor's
    total stays, to a neutron at an aperture's edge in the 2047, and so does
    its weight (1e-4: d ln R = 2 dq / W on the mirror's edge, q to a few
    1e-7, for some ten reflections there)."""
    slow = dict(E0=0, dE=0, Lambda0=15.0, dLambda=4.0)
    a, b = _chain(source=slow), _chain(source=slow)
    for ins, variant in ((a, None), (b, "thread")):
        st = engine.run_instrument(ins, n, seed=77, first=5,
                                   floattype="float32", variant=variant)
        assert st.processed == n
    for ta, tb in zip(gpu_tallies(a).values(), gpu_tallies(b).values()):
        assert tb[0].sum() > 0.4 * n
        assert abs(ta[0].sum() - tb[0].sum()) <= (1 if n == 2047 else 0)
        if ta[0].sum() == tb[0].sum():
            assert ta[1].sum() == pytest.approx(tb[1].sum(), rel=1e-4)
