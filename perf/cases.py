"""Performance cases: the runs a user of this package makes, through its public
entry points, with the work each cannot do without.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the instrument (and chain, graph, neutrons) in hand
    run(state)           one pass; returns the monitors' tallies, the
                         gradients or the processed neutrons
    work(case)           bytes and floating-point operations of one pass
    exact(case, seed)    the same outputs in 64 bits from plain torch, for the
                         guide and sphere instruments

A case has a `call` (which entry point), an `instrument` (a builder of
acc_gb300.instruments), a `floattype` and an `ncount`:

    "run"      engine.run_instrument, then every monitor's `out`: what
               run_script.run does for a script
    "grad"     autograd.GradRun forward and backward: fits of sample and
               coating parameters
    "graph"    engine.BatchedGraph over `nvariants` instruments: incident
               energy scans
    "process"  engine.process_buffer of one guide on a host neutron array:
               the components' buffered mode
"""

import math

import numpy as np
import torch

from acc_gb300 import engine, instruments
from acc_gb300.autograd import GradRun
from acc_gb300.components.monitors.MonitorBase import MonitorBase
from acc_gb300.components.optics.guide import Guide


def listed():
    return [
        # a first look at a script: few neutrons in the default precision,
        # all launch and host latency
        dict(name="sphere_fp64_1k", call="run", instrument="sphere_theta_tof",
             floattype="float64", ncount=1009),
        # the same instrument at production statistics in FP32
        dict(name="sphere_fp32_50m", call="run",
             instrument="sphere_theta_tof", floattype="float32",
             ncount=50_000_017),
        # the benchmark's guide chain: production statistics in FP32, and
        # in the default precision
        dict(name="guide_fp32_100m", call="run", instrument="guide_chain",
             floattype="float32", ncount=100_000_000),
        dict(name="guide_fp64_10m", call="run", instrument="guide_chain",
             floattype="float64", ncount=9_999_991),
        # a segmented elliptic guide in the default precision
        dict(name="tapered_fp64_1m", call="run",
             instrument="tapered_guide_chain", floattype="float64",
             ncount=1_000_003),
        # a whole instrument: VERDI, 26 components
        dict(name="verdi_fp32_10m", call="run", instrument="verdi",
             floattype="float32", ncount=10_000_000),
        # multiple scattering: the UN benchmark in FP32, the reference's
        # hollow-cylinder test instrument in the default precision
        dict(name="un_ms_fp32_3m", call="run", instrument="un_ms",
             floattype="float32", ncount=3_000_000),
        dict(name="hollow_ms_fp64_300k", call="run",
             instrument="ms_hollow_cylinder", floattype="float64",
             ncount=300_007),
        # one forward and one backward pass of a fit: S(Q, E) table with the
        # sample's coefficients, and powder structure factors with a coating
        dict(name="sqe_grad_fp32_20m", call="grad",
             instrument="sqe_hollow_cylinder", floattype="float32",
             ncount=20_000_003),
        dict(name="powder_grad_fp32_50m", call="grad",
             instrument="powder_banked", floattype="float32",
             ncount=50_000_000, ntubes=32, npixels=64, ntof=100),
        # an incident-energy scan: one launch over many instruments
        dict(name="scan_fp32_32x2m", call="graph",
             instrument="sphere_variants", floattype="float32",
             ncount=66_000_001, nvariants=32),
        # the buffered mode on neutrons in host memory, default precision
        dict(name="process_guide_fp64_500k", call="process",
             instrument="guide", floattype="float64", ncount=500_009),
    ]


# (call, instrument, floattype): the most neutrons a drawn case takes
_MOST = {
    ("run", "sphere_theta_tof", "float32"): 5e7,
    ("run", "sphere_theta_tof", "float64"): 1e7,
    ("run", "guide_chain", "float32"): 1e8,
    ("run", "guide_chain", "float64"): 1e7,
    ("run", "tapered_guide_chain", "float32"): 1e7,
    ("run", "tapered_guide_chain", "float64"): 1e6,
    ("run", "verdi", "float32"): 1e7,
    ("run", "un_ms", "float32"): 3e6,
    ("run", "un_ms", "float64"): 6e5,
    ("run", "ms_hollow_cylinder", "float32"): 1e6,
    ("run", "ms_hollow_cylinder", "float64"): 3e5,
    ("grad", "sqe_hollow_cylinder", "float32"): 2e7,
    ("grad", "sqe_hollow_cylinder", "float64"): 2e6,
    ("grad", "powder_banked", "float32"): 5e7,
    ("graph", "sphere_variants", "float32"): 6.6e7,
    ("process", "guide", "float64"): 5e5,
    ("process", "guide", "float32"): 5e5,
}


def draw(rng):
    call, ins, ft = rng.choice(sorted(_MOST))
    most = _MOST[call, ins, ft]
    n = int(math.exp(rng.uniform(math.log(1e3), math.log(most)))) | 1
    case = dict(call=call, instrument=ins, floattype=ft, ncount=n)
    if ins == "tapered_guide_chain":
        case["nseg"] = rng.randint(20, 120)
    if ins == "sphere_theta_tof":
        case["ntheta"] = rng.randint(30, 180)
        case["ntof"] = rng.randint(20, 200)
    if ins == "powder_banked":
        case.update(ntubes=rng.randint(4, 32), npixels=rng.randint(8, 64),
                    ntof=rng.randint(25, 100))
    if call == "graph":
        case["nvariants"] = rng.randint(2, 48)
    return case


# ------------------------------------------------------------------ inputs
_OPTIONS = ("nseg", "ntheta", "ntof", "ntubes", "npixels")


def _instrument(case):
    kw = {k: case[k] for k in _OPTIONS if k in case}
    return getattr(instruments, case["instrument"])(**kw)


def _philox_seed(seed):
    return 1 + 7919 * int(seed)


def _scan(case, seed):
    """Incident energies log-uniform in 20-500 meV, counts log-uniform over
    a decade with the case's total, one Philox seed each."""
    n = case["nvariants"]
    ins, counts, seeds = instruments.sphere_variants(
        n, seed=int(seed) % (1 << 32), nmin=1.0, nmax=10.0)
    share = np.exp(np.random.default_rng([int(seed), 1]).uniform(
        0.0, math.log(10.0), n))
    counts = [max(1, int(c)) for c in share / share.sum() * case["ncount"]]
    return ins, counts, seeds


def _guide_neutrons(case, seed):
    """Neutrons leaving a source plane 1 m before a 5 x 5 cm entrance, as a
    saved beam holds them: 5-100 meV, a few mrad of divergence."""
    n = case["ncount"]
    r = np.random.default_rng(int(seed))
    a = np.zeros((n, 10))
    a[:, 0:2] = r.uniform(-0.025, 0.025, (n, 2))
    v = 437.393377 * np.sqrt(r.uniform(5.0, 100.0, n))
    d = r.normal(0.0, 5e-3, (n, 2))
    a[:, 3] = v * d[:, 0]
    a[:, 4] = v * d[:, 1]
    a[:, 5] = v
    a[:, 8] = r.uniform(0.0, 1e-3, n)
    a[:, 9] = r.uniform(0.1, 1.0, n)
    return a


_GUIDE = dict(w1=0.05, h1=0.05, w2=0.05, h2=0.05, l=10.0)


def prepare(case, seed):
    n, ft, s = case["ncount"], case["floattype"], _philox_seed(seed)
    state = dict(case=case, seed=s)
    if case["call"] == "run":
        state["ins"] = _instrument(case)
    elif case["call"] == "graph":
        ins, counts, seeds = _scan(case, seed)
        state["graph"] = engine.BatchedGraph(ins, counts, seeds, floattype=ft)
        state["ins"] = ins
    elif case["call"] == "process":
        state["guide"] = Guide("guide", **_GUIDE, **instruments.COATING)
        state["neutrons"] = _guide_neutrons(case, seed)
    else:
        ins = _instrument(case)
        mon = [c for c in ins.components if isinstance(c, MonitorBase)][-1]
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        if case["instrument"] == "powder_banked":
            sample = ins.components[-2]
            guides = [c for c in ins.components if isinstance(c, Guide)]
            f2 = [p.F_squared for p in sample.kernel.peaks]
            params = {"F2": ("powder_F2", sample), "m": ("guide_m", guides)}
            values = {"F2": torch.tensor(f2, dtype=torch.float64),
                      "m": torch.tensor(3.0, dtype=torch.float64)}
        else:
            sample = ins.components[1]
            params = {"S": ("sqe_table", sample), "mu": ("hss_mu", sample),
                      "sigma": ("hss_sigma", sample)}
            values = {"S": torch.from_numpy(instruments.sqe_table()).cuda(),
                      "mu": torch.tensor(10.0, dtype=torch.float64),
                      "sigma": torch.tensor(25.0, dtype=torch.float64)}
        state["fit"] = GradRun(ins, mon, n, seed=s, floattype=ft,
                               params=params)
        state["values"] = {k: v.requires_grad_() for k, v in values.items()}
        # dL/dH of a weighted least-squares loss: random signs and sizes
        state["weight"] = torch.randn(mon.hist_shape, generator=g,
                                      dtype=torch.float64, device="cuda")
    return state


# -------------------------------------------------------------------- runs
def run(state):
    case = state["case"]
    if case["call"] == "run":
        mons = [c for c in state["ins"].components
                if isinstance(c, MonitorBase)]
        for m in mons:
            m.reset()
        engine.run_instrument(state["ins"], case["ncount"],
                              seed=state["seed"],
                              floattype=case["floattype"])
        return [m.out for m in mons]
    if case["call"] == "graph":
        mons = [ins.components[-1] for ins in state["ins"]]
        for m in mons:
            m.reset()
        state["graph"].launch()
        engine.read_status(expected=state["graph"].total)
        return [m.out for m in mons]
    if case["call"] == "process":
        return engine.process_buffer([state["guide"]], state["neutrons"],
                                     seed=state["seed"],
                                     floattype=case["floattype"])
    hist = state["fit"](**state["values"])
    leaves = list(state["values"].values())
    grads = torch.autograd.grad(hist, leaves, grad_outputs=state["weight"])
    return {"hist": hist.detach(),
            "grads": dict(zip(state["values"], grads))}


# -------------------------------------------------------------------- work
# Floating-point operations a neutron cannot do without (mean over the
# neutrons of the instrument; additions, multiplications, divisions, roots
# and function values each count one): source draw ~45, a guide's entry ~8
# and ~45 a reflection (1.2 reflections in the first guide, 7.5% of the
# neutrons reach the second), shape crossings ~40 each, a monitor ~15, a
# multiple-scattering call ~150, a straight segment of a tapered guide ~12.
_FLOPS = {"sphere_theta_tof": 150, "sphere_variants": 150,
          "guide_chain": 130, "tapered_guide_chain": 900, "verdi": 900,
          "un_ms": 1500, "ms_hollow_cylinder": 2000,
          "sqe_hollow_cylinder": 250, "powder_banked": 140, "guide": 120}


def _bins(case):
    if case["instrument"] in ("sphere_theta_tof", "sphere_variants"):
        return case.get("ntheta", 180) * case.get("ntof", 200)
    if case["instrument"] == "powder_banked":
        return 8 * case["ntubes"] * case["npixels"] * case["ntof"]
    return {"guide_chain": 10_200, "tapered_guide_chain": 62_500,
            "verdi": 1_000_000, "un_ms": 15_000,
            "ms_hollow_cylinder": 8_100,
            "sqe_hollow_cylinder": 10_000}[case["instrument"]]


def work(case):
    n = case["ncount"]
    flops = float(n) * _FLOPS[case["instrument"]]
    if case["call"] == "process":
        return {"bytes": 160.0 * n, "flops": flops}
    # the tallies (N, sum p, sum p^2) written once and read back once
    nbytes = 48.0 * _bins(case) * case.get("nvariants", 1)
    if case["call"] == "grad":
        # the backward pass follows the same neutrons, reads dL/dH and adds
        # one gradient per parameter
        return {"bytes": nbytes + 8.0 * _bins(case), "flops": 2 * flops}
    return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------- the same outputs in 64 bits
_V2K, _SE2V, _VS2E = 1.58825361e-3, 437.393377, 5.22703725e-6
_M32 = 0xFFFFFFFF
_CHUNK = 1 << 22


def _philox_uniforms(seed, index, block):
    """Five 24-bit uniforms of Philox4x32-10, counter (index, block, 0)."""
    x0, x1 = index & _M32, (index >> 32) & _M32
    x2, x3 = torch.full_like(index, block), torch.zeros_like(index)
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for _ in range(10):
        a, b = x0 * 0xD2511F53, x2 * 0xCD9E8D57  # the low 64 bits
        x0, x1, x2, x3 = (((b >> 32) & _M32) ^ x1 ^ k0, b & _M32,
                          ((a >> 32) & _M32) ^ x3 ^ k1, a & _M32)
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    w = 0xFFFFFF
    u = (x0 & w, ((x0 >> 24) | (x1 << 8)) & w, ((x1 >> 16) | (x2 << 16)) & w,
         x2 >> 8, x3 & w)
    return [v.double() * 2.0 ** -24 for v in u]


class _Beam:
    """Columns x y z vx vy vz t p of the neutrons of one chunk."""

    def __init__(self, **cols):
        self.__dict__.update(cols)

    def take(self, m):
        return _Beam(**{k: v[m] for k, v in self.__dict__.items()})

    def move(self, dt):
        for a in "xyz":
            setattr(self, a, getattr(self, a) + getattr(self, "v" + a) * dt)
        self.t = self.t + dt


def _source(u, radius, dist, xw, yh, E0, dE):
    r, phi = torch.sqrt(u[1].float()).double() * radius, u[0] * (2 * math.pi)
    x, y = r * torch.cos(phi), r * torch.sin(phi)
    tx, ty = xw * (u[2] * 2 - 1) / 2, yh * (u[3] * 2 - 1) / 2
    solid = xw * yh * dist / (tx * tx + ty * ty + dist * dist) ** 1.5
    area = 1e4 * math.pi * radius * radius  # cm^2, at unit flux
    dx, dy = -tx - x, -ty - y
    v = _SE2V * torch.sqrt(E0 + dE * (u[4] * 2 - 1))
    s = v / torch.sqrt(dx * dx + dy * dy + dist * dist)
    return _Beam(x=x, y=y, z=torch.zeros_like(x), vx=s * dx, vy=s * dy,
                 vz=s * dist, t=torch.zeros_like(x), p=area * solid)


def _through_guide(b, w1, h1, w2, h2, l, R0, Qc, alpha, m, W):
    """Reflect `b` down a guide; the columns at the last reflection, p = -1
    for the neutrons outside the opening and 0 for the absorbed ones."""
    start = b.take(slice(None))
    start.move(-b.z / b.vz)
    out = (start.x.abs() >= w1 / 2) | (start.y.abs() >= h1 / 2)
    for name, v in start.__dict__.items():  # the absorbed ones stay put
        b.__dict__[name] = torch.where(out, b.__dict__[name], v)
    b.p = torch.where(out, -1.0, b.p)
    live = torch.nonzero(~out).reshape(-1)
    ww, hh, inf = (w2 - w1) / 2, (h2 - h1) / 2, math.inf
    while live.numel():
        c = b.take(live)
        av, bv, ah, bh = l * c.vx, ww * c.vz, l * c.vy, hh * c.vz
        cv, ch = -w1 / 2 * l - c.z * ww, -h1 / 2 * l - c.z * hh
        vn = torch.stack([bv + av, bv - av, bh + ah, bh - ah])
        d = torch.stack([cv - c.x * l, cv + c.x * l, ch - c.y * l,
                         ch + c.y * l])
        t = torch.where(vn < 0, d / vn, inf)
        t, i = t.min(0)
        hit = t < (l - c.z) / c.vz
        c, t, i, live = c.take(hit), t[hit], i[hit], live[hit]
        vn = vn[:, hit].gather(0, i[None])[0]
        c.move(t)
        slope = torch.where(i < 2, ww, torch.full_like(t, hh))
        n2 = l * l + slope * slope
        q, k = _V2K * -2 * vn / torch.sqrt(n2), 2 * vn / n2
        k1 = torch.where((i == 0) | (i == 2), -k, k) * l
        c.vx, c.vy = c.vx + k1 * (i < 2), c.vy + k1 * (i >= 2)
        c.vz = c.vz - k * slope
        x = (q - m * Qc) / W
        edge = R0 * (1 - torch.tanh(x)) * (1 - alpha * (q - Qc)) / 2
        c.p = c.p * torch.where(q > Qc, torch.where(x < 10, edge, 0.0), R0)
        for name, v in c.__dict__.items():
            b.__dict__[name][live] = v
        live = live[c.p > 0]
    return b


def _tally(hist, bins, p):
    for row, v in zip(hist, (torch.ones_like(p), p, p * p)):
        row.index_add_(0, bins, v)


def _bin(v, lo, hi, n):
    return ((v - lo) / (hi - lo) * n).floor().long().clamp(0, n - 1)


def _exact_guide(n, seed):
    psd = torch.zeros(3, 10_000, dtype=torch.float64, device="cuda")
    emon = torch.zeros(3, 200, dtype=torch.float64, device="cuda")
    c = instruments.COATING
    for first in range(0, n, _CHUNK):
        i = torch.arange(first, min(n, first + _CHUNK), device="cuda")
        b = _source(_philox_uniforms(seed, i, 0), 0.05, 1.0, 0.05, 0.05,
                    52.5, 47.5)
        b.z = b.z - 1.0
        b = _through_guide(b, 0.05, 0.05, 0.05, 0.05, 10.0, **c)
        b = b.take(b.p > 0)
        b.z = b.z - 10.001
        b = _through_guide(b, 0.05, 0.05, 0.02, 0.02, 5.0, **c)
        b = b.take(b.p > 0)
        b.z = b.z - 5.001
        b.move(-b.z / b.vz)
        b = b.take((b.x.abs() < 0.03) & (b.y.abs() < 0.03))
        _tally(psd, _bin(b.x, -0.03, 0.03, 100) * 100 +
               _bin(b.y, -0.03, 0.03, 100), b.p)
        E = (b.vx * b.vx + b.vy * b.vy + b.vz * b.vz) * _VS2E
        m = (E > 0) & (E < 100.0)
        _tally(emon, _bin(E[m], 0.0, 100.0, 200), b.p[m])
    return [psd.reshape(3, 100, 100).cpu().numpy(), emon.cpu().numpy()]


def _crossings(b, radius):
    """(hit, t1, t2) of the rays with a sphere around the origin."""
    rv = b.x * b.vx + b.y * b.vy + b.z * b.vz
    v2 = b.vx * b.vx + b.vy * b.vy + b.vz * b.vz
    d = rv * rv - v2 * (b.x * b.x + b.y * b.y + b.z * b.z - radius * radius)
    s = torch.sqrt(d.clamp(min=0))
    return d >= 0, (-rv - s) / v2, (-rv + s) / v2


def _exact_sphere(n, seed, E0, dE, nth, nt):
    hist = torch.zeros(3, nth * nt, dtype=torch.float64, device="cuda")
    for first in range(0, n, _CHUNK):
        i = torch.arange(first, min(n, first + _CHUNK), device="cuda")
        u = _philox_uniforms(seed, i, 0) + _philox_uniforms(seed, i, 1)
        b = _source(u, 0.05, 5.0, 0.01, 0.01, E0, dE)
        b.z = b.z - 5.0
        hit, t1, t2 = _crossings(b, 0.01)
        inside = torch.where(hit, u[5] * (t2 - t1), 0.0)
        b.move(torch.where(hit, t1 + inside, 0.0))
        v = torch.sqrt(b.vx * b.vx + b.vy * b.vy + b.vz * b.vz)
        mu = 25.0 / v * 2200 + 25.0
        cost, phi = u[6] * 2 - 1, u[7] * (2 * math.pi)
        sint = torch.sqrt(1 - cost * cost)
        for a, w in (("vx", sint * torch.cos(phi)),
                     ("vy", sint * torch.sin(phi)), ("vz", cost)):
            b.__dict__[a] = torch.where(hit, v * w, b.__dict__[a])
        out = torch.where(hit, _crossings(b, 0.01)[2], 0.0)
        b.p = torch.where(hit, b.p * v * (t2 - t1) * 25.0 *
                          torch.exp(-mu * v * (inside + out)), b.p)
        b.move(out)
        hit, t1, t2 = _crossings(b, 3.0)
        b.move(torch.where(t1 < 0, t2, t1))
        theta = torch.atan2(torch.hypot(b.x, b.y), b.z)
        m = hit & (t2 >= 0) & (b.t >= 0) & (b.t < 0.01)
        _tally(hist, _bin(theta[m], 0.0, math.pi, nth) * nt +
               _bin(b.t[m], 0.0, 0.01, nt), b.p[m])
    return hist.reshape(3, nth, nt).cpu().numpy()


def exact(case, seed):
    s, n = _philox_seed(seed), case["ncount"]
    if case["call"] == "run" and case["instrument"] == "guide_chain":
        return _exact_guide(n, s)
    if case["call"] == "run" and case["instrument"] == "sphere_theta_tof":
        return [_exact_sphere(n, s, 60.0, 10.0, case.get("ntheta", 180),
                              case.get("ntof", 200))]
    if case["call"] == "graph":
        ins, counts, seeds = _scan(case, seed)
        return [_exact_sphere(c, k, float(i.components[0].propagate_params[7]),
                              0.0, 180, 200)
                for i, c, k in zip(ins, counts, seeds)]
    if case["call"] == "process":
        a = torch.from_numpy(_guide_neutrons(case, seed)).cuda()
        if case["floattype"] == "float32":
            a = a.float().double()
        b = _Beam(**{k: a[:, j].clone() for j, k in
                     zip((0, 1, 2, 3, 4, 5, 8, 9),
                         ("x", "y", "z", "vx", "vy", "vz", "t", "p"))})
        b = _through_guide(b, *_GUIDE.values(), **instruments.COATING)
        for j, k in zip((0, 1, 2, 3, 4, 5, 8, 9),
                        ("x", "y", "z", "vx", "vy", "vz", "t", "p")):
            a[:, j] = b.__dict__[k]
        return a.cpu().numpy()
    return None
