// wave.cuh -- the path-regeneration kernels of chains with guides.
//
// One neutron per thread leaves most of a warp idle behind its longest path:
// in the guide chain nine neutrons of ten die at their first reflection and
// a few make ten.  Here a warp runs three kinds of passes, each with its
// lanes full:
//
//   front   32 new neutrons from the source to the first reflection of the
//           first guide, in straight-line code with a uniform component
//           index; the survivors wait in the warp's flight queue
//   bounce  every lane holds a neutron inside some guide and makes one
//           reflection; lanes that come free take the next neutron of the
//           flight queue
//   tail    32 neutrons that left the last guide, through the components
//           after it (monitors, a sample, a detector), from the tail queue
//
// Every neutron goes through the same components in the same order on its own
// Philox stream as in the thread kernel: in FP64 with the same results, in
// FP32 with roundings of its own (kWave), which move a neutron within an ulp
// of a bin's edge into the next bin; the FP32 backward replays with the thread
// kernel's roundings.  Between the bounce loops no lane holds a neutron (the
// loop puts back what it has in flight), so that each phase has the registers
// to itself.
//
// Bound by instruction issue (FP32) and by the FP64 pipe.  Measured on the
// guide chain, where nine neutrons of ten die at their first reflection and
// 1.8% reach the monitors:
//   FP32, 1e8 neutrons: 3.79 -> 2.16 ms against one loop that swept
//   the chain a component at a time (35.2 warp instructions a neutron on 23
//   lanes, two of three of them control flow, range tests of the rounded
//   divisions and spills);
//   FP64, 1e7 neutrons: 23.9 -> 2.02 ms against one neutron per thread
//   (8.6 lanes on a pipe that costs a warp instruction 16 clocks whatever
//   its lanes), most of it from the screen below.
#pragma once

namespace mcv {

// A queue holds up to 63 neutrons: a pass adds at most 32, and runs only
// while fewer than 32 wait.
constexpr int kWaveCap = 64;

// What a waiting neutron is: its state without the spin (which the sources of
// these chains leave 0 and nothing changes), its index,
// `meta`: component (bits 0-5), inside a guide (6), uniforms left in the
// current Philox block (7-9), the next block (10-31), and its reflections in
// the guide so far.
template <typename R>
constexpr int kWaveWords = (sizeof(R) == 8 ? 16 : 9) + 4;

template <typename R>
__device__ __forceinline__ void wave_store(uint32_t* q, const Neutron<R>& n,
                                           uint32_t c0, uint32_t c1,
                                           uint32_t meta, uint32_t nb) {
  int k = 0;
  auto put = [&](uint32_t w) { q[kWaveCap * k++] = w; };
  auto val = [&](R v) {
    if constexpr (sizeof(R) == 4) {
      put(__float_as_uint(v));
    } else {
      put((uint32_t)__double2loint(v));
      put((uint32_t)__double2hiint(v));
    }
  };
  val(n.x);
  val(n.y);
  val(n.z);
  val(n.vx);
  val(n.vy);
  val(n.vz);
  if constexpr (sizeof(R) == 4) {
    val(n.t.hi);
    val(n.t.lo);
  } else {
    val(n.t.t);
  }
  val(n.p);
  put(c0);
  put(c1);
  put(meta);
  put(nb);
}

template <typename R>
__device__ __forceinline__ void wave_load(const uint32_t* q, Neutron<R>& n,
                                          uint32_t& c0, uint32_t& c1,
                                          uint32_t& meta, uint32_t& nb) {
  int k = 0;
  auto get = [&]() { return q[kWaveCap * k++]; };
  auto val = [&]() -> R {
    if constexpr (sizeof(R) == 4) {
      return __uint_as_float(get());
    } else {
      const uint32_t lo = get();
      return __hiloint2double((int)get(), (int)lo);
    }
  };
  n.x = val();
  n.y = val();
  n.z = val();
  n.vx = val();
  n.vy = val();
  n.vz = val();
  n.sx = n.sy = R(0);
  if constexpr (sizeof(R) == 4) {
    n.t.hi = val();
    n.t.lo = val();
  } else {
    n.t.t = val();
  }
  n.p = val();
  c0 = get();
  c1 = get();
  meta = get();
  nb = get();
}

__device__ __forceinline__ uint32_t wave_meta(int c, int inside,
                                              const PhiloxStream& r) {
  return (uint32_t)c | ((uint32_t)inside << 6) | ((uint32_t)r.left << 7) |
         (r.c2 << 10);
}

// a neutron's stream again, at the position its meta word holds
__device__ __forceinline__ PhiloxStream wave_stream(uint64_t seed, uint32_t c0,
                                                    uint32_t c1,
                                                    uint32_t meta) {
  PhiloxStream r(seed, (uint64_t)c0 | ((uint64_t)c1 << 32), 0u);
  const int left = (int)(meta >> 7 & 7u);
  r.c2 = meta >> 10;
  if (left) {
    --r.c2;
    r.refill();
    while (r.left > left) r.next();
  }
  return r;
}

// One component of the chain on one neutron, out of line: for the places
// that few lanes or few chains reach (components ahead of the first guide
// other than a plain source, and between guides).
template <typename R>
__device__ __noinline__ int wave_component(Neutron<R>& n, PhiloxStream& rng,
                                           const mcv_chain& ch, int k,
                                           double* smt) {
  NoTrack trk;
  return run_component<R>(n, rng, ch.comp[k], trk, ch, smt);
}

// ---------------------------------------------------------------- screening
// FP64 chains whose source is followed at once by a guide: most neutrons end
// at their first reflection, beyond the mirror's reach.  GB300 retires 2
// FP64 lanes a clock and SM against 128 FP32 lanes, so the front first
// follows the neutron to its first wall in FP32 with an error bound on every
// quantity, and drops it when it certainly is outside the opening or
// certainly meets, first, a wall it certainly does not survive.  Every other
// neutron (13% of the guide chain's) is then run in FP64 from its source
// draws: what reaches a tally never depends on the FP32 values.
struct WaveScreen {
  int on;
  // the source's and the guide's parameters, and the entrance's offset, from
  // the doubles (fp[] is the FP32 kernels')
  float a[11], g[5], ox, oy;
  float f;           // (distance to the entrance) / (distance to the target)
  float e_pos, e_m;  // error bounds: position at the entrance, wall approach
  float kx, ky;      // q = k vz m: 2 V2K / sqrt(l^2 + slope^2)
  float qdead;       // certainly absorbed at or beyond this q
};

__device__ inline void wave_screen_setup(WaveScreen& s, const mcv_chain& ch) {
  s.on = 0;
  if (ch.ncomp < 2 || ch.comp[0].opcode != MCV_OP_SOURCE_SIMPLE ||
      ch.comp[1].opcode != MCV_OP_GUIDE ||
      !(ch.comp[1].flags & kFlagIdentityRot))
    return;
  const double* a = ch.comp[0].dp;
  const double* g = ch.comp[1].dp;
  const double dist = a[9], oz = ch.off[1][2], l = g[4], W = g[9];
  // the slowest neutron moves forward, the weight is finite and the guide
  // lies downstream; anything else runs unscreened
  const bool slow = ch.comp[0].ip[1] ? !(a[3] - fabs(a[4]) > 0)
                                     : !(a[5] - fabs(a[6]) > 0);
  if (slow || !(dist > 0) || !(oz > 0) || !(l > 0) || !(W > 0) ||
      !isfinite(a[10]) || !(a[10] > 0) || !(a[7] > 0) || !(a[8] > 0))
    return;
  // The speed's relative error in FP32: E0 + dE (2 u - 1) keeps a few units
  // of 2^-24 (E0 + |dE|), and the slowest neutron has E0 - |dE| of it (the
  // wavelength likewise).  A band that reaches down so far that this exceeds
  // a percent runs unscreened.
  const int at = ch.comp[0].ip[1] ? 3 : 5;
  const double mean = a[at], half = fabs(a[at + 1]);
  const double e_v = ldexp(8.0, -24) * (fabs(mean) + half) / (mean - half);
  if (!(e_v < 1e-2)) return;
  const double q = fmax(g[6], g[8] * g[6] + 10.0 * W);
  const double reach = fabs(a[0]) + fabs(a[1]) + fabs(a[2]) + a[7] + a[8];
  for (int k = 0; k < 11; ++k) s.a[k] = (float)a[k];
  for (int k = 0; k < 5; ++k) s.g[k] = (float)g[k];
  s.ox = (float)ch.off[1][0];
  s.oy = (float)ch.off[1][1];
  s.f = (float)(oz / dist);
  // FP32 rounding of a few operations on values up to `reach` and the
  // hardware sine and cosine (2^-21.4) are below 2e-6 of it
  s.e_pos = (float)(1e-5 * (reach * (1.0 + oz / dist) +
                            fabs(ch.off[1][0]) + fabs(ch.off[1][1]) +
                            fabs(g[2]) + fabs(g[3])));
  s.e_m = (float)(1e-5 * (l * reach / dist + fabs(g[0]) + fabs(g[1])));
  s.kx = (float)(2 * kV2K / sqrt(l * l + g[0] * g[0]));
  s.ky = (float)(2 * kV2K / sqrt(l * l + g[1] * g[1]));
  // 1e-4 for the other factors of q (a few 2^-22); e_v bounds the speed's
  // error, a square root halves the energy's and 1 / (1 - e) of a wavelength
  // stays below 1 + 2 e
  s.qdead = (float)(q * (1.0 + 1e-4 + 2.0 * e_v));
  s.on = isfinite(s.f) && isfinite(s.e_pos) && isfinite(s.e_m) &&
         isfinite(s.kx) && isfinite(s.ky) && isfinite(s.qdead) &&
         s.qdead > 0.f && dist > 1e-6 && dist < 1e6 && reach < 1e6 &&
         l < 1e6;
}

// true when the neutron certainly ends at the first guide's opening or first
// reflection
__device__ __forceinline__ bool wave_screen_dead(const WaveScreen& s,
                                                 const mcv_chain& ch,
                                                 PhiloxStream& rng) {
  const int* const ip = ch.comp[0].ip;
  const float u1 = rng.next(), u2 = rng.next(), u3 = rng.next(),
              u4 = rng.next(), u5 = rng.next();
  float x, y;
  if (ip[0]) {
    x = s.a[0] * (u1 - 0.5f);
    y = s.a[1] * (u2 - 0.5f);
  } else {
    const float r = sqrtf(u2) * s.a[2];
    float sn, cs;
    m_sincos_2pi(u1, &sn, &cs);
    x = r * cs;
    y = r * sn;
  }
  const float dist = s.a[9];
  const float dx = -s.a[7] * (u3 - 0.5f) - x;
  const float dy = -s.a[8] * (u4 - 0.5f) - y;
  const float v = ip[1] ? float(kK2V * 2 * kPi) /
                                (s.a[3] + s.a[4] * (2.f * u5 - 1.f))
                          : float(kSE2V) *
                                sqrtf(s.a[5] + s.a[6] * (2.f * u5 - 1.f));
  const float vz = v * dist * rsqrtf(dx * dx + dy * dy + dist * dist);
  const float px = fmaf(dx, s.f, x - s.ox);
  const float py = fmaf(dy, s.f, y - s.oy);
  const float hw = s.g[2], hh = s.g[3];
  if (fabsf(px) > hw + s.e_pos || fabsf(py) > hh + s.e_pos) return true;
  if (!(fabsf(px) < hw - s.e_pos && fabsf(py) < hh - s.e_pos)) return false;
  // the wall ahead on each side: m is its approach over the guide's length
  // (per unit l), d its distance; it is met at the fraction d / m of l
  const float sl = s.g[4] / dist, lx = dx * sl, ly = dy * sl;
  const float m[4] = {-s.g[0] - lx, -s.g[0] + lx, -s.g[1] - ly,
                      -s.g[1] + ly};
  const float d[4] = {hw + px, hw - px, hh + py, hh - py};
  float first = 1.f;  // the latest the first wall can be met; 1: the exit
  bool met = false;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    const float hi = (d[w] + s.e_pos) / (m[w] - s.e_m);
    if (m[w] > s.e_m && hi < first * 0.9999f) {
      first = hi;
      met = true;
    }
  }
  bool dead = met;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    const bool could = m[w] > -s.e_m &&
                       (d[w] - s.e_pos) <= first * 1.0001f * (m[w] + s.e_m);
    const float q = (w < 2 ? s.kx : s.ky) * vz * (m[w] - s.e_m);
    if (could && !(q > s.qdead)) dead = false;
  }
  return dead;
}

// ------------------------------------------------------------------- kernel
// Shared memory of one warp, in bytes: the flight and tail queues and, FP64,
// the indices that passed the screen.
template <typename R>
__host__ __device__ constexpr size_t wave_warp_bytes() {
  return sizeof(uint32_t) * kWaveCap *
         (2 * (size_t)kWaveWords<R> + (sizeof(R) == 8 ? 1 : 0));
}

// `tail_min`: the tail runs once this many neutrons wait for it (32; 1 runs
// it without waiting).  With kSmem, the dynamic shared memory starts with
// `tally_words` doubles of monitor tallies (MCV_COMP_SMEM_TALLY), zeroed here
// and added to the global tallies when the block ends.
template <typename R, bool kSmem = false>
__global__ void __launch_bounds__(kMaxThreads, sizeof(R) == 4 ? 4 : 2)
    wave_kernel(const __grid_constant__ mcv_chain ch, uint64_t n,
                uint64_t first, uint64_t seed, int tail_min, int tally_words,
                DevStatus* st) {
  extern __shared__ __align__(16) uint32_t wave_smem[];
  __shared__ WaveScreen screen;
  __shared__ GuideInv inv[sizeof(R) == 8 ? MCV_MAX_COMPONENTS : 1];
  if constexpr (!kSmem) tally_words = 0;
  double* const smt = kSmem ? (double*)wave_smem : nullptr;
  const int nc = ch.ncomp;
  if constexpr (kSmem) {
    for (int i = threadIdx.x; i < tally_words; i += blockDim.x) smt[i] = 0.0;
  }
  if constexpr (sizeof(R) == 8) {
    if (threadIdx.x == 0) wave_screen_setup(screen, ch);
    for (int k = threadIdx.x; k < nc; k += blockDim.x)
      if (ch.comp[k].opcode == MCV_OP_GUIDE) inv[k] = guide_inv(ch.comp[k]);
  }
  if constexpr (kSmem || sizeof(R) == 8) __syncthreads();
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned below = (1u << lane) - 1u;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t per = (n + nwarps - 1) / nwarps;
  uint64_t next = warp * per;
  const uint64_t end = next + per < n ? next + per : n;
  // the screen's queue holds 32-bit offsets into the warp's range
  const bool screening =
      sizeof(R) == 8 && screen.on && per <= 0xffffffffull;
  int g1 = -1, last_guide = -1;
  for (int k = 0; k < nc; ++k)
    if (ch.comp[k].opcode == MCV_OP_GUIDE) {
      if (g1 < 0) g1 = k;
      last_guide = k;
    }
  uint32_t* const q1 = wave_smem + 2 * tally_words +
                       (threadIdx.x >> 5) * (wave_warp_bytes<R>() / 4);
  uint32_t* const q2 = q1 + kWaveWords<R> * kWaveCap;
  uint32_t* const q0 = q2 + kWaveWords<R> * kWaveCap;
  int h1 = 0, n1 = 0, h2 = 0, n2 = 0, h0 = 0, n0 = 0;  // warp-uniform
  Counters k{0, 0, 0, 0};
  NoTrack trk;

  // every lane of the warp calls it; the lanes with `mine` append `m`
  auto push = [&](uint32_t* q, int h, int& cnt, bool mine,
                  const Neutron<R>& m, uint32_t i0, uint32_t i1,
                  uint32_t meta_, int nb_) {
    const unsigned pm = __ballot_sync(kFull, mine);
    if (mine) {
      const int slot = (h + cnt + __popc(pm & below)) % kWaveCap;
      wave_store<R>(q + slot, m, i0, i1, meta_, (uint32_t)nb_);
    }
    cnt += __popc(pm);
    __syncwarp();
  };
  auto retire = [&](bool nan) {
    if (nan) k.nonfinite++;
    k.processed++;
  };
  auto tail = [&]() {
    const int m = n2 < 32 ? n2 : 32;
    if ((int)lane < m) {
      Neutron<R> t;
      uint32_t i0, i1, mt, tb;
      const int slot = (h2 + (int)lane) % kWaveCap;
      wave_load<R>(q2 + slot, t, i0, i1, mt, tb);
      PhiloxStream rng = wave_stream(seed, i0, i1, mt);
      bool alive = true;
      for (int kc = last_guide + 1; kc < nc; ++kc) {
        if (!alive) continue;
        if (kc > last_guide + 1) apply_transform<R>(t, ch, kc);
        k.overflow += run_component<R>(t, rng, ch.comp[kc], trk, ch, smt);
        if (!(t.p > 0)) alive = false;
      }
      retire(m_isnan(t.p));
    }
    h2 = (h2 + m) % kWaveCap;
    n2 -= m;
    __syncwarp();
  };
  // FP64: the next 32 neutrons that the screen does not drop
  auto screened = [&](uint64_t& idx) -> bool {
    while (n0 < 32 && next < end) {
      idx = next + lane;
      bool keep = idx < end;
      if (keep) {
        PhiloxStream rs(seed, first + idx, 0u);
        if (wave_screen_dead(screen, ch, rs)) {
          keep = false;
          k.processed++;
        }
      }
      const unsigned pm = __ballot_sync(kFull, keep);
      if (keep)
        q0[(h0 + n0 + __popc(pm & below)) % kWaveCap] =
            (uint32_t)(idx - warp * per);
      n0 += __popc(pm);
      next = next + 32 < end ? next + 32 : end;
      __syncwarp();
    }
    const int m = n0 < 32 ? n0 : 32;
    idx = warp * per + q0[(h0 + (int)lane) % kWaveCap];
    h0 = (h0 + m) % kWaveCap;
    n0 -= m;
    __syncwarp();
    return (int)lane < m;
  };
  // 32 new neutrons up to their first reflection
  auto front = [&]() {
    uint64_t idx = next + lane;
    bool alive = idx < end;
    if (screening) alive = screened(idx);
    else next = next + 32 < end ? next + 32 : end;
    Neutron<R> m;
    zero_neutron(m);
    PhiloxStream rng(seed, first + idx, 0u);
    int mc = g1, in = 0;
    if (alive) {
      int kc = 0;
      if (ch.comp[0].opcode == MCV_OP_SOURCE_SIMPLE) {
        source_simple<R, true>(m, rng, ch.comp[0]);
        if constexpr (sizeof(R) == 4) m.p *= weight_up<R>(ch);
        alive = m.p > 0;
        kc = 1;
      }
      for (; kc < g1; ++kc) {
        if (!alive) continue;
        if (kc > 0) apply_transform<R>(m, ch, kc);
        Neutron<R> tmp = m;
        PhiloxStream rt = rng;
        k.overflow += wave_component<R>(tmp, rt, ch, kc, smt);
        m = tmp;
        rng = rt;
        if (!(m.p > 0)) alive = false;
      }
      if (alive) {
        if (g1 > 0) apply_transform<R>(m, ch, g1);
        const mcv_component& g = ch.comp[g1];
        alive = guide_enter<R, true>(m, g);
        if (alive) {
          in = 1;
          if (guide_bounce<R, true>(m, g, trk, &inv[sizeof(R) == 8 ? g1 : 0])) {
            in = 0;
            alive = m.p > 0 && g1 + 1 < nc;
            if (alive) {
              mc = g1 + 1;
              apply_transform<R>(m, ch, mc);
            }
          }
        }
      }
      if (!alive) retire(m_isnan(m.p));
    }
    const bool tl = alive && mc > last_guide;
    const uint32_t mt = wave_meta(mc, in, rng);
    push(q1, h1, n1, alive && !tl, m, rng.c0, rng.c1, mt, in);
    if (__any_sync(kFull, tl)) push(q2, h2, n2, tl, m, rng.c0, rng.c1, mt, 0);
  };

  // Between the bounce loops no lane holds a neutron: the heavy phases have
  // the registers to themselves.  q1 always has room for what the bounce
  // loop puts back: it left at most 31 there when it filled the lanes.
  for (;;) {
    const bool more = next < end || n0 > 0;
    if (n2 >= tail_min || (n2 > 0 && n1 == 0 && !more)) {
      tail();
      continue;
    }
    if (n1 < 32 && more) {
      front();
      continue;
    }
    if (n1 == 0) break;
    Neutron<R> nt;
    zero_neutron(nt);
    uint32_t c0 = 0, c1 = 0, meta = 0;
    int c = -1;      // the component of the lane's neutron; -1 idle
    int inside = 0;  // in a guide, entered
    int nb = 0;      // reflections in that guide so far
    for (;;) {
      const unsigned idle = __ballot_sync(kFull, c < 0);
      const int nidle = __popc(idle);
      if (n2 >= tail_min || (more && n1 < nidle) ||
          (idle == kFull && n1 == 0)) {
        push(q1, h1, n1, c >= 0, nt, c0, c1,
             (meta & ~0x7fu) | (uint32_t)c & 63u | (uint32_t)inside << 6, nb);
        break;
      }
      if (idle && n1) {
        const int np = nidle < n1 ? nidle : n1;
        const int rank = __popc(idle & below);
        if (c < 0 && rank < np) {
          const int slot = (h1 + rank) % kWaveCap;
          uint32_t tb;
          wave_load<R>(q1 + slot, nt, c0, c1, meta, tb);
          c = (int)(meta & 63u);
          inside = (int)(meta >> 6 & 1u);
          nb = (int)tb;
        }
        h1 = (h1 + np) % kWaveCap;
        n1 -= np;
        __syncwarp();
      }
      // the lanes between two guides
      if (__any_sync(kFull, c >= 0 && !inside)) {
        for (int kc = g1 + 1; kc <= last_guide; ++kc) {
          if (c != kc || inside) continue;
          if (ch.comp[kc].opcode == MCV_OP_GUIDE) {
            inside = guide_enter<R, true>(nt, ch.comp[kc]);
            nb = 0;
            if (!inside) {
              retire(m_isnan(nt.p));
              c = -1;
            }
            continue;
          }
          Neutron<R> tmp = nt;
          PhiloxStream rt = wave_stream(seed, c0, c1, meta);
          k.overflow += wave_component<R>(tmp, rt, ch, kc, smt);
          nt = tmp;
          if (!(nt.p > 0)) {
            retire(m_isnan(nt.p));
            c = -1;
          } else {
            c = kc + 1;
            meta = wave_meta(c, 0, rt);
            apply_transform<R>(nt, ch, c);
          }
        }
      }
      // one reflection for every lane inside a guide, whichever guide it is
      // in (that guide's parameters are read per lane)
      bool tl = false;
      if (inside) {
        bool done =
            guide_bounce<R, true>(nt, ch.comp[c], trk, &inv[sizeof(R) == 8 ? c : 0]);
        if (!done && ++nb >= MCV_MAX_BOUNCES) {
          done = true;
          k.overflow++;
        }
        if (done) {
          inside = 0;
          if (!(nt.p > 0) || c + 1 >= nc) {
            retire(m_isnan(nt.p));
            c = -1;
          } else {
            ++c;
            apply_transform<R>(nt, ch, c);
            tl = c > last_guide;
          }
        }
      }
      if (__any_sync(kFull, tl)) {
        push(q2, h2, n2, tl, nt, c0, c1, meta, 0);
        if (tl) c = -1;
      }
    }
  }
  flush_counters(k, st);
  if constexpr (kSmem) {
    // the block's shared-memory tallies into the global ones
    __syncthreads();
    for (int kc = 0; kc < nc; ++kc) {
      const mcv_component& cp = ch.comp[kc];
      if (!(cp.flags & kFlagSmemTally) || !cp.tally) continue;
      const int m = 3 * (int)comp_nbins(cp);
      const double* src = smt + cp.ip[6];
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const double v = src[i];
        if (v != 0.0) atomicAdd(cp.tally + i, v);
      }
    }
  }
}

}  // namespace mcv
