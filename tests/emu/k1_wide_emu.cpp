// Host emulator of wide K1 programs -- TEST INFRASTRUCTURE ONLY.
//
// Plans parts the way the library does for the device (plan_passes) and runs
// the wide programs on a host array as the kernel does: tile copy into the
// folded shared layout, register groups of 32 amplitudes, steps (sign words,
// factor tables, phase runs, rotations, controlled X and swaps), the direct
// store.  Every offset is range-checked.  Passes of chunks that
// do not qualify for a wide program are counted, not run.  Nothing in the
// product loads this file.
#include <chrono>
#include <cmath>
#include <complex>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <stdexcept>
#include <vector>

#include "internal.h"

namespace hisv {
static char g_err[512];
int set_error(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}
int k1_reg_bits(int) { return 4; }
int current_tile_hint() { return 0; }
}  // namespace hisv

using namespace hisv;
using C = std::complex<double>;

namespace {

uint64_t deposit(uint64_t x, const Runs& r) {
  uint64_t out = 0;
  for (int i = 0; i < r.n; ++i) out |= ((x >> r.src[i]) & ((1ull << r.len[i]) - 1ull)) << r.dst[i];
  return out;
}

void need(bool ok, const char* what) {
  if (!ok) throw std::runtime_error(what);
}

constexpr int kPairA[10] = {0, 0, 0, 0, 1, 1, 1, 2, 2, 3}, kPairB[10] = {1, 2, 3, 4, 2, 3, 4, 3, 4, 4};

struct Emu {
  const WideProgram& P;
  int ab;
  C rnd(C x) const { return ab == 16 ? x : C(float(x.real()), float(x.imag())); }
  C coef(int i) const {
    need(i > 0 && i < P.ncoef, "coefficient out of range");
    return C(P.coef[i].x, P.coef[i].y);
  }
  C amp_coef(int i) const {
    need(i > 0 && i < P.ncoef, "coefficient out of range");
    if (ab == 16) return coef(i);
    float f[2];
    std::memcpy(f, &P.coef[i], sizeof(f));
    return C(f[0], f[1]);
  }
  C turn(C v, C c) const {
    double x = v.real(), y = v.imag();
    x = std::fma(-c.real(), y, x);
    y = std::fma(c.imag(), x, y);
    x = std::fma(-c.real(), y, x);
    return rnd(C(x, y));
  }
  void rotate(std::vector<C>& v, int j, const WideStep& S, uint32_t z) const {
    const C cy = amp_coef(S.rot[j]) * (((z >> j) & 1) ? -1.0 : 1.0);
    const int form = (S.forms >> (2 * j)) & 3;
    for (int a = 0; a < (1 << kWideBits); ++a) {
      if ((a >> j) & 1) continue;
      C &A = v[a], &B = v[a | 1 << j];
      if ((S.zmask >> j) & 1) B = turn(B, amp_coef(S.rot[j] + 1));
      if (!(form & 2)) A = rnd(A + cy.real() * B);
      B = rnd(B + cy.imag() * A);
      if (!(form & 1)) A = rnd(A + cy.real() * B);
    }
  }
  bool holds(uint32_t cthr, uint64_t couter, uint32_t thr, uint64_t gbase) const {
    return (thr & cthr) == cthr && (gbase & couter) == couter;
  }
  void step(std::vector<C>& v, const WideStep& S, uint32_t thr, uint64_t gbase, uint32_t& z) const {
    need(S.first_sign + S.nsigns <= P.nsigns, "sign out of range");
    for (int i = S.first_sign; i < S.first_sign + S.nsigns; ++i)
      if (holds(P.signs[i].cthr, P.signs[i].couter, thr, gbase)) z ^= P.signs[i].bits;
    if (S.table)
      for (unsigned e = 1; e < (1u << kWideBits); ++e) v[e] = rnd(amp_coef(S.table + e) * v[e]);
    if (S.apply) {
      for (uint32_t e = 0; e < (1u << kWideBits); ++e)
        if (__builtin_popcount((e | 32u) & z) & 1) v[e] = -v[e];
      z = 0;
    }
    int o = S.first_op;
    need(o + S.nruns + S.nperms <= P.nwops, "op out of range");
    for (int end = o + S.nruns; o < end; ++o) {
      const WideOp& op = P.ops[o];
      if (op.code == wk_neg) {
        need(op.reg < 10, "bad pair");
        for (int a = 0; a < (1 << kWideBits); ++a)
          if (((a >> kPairA[op.reg]) & 1) && ((a >> kPairB[op.reg]) & 1)) v[a] = -v[a];
        continue;
      }
      need(op.code == wk_run && op.first + op.n <= P.nconds, "bad phase run");
      C f = op.coef ? coef(op.coef) : C(1.0);
      for (int i = op.first; i < op.first + op.n; ++i)
        if (holds(P.conds[i].cthr, P.conds[i].couter, thr, gbase)) f *= coef(int(P.conds[i].coef));
      for (uint32_t e = 0; e < (1u << kWideBits); ++e)
        if ((e & op.reg) == op.reg) v[e] = rnd(f * v[e]);
    }
    for (int j = 0; j < kWideBits; ++j)
      if (S.rot[j]) rotate(v, j, S, z);
    for (int end = o + S.nperms; o < end; ++o) {
      const WideOp& op = P.ops[o];
      if (op.code == wk_cx) {
        const uint32_t m = holds(op.cthr, op.couter, thr, gbase) ? op.elems : 0u;
        for (int a = 0; a < (1 << kWideBits); ++a)
          if (!((a >> op.reg) & 1) && ((m >> a) & 1)) std::swap(v[a], v[a | 1 << op.reg]);
      } else {
        need(op.code == wk_swap && op.reg < 10, "bad op");
        for (int a = 0; a < (1 << kWideBits); ++a)
          if (((a >> kPairA[op.reg]) & 1) && !((a >> kPairB[op.reg]) & 1))
            std::swap(v[a], v[(a ^ (1 << kPairA[op.reg])) | 1 << kPairB[op.reg]]);
      }
    }
  }
  void run(std::vector<C>& sv) const {
    const int nthr = 1 << (P.m - kWideBits), bits = P.m - kWideBits, sh = ab == 8 ? 1 : 0;
    const size_t tile_bytes = size_t(ab) << P.m;
    need(P.m <= kWideMaxTileBits && bits >= 5 && bits <= kWideMaxThrBits && P.ngroups >= 1, "bad shape");
    need(P.per_thr <= kWideMaxChunks && P.ngroups <= kWideMaxGroups && P.nsteps <= kWideMaxSteps &&
             P.nsigns <= kWideMaxSigns && P.nconds <= kWideMaxConds && P.nwops <= kWideMaxOps &&
             P.ncoef <= kWideMaxCoef,
         "program out of range");
    std::vector<C> buf(tile_bytes / ab);
    std::vector<std::vector<C>> regs(nthr, std::vector<C>(1 << kWideBits));
    for (uint64_t tile = 0; tile < P.ntiles; ++tile) {
      const uint64_t gbase = deposit(tile, P.outer);
      std::vector<char> written(buf.size(), 0);
      for (int t = 0; t < nthr; ++t) {
        uint64_t gt = 0;
        uint32_t ct = 0;
        for (int b = 0; b < bits; ++b)
          if ((t >> b) & 1) {
            gt += P.gthr[b];
            ct ^= P.cthr[b];
          }
        for (int k = 0; k < P.per_thr; ++k) {
          const uint64_t g = gbase + gt + P.gchunk[k];
          const uint32_t a = ct ^ P.cslot[k];
          need(g + (1u << sh) <= sv.size() && a + 16 <= tile_bytes && a % 16 == 0, "copy out of range");
          for (int s = 0; s < (1 << sh); ++s) {
            buf[a / ab + s] = sv[g + s];
            written[a / ab + s] = 1;
          }
        }
      }
      for (char c : written) need(c, "tile not covered by the copy");
      for (int g = 0; g < P.ngroups; ++g) {
        const WideGroup& G = P.groups[g];
        const bool last = g == P.ngroups - 1;
        need(G.first_step + G.num_steps <= P.nsteps, "step out of range");
        for (int t = 0; t < nthr; ++t) {
          uint32_t tw = 0;
          for (int b = 0; b < kWideMaxThrBits; ++b)
            if ((t >> b) & 1) tw ^= G.tw[b];  // (t < 2^7: never the flips' entry)
          const uint32_t thr = tw & 0xffffu, a0 = tw >> 16;
          auto at = [&](int e) {
            uint32_t a = a0;
            for (int j = 0; j < kWideBits; ++j)
              if ((e >> j) & 1) a ^= G.dx[j];
            need(a + ab <= tile_bytes && a % ab == 0, "tile offset out of range");
            return a / ab;
          };
          std::vector<C>& v = regs[t];
          for (unsigned e = 0; e < (1u << kWideBits); ++e) v[e] = buf[at(e)];
          uint32_t z = 0;
          for (int s = G.first_step; s < G.first_step + G.num_steps; ++s)
            step(v, P.steps[s], thr, gbase, z);
          need(z == 0, "signs left at the end of a group");
          if (last) {
            uint64_t p = gbase + P.sbase;
            for (int b = 0; b < bits; ++b)
              if ((t >> b) & 1) p += P.sthr[b];
            for (unsigned e = 0; e < (1u << kWideBits); ++e) {
              uint64_t q = p;
              for (int j = 0; j < kWideBits; ++j)
                if ((e >> j) & 1) q += P.sreg[j];
              need(q < sv.size(), "store out of range");
              sv[q] = v[e];
            }
          } else {
            for (unsigned e = 0; e < (1u << kWideBits); ++e) {
              need((a0 ^ G.tw[kWideFlipEntry]) < tile_bytes, "flip offset out of range");
              need((at(e) * ab ^ G.tw[kWideFlipEntry]) == at(e ^ G.flip) * ab, "flip offset");
              buf[at(e ^ G.flip)] = v[e];
            }
          }
        }
      }
    }
  }
};

}  // namespace

extern "C" {

const char* wide_last_error() { return g_err; }

// Plan parts (mode 0: one by one, frames carried and flushed by the last; 1:
// each on its own; 2: as one call, gates moving into earlier parts' passes; 3: as
// one call, every part with its own passes, as hs_parts_run_timed) on a
// state whose qubit q sits in slot q2s[q], run the wide passes on `amps` (slot order,
// 2^n complex128, in/out; complex64 rounds).  stats: {passes, wide passes,
// groups, steps, tables}.
int wide_parts_run(int n, int dtype, const hs_gate* gates, const int32_t* offs, int nparts,
                   const int32_t* q2s_in, int tile_hint, int mode, double* amps,
                   int32_t* stats) {
  const int ab = int(amp_bytes(dtype));
  std::vector<C> sv(size_t(1) << n);
  for (size_t i = 0; i < sv.size(); ++i) {
    sv[i] = C(amps[2 * i], amps[2 * i + 1]);
    if (ab == 8) sv[i] = C(float(sv[i].real()), float(sv[i].imag()));
  }
  std::vector<int> q2s(q2s_in, q2s_in + n);
  Frames fr;
  fr.reset(n);
  int32_t st[5] = {0, 0, 0, 0, 0};
  const PassSink sink = [&](PlannedPass& ps) -> int {
    ++st[0];
    if (!ps.wide) return HS_OK;
    ++st[1];
    st[2] += ps.wide->ngroups;
    st[3] += ps.wide->nsteps;
    for (int s = 0; s < ps.wide->nsteps; ++s) st[4] += ps.wide->steps[s].table != 0;
    try {
      Emu{*ps.wide, ab}.run(sv);
    } catch (const std::exception& e) {
      std::snprintf(g_err, sizeof(g_err), "%s", e.what());
      return HS_E_INVALID;
    }
    return HS_OK;
  };
  std::vector<std::vector<LoweredGate>> parts(nparts);
  for (int p = 0; p < nparts; ++p) {
    parts[p].resize(offs[p + 1] - offs[p]);
    for (int i = offs[p]; i < offs[p + 1]; ++i) {
      const int rc = lower_gate(gates[i], n, &parts[p][i - offs[p]]);
      if (rc != HS_OK) return rc;
    }
  }
  if (mode >= 2) {
    const int rc = plan_parts(n, q2s, parts, &fr, true, tile_hint, dtype, mode == 2, sink);
    if (rc != HS_OK) return rc;
  } else {
    for (int p = 0; p < nparts; ++p) {
      std::vector<PlannedPass> passes;
      if (mode == 1) fr.reset(n);
      int rc = plan_passes(n, q2s, parts[p], &fr, mode == 1 || p == nparts - 1, tile_hint, dtype,
                           &passes);
      for (auto& ps : passes)
        if (rc == HS_OK) rc = sink(ps);
      if (rc != HS_OK) return rc;
    }
  }
  for (size_t i = 0; i < sv.size(); ++i) {
    amps[2 * i] = sv[i].real();
    amps[2 * i + 1] = sv[i].imag();
  }
  if (stats) std::memcpy(stats, st, sizeof(st));
  return HS_OK;
}
}

// Plans parts as one call without running them: {passes}, seconds {to the first pass, in all}.
extern "C" int wide_plan_time(int n, int dtype, const hs_gate* gates, const int32_t* offs,
                              int nparts, int32_t* passes, double* seconds) {
  std::vector<std::vector<LoweredGate>> parts(nparts);
  for (int p = 0; p < nparts; ++p) {
    parts[p].resize(offs[p + 1] - offs[p]);
    for (int i = offs[p]; i < offs[p + 1]; ++i) {
      const int rc = lower_gate(gates[i], n, &parts[p][i - offs[p]]);
      if (rc != HS_OK) return rc;
    }
  }
  std::vector<int> q2s(n);
  for (int q = 0; q < n; ++q) q2s[q] = q;
  Frames fr;
  fr.reset(n);
  *passes = 0;
  const auto t0 = std::chrono::steady_clock::now();
  auto now = [&] { return std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count(); };
  const int rc = plan_parts(n, q2s, parts, &fr, true, 0, dtype, true, [&](PlannedPass&) {
    if (++*passes == 1) seconds[0] = now();
    return HS_OK;
  });
  seconds[1] = now();
  return rc;
}
