// Host planner for K1: turns a gate sequence (one part, or the parts of one
// call) into tile programs.
//
// The reference runs a part by gathering, for each assignment of the outer
// qubits, the 2^k amplitudes of the part's qubits into an inner state vector,
// applying every gate there and scattering back (execute.hpp:318-470,
// state_vector.hpp:617-673; the loop nest of loop.hpp:468-962).  Here a tile
// is the same gather, widened by the three lowest slots so that every global
// access moves whole 128-byte lines of complex128 (the GPU form of opt_slots,
// execute.hpp:184-199).
// Chunks of rotations, diagonal gates, controlled X and swaps become wide
// programs (32 amplitudes per thread, kernels_wide.cu; plan_wide_chunk below);
// the rest of this comment is about the others, and about the rewriting that
// both share.
// Each tile is held by one CTA: 2^R amplitudes per thread in registers, where
// R tile bits are "register bits".  A non-diagonal gate's targets must be
// register bits; consecutive gates whose targets fit in R bits form a group,
// and between groups the tile is exchanged through shared memory so that the
// next group's targets become register bits.  Diagonal gates (Z, S, T, RZ,
// controlled phases, RZZ, ...) only scale amplitudes by a phase chosen from
// index bits, so they run in any layout and their qubits need not be in the
// tile at all.  Controls are index predicates wherever their bits are, as
// control_offset is in StateVector::apply (state_vector.hpp:410-417).
//
// Before that, the gate sequence is rewritten (Frames, internal.h): an
// uncontrolled one-qubit gate U on qubit q, preceded by the pending diagonal
// diag(1, r_q), is factored (Z-Y-Z Euler form) as
//     U diag(1, r_q) = diag(a0, a1) * RY(theta) * diag(1, e^{i beta}),
// with |beta| <= pi/2 (otherwise Z = diag(1, -1) moves to the left factor:
// RY(theta) Z = Z RY(-theta)).  RY(theta) diag(1, e^{i beta}) is applied as
// exact plane rotations, each written as three in-place shears (x -= t y;
// y += s x; x -= t y, with t = tan(angle/2), s = sin(angle)): the phase turns
// the (re, im) plane of the pair's second amplitude by beta, RY the (first,
// second) plane of the pair's real and of its imaginary parts by theta/2.
// 9 FP64 FMA per amplitude pair (6 without the phase), every one updating a
// register in place, so the kernel's op dispatch needs no register moves.
// For complex128 states the RY part is instead written, when cos(theta/2) >=
// 0.4, as two shears and a real diagonal scale that joins the pending factor
// (factor_rotation): 7 FMA per pair.  diag(a0, a1) (times that scale) joins
// the pending diagonal, which commutes with every diagonal gate (CZ, phases)
// and is absorbed by the next one-qubit gate on q.
// Diagonal one-qubit gates (S, T, RZ, ...) only update the pending diagonal.
// Whatever is pending at the end of a call is applied by one flush op.  The
// result is the reference's state up to rounding.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstddef>
#include <cstring>

#include "internal.h"

namespace hisv {

bool Frames::identity() const {
  if (G != cplx(1.0, 0.0)) return false;
  for (const auto& x : r)
    if (x != cplx(1.0, 0.0)) return false;
  return true;
}

namespace {

void build_runs(const std::vector<int>& dst_of_src, Runs* r) {
  // dst_of_src[i] = destination bit of source bit i; merge consecutive bits.
  r->n = 0;
  int i = 0;
  const int len = int(dst_of_src.size());
  while (i < len) {
    int j = i + 1;
    while (j < len && dst_of_src[j] == dst_of_src[j - 1] + 1) ++j;
    r->src[r->n] = uint8_t(i);
    r->len[r->n] = uint8_t(j - i);
    r->dst[r->n] = uint8_t(dst_of_src[i]);
    ++r->n;
    i = j;
  }
}

bool exact(cplx a, double re, double im = 0.0) { return a.real() == re && a.imag() == im; }

bool is_diagonal(const LoweredGate& g) {
  const int d = g.nt == 1 ? 2 : 4;
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c)
      if (r != c && !exact(g.m[d * r + c], 0)) return false;
  return true;
}

// ---- the factored rotation ---------------------------------------------------
// Applied to the stored pair (A, B) = (amplitude with the qubit 0, with it 1):
// first the phase b1 = e^{i beta} on B as the three shears of its (re, im)
// plane (tan(beta/2), sin(beta)), then real shears on the (A.re, B.re) and
// (A.im, B.im) planes with one coefficient pair (t, s):
//   form 0:  A += t B;  B += s A;  A += t B
//   form 1:  A += t B;  B += s A
//   form 2:             B += s A;  A += t B
// and the left diagonal diag(g0, g1) joins the pending factors.
struct Rot {
  bool has_z;        // phase part present (beta != 0)
  double tz, sz;     // shears of the phase: tan(beta/2), sin(beta)
  cplx b1;           // e^{i beta}
  int form;
  double t, s;
  cplx g0, g1;       // left diagonal
  bool flip;         // wide programs: X after the shears (and the left diagonal of X)
  bool none;         // with flip: no shears at all (an anti-diagonal gate)
};

// Two-shear forms are used when cos(theta/2) >= kShearPivot: their
// coefficients stay below ~3 and the pending scale of a qubit within
// [kShearPivot^2, kShearPivot^-2].
constexpr double kShearPivot = 0.4;
// Wide programs write the other rotations as X times one whose cosine is their
// sine, X being a relabelling of the thread's elements that costs nothing; so
// every rotation takes two shears.  Complex64 states turn at a larger cosine:
// a qubit's pending scale then stays within [0.36, 2.8], and the product over
// 40 qubits, with the global factor's 2^+-24, within the type's exponents.
constexpr double kFlipPivotC64 = 0.6;

// W = U diag(1, r): U unitary, r the qubit's pending factor, so W's first
// column is a unit vector and its second |r| = rho times one.  With
// Wn = W diag(1, 1/rho) = diag(a0, a1) RY diag(1, b1) (Z-Y-Z; RY = [[c, -sg],
// [sg, c]], c = cos(theta/2) >= 0, |arg b1| <= pi/2):
//   W = diag(a0, a1) M diag(1, b1),  M = RY diag(1, rho) = [[c, -sg rho], [sg, c rho]],
// and M is written as shears times a left diagonal:
//   form 0 (exact rotation): M = diag(1, rho) S3, S3 the three shears with
//     t = -rho tan(theta/4), s = sg / rho (rho never changes);
//   form 1 (scaled, rho <= 1): M = diag(c, rho / c) [[1, 0], [s, 1]] [[1, t], [0, 1]],
//     t = -sg rho / c, s = sg c / rho (rho grows to rho / c^2);
//   form 2 (scaled, rho > 1): M = diag(1 / c, c rho) [[1, t], [0, 1]] [[1, 0], [s, 1]],
//     s = sg / (c rho), t = -sg c rho (rho shrinks to c^2 rho).
// Forms 1 and 2 take 4 FMA per pair instead of 6 and leave a real scale on
// the qubit's two values, which the frames carry (`scaled`: complex128, and
// complex64 calls with flips; other complex64 calls keep form 0).  False when W is not of the form above to
// 1e-12 (custom C1 matrices need not be).
// `pivot` > 0: cosines below it are turned (Rot::flip).

// Whether W (its second column scaled to a unit vector) is of that form to `tol`.
// A lower left entry of exactly 0 is not: the gate is diagonal, or its upper
// right entry is the rounding residue of a product that should have been
// (custom C1 matrices), and it is applied as the matrix it is.
bool rotates(const cplx& w0, const cplx& w1, const cplx& w2, const cplx& w3, double tol) {
  const double c = std::abs(w0), s = std::abs(w2);
  return s != 0.0 && std::fabs(c * c + s * s - 1.0) <= tol &&
         std::norm(std::conj(w0) * w1 + std::conj(w2) * w3) <= tol * tol;
}

bool factor_rotation(const cplx* W, bool scaled, double pivot, Rot* R) {
  R->flip = R->none = false;
  const double c = std::abs(W[0]), s = std::abs(W[2]);
  const double rho = std::hypot(std::abs(W[1]), std::abs(W[3]));
  if (!(rho > 0.0) || !std::isfinite(rho)) return false;
  const cplx w1 = W[1] / rho, w3 = W[3] / rho;
  if (!rotates(W[0], w1, W[2], w3, 1e-12)) return false;
  if (c < pivot) {  // W = X V = X diag(g0, g1) M diag(1, b1) = diag(g1, g0) X M diag(1, b1)
    if (c == 0.0) {
      *R = Rot{false, 0.0, 0.0, cplx(1.0), 1, 0.0, 0.0, W[1], W[2], true, true};
      return true;
    }
    const cplx V[4] = {W[2], W[3], W[0], W[1]};
    if (!factor_rotation(V, scaled, 0.0, R)) return false;
    std::swap(R->g0, R->g1);
    R->flip = true;
    return true;
  }
  cplx a0, a1, b1;
  double cc = c, ss = s;
  if (c > 0.0) {
    a0 = W[0] / c;
    a1 = W[2] / s;
    // (a0, a1 are of modulus 1: dividing by them is multiplying by the conjugate)
    b1 = c >= s ? w3 * std::conj(a1) : -w1 * std::conj(a0);
    b1 /= std::abs(b1);
  } else {  // anti-diagonal
    a0 = -w1;
    a1 = W[2];
    b1 = 1.0;
    cc = 0.0;
    ss = 1.0;
  }
  // the norms of the rows are 1 to 1e-12; keep the phases unit-modulus (by the
  // exact modulus: the square root of a norm this close to 1 rounds to 1 and
  // doubles the state's error)
  a0 /= std::abs(a0);
  a1 /= std::abs(a1);
  const double nrm = std::hypot(cc, ss);
  cc /= nrm;
  ss /= nrm;
  double sign = 1.0;
  if (b1.real() < 0.0) {
    // RY(theta) diag(1, b1) = Z RY(-theta) diag(1, -b1): |arg(-b1)| <= pi/2
    b1 = -b1;
    a1 = -a1;
    sign = -1.0;
  }
  const double sg = sign * ss;
  double g0 = 1.0, g1 = rho;
  if (scaled && cc >= kShearPivot) {
    if (rho <= 1.0) {
      R->form = 1;
      R->t = -sg * rho / cc;
      R->s = sg * cc / rho;
      g0 = cc;
      g1 = rho / cc;
    } else {
      R->form = 2;
      R->s = sg / (cc * rho);
      R->t = -sg * cc * rho;
      g0 = 1.0 / cc;
      g1 = cc * rho;
    }
  } else {
    // tan(theta/4) = s / (1 + c) (half-angle formula for theta/2, c >= 0)
    R->form = 0;
    R->t = -rho * sg / (1.0 + cc);
    R->s = sg / rho;
  }
  R->g0 = a0 * g0;
  R->g1 = a1 * g1;
  R->has_z = !(b1.real() == 1.0 && b1.imag() == 0.0);
  // tan(beta/2) = sin(beta) / (1 + cos(beta)), cos(beta) >= 0
  R->tz = R->has_z ? b1.imag() / (1.0 + b1.real()) : 0.0;
  R->sz = R->has_z ? b1.imag() : 0.0;
  R->b1 = b1;
  return true;
}

// ---- rewritten gates -----------------------------------------------------------
enum RKind { RK_MATRIX = 0, RK_ROT = 1, RK_FLUSH = 2 };

struct RGate {
  RKind kind = RK_MATRIX;
  int part = 0;               // the part its gate came from
  LoweredGate g;              // targets / controls (and the matrix for RK_MATRIX)
  Rot rot;                    // RK_ROT
  std::vector<int> flq;       // RK_FLUSH: qubits
  std::vector<cplx> flr;      //           their factors r_q (applied where the bit is 1)
  cplx flG{1.0, 0.0};         //           global factor
};

bool is_swap4(const cplx* m) {
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      const bool one = (r == 0 && c == 0) || (r == 3 && c == 3) || (r == 1 && c == 2) ||
                       (r == 2 && c == 1);
      if (!exact(m[4 * r + c], one ? 1.0 : 0.0)) return false;
    }
  return true;
}

// phase r on the |1> of qubit q, as a diagonal one-qubit gate
RGate phase_gate(int q, cplx r) {
  RGate x;
  x.g.nt = 1;
  x.g.targets[0] = q;
  x.g.nc = 0;
  x.g.m[0] = 1.0;
  x.g.m[1] = x.g.m[2] = 0.0;
  x.g.m[3] = r;
  return x;
}

bool is_x(const cplx* m) {
  return exact(m[0], 0) && exact(m[1], 1) && exact(m[2], 1) && exact(m[3], 0);
}

// A controlled or two-qubit diagonal gate of unit factors as phases on sets of
// qubits (one-qubit phases and the global one join the pending diagonal, the
// others become phase gates): diag(d0, d1) on t under the controls C is d0 on C
// times d1 / d0 on C and t; a two-target diag takes the four sets of its
// targets.  False when some factor is not of unit modulus (custom C1, C2).
bool split_diagonal(const LoweredGate& g, Frames* F, std::vector<RGate>* out) {
  const int d = g.nt == 1 ? 2 : 4;
  cplx f[4];
  for (int i = 0; i < d; ++i) {
    f[i] = g.m[d * i + i];
    if (std::fabs(std::norm(f[i]) - 1.0) > 2e-12) return false;
  }
  const cplx one(1.0, 0.0);
  auto over = [&](cplx a, cplx b) { return b == one ? a : a / b; };
  // factor c on the controls and `nt` of the targets
  auto put = [&](int nt, int ta, int tb, cplx c) {
    if (c == one) return;
    if (g.nc + nt == 0) {
      F->G *= c;
    } else if (g.nc + nt == 1) {
      F->r[nt ? ta : g.controls[0]] *= c;
    } else {
      out->push_back(phase_gate(nt ? ta : g.controls[g.nc - 1], c));
      LoweredGate& x = out->back().g;
      x.nc = nt ? g.nc : g.nc - 1;
      for (int i = 0; i < x.nc; ++i) x.controls[i] = g.controls[i];
      if (nt > 1) x.controls[x.nc++] = tb;
    }
  };
  const int t0 = g.targets[0], t1 = g.targets[1];
  if (g.nt == 2 && g.nc == HS_MAX_CONTROLS) return false;  // no room for the second target
  put(0, 0, 0, f[0]);
  if (g.nt == 1) {
    put(1, t0, 0, over(f[1], f[0]));
  } else {  // reference index i = 2*b(t0) + b(t1)
    put(1, t0, 0, over(f[2], f[0]));
    put(1, t1, 0, over(f[1], f[0]));
    put(2, t0, t1, over(f[3] * f[0], f[1] * f[2]));
  }
  return true;
}

RGate flush_gate(Frames* F) {
  RGate x;
  x.kind = RK_FLUSH;
  x.g.nt = 0;
  x.g.nc = 0;
  for (int q = 0; q < int(F->r.size()); ++q)
    if (F->r[q] != cplx(1.0, 0.0)) {
      x.flq.push_back(q);
      x.flr.push_back(F->r[q]);
      F->r[q] = 1.0;
    }
  x.flG = F->G;
  F->G = 1.0;
  return x;
}

// |G| outside 2^+-lim
bool out_of_range(cplx G, double lim) {
  const double top = std::ldexp(1.0, int(2 * lim)), g = std::norm(G);
  return !(g <= top && g * top >= 1.0);
}

// `scaled`: rotations may leave real scales in the frames (factor_rotation);
// `lim`: the global factor's scale is flushed once it leaves 2^+-lim; `split`:
// diagonal gates become phases (split_diagonal), for wide programs.
void rewrite_gate(const LoweredGate& g, Frames* F, bool scaled, double pivot, double lim,
                  bool split, std::vector<RGate>* out) {
  if (g.nt == 0) return;
  const bool diag = is_diagonal(g);
  if (g.nt == 1 && g.nc == 0) {
    const int q = g.targets[0];
    const cplx rq = F->r[q];
    if (diag) {
      if (g.m[0] != cplx(0.0, 0.0)) {  // joins the pending diagonal
        F->G *= g.m[0];
        F->r[q] = g.m[3] * rq / g.m[0];
      } else {  // degenerate (custom C1): applied with the pending factor
        RGate x;
        x.g = g;
        x.g.m[3] *= rq;
        F->r[q] = 1.0;
        out->push_back(x);
      }
      return;
    }
    cplx W[4] = {g.m[0], g.m[1] * rq, g.m[2], g.m[3] * rq};
    RGate x;
    x.g = g;
    if (factor_rotation(W, scaled, pivot, &x.rot)) {
      x.kind = RK_ROT;
      F->G *= x.rot.g0;
      F->r[q] = x.rot.g1 / x.rot.g0;
    } else {
      for (int k = 0; k < 4; ++k) x.g.m[k] = W[k];
      F->r[q] = 1.0;
    }
    out->push_back(x);
    if (out_of_range(F->G, lim)) {
      // bring the stored amplitudes' scale back (one multiply of the state)
      Frames sc;
      sc.G = std::abs(F->G);
      out->push_back(flush_gate(&sc));
      F->G /= std::abs(F->G);
    }
    return;
  }
  if (diag) {  // controlled or two-qubit diagonal: commutes with the pending diagonal
    if (split && split_diagonal(g, F, out)) return;
    RGate x;
    x.g = g;
    out->push_back(x);
    return;
  }
  if (g.nt == 2 && g.nc == 0) {
    const int t0 = g.targets[0], t1 = g.targets[1];
    RGate x;
    x.g = g;
    if (is_swap4(g.m)) {
      std::swap(F->r[t0], F->r[t1]);
    } else {
      // absorb diag(1, r_t0) (x) diag(1, r_t1); reference index i = 2*b(t0) + b(t1)
      for (int c = 0; c < 4; ++c) {
        cplx d = 1.0;
        if (c & 2) d *= F->r[t0];
        if (c & 1) d *= F->r[t1];
        for (int r = 0; r < 4; ++r) x.g.m[4 * r + c] *= d;
      }
      F->r[t0] = F->r[t1] = 1.0;
    }
    out->push_back(x);
    return;
  }
  // controlled non-diagonal gate: apply the pending factors of its targets first
  for (int i = 0; i < g.nt; ++i) {
    const int t = g.targets[i];
    if (F->r[t] != cplx(1.0, 0.0)) {
      out->push_back(phase_gate(t, F->r[t]));
      F->r[t] = 1.0;
    }
  }
  RGate x;
  x.g = g;
  out->push_back(x);
}

// some parts of a call, in order
using Parts = std::vector<const std::vector<LoweredGate>*>;

// every part in turn; the gates keep their part's number
void rewrite(const Parts& parts, Frames* F, bool scaled, double pivot, double lim, bool split,
             std::vector<RGate>* out) {
  for (size_t p = 0; p < parts.size(); ++p) {
    const size_t first = out->size();
    for (const auto& g : *parts[p]) rewrite_gate(g, F, scaled, pivot, lim, split, out);
    for (size_t i = first; i < out->size(); ++i) (*out)[i].part = int(p);
  }
}

// ---- slot view -------------------------------------------------------------------
struct SlotGate {
  const RGate* rg;
  bool diag;
  int nt;
  int ts[2];                 // non-diagonal target slots
  uint64_t tmask;            // the same as a mask
  uint64_t dmask;            // slots it acts on diagonally: controls, diagonal targets
};

int coef_count(const SlotGate& sg) {
  const RGate& r = *sg.rg;
  if (r.kind == RK_ROT) return 4;  // a pair, aligned, after the two reserved entries
  if (r.kind == RK_FLUSH) return 1 + int(r.flq.size());
  if (sg.diag) return 4;
  return r.g.nt == 1 ? 4 : 16;
}

struct Layout {
  const std::vector<int>* tbit_of_slot;  // slot -> tile bit or -1
  int regpos_of_tbit[kMaxTileBits];      // tile bit -> register position or -1
};

// where a slot's bit sits for the group: register / thread / outer
void locate(const Layout& L, int slot, uint8_t* where, uint8_t* pos) {
  const int tb = (*L.tbit_of_slot)[slot];
  if (tb < 0) {
    *where = TW_OUT;
    *pos = uint8_t(slot);
  } else if (L.regpos_of_tbit[tb] >= 0) {
    *where = TW_REG;
    *pos = uint8_t(L.regpos_of_tbit[tb]);
  } else {
    *where = TW_THR;
    *pos = uint8_t(tb);
  }
}

void add_mask_bit(const Layout& L, int slot, DevOp* op) {
  uint8_t w, p;
  locate(L, slot, &w, &p);
  if (w == TW_OUT)
    op->couter |= 1ull << p;
  else if (w == TW_REG)
    op->creg |= uint16_t(1u << p);
  else
    op->cthr |= 1u << p;
}

struct Emitter {
  PartProgram* P;
  const std::vector<int>* q2s;
  void push(cplx c) {
    P->coef[P->ncoef].x = c.real();
    P->coef[P->ncoef].y = c.imag();
    ++P->ncoef;
  }
  void add(const DevOp& op) { P->ops[P->nops++] = op; }
  DevOp blank() {
    DevOp op;
    std::memset(&op, 0, sizeof(op));
    op.coef = uint16_t(P->ncoef);
    return op;
  }
};

void emit_matrix(const SlotGate& sg, const Layout& L, Emitter& E) {
  const LoweredGate& g = sg.rg->g;
  DevOp op = E.blank();
  for (int i = 0; i < g.nc; ++i) add_mask_bit(L, (*E.q2s)[g.controls[i]], &op);
  const cplx* m = g.m;
  const bool ctrl = op.creg != 0 || op.cthr != 0 || op.couter != 0;
  if (sg.diag) {
    const int s0 = (*E.q2s)[g.targets[0]];
    if (g.nt == 1 && exact(m[0], 1)) {
      // phase on the |1> of the target: a mask over controls + target
      add_mask_bit(L, s0, &op);
      if (exact(m[3], -1)) {
        op.kind = OPD_NEG;
        op.code = uint8_t(kc_neg + op.creg);
      } else {
        op.kind = OPD_PHASE;
        op.code = uint8_t(kc_ph + op.creg);
        E.push(m[3]);
      }
    } else {
      op.kind = OPD_DIAG;
      op.code = kc_diag;
      locate(L, s0, &op.t0w, &op.t0p);
      if (g.nt == 1) {
        E.push(m[0]);
        E.push(m[3]);
      } else {
        // device index q = b(t0) | b(t1) << 1; reference index i = 2*b(t0) + b(t1)
        locate(L, (*E.q2s)[g.targets[1]], &op.t1w, &op.t1p);
        E.push(m[0]);   // q=0: i=0
        E.push(m[10]);  // q=1: b0=1,b1=0 -> i=2
        E.push(m[5]);   // q=2: b0=0,b1=1 -> i=1
        E.push(m[15]);  // q=3: i=3
      }
    }
  } else if (g.nt == 1) {
    uint8_t w;
    locate(L, sg.ts[0], &w, &op.ja);
    op.kind = OP1_DENSE;
    for (int k = 0; k < 4; ++k) E.push(m[k]);
    op.code = uint8_t((ctrl ? kc_c1 : kc_d1) + op.ja);
  } else {
    uint8_t w, p0, p1;
    locate(L, sg.ts[0], &w, &p0);
    locate(L, sg.ts[1], &w, &p1);
    op.ja = std::min(p0, p1);
    op.jb = std::max(p0, p1);
    // device index q = b(ja) | b(jb) << 1; reference index i = 2*b(t0) + b(t1)
    auto ref_index = [&](int q) { return p0 < p1 ? (((q & 1) << 1) | (q >> 1)) : q; };
    cplx md[16];
    for (int qo = 0; qo < 4; ++qo)
      for (int qi = 0; qi < 4; ++qi) md[4 * qo + qi] = m[4 * ref_index(qo) + ref_index(qi)];
    static const int pair_index[4][4] = {{-1, 0, 1, 2}, {-1, -1, 3, 4}, {-1, -1, -1, 5},
                                         {-1, -1, -1, -1}};
    const int pi = pair_index[op.ja][op.jb];
    if (is_swap4(md)) {
      op.kind = OP2_SWAP;
      op.code = uint8_t(kc_sw + pi);
    } else {
      op.kind = OP2_DENSE;
      for (int k = 0; k < 16; ++k) E.push(md[k]);
      op.code = uint8_t((ctrl ? kc_c2 : kc_d2) + pi);
    }
  }
  E.add(op);
}

void emit_rot(const SlotGate& sg, const Layout& L, Emitter& E) {
  DevOp op = E.blank();
  uint8_t w;
  locate(L, sg.ts[0], &w, &op.ja);
  const Rot& r = sg.rg->rot;
  op.kind = OP1_ROT;
  op.code = uint8_t((r.has_z ? kc_zy : kc_y) + op.ja);
  op.form = uint32_t(r.form);
  // coefficient pairs start at even indices >= 2 (pair 0 marks "none")
  while (E.P->ncoef < 2 || (E.P->ncoef & 1)) E.push(0.0);
  op.coef = uint16_t(E.P->ncoef);
  E.push(cplx(r.t, r.s));
  E.push(r.has_z ? cplx(r.tz, r.sz) : cplx(0.0, 0.0));
  E.add(op);
}

// register-bit factors become phase ops; thread / outer ones and G one flush op
int emit_flush(const SlotGate& sg, const Layout& L, Emitter& E) {
  const RGate& r = *sg.rg;
  std::vector<int> rest;
  for (size_t i = 0; i < r.flq.size(); ++i) {
    uint8_t w, p;
    locate(L, (*E.q2s)[r.flq[i]], &w, &p);
    if (w == TW_REG) {
      DevOp op = E.blank();
      op.kind = OPD_PHASE;
      op.creg = uint16_t(1u << p);
      op.code = uint8_t(kc_ph + op.creg);
      E.push(r.flr[i]);
      E.add(op);
    } else {
      rest.push_back(int(i));
    }
  }
  if (rest.empty() && r.flG == cplx(1.0, 0.0)) return HS_OK;
  PartProgram* P = E.P;
  if (P->nfl + int(rest.size()) > kMaxFlush)
    return set_error(HS_E_UNSUPPORTED, "frame flush of %d entries exceeds %d", int(rest.size()),
                     kMaxFlush);
  DevOp op = E.blank();
  op.kind = OPD_FLUSH;
  op.code = kc_flush;
  op.fl_first = uint16_t(P->nfl);
  op.fl_n = uint16_t(rest.size());
  E.push(r.flG);
  for (int i : rest) {
    uint8_t w, p;
    locate(L, (*E.q2s)[r.flq[i]], &w, &p);
    P->flw[P->nfl] = w;
    P->flp[P->nfl] = p;
    ++P->nfl;
    E.push(r.flr[i]);
  }
  E.add(op);
  return HS_OK;
}

// does op x act on register bit j (target, control or mask)?
bool touches_reg(const DevOp& x, int j) {
  if (x.kind == OP1_ROT || x.kind == OP1_DENSE) {
    if (x.ja == j) return true;
  } else if (x.kind == OP2_DENSE || x.kind == OP2_SWAP) {
    if (x.ja == j || x.jb == j) return true;
  } else if (x.kind == OPD_DIAG) {
    if ((x.t0w == TW_REG && x.t0p == j) || (x.t1w == TW_REG && x.t1p == j)) return true;
  }
  return ((x.creg >> j) & 1) != 0;
}

bool diagonal_op(const DevOp& x) { return x.kind >= OPD_PHASE; }

// the sign word entry of a sign flip on register elements (mask creg) whose
// thread / outer condition is at most one bit
bool sign_entry(const DevOp& x, uint32_t* entry) {
  if (x.kind != OPD_NEG || x.creg == 0 || x.creg > 15) return false;
  const int nthr = __builtin_popcount(x.cthr), nout = __builtin_popcountll(x.couter);
  if (nthr + nout > 1) return false;
  uint32_t kind = 0, pos = 0;
  if (nthr) {
    kind = 1;
    pos = uint32_t(__builtin_ctz(x.cthr));
  } else if (nout) {
    kind = 2;
    pos = uint32_t(__builtin_ctzll(x.couter));
  }
  *entry = uint32_t(x.creg) | kind << 4 | pos << 6;
  return true;
}

// Pack the group's ops into rounds (RoundDesc) by list scheduling: op b must
// follow an earlier op a only when both act on a common register bit and not
// both are diagonal (ops act non-diagonally on register bits alone, so
// anything else commutes).  Each round takes, per register bit, the first
// rotation whose predecessors are all in earlier rounds, then every other op
// whose predecessors are scheduled (this round's rotations included), in
// program order.
void build_rounds(PartProgram* P, GroupDesc* gd) {
  gd->first_round = uint16_t(P->nrounds);
  const int o0 = gd->first_op, n = gd->num_ops;
  std::vector<uint16_t> regs(n, 0);  // register bits each op acts on
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < kRegBits; ++j)
      if (touches_reg(P->ops[o0 + i], j)) regs[i] |= uint16_t(1u << j);
  std::vector<std::vector<int>> preds(n);
  for (int b = 0; b < n; ++b)
    for (int a = 0; a < b; ++a)
      if ((regs[a] & regs[b]) && !(diagonal_op(P->ops[o0 + a]) && diagonal_op(P->ops[o0 + b])))
        preds[b].push_back(a);
  // 0: unscheduled, 1: in an earlier round, 2: in this round
  std::vector<int> state(n, 0);
  int left = n;
  auto ready = [&](int b, int need) {
    for (int a : preds[b])
      if (state[a] == 0 || state[a] > need) return false;
    return true;
  };
  while (left > 0) {
    uint32_t mask = 0, zmask = 0, pair[4] = {0, 0, 0, 0}, form[4] = {0, 0, 0, 0};
    const uint32_t first_other = uint32_t(P->nothers);
    uint32_t num_other = 0;
    for (int b = 0; b < n; ++b) {
      const DevOp& x = P->ops[o0 + b];
      if (state[b] || x.kind != OP1_ROT || ((mask >> x.ja) & 1) || !ready(b, 1)) continue;
      // an earlier unscheduled rotation on the same bit goes first
      bool first = true;
      for (int a = 0; a < b; ++a)
        if (!state[a] && P->ops[o0 + a].kind == OP1_ROT && P->ops[o0 + a].ja == x.ja) first = false;
      if (!first) continue;
      mask |= 1u << x.ja;
      if (x.code < kc_y) zmask |= 1u << x.ja;
      pair[x.ja] = x.coef / 2u;
      form[x.ja] = x.form;
      state[b] = 2;
      --left;
    }
    // sign flips on register elements with at most one thread / outer
    // condition go to the round's sign word (applied before its other ops:
    // valid while every other op placed before them is diagonal)
    uint64_t signs = 0;
    int nsign = 0;
    bool others_diag = true;
    for (bool grew = true; grew;) {
      grew = false;
      for (int b = 0; b < n; ++b) {
        const DevOp& x = P->ops[o0 + b];
        if (state[b] || x.kind == OP1_ROT || !ready(b, 2)) continue;
        uint32_t entry = 0;
        if (others_diag && nsign < 4 && sign_entry(x, &entry)) {
          signs |= uint64_t(entry) << (16 * nsign++);
        } else {
          P->others[P->nothers++] = uint8_t(o0 + b);
          ++num_other;
          if (!diagonal_op(x)) others_diag = false;
        }
        state[b] = 2;
        --left;
        grew = true;
      }
    }
    P->signs[P->nrounds] = signs;
    P->rounds[P->nrounds++] = round_pack(zmask, first_other, num_other, pair, form);
    for (int b = 0; b < n; ++b)
      if (state[b] == 2) state[b] = 1;
  }
  gd->num_rounds = uint16_t(P->nrounds - gd->first_round);
}

// ---- shared-memory layout ----------------------------------------------------
// Slot s of the tile (16 bytes) sits at s ^ fold(s), fold(s) = XOR over the
// set bits k of s of fold[k] (3 bits: a move within the 128-byte row).
uint32_t fold_of(const uint8_t* fold, uint32_t s) {
  uint32_t r = 0;
  for (; s; s &= s - 1) r ^= fold[__builtin_ctz(s)];
  return r;
}

// Byte offset change of setting tile bit tbit (the map is linear over GF(2)).
uint32_t smem_dx(const uint8_t* fold, int tbit, int dtype) {
  const int sh = dtype == HS_DTYPE_C64 ? 1 : 0;
  const uint32_t b = 1u << tbit;
  const uint32_t slot = b >> sh;
  return ((slot ^ fold_of(fold, slot)) << 4) ^ ((b & ((1u << sh) - 1u)) * uint32_t(amp_bytes(dtype)));
}

// Pick fold so that, in every register group, the lanes of one access phase
// (8 lanes of 16 bytes for complex128, 16 of 8 bytes for complex64) hit
// distinct banks: the lanes differ in the group's lowest thread tile bits,
// whose images (slot bits 0..2 after the fold, plus the in-slot bit for
// complex64) must be linearly independent.  Slot bits 0..2 keep fold 0, so
// the chunked tile copy (lanes over consecutive slots) is conflict-free too.
// Small backtracking search, the fixed fold of the earlier layout (bit k >= 3
// onto bit k mod 3) first; kept when no assignment is found.
// `regs`: bit mask of the register tile bits of each group; fold: 16 entries.
void choose_fold(uint8_t* fold, int m, int rbits, const std::vector<uint32_t>& regs, int dtype) {
  const int sh = dtype == HS_DTYPE_C64 ? 1 : 0;
  const int nslot = m - sh;
  const int lane_bits = std::min(dtype == HS_DTYPE_C64 ? 4 : 3, m - rbits);
  std::memset(fold, 0, 16);
  for (int k = 3; k < nslot; ++k) fold[k] = uint8_t(1u << (k % 3));
  if (lane_bits < 1 || nslot <= 3) return;
  // constraints: the lane tile bits of each group
  struct Lanes {
    int n;
    int bit[4];
    const int* begin() const { return bit; }
    const int* end() const { return bit + n; }
  };
  std::vector<Lanes> cons;
  cons.reserve(regs.size());
  for (uint32_t reg : regs) {
    Lanes lb{};
    for (int b = 0; b < m && lb.n < lane_bits; ++b)
      if (!((reg >> b) & 1u)) lb.bit[lb.n++] = b;
    cons.push_back(lb);
  }
  auto vec = [&](const uint8_t* F, int tbit) -> uint32_t {
    if (tbit < sh) return 8u << tbit;  // in-slot bit: its own dimension
    const int k = tbit - sh;
    return (k < 3 ? (1u << k) : 0u) ^ F[k];
  };
  // the lanes' images must have full rank: min(lanes, 3 slot bits + the
  // in-slot bit when a lane bit is one) -- complex64 lanes that share the
  // in-slot half can at best hit every bank pair twice
  auto independent = [&](const uint8_t* F, const Lanes& lb) {
    int dims = 3;
    for (int b : lb) dims += b < sh;
    const int want = std::min(lb.n, dims);
    uint32_t basis[8];
    int rank = 0;
    for (int b : lb) {
      uint32_t x = vec(F, b);
      for (int i = 0; i < rank; ++i) x = std::min(x, x ^ basis[i]);
      if (x) basis[rank++] = x;
      for (int i = rank - 1; i > 0 && basis[i] > basis[i - 1]; --i) std::swap(basis[i], basis[i - 1]);
    }
    return rank >= want;
  };
  // the highest slot bit each constraint involves (checked once it is set)
  auto top = [&](const Lanes& lb) {
    int t = -1;
    for (int b : lb) t = std::max(t, b - sh);
    return t;
  };
  uint8_t F[16];
  std::memcpy(F, fold, sizeof(F));
  bool ok = true;
  for (const auto& c : cons)
    if (!independent(F, c)) ok = false;
  if (ok) return;
  int budget = 20000;
  auto dfs = [&](auto& self, int k) -> bool {
    if (--budget < 0) return false;
    if (k >= nslot) return true;
    const uint8_t first = uint8_t(1u << (k % 3));
    for (int i = 0; i < 8; ++i) {
      const uint8_t cand = uint8_t(i == 0 ? first : (i == first ? 0 : i));
      F[k] = cand;
      bool good = true;
      for (const auto& c : cons)
        if (top(c) == k && !independent(F, c)) {
          good = false;
          break;
        }
      if (good && self(self, k + 1)) return true;
    }
    F[k] = first;
    return false;
  };
  // constraints that involve only slot bits 0..2 do not depend on fold
  if (dfs(dfs, 3)) std::memcpy(fold, F, sizeof(F));
}

void finish_layout(PartProgram* P, int dtype) {
  std::vector<uint32_t> regs(P->ngroups, 0);
  for (int g = 0; g < P->ngroups; ++g)
    for (int j = 0; j < P->rbits; ++j) regs[g] |= 1u << P->groups[g].reg_tbit[j];
  choose_fold(P->fold, P->m, P->rbits, regs, dtype);
  for (int g = 0; g < P->ngroups; ++g)
    for (int j = 0; j < P->rbits; ++j)
      P->groups[g].dx[j] = smem_dx(P->fold, P->groups[g].reg_tbit[j], dtype);
}

// ---- register groups -----------------------------------------------------------
// A second-level acyclic partition of a chunk: a group takes, in circuit order,
// every remaining gate whose non-diagonal targets fit the R register bits and
// that does not have to follow a gate left for a later group.
void take_group(const std::vector<SlotGate>& sgs, const std::vector<int>& remaining,
                const std::vector<int>& tbit_of_slot, int R, uint32_t* regs,
                std::vector<int>* members, std::vector<int>* rest) {
  uint64_t blocked = 0;  // slots held back by a deferred gate
  for (int x : remaining) {
    const SlotGate& g = sgs[x];
    uint32_t r2 = *regs;
    for (int i = 0; i < g.nt; ++i) r2 |= 1u << tbit_of_slot[g.ts[i]];
    if (((g.tmask | g.dmask) & blocked) || __builtin_popcount(r2) > R) {
      blocked |= g.tmask | g.dmask;
      rest->push_back(x);
      continue;
    }
    *regs = r2;
    members->push_back(x);
  }
}

// The same with the slots' roles told apart (wide programs): a gate acts
// diagonally on its controls and on every slot of a diagonal gate, and two
// gates that meet on such slots only commute.  Fewer groups than take_group,
// whose grouping the cost model's features are counted with.
void take_group_roles(const std::vector<SlotGate>& sgs, const std::vector<int>& remaining,
                      const std::vector<int>& tbit_of_slot, int R, uint32_t* regs,
                      std::vector<int>* members, std::vector<int>* rest) {
  uint64_t held_t = 0, held_d = 0;  // slots of deferred gates: targets, diagonal roles
  for (int x : remaining) {
    const SlotGate& g = sgs[x];
    uint32_t r2 = *regs;
    for (int i = 0; i < g.nt; ++i) r2 |= 1u << tbit_of_slot[g.ts[i]];
    if ((g.tmask & (held_t | held_d)) || (g.dmask & held_t) || __builtin_popcount(r2) > R) {
      held_t |= g.tmask;
      held_d |= g.dmask;
      rest->push_back(x);
      continue;
    }
    *regs = r2;
    members->push_back(x);
  }
}

// ---- wide programs (WideProgram, internal.h) --------------------------------------
// Whether a state of n qubits runs wide programs where its chunks qualify.
bool use_wide(int n, int dtype) {
  return k1_reg_bits(dtype) == kRegBits && n >= kWideMinTileBits;
}

// Whether gates of later parts may move into earlier passes.  Complex64 calls
// keep their parts' passes: hs_parts_run_timed, which times the parts one by one,
// gives the same bits there.
bool moves_gates(int dtype) { return dtype == HS_DTYPE_C128; }

// Gates a wide program can hold: rotations, flushes, phases, X under any
// controls, and the plain swap.
bool wide_gate(const SlotGate& s) {
  const RGate& r = *s.rg;
  if (r.kind != RK_MATRIX) return true;
  if (s.diag) return r.g.nt == 1 && exact(r.g.m[0], 1);
  if (r.g.nt == 1) return r.g.nc > 0 && is_x(r.g.m);
  return r.g.nc == 0 && is_swap4(r.g.m);
}

// A set of a group's ops.
constexpr int kRecWords = 3;
struct RecSet {
  uint64_t w[kRecWords];  // (RecSet{} is the empty one)
  void add(int i) { w[i >> 6] |= 1ull << (i & 63); }
  RecSet& operator|=(const RecSet& o) {
    for (int k = 0; k < kRecWords; ++k) w[k] |= o.w[k];
    return *this;
  }
  RecSet operator|(const RecSet& o) const {
    RecSet r = *this;
    return r |= o;
  }
  RecSet minus(const RecSet& o) const {
    RecSet r;
    for (int k = 0; k < kRecWords; ++k) r.w[k] = w[k] & ~o.w[k];
    return r;
  }
  bool within(const RecSet& o) const {
    for (int k = 0; k < kRecWords; ++k)
      if (w[k] & ~o.w[k]) return false;
    return true;
  }
  template <typename F>
  void each(F&& f) const {  // in order
    for (int k = 0; k < kRecWords; ++k)
      for (uint64_t x = w[k]; x; x &= x - 1) f(64 * k + __builtin_ctzll(x));
  }
};

// Whether every gate of a call ends up in wide programs, which alone hold
// rotations with a flip: the kinds wide_gate takes, and pending factors (from
// earlier calls, custom gates among them) that factor_rotation can take in.
bool all_wide(const Parts& parts, const Frames& F) {
  for (const cplx& r : F.r)
    if (!(std::norm(r) > 1e-6 && std::norm(r) < 1e6)) return false;
  for (const auto* gates : parts)
    for (const LoweredGate& g : *gates) {
      if (g.nt == 0) continue;
      if (is_diagonal(g)) {
        for (int i = 0; i < (g.nt == 1 ? 2 : 4); ++i)
          if (std::fabs(std::norm(g.m[(g.nt == 1 ? 3 : 5) * i]) - 1.0) > 2e-12) return false;
        if (g.nt == 2 && g.nc == HS_MAX_CONTROLS) return false;
      } else if (g.nt == 1 && g.nc == 0) {
        // a rotation, well within what factor_rotation asks for
        const double tol = 2.5e-13;
        if (!(std::fabs(std::norm(g.m[1]) + std::norm(g.m[3]) - 1.0) <= tol &&
              rotates(g.m[0], g.m[1], g.m[2], g.m[3], tol)))
          return false;
      } else if (!(g.nt == 1 && is_x(g.m)) && !(g.nt == 2 && g.nc == 0 && is_swap4(g.m))) {
        return false;
      }
    }
  return true;
}

// An op of a group before it is scheduled.
struct WideRec {
  enum Kind { kRot, kNeg, kPhase, kCx, kSwap } kind;
  uint32_t mask = 0;     // register bits it acts on (a cx's controls included)
  uint32_t target = 0;   // of these, the ones it acts on non-diagonally
  int j = 0, jb = 0;
  uint32_t cthr = 0;     // thread / outer condition
  uint64_t couter = 0;
  cplx c{1.0, 0.0};      // kPhase
  const Rot* rot = nullptr;
  bool z = false;        // kRot: its phase part is still to be applied
  bool global = false;   // kPhase: a flush's global factor
  bool done = false;
  bool diag() const { return kind == kNeg || kind == kPhase; }
  bool uniform() const { return cthr == 0 && couter == 0; }
};

void wide_records(const SlotGate& sg, const Layout& L, const std::vector<int>& q2s,
                  std::vector<WideRec>* out) {
  const RGate& r = *sg.rg;
  auto bit = [&](int q, WideRec* w) {  // adds qubit q to the masks
    uint8_t where, pos;
    locate(L, q2s[q], &where, &pos);
    if (where == TW_OUT)
      w->couter |= 1ull << pos;
    else if (where == TW_REG)
      w->mask |= 1u << pos;
    else
      w->cthr |= 1u << pos;
  };
  auto regpos = [&](int slot) { return L.regpos_of_tbit[(*L.tbit_of_slot)[slot]]; };
  WideRec w;
  if (r.kind == RK_FLUSH) {
    w.kind = WideRec::kPhase;
    for (size_t i = 0; i < r.flq.size(); ++i) {
      WideRec x = w;
      bit(r.flq[i], &x);
      x.c = r.flr[i];
      out->push_back(x);
    }
    w.c = r.flG;
    w.global = true;
    out->push_back(w);
    return;
  }
  const LoweredGate& g = r.g;
  if (r.kind == RK_ROT) {
    w.kind = WideRec::kRot;
    w.j = regpos(sg.ts[0]);
    w.mask = w.target = 1u << w.j;
    w.rot = &r.rot;
    w.z = r.rot.has_z;
  } else if (sg.diag) {
    for (int i = 0; i < g.nc; ++i) bit(g.controls[i], &w);
    bit(g.targets[0], &w);
    w.kind = exact(g.m[3], -1) ? WideRec::kNeg : WideRec::kPhase;
    w.c = g.m[3];
  } else if (g.nt == 1) {
    w.kind = WideRec::kCx;
    for (int i = 0; i < g.nc; ++i) bit(g.controls[i], &w);
    w.j = regpos(sg.ts[0]);
    w.target = 1u << w.j;
    w.mask |= w.target;
  } else {
    w.kind = WideRec::kSwap;
    const int a = regpos(sg.ts[0]), b = regpos(sg.ts[1]);
    w.j = std::min(a, b);
    w.jb = std::max(a, b);
    w.mask = w.target = 1u << a | 1u << b;
  }
  out->push_back(w);
}

// Schedules a group's ops into steps.  Op b has to follow an earlier op a when
// they share a register bit on which one of them is not diagonal.  A step runs
// its diagonal ops (signs, factor table, phase runs), then its rotations, then
// its controlled X and swaps.  Conditional signs join the thread's sign word as
// soon as they may; other diagonal ops wait until a step acts on their bits, so
// that runs with one register mask are shared; the phase parts of every
// rotation that is next on its bit and the register-only factors of modulus 1
// join the table of the first step that needs one.  `reserve`: coefficients to
// be left for the program's later groups.
//
// Flips (Rot::flip) relabel the elements: element e holds the amplitude of
// register index e ^ xm.  A rotation on a flipped bit has its pair's roles, so
// its two shears, exchanged; its phase turns the other amplitude back instead,
// up to a global factor that `gamma` collects for the next flush; diagonal ops
// are written for e ^ xm (a condition "bit is 0" as the unconditional factor
// times its inverse on the bit, a CZ as one and a Z).  The group's end stores
// element e where e ^ xm belongs.
int wide_steps(std::vector<WideRec>& rec, int dtype, WideProgram* P, WideGroup* G, int reserve,
               cplx* gamma) {
  const int n = int(rec.size()), size = 1 << kWideBits;
  G->first_step = uint16_t(P->nsteps);
  // dependencies as bit sets over the ops: the last non-diagonal op on a bit,
  // and for a non-diagonal op the diagonal ones since (what came before those
  // follows from them)
  if (n > kRecWords * 64) return set_error(HS_E_UNSUPPORTED, "%d ops in a group", n);
  RecSet preds[kRecWords * 64], done{}, diag{}, perm{};
  uint8_t queue[kWideBits][kRecWords * 64];  // the non-diagonal ops of each bit, in order
  int queued[kWideBits] = {}, head[kWideBits] = {};
  {
    int last[kWideBits];
    RecSet since[kWideBits] = {};
    for (int j = 0; j < kWideBits; ++j) last[j] = -1;
    for (int b = 0; b < n; ++b) {
      RecSet p{};
      for (int j = 0; j < kWideBits; ++j) {
        if (!((rec[b].mask >> j) & 1u)) continue;
        if (last[j] >= 0) p.add(last[j]);
        if ((rec[b].target >> j) & 1u) {
          p |= since[j];
          last[j] = b;
          queue[j][queued[j]++] = uint8_t(b);
          since[j] = RecSet{};
        } else {
          since[j].add(b);
        }
      }
      preds[b] = p;
      if (rec[b].diag()) diag.add(b);
      if (rec[b].kind == WideRec::kCx || rec[b].kind == WideRec::kSwap) perm.add(b);
    }
  }
  int left = n;
  bool pend_any = false;      // signs wait in the word
  uint32_t pend = 0;          // register bits they act on
  auto push_coef = [&](cplx c) {
    P->coef[P->ncoef].x = c.real();
    P->coef[P->ncoef].y = c.imag();
    return P->ncoef++;
  };
  auto push_amp_coef = [&](cplx c) {  // in the amplitudes' precision
    if (dtype == HS_DTYPE_C128) return push_coef(c);
    const float f[2] = {float(c.real()), float(c.imag())};
    std::memcpy(&P->coef[P->ncoef], f, sizeof(f));
    return P->ncoef++;
  };
  // a diagonal op may run at the start of this step: everything it follows is done
  auto available = [&](int i) { return preds[i].within(done); };
  // a non-diagonal op may run in this step: what it follows is done, or is a
  // diagonal op that may run at the start of the step (`open`)
  RecSet open{};
  auto ready = [&](int i) { return preds[i].within(done | open); };
  // a conditional sign of the thread or of one register bit
  auto is_sign = [&](int i) {
    return rec[i].kind == WideRec::kNeg && (rec[i].mask & (rec[i].mask - 1)) == 0 &&
           !(rec[i].uniform() && rec[i].mask != 0);
  };
  // a factor of modulus 1 on register bits alone
  auto unit = [&](int i) {
    return rec[i].uniform() && rec[i].mask != 0 && std::fabs(std::norm(rec[i].c) - 1.0) < 1e-12;
  };
  auto finish = [&](int i) {
    rec[i].done = true;
    done.add(i);
    --left;
  };
  uint32_t xm = 0;
  struct Piece {  // a factor of a run
    uint32_t mask, cthr;
    uint64_t couter;
    cplx c;
  };
  std::vector<Piece> pieces;
  std::vector<int> perms, run;
  auto is_pair = [&](int i) {
    return rec[i].kind == WideRec::kNeg && rec[i].uniform() && __builtin_popcount(rec[i].mask) == 2;
  };
  while (left > 0 || pend_any) {
    if (P->nsteps >= kWideMaxSteps) return set_error(HS_E_UNSUPPORTED, "too many steps in a pass");
    WideStep& S = P->steps[P->nsteps++];
    std::memset(&S, 0, sizeof(S));
    S.first_sign = uint16_t(P->nsigns);
    S.first_op = uint16_t(P->nwops);
    open = RecSet{};
    diag.minus(done).each([&](int i) {
      if (available(i)) open.add(i);
    });
    // ---- the step's non-diagonal ops
    int rot[kWideBits];
    uint32_t touched = 0, moved = 0;  // register bits acted on; by controlled X and swaps
    perms.clear();
    for (int j = 0; j < kWideBits; ++j) {
      rot[j] = -1;
      while (head[j] < queued[j] && rec[queue[j][head[j]]].done) ++head[j];
      if (head[j] == queued[j]) continue;
      const int i = queue[j][head[j]];  // (a later op on the bit has to follow it)
      if (rec[i].kind == WideRec::kRot && ready(i)) {
        rot[j] = i;
        touched |= 1u << j;
      }
    }
    perm.minus(done).each([&](int i) {
      RecSet here = done | open;  // the step's rotations and earlier perms run first
      for (int j = 0; j < kWideBits; ++j)
        if (rot[j] >= 0) here.add(rot[j]);
      for (int a : perms) here.add(a);
      if (preds[i].within(here)) {
        perms.push_back(i);
        moved |= rec[i].target;
      }
    });
    touched |= moved;
    const bool last = touched == 0;  // diagonal ops alone are left
    if (xm) {
      // runs with several flipped bits, or more pieces than there is room for:
      // undo those flips first (a step of plain X)
      uint32_t undo = 0;
      int extra = 0;
      open.each([&](int i) {
        if (is_sign(i) || is_pair(i) || !(rec[i].mask & xm) || !(last || (rec[i].mask & touched)))
          return;
        if (__builtin_popcount(rec[i].mask & xm) > 1 || rec[i].c == cplx(0.0, 0.0))
          undo |= rec[i].mask & xm;
        ++extra;
      });
      const int room = std::min(kWideMaxConds - P->nconds, kWideMaxOps - 8 - P->nwops) -
                       (reserve / 2 + left);
      if (extra > room) undo |= xm;
      if (undo) {
        S.apply = pend_any && (pend & undo);
        if (S.apply) {
          pend_any = false;
          pend = 0;
        }
        for (int j = 0; j < kWideBits; ++j) {
          if (!((undo >> j) & 1u)) continue;
          WideOp& op = P->ops[P->nwops++];
          std::memset(&op, 0, sizeof(op));
          op.code = wk_cx;
          op.reg = uint8_t(j);
          op.elems = ~0u;
          ++S.nperms;
        }
        xm &= ~undo;
        continue;
      }
    }
    // ---- diagonal ops
    run.clear();
    auto add_sign = [&](uint32_t bits, uint32_t cthr, uint64_t couter) {
      WideSign& q = P->signs[P->nsigns++];
      q.bits = bits;
      q.cthr = cthr;
      q.couter = couter;
      ++S.nsigns;
      pend_any = true;
      pend |= bits & 31u;
    };
    open.each([&](int i) {
      if (is_sign(i)) {
        add_sign(rec[i].mask == 0 || (rec[i].mask & xm) ? rec[i].mask | 32u : rec[i].mask,
                 rec[i].cthr, rec[i].couter);
        finish(i);
      } else if (last || (rec[i].mask & touched)) {
        run.push_back(i);
      }
    });
    // phase parts: of the rotations next on their bits
    int zs[kWideBits], nz = 0;
    bool need = false;
    for (int j = 0; j < kWideBits; ++j) {
      if (head[j] == queued[j]) continue;
      const int i = queue[j][head[j]];
      // (nothing non-diagonal on the bit is ahead of it)
      if (rec[i].kind == WideRec::kRot && rec[i].z) {
        zs[nz++] = i;
        need |= rot[j] == i;
      }
    }
    // multiply-adds per amplitude of a table (2^R - 1 complex factors) and of
    // the same work op by op; a negation counts its integer operations
    double single = 1.5 * nz;
    bool any = need;
    for (int i : run)
      if (unit(i)) {
        any = true;
        const int bits = __builtin_popcount(rec[i].mask);
        single += rec[i].kind == WideRec::kNeg && bits == 2 ? 0.5 : 4.0 / (1 << bits);
      }
    if (any && single > 4.0 * (size - 1) / size &&
        P->ncoef + size + reserve + 2 * n <= kWideMaxCoef) {
      cplx f[1 << kWideBits], by_bit[kWideBits];
      for (auto& x : by_bit) x = 1.0;
      for (int k = 0; k < nz; ++k) {
        by_bit[rec[zs[k]].j] = rec[zs[k]].rot->b1;
        rec[zs[k]].z = false;
      }
      f[0] = 1.0;
      for (int e = 1; e < size; ++e)  // the lowest set bit's factor times the others'
        f[e] = f[e & (e - 1)] * by_bit[__builtin_ctz(unsigned(e))];
      open.minus(done).each([&](int i) {  // every such factor that may run now
        if (!unit(i)) return;
        for (uint32_t e = rec[i].mask; e < uint32_t(size); e = (e + 1) | rec[i].mask)
          f[e] *= rec[i].c;
        run.erase(std::remove(run.begin(), run.end(), i), run.end());
        finish(i);
      });
      S.table = uint16_t(P->ncoef);
      const cplx first = f[xm];  // element 0's, left out of the table
      *gamma *= first;
      for (int e = 0; e < size; ++e)
        push_amp_coef(xm ? f[uint32_t(e) ^ xm] * std::conj(first) : f[e]);
    }
    // pairs on flipped bits leave a Z on the other bit
    for (int i : run)
      if (is_pair(i) && (rec[i].mask & xm)) {
        const uint32_t a = rec[i].mask & (0u - rec[i].mask), b = rec[i].mask ^ a;
        add_sign(((xm & a) ? b : 0u) | ((xm & b) ? a : 0u) | ((xm & a) && (xm & b) ? 32u : 0u), 0, 0);
      }
    S.apply = pend_any && ((pend & moved) || (last && left == int(run.size())));
    if (S.apply) {
      pend_any = false;
      pend = 0;
    }
    // negations of register pairs, then runs, one per register mask
    pieces.clear();
    for (int i : run) {
      const WideRec& x = rec[i];
      if (is_pair(i)) {
        WideOp& op = P->ops[P->nwops++];
        std::memset(&op, 0, sizeof(op));
        op.code = wk_neg;
        op.reg = uint8_t(wide_pair(__builtin_ctz(x.mask), 31 - __builtin_clz(x.mask)));
        ++S.nruns;
      } else if (x.mask & xm) {  // one flipped bit: on 0 = everywhere, undone on 1
        pieces.push_back({x.mask & ~xm, x.cthr, x.couter, x.c});
        pieces.push_back({x.mask, x.cthr, x.couter, 1.0 / x.c});
      } else {
        cplx c = x.c;
        if (x.global) {
          c *= *gamma;
          *gamma = 1.0;
        }
        if (c != cplx(1.0, 0.0)) pieces.push_back({x.mask, x.cthr, x.couter, c});
      }
      finish(i);
    }
    for (size_t k = 0; k < pieces.size(); ++k) {
      const uint32_t mask = pieces[k].mask;
      if (mask > 31u) continue;  // taken by an earlier run
      WideOp& op = P->ops[P->nwops++];
      std::memset(&op, 0, sizeof(op));
      op.code = wk_run;
      op.reg = uint8_t(mask);
      op.first = uint16_t(P->nconds);
      cplx c = 1.0;
      for (size_t l = k; l < pieces.size(); ++l) {
        Piece& x = pieces[l];
        if (x.mask != mask) continue;
        if (x.cthr == 0 && x.couter == 0) {
          c *= x.c;
        } else {
          WideCond& q = P->conds[P->nconds++];
          q.cthr = x.cthr;
          q.couter = x.couter;
          q.coef = uint32_t(push_coef(x.c));
          ++op.n;
        }
        x.mask = ~0u;
      }
      if (c != cplx(1.0, 0.0)) op.coef = uint16_t(push_coef(c));
      ++S.nruns;
    }
    uint32_t flips = 0;
    for (int j = 0; j < kWideBits; ++j) {
      if (rot[j] < 0) continue;
      const Rot& r = *rec[rot[j]].rot;
      const bool turned = (xm >> j) & 1u;  // the pair's roles are exchanged
      if (!r.none) {
        S.forms |= uint16_t((turned ? 3 - r.form : r.form) << (2 * j));
        S.rot[j] = uint16_t(push_amp_coef(turned ? cplx(r.s, r.t) : cplx(r.t, r.s)));
        if (rec[rot[j]].z) {
          S.zmask |= uint8_t(1u << j);
          push_amp_coef(turned ? cplx(-r.tz, -r.sz) : cplx(r.tz, r.sz));
          if (turned) *gamma *= r.b1;
        }
      }
      if (r.flip) flips |= 1u << j;
      finish(rot[j]);
    }
    xm ^= flips;
    for (int i : perms) {
      WideOp& op = P->ops[P->nwops++];
      std::memset(&op, 0, sizeof(op));
      if (rec[i].kind == WideRec::kCx) {
        op.code = wk_cx;
        op.reg = uint8_t(rec[i].j);
        const uint32_t ctl = rec[i].mask & ~rec[i].target;
        for (uint32_t e = 0; e < uint32_t(size); ++e)
          if (((e ^ xm) & ctl) == ctl) op.elems |= 1u << e;
      } else {
        const uint32_t a = (xm >> rec[i].j) & 1u, b = (xm >> rec[i].jb) & 1u;
        if (a != b) xm ^= rec[i].mask;  // the flips change places too
        op.code = wk_swap;
        op.reg = uint8_t(wide_pair(rec[i].j, rec[i].jb));
      }
      op.cthr = rec[i].cthr;
      op.couter = rec[i].couter;
      ++S.nperms;
      finish(i);
    }
  }
  G->flip = uint8_t(xm);
  G->num_steps = uint16_t(P->nsteps - G->first_step);
  return HS_OK;
}

// the shared-memory layout and the copy / store tables
void finish_wide(WideProgram* P, const std::vector<uint32_t>& regs, int dtype) {
  const int sh = dtype == HS_DTYPE_C64 ? 1 : 0;
  const int thr_bits = P->m - kWideBits;
  choose_fold(P->fold, P->m, kWideBits, regs, dtype);
  uint64_t slot[kWideMaxTileBits];  // global and shared offset of each tile bit
  uint32_t off[kWideMaxTileBits];
  for (int b = 0; b < P->m; ++b) {
    slot[b] = uint64_t(1) << P->tile_slot[b];
    off[b] = smem_dx(P->fold, b, dtype);
  }
  for (int g = 0; g < P->ngroups; ++g) {
    WideGroup& G = P->groups[g];
    for (int j = 0; j < kWideBits; ++j) {
      G.dx[j] = off[G.reg_tbit[j]];
      if ((G.flip >> j) & 1u) G.tw[kWideFlipEntry] ^= G.dx[j];
    }
    int b = 0;
    for (int tb = 0; tb < P->m; ++tb) {
      if ((regs[g] >> tb) & 1u) continue;
      G.tw[b] = 1u << tb | off[tb] << 16;
      if (g == P->ngroups - 1) P->sthr[b] = slot[tb];
      ++b;
    }
  }
  const WideGroup& last = P->groups[P->ngroups - 1];
  for (int j = 0; j < kWideBits; ++j) {  // (a flipped bit's element 0 is the one with the bit set)
    const bool f = (last.flip >> j) & 1u;
    P->sreg[j] = f ? -int64_t(slot[last.reg_tbit[j]]) : int64_t(slot[last.reg_tbit[j]]);
    if (f) P->sbase += slot[last.reg_tbit[j]];
  }
  // chunk c = t + k * threads holds tile indices [c << sh, (c + 1) << sh)
  P->per_thr = ((1 << P->m) >> sh) >> thr_bits;
  for (int b = 0; b < thr_bits; ++b) {
    P->gthr[b] = slot[b + sh];
    P->cthr[b] = off[b + sh];
  }
  P->gchunk[0] = 0;
  P->cslot[0] = 0;
  for (int k = 1; k < P->per_thr; ++k) {
    const int b = __builtin_ctz(unsigned(k)) + sh + thr_bits, rest = k & (k - 1);
    P->gchunk[k] = P->gchunk[rest] | slot[b];
    P->cslot[k] = P->cslot[rest] ^ off[b];
  }
}

// A chunk (gates of sgs, every one a wide_gate) as wide programs: one, or more
// where its groups outgrow a program.
int plan_wide_chunk(int n, int dtype, const std::vector<int>& q2s,
                    const std::vector<SlotGate>& sgs, std::vector<int> remaining,
                    const std::vector<int>& tile, const std::vector<int>& tbit_of_slot,
                    cplx* gamma, std::vector<PlannedPass>* passes) {
  const int m = int(tile.size());
  WideProgram* P = nullptr;
  std::vector<uint32_t> regs_of;
  auto new_program = [&]() {
    if (P) finish_wide(P, regs_of, dtype);
    regs_of.clear();
    passes->emplace_back();
    passes->back().wide.reset(new WideProgram);
    P = passes->back().wide.get();
    // the lists are written entry by entry; only what is read is initialised
    std::memset(P, 0, offsetof(WideProgram, groups));
    P->n = n;
    P->m = m;
    P->ntiles = 1ull << (n - m);
    P->ncoef = 1;
    build_runs(tile, &P->tile);
    for (int b = 0; b < m; ++b) P->tile_slot[b] = uint8_t(tile[b]);
    std::vector<int> outer;
    outer.reserve(n);
    for (int s = 0; s < n; ++s)
      if (tbit_of_slot[s] < 0) outer.push_back(s);
    build_runs(outer, &P->outer);
  };
  new_program();
  std::vector<int> members, rest;
  std::vector<WideRec> rec;
  members.reserve(remaining.size());
  rec.reserve(remaining.size() + 2);
  while (!remaining.empty()) {
    uint32_t rmask = 0;
    members.clear();
    rest.clear();
    rec.clear();
    take_group_roles(sgs, remaining, tbit_of_slot, kWideBits, &rmask, &members, &rest);
    if (P->ngroups == kWideMaxGroups) new_program();
    WideGroup& G = P->groups[P->ngroups++];
    std::memset(&G, 0, sizeof(G));
    // free register bits take the highest tile bits, so that the lanes stay on
    // the low, contiguous slots
    for (int b = m - 1; b >= 0 && __builtin_popcount(rmask) < kWideBits; --b) rmask |= 1u << b;
    regs_of.push_back(rmask);
    Layout L;
    L.tbit_of_slot = &tbit_of_slot;
    for (int b = 0, j = 0; b < kMaxTileBits; ++b) {
      L.regpos_of_tbit[b] = -1;
      if ((rmask >> b) & 1u) {
        G.reg_tbit[j] = uint8_t(b);
        L.regpos_of_tbit[b] = j++;
      }
    }
    for (int x : members) wide_records(sgs[x], L, q2s, &rec);
    P->nops += int(rec.size());
    // every later op needs at most two coefficients
    int reserve = 2;
    for (int x : rest)
      reserve += sgs[x].rg->kind == RK_FLUSH ? 2 + 2 * int(sgs[x].rg->flq.size()) : 2;
    HS_TRY(wide_steps(rec, dtype, P, &G, reserve, gamma));
    remaining.swap(rest);
  }
  finish_wide(P, regs_of, dtype);
  return HS_OK;
}

// What a program has room for, as the chunk grows.
struct ChunkRoom {
  int ops = 0, coefs = 0, fls = 0;
  bool add(const SlotGate& g) {
    const bool fl = g.rg->kind == RK_FLUSH;
    const int f = fl ? int(g.rg->flq.size()) : 0, o = fl ? 1 + f : 1, c = coef_count(g);
    if (ops + o > kMaxOps || coefs + c > kMaxCoef || fls + f > kMaxFlush) return false;
    ops += o;
    coefs += c;
    fls += f;
    return true;
  }
};

// Lists that a call's windows share.
struct PlanLists {
  std::vector<RGate> rg;
  std::vector<SlotGate> sgs;
};

// The planner of both program kinds, for some parts of a call: into `programs`
// (PartPrograms only) or, with `sink`, as PartPrograms and WidePrograms, handed
// over pass by pass.  A pass takes what fits of the first part left (in order, up
// to the first gate that does not fit).  Given a sink, a pass of wide gates also
// takes, where that saves passes, every gate of the parts after it that fits the
// tile and has to follow no gate left behind: a part bounded by the qubits its
// gates touch leaves room in the tile, which holds targets alone, and parts so
// used up cost no pass of their own (27 qubits, parts of 9 touched qubits: 9
// passes instead of 13; 20 random layers of 20 qubits in parts of 10: 9 instead
// of 26).  `flips`: rotations beyond the pivot become flips (all_wide).
int plan_chunks(int n, const std::vector<int>& q2s, const Parts& gates, Frames* fr, bool flush,
                int tile_bits_hint, int dtype, bool flips, PlanLists* lists,
                std::vector<PartProgram>* programs, const PassSink* sink) {
  if (n < 1 || n > 63) return set_error(HS_E_INVALID, "bad qubit count %d", n);
  if (int(fr->r.size()) != n) fr->reset(n);
  std::vector<RGate>& rg = lists->rg;
  rg.clear();
  size_t count = 2;
  for (const auto* g : gates) count += g->size();
  rg.reserve(count);
  // keep the carried scale within a few dozen binary orders (it moves with
  // the scaled rotation forms and non-unitary diagonal gates)
  const double lim = dtype == HS_DTYPE_C64 ? 24.0 : 48.0;
  const bool wide = sink && use_wide(n, dtype);
  const double pivot = !flips ? 0.0 : dtype == HS_DTYPE_C128 ? kShearPivot : kFlipPivotC64;
  rewrite(gates, fr, dtype == HS_DTYPE_C128 || flips, pivot, lim, wide, &rg);
  if (flush) {
    if (!fr->identity()) {
      rg.push_back(flush_gate(fr));
      rg.back().part = int(gates.size()) - 1;
    }
  } else if (out_of_range(fr->G, lim)) {
    Frames scale;
    scale.G = std::abs(fr->G);
    rg.push_back(flush_gate(&scale));
    fr->G /= std::abs(fr->G);
  }
  // one tile buffer per CTA: up to 2^12 amplitudes (64 KiB of complex128)
  const int max_tile = std::min(n, max_tile_bits(dtype));
  const int rbits = k1_reg_bits(dtype);
  // automatic size: complex128 tiles of 2^10 (CTAs of 64 threads x 16
  // amplitudes, ten per SM), complex64 tiles of 2^12
  const int auto_m = dtype == HS_DTYPE_C128 ? 10 : max_tile;
  const int m_target = std::min(max_tile, tile_bits_hint > 0 ? tile_bits_hint : auto_m);
  // keep the three lowest slots in the tile where they fit, so that global
  // accesses come in contiguous runs of at least 8 amplitudes (128 bytes of
  // complex128: whole L2 lines; with 64-byte runs the other half of each
  // line is fetched as well and often evicted before its own tile reads it
  // -- 3.7% slower at 33 qubits)
  const int low_min = std::min(n, 3);
  std::vector<SlotGate>& sgs = lists->sgs;
  sgs.clear();
  sgs.reserve(rg.size());
  for (const auto& r : rg) {
    SlotGate s;
    s.rg = &r;
    s.nt = 0;
    s.tmask = s.dmask = 0;
    if (r.kind == RK_FLUSH) {
      s.diag = true;
      for (int q : r.flq) s.dmask |= 1ull << q2s[q];
    } else {
      s.diag = r.kind == RK_MATRIX && is_diagonal(r.g);
      for (int i = 0; i < r.g.nt; ++i) {
        const int t = q2s[r.g.targets[i]];
        if (s.diag) {
          s.dmask |= 1ull << t;
        } else {
          s.tmask |= 1ull << t;
          s.ts[s.nt++] = t;
        }
      }
      for (int i = 0; i < r.g.nc; ++i) s.dmask |= 1ull << q2s[r.g.controls[i]];
    }
    sgs.push_back(s);
  }
  auto low_union_size = [&](uint64_t t, int lows) {
    return __builtin_popcountll(t | ((1ull << lows) - 1ull));
  };
  // a chunk only needs the low slots the 16-byte chunk copy requires (slot 0
  // for complex64); where the targets leave room the tile takes all three:
  // shorter runs cost less than another pass
  const int low_need = std::min(n, dtype == HS_DTYPE_C64 ? 1 : 0);
  // ---- chunks: gates whose non-diagonal target slots (+ low slots) fit one tile
  struct Chunk {
    std::vector<int> gates;
    uint64_t tset = 0;
    bool wide = false;
  };
  // the next gate joins the chunk if it is of the same part and fits
  auto join = [&](Chunk* c, ChunkRoom* room, int x, int part) -> bool {
    const SlotGate& g = sgs[x];
    if (g.rg->part != part || low_union_size(c->tset | g.tmask, low_need) > max_tile ||
        !room->add(g))
      return false;
    c->tset |= g.tmask;
    c->gates.push_back(x);
    c->wide = c->wide && wide_gate(g);
    return true;
  };
  std::vector<Chunk> chunks, merged;
  for (int x = 0; x < int(sgs.size());) {
    chunks.emplace_back();
    Chunk& c = chunks.back();
    c.wide = wide;
    c.gates.reserve(std::min<size_t>(sgs.size() - size_t(x), 64));
    ChunkRoom room;
    const int part = sgs[x].rg->part;
    while (x < int(sgs.size()) && join(&c, &room, x, part)) ++x;
    if (c.gates.empty()) return set_error(HS_E_INVALID, "gate does not fit a tile");
  }
  // The same with gates moved forward.  Every chunk walks the gates that are left,
  // which plan_parts bounds.
  auto cut_merged = [&](std::vector<Chunk>* out) {
    std::vector<int> left(sgs.size()), rest;
    for (size_t x = 0; x < sgs.size(); ++x) left[x] = int(x);
    while (!left.empty()) {
      out->emplace_back();
      Chunk& c = out->back();
      ChunkRoom room;
      const int part = sgs[left[0]].rg->part;
      c.wide = true;
      size_t i = 0;
      while (i < left.size() && join(&c, &room, left[i], part)) ++i;
      rest.clear();
      if (c.wide && low_union_size(c.tset, low_min) <= max_tile) {
        uint64_t held_t = 0, held_d = 0;  // slots of gates left behind, as in take_group_roles
        const uint64_t every = (1ull << n) - 1ull;
        for (; i < left.size() && held_t != every; ++i) {
          const SlotGate& g = sgs[left[i]];
          if ((g.tmask & (held_t | held_d)) || (g.dmask & held_t) || !wide_gate(g) ||
              low_union_size(c.tset | g.tmask, low_min) > max_tile || !room.add(g)) {
            held_t |= g.tmask;
            held_d |= g.dmask;
            rest.push_back(left[i]);
            continue;
          }
          c.tset |= g.tmask;
          c.gates.push_back(left[i]);
        }
      }
      rest.insert(rest.end(), left.begin() + i, left.end());
      left.swap(rest);
    }
  };
  // moving gates between passes pays where it saves passes: as many passes with
  // other gates in them only change places of work and widen tiles
  if (wide && moves_gates(dtype) && gates.size() > 1) {
    cut_merged(&merged);
    if (merged.size() < chunks.size()) chunks.swap(merged);
  }
  std::vector<PlannedPass> passes;
  cplx gamma = 1.0;  // global factor the wide programs leave (wide_steps)
  for (const Chunk& c : chunks) {
    const std::vector<int>& chunk = c.gates;
    const bool wide_chunk = c.wide;
    uint64_t tset = c.tset;
    // wide chunks with controlled X or swaps on states beyond the L2 take the
    // largest tile (CTAs of four warps): 7.35 against 7.97 ms for 8 random
    // layers of 26 qubits; in the L2, and without them, 2^10 is the faster
    const bool big = wide_chunk && tile_bits_hint <= 0 && (amp_bytes(dtype) << n) > (128ull << 20) &&
                     std::any_of(chunk.begin(), chunk.end(), [&](int x) {
                       return sgs[x].rg->kind == RK_MATRIX && !sgs[x].diag;
                     });
    // ---- tile: non-diagonal target slots + lowest slots up to the target size
    const int m = std::min(max_tile, std::max(big ? kWideMaxTileBits : m_target,
                                              low_union_size(tset, low_min)));
    for (int s = 0; s < n && __builtin_popcountll(tset) < m; ++s) tset |= 1ull << s;
    std::vector<int> tile;
    tile.reserve(m);
    for (int s = 0; s < n; ++s)
      if ((tset >> s) & 1ull) tile.push_back(s);
    const int R = std::min(rbits, m);
    std::vector<int> tbit_of_slot(n, -1);
    for (int i = 0; i < m; ++i) tbit_of_slot[tile[i]] = i;
    passes.clear();
    auto hand_over = [&]() -> int {
      for (auto& p : passes) {
        if (p.part) finish_layout(p.part.get(), dtype);
        if (p.nops() > 0) HS_TRY((*sink)(p));  // (a pass without ops has nothing to do)
      }
      return HS_OK;
    };
    if (wide_chunk && m >= kWideMinTileBits) {
      HS_TRY(plan_wide_chunk(n, dtype, q2s, sgs, chunk, tile, tbit_of_slot, &gamma, &passes));
      HS_TRY(hand_over());
      continue;
    }
    PartProgram* P = nullptr;
    auto new_program = [&]() {
      if (sink) {
        passes.emplace_back();
        passes.back().part.reset(new PartProgram);
        P = passes.back().part.get();
      } else {
        programs->emplace_back();
        P = &programs->back();
      }
      std::memset(P, 0, sizeof(*P));
      P->n = n;
      P->m = m;
      P->ntiles = 1ull << (n - m);
      P->rbits = R;
      build_runs(tile, &P->tile);
      for (int b = 0; b < m; ++b) P->tile_slot[b] = uint8_t(tile[b]);
      std::vector<int> outer;
      for (int s = 0; s < n; ++s)
        if (tbit_of_slot[s] < 0) outer.push_back(s);
      build_runs(outer, &P->outer);
    };
    new_program();
    // ---- groups
    std::vector<int> remaining = chunk;
    while (!remaining.empty()) {
      uint32_t rmask = 0;
      std::vector<int> regs, members, later;
      take_group(sgs, remaining, tbit_of_slot, R, &rmask, &members, &later);
      if (P->ngroups == kMaxGroups) new_program();  // a new pass (rare)
      GroupDesc& gd = P->groups[P->ngroups++];
      std::memset(&gd, 0, sizeof(gd));
      // fill the register set with the highest unused tile bits so that the
      // thread (lane) bits stay on the low, contiguous slots
      for (int b = m - 1; b >= 0 && __builtin_popcount(rmask) < R; --b) rmask |= 1u << b;
      for (int b = 0; b < m; ++b)
        if ((rmask >> b) & 1u) regs.push_back(b);
      for (int j = 0; j < R; ++j) gd.reg_tbit[j] = uint8_t(regs[j]);
      std::vector<int> thr;
      for (int b = 0; b < m; ++b)
        if (std::find(regs.begin(), regs.end(), b) == regs.end()) thr.push_back(b);
      build_runs(thr, &gd.thr);
      Layout L;
      L.tbit_of_slot = &tbit_of_slot;
      for (int b = 0; b < kMaxTileBits; ++b) L.regpos_of_tbit[b] = -1;
      for (int j = 0; j < R; ++j) L.regpos_of_tbit[regs[j]] = j;
      gd.first_op = uint16_t(P->nops);
      Emitter E{P, &q2s};
      for (int x : members) {
        const SlotGate& sg = sgs[x];
        if (sg.rg->kind == RK_ROT && sg.rg->rot.flip)
          return set_error(HS_E_UNSUPPORTED, "a flipped rotation outside a wide program");
        if (sg.rg->kind == RK_ROT)
          emit_rot(sg, L, E);
        else if (sg.rg->kind == RK_FLUSH)
          HS_TRY(emit_flush(sg, L, E));
        else
          emit_matrix(sg, L, E);
      }
      gd.num_ops = uint16_t(P->nops - gd.first_op);
      build_rounds(P, &gd);
      remaining = later;
    }
    if (sink) HS_TRY(hand_over());
  }
  if (gamma != cplx(1.0, 0.0) && !flush) {
    fr->G *= gamma;
  } else if (gamma != cplx(1.0, 0.0)) {
    // left by rotations planned after the flush (their qubits had nothing
    // pending): a flush of its own
    Frames g;
    g.reset(n);
    g.G = gamma;
    return plan_chunks(n, q2s, {}, &g, true, tile_bits_hint, dtype, false, lists, nullptr, sink);
  }
  if (!sink)
    for (auto& P : *programs) finish_layout(&P, dtype);
  return HS_OK;
}

}  // namespace

int plan_gates(int n, const std::vector<int>& q2s, const std::vector<LoweredGate>& gates,
               Frames* fr, bool flush, int tile_bits_hint, int dtype,
               std::vector<PartProgram>* programs) {
  programs->clear();
  PlanLists lists;
  return plan_chunks(n, q2s, {&gates}, fr, flush, tile_bits_hint, dtype, false, &lists, programs,
                     nullptr);
}

namespace {

// The parts of a call, window by window: a window's passes are on the device
// before the next window is rewritten, and what a chunk walks stays bounded, so
// planning is linear in the gates.  Where gates may move (`merge`) a window takes
// whole parts up to window_gates (one part at least); elsewhere it is one part.
// No gate moves across a window's border, which costs a pass or two there: on
// large states, where a pass takes longer than planning hundreds of gates, windows
// are larger (33 qubits, 1960 gates in parts of touched qubits: 54 passes in
// windows of 1024 gates, 51 in one).  Up to 22 qubits half a millisecond of
// planning is ahead of a call's first pass.
size_t window_gates(int n) { return size_t(1024) << std::clamp(n - 22, 0, 4); }

int plan_call(int n, const std::vector<int>& q2s, const Parts& parts, Frames* fr, bool flush,
              int tile_bits_hint, int dtype, bool merge, const PassSink& sink) {
  if (int(fr->r.size()) != n) fr->reset(n);
  const bool wide = use_wide(n, dtype);
  const bool flips = wide && (tile_bits_hint <= 0 || tile_bits_hint >= kWideMinTileBits) &&
                     all_wide(parts, *fr);
  const size_t most = wide && merge && moves_gates(dtype) ? window_gates(n) : 0;
  size_t i = 0;
  int first = 0;
  const PassSink tagged = [&](PlannedPass& p) {
    p.of_part = first;
    return sink(p);
  };
  PlanLists lists;
  Parts window;
  do {
    window.clear();
    first = int(i);
    for (size_t count = 0; i < parts.size(); ++i) {
      count += parts[i]->size();
      if (!window.empty() && count > most) break;
      window.push_back(parts[i]);
    }
    HS_TRY(plan_chunks(n, q2s, window, fr, flush && i == parts.size(), tile_bits_hint, dtype, flips,
                       &lists, nullptr, &tagged));
  } while (i < parts.size());
  return HS_OK;
}

}  // namespace

int plan_parts(int n, const std::vector<int>& q2s,
               const std::vector<std::vector<LoweredGate>>& parts, Frames* fr, bool flush,
               int tile_bits_hint, int dtype, bool merge, const PassSink& sink) {
  Parts all;
  all.reserve(parts.size());
  for (const auto& p : parts) all.push_back(&p);
  return plan_call(n, q2s, all, fr, flush, tile_bits_hint, dtype, merge, sink);
}

int plan_passes(int n, const std::vector<int>& q2s, const std::vector<LoweredGate>& gates,
                Frames* fr, bool flush, int tile_bits_hint, int dtype,
                std::vector<PlannedPass>* passes) {
  passes->clear();
  const PassSink sink = [&](PlannedPass& p) {
    passes->push_back(std::move(p));
    return HS_OK;
  };
  return plan_call(n, q2s, {&gates}, fr, flush, tile_bits_hint, dtype, false, sink);
}

int plan_part(int n, const std::vector<int>& q2s, const std::vector<LoweredGate>& gates,
              int tile_bits_hint, int dtype, std::vector<PartProgram>* programs) {
  Frames fr;
  fr.reset(n);
  return plan_gates(n, q2s, gates, &fr, true, tile_bits_hint, dtype, programs);
}

}  // namespace hisv
