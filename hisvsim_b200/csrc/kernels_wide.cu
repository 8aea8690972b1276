// K1, wide form: the part kernel with 32 amplitudes per thread, for programs of
// rotations, diagonal gates, controlled X and swaps (WideProgram, internal.h;
// planned by plan_wide_chunk).  The same pass as kernels_part.cu -- a CTA holds
// one 2^m tile at a time, copied in by cp.async while the previous tile's last
// register group runs, exchanged through shared memory between groups, stored
// straight from the last group's registers -- for the same entry points.
#include <atomic>
#include <type_traits>

#include "bounds.cuh"
#include "internal.h"

namespace hisv {
namespace {

constexpr int E = 1 << kWideBits;                              // amplitudes per thread
constexpr int kThreads = 1 << (kWideMaxTileBits - kWideBits);  // most threads of a CTA

// Resident CTAs of 128 threads per SM (their register budget).  32 amplitudes
// take 128 (complex128) or 64 (complex64) registers: three CTAs hold the
// kernel to 168, five to 96.  Half as many amplitudes per thread with five
// CTAs of 96 registers exchange the tile more often and decode twice as many
// steps per amplitude: 111 against 95 ms for the 30-qubit U3 + CZ circuit of
// 8 layers (complex128), 100 against 71 ms in complex64.
template <typename V>
struct WideTraits;
template <>
struct WideTraits<double2> {
  using T = double;
  static constexpr int blocks = 3;
};
template <>
struct WideTraits<float2> {
  using T = float;
  static constexpr int blocks = 5;
};

template <int J>
__device__ __forceinline__ constexpr int ins0(int p) {  // insert a 0 bit at J
  return ((p >> J) << (J + 1)) | (p & ((1 << J) - 1));
}

__device__ __forceinline__ double flip(double x, uint32_t sm) {
  return __hiloint2double(__double2hiint(x) ^ int(sm), __double2loint(x));
}
__device__ __forceinline__ float flip(float x, uint32_t sm) {
  return __int_as_float(__float_as_int(x) ^ int(sm));
}

// coefficient i in the amplitudes' precision.  It is read from the parameter
// space with a warp-uniform index; from a copy in shared memory the factor
// tables took as much of the load pipe as the tile exchange (7% slower at 30
// qubits), and the copy cost a resident CTA on 2^11 tiles.
template <typename V>
__device__ __forceinline__ V amp_coef(const WideProgram& P, int i) {
  return *reinterpret_cast<const V*>(&P.coef[i]);
}

// a += s * b on both components
__device__ __forceinline__ void shear(double2& a, double s, const double2& b) {
  a.x = fma(s, b.x, a.x);
  a.y = fma(s, b.y, a.y);
}
// one packed multiply-add for a complex64 amplitude
__device__ __forceinline__ void shear(float2& a, float s, const float2& b) {
  uint64_t r;
  asm("{.reg .b64 a, b, s;\n\t"
      "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b64 s, {%5, %5};\n\t"
      "fma.rn.f32x2 %0, s, b, a;}"
      : "=l"(r)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(s));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
}

// e^{i beta} on v: three in-place shears of its (re, im) plane, c = (tan(beta/2), sin(beta))
template <typename V>
__device__ __forceinline__ void turn(V& v, const V c) {
  v.x = fma(-c.x, v.y, v.x);
  v.y = fma(c.y, v.x, v.y);
  v.x = fma(-c.x, v.y, v.x);
}

// rotation on register bit J: its phase part first where `turned`, then the
// shears of `form` (RoundDesc), negated by a pending Z on the bit (zs: the sign
// bit or 0)
template <int J, typename V>
__device__ __forceinline__ void rotate(V (&v)[E], const WideProgram& P, int ci,
                                       uint32_t form, bool turned, uint32_t zs) {
  V cy = amp_coef<V>(P, ci);
  cy.x = flip(cy.x, zs);
  cy.y = flip(cy.y, zs);
#define A(p) v[ins0<J>(p)]
#define B(p) v[ins0<J>(p) | (1 << J)]
  if (turned) {
    const V cz = amp_coef<V>(P, ci + 1);
#pragma unroll
    for (int p = 0; p < E / 2; ++p) turn(B(p), cz);
  }
  if (!(form & 2u)) {
#pragma unroll
    for (int p = 0; p < E / 2; ++p) shear(A(p), cy.x, B(p));
  }
#pragma unroll
  for (int p = 0; p < E / 2; ++p) shear(B(p), cy.y, A(p));
  if (!(form & 1u)) {
#pragma unroll
    for (int p = 0; p < E / 2; ++p) shear(A(p), cy.x, B(p));
  }
#undef A
#undef B
}

// the pending signs z: element e is negated when e's register bits and the
// thread's own bit (5) meet an odd number of set bits
template <typename V>
__device__ __forceinline__ void apply_signs(V (&v)[E], uint32_t z) {
  uint32_t lo[4];  // sign of the two lowest bits and the thread
#pragma unroll
  for (int e = 0; e < 4; ++e)
    lo[e] = ((z << 26) ^ ((e & 1) ? z << 31 : 0u) ^ ((e & 2) ? z << 30 : 0u)) & 0x80000000u;
  uint32_t hi = 0;
#pragma unroll
  for (int i = 0; i < E / 4; ++i) {  // the upper bits in Gray-code order
    const int h = i ^ (i >> 1);
    if (i > 0) hi ^= (z << ((i & 1) ? 29 : (i & 2) ? 28 : 27)) & 0x80000000u;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      V& x = v[4 * h + e];
      x.x = flip(x.x, lo[e] ^ hi);
      x.y = flip(x.y, lo[e] ^ hi);
    }
  }
}

// a *= f, every result in its operand's register (as written in the usual way
// the product needs the old a.x to the end and two moves per component)
template <typename V>
__device__ __forceinline__ void cmul(V& a, const V f) {
  const typename WideTraits<V>::T t = f.y * a.x;
  a.x *= f.x;
  a.x = fma(-f.y, a.y, a.x);
  a.y = fma(f.x, a.y, t);
}

// factor f on the elements with register bit J set
template <int J, typename V>
__device__ __forceinline__ void factor_bit(V (&v)[E], const V f) {
#pragma unroll
  for (int p = 0; p < E / 2; ++p) cmul(v[ins0<J>(p) | (1 << J)], f);
}

// X on register bit J for the pairs whose bit in w (the element with the
// target 0) is set
template <int J, typename V>
__device__ __forceinline__ void exchange(V (&v)[E], uint32_t w) {
#pragma unroll
  for (int p = 0; p < E / 2; ++p) {
    const int e0 = ins0<J>(p), e1 = e0 | (1 << J);
    const bool f = (w >> e0) & 1u;
    const V a = v[e0], b = v[e1];
    v[e0].x = f ? b.x : a.x;
    v[e0].y = f ? b.y : a.y;
    v[e1].x = f ? a.x : b.x;
    v[e1].y = f ? a.y : b.y;
  }
}

// swap of register bits JA < JB.  `f` is always true; as a run-time value it
// keeps the exchange in place (select instructions): as plain moves the
// compiler renames registers in every case of the switch and spills
template <int JA, int JB, typename V>
__device__ __forceinline__ void swap_bits(V (&v)[E], bool f) {
#pragma unroll
  for (int p = 0; p < E / 4; ++p) {
    const int x = ins0<JB>(ins0<JA>(p)), e0 = x | (1 << JA), e1 = x | (1 << JB);
    const V a = v[e0], b = v[e1];
    v[e0].x = f ? b.x : a.x;
    v[e0].y = f ? b.y : a.y;
    v[e1].x = f ? a.x : b.x;
    v[e1].y = f ? a.y : b.y;
  }
}

// a phase run: the factors whose conditions hold, multiplied up in FP64 and
// applied to the elements its register mask selects
template <typename V>
__device__ __forceinline__ void phase_run(V (&v)[E], const WideOp& op, const WideProgram& P,
                                          uint32_t thr, uint64_t gbase) {
  using T = typename WideTraits<V>::T;
  double2 f = op.coef ? P.coef[op.coef] : make_double2(1.0, 0.0);
  for (int i = op.first, end = i + op.n; i < end; ++i) {
    const WideCond& q = P.conds[i];
    if ((thr & q.cthr) == q.cthr && (gbase & q.couter) == q.couter) {
      const double2 c = P.coef[q.coef];
      f = make_double2(fma(-c.y, f.y, c.x * f.x), fma(c.y, f.x, c.x * f.y));
    }
  }
  V g;
  g.x = T(f.x);
  g.y = T(f.y);
  switch (op.reg) {
    case 0:
#pragma unroll
      for (int e = 0; e < E; ++e) cmul(v[e], g);
      break;
    case 1: factor_bit<0>(v, g); break;
    case 2: factor_bit<1>(v, g); break;
    case 4: factor_bit<2>(v, g); break;
    case 8: factor_bit<3>(v, g); break;
    case 16: factor_bit<4>(v, g); break;
    default:
#pragma unroll
      for (int e = 3; e < E; ++e)
        if ((uint32_t(e) & op.reg) == op.reg) cmul(v[e], g);
  }
}

// CZ of register bits JA < JB: negates their elements
template <int JA, int JB, typename V>
__device__ __forceinline__ void negate(V (&v)[E]) {
#pragma unroll
  for (int p = 0; p < E / 4; ++p) {
    V& x = v[ins0<JB>(ins0<JA>(p)) | (1 << JA) | (1 << JB)];
    x.x = flip(x.x, 0x80000000u);
    x.y = flip(x.y, 0x80000000u);
  }
}

// F<JA, JB>(...) for the register pair of index I (wide_pair)
#define HS_WIDE_PAIRS(I, F, ...)                  \
  switch (I) {                                    \
    case 0: F<0, 1>(__VA_ARGS__); break;          \
    case 1: F<0, 2>(__VA_ARGS__); break;          \
    case 2: F<0, 3>(__VA_ARGS__); break;          \
    case 3: F<0, 4>(__VA_ARGS__); break;          \
    case 4: F<1, 2>(__VA_ARGS__); break;          \
    case 5: F<1, 3>(__VA_ARGS__); break;          \
    case 6: F<1, 4>(__VA_ARGS__); break;          \
    case 7: F<2, 3>(__VA_ARGS__); break;          \
    case 8: F<2, 4>(__VA_ARGS__); break;          \
    default: F<3, 4>(__VA_ARGS__); break;         \
  }

template <typename V>
__device__ __forceinline__ void permute(V (&v)[E], const WideOp& op, uint32_t thr,
                                        uint64_t gbase) {
  const bool ok = (thr & op.cthr) == op.cthr && (gbase & op.couter) == op.couter;
  if (op.code == wk_cx) {
    if (!__any_sync(0xffffffffu, ok)) return;  // (an outer control is the same for the warp)
    const uint32_t w = ok ? op.elems : 0u;
    switch (op.reg) {
      case 0: exchange<0>(v, w); break;
      case 1: exchange<1>(v, w); break;
      case 2: exchange<2>(v, w); break;
      case 3: exchange<3>(v, w); break;
      default: exchange<4>(v, w); break;
    }
    return;
  }
  HS_WIDE_PAIRS(op.reg, swap_bits, v, ok)
}

__device__ __forceinline__ void cp_async16(uint32_t saddr, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ uint64_t deposit(uint64_t x, const Runs& r) {
  uint64_t out = 0;
  for (int i = 0; i < r.n; ++i)
    out |= ((x >> r.src[i]) & ((1ull << r.len[i]) - 1ull)) << r.dst[i];
  return out;
}

// A tile: its number and its offset.
struct NextTile {
  uint64_t base;
  uint64_t tile;
};

// deposit by a whole warp, a run per lane (a loop over the runs costs 0.6 us, on
// the path of a tile of 10)
__device__ __forceinline__ uint64_t warp_deposit(uint32_t x, const Runs& r) {
  const int i = int(threadIdx.x & 31u);
  uint64_t v = 0;
  if (i < r.n) v = ((uint64_t(x) >> r.src[i]) & ((1ull << r.len[i]) - 1ull)) << r.dst[i];
  return uint64_t(__reduce_or_sync(0xffffffffu, uint32_t(v >> 32))) << 32 |
         __reduce_or_sync(0xffffffffu, uint32_t(v));
}

// Tiles are handed out in order, by a counter of the state's (P.ticket, 0 between
// launches: a launch counts to its number of tiles and wraps).  The tiles in
// flight are then always neighbours, and the sectors and DRAM pages that
// neighbouring tiles share are read and written once.  With every CTA on a fixed
// stride of tiles the CTAs drift apart and meet their neighbours' sectors after
// they left the L2: complex128, 33 qubits in frontier parts of 12, 7 layers, 1661
// ms against 815; 30 qubits in parts of 9, where whole lines are read, 145
// against 122.  Small launches, and states without a counter, keep the stride
// (ORDERED = false; launch below).
// OPS: the program has other ops than rotations, signs, tables and negations
template <bool OPS, bool ORDERED, typename V>
__global__ void __launch_bounds__(kThreads, WideTraits<V>::blocks)
    k1_wide(V* __restrict__ sv, const __grid_constant__ WideProgram P) {
  extern __shared__ __align__(128) unsigned char smem_raw[];  // the tile, then two NextTile
  const uint32_t t = threadIdx.x;
  const uint32_t tile_bytes = uint32_t(sizeof(V)) << P.m;
  const uint64_t size = 1ull << P.n;  // amplitudes of the state (bounds checks)
  const uint32_t sb = uint32_t(__cvta_generic_to_shared(smem_raw));
  auto issue = [&](uint64_t gbase) {
    uint64_t gt = 0;
    uint32_t ct = 0;
#pragma unroll
    for (int b = 0; b < kWideMaxThrBits; ++b)
      if ((t >> b) & 1u) {
        gt += P.gthr[b];
        ct ^= P.cthr[b];
      }
    const V* base = sv + gbase + gt;
#pragma unroll 4
    for (int k = 0; k < P.per_thr; ++k)
      if (HS_IN_BOUNDS(gbase + gt + P.gchunk[k] + 16 / sizeof(V) <= size &&
                           (ct ^ P.cslot[k]) + 16u <= tile_bytes,
                       kBoundsK1))
        cp_async16(sb + (ct ^ P.cslot[k]), base + P.gchunk[k]);
    cp_async_commit();
  };
  std::conditional_t<ORDERED, uint32_t, uint64_t> tile = blockIdx.x;
  uint64_t gbase = tile < P.ntiles ? deposit(tile, P.outer) : 0;
  // ORDERED: the tile after the present one, known a tile ahead: written by warp 0
  // into one entry while the other is read.  One number per tile: a launch draws
  // ntiles in all
  NextTile* N = reinterpret_cast<NextTile*>(smem_raw + (sizeof(V) << P.m));
  auto draw = [&](NextTile* to) {
    if (t >= 32u) return;
    uint32_t x = 0;
    if (t == 0) x = atomicInc(P.ticket, uint32_t(P.ntiles - 1));
    x = gridDim.x + __shfl_sync(0xffffffffu, x, 0);
    const uint64_t base = warp_deposit(x, P.outer);
    if (t == 0) {
      to->tile = x;
      to->base = base;
    }
  };
  // the stride: the next tile's offset by one addition in the scattered outer bits
  // (the carries run through the other bits, which are set)
  const uint64_t omask = ORDERED ? 0 : deposit(P.ntiles - 1, P.outer);
  const uint64_t ostep = ORDERED ? 0 : deposit(uint64_t(gridDim.x), P.outer);
  if (tile < P.ntiles) issue(gbase);
  if constexpr (ORDERED) draw(N);
  cp_async_wait();
  __syncthreads();
  V v[E];
  while (tile < P.ntiles) {
    const uint64_t next = tile + gridDim.x;
    const uint64_t gnext = !ORDERED && next < P.ntiles ? (((gbase | ~omask) + ostep) & omask) : 0;
    for (int g = 0; g < P.ngroups; ++g) {
      const WideGroup& G = P.groups[g];
      const bool last = g == P.ngroups - 1;
      // tile index bits of this thread (low half) and its shared offset (high half)
      uint32_t tw = 0;
#pragma unroll
      for (int b = 0; b < kWideMaxThrBits; ++b) tw ^= (0u - ((t >> b) & 1u)) & G.tw[b];
      const uint32_t thr = tw & 0xffffu, a0 = tw >> 16;
      auto ux = [&](int e) {
        uint32_t d = 0;
#pragma unroll
        for (int j = 0; j < kWideBits; ++j)
          if ((e >> j) & 1) d ^= G.dx[j];
        return d;
      };
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (HS_IN_BOUNDS((a0 ^ ux(e)) + sizeof(V) <= tile_bytes, kBoundsK1))
          v[e] = *reinterpret_cast<const V*>(smem_raw + (a0 ^ ux(e)));
      if (last) {
        // every thread holds its registers of the last group: the buffer takes
        // the next tile while this one is finished and stored
        __syncthreads();
        if constexpr (ORDERED) {
          if (N->tile < P.ntiles) issue(N->base);
        } else {
          if (next < P.ntiles) issue(gnext);
        }
      }
      uint32_t z = 0;  // pending signs (WideSign)
      for (int s = G.first_step, s_end = s + G.num_steps; s < s_end; ++s) {
        const uint64_t* sw = reinterpret_cast<const uint64_t*>(&P.steps[s]);
        const uint64_t w0 = sw[0], w1 = sw[1], w2 = sw[2];
        const int table = int(w1 >> 16) & 0xffff;
        for (int i = int(w1 >> 32) & 0xffff, end = i + (int(w2 >> 32) & 0xff); i < end; ++i) {
          const WideSign& q = P.signs[i];
          if ((thr & q.cthr) == q.cthr && (gbase & q.couter) == q.couter) z ^= q.bits;
        }
        if (table) {
          if (!HS_IN_BOUNDS(table + E <= P.ncoef, kBoundsK1)) continue;
#pragma unroll
          for (int e = 1; e < E; ++e) cmul(v[e], amp_coef<V>(P, table + e));
        }
        if (w2 & 0xff000000u) {
          apply_signs(v, z);
          z = 0;
        }
        int op = int(w1 >> 48);
        for (int end = op + (int(w2 >> 40) & 0xff); op < end; ++op) {
          const WideOp& o = P.ops[op];
          if (!OPS || o.code == wk_neg) {
            HS_WIDE_PAIRS(o.reg, negate, v)
          } else {
            phase_run(v, o, P, thr, gbase);
          }
        }
        const uint32_t forms = uint32_t(w2);
#define SLOT(J, W)                                                                      \
  if (const int ci = int(W) & 0xffff)                                                   \
    if (HS_IN_BOUNDS(ci < P.ncoef, kBoundsK1))                                          \
      rotate<J>(v, P, ci, forms >> (2 * J), (forms >> (16 + J)) & 1u,             \
                (z << (31 - J)) & 0x80000000u);
        SLOT(0, w0) SLOT(1, w0 >> 16) SLOT(2, w0 >> 32) SLOT(3, w0 >> 48) SLOT(4, w1)
#undef SLOT
        if constexpr (OPS)
          for (int end = op + (int(w2 >> 48) & 0xff); op < end; ++op)
            permute(v, P.ops[op], thr, gbase);
      }
      if (last) {
        // elements in Gray-code order: each address is the previous one plus
        // or minus one register bit's offset (one live pointer)
        V* p = sv + gbase + P.sbase;
#pragma unroll
        for (int b = 0; b < kWideMaxThrBits; ++b)
          if ((t >> b) & 1u) p += P.sthr[b];
#pragma unroll
        for (int i = 0; i < E; ++i) {
          const int e = i ^ (i >> 1);
          if (i > 0) {
            constexpr int kLow[5] = {1, 2, 4, 8, 16};
            const int j = (i & kLow[0]) ? 0 : (i & kLow[1]) ? 1 : (i & kLow[2]) ? 2 : (i & kLow[3]) ? 3 : 4;
            if ((e >> j) & 1) p += P.sreg[j]; else p -= P.sreg[j];
          }
          if (HS_IN_BOUNDS(uint64_t(p - sv) < size, kBoundsK1)) __stcs(p, v[e]);
        }
        if constexpr (ORDERED) {
          tile = uint32_t(N->tile);
          gbase = N->base;
          // the other entry, while the copies are awaited
          N = reinterpret_cast<NextTile*>(reinterpret_cast<uintptr_t>(N) ^ sizeof(NextTile));
          if (tile < P.ntiles) draw(N);
        }
        cp_async_wait();  // the next tile's copies (the only ones in flight)
      } else {
        const uint32_t a1 = a0 ^ G.tw[kWideFlipEntry];
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (HS_IN_BOUNDS((a1 ^ ux(e)) + sizeof(V) <= tile_bytes, kBoundsK1))
            *reinterpret_cast<V*>(smem_raw + (a1 ^ ux(e))) = v[e];
      }
      __syncthreads();
    }
    if constexpr (!ORDERED) {
      tile += gridDim.x;
      gbase = gnext;
    }
  }
}

// CTAs of the kernel that are resident at once, looked up once per device and tile
// size (the calls cost as much host time as the launch of a small pass)
template <bool OPS, bool ORDERED, typename V>
int resident_ctas(int m, size_t smem, int* most) {
  static std::atomic<int> resident[64][kWideMaxTileBits + 1];
  int dev = 0;
  HS_CUDA(cudaGetDevice(&dev));
  std::atomic<int>& cached = resident[dev & 63][m];
  *most = cached.load(std::memory_order_relaxed);
  if (*most >= 1) return HS_OK;
  constexpr auto kernel = k1_wide<OPS, ORDERED, V>;
  HS_TRY(smem_optin(reinterpret_cast<const void*>(kernel)));
  HS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(most, kernel, 1 << (m - kWideBits), smem));
  if (*most < 1) return set_error(HS_E_UNSUPPORTED, "K1 tile does not fit an SM (m=%d)", m);
  *most *= device_sms();
  cached.store(*most, std::memory_order_relaxed);
  return HS_OK;
}

template <bool OPS, typename V>
int launch(V* sv, const WideProgram& P, cudaStream_t s) {
  const int threads = 1 << (P.m - kWideBits);
  const size_t tile = sizeof(V) << P.m;
  int most = 0;
  HS_TRY((resident_ctas<OPS, false, V>(P.m, tile, &most)));
  // Few tiles per CTA keep the stride: it spreads the last ones evenly, while
  // numbers drawn a tile ahead go to whichever CTAs start first, several on one SM
  // (1.4 tiles per CTA, complex64 22 qubits: 233 us with the stride, 276 in order;
  // 2.3, complex128 22 qubits: 322, 328; 4.6, 23 qubits: 631, 609).
  if (P.ticket && P.ntiles >= 4 * uint64_t(most)) {
    const size_t smem = tile + 2 * sizeof(NextTile);
    HS_TRY((resident_ctas<OPS, true, V>(P.m, smem, &most)));
    k1_wide<OPS, true, V><<<most, threads, smem, s>>>(sv, P);
  } else {
    const int grid = P.ntiles < uint64_t(most) ? int(P.ntiles) : most;
    k1_wide<OPS, false, V><<<grid, threads, tile, s>>>(sv, P);
  }
  HS_CUDA(cudaGetLastError());
  return HS_OK;
}

template <typename V>
int launch_typed(V* sv, const WideProgram& P, cudaStream_t s) {
  bool ops = false;
  for (int i = 0; i < P.nwops; ++i) ops |= P.ops[i].code != wk_neg;
  return ops ? launch<true>(sv, P, s) : launch<false>(sv, P, s);
}

}  // namespace

#ifdef HS_BOUNDS
HS_BOUNDS_TAKE(bounds_take_wide)
#endif

int launch_wide(void* amp, int dtype, const WideProgram& P, cudaStream_t s) {
  if (dtype == HS_DTYPE_C128) return launch_typed(static_cast<double2*>(amp), P, s);
  return launch_typed(static_cast<float2*>(amp), P, s);
}

}  // namespace hisv
