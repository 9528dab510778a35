// Register-resident batched line FFT and the pass kernels built on it
// (k_lines: strided x / y passes; k_stage: the stage epilogue; k_p3, k_p3x: the
// z pass with the cross product; k_nz_max: the N-grid z pass).
//
// NLINES lines of length L are transformed by a Stockham auto-sort whose
// stages live in registers: the first stage reads its butterfly inputs
// straight from global memory (through the pass's load functor, which also
// applies zero-padding and derivative factors; inputs that are padding for
// every butterfly are compile-time zeros whose additions are skipped), every
// later stage reads them from a shared-memory exchange buffer written by the
// stage before, and the last stage hands its outputs straight to the pass's
// store functor (which applies truncation).  With the FP32 plans (two stages
// for every padded length up to 768) each element crosses shared memory once.
//
// Thread-to-butterfly maps: interleaved lines (x / y passes, MapInterleaved):
// thread g handles butterfly j = g / NLINES of line l = g % NLINES, so
// consecutive lanes take consecutive lines and global accesses are row
// segments of NLINES elements; contiguous lines (z passes, MapContig):
// consecutive lanes take consecutive butterflies of one line.
#pragma once

#include <type_traits>

#include "vk_fix.cuh"
#include "vk_kernels.cuh"
#include "vk_reduce.cuh"

// k_p3 (FP32) unpacks the forward's kept modes from the last stage's
// registers (1) or through shared memory after a barrier (0)
#ifndef VK_P3_ROW_UNPACK
#define VK_P3_ROW_UNPACK 1
#endif

namespace vk {

// At most two stages up to L = 768, with composite in-register radices; the
// larger radix goes first, where it carries no twiddles (and where padded
// inputs prune it).
__host__ __device__ constexpr int rplan_stages_f(int L) {
  return (L == 8 || L == 12 || L == 16 || L == 24) ? 1
       : (L == 32 || L == 48 || L == 64 || L == 96 || L == 128 || L == 192 || L == 256 || L == 384 || L == 512 || L == 768) ? 2
       : -1;
}
__host__ __device__ constexpr int rplan_radix_f(int L, int s) {
  return L <= 24 ? L
       : L == 32 ? (s == 0 ? 8 : 4)
       : L == 48 ? (s == 0 ? 16 : 3)
       : L == 64 ? (s == 0 ? 16 : 4)
       : L == 96 ? (s == 0 ? 16 : 6)
       : L == 128 ? (s == 0 ? 16 : 8)
       : L == 192 ? (s == 0 ? 16 : 12)
       : L == 256 ? 16
       : L == 384 ? (s == 0 ? 24 : 16)
       : L == 512 ? (s == 0 ? 32 : 16)
       : L == 768 ? (s == 0 ? 32 : 24)
       : 1;
}
// Contiguous lines (z passes) keep the radix-16 stage first where the
// larger radix would put the first-stage writes (stride RAD positions) on
// shared-memory banks that the one-slot-per-128-bytes padding cannot spread.
__host__ __device__ constexpr int rplan_radix_fc(int L, int s) {
  return L == 384 ? (s == 0 ? 16 : 24) : rplan_radix_f(L, s);
}
// FP64 lines run in fixed point with the plans of vk_fix.cuh.
template <typename R, bool CONTIG = false> __host__ __device__ constexpr int rstages(int L) {
  return sizeof(R) == 4 ? rplan_stages_f(L) : fx_supported(L) ? fx_stages(L) : -1;
}
template <typename R, bool CONTIG = false> __host__ __device__ constexpr int rradix(int L, int s) {
  return sizeof(R) == 4 ? (CONTIG ? rplan_radix_fc(L, s) : rplan_radix_f(L, s)) : fx_radix(L, s);
}
// threads of a CTA: one butterfly per thread in the widest stage (FP64 plans of
// two stages above 96 points: in the first stage, and a line of the second; of
// three stages: in all but the last)
template <typename R, int L, int NLINES, bool CONTIG = false, int S = 0>
__host__ __device__ constexpr int rthreads() {
  if constexpr (sizeof(R) == 8) {
    constexpr int nb0 = L / fx_radix(L, 0), nb1 = L / fx_radix(L, 1);
    return round32(L <= 96 || fx_stages(L) == 3 ? cmax(nb0, nb1) * NLINES : cmax(nb0 * NLINES, CONTIG ? nb1 : 0));
  } else if constexpr (S >= rstages<R, CONTIG>(L)) {
    return 32;
  } else {
    return cmax(round32(L / rradix<R, CONTIG>(L, S) * NLINES), rthreads<R, L, NLINES, CONTIG, S + 1>());
  }
}
// Per-stage twiddle tables (shared memory): stage S >= 1 of a plan reads
// W_L^(r k TWS) for r = 1..RAD-1, k = 0..NS-1 at (r-1) NS + k, so that lanes
// with consecutive k read consecutive entries (no bank conflicts) and lanes
// with the same k read the same entry.
template <typename R, bool CONTIG>
__host__ __device__ constexpr int stage_ns(int L, int S) {
  int ns = 1;
  for (int s = 0; s < S; ++s) ns *= rradix<R, CONTIG>(L, s);
  return ns;
}
template <typename R, bool CONTIG>
__host__ __device__ constexpr int twtab_off(int L, int S) {
  int off = 0;
  for (int s = 1; s < S; ++s) off += (rradix<R, CONTIG>(L, s) - 1) * stage_ns<R, CONTIG>(L, s);
  return off;
}
template <typename R, bool CONTIG>
__host__ __device__ constexpr int twtab_elems(int L) {
  return cmax(1, twtab_off<R, CONTIG>(L, rstages<R, CONTIG>(L)));
}

// FP32 with 8 lines: the first stage writes at stride RAD0 positions, so a
// padding slot after every RAD0 positions spreads a warp over both halves of
// the 32 banks.  FP64 rows of 8 lines are already 128 bytes.
template <typename R, int L, int NLINES>
__host__ __device__ constexpr bool rpad() { return sizeof(R) == 4 && NLINES < 16 && rstages<R>(L) > 1; }
template <typename R, int L, int NLINES>
__host__ __device__ constexpr int rsmem_elems() {
  return rstages<R>(L) > 1 ? (L + (rpad<R, L, NLINES>() ? L / rradix<R>(L, 0) : 0)) * NLINES : 0;
}
template <typename R, int L, int NLINES, int S>
__device__ __forceinline__ int ridx(int pos, int l) {
  if constexpr (S == 0 && rpad<R, L, NLINES>()) {
    return (pos + pos / rradix<R>(L, 0)) * NLINES + l;
  } else {
    return pos * NLINES + l;
  }
}

// Resident CTAs per SM of the fixed-point kernels, through the registers they
// may take: three-stage plans (radices up to 8: 32 registers of data) run best
// with 1152 threads of 56 registers per SM, two-stage plans (up to radix 16: 64
// of data) with 512 of 128 (N = 256 P2: 1.35 ms with two stages and 384
// threads, 1.39 with three and 768, 1.22 with three and 1152; N = 128 P2: 0.168
// ms with 384 threads, 0.150 with 512).
template <int L, int NT>
__host__ __device__ constexpr int fx_min_blocks() { return cmax(1, (fx_stages(L) == 3 ? 1152 : 512) / NT); }

// Minimum resident CTAs per SM requested from the compiler (caps registers):
// 24 warps per SM for the strided FP32 passes where the plan allows it; one or
// two CTAs for the 768-point plans and for the adjoint's multi-field kernel
// (EPI), whose shared memory limits residency anyway.  FP64: fx_min_blocks.
template <typename R, int L, int NT, bool EPI = false>
__host__ __device__ constexpr int lines_min_blocks() {
  if constexpr (sizeof(R) == 8) {
    return fx_min_blocks<L, NT>();
  } else {
    return L >= 768 ? (EPI ? 1 : 2) : EPI ? cmax(1, 512 / NT) : L >= 512 ? 2 : L >= 384 ? (NT >= 384 ? 2 : 3)
         : NT < 128 ? 4 : cmax(1, 768 / NT);
  }
}

// Thread-to-butterfly maps and exchange layouts.
// Interleaved lines (x / y passes, element p of line l at p * NLINES + l):
// consecutive lanes take consecutive lines, so every thread keeps one line.
template <typename R, int L, int NLINES>
struct MapInterleaved {
  static constexpr bool CONTIG = false;
  template <int NB> __device__ __forceinline__ static int line(int g) { return g % NLINES; }
  template <int NB> __device__ __forceinline__ static int bfly(int g) { return g / NLINES; }
  template <int S> __device__ __forceinline__ static int idx(int pos, int l) { return ridx<R, L, NLINES, S>(pos, l); }
  template <int STEP, int BASE> __device__ __forceinline__ static int step(int, int r) { return r * STEP * NLINES; }
  static constexpr int elems() { return rsmem_elems<R, L, NLINES>(); }
};
// Contiguous lines (z passes, element p of line l at l * LP + zi(p), one
// padding slot per 128 bytes): consecutive lanes take consecutive
// butterflies of a line, so global accesses along a line coalesce.
template <typename R, int L, int NLINES>
struct MapContig {
  static constexpr bool CONTIG = true;
  template <int NB> __device__ __forceinline__ static int line(int g) { return g / NB; }
  template <int NB> __device__ __forceinline__ static int bfly(int g) { return g % NB; }
  template <int S> __device__ __forceinline__ static int idx(int pos, int l) { return l * zpad_len<R>(L) + zi<R>(pos); }
  static constexpr int elems() { return NLINES * zpad_len<R>(L); }
  // offset of position pos + r STEP from that of pos (BASE divides pos): a
  // constant where whole padding rows are stepped over, or none is left
  template <int STEP, int BASE> __device__ __forceinline__ static int step(int pos, int r) {
    return STEP % zrow<R>() == 0 || (BASE % zrow<R>() == 0 && (r + 1) * STEP <= zrow<R>())
               ? zi<R>(r * STEP) : zi<R>(pos + r * STEP) - zi<R>(pos);
  }
};

// Inputs of the first stage at positions p in [Z0, Z1) are known to be zero
// (zero-padded modes): butterflies whose input r lies there for every j (all
// of [r NB, r NB + NB) inside the range) skip its first-layer additions.
__host__ __device__ constexpr unsigned zero_mask(int nb, int rad, int z0, int z1) {
  unsigned m = 0u;
  for (int r = 0; r < rad && r < 32; ++r)
    if (z0 < z1 && r * nb >= z0 && r * nb + nb <= z1) m |= 1u << r;
  return m;
}

// Store functors with a row<RAD, NS>(l, j, v) member take the last stage's
// whole butterfly (outputs at positions j + NS r, r < RAD) in one call, so
// that they can combine outputs across lanes (contiguous lines only).
template <class ST, class = void> struct StoreTakesRows : std::false_type {};
template <class ST> struct StoreTakesRows<ST, std::void_t<decltype(ST::kRowStore)>> : std::true_type {};

template <typename R, int L, bool INV, int NT, int NLINES, class MAP, int S, int NS, bool SL = false, bool TT = false,
          int Z0 = 0, int Z1 = 0>
struct RegStage {
  static constexpr int RAD = rradix<R, MAP::CONTIG>(L, S);
  static constexpr int NB = L / RAD;            // butterflies per line
  static constexpr int G = NB * NLINES;         // butterflies per stage
  static constexpr int Q = (G + NT - 1) / NT;
  static constexpr bool LAST = S + 1 == rstages<R, MAP::CONTIG>(L);
  static constexpr int TWS = L / (NS * RAD);    // twiddle table stride

  // ld(l, p) -> raw input of position p of line l (memory loads only),
  // pp(l, p, raw) -> the complex input (arithmetic on the loaded values),
  // st(l, p, v) takes output p.  All loads of the first stage are issued
  // before any arithmetic on them: in-order issue would otherwise wait on each
  // load before issuing the next.
  template <class LD, class PP, class ST>
  __device__ __forceinline__ static void run(C2<R>* xb, const C2<R>* __restrict__ tw, const LD& ld, const PP& pp,
                                             const ST& st) {
    const int tid = threadIdx.x;
    C2<R> v[Q][RAD];
    if constexpr (S == 0) {
      // raw inputs wider than one complex value are staged in chunks of
      // 192 bytes per thread (registers)
      using Raw = decltype(ld(0, 0));
      constexpr int CH = sizeof(Raw) > sizeof(C2<R>) ? cmin(RAD, (int)(192 / sizeof(Raw))) : RAD;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int g = tid + q * NT;
        if (G % NT == 0 || g < G) {
          const int l = MAP::template line<NB>(g);
          const int j = MAP::template bfly<NB>(g);
          __builtin_assume(j >= 0 && j < NB);
          __builtin_assume(l >= 0 && l < NLINES);
#pragma unroll
          for (int r0 = 0; r0 < RAD; r0 += CH) {
            Raw raw[CH];
#pragma unroll
            for (int r = 0; r < CH; ++r) {
              if (r0 + r < RAD) raw[r] = ld(l, j + (r0 + r) * NB);
            }
#pragma unroll
            for (int r = 0; r < CH; ++r) {
              if (r0 + r < RAD) v[q][r0 + r] = pp(l, j + (r0 + r) * NB, raw[r]);
            }
          }
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int g = tid + q * NT;
        if (G % NT == 0 || g < G) {
          const int l = MAP::template line<NB>(g);
          const int j = MAP::template bfly<NB>(g);
          __builtin_assume(j >= 0 && j < NB);
          __builtin_assume(l >= 0 && l < NLINES);
#pragma unroll
          for (int r = 0; r < RAD; ++r) v[q][r] = xb[MAP::template idx<S - 1>(j + r * NB, l)];
        }
      }
    }
    // a later stage writes the buffer it has just read: wait for all readers
    // (the last stage too when its outputs go back into the buffer, SL)
    if constexpr (S > 0 && (!LAST || SL)) __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int g = tid + q * NT;
      if (G % NT == 0 || g < G) {
        const int l = MAP::template line<NB>(g);
        const int j = MAP::template bfly<NB>(g);
        __builtin_assume(j >= 0 && j < NB);
        __builtin_assume(l >= 0 && l < NLINES);
        const int k = j % NS;
        C2<R> w[RAD];
        if constexpr (S > 0) {
#pragma unroll
          for (int r = 1; r < RAD; ++r) {
            if constexpr (TT) {
              w[r] = tw[twtab_off<R, MAP::CONTIG>(L, S) + (r - 1) * NS + k];
            } else {
              w[r] = tw[r * k * TWS];
            }
          }
        }
        dft<R, INV, RAD, (S > 0), S == 0 ? zero_mask(NB, RAD, Z0, Z1) : 0u>(v[q], w);
        const int base = (j - k) * RAD + k;
        if constexpr (LAST && StoreTakesRows<ST>::value) {
          // the whole butterfly (outputs j + NS r, j = base < NS) at once
          static_assert(MAP::CONTIG && G % 32 == 0 && NT % 32 == 0 && NB == NS && (NS == 16 || NS == 32),
                        "row stores: whole warps, butterfly j on lane j of an NS-lane group");
          st.template row<RAD, NS>(l, base, v[q]);
        } else if constexpr (LAST) {
#pragma unroll
          for (int r = 0; r < RAD; ++r) st(l, base + r * NS, v[q][r]);
        } else {
#pragma unroll
          for (int r = 0; r < RAD; ++r) xb[MAP::template idx<S>(base + r * NS, l)] = v[q][r];
        }
      }
    }
    if constexpr (!LAST) {
      __syncthreads();
      RegStage<R, L, INV, NT, NLINES, MAP, S + 1, NS * RAD, SL, TT, Z0, Z1>::run(xb, tw, ld, pp, st);
    }
  }
};

// FP64 lines in fixed point.
//
// Stage 0: one butterfly per thread.  Its bound of the inputs' magnitudes
// (fx_bound) is maximised over the line's threads, by shuffles where a line's
// butterflies share a warp (contiguous lines) and through shared memory
// otherwise, and gives the line's exponent.  The later stages loop over their
// butterflies in rounds of NT threads (whole lines per round where they write
// back into the exchange buffer), so that a CTA needs no more threads than stage
// 0 keeps busy.
//
// Contiguous lines carry two real lines, Z = X + i Y: one field at two neighbouring
// columns, which are of one size as a rule, as they share the exponent.

// The exponent of an output, v 2^q; FX_Q_NAN where an input is a NaN or an
// infinity: every output of the line is NaN.
constexpr int FX_Q_NAN = 1 << 24;
constexpr int FX_K_NAN = 0x7fff;   // the bound of such inputs
// bounds below FX_K_LOW may come from denormals, which 2^FX_UP makes normal
constexpr int FX_K_LOW = 80, FX_UP = 200;
__device__ __forceinline__ int fx_line_q(int k, int growth) {
  return k == FX_K_NAN ? FX_Q_NAN : fx_quantum(k) + growth;
}
// v 2^q, q20 = q << 20 (within the normal range)
__device__ __forceinline__ double fx_to_double(long long v, int q20) {
  const double d = __ll2double_rn(v);
  const int h = __double2hiint(d);
  return __hiloint2double(h != 0 ? h + q20 : 0, __double2loint(d));
}
// Exponents outside [-960, 900] are split: the first factor leaves every |v| >= 1
// normal, the second (the rest, or a NaN) rounds once.
__device__ __forceinline__ int fx_near_q(int q) { return min(max(q, -960), 900); }
__device__ __forceinline__ double fx_rest(int q) {
  const int rest = q - fx_near_q(q);
  return q >= FX_Q_NAN / 2 ? __longlong_as_double(0x7ff8000000000000ll)
                           : __hiloint2double((1023 + min(max(rest, -1000), 1000)) << 20, 0);
}
// Integers as doubles, put(r, u 2^q).  Two texts, so that the usual one converts and
// stores value by value (with the rest's factor as a branch before the stores: N = 256
// P2 1.21 ms against 1.18, P4 0.56 against 0.53).
template <int R, class PUT> __device__ __forceinline__ void fx_results(const fx2* u, int q, const PUT& put) {
  const int n = fx_near_q(q), h = n << 20;
  if (n == q) {
#pragma unroll
    for (int r = 0; r < R; ++r) put(r, make_double2(fx_to_double(u[r].x, h), fx_to_double(u[r].y, h)));
  } else {
    long long any = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) any |= u[r].x | u[r].y;
    const double f = any == 0 && q < FX_Q_NAN / 2 ? 1.0 : fx_rest(q);
    const bool scale = f != 1.0;   // (lines of zeros pass without the FP64 pipe)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      double2 d = make_double2(fx_to_double(u[r].x, h), fx_to_double(u[r].y, h));
      if (scale) d = make_double2(d.x * f, d.y * f);
      put(r, d);
    }
  }
}
__device__ __forceinline__ int fx_magnitude(double2 v) {
  return max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff);
}
__device__ __forceinline__ long long fx_integer(double v, int k) {
  return fx_from_double(__double2hiint(v), __double2loint(v), k);
}

// words that the maximum over a contiguous line's threads takes in shared memory
template <int L, int NLINES> __host__ __device__ constexpr int fx_contig_parts() {
  return 32 % (L / fx_radix(L, 0)) == 0 ? 1 : L / fx_radix(L, 0) * NLINES / 16;
}

// SL: the last stage writes back into the exchange.
template <int L, bool INV, int NT, int NLINES, class MAP, bool SL, int Z0, int Z1>
struct FxLines {
  static constexpr int ST = fx_stages(L);
  static constexpr int R0 = fx_radix(L, 0), NB0 = L / R0, G0 = NB0 * NLINES;
  // the last stage: radix, butterflies, and its twiddles' place in the table
  static constexpr int R1 = fx_radix(L, ST - 1), NB1 = L / R1, G1 = NB1 * NLINES;
  static constexpr int TW1 = twtab_off<double, MAP::CONTIG>(L, ST - 1);
  static constexpr int TG = fx_total_growth(L);
  static constexpr unsigned ZM = zero_mask(NB0, R0, Z0, Z1);
  static constexpr int NW0 = (G0 + 31) / 32;
  static_assert(G0 <= NT, "one first-stage butterfly per thread");
  static_assert(!MAP::CONTIG || 32 % NB0 == 0 || NB0 % 16 == 0, "groups of lanes keep one contiguous line");
  // words of the part array of line_max
  static constexpr int PARTS = MAP::CONTIG ? fx_contig_parts<L, NLINES>() : NW0 * NLINES;
  static_assert(MAP::CONTIG || (32 % NLINES == 0 && !SL), "interleaved lines tile a warp");

  // maximum over a line's threads
  __device__ __forceinline__ static int line_max(int m, int* part) {
    if constexpr (MAP::CONTIG && 32 % NB0 == 0) {
#pragma unroll
      for (int o = 1; o < NB0; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    } else if constexpr (MAP::CONTIG) {   // a line's threads are whole groups of 16 lanes
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      const int g = threadIdx.x;
      if (g < G0 && g % 16 == 0) part[g / 16] = m;
      __syncthreads();
      const int l = g < G0 ? g / NB0 : 0;
      m = part[l * (NB0 / 16)];
#pragma unroll
      for (int i = 1; i < NB0 / 16; ++i) m = max(m, part[l * (NB0 / 16) + i]);
    } else {
#pragma unroll
      for (int o = NLINES; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      const int w = threadIdx.x / 32, ln = threadIdx.x % 32;
      if (w < NW0 && ln < NLINES) part[w * NLINES + ln] = m;
      __syncthreads();
      m = part[ln % NLINES];
#pragma unroll
      for (int i = 1; i < NW0; ++i) m = max(m, part[i * NLINES + ln % NLINES]);
    }
    return m;
  }

  // Stage 0 from doubles.  fill(l, j, d): the inputs at positions j + r NB0 of line l
  // (those of ZM excepted).  Returns the exponent of the thread's line (interleaved:
  // the line of the thread in all stages; contiguous: also in line_q[l]).
  template <class FILL>
  __device__ __forceinline__ static int front(fx2* xb, const FILL& fill, int* part, int* line_q) {
    const int g = threadIdx.x;
    const int l0 = MAP::template line<NB0>(g), j0 = MAP::template bfly<NB0>(g);
    const bool act = G0 == NT || g < G0;
    double2 d[R0];
    int k = 0;
    if (act) {
      __builtin_assume(j0 >= 0 && j0 < NB0);
      __builtin_assume(l0 >= 0 && l0 < NLINES);
      fill(l0, j0, d);
      int top = 0;
#pragma unroll
      for (int r = 0; r < R0; ++r)
        if (!((ZM >> r) & 1u)) top = max(top, fx_magnitude(d[r]));
      float sum = 0.f;
#pragma unroll
      for (int r = 0; r < R0; ++r)
        if (!((ZM >> r) & 1u)) sum += fx_relative(fx_magnitude(d[r]), top);
      k = top == 0 ? 0 : top >= 0x7ff00000 ? FX_K_NAN : fx_bound(top, sum);
    }
    k = max(line_max(k, part), 1);
    int up = 0;
    if (k < FX_K_LOW) {   // 2^up makes denormals normal
      up = FX_UP;
      k += up;
      if (act) {
        int any = 0;
#pragma unroll
        for (int r = 0; r < R0; ++r)
          if (!((ZM >> r) & 1u)) any |= fx_magnitude(d[r]) | __double2loint(d[r].x) | __double2loint(d[r].y);
        if (any != 0) {
          const double f = __hiloint2double((1023 + FX_UP) << 20, 0);
#pragma unroll
          for (int r = 0; r < R0; ++r)
            if (!((ZM >> r) & 1u)) d[r] = make_double2(d[r].x * f, d[r].y * f);
        }
      }
    }
    const int q = fx_line_q(k, TG) - up;
    if (act) {
      fx2 v[R0];
#pragma unroll
      for (int r = 0; r < R0; ++r)
        v[r] = (ZM >> r) & 1u ? fx2{0, 0} : fx2{fx_integer(d[r].x, k), fx_integer(d[r].y, k)};
      if (MAP::CONTIG && j0 == 0) line_q[l0] = q;
      first_dft(v, xb, l0, j0);
    }
    return q;
  }

  // a first-stage butterfly into the exchange
  __device__ __forceinline__ static void first_dft(fx2* v, fx2* xb, int l, int j) {
    FxDft<R0, INV>::run(v);
    v[0] = fx_multiple<FX_GROWTH>(v[0]);
    fx2* dst = xb + MAP::template idx<0>(j * R0, l);
#pragma unroll
    for (int r = 0; r < R0; ++r) dst[MAP::template step<1, R0>(j * R0, r)] = v[r];
  }
  // twiddles and DFT of a later stage's butterfly: twiddle index k of ns
  template <int RAD, int OFF>
  __device__ __forceinline__ static void later_dft(fx2* u, const fxtw* __restrict__ tw, int k, int ns) {
    u[0] = fx_shift<FX_GROWTH>(u[0]);
#pragma unroll
    for (int r = 1; r < RAD; ++r) u[r] = fx_twiddle<INV>(u[r], tw[OFF + (r - 1) * ns + k]);
    FxDft<RAD, INV>::run(u);
  }
  // The middle stage of a three-stage plan on nl lines, in place (begins with the
  // exchange complete and ends so).
  __device__ __forceinline__ static void middle(fx2* xb, const fxtw* __restrict__ tw, int nl) {
    constexpr int RM = fx_radix(L, 1), NBM = L / RM, GM = NBM * NLINES;
    static_assert(GM <= NT, "one butterfly per thread");
    const int l = MAP::template line<NBM>(threadIdx.x), j = MAP::template bfly<NBM>(threadIdx.x);
    const bool act = MAP::CONTIG ? l < nl : GM == NT || (int)threadIdx.x < GM;
    fx2 u[RM];
    if (act) {
      __builtin_assume(j >= 0 && j < NBM);
      __builtin_assume(l >= 0 && l < NLINES);
      const fx2* src = xb + MAP::template idx<0>(j, l);
#pragma unroll
      for (int r = 0; r < RM; ++r) u[r] = src[MAP::template step<NBM, 1>(j, r)];
    }
    __syncthreads();
    if (act) {
      const int k = j % R0;
      later_dft<RM, 0>(u, tw, k, R0);
      u[0] = fx_multiple<FX_GROWTH>(u[0]);
      const int p0 = (j - k) * RM + k;
      fx2* dst = xb + MAP::template idx<0>(p0, l);
#pragma unroll
      for (int r = 0; r < RM; ++r) dst[MAP::template step<R0, 1>(p0, r)] = u[r];
    }
    __syncthreads();
  }
  // The last stage of nl lines, in rounds (whole lines, or butterflies of all
  // lines); the exchange is complete.  em(u, l, j) takes a butterfly's outputs
  // (positions j + r NB1), all threads of whose line have read theirs (SL).
  template <class EM>
  __device__ __forceinline__ static void back(const fx2* xb, const fxtw* __restrict__ tw, int nl, const EM& em) {
    constexpr int RL = MAP::CONTIG ? cmin(NT / NB1, NLINES) : NLINES;   // lines of a round
    constexpr int PER = MAP::CONTIG ? RL * NB1 : NT;                    // butterflies of a round
    static_assert(RL >= 1, "a round holds a line");
    const int total = MAP::CONTIG ? nl * NB1 : G1;
#pragma unroll 1
    for (int g0 = 0; g0 < total; g0 += PER) {
      const int g = g0 + (int)threadIdx.x;
      const int l = MAP::template line<NB1>(g), j = MAP::template bfly<NB1>(g);
      const bool act = (PER == NT || (int)threadIdx.x < PER) && g < total;
      fx2 u[R1];
      if (act) {
        __builtin_assume(j >= 0 && j < NB1);
        __builtin_assume(l >= 0 && l < NLINES);
        const fx2* src = xb + MAP::template idx<0>(j, l);
#pragma unroll
        for (int r = 0; r < R1; ++r) u[r] = src[MAP::template step<NB1, 1>(j, r)];
      }
      if constexpr (SL) __syncthreads();
      if (act) {
        later_dft<R1, TW1>(u, tw, j, NB1);
        em(u, l, j);
      }
    }
  }

  // From doubles to doubles, times 2^xe: st(l, p, v).
  template <class FILL, class STF>
  __device__ __forceinline__ static void run(fx2* xb, const fxtw* __restrict__ tw, const FILL& fill, const STF& st,
                                             int xe) {
    __shared__ int part[PARTS];
    __shared__ int line_q[MAP::CONTIG ? NLINES : 1];
    const int q0 = front(xb, fill, part, line_q);
    __syncthreads();
    if constexpr (ST == 3) middle(xb, tw, NLINES);
    back(xb, tw, NLINES, [&](const fx2* u, int l, int j) {
      fx_results<R1>(u, (MAP::CONTIG ? line_q[l] : q0) + xe, [&](int r, double2 v) { st(l, j + r * NB1, v); });
    });
  }
  // From doubles to integers in the exchange, with the exponents line_q (contiguous
  // lines): see fx_unpack.
  template <class FILL>
  __device__ __forceinline__ static void run_integers(fx2* xb, const fxtw* __restrict__ tw, const FILL& fill, int* part,
                                                      int* line_q) {
    static_assert(MAP::CONTIG && SL, "in place");
    front(xb, fill, part, line_q);
    __syncthreads();
    if constexpr (ST == 3) middle(xb, tw, NLINES);
    back(xb, tw, NLINES, [&](const fx2* u, int l, int j) {
      fx2* dst = xb + MAP::template idx<0>(j, l);
#pragma unroll
      for (int r = 0; r < R1; ++r) dst[MAP::template step<NB1, 1>(j, r)] = u[r];
    });
    __syncthreads();
  }
};

// Mode k of X and Y from a line of Z: z and its mirror image w, exponent q
// (X = (z + conj w) / 2, Y = (z - conj w) / 2i).
__device__ __forceinline__ void fx_unpack(fx2 z, fx2 w, int q, double2& X, double2& Y) {
  const int n = fx_near_q(--q), h = n << 20;
  X = make_double2(fx_to_double(z.x + w.x, h), fx_to_double(z.y - w.y, h));
  Y = make_double2(fx_to_double(z.y + w.y, h), fx_to_double(w.x - z.x, h));
  if (n != q) {
    const double f = fx_rest(q);
    X = make_double2(X.x * f, X.y * f);
    Y = make_double2(Y.x * f, Y.y * f);
  }
}

// fill functor of FxLines::front from ld / pp: all loads of a chunk are issued before
// any arithmetic on them (chunks of 256 bytes per thread where the raw inputs
// are wider than one complex value)
template <int L, int Z0, int Z1, class LD, class PP> struct FxFill {
  const LD& ld;
  const PP& pp;
  __device__ __forceinline__ void operator()(int l, int j, double2* d) const {
    constexpr int R0 = fx_radix(L, 0), NB0 = L / R0;
    constexpr unsigned ZM = zero_mask(NB0, R0, Z0, Z1);
    using Raw = decltype(ld(0, 0));
    constexpr int CH = sizeof(Raw) > sizeof(double2) ? cmin(R0, (int)(256 / sizeof(Raw))) : R0;
#pragma unroll
    for (int r0 = 0; r0 < R0; r0 += CH) {
      Raw raw[CH];
#pragma unroll
      for (int r = 0; r < CH; ++r)
        if (r0 + r < R0 && !((ZM >> (r0 + r)) & 1u)) raw[r] = ld(l, j + (r0 + r) * NB0);
#pragma unroll
      for (int r = 0; r < CH; ++r)
        if (r0 + r < R0 && !((ZM >> (r0 + r)) & 1u)) d[r0 + r] = pp(l, j + (r0 + r) * NB0, raw[r]);
    }
  }
};

// Transform NLINES lines (FP32).  All NT threads must call it; the exchange buffer
// xb (MAP::elems() elements) must not be in use by any thread.  Returns with
// no synchronisation after the last stage.
// SL: the store functor writes into xb itself (in place), so the last stage
// also waits for all readers before storing.  tw is the per-stage table of
// load_twtab (shared memory).
template <typename R, int L, bool INV, int NT, int NLINES, class MAP = MapInterleaved<R, L, NLINES>, bool SL = false,
          bool TT = false, int Z0 = 0, int Z1 = 0, class LD, class PP, class ST>
__device__ __forceinline__ void fft_lines(C2<R>* xb, const C2<R>* __restrict__ tw, const LD& ld, const PP& pp,
                                          const ST& st) {
  static_assert(rstages<R>(L) > 0 && sizeof(R) == 4, "unsupported FFT length, or not FP32");
  RegStage<R, L, INV, NT, NLINES, MAP, 0, 1, SL, TT, Z0, Z1>::run(xb, tw, ld, pp, st);
}
// pp for inputs that need no arithmetic after the load
struct PrepNone {
  template <class T> __device__ __forceinline__ T operator()(int, int, const T& v) const { return v; }
};
// pp of a c2r over lines of L points: Z = X + i Y with the Hermitian extension
template <typename R, int L> struct ZPack {
  __device__ __forceinline__ C2<R> operator()(int, int p, const C2x2<R>& r) const {
    const C2<R> X = r.a, Y = r.b;
    if (p == 0 || 2 * p == L) return cmk<R>(X.x, Y.x);   // c2r drops these imaginary parts
    return 2 * p < L ? cmk<R>(X.x - Y.y, X.y + Y.x) : cmk<R>(X.x + Y.y, Y.x - X.y);
  }
};

// Per-stage twiddle tables in shared memory: the stages read them through the
// shared-memory pipe instead of the L1/texture path, which the global loads
// and stores of the passes keep busy, and without bank conflicts.  No barrier
// is needed before the FFT: the first stage reads no twiddles and ends with
// one.
template <typename R, int L, bool CONTIG, int NT>
__device__ __forceinline__ void load_twtab(C2<R>* tab, const C2<R>* __restrict__ tw) {
  constexpr int ST = rstages<R, CONTIG>(L);
  for (int S = 1; S < ST; ++S) {
    const int rad = rradix<R, CONTIG>(L, S), ns = stage_ns<R, CONTIG>(L, S);
    const int tws = L / (ns * rad), off = twtab_off<R, CONTIG>(L, S);
    for (int i = threadIdx.x; i < (rad - 1) * ns; i += NT) {
      const int r = i / ns + 1, k = i - (r - 1) * ns;
      if constexpr (sizeof(R) == 8) {   // in the units of the stage
        reinterpret_cast<fxtw*>(tab)[off + i] =
            fx_stage_twiddle(reinterpret_cast<const fxtw*>(tw)[r * k * tws], fx_growth(rad));
      } else {
        tab[off + i] = tw[r * k * tws];
      }
    }
  }
}

// Positions [lo, hi) of a pass's input lines that are zero-padding for every
// line (Op::ZERO_LO / ZERO_HI; none by default).
template <class Op, class = void> struct OpZeroRange { static constexpr int lo = 0, hi = 0; };
template <class Op> struct OpZeroRange<Op, std::void_t<decltype(Op::ZERO_LO)>> {
  static constexpr int lo = Op::ZERO_LO, hi = Op::ZERO_HI;
};

// Power of two that an op's FP64 outputs carry (Op::exp2<K>(); 0 by default)
template <class Op, int K, class = void> struct OpExp2 { static constexpr int value = 0; };
template <class Op, int K> struct OpExp2<Op, K, std::void_t<decltype(Op::template exp2<K>())>> {
  static constexpr int value = Op::template exp2<K>();
};

// Ops that supply prefetch_row(f, lam0, nl, t) (an L2 hint for row t of a
// later CTA's input tile)
template <class Op, class = void> struct OpHasPrefetch : std::false_type {};
template <class Op>
struct OpHasPrefetch<Op, std::void_t<decltype(std::declval<const Op&>().prefetch_row(0, 0, 0, 0))>> : std::true_type {};

// Generic strided pass: NLINES consecutive lines lam = outer * hz + z of one
// field per CTA (blockIdx.x = f + nfields * tile), so no z tile is partly
// empty.  Op supplies kind(f) in [0, NKIND) (fields of one kind share their
// load/prep code, which is specialised per kind), load<K>(f, outer, z, p)
// (memory loads only, zero for padded positions), prep<K>(f, outer, z, p,
// raw), out_index(p) (-1: dropped) and store(f, outer, z, i, v).  Lines past
// the end (lam >= nlines) load line 0 and store nothing.  pf: blocks ahead
// whose input rows are prefetched into L2 (0 = none).

template <typename R, int L, bool INV, int NLINES, int NT, class Op>
__global__ void __launch_bounds__(NT, lines_min_blocks<R, L, NT>())
k_lines(Op op, const C2<R>* __restrict__ tw, int nlines, int pf) {
  static_assert(NT % NLINES == 0, "a thread keeps one line in every stage");
  extern __shared__ __align__(16) unsigned char vk_smem[];
  __shared__ C2<R> tw_s[twtab_elems<R, false>(L)];
  load_twtab<R, L, false, NT>(tw_s, tw);
  grid_depend();
  // the input rows of the CTA pf blocks ahead (ops with prefetch_row, whole
  // tiles whose rows are whole 128-byte lines)
  if constexpr (OpHasPrefetch<Op>::value && NLINES * sizeof(C2<R>) == 128) {
    const int b = (int)blockIdx.x + pf;
    if (pf > 0 && b < (int)gridDim.x) {
      const int lam0 = (b / op.nfields) * NLINES;
      if (lam0 + NLINES <= nlines)
        for (int t = threadIdx.x; t < L; t += NT) op.prefetch_row(b % op.nfields, lam0, NLINES, t);
    }
  }
  C2<R>* xb = reinterpret_cast<C2<R>*>(vk_smem);
  const int f = blockIdx.x % op.nfields;
  const int tile = blockIdx.x / op.nfields;
  const int lam = tile * NLINES + (int)(threadIdx.x % NLINES);
  const bool ok = lam < nlines;
  const int outer = ok ? lam / op.h_() : 0;
  const int z = ok ? lam - outer * op.h_() : 0;
  const int kd = op.kind(f);
  auto st = [&](int, int p, C2<R> v) {
    const int i = op.out_index(p);
    if (ok && i >= 0) op.store(f, outer, z, i, v);
  };
  if constexpr (sizeof(R) == 8) {
    // one transform for all kinds, whose loads alone differ: the transform's
    // code is large, and CTAs of several kinds share an SM's instruction cache
    constexpr int Z0 = OpZeroRange<Op>::lo, Z1 = OpZeroRange<Op>::hi;
    auto fill = [&](int l, int j, double2* d) {
      sfor<Op::NKIND>([&](auto kc) {
        constexpr int K = decltype(kc)::value;
        if (kd != K) return;   // uniform over the CTA
        const auto ld = [&](int, int p) { return op.template load<K>(f, outer, z, p); };
        const auto pp = [&](int, int p, const auto& raw) { return op.template prep<K>(f, outer, z, p, raw); };
        FxFill<L, Z0, Z1, decltype(ld), decltype(pp)>{ld, pp}(l, j, d);
      });
    };
    int xe = 0;
    sfor<Op::NKIND>([&](auto kc) {
      constexpr int K = decltype(kc)::value;
      if (kd == K) xe = OpExp2<Op, K>::value;
    });
    FxLines<L, INV, NT, NLINES, MapInterleaved<R, L, NLINES>, false, Z0, Z1>::run(
        reinterpret_cast<fx2*>(xb), reinterpret_cast<const fxtw*>(tw_s), fill, st, xe);
  } else {
  sfor<Op::NKIND>([&](auto kc) {
    constexpr int K = decltype(kc)::value;
    if (kd != K) return;   // uniform over the CTA
    fft_lines<R, L, INV, NT, NLINES, MapInterleaved<R, L, NLINES>, false, true, OpZeroRange<Op>::lo,
              OpZeroRange<Op>::hi>(
        xb, tw_s, [&](int, int p) { return op.template load<K>(f, outer, z, p); },
        [&](int, int p, const auto& raw) { return op.template prep<K>(f, outer, z, p, raw); }, st);
  });
  }
}

// ---------------------------------------------------------------------------
// P5 is two kernels: k_lines<OpXFwdTrunc> (x-forward of the three cross-product
// fields, keep N of M modes) and k_stage, mode by mode: scale N^3/M^3
// (dealiased.rs:102-109), Leray projection (spectral_ops.rs:114-151) and the
// stage epilogue.  Fused, one CTA held the transform's and the epilogue's
// registers and the kept modes of three fields in shared memory and ran the two
// one after the other at 12 to 24 warps per SM.  Apart they cost one more write
// and read of the three fields (6 N^2 H elements) and are faster: FP64 (FP64
// pipe, about 38 operations per mode) N = 256 1.09 -> 0.98 ms, N = 128 0.164 ->
// 0.140, N = 64 0.037 -> 0.031; FP32 (memory) N = 512 3.04 -> 2.37, N = 256
// 0.294 -> 0.261, N = 128 0.043 -> 0.041.
// ---------------------------------------------------------------------------
template <typename R> struct P5Args {
  R s_out, ks;
  const C2<R>* in; size_t fsin;   // (N, N, H), kept modes
  StageArgs<R> st;
};

// The CTA's row of the fused diagnostics: Tier-1 sums by a fixed shuffle /
// warp-order tree, then the shell histogram.
template <int NT, typename R>
__device__ __forceinline__ void diag_row(const StageArgs<R>& st, bool d_t1, bool d_sp, const double* dsum,
                                         const double* hist) {
  __shared__ double wsum[4][NT / 32];
  const bool has_row = (int)blockIdx.x < st.dpart_rows;
  double* row = st.dpart + (size_t)(has_row ? blockIdx.x : 0) * (4 + st.nsh);
  if (d_t1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double v = dsum[j];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) == 0) wsum[j][threadIdx.x / 32] = v;
    }
  }
  __syncthreads();
  if (d_t1 && has_row && threadIdx.x < 4) {
    double v = 0.0;
    for (int w = 0; w < NT / 32; ++w) v += wsum[threadIdx.x][w];
    row[threadIdx.x] = v;
  }
  if (d_sp && has_row)
    for (int i = threadIdx.x; i < st.nsh; i += NT) row[4 + i] = hist[i];
}

// Work and threads per CTA of k_stage (p5_ctas CTAs, which also sizes the
// diagnostics' rows).  FP64: one mode per thread and iteration, in array order
// (two need registers that it has not: N = 256 0.978 -> 1.006 ms).  FP32: the
// two modes (kx, ky, kz) and (-kx, ky, kz), whose loads are in flight together
// and which share |k|^2 and the coefficients: a gather from the table touches
// 32 cache lines per warp.
template <typename R, int N> struct StageGrid {
  static constexpr int PER = P5_LINES * N;
  static constexpr int NT = cmin(256, cmax(32, PER));
  static constexpr int MB = cmin(16, 768 / NT);   // 84 registers
  static constexpr int TOTAL = (sizeof(R) == 4 ? N / 2 + 1 : N) * N * (N / 2 + 1);
};

// DIAG: the instance for final stages whose new state also feeds the fused
// diagnostics (a.st.diag bits): per thread FP64 sums of the Tier-1 terms and a
// per-CTA FP64 shell histogram in shared memory (nsh doubles), written as row
// blockIdx.x of a.st.dpart; the rows are added by the Neumaier column reduction,
// as the separate reduction passes do.
template <typename R, int N, bool DIAG>
__global__ void __launch_bounds__(StageGrid<R, N>::NT, DIAG ? 1 : StageGrid<R, N>::MB) k_stage(P5Args<R> a) {
  constexpr int H = N / 2 + 1, NT = StageGrid<R, N>::NT, PER = StageGrid<R, N>::PER;
  constexpr int TOTAL = StageGrid<R, N>::TOTAL;
  __shared__ R kxy[N], kz_s[H];   // wave numbers (their conversion is an FP64 operation in the FP64 form)
  extern __shared__ __align__(16) unsigned char vk_smem[];
  double* hist = reinterpret_cast<double*>(vk_smem);   // DIAG: nsh shells
  const bool d_t1 = DIAG && (a.st.diag & DIAG_TIER1);
  const bool d_sp = DIAG && (a.st.diag & DIAG_SPECTRUM);
  for (int i = threadIdx.x; i < N; i += NT) kxy[i] = a.ks * (R)signed_k(i, N);
  for (int i = threadIdx.x; i < H; i += NT) kz_s[i] = a.ks * (R)i;
  if (d_sp)
    for (int i = threadIdx.x; i < a.st.nsh; i += NT) hist[i] = 0.0;
  grid_depend();
  __syncthreads();
  double dsum[4] = {0.0, 0.0, 0.0, 0.0};
  const bool ks_one = a.st.ks == 1.0;
  const int end = min((int)(blockIdx.x + 1) * PER, TOTAL);
  // diagnostics of a new mode u at (kx, ky, z)
  const auto diag = [&](int kx, int ky, int z, const C2<R>* u) {
    const R w = (z == 0 || z == N / 2) ? R(1) : R(2);   // R2C weight, exact in R
    if (d_t1) {
      R e, en, he, sh;
      tier1_terms<R>(a.ks * (R)kx, a.ks * (R)ky, a.ks * (R)z, u, e, en, he, sh);
      dsum[0] += (double)(w * e); dsum[1] += (double)(w * en);
      dsum[2] += (double)(w * he); dsum[3] += (double)(w * sh);
    }
    if (d_sp) {
      const int shell = shell_of(kx, ky, z, a.st.ks, ks_one);
      if (shell < a.st.nsh) atomicAdd(&hist[shell], (double)(w * spectrum_term<R>(u)));
    }
  };
  const auto locate = [](unsigned i, int& ix, int& iy, int& z) {
    const unsigned row = i / (unsigned)H;
    z = (int)(i - row * H);
    iy = (int)(row % N);
    ix = (int)(row / N);
  };
  if constexpr (sizeof(R) == 8) {
    const StageF64 stage(a.st, a.s_out);
#pragma unroll 1
    for (int e = blockIdx.x * PER + threadIdx.x; e < end; e += NT) {
      int ix, iy, z;
      locate(e, ix, iy, z);
      const int kxi = signed_k(ix, N), kyi = signed_k(iy, N);
      StageF64::Mode md;
      md.idx = e;
      md.m = kxi * kxi + kyi * kyi + z * z;
      stage.load(md);
      double2 v[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) v[c] = a.in[(size_t)c * a.fsin + e];
      const double kx = kxy[ix], ky = kxy[iy], kz = kz_s[z];
      const double dr = fma(kz, v[2].x, fma(ky, v[1].x, kx * v[0].x)) * md.ik2;
      const double di = fma(kz, v[2].y, fma(ky, v[1].y, kx * v[0].y)) * md.ik2;
      const double2 nl[3] = {make_double2(fma(-kx, dr, v[0].x), fma(-kx, di, v[0].y)),
                             make_double2(fma(-ky, dr, v[1].x), fma(-ky, di, v[1].y)),
                             make_double2(fma(-kz, dr, v[2].x), fma(-kz, di, v[2].y))};
      double2 un[3];
      stage.apply(md, nl, un);
      if constexpr (DIAG) diag(kxi, kyi, z, un);
    }
  } else {
#pragma unroll 1
    for (int e = blockIdx.x * PER + threadIdx.x; e < end; e += NT) {
      int ix, iy, z;   // ix <= N / 2
      locate((unsigned)e, ix, iy, z);
      const bool ok[2] = {true, ix > 0 && ix < N / 2};
      const size_t idx[2] = {(size_t)e, ok[1] ? ((size_t)(N - ix) * N + iy) * H + z : (size_t)e};
      const int kxi = signed_k(ix, N), kyi = signed_k(iy, N);
      const R kx = kxy[ix], ky = kxy[iy], kz = kz_s[z];
      C2<R> nl[2][3];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
#pragma unroll
        for (int c = 0; c < 3; ++c) nl[q][c] = a.in[(size_t)c * a.fsin + idx[q]];
      }
      const R k2 = (kx * kx + ky * ky) + kz * kz;
      const R inv = k2 < R(1e-30) ? R(0) : R(1) / k2;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const R k = q == 0 ? kx : -kx;
#pragma unroll
        for (int c = 0; c < 3; ++c) nl[q][c] = cscale<R>(nl[q][c], a.s_out);
        const C2<R> kd = cmk<R>((k * nl[q][0].x + ky * nl[q][1].x) + kz * nl[q][2].x,
                                (k * nl[q][0].y + ky * nl[q][1].y) + kz * nl[q][2].y);
        nl[q][0] = cmk<R>(nl[q][0].x - k * kd.x * inv, nl[q][0].y - k * kd.y * inv);
        nl[q][1] = cmk<R>(nl[q][1].x - ky * kd.x * inv, nl[q][1].y - ky * kd.y * inv);
        nl[q][2] = cmk<R>(nl[q][2].x - kz * kd.x * inv, nl[q][2].y - kz * kd.y * inv);
      }
      const int m = kxi * kxi + kyi * kyi + z * z;
      if constexpr (!DIAG) {
        stage_apply_n<R, 2>(a.st, idx, m, k2, nl, ok);
      } else {
        C2<R> un[2][3];
        stage_apply_n<R, 2, true>(a.st, idx, m, k2, nl, ok, un);
        diag(kxi, kyi, z, un[0]);
        if (ok[1]) diag(-kxi, kyi, z, un[1]);
      }
    }
  }
  if constexpr (DIAG) diag_row<NT>(a.st, d_t1, d_sp, dsum, hist);
}

// ---------------------------------------------------------------------------
// P3 on the register engine (FP32; FP64: k_p3x below): per CTA CP column pairs.  Inverse lines (6 CP):
// l = t * 2CP + c, the packed pair t of column c ((u_x, u_y), (u_z, w_x),
// (w_y, w_z)); the first stage packs straight from global memory with the
// Hermitian extension (z-line helpers above), the last stage writes the
// physical values to buffer B.  The cross product then writes the forward
// lines (3 CP) to buffer A: l = t * CP + pr with (c_x^A + i c_y^A),
// (c_z^A + i c_z^B), (c_x^B + i c_y^B) for the columns A, B of pair pr.  The
// forward transform reads A, exchanges through B and writes its spectra back
// to A, from where the kept H modes are unpacked and stored.
// ---------------------------------------------------------------------------
template <typename R, int M, int CP>
__host__ __device__ constexpr int p3_threads() {
  return cmin(rthreads<R, M, 6 * CP, true>(), 384);
}
// One column pair per CTA (M >= 384): the inverse writes its physical values
// in place, the cross product overwrites three of the six lines position by
// position (each position of the pair is read and written by one thread),
// and the forward exchanges through the other three, so the CTA needs 6
// lines of shared memory instead of 12.
#ifndef VK_P3_INPLACE
#define VK_P3_INPLACE 1
#endif
template <int CP> __host__ __device__ constexpr bool p3_inplace() { return VK_P3_INPLACE && CP == 1; }
template <typename R, int M, int CP>
__host__ __device__ constexpr int p3_smem_lines() { return (p3_inplace<CP>() ? 6 : 12) * CP; }

// Hermitian unpack of a forward line from the last stage's registers:
// butterfly j (lane j of an NS-lane group) holds Z(k) at k = j + NS r, r <
// RAD; the unpack of mode k needs Z(L - k), which is output RAD - 1 - r of
// lane NS - j of the same group, or, for j = 0, output (RAD - r) mod RAD of
// this lane.  f(k, X, Y) receives the two real fields' modes k < H.  All
// lanes of the warp must call it.
template <typename R, int RAD, int NS, int H, class F>
__device__ __forceinline__ void unpack_rows(int j, const C2<R>* v, const F& f) {
  const int lane = threadIdx.x & 31;
  const int src = (lane & ~(NS - 1)) | ((NS - j) & (NS - 1));
#pragma unroll
  for (int r = 0; r * NS < H; ++r) {
    const C2<R> zs = cmk<R>(__shfl_sync(0xffffffffu, v[RAD - 1 - r].x, src),
                            __shfl_sync(0xffffffffu, v[RAD - 1 - r].y, src));
    const C2<R> z = v[r];
    const C2<R> w = j == 0 ? v[(RAD - r) % RAD] : zs;
    const int k = j + NS * r;
    if (k >= H) continue;
    f(k, cmk<R>(R(0.5) * (z.x + w.x), R(0.5) * (z.y - w.y)), cmk<R>(R(0.5) * (z.y + w.y), R(0.5) * (w.x - z.x)));
  }
}

// Row unpack of the forward z transform of k_p3 (forward line l = t CP + pr):
// the kept modes go straight to global memory, in the layout of k_p3's
// shared-memory unpack below.
template <typename R, int M, int CP>
struct P3RowUnpack {
  static constexpr bool kRowStore = true;
  C2<R>* out; size_t fsout; int ncols; int col0;
  template <int RAD, int NS>
  __device__ __forceinline__ void row(int l, int j, const C2<R>* v) const {
    constexpr int H = M / 3 + 1;
    const int t = l / CP, pr = l - t * CP;
    const int ca = col0 + 2 * pr, cb = ca + 1;
    unpack_rows<R, RAD, NS, H>(j, v, [&](int k, const C2<R>& X, const C2<R>& Y) {
      if (t == 0) {
        if (ca < ncols) {
          out[(size_t)ca * H + k] = X;
          out[fsout + (size_t)ca * H + k] = Y;
        }
      } else if (t == 1) {
        if (ca < ncols) out[2 * fsout + (size_t)ca * H + k] = X;
        if (cb < ncols) out[2 * fsout + (size_t)cb * H + k] = Y;
      } else {
        if (cb < ncols) {
          out[(size_t)cb * H + k] = X;
          out[fsout + (size_t)cb * H + k] = Y;
        }
      }
    });
  }
};
// Forward z transforms of NF lines unpack from registers where the last
// stage allows it: FP32 plans whose last stage has 16 or 32 butterflies per
// line over whole warps
template <typename R, int M, int NF, int NT>
__host__ __device__ constexpr bool z_row_unpack() {
  if (VK_P3_ROW_UNPACK == 0) return false;
  constexpr int S = rstages<R, true>(M);
  constexpr int RAD = rradix<R, true>(M, S - 1);
  constexpr int NB = M / RAD;
  return (NB == 16 || NB == 32) && (NB * NF) % 32 == 0 && NT % 32 == 0;
}

template <typename R, int M, int CP, int NT>
__global__ void __launch_bounds__(NT, M >= 768 ? (p3_inplace<CP>() ? 3 : 1) : cmax(1, 512 / NT))
k_p3(P3Args<R> a, const C2<R>* __restrict__ tw, int pf) {
  constexpr int N = 2 * M / 3;
  constexpr int H = N / 2 + 1;
  constexpr int LP = zpad_len<R>(M);
  constexpr int NI = 6 * CP, NF = 3 * CP;
  constexpr bool INPL = p3_inplace<CP>();
  extern __shared__ __align__(16) unsigned char vk_smem[];
  __shared__ C2<R> tw_s[twtab_elems<R, true>(M)];
  // L2 prefetch of the six input ranges of the CTA pf blocks ahead (2 CP columns
  // of H complex values per field, a multiple of 16 bytes at a 16-byte boundary)
  {
    const int b = (int)blockIdx.x + pf;
    if (pf > 0 && threadIdx.x < 6 && b < (int)gridDim.x && (b + 1) * 2 * CP <= a.ncols)
      prefetch_l2_bulk(a.in + (size_t)threadIdx.x * a.fsin + (size_t)b * (2 * CP * H), 2 * CP * H * sizeof(C2<R>));
  }
  load_twtab<R, M, true, NT>(tw_s, tw);
  grid_depend();
  C2<R>* A = reinterpret_cast<C2<R>*>(vk_smem);
  C2<R>* B = INPL ? A : A + NI * LP;
  C2<R>* XF = INPL ? A + NF * LP : B;   // exchange of the forward transform
  const int col0 = blockIdx.x * 2 * CP;
  // positions H .. M - H of the packed lines are the z zero-padding
  fft_lines<R, M, true, NT, NI, MapContig<R, M, NI>, INPL, true, H, M - H + 1>(
      A, tw_s,
      [&](int l, int p) -> C2x2<R> {
        const int t = l / (2 * CP);
        const int col = col0 + l % (2 * CP);
        const bool lo = p < H;
        C2x2<R> r{};
        if (col < a.ncols && (lo || p > M - H)) {
          const C2<R>* src = a.in + (size_t)col * H + (lo ? p : M - p);
          r.a = src[(size_t)(2 * t) * a.fsin];
          r.b = src[(size_t)(2 * t + 1) * a.fsin];
        }
        return r;
      },
      [&](int, int p, const C2x2<R>& r) -> C2<R> {   // Z = X + i Y with the Hermitian extension
        const C2<R> X = r.a, Y = r.b;
        if (p == 0) return cmk<R>(X.x, Y.x);
        return p < H ? cmk<R>(X.x - Y.y, X.y + Y.x) : cmk<R>(X.x + Y.y, Y.x - X.y);
      },
      [&](int l, int p, C2<R> v) { B[l * LP + zi<R>(p)] = v; });
  __syncthreads();
  for (int e = threadIdx.x; e < CP * M; e += NT) {
    const int pr = e / M, p = e % M;
    const int zp = zi<R>(p);
    R c[2][3];
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      const int col = 2 * pr + cc;
      const C2<R> z1 = B[col * LP + zp], z2 = B[(2 * CP + col) * LP + zp], z3 = B[(4 * CP + col) * LP + zp];
      const R ux = z1.x, uy = z1.y, uz = z2.x, wx = z2.y, wy = z3.x, wz = z3.y;
      c[cc][0] = uy * wz - uz * wy;
      c[cc][1] = uz * wx - ux * wz;
      c[cc][2] = ux * wy - uy * wx;
    }
    A[pr * LP + zp] = cmk<R>(c[0][0], c[0][1]);
    A[(CP + pr) * LP + zp] = cmk<R>(c[0][2], c[1][2]);
    A[(2 * CP + pr) * LP + zp] = cmk<R>(c[1][0], c[1][1]);
  }
  __syncthreads();
  if constexpr (z_row_unpack<R, M, NF, NT>()) {
    // the kept modes unpacked from the last stage's registers
    fft_lines<R, M, false, NT, NF, MapContig<R, M, NF>, false, true>(
        XF, tw_s, [&](int l, int p) { return A[l * LP + zi<R>(p)]; }, PrepNone{},
        P3RowUnpack<R, M, CP>{a.out, a.fsout, a.ncols, col0});
    return;
  }
  fft_lines<R, M, false, NT, NF, MapContig<R, M, NF>, false, true>(
      XF, tw_s, [&](int l, int p) { return A[l * LP + zi<R>(p)]; }, PrepNone{},
      [&](int l, int p, C2<R> v) { A[l * LP + zi<R>(p)] = v; });
  __syncthreads();
  for (int e = threadIdx.x; e < CP * 3 * H; e += NT) {
    const int k = e % H;
    const int t = (e / H) % 3;
    const int pr = e / (3 * H);
    C2<R> X, Y;
    zunpack<R>(A + (t * CP + pr) * LP, M, k, X, Y);
    const int ca = col0 + 2 * pr, cb = ca + 1;
    if (t == 0) {
      if (ca < a.ncols) {
        a.out[(size_t)ca * H + k] = X;
        a.out[a.fsout + (size_t)ca * H + k] = Y;
      }
    } else if (t == 1) {
      if (ca < a.ncols) a.out[2 * a.fsout + (size_t)ca * H + k] = X;
      if (cb < a.ncols) a.out[2 * a.fsout + (size_t)cb * H + k] = Y;
    } else {
      if (cb < a.ncols) {
        a.out[(size_t)cb * H + k] = X;
        a.out[a.fsout + (size_t)cb * H + k] = Y;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// P3 in the FP64 form, with the fields, their cross products and the spectra as
// integers from the first stage of the inverse to the unpacked modes (doubles in
// between would cost 12 conversions and FP64 operations per position on the pipe
// that is scarce).
//
// Inverse lines l = f CP + pr: field f (u, omega) of the two columns of pair pr,
// neighbours that are of one size as a rule.  The last inverse stage leaves the
// fields in place with each line's exponent and the OR of the high words'
// magnitudes, which gives the shift that brings the line to 62 bits; a product keeps
// the upper 60 of its 124 bits.  Every field and every component has its exponent, so
// that a small component keeps its bits beside a large one.  Forward lines i CP + pr:
// component i of the two columns; they exchange through the lines 3 CP further on.  The forward first stage shifts its line right by
// what its largest butterfly needs (rounded), at most 6 bits.
//
// The inverse runs as a forward transform of lines with real and imaginary
// parts exchanged, so that both directions are one text (p3x_second) and one
// twiddle table.
// ---------------------------------------------------------------------------
struct FxPair {
  int s[6];      // left shifts of the fields
  int d[3][2];   // per component: right shifts of the two products
  int e[3];      // exponents of the components (FX_Q_NAN: a NaN among the fields)
};
__device__ __forceinline__ long long fx_rshift(long long v, int d) {   // v 2^-d, rounded
  return d > 0 ? ((v >> min(d - 1, 62)) + 1) >> 1 : v;
}
// a b, upper 64 of 128 bits (below 2^62 each, split): one cross term is floored and
// one rounded up, so that the means cancel and a zero factor gives zero
__device__ __forceinline__ long long fx_mulhi(fxsplit a, fxsplit b) {
  return fx_wide(a.h, b.h) + (long long)(fx_madhi(a.h, b.l, 0) - fx_madhi(a.l, -b.h, 0));
}
// a b - c d, the same
__device__ __forceinline__ long long fx_det(fxsplit a, fxsplit b, fxsplit c, fxsplit d) {
  const int t = fx_madhi(a.h, b.l, fx_madhi(c.l, -d.h, 0)), u = fx_madhi(c.h, d.l, fx_madhi(a.l, -b.h, 0));
  return fx_wide(a.h, b.h) - fx_wide(c.h, d.h) + (long long)(t - u);
}
// u x omega of a column; d: right shifts of the products (none: aligned)
__device__ __forceinline__ void fx_cross(const fxsplit* f, bool aligned, const int (*d)[2], long long* c) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    if (aligned) {
      c[i] = fx_det(f[j], f[3 + k], f[k], f[3 + j]);
    } else {
      c[i] = fx_rshift(fx_mulhi(f[j], f[3 + k]), d[i][0]) - fx_rshift(fx_mulhi(f[k], f[3 + j]), d[i][1]);
    }
  }
}

template <int M, int CP> __host__ __device__ constexpr int p3x_threads() {
  return rthreads<double, M, 6 * CP, true>();
}

// Dynamic shared memory of k_p3x.
template <int M, int CP> struct P3X {
  static constexpr int LP = zpad_len<double>(M);
  static constexpr int NI = 6 * CP, NF = 3 * CP;
  static constexpr int TW = NI * LP;                                 // in units of fx2
  static constexpr int INTS = TW + twtab_elems<double, true>(M);
  static constexpr int BYTES = INTS * 16 + 2 * NI * 4 + CP * ((int)sizeof(FxPair) + 4) + fx_contig_parts<M, NI>() * 4;
  __device__ __forceinline__ static fx2* lines() {
    extern __shared__ __align__(16) unsigned char vk_smem[];
    return reinterpret_cast<fx2*>(vk_smem);
  }
  __device__ __forceinline__ static fxtw* twiddles() { return reinterpret_cast<fxtw*>(lines() + TW); }
  __device__ __forceinline__ static int* line_q() { return reinterpret_cast<int*>(lines() + INTS); }
  __device__ __forceinline__ static int* field_m() { return line_q() + NI; }
  __device__ __forceinline__ static int* apart() { return field_m() + NI; }   // a pair's products need shifts
  __device__ __forceinline__ static FxPair* pairs() { return reinterpret_cast<FxPair*>(apart() + CP); }
  __device__ __forceinline__ static int* part() { return reinterpret_cast<int*>(pairs() + CP); }   // FxLines::PARTS
};
// Stages after the first of nl lines, from xs to ds (element offsets), with the
// fields' magnitudes where they are wanted.
// Inlined twice: as one function it spills (N = 256 3.2 ms against 2.9), as a
// loop over the directions more so (3.7).
template <int M, int CP, int NT>
__device__ __forceinline__ void p3x_second(int xs, int ds, int nl, bool maxima) {
  using P = P3X<M, CP>;
  using Inv = FxLines<M, false, NT, P::NI, MapContig<double, M, P::NI>, true, 0, 0>;
  if constexpr (Inv::ST == 3) Inv::middle(P::lines() + xs, P::twiddles(), nl);
  Inv::back(P::lines() + xs, P::twiddles(), nl, [&](const fx2* u, int l, int j) {
    fx2* dst = P::lines() + ds + l * P::LP + zi<double>(j);
    int m = 0;
#pragma unroll
    for (int r = 0; r < Inv::R1; ++r) {
      const int hx = (int)(u[r].x >> 32), hy = (int)(u[r].y >> 32);
      m |= (hx ^ (hx >> 31)) | (hy ^ (hy >> 31));
      dst[MapContig<double, M, P::NI>::template step<Inv::NB1, 1>(j, r)] = u[r];
    }
    if (maxima) {
      if constexpr (Inv::NB1 % 32 == 0) m = __reduce_or_sync(0xffffffffu, m);   // a warp holds butterflies of one line
      if (Inv::NB1 % 32 != 0 || threadIdx.x % 32 == 0) atomicOr(P::field_m() + l, m);
    }
  });
}

// The shifts and exponents of a pair: component i (one thread each).
template <int M, int CP>
__device__ __forceinline__ void p3x_pair(int pr, int i) {
  using P = P3X<M, CP>;
  int s[6], e[6];
  bool nan = false;
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    const int l = f * CP + pr;
    const int q = P::line_q()[l];
    nan = nan || q >= FX_Q_NAN / 2;
    s[f] = __clz(P::field_m()[l]) - 2;
    e[f] = q - s[f];
  }
  // up to three of the 62 bits bring the components of u, and of omega, to one exponent
#pragma unroll
  for (int g = 0; g < 6; g += 3) {
    const int top = max(max(e[g], e[g + 1]), e[g + 2]);
#pragma unroll
    for (int f = g; f < g + 3; ++f) {
      const int low = top - e[f];
      if (low <= 3 && low <= s[f]) {
        s[f] -= low;
        e[f] = top;
      }
    }
  }
  const auto pick = [](const int* v, int f) { return f == 0 ? v[0] : f == 1 ? v[1] : v[2]; };
  const int j = i == 2 ? 0 : i + 1, k = i == 0 ? 2 : i - 1;
  const int a = pick(e, j) + pick(e + 3, k), b = pick(e, k) + pick(e + 3, j);
  FxPair& out = P::pairs()[pr];
  out.d[i][0] = max(b - a, 0);
  out.d[i][1] = max(a - b, 0);
  out.e[i] = nan ? FX_Q_NAN : max(a, b) + 64;
  if (a != b) P::apart()[pr] = 1;
  if (i == 0) {
#pragma unroll
    for (int f = 0; f < 6; ++f) out.s[f] = s[f];
  }
}

template <int M, int CP, int NT>
__global__ void __launch_bounds__(NT, fx_min_blocks<M, NT>())
k_p3x(P3Args<double> a, const fxtw* __restrict__ tw) {
  constexpr int N = 2 * M / 3;
  constexpr int H = N / 2 + 1;
  constexpr int LP = zpad_len<double>(M);
  constexpr int NI = 6 * CP, NF = 3 * CP;
  using Inv = FxLines<M, false, NT, NI, MapContig<double, M, NI>, true, H, M - H + 1>;
  using Fwd = FxLines<M, false, NT, NF, MapContig<double, M, NF>, true, 0, 0>;
  using P = P3X<M, CP>;
  static_assert(NT >= 3 * CP, "a thread per pair and component");
  fx2* A = P::lines();
  int* line_q = P::line_q();
  load_twtab<double, M, true, NT>(reinterpret_cast<double2*>(P::twiddles()), reinterpret_cast<const double2*>(tw));
  grid_depend();
  const int col0 = blockIdx.x * 2 * CP;
  const int tid = threadIdx.x;
  for (int i = tid; i < NI + CP; i += NT) P::field_m()[i] = 0;   // apart() too
  {
    // inverse: positions H .. M - H are the z zero-padding
    const auto ld = [&](int l, int p) -> C2x2<double> {
      const int f = l / CP, col = col0 + 2 * (l - f * CP);
      const bool lo = p < H;
      C2x2<double> r{};
      if (lo || p > M - H) {
        const double2* src = a.in + (size_t)f * a.fsin + (size_t)col * H + (lo ? p : M - p);
        if (col < a.ncols) r.a = src[0];
        if (col + 1 < a.ncols) r.b = src[H];
      }
      return r;
    };
    // Z = X + i Y with the Hermitian extension, parts exchanged
    const auto pp = [&](int, int p, const C2x2<double>& r) -> double2 {
      if (p == 0) return make_double2(r.b.x, r.a.x);
      return p < H ? make_double2(r.a.y + r.b.x, r.a.x - r.b.y) : make_double2(r.b.x - r.a.y, r.a.x + r.b.y);
    };
    Inv::front(A, FxFill<M, H, M - H + 1, decltype(ld), decltype(pp)>{ld, pp}, P::part(), line_q);
  }
  __syncthreads();
  p3x_second<M, CP, NT>(0, 0, NI, true);
  __syncthreads();
  if (tid < 3 * CP) p3x_pair<M, CP>(tid / 3, tid % 3);
  __syncthreads();
  for (int e = tid; e < CP * M; e += NT) {
    const int pr = e / M, p = e % M;
    const FxPair& f = P::pairs()[pr];
    const bool aligned = P::apart()[pr] == 0;
    fx2* x = A + pr * LP + zi<double>(p);
    fxsplit va[6], vb[6];   // the columns (parts exchanged)
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const fx2 z = x[i * CP * LP];
      va[i] = fx_split(z.y << f.s[i]);
      vb[i] = fx_split(z.x << f.s[i]);
    }
    long long ca[3], cb[3];
    fx_cross(va, aligned, f.d, ca);
    fx_cross(vb, aligned, f.d, cb);
#pragma unroll
    for (int i = 0; i < 3; ++i) x[i * CP * LP] = fx2{ca[i], cb[i]};
  }
  __syncthreads();
  {
    const int l = MapContig<double, M, NF>::template line<Fwd::NB0>(tid);
    const int j = MapContig<double, M, NF>::template bfly<Fwd::NB0>(tid);
    const bool act = tid < Fwd::G0;
    fx2 v[Fwd::R0];
    int sum = 0;
    if (act) {
      __builtin_assume(j >= 0 && j < Fwd::NB0);
      __builtin_assume(l >= 0 && l < NF);
#pragma unroll
      for (int r = 0; r < Fwd::R0; ++r) {
        v[r] = A[l * LP + zi<double>(j) + MapContig<double, M, NF>::template step<Fwd::NB0, 1>(j, r)];
        const int hx = (int)(v[r].x >> 32), hy = (int)(v[r].y >> 32);
        sum += max(hx ^ (hx >> 31), hy ^ (hy >> 31)) >> 5;
      }
      sum += Fwd::R0;                                // the shifted-out bits
      sum += (sum >> 2) + (sum >> 3) + (sum >> 4) + 3;   // times 1.4375 > sqrt(2), rounded up
    }
    // |z| sums below 2^(37 + bits); to 2^62
    const int sh = max(0, 37 + 32 - __clz(Fwd::line_max(sum, P::part())) - 62);
    if (act) {
      const long long half = (1ll << sh) >> 1;
#pragma unroll
      for (int r = 0; r < Fwd::R0; ++r) v[r] = fx2{(v[r].x + half) >> sh, (v[r].y + half) >> sh};
      Fwd::first_dft(v, A + NF * LP, l, j);
      if (j == 0) line_q[l] = P::pairs()[l % CP].e[l / CP] + sh + Fwd::TG;
    }
  }
  __syncthreads();
  p3x_second<M, CP, NT>(NF * LP, 0, NF, false);
  __syncthreads();
  for (int e = tid; e < NF * H; e += NT) {
    const int l = e / H, k = e - l * H;
    const int i = l / CP, col = col0 + 2 * (l - i * CP);
    const fx2* line = A + l * LP;
    double2 X, Y;
    fx_unpack(line[zi<double>(k)], line[zi<double>(k == 0 ? 0 : M - k)], line_q[l], X, Y);
    double2* dst = a.out + (size_t)i * a.fsout + (size_t)col * H + k;
    if (col < a.ncols) dst[0] = X;
    if (col + 1 < a.ncols) dst[H] = Y;
  }
}

// ---------------------------------------------------------------------------
// N-grid z pass on the register engine: c2r of u and/or omega (already x/y
// inverted and scaled by 1/N^3) packed in pairs, and max |u|^2, max |omega|^2
// over the N^3 grid (solver.rs:180-218 and :537-567).  Lines per column pair, FP32:
// BOTH: l = 6 pr + 3 cc + t, the pair t of column cc; otherwise l = 3 pr + cc
// (f0 + i f1 of column cc) and 3 pr + 2 (f2 of both columns).  FP64: field f of both
// columns, l = f CP + pr (k_p3x's lines).  The inverse writes its physical values in
// place; the maxima follow.
// ---------------------------------------------------------------------------
template <typename R, int N, int CP, bool BOTH>
__host__ __device__ constexpr int nz_threads() {
  return cmin(rthreads<R, N, (BOTH ? 6 : 3) * CP, true>(), 384);
}

template <typename R, int N, int CP, bool BOTH, int NT>
__global__ void __launch_bounds__(NT, sizeof(R) == 8 ? fx_min_blocks<N, NT>() : N >= 512 ? 1 : cmax(1, 512 / NT))
k_nz_max(NZArgs<R> a, const C2<R>* __restrict__ tw, int pf) {
  constexpr int H = N / 2 + 1;
  constexpr int LPP = BOTH ? 6 : 3;   // lines per column pair
  constexpr int NL = LPP * CP;
  constexpr int LP = zpad_len<R>(N);
  extern __shared__ __align__(16) unsigned char vk_smem[];
  C2<R>* lines = reinterpret_cast<C2<R>*>(vk_smem);
  __shared__ C2<R> tw_s[twtab_elems<R, true>(N)];
  __shared__ double red[2][32];
  __shared__ int redn;
  // L2 prefetch of the input ranges of the CTA pf blocks ahead (FP32: per
  // field 2 CP columns of H complex values, a multiple of 16 bytes at a
  // 16-byte boundary)
  if constexpr (sizeof(R) == 4) {
    const int b = (int)blockIdx.x + pf;
    if (pf > 0 && threadIdx.x < (BOTH ? 6 : 3) && b < (int)gridDim.x && (b + 1) * 2 * CP <= a.ncols)
      prefetch_l2_bulk(a.in + (size_t)threadIdx.x * a.fs + (size_t)b * (2 * CP * H), 2 * CP * H * sizeof(C2<R>));
  }
  load_twtab<R, N, true, NT>(tw_s, tw);
  grid_depend();
  if (threadIdx.x == 0) redn = 0;
  const int col0 = blockIdx.x * 2 * CP;
  if constexpr (sizeof(R) == 8) {
    const auto ld = [&](int l, int p) -> C2x2<R> {
      const int f = l / CP, c = col0 + 2 * (l - f * CP);
      const C2<R>* src = a.in + (size_t)f * a.fs + (size_t)c * H + (p < H ? p : N - p);
      C2x2<R> r{};
      if (c < a.ncols) r.a = src[0];
      if (c + 1 < a.ncols) r.b = src[H];
      return r;
    };
    FxLines<N, true, NT, NL, MapContig<R, N, NL>, true, 0, 0>::run(
        reinterpret_cast<fx2*>(lines), reinterpret_cast<const fxtw*>(tw_s),
        FxFill<N, 0, 0, decltype(ld), ZPack<R, N>>{ld, ZPack<R, N>{}},
        [&](int l, int p, C2<R> v) { lines[l * LP + zi<R>(p)] = v; }, 0);
  } else {
    fft_lines<R, N, true, NT, NL, MapContig<R, N, NL>, true, true>(
        lines, tw_s,
        [&](int l, int p) -> C2x2<R> {
          const int pr = l / LPP, j = l % LPP;
          int fx, fy, cx, cy;
          if (BOTH) {
            const int cc = j / 3, t = j % 3;
            fx = 2 * t; fy = 2 * t + 1;
            cx = cy = col0 + 2 * pr + cc;
          } else if (j < 2) {
            fx = 0; fy = 1;
            cx = cy = col0 + 2 * pr + j;
          } else {
            fx = fy = 2;
            cx = col0 + 2 * pr;
            cy = cx + 1;
          }
          const int k = p < H ? p : N - p;
          C2x2<R> r{};
          if (cx < a.ncols) r.a = a.in[(size_t)fx * a.fs + (size_t)cx * H + k];
          if (cy < a.ncols) r.b = a.in[(size_t)fy * a.fs + (size_t)cy * H + k];
          return r;
        },
        ZPack<R, N>{},
        [&](int l, int p, C2<R> v) { lines[l * LP + zi<R>(p)] = v; });
  }
  __syncthreads();
  // maxima in the working precision (the FP32-bulk form keeps FP64 only for
  // the dt arithmetic that consumes them)
  R m1 = R(0), m2 = R(0);
  int bad = 0;
  for (int e = threadIdx.x; e < CP * N; e += NT) {
    const int pr = e / N, p = e % N;
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
      if (col0 + 2 * pr + cc >= a.ncols) continue;
      if constexpr (BOTH) {
        R ux, uy, uz, wx, wy, wz;
        if constexpr (sizeof(R) == 8) {
          const auto at = [&](int f) {
            const C2<R> v = lines[(f * CP + pr) * LP + zi<R>(p)];
            return cc == 0 ? v.x : v.y;
          };
          ux = at(0); uy = at(1); uz = at(2); wx = at(3); wy = at(4); wz = at(5);
        } else {
          const C2<R>* L0 = lines + (6 * pr + 3 * cc) * LP;
          const C2<R> A = L0[zi<R>(p)], B = L0[LP + zi<R>(p)], C = L0[2 * LP + zi<R>(p)];
          ux = A.x; uy = A.y; uz = B.x; wx = B.y; wy = C.x; wz = C.y;
        }
        const R s1 = ux * ux + uy * uy + uz * uz;
        const R s2 = wx * wx + wy * wy + wz * wz;
        bad |= (s1 != s1) | (s2 != s2);
        m1 = fmax(m1, s1);
        m2 = fmax(m2, s2);
      } else {
        R fx, fy, fz;
        if constexpr (sizeof(R) == 8) {
          const C2<R> A = lines[pr * LP + zi<R>(p)], B = lines[(CP + pr) * LP + zi<R>(p)],
                      C = lines[(2 * CP + pr) * LP + zi<R>(p)];
          fx = cc == 0 ? A.x : A.y; fy = cc == 0 ? B.x : B.y; fz = cc == 0 ? C.x : C.y;
        } else {
          const C2<R> A = lines[(3 * pr + cc) * LP + zi<R>(p)];
          const C2<R> Z = lines[(3 * pr + 2) * LP + zi<R>(p)];
          fx = A.x; fy = A.y; fz = cc == 0 ? Z.x : Z.y;
        }
        const R s = fx * fx + fy * fy + fz * fz;
        bad |= (s != s);
        m1 = fmax(m1, s);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
  }
  const int w = threadIdx.x / 32, ln = threadIdx.x % 32;
  if (bad) atomicOr(&redn, 1);
  if (ln == 0) { red[0][w] = (double)m1; red[1][w] = (double)m2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r1 = 0.0, r2 = 0.0;
    for (int i = 0; i < NT / 32; ++i) { r1 = fmax(r1, red[0][i]); r2 = fmax(r2, red[1][i]); }
    if (BOTH) {
      atomic_max_pos(&a.out->umax2, r1);
      atomic_max_pos(&a.out->wmax2, r2);
    } else if (a.which == 2) {
      atomic_max_pos(&a.out->wmax2, r1);
    } else {
      atomic_max_pos(&a.out->umax2, r1);
    }
    if (redn) atomicOr(&a.out->nan_flag, 1);
  }
}

// ---------------------------------------------------------------------------
// Standalone backend z passes (FftBackend::r2c_3d / c2r_3d z stage,
// ndrustfft_backend.rs:33-57).  Real lines of length L, two columns per complex
// line, CP lines per CTA: r2c reads the pair into the first stage, leaves the
// spectrum in shared memory and unpacks it; c2r packs the half spectra (with
// the Hermitian extension) in the first stage's loads and stores the two real
// columns from the last stage's registers.
// ---------------------------------------------------------------------------
template <typename R> struct FZArgs {
  int ncols;                  // nx*ny
  R* real; C2<R>* cplx;       // (ncols, L) real, (ncols, L/2+1) complex
  R scale;                    // c2r: 1/(nx ny nz)
};
// lines per CTA: about 192 threads in the wider stage
template <typename R, int L> __host__ __device__ constexpr int fz_pairs() {
  int rad = rradix<R, true>(L, 0);
  for (int s = 1; s < rstages<R, true>(L); ++s) rad = cmin(rad, rradix<R, true>(L, s));
  return cmax(1, 192 * rad / L);
}
template <typename R, int L, int NT>
__host__ __device__ constexpr int fz_min_blocks() { return sizeof(R) == 8 ? fx_min_blocks<L, NT>() : cmax(1, 768 / NT); }

template <typename R, int L, int CP, int NT>
__global__ void __launch_bounds__(NT, fz_min_blocks<R, L, NT>()) k_fz_r2c(FZArgs<R> a, const C2<R>* __restrict__ tw) {
  constexpr int H = L / 2 + 1;
  constexpr int LP = zpad_len<R>(L);
  extern __shared__ __align__(16) unsigned char vk_smem[];
  __shared__ C2<R> tw_s[twtab_elems<R, true>(L)];
  load_twtab<R, L, true, NT>(tw_s, tw);
  grid_depend();
  C2<R>* lines = reinterpret_cast<C2<R>*>(vk_smem);
  const int col0 = blockIdx.x * 2 * CP;
  const auto ld = [&](int l, int p) -> C2<R> {
    const int c = col0 + 2 * l;
    const R* x = a.real + (size_t)c * L + p;
    return cmk<R>(c < a.ncols ? x[0] : R(0), c + 1 < a.ncols ? x[L] : R(0));
  };
  if constexpr (sizeof(R) == 8) {
    using Fwd = FxLines<L, false, NT, CP, MapContig<R, L, CP>, true, 0, 0>;
    __shared__ int part[Fwd::PARTS], line_q[CP];
    fx2* z = reinterpret_cast<fx2*>(lines);
    Fwd::run_integers(z, reinterpret_cast<const fxtw*>(tw_s),
                      FxFill<L, 0, 0, decltype(ld), PrepNone>{ld, PrepNone{}}, part, line_q);
    for (int e = threadIdx.x; e < CP * H; e += NT) {
      const int l = e / H, k = e - l * H;
      const int c = col0 + 2 * l;
      if (c >= a.ncols) break;
      C2<R> X, Y;
      fx_unpack(z[l * LP + zi<R>(k)], z[l * LP + zi<R>(k == 0 ? 0 : L - k)], line_q[l], X, Y);
      C2<R>* dst = a.cplx + (size_t)c * H + k;
      dst[0] = X;
      if (c + 1 < a.ncols) dst[H] = Y;
    }
    return;
  } else {
    fft_lines<R, L, false, NT, CP, MapContig<R, L, CP>, true, true>(
        lines, tw_s, ld, PrepNone{}, [&](int l, int p, C2<R> v) { lines[l * LP + zi<R>(p)] = v; });
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * CP * H; e += NT) {
      const int col = e / H, k = e % H;
      if (col0 + col >= a.ncols) break;
      C2<R> X, Y;
      zunpack<R>(lines + (col / 2) * LP, L, k, X, Y);
      a.cplx[(size_t)(col0 + col) * H + k] = col % 2 == 0 ? X : Y;
    }
  }
}

template <typename R, int L, int CP, int NT>
__global__ void __launch_bounds__(NT, fz_min_blocks<R, L, NT>()) k_fz_c2r(FZArgs<R> a, const C2<R>* __restrict__ tw) {
  constexpr int H = L / 2 + 1;
  extern __shared__ __align__(16) unsigned char vk_smem[];
  __shared__ C2<R> tw_s[twtab_elems<R, true>(L)];
  load_twtab<R, L, true, NT>(tw_s, tw);
  grid_depend();
  const int col0 = blockIdx.x * 2 * CP;
  const auto ld = [&](int l, int p) -> C2x2<R> {
    const int c = col0 + 2 * l;
    const C2<R>* x = a.cplx + (size_t)c * H + (p < H ? p : L - p);
    C2x2<R> r{};
    if (c < a.ncols) r.a = x[0];
    if (c + 1 < a.ncols) r.b = x[H];
    return r;
  };
  const auto st = [&](int l, int p, C2<R> z) {
    const int c = col0 + 2 * l;
    R* x = a.real + (size_t)c * L + p;
    if (c < a.ncols) x[0] = z.x * a.scale;
    if (c + 1 < a.ncols) x[L] = z.y * a.scale;
  };
  if constexpr (sizeof(R) == 8) {
    FxLines<L, true, NT, CP, MapContig<R, L, CP>, false, 0, 0>::run(
        reinterpret_cast<fx2*>(vk_smem), reinterpret_cast<const fxtw*>(tw_s),
        FxFill<L, 0, 0, decltype(ld), ZPack<R, L>>{ld, ZPack<R, L>{}}, st, 0);
  } else {
    fft_lines<R, L, true, NT, CP, MapContig<R, L, CP>, false, true>(
        reinterpret_cast<C2<R>*>(vk_smem), tw_s, ld, ZPack<R, L>{}, st);
  }
}

}  // namespace vk
