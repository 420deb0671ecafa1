// Version 5 of the LU-SGS sweeps: the pipelined wavefront of lusgs.cuh (same tiles, same order of
// the dependencies) with the flux-difference terms computed on the producing side and every role of
// a step on its own warps, joined by mbarriers instead of by CTA-wide barriers.
//
// What bounds a sweep is the time of one step of a tile: a block's sweep is a chain of about
// nx + ny + nz of them.  Versions 3 and 4 take 2,000-3,000 cycles a step on B200: the same U + DU,
// reciprocal density and pressure are evaluated by three direction threads, each of its divisions
// is a subroutine of ~125 cycles with a branch, and two CTA barriers, sector bookkeeping and the
// final divisions sit in the chain.  Here
//   * a cell, once its DU is known, evaluates the three terms
//       0.5 (F(U+DU) - F(U)).n S + 0.5 w Lc DU + Lv DU        (sub_LU_SGS.f90:38-117, 135-157)
//     of its downstream faces itself, so U + DU, 1/rho and p exist once per cell, a cell's
//     neighbours need nothing of it but these terms, and they cross a tile edge as data (below);
//   * the quotients by one denominator share its reciprocal: r = RN(1/b), q = RN(x r),
//     q' = RN(q + r RN(x - b q)), the FMA division of Markstein (IBM J. Res. Dev. 34, 1990; Cornea,
//     Harrison and Tang, "Scientific Computing on Itanium", 2002), correctly rounded, hence the
//     bits of x / b, without a branch.  Large operands, small denominators, infinities and NaN take
//     the plain division (bad_den, bad_num).  Small numerators do not: -0 / b gives +0, and a
//     numerator whose remainder x - b q is subnormal (below about 2^-969 in FP64, 2^-103 in FP32)
//     can give a quotient one unit off.
//
// Warps of a CTA (TC columns per tile, TC = 32 or 64; RW = TC / 32 warps per group):
//   L (2 RW)    loads every input plane of the tile in blocks of WB steps, two blocks deep: a request
//               covers 32 / WB columns times WB consecutive i (a step's own cells lie on 32 different
//               rows, one sector each, and the L1 miss path takes one sector a cycle, 33 cycles a
//               warp request: 44 of them a step bounded the first form of this kernel).  The copies
//               (cp.async) land in rows by step, so a step's cells are one conflict-free row.  L also
//               stores the finished DU of a block, row-wise the same way;
//   D0, D1, D2  direction d: DU of the column's cell (each of the three evaluates it: cheaper than
//               a second barrier), then the term of the downstream face in direction d, into the
//               next step's slot, and the old state's flux of the next step's face; a step is one
//               straight-line block, so that these chains overlap;
//   P0, P1      the diagonal, 1/rho and E - kinetic energy of the old state into the ring of slots
//               (even and odd steps);
//   E           one warp: the terms that come from the upstream tiles.
// One named barrier of the D warps per step (the terms of step t before step t + 1 reads them); P
// and E run up to SLOTS steps ahead through the ring (full / empty mbarriers), L two blocks.
//
// Cross-tile terms: an edge column's terms are stored to a buffer of this tile (edge_off), one
// 8-byte word per value and step, and the consuming tile's warp E polls the words themselves: a
// word holds the sentinel until its value is stored, and E puts the sentinel back after reading it, so
// the buffer is ready for the next sweep.  The sentinel is a signalling NaN: FP64 arithmetic carries a
// quiet NaN's payload on (all ones, say, from a state filled with 0xFF), but the result of an operation
// on a signalling NaN is a quiet one (IEEE 754, 6.2; checked on B200 for add, mul and fma), and every
// term is the result of an operation.  No flag, no fence: one store and one L2 read between tiles.
// The wait is bounded (L.spin_limit, lu5_wait.h); E then sets the error flag and delivers zeros without
// waiting until the tile ends, and the tiles not yet begun are skipped, in this launch and in those
// before the host has read the flag: a failure costs about two bounds, not one per tile.  Deadlock
// freedom is that of lusgs.cuh: tiles are handed out in topological order to resident CTAs.
//
// Measured (B200, ms lower + upper sweep, the best of versions 3 and 4 -> this): config 2 (2.09 M
// cells, 8 blocks) FP64 0.690 + 0.669 -> 0.491 + 0.493, mixed 0.623 + 0.664 -> 0.426 + 0.430; 64
// airfoils mixed 0.742 + 0.704 -> 0.459 + 0.435; wing-body (7.8 M cells, SST) mixed 1.62 + 1.65 -> 1.30
// + 1.29; one 129 x 33 airfoil FP64 0.194 -> 0.110 a sweep, the 129 x 65 x 17 channel 0.33 -> 0.16.  A
// step takes about 1,400 cycles: a D warp's ~320 instructions at four to five cycles each (a chain of
// dependent FP64 operations and shared-memory reads), beside the SM's load path at about half of its
// rate (ncu on the channel, a step of a tile: 1,558 warp instructions of all roles, 666 wavefronts, of
// which 263 shared-memory loads, 198 of L's copies and 70 stores).  Tried on top and slower: step
// counters with acquire loads in place of the mbarriers (+3 %), DU shared between the D warps by
// variables with a second barrier (FP64 +15 %, mixed even), next step's mbarriers probed a step ahead
// (even), two CTAs per SM at 168 registers with one P and one L warp (config 2 FP64 +90 %: the single L
// warp bounds it), 64-column tiles (+60 %), face geometry and state loaded by the D and P warps
// themselves into registers (+20 to 40 %).
#pragma once
#include "lu5_wait.h"
#include "lusgs.cuh"

namespace ocfd {

// ns between a loader warp's requests: keeps bursts off the load path (wing-body sweep 1.37 -> 1.31 ms).
// Flat from 300 to 400 (257x97x86 FP64 step 2.60 ms); 150 gives 2.64 ms, 700 gives 2.68 ms.
constexpr int LU5_PACE = 300;
constexpr long long LU5_EMPTY = 0x7ff25ec0de5c0ffeLL;  // the sentinel of an edge word: a signalling NaN (quiet bit clear)

// ---- division by a shared reciprocal -------------------------------------------------------
// (rcp_rn, div_by and expo of double are in physics.cuh)
__device__ __forceinline__ float rcp_rn(float b) { return __frcp_rn(b); }
__device__ __forceinline__ float div_by(float x, float b, float r) {
  const float q = __fmul_rn(x, r);
  return __fmaf_rn(__fmaf_rn(-b, q, x), r, q);
}
// the exponent word of |x|, and whether operands lie outside the range div_by is exact in
__device__ __forceinline__ unsigned expo(float x) { return (unsigned)__float_as_int(x) & 0x7fffffffu; }
__device__ __forceinline__ bool bad_den(double b) { return expo(b) - 0x20000000u > 0x3fc00000u; }  // |b| in 2^-511 .. 2^509
__device__ __forceinline__ bool bad_num(unsigned e, double) { return e > 0x5fc00000u; }
__device__ __forceinline__ bool bad_den(float b) { return expo(b) - 0x20800000u > 0x3e800000u; }   // 2^-62 .. 2^63
__device__ __forceinline__ bool bad_num(unsigned e, float) { return e > 0x5f000000u; }

// The expressions of the flux difference.  FP64 rounds every operation, as the reference; the mixed
// form contracts them exactly as versions 3 and 4 compile (which product of a sum enters the FMA
// unrounded was found by comparing bits on random states; the compiler may choose otherwise in other
// code), so that every version of the sweep gives the same bits (halving the face area and radius first
// is exact but where an FP32 product is subnormal).
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double mad2(double a, double b, double c, double d) { return __dadd_rn(__dmul_rn(a, b), __dmul_rn(c, d)); }  // a b + c d
__device__ __forceinline__ float mad2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ double msub(double a, double b, double c) { return __dsub_rn(__dmul_rn(a, b), c); }  // a b - c
__device__ __forceinline__ float msub(float a, float b, float c) { return __fmaf_rn(a, b, -c); }
__device__ __forceinline__ double dot3(const double* u, const double* n) { return __dadd_rn(mad2(u[1], n[0], u[2], n[1]), __dmul_rn(u[3], n[2])); }
__device__ __forceinline__ float dot3(const float* u, const float* n) { return __fmaf_rn(u[3], n[2], mad2(u[1], n[0], u[2], n[1])); }
__device__ __forceinline__ double sq3(const double* u) { return __dadd_rn(mad2(u[1], u[1], u[2], u[2]), __dmul_rn(u[3], u[3])); }
__device__ __forceinline__ float sq3(const float* u) { return __fmaf_rn(u[3], u[3], mad2(u[1], u[1], u[2], u[2])); }

// ---- mbarriers -----------------------------------------------------------------------------
__device__ __forceinline__ void mb_init(unsigned a, int n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(n) : "memory"); }
__device__ __forceinline__ bool mb_try(unsigned a, unsigned parity) {
  unsigned ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mb_arrive(unsigned a) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory"); }
// waits for the phase of the given parity; bounded (another role of the CTA always makes progress:
// the bound only turns a defect into an error).  tries: the thread's bound, 0 once it has run out: its
// later waits end after one try (the tile is lost, every access stays in its place)
__device__ __forceinline__ void mb_wait(unsigned a, unsigned parity, int& tries, int* err) {
  for (int n = 0; !mb_try(a, parity);)
    if (++n > tries) { tries = 0; atomicExch(err, 1); return; }
}
__device__ __forceinline__ long long ld_word(const long long* p) {
  long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_word32(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(long long* p, long long v) { asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory"); }

// one element of at most 8 bytes into shared memory, and this thread's copies onto an mbarrier
template <class X>
__device__ __forceinline__ void cp_elem(unsigned dst, const X* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"((int)sizeof(X)) : "memory");
}
__device__ __forceinline__ void cp_arrive(unsigned a) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(a) : "memory"); }

// N values of one term
template <int N>
struct alignas(8 * N) Lu5Vec {
  double v[N];
};

// ---- shared memory (byte offsets) -------------------------------------------------------------
// Input rows: one row of TC cells per stream and step, 2 WB rows per stream (two blocks).  The row
// pitch is TC + 2 doubles or TC + 4 floats: the copies of a request (32 / WB columns x WB steps, a
// column's step being its i plus its skew) then fall into different banks.
// The right-hand side's rows hold doubles in every form: DU overwrites them.
// Slots (one per step, SLOTS of them): the terms of the three directions for the step's cells, a
// row of TC own columns followed by TC places for the upstream edges (placed so that a warp's read
// of own and edge columns is free of bank conflicts), and what P computes.
template <class T, int NV, bool UPPER, int TC>
struct Lu5Smem {
  using RT = typename std::conditional<UPPER, double, T>::type;  // right-hand side: Res (lower) or DU* (upper)
  static constexpr int WB = TC == 64 ? 4 : 8, ROWS = 2 * WB, SLOTS = TC == 64 ? 3 : 4;
  static constexpr int PB = (TC + 2) * 8, PT = sizeof(T) == 8 ? PB : (TC + 4) * 4;
  static constexpr int U = 0, R = U + NV * ROWS * PB, VOL = R + NV * ROWS * PB, DT = VOL + ROWS * PB;
  static constexpr int LC = DT + ROWS * PT, LV = LC + 3 * ROWS * PT, N = LV + 3 * ROWS * PT, S = N + 9 * ROWS * PT;
  static constexpr int SLOT0 = S + 3 * ROWS * PT;
  static constexpr int NA = sizeof(T) == 8 ? (NV == 6 ? 4 : 2) : (NV == 6 ? 2 : 1);  // diagonal: (value and) reciprocal, SA's own
  static constexpr int AS = 2 * TC + 2;  // the place behind the edges stays zero
  // a term's values lie in pairs of variables (one 16-byte access) for NV = 6: sweep -4 % on the SA
  // airfoil and wing; padding an odd NV costs more than it saves (SST airfoil 0.242 -> 0.270 ms)
  static constexpr int VP = NV % 2 == 0 ? 2 : 1, NP2 = NV / VP, VB = 8 * VP;
  static constexpr int ACC = 0, AL = ACC + 3 * NP2 * AS * VB, Q = AL + NA * TC * 8;  // Q: 1/rho, E - kinetic energy
  static constexpr int SU = Q + 2 * TC * (int)sizeof(T);                         // mixed form: the state in FP32
  static constexpr int SLOT = (SU + (sizeof(T) == 4 ? NV * TC * 4 : 0) + 15) / 16 * 16;
  static constexpr int BYTES = SLOT0 + SLOTS * SLOT;
  static_assert(SLOT0 % 16 == 0 && BYTES <= 227 * 1024, "shared memory of one CTA");
};
template <class T, int NV, bool UPPER, int TC>
inline size_t lu5_smem() { return (size_t)Lu5Smem<T, NV, UPPER, TC>::BYTES; }
template <int TC>
constexpr int lu5_threads() { return 7 * TC + 32; }

template <class T, int NV, bool UPPER, int TC>
__global__ void __launch_bounds__(7 * TC + 32, 1) k_lusgs_wave5(Arena<T> A, LuArgs L) {
  using SM = Lu5Smem<T, NV, UPPER, TC>;
  using RT = typename SM::RT;
  using VT = Lu5Vec<SM::VP>;
  using T2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
  constexpr int SLOTS = SM::SLOTS, WB = SM::WB, RW = TC / 32, NA = SM::NA, PB = SM::PB, PT = SM::PT, ROWS = SM::ROWS;
  constexpr bool FP64 = sizeof(T) == 8;
  constexpr int AS5 = NV == 6 ? 2 : 0;  // the SA variable's own diagonal (FP64 form: value, reciprocal)
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ __align__(8) unsigned long long s_bar[3 * SLOTS + 4];
  __shared__ int s_tile, s_err;
  const long long tb = A.tot_box, tf = A.tot_face, tc = A.tot_cell;
  const int TJ = L.TJ, TK = L.TK;
  const int tid = threadIdx.x, role = tid / TC, c = tid % TC, lane = tid & 31;  // roles 0..2: D, 3, 4: P, 5, 6: L, 7: E
  const int lj = c % TJ, lk = c / TJ;
  if (TJ * TK != TC || TK < 2 || TJ < 4 || TJ + TK > TC / 2 + 2) {  // a tile shape the edge and bank layouts do not cover: refuse
    if (tid == 0) atomicExch(L.err, 1);
    return;
  }
  // full (P's values), full (upstream terms), empty barrier of each slot; full and empty of the two row blocks
  const unsigned fullP = (unsigned)__cvta_generic_to_shared(s_bar), fullE = fullP + 8 * SLOTS, empty0 = fullP + 16 * SLOTS;
  const unsigned fullR = fullP + 24 * SLOTS, emptyR = fullR + 16;
  if (tid == 0) {
    for (int q = 0; q < SLOTS; q++) { mb_init(fullP + 8 * q, RW); mb_init(fullE + 8 * q, 1); mb_init(empty0 + 8 * q, 3 * RW); }
    for (int q = 0; q < 2; q++) { mb_init(fullR + 8 * q, 2 * TC); mb_init(emptyR + 8 * q, 3 * RW); }
  }
  for (int q = tid; q < SLOTS * 3 * SM::NP2; q += lu5_threads<TC>())  // the zero places
    reinterpret_cast<VT*>(s_dyn + SM::SLOT0 + q / (3 * SM::NP2) * SM::SLOT + SM::ACC)[(q % (3 * SM::NP2)) * SM::AS + 2 * TC] = VT{};
  // steps and row blocks this CTA has done (the same in every role): slot it % SLOTS, round
  // it / SLOTS; block buffer ib % 2, round ib / 2
  unsigned it = 0, ib = 0;
  int tries = lu5_tries(L.spin_limit);
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const int e = ld_word32(L.err), n = atomicAdd(&L.counter[UPPER ? 1 : 0], 1);  // both in flight at once
      s_err = e;
      s_tile = n;
    }
    __syncthreads();
    const int q = s_tile;
    if (q >= L.ntiles) {  // the last CTA to ask leaves the counter at 0 for the next sweep
      if (tid == 0 && q == L.ntiles + (int)gridDim.x - 1) L.counter[UPPER ? 1 : 0] = 0;
      break;
    }
    if (s_err) continue;  // a wait has run out, in this launch or one before: the sweep is lost
    const LuTile tl = UPPER ? L.rtiles[q] : L.tiles[q];
    const BlkD& B = A.blk[tl.blk];
    const SolveP& s = A.sp[B.solve];
    const int nxm = B.nx - 1, nym = B.ny - 1, nzm = B.nz - 1;
    const int j = UPPER ? (tl.j0 + TJ - 1 - lj) : (tl.j0 + lj);
    const int k = UPPER ? (tl.k0 + TK - 1 - lk) : (tl.k0 + lk);
    const bool active = j >= 1 && j <= nym && k >= 1 && k <= nzm;
    const int* tb3 = L.tile_of + 3 * tl.blk;
    const int first = tb3[0], nJ = tb3[1], nK = tb3[2];
    const int J = (tl.j0 - 1) / TJ, K = (tl.k0 - 1) / TK;
    const int nsteps = nxm + TJ + TK - 2, nblk = (nsteps + WB - 1) / WB;
    auto on_at = [&](int t) { const int il = t - lj - lk; return active && il >= 0 && il < nxm; };
    auto slot_of = [&](unsigned n) { return s_dyn + SM::SLOT0 + (n % SLOTS) * SM::SLOT; };
    auto row_of = [&](int t) { return (int)((ib + t / WB) & 1) * WB + t % WB; };  // the row of step t in every stream
    if (role < 3) {
      // ------------------------------------------------------------------ direction warps
      const int d = role;
      const double w = s.w_lu;
      const bool visc = NV >= 6 || s.viscous == 1;  // a turbulence model implies the viscous terms
      const T g1 = (T)(s.gamma - 1.0), half = (T)0.5;
      const bool has_j = UPPER ? j != nym : j != 1, has_k = UPPER ? k != nzm : k != 1;  // upstream neighbours
      // places of the upstream terms: the own column's, its neighbours' (or the upstream edges' behind
      // them), or the zero place where there is no neighbour
      const int a_i = c * SM::VB, a_z = 2 * TC * SM::VB;
      const int a_j = (SM::NP2 * SM::AS + (!has_j ? 2 * TC : (lj > 0 ? c - 1 : TC + c + TJ - 1))) * SM::VB;
      const int a_k = (2 * SM::NP2 * SM::AS + (!has_k ? 2 * TC : (lk > 0 ? c - TJ : TC + TC - TJ + lj))) * SM::VB;
      // does this column's term leave the tile?  Edge words: j edge [step][m][lk], then k edge [step][m][lj]
      const bool out = d == 1 ? (lj == TJ - 1 && (UPPER ? J > 0 : J < nJ - 1)) : (d == 2 && lk == TK - 1 && (UPPER ? K > 0 : K < nK - 1));
      const int ow = d == 1 ? TK : TJ;
      long long* const eout = L.edge + L.edge_off[first + J + nJ * K] + (d == 1 ? lk : (long long)nsteps * NV * TK + lj);
      struct Cell {
        T U[NV], r0, ei, g[6];  // state, 1/rho, E - kinetic energy; downstream face: normal, area / 2; w Lc / 2, Lv
        RT R[NV];
        double al[NA];
      };
      auto take = [&](Cell& x, const unsigned char* sl, int row) {
        const unsigned char* const r8 = s_dyn + row * PB + c * 8;
        const unsigned char* const rt = s_dyn + row * PT + c * (int)sizeof(T);
#pragma unroll
        for (int m = 0; m < NV; m++) {
          if (FP64) {
            const double u = *reinterpret_cast<const double*>(r8 + SM::U + m * ROWS * PB);
            x.U[m] = (T)(m >= 5 ? clamp0(u) : u);
          } else {
            x.U[m] = reinterpret_cast<const T*>(sl + SM::SU)[m * TC + c];
          }
          x.R[m] = *reinterpret_cast<const RT*>(s_dyn + SM::R + (m * ROWS + row) * PB + c * (int)sizeof(RT));
        }
#pragma unroll
        for (int m = 0; m < 3; m++) x.g[m] = *reinterpret_cast<const T*>(rt + SM::N + (3 * d + m) * ROWS * PT);
        // halving is exact: 0.5 (DF S + w Lc DU) = DF (S / 2) + (w Lc / 2) DU in every rounding
        x.g[3] = (T)(UPPER ? -0.5 : 0.5) * *reinterpret_cast<const T*>(rt + SM::S + d * ROWS * PT);
        x.g[4] = (T)0.5 * (T)(w * (double)*reinterpret_cast<const T*>(rt + SM::LC + d * ROWS * PT));
        x.g[5] = *reinterpret_cast<const T*>(rt + SM::LV + d * ROWS * PT);
        if constexpr (NA == 1) {
          x.al[0] = reinterpret_cast<const double*>(sl + SM::AL)[c];
        } else {
#pragma unroll
          for (int m = 0; m < NA / 2; m++) {
            const double2 p = reinterpret_cast<const double2*>(sl + SM::AL)[m * TC + c];
            x.al[2 * m] = p.x;
            x.al[2 * m + 1] = p.y;
          }
        }
        const T2 q = reinterpret_cast<const T2*>(sl + SM::Q)[c];
        x.r0 = q.x;
        x.ei = q.y;
      };
      // F(U).n of the old state (plain: by plain division); true: operands div_by does not cover
      auto old_flux = [&](const Cell& x, T* F, bool plain) -> bool {
        const T dot = dot3(x.U, x.g);
        const T un = plain ? dot / x.U[0] : div_by(dot, x.U[0], x.r0);
        const T p = mul_rn(g1, x.ei);
        F[0] = x.U[0] * un;
#pragma unroll
        for (int m = 1; m < 4; m++) F[m] = NV == 7 && m == 3 ? mad2(p, x.g[2], x.U[3], un) : mad2(x.U[m], un, p, x.g[m - 1]);
        F[4] = add_rn(x.U[4], p) * un;
#pragma unroll
        for (int m = 5; m < NV; m++) F[m] = x.U[m] * un;
        return bad_den(x.U[0]) || bad_num(expo(dot), dot);
      };
      // DU of the cell (sub_LU_SGS.f90:63-72 lower, 108-117 upper) from the sum xs, and the term v of
      // its downstream face; plain and the result as above
      auto cell = [&](const Cell& x, const T* F, const double* xs, double* DU, double* v, bool plain) -> bool {
        unsigned e = 0;
#pragma unroll
        for (int m = 0; m < NV; m++) {
          if (FP64) {
            const int q5 = m == 5 ? AS5 : 0;
            DU[m] = plain ? xs[m] / x.al[q5] : div_by(xs[m], x.al[q5], x.al[q5 + 1]);
            if (UPPER) DU[m] = (double)x.R[m] + DU[m];
            e = max(e, expo(xs[m]));
          } else {  // the mixed form multiplies by the diagonal's FP64 reciprocal
            const double ra = x.al[NV == 6 && m == 5 ? 1 : 0];
            DU[m] = UPPER ? __fma_rn(xs[m], ra, (double)x.R[m]) : __dmul_rn(xs[m], ra);
          }
        }
        bool bad = FP64 && (bad_num(e, 0.0) || bad_den(x.al[0]) || bad_den(x.al[AS5 < NA ? AS5 : 0]));
        T U2[NV];
#pragma unroll
        for (int m = 0; m < NV; m++) U2[m] = (T)__dadd_rn((double)x.U[m], DU[m]);  // DU rounded first, in the mixed form too
        const T r2 = rcp_rn(U2[0]);
        const T dot = dot3(U2, x.g), kin = half * sq3(U2);
        const T un = plain ? dot / U2[0] : div_by(dot, U2[0], r2);
        const T ke = plain ? kin / U2[0] : div_by(kin, U2[0], r2);
        bad = bad || bad_den(U2[0]) || bad_num(max(expo(dot), expo(kin)), dot);
        const T p = mul_rn(g1, U2[4] - ke);
        T DF[NV];
        DF[0] = msub(U2[0], un, F[0]);
#pragma unroll
        for (int m = 1; m < 4; m++) DF[m] = (m == 3 || (NV == 7 && m == 2) ? mad2(p, x.g[m - 1], U2[m], un) : mad2(U2[m], un, p, x.g[m - 1])) - F[m];
        DF[4] = msub(add_rn(U2[4], p), un, F[4]);
#pragma unroll
        for (int m = 5; m < NV; m++) DF[m] = msub(U2[m], un, F[m]);
#pragma unroll
        for (int m = 0; m < NV; m++) {
          if (!FP64) {  // off-diagonal products in FP32, the sum stays FP64
            const float du = (float)DU[m], y = __fmaf_rn((float)DF[m], (float)x.g[3], __fmul_rn((float)x.g[4], du));
            v[m] = (double)(visc ? __fmaf_rn((float)x.g[5], du, y) : y);
          } else {
            const double y = mad2((double)DF[m], (double)x.g[3], (double)x.g[4], DU[m]);
            v[m] = visc ? y + (double)x.g[5] * DU[m] : y;
          }
        }
        return bad;
      };
      T F[2][NV];
      Cell x[2];
      mb_wait(fullP + 8 * (it % SLOTS), (it / SLOTS) & 1, tries, L.err);
      take(x[0], slot_of(it), row_of(0));
      if (old_flux(x[0], F[0], false)) old_flux(x[0], F[0], true);
      for (int t0 = 0; t0 < nsteps; t0 += 2) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int t = t0 + u;
          if (t >= nsteps) break;
          const unsigned n = it + t;
          const unsigned char* const sl = slot_of(n);
          unsigned char* const ns = slot_of(n + 1);
          Cell& xc = x[u];
          Cell& xn = x[1 - u];
          // the upstream terms of this step and P's values of the next one (there is none after the
          // last); P has read its inputs from the rows of that step, so D may
          {
            const unsigned ea = fullE + 8 * (n % SLOTS), ep = (n / SLOTS) & 1;
            const unsigned pa = t + 1 < nsteps ? fullP + 8 * ((n + 1) % SLOTS) : ea, pp = t + 1 < nsteps ? ((n + 1) / SLOTS) & 1 : ep;
            const bool e0 = mb_try(ea, ep), p0 = mb_try(pa, pp);
            if (!(e0 && p0)) { mb_wait(ea, ep, tries, L.err); mb_wait(pa, pp, tries, L.err); }
          }
          cta_bar_id<1, 3 * TC>();  // the terms of step t - 1 are in slot t
          double xs[NV];
          {
            const unsigned char* const acc = sl + SM::ACC;
            const int ai = t - lj - lk > 0 ? a_i : a_z;
#pragma unroll
            for (int p = 0; p < SM::NP2; p++) {
              const VT b0 = *reinterpret_cast<const VT*>(acc + ai + p * SM::AS * SM::VB);
              const VT b1 = *reinterpret_cast<const VT*>(acc + a_j + p * SM::AS * SM::VB);
              const VT b2 = *reinterpret_cast<const VT*>(acc + a_k + p * SM::AS * SM::VB);
#pragma unroll
              for (int e = 0; e < SM::VP; e++) {
                const int m = SM::VP * p + e;
                xs[m] = UPPER ? b0.v[e] + b1.v[e] + b2.v[e] : (double)xc.R[m] + b0.v[e] + b1.v[e] + b2.v[e];
              }
            }
          }
          take(xn, ns, row_of(t + 1));
          const bool on = on_at(t);
          double DU[NV], v[NV];
          const bool bad = cell(xc, F[u], xs, DU, v, false);
          const bool badn = old_flux(xn, F[1 - u], false);
          if ((bad && on) || badn) {
            cell(xc, F[u], xs, DU, v, true);
            old_flux(xn, F[1 - u], true);
          }
          VT* const nacc = reinterpret_cast<VT*>(ns + SM::ACC) + d * SM::NP2 * SM::AS + c;
#pragma unroll
          for (int p = 0; p < SM::NP2; p++) {
            VT x2;
#pragma unroll
            for (int e = 0; e < SM::VP; e++) x2.v[e] = v[SM::VP * p + e];
            nacc[p * SM::AS] = x2;
          }
          if (out && on) {
#pragma unroll
            for (int m = 0; m < NV; m++) st_word(eout + t * (NV * ow) + m * ow, __double_as_longlong(v[m]));
          }
          if (d == 0) {  // over the right-hand side's row of this step
            double* const o = reinterpret_cast<double*>(s_dyn + SM::R + row_of(t) * PB) + c;
#pragma unroll
            for (int m = 0; m < NV; m++) o[m * ROWS * (PB / 8)] = DU[m];
          }
          __syncwarp();
          if (lane == 0) {
            mb_arrive(empty0 + 8 * (n % SLOTS));  // this warp's reads of slot t are done
            if (t % WB == WB - 1 || t == nsteps - 1) mb_arrive(emptyR + 8 * ((ib + t / WB) & 1));  // and the block's
          }
        }
      }
    } else if (role < 5) {
      // ------------------------------------------------------------------ diagonal and old-state values
      const double w = s.w_lu;
      const bool visc = NV >= 6 || s.viscous == 1, dual = s.time_method == -1;
      const double sfac1 = dual ? A.sfac[1] : 0.0;
      const T half = (T)0.5;
      for (int t = role - 3; t < nsteps; t += 2) {  // even or odd steps of the tile
        const unsigned n = it + t, rb = ib + t / WB;
        unsigned char* const sl = slot_of(n);
        if (t % WB < 2) mb_wait(fullR + 8 * (rb & 1), (rb >> 1) & 1, tries, L.err);  // this warp's first step of the block
        const int row = row_of(t);
        const unsigned char* const r8 = s_dyn + row * PB + c * 8;
        const unsigned char* const rt = s_dyn + row * PT + c * (int)sizeof(T);
        T U[NV];
#pragma unroll
        for (int m = 0; m < NV; m++) {
          const double u = *reinterpret_cast<const double*>(r8 + SM::U + m * ROWS * PB);
          U[m] = (T)(m >= 5 ? clamp0(u) : u);
        }
        const double vol = *reinterpret_cast<const double*>(r8 + SM::VOL);
        const double dtd = (double)*reinterpret_cast<const T*>(rt + SM::DT);
        double lc[3], lvd[3];
#pragma unroll
        for (int m = 0; m < 3; m++) {
          lc[m] = (double)*reinterpret_cast<const T*>(rt + SM::LC + m * ROWS * PT);
          lvd[m] = (double)*reinterpret_cast<const T*>(rt + SM::LV + m * ROWS * PT);
        }
        const T r0 = rcp_rn(U[0]);
        const T kin = half * sq3(U);
        T ke = div_by(kin, U[0], r0);
        // the diagonal (sub_LU_SGS.f90:50-62, 90-92)
        double vdt = div_by(vol, dtd, rcp_rn(dtd));
        if (bad_den(U[0]) || bad_num(expo(kin), kin) || bad_den(dtd) || bad_num(expo(vol), 0.0)) { ke = kin / U[0]; vdt = vol / dtd; }
        const T ei = U[4] - ke;
        const double a0 = vdt + w * (lc[0] + lc[1] + lc[2]);
        double al = a0, als = a0;
        if (visc) {
          const double lv = lvd[0] + lvd[1] + lvd[2];
          al = al + 2.0 * lv;
          als = als + 2.0 * lv;
          if (NV == 6) {  // lower: + (Lv sum); upper: + Lv1 + Lv2 + Lv3 term by term
            if (!UPPER) als = als + lv;
            else als = als + lvd[0] + lvd[1] + lvd[2];
          }
        }
        if (dual) {  // dual time: + Sfac1 vol (sub_LU_SGS.f90:39, 92)
          al = al + sfac1 * vol;
          als = als + sfac1 * vol;
        }
        double ra = rcp_rn(al), ras = NV == 6 ? rcp_rn(als) : 0.0;
        if (bad_den(al) || (NV == 6 && bad_den(als))) { ra = 1.0 / al; ras = 1.0 / als; }
        mb_wait(empty0 + 8 * (n % SLOTS), (n / SLOTS + 1) & 1, tries, L.err);  // the slot's last readers are done
        if constexpr (NA == 1) {
          reinterpret_cast<double*>(sl + SM::AL)[c] = ra;
        } else {
          double2* const pa = reinterpret_cast<double2*>(sl + SM::AL) + c;
          pa[0] = FP64 ? make_double2(al, ra) : make_double2(ra, ras);
          if (NA == 4) pa[TC] = make_double2(als, ras);
        }
        T2 q2;
        q2.x = r0;
        q2.y = ei;
        reinterpret_cast<T2*>(sl + SM::Q)[c] = q2;
        if (!FP64) {
#pragma unroll
          for (int m = 0; m < NV; m++) reinterpret_cast<T*>(sl + SM::SU)[m * TC + c] = U[m];
        }
        __syncwarp();
        if (lane == 0) mb_arrive(fullP + 8 * (n % SLOTS));
      }
    } else if (role < 7) {
      // ------------------------------------------------------------------ input rows in, DU out
      constexpr int LW = 2 * RW, CR = 32 / WB, NR = TC / CR / LW;  // loader warps; columns per request; requests per stream and warp
      const int lw = (tid - 5 * TC) / 32, iw = lane % WB;
      long long cb[NR], bb[NR], fb[NR];
      int sk[NR], col[NR];
      bool act[NR], dj[NR], dk[NR];
#pragma unroll
      for (int r = 0; r < NR; r++) {
        col[r] = (lw * NR + r) * CR + lane / WB;
        const int qj = col[r] % TJ, qk = col[r] / TJ;
        const int jj = UPPER ? (tl.j0 + TJ - 1 - qj) : (tl.j0 + qj), kk = UPPER ? (tl.k0 + TK - 1 - qk) : (tl.k0 + qk);
        act[r] = jj >= 1 && jj <= nym && kk >= 1 && kk <= nzm;
        // idle columns and steps load a cell of the block that nobody uses
        const int jc = min(max(jj, 1), nym), kc = min(max(kk, 1), nzm);
        sk[r] = qj + qk;
        dj[r] = jc > 1;
        dk[r] = kc > 1;
        cb[r] = B.ocell - 1 + (long long)nxm * ((jc - 1) + (long long)nym * (kc - 1));
        bb[r] = B.obox + 3 + (long long)B.NX * ((jc + 3) + (long long)B.NY * (kc + 3));
        fb[r] = B.oface - 1 + (long long)B.nx * ((jc - 1) + (long long)B.ny * (kc - 1));
      }
      const unsigned base = (unsigned)__cvta_generic_to_shared(s_dyn);
      const long long sj = B.nx, sk2 = (long long)B.nx * B.ny;
      for (int wb = 0; wb < nblk + 2; wb++) {
        const unsigned gb = ib + wb;
        const int row = (int)(gb & 1) * WB + iw;
        if (wb >= 2) {  // block wb - 2 is done: its DU to memory, then its rows are free
          mb_wait(emptyR + 8 * (gb & 1), ((gb - 2) >> 1) & 1, tries, L.err);
          // its copies have landed long since, unless a wait ran out: none may be in flight at the kernel's end
          // (cp.async.wait_all there instead costs 1 us a sweep, even behind a branch that is never taken)
          mb_wait(fullR + 8 * (gb & 1), ((gb - 2) >> 1) & 1, tries, L.err);
          const int t = (wb - 2) * WB + iw;
#pragma unroll
          for (int r = 0; r < NR; r++) {
            const int il = t - sk[r];
            if (act[r] && il >= 0 && il < nxm) {
              double* const o = A.DU + cb[r] + (UPPER ? nxm - il : il + 1);
              const double* const v = reinterpret_cast<const double*>(s_dyn + SM::R + row * PB) + col[r];
#pragma unroll
              for (int m = 0; m < NV; m++) o[m * tc] = v[m * ROWS * (PB / 8)];
            }
          }
        }
        if (wb >= nblk) continue;
        cta_bar_id<2, 2 * TC>();  // every loader warp has read the rows
        const int t = wb * WB + iw;
#pragma unroll
        for (int r = 0; r < NR; r++) {
          if (wb >= 2) __nanosleep(LU5_PACE);  // leaves the load path to D's reads in between
          const int il = min(max(t - sk[r], 0), nxm - 1), i = UPPER ? nxm - il : il + 1;
          const unsigned d8 = base + row * PB + col[r] * 8, dt_ = base + row * PT + col[r] * (int)sizeof(T);
          const double* const pU = A.U + bb[r] + i;
          const long long ci = cb[r] + i, f = fb[r] + i;
#pragma unroll
          for (int m = 0; m < NV; m++) {
            cp_elem(d8 + SM::U + m * ROWS * PB, pU + m * tb);
            if (UPPER) cp_elem(d8 + SM::R + m * ROWS * PB, A.DU + ci + m * tc);  // DU* of the lower sweep
            else cp_elem(base + SM::R + (m * ROWS + row) * PB + col[r] * (int)sizeof(T), A.Res + ci + m * tc);
          }
          cp_elem(d8 + SM::VOL, A.vold + ci);
          cp_elem(dt_ + SM::DT, A.dt + ci);
          // the downstream face of direction m: its normal is the lower face's of the downstream cell,
          // its area the lower face's (lower sweep) or the upper face's of that cell (upper sweep,
          // sub_LU_SGS.f90:96-97); without a downstream cell the term is not used
#pragma unroll
          for (int m = 0; m < 3; m++) {
            cp_elem(dt_ + SM::LC + m * ROWS * PT, A.Lc + ci + m * tc);
            cp_elem(dt_ + SM::LV + m * ROWS * PT, A.Lv + ci + m * tc);
            const long long st = m == 0 ? 1 : (m == 1 ? sj : sk2);
            const long long fn = UPPER ? ((m == 0 ? i > 1 : (m == 1 ? dj[r] : dk[r])) ? f - st : f) : f + st;
            const T* const pn = A.M + (M_NI1 + 3 * m) * tf + fn;
            cp_elem(dt_ + SM::N + (3 * m) * ROWS * PT, pn);
            cp_elem(dt_ + SM::N + (3 * m + 1) * ROWS * PT, pn + tf);
            cp_elem(dt_ + SM::N + (3 * m + 2) * ROWS * PT, pn + 2 * tf);
            cp_elem(dt_ + SM::S + m * ROWS * PT, A.M + (M_SI + m) * tf + (UPPER ? f : f + st));
          }
        }
        cp_arrive(fullR + 8 * (gb & 1));
      }
    } else {
      // ------------------------------------------------------------------ terms from the upstream tiles
      constexpr int EPL = (NV * (TC / 2 + 2) + 31) / 32, W = EPL > 4 ? 2 : 4;  // words per lane and step; steps polled at once
      const bool up_j = UPPER ? J < nJ - 1 : J > 0, up_k = UPPER ? K < nK - 1 : K > 0;
      long long* src[EPL];
      int lo[EPL], stride[EPL], dst[EPL];
      const int step_j = first + (UPPER ? J + 1 : J - 1) + nJ * K, step_k = first + J + nJ * (UPPER ? K + 1 : K - 1);
#pragma unroll
      for (int e = 0; e < EPL; e++) {
        const int x = lane + 32 * e;
        src[e] = nullptr; lo[e] = 0; stride[e] = 0; dst[e] = 0;
        if (x < NV * TK) {  // j edge: the upstream tile's column (TJ - 1, ek), TJ - 1 steps later there
          const int m = x / TK, ek = x % TK, kk = UPPER ? tl.k0 + TK - 1 - ek : tl.k0 + ek;
          if (up_j && kk >= 1 && kk <= nzm) {
            src[e] = L.edge + L.edge_off[step_j] + ((long long)(TJ - 1) * NV + m) * TK + ek;
            stride[e] = NV * TK; lo[e] = ek; dst[e] = ((SM::NP2 + m / SM::VP) * SM::AS + TC + ek * TJ + TJ - 1) * SM::VP + m % SM::VP;
          }
        } else if (x < NV * (TJ + TK)) {  // k edge
          const int m = (x - NV * TK) / TJ, ej = (x - NV * TK) % TJ, jj = UPPER ? tl.j0 + TJ - 1 - ej : tl.j0 + ej;
          if (up_k && jj >= 1 && jj <= nym) {
            src[e] = L.edge + L.edge_off[step_k] + (long long)nsteps * NV * TK + ((long long)(TK - 1) * NV + m) * TJ + ej;
            stride[e] = NV * TJ; lo[e] = ej; dst[e] = ((2 * SM::NP2 + m / SM::VP) * SM::AS + TC + TC - TJ + ej) * SM::VP + m % SM::VP;
          }
        }
      }
      const int rounds = lu5_rounds(L.spin_limit);
      int spins = 0;
      bool gave_up = false;
      int t = 0;
      while (t < nsteps) {
        long long v[W][EPL];
        int ready = 0;
        bool all = true;
#pragma unroll
        for (int g = 0; g < W; g++)
#pragma unroll
          for (int e = 0; e < EPL; e++) {
            const int il = t + g - lo[e];
            v[g][e] = 0;
            if (src[e] && il >= 0 && il < nxm && !gave_up) v[g][e] = ld_word(src[e] + (long long)(t + g) * stride[e]);
          }
#pragma unroll
        for (int g = 0; g < W; g++) {
          bool here = t + g < nsteps;
#pragma unroll
          for (int e = 0; e < EPL; e++) here &= v[g][e] != LU5_EMPTY;
          all = all && __all_sync(0xffffffffu, here);
          ready += all ? 1 : 0;
        }
        if (ready == 0) {
          if (++spins > rounds) {
            gave_up = true;
            if (lane == 0) atomicExch(L.err, 1);
          }
          continue;
        }
        spins = 0;
#pragma unroll
        for (int g = 0; g < W; g++) {
          if (g >= ready) break;
          const unsigned n = it + t + g;
          double* const acc = reinterpret_cast<double*>(slot_of(n) + SM::ACC);
          mb_wait(empty0 + 8 * (n % SLOTS), (n / SLOTS + 1) & 1, tries, L.err);
#pragma unroll
          for (int e = 0; e < EPL; e++) {
            const int il = t + g - lo[e];
            if (src[e] && il >= 0 && il < nxm) {
              acc[dst[e]] = __longlong_as_double(v[g][e]);
              st_word(src[e] + (long long)(t + g) * stride[e], LU5_EMPTY);
            }
          }
          __syncwarp();
          if (lane == 0) mb_arrive(fullE + 8 * (n % SLOTS));
        }
        t += ready;
      }
    }
    it += nsteps;
    ib += nblk;
  }
}

template <class T, int NV, int TC>
inline void lu_wave5_prepare() {
  cudaFuncSetAttribute(k_lusgs_wave5<T, NV, false, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lu5_smem<T, NV, false, TC>());
  cudaFuncSetAttribute(k_lusgs_wave5<T, NV, true, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lu5_smem<T, NV, true, TC>());
}

}  // namespace ocfd
