// kernels.cuh -- sm_103a kernels of the BSAM adaptive FAS V-cycle (FP64).
//
// Every kernel restates one step of the reference's MATLAB solve path in the
// reference's floating-point operation order (the library is compiled with
// --fmad=false, so no multiply-add is contracted).  Work is flattened per
// level over all patches: a level's items (colour cells, cells, coarse
// cells, ...) are numbered consecutively patch after patch and cut into
// 256-item blocks; `blk_p0[b]` names the patch that holds block b's first
// item, `beg[p]..beg[p+1]` the items of patch p.
//
// Memory layout in HBM: one array per field with every patch of every level
// concatenated, each patch column-major (x fastest) like the reference; the
// solution Q and the coarse shadows QC carry their one-cell ghost frame.
//
// Launch chaining (programmatic dependent launch): a kernel first loads what
// no kernel of the solve writes (patch records, coefficients, ghost rules,
// index tables), then executes griddepcontrol.wait, after which it reads and
// writes the solution state, and only then griddepcontrol.launch_dependents:
// one kernel ahead is resident, and its static loads run beside this one's
// work.  (With the trigger at entry the waiting blocks of many kernels pile
// up, each grid's blocks go wherever those before it left room, and an
// FP64-heavy kernel runs on part of the SMs: the starfish's second-finest
// prolongation took 13-20 us instead of 3.9, its smoother passes 4.9 instead
// of 3.9, an iteration 469 instead of 409 us.)  Every thread executes the
// wait before it exits, so no kernel completes before its predecessor.
#pragma once
#include <cooperative_groups.h>
#include <cstdint>
#include <cuda_runtime.h>

#include "stencil.cuh"

namespace bsam {

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// the wait of a kernel that writes operands which its successors read before
// their own wait (coefficients, sources): no early trigger, so that the next
// kernel starts when this one's stores are visible
__device__ __forceinline__ void chain_wait_static() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// a solution load; kCG: from L2 (ld.global.cg), for kernels whose blocks
// read values other blocks of the same launch wrote after a cluster barrier
// (another SM's L1 may hold an older copy of the line)
template <bool kCG, class T>
__device__ __forceinline__ T ld_sol(const T *p) {
  if constexpr (kCG) return __ldcg(p);
  else return *p;
}

// A double product on the integer pipe, correctly rounded (to nearest, ties to
// even): the 53-bit significands' product from four 32-bit multiply-adds,
// one bit of normalisation, rounding by a carry.  Operands that are zero,
// denormal, infinite or NaN and results near the ends of the exponent range
// take the multiply instruction.  GB300 starts a warp's FP64 operation every
// 19 cycles per SM and four warps' integer operations every cycle, so a
// kernel bound by the FP64 pipe gains from moving products over: the
// smoother's update (five products, four additions) ran at 55.9 G/s with
// none, 99.0 with four and 104.1 with five of its products formed this way.
__device__ __noinline__ double mul_fp64_pipe(double a, double b) { return a * b; }
__device__ __forceinline__ double mul_int_pipe(double a, double b) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  // significands: a's in 53 bits, b's at the top of 64
  const unsigned a1 = (ah & 0xfffffu) | 0x100000u;
  const unsigned b1 = __funnelshift_l(bl, (bh & 0xfffffu) | 0x100000u, 11), b0 = bl << 11;
  const uint64_t p = (uint64_t)al * b0;
  const uint64_t t = (uint64_t)al * b1 + (p >> 32);
  const uint64_t u = (uint64_t)a1 * b0 + (uint32_t)t;
  const uint64_t hi = (uint64_t)a1 * b1 + (t >> 32) + (u >> 32);   // in [2^51, 2^53)
  const unsigned hh = (unsigned)(hi >> 32), hl = (unsigned)hi, l1 = (unsigned)u, l0 = (unsigned)p;
  const unsigned n = (~hh >> 20) & 1u;                             // below 2^52: one bit more
  const unsigned h1 = __funnelshift_l(hl, hh, n), h0 = __funnelshift_l(l1, hl, n), r = __funnelshift_l(l0, l1, n);
  const unsigned rest = r | ((l0 << n) ? 1u : 0u);                 // what is cut off, its tail as one bit
  uint64_t m = ((uint64_t)h1 << 32) | h0;
  m += ((uint64_t)rest + 0x7fffffffu + (h0 & 1u)) >> 32;
  const unsigned ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
  const unsigned e = ea + eb - (1023u << 20) - (n << 20);          // the result's exponent field minus one
  double q = __hiloint2double((int)(((unsigned)(m >> 32) + e) ^ ((ah ^ bh) & 0x80000000u)), (int)(unsigned)m);
  const bool in = ea - 0x00100000u < 0x7fe00000u && eb - 0x00100000u < 0x7fe00000u && (int)e >= 0x00100000 &&
                  (int)e < 0x7fd00000;
  if (!in) q = mul_fp64_pipe(a, b);
  return q;
}
// the product on the pipe of choice
template <bool kInt>
__device__ __forceinline__ double mul_on(double a, double b) {
  return kInt ? mul_int_pipe(a, b) : a * b;
}
template <bool kInt>
__device__ __forceinline__ float mul_on(float a, float b) {
  return a * b;
}

// 3 x and 9 x on the integer pipe, correctly rounded: the significand times K
// has one or two bits (K = 9: three or four) too many, which are rounded to
// nearest even; zeros, denormals, infinities, NaN and results beyond the
// range take the multiply instruction
template <int K>
__device__ __forceinline__ double times_int_pipe(double x) {
  static_assert(K == 3 || K == 9, "");
  constexpr int kLog = K == 3 ? 1 : 3;
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const uint64_t m = ((uint64_t)((h & 0xfffffu) | 0x100000u) << 32) | l;
  const uint64_t w = m + (m << kLog);
  const unsigned n = kLog + ((unsigned)(w >> (53 + kLog)) & 1u);       // bits to drop
  const uint64_t r = (w + ((1u << (n - 1)) - 1u) + ((unsigned)(w >> n) & 1u)) >> n;
  const unsigned e = h & 0x7ff00000u;
  // the significand's leading bit adds the one that the exponent field lacks
  const double q = __hiloint2double((int)((unsigned)(r >> 32) + ((h & 0xfff00000u) + ((n - 1) << 20))), (int)(unsigned)r);
  const bool in = e - 0x00100000u < 0x7f800000u;                       // 1 <= exponent field <= 2040
  return in ? q : mul_fp64_pipe(x, (double)K);
}
// x / 16: the exponent field less four
__device__ __forceinline__ double sixteenth_int_pipe(double x) {
  const unsigned h = (unsigned)__double2hiint(x);
  const bool in = (h & 0x7ff00000u) - 0x00500000u < 0x7fa00000u;       // 5 <= exponent field <= 2046
  return in ? __hiloint2double((int)(h - 0x00400000u), __double2loint(x)) : mul_fp64_pipe(x, 0.0625);
}
template <int K, bool kInt, class T>
__device__ __forceinline__ T times(T x) {
  if constexpr (kInt && sizeof(T) == 8) return times_int_pipe<K>(x);
  else return T(K) * x;
}
template <bool kInt, class T>
__device__ __forceinline__ T sixteenth(T x) {
  if constexpr (kInt && sizeof(T) == 8) return sixteenth_int_pipe(x);
  else return x / 16;
}

// per-patch metadata on the device
struct PatchD {
  int mx, my, par0, level;
  int q_off, c_off, dew_off, dns_off;
  int qc_off, bcg_off, cfd_off, pc_off;
  int win_off, fp_off, corr_off, pe_off;   // pe_off: perimeter ghost-rule table
  int bc[4];
  int inst;                    // instance of a batch (0 for a single hierarchy)
  int pflags;                  // bit0: level >= the instance's root (in the norms)
                               // bit1: QC refreshed by the residual (level >= root+1)
  int ilo, jlo;                // 1-based origin of the patch box in the level's index space
};

// the arrays one V-cycle works on, in its value type T: the FP64 solve
// (T = double) or the FP32 correction cycle of the mixed form (T = float:
// Q is the correction, F its right-hand side, coefficients FP32 copies)
template <class T>
struct FieldsT {
  T *Q, *F, *QC;
  const double *FTrue;         // FP64 source (residual only)
  const T *CC, *ID, *DeW, *DnS, *bcg, *cfd, *pcoef;
  const uint8_t *flags;        // bit0 covered by a finer level, bit1 correction target
  const int *win, *fp;         // window gathers, footprint scatters (2 ints/cell)
  const int *active;           // per instance: 1 while its V-cycles continue (below)
  int lsh;                     // the launch's (finer) level lives at Q + lsh: 0, or its second copy
                               // between the two relaxations of the tile form (tile.cuh)
};
// `active` is written only by k_solve_step, the last kernel of a launch
// chain, and the host synchronises before the next chain (or writes it with
// a stream-ordered copy).  Within a chain no kernel can still be in its
// pre-wait part when k_solve_step's body runs (every kernel completes
// only after its predecessor), so kernels read `active` before
// griddepcontrol.wait and the blocks of a frozen instance skip their loads.
using Fields = FieldsT<double>;

// FP64 view of a value of either type (a no-op for double).  A float is
// widened on the integer pipe: the conversion instruction shares the FP64
// pipe (one warp every 19 cycles per SM), and the mixed form's coarse load
// converts as many values as it does FP64 operations.  A denormal is brought
// to the normal range first (an exact FP32 product).
__device__ __forceinline__ double dbl(double x) { return x; }
__device__ __forceinline__ double dbl(float x) {
  unsigned u = __float_as_uint(x), off = 0x38000000u;   // (1023 - 127) << 20
  const unsigned m = u & 0x7fffffffu;
  if (m < 0x00800000u) {
    u = __float_as_uint(x * 16777216.0f);
    off = m ? 0x38000000u - (24u << 20) : 0u;
  }
  if (m >= 0x7f800000u) off = 0x70000000u;              // infinity, NaN
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + off)), (int)(u << 29));
}

// one level's work decomposition for one kind of item
struct Decomp {
  const int *beg;              // [np+1] item prefix per patch (level-local)
  const int *blk_p0;           // [nblocks] first patch of each block
  int n, nblocks;
};

// Division by a level's constant h^2, correctly rounded without a divide: a
// double division is a chain of about nine dependent FP64 operations (556
// cycles on GB300, one operation takes 64).  r = RN(1/d) comes from the host.
// ops 1: d is a power of two, x r is exact.  ops 3: q = RN(x r), then
// RN(q + r RN(x - q d)), the last two fused -- the quotient step of Markstein
// (IBM J. Res. Dev. 34, 1990): correctly rounded if r is the correctly
// rounded reciprocal and q is within an ulp, which holds while |r d - 1| is
// below a quarter ulp of 1 (the host checks it per constant).  ops 5: the step
// twice; the first brings q within an ulp for any d.  Outside the exponent
// range [elo, elo + espan] an intermediate could leave the normal range: a
// true division there, and the signed zero of the first product for x = 0.
// A colour pass of a 15 x 11-based ragged level (660 cells): 4.1 us with
// divisions, 3.6 with this; the three-level ragged solve 4.23 -> 3.95 ms.
template <class T>
struct DivK {
  T d, r;
  int ops, kexp;               // kexp: what x / d adds to x's high word (ops 1)
  unsigned elo, espan;
};
using DivC = DivK<double>;

__device__ __forceinline__ unsigned exp_bits(double x) { return ((unsigned)__double2hiint(x) >> 20) & 0x7ffu; }
__device__ __forceinline__ bool is_zero(double x) {
  return (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) == 0u;
}
__device__ __forceinline__ unsigned exp_bits(float x) { return (__float_as_uint(x) >> 23) & 0xffu; }
__device__ __forceinline__ bool is_zero(float x) { return (__float_as_uint(x) << 1) == 0u; }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

__device__ __noinline__ double div_out_of_line(double x, double d) { return x / d; }
__device__ __noinline__ float div_out_of_line(float x, float d) { return x / d; }

// kPow2: the kernel's variant for levels where every constant is a power of
// two (ops 1), which carries none of the other code
template <bool kPow2, bool kInt = false>
__device__ __forceinline__ double div_c(double x, const DivC &D) {
  const double q0 = mul_on<kInt>(x, D.r);
  if (kPow2 || D.ops == 1) return q0;
  double q = __fma_rn(__fma_rn(-q0, D.d, x), D.r, q0);
  if (D.ops == 5) q = __fma_rn(__fma_rn(-q, D.d, x), D.r, q);
  if (exp_bits(x) - D.elo > D.espan) q = is_zero(x) ? q0 : div_out_of_line(x, D.d);
  return q;
}

// The face coefficients of an operator on a power-of-two level, scaled by the
// exact 1/h^2 on the integer pipe before they are used: (D 2^-k) dq ==
// (D dq) 2^-k in floating point, so the operator's two divisions fall away
// (relax_cell's packed operands rely on the same).  Coefficients whose scaled
// exponent could leave the normal range (faces_in false for any of a cell's)
// are multiplied instead.
template <int kN>
__device__ __forceinline__ bool faces_in(const double (&c)[kN], const DivC &D) {
  bool in = true;
#pragma unroll
  for (int i = 0; i < kN; ++i) in = in && exp_bits(c[i]) - D.elo <= D.espan;
  return in;
}
template <int kN>
__device__ __forceinline__ void scale_faces(double (&c)[kN], const DivC &D, bool in) {
#pragma unroll
  for (int i = 0; i < kN; ++i)
    c[i] = in ? __hiloint2double(__double2hiint(c[i]) + D.kexp, __double2loint(c[i])) : c[i] * D.r;
}

// The quotients of several values at once, the first kX by dx and the rest by
// dy: the steps of all of them overlap (an update's four were a chain of
// about 1,000 cycles, one after the other because each has its out-of-range
// branch), the range is looked at once, and the second step is taken if
// either constant wants it (it leaves a correct quotient as it is).
// Six passes of a tile: FP64 12 x 256 threads 10.3 us -> 8.5, FP32 9.2 -> 6.7
// (three steps and a range test for FP32, where a divide alone is as short);
// ragged three-level solve 2.86 -> 2.66 ms, ragged mixed solve 1.89 -> 1.78.
template <int kX, int kN, bool kInt, class T>
__device__ __forceinline__ void div_group(T (&x)[kN], const DivK<T> &dx, const DivK<T> &dy) {
  T q[kN];
  bool out = false;
#pragma unroll
  for (int i = 0; i < kN; ++i) {
    const DivK<T> &D = i < kX ? dx : dy;
    const T q0 = mul_on<kInt>(x[i], D.r);
    q[i] = fma_rn(fma_rn(-q0, D.d, x[i]), D.r, q0);
    out = out || exp_bits(x[i]) - D.elo > D.espan;
  }
  if (dx.ops == 5 || dy.ops == 5) {
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      const DivK<T> &D = i < kX ? dx : dy;
      q[i] = fma_rn(fma_rn(-q[i], D.d, x[i]), D.r, q[i]);
    }
  }
  if (out) {
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      const DivK<T> &D = i < kX ? dx : dy;
      if (exp_bits(x[i]) - D.elo > D.espan) q[i] = is_zero(x[i]) ? x[i] * D.r : div_out_of_line(x[i], D.d);
    }
  }
#pragma unroll
  for (int i = 0; i < kN; ++i) x[i] = q[i];
}

// one FP32 quotient
template <bool kPow2, bool kInt = false>
__device__ __forceinline__ float div_c(float x, const DivK<float> &D) { return x / D.d; }

struct LevelD {
  const PatchD *patches;       // this level's patches
  double hx, hy;
  DivC dx, dy;                 // division by hx^2, hy^2
  int pow2;                    // hx2 and hy2 are powers of two
  float fhx, fhy;              // FP32 copies for the correction cycle
  DivK<float> fdx, fdy;
};

// the level's cell sizes in the cycle's value type
template <class T, class D2> struct LevelH {
  T hx, hy;
  D2 dx, dy;                   // what div_c and div_group divide by
};
__device__ __forceinline__ LevelH<double, DivC> level_h(const LevelD &L, double) { return {L.hx, L.hy, L.dx, L.dy}; }
__device__ __forceinline__ LevelH<float, DivK<float>> level_h(const LevelD &L, float) {
  return {L.fhx, L.fhy, L.fdx, L.fdy};
}

// `b` is the block index within the decomposition
__device__ __forceinline__ int find_patch(const Decomp &D, int b, int g) {
  int p = __ldg(D.blk_p0 + b);
  while (g >= __ldg(D.beg + p + 1)) ++p;
  return p;
}

// op2d (ebKernels.m:13-25) at one cell from its face fluxes (kPow2: formed
// with scale_faces' coefficients)
template <bool kPow2, bool kInt = false>
__device__ __forceinline__ double op_flux(double feE, double feW, double fnN, double fnS, double cc, double q,
                                          const LevelD &L) {
  if (kPow2) return (-(feE - feW) - (fnN - fnS)) + mul_on<kInt>(cc, q);
  double d[2] = {-(feE - feW), fnN - fnS};
  div_group<1, 2, kInt>(d, L.dx, L.dy);
  return (d[0] - d[1]) + mul_on<kInt>(cc, q);
}

// the same from its values and (unscaled) coefficients
template <bool kPow2>
__device__ __forceinline__ double op_pre(double q, double qe, double qw, double qn, double qs, double dE, double dW,
                                         double dN, double dS, double cc, const LevelD &L) {
  const double feE = dE * (qe - q), feW = dW * (q - qw), fnN = dN * (qn - q), fnS = dS * (q - qs);
  if (kPow2) return (div_c<true>(-(feE - feW), L.dx) - div_c<true>(fnN - fnS, L.dy)) + cc * q;
  double d[2] = {-(feE - feW), fnN - fnS};
  div_group<1, 2, false>(d, L.dx, L.dy);
  return (d[0] - d[1]) + cc * q;
}

// the same at interior cell (li, lj) of a padded array
template <bool kPow2 = false>
__device__ __forceinline__ double op_cell_r(const double *__restrict__ Qa, int ldq, const double *__restrict__ DeW,
                                            const double *__restrict__ DnS, double cc, int mx, int li, int lj,
                                            const LevelD &L) {
  const int c = (li + 1) + (lj + 1) * ldq;
  return op_pre<kPow2>(Qa[c], Qa[c + 1], Qa[c - 1], Qa[c + ldq], Qa[c - ldq], DeW[(li + 1) + lj * (mx + 1)],
                DeW[li + lj * (mx + 1)], DnS[li + (lj + 1) * mx], DnS[li + lj * mx], cc, L);
}

// ---------------------------------------------------------------------------
// Ghost rules (EllipticBSAM/src/ebFillGhosts.m:17-94, ebInterpCf.m:36-154).
// The three ordered stages (coarse-fine interpolation, same-level copy,
// physical closure) are resolved on the host into one final rule per ghost
// cell.  Value rules read only interior cells, parent cells (the coarse
// window is read from the parent's Q, which is what the QC ring holds) or
// boundary data; a physical corner evaluates its two face-ghost rules
// itself, so a level's ghost frame is filled in one pass.
enum GhostType : int8_t {
  G_COPY = 0, G_QIF = 1, G_QIF_END = 2, G_LIF = 3, G_LIF_CORNER = 4,
  G_DIRICHLET = 5, G_NEUMANN = 6, G_RING = 7, G_PHYS_CORNER = 8
};

// A physical corner's two face rules resolved at upload, with the operand
// slots as a kernel holds them (GhostPrep): read through the items, one
// after the other, they kept the corner's warp 3 us behind every other.
struct __align__(16) GhostRule {
  int ty, a, b, c, d, e, la, lb, lc;
  int g, nb, x;                // boundary datum, Neumann side; rule 0: the corner's interior operand, 1: its stride
};
struct CornerRec {
  GhostRule r[2];
};

struct GhostItems {
  const int8_t *type;
  const int *dst, *a, *b, *c, *d, *e;   // a corner's d: its CornerRec
  const int *inst;             // instance per item (batches only, else null)
  const CornerRec *corner;
};

// the value of a COPY / QIF / QIF_END / LIF rule from its five operands
template <class T>
__device__ __forceinline__ T rule_value(int type, T qa, T qb, T qc, T qd, T qe) {
  const T A1 = T(-1.0 / 5.0), A2 = T(2.0 / 3.0), A3 = T(8.0 / 15.0);
  const T B1 = T(5.0 / 32.0), B2 = T(15.0 / 16.0), B3 = T(-3.0 / 32.0);
  const T c23 = T(2.0 / 3.0), c13 = T(1.0 / 3.0);
  switch (type) {
    case G_COPY: return qa;
    case G_QIF: return (A1 * qa + A2 * qb) + A3 * qc;
    case G_QIF_END: return (A1 * qa + A2 * qb) + A3 * ((B1 * qc + B2 * qd) + B3 * qe);
    default: return (c23 * qc + c23 * qa) - c13 * qb;   // G_LIF
  }
}

// A ghost item in two stages, so that every load it needs is in flight at
// once: ghost_prep reads the item's static indices and boundary value (before
// a kernel's programmatic-launch wait), ghost_apply requests all of its solution
// operands and its boundary value before it looks at the rule's kind, so
// the lanes of a warp that fill different kinds of ghosts wait for one round
// of loads together.  Operand slots a kind does not read repeat its first
// operand.
//
// GhostAlt: the operands of a level's ghost items for the fill that follows
// the restriction of the level above into it, fused into one launch with
// that restriction (k_restrict_fill).  A solution operand that the
// restriction overwrites (a cell under the finer level's footprint) is coded
// -1 - j, and the item forms its value itself from the four fine cells of
// entry j of `rt` with restrict_cell's arithmetic -- the value the
// restriction stores -- so the fill reads nothing the same launch writes.
struct GhostAlt {
  const int *a, *b, *c;        // operand slots (d and e are parent cells: never restricted)
  const int2 *rt;              // (first fine cell in Q, fine row stride)
  const CornerRec *corner;     // with these operands
  int sh;                      // where the finer level lives (FieldsT::lsh)
};

template <class T>
struct GhostPrep {
  int8_t ty;
  int dst, a, b, c, d, e;
  int la, lb, lc;              // GhostAlt: row stride of the four fine cells from a / b / c on, 0: a plain cell
  T g;                         // a physical rule's boundary part: 8/3 g or h g
};

__device__ __forceinline__ int ghost_cells(const GhostAlt *A, int code, int &ld) {
  ld = 0;
  if (code >= 0) return code;
  const int2 r = __ldg(A->rt + (-1 - code));
  ld = r.y;
  return r.x + A->sh;
}

template <class T, bool kAlt = false>
__device__ __forceinline__ GhostPrep<T> ghost_prep(const GhostItems &G, int i, int8_t ty, int dst, const T *bcg, T hx,
                                                   T hy, const GhostAlt *A = nullptr) {
  GhostPrep<T> P;
  P.ty = ty;
  P.dst = dst;
  P.la = P.lb = P.lc = 0;
  const int pa = __ldg(G.a + i);
  const bool ub = ty == G_QIF || ty == G_QIF_END || ty == G_LIF || ty == G_DIRICHLET;
  const bool uc = ty == G_QIF || ty == G_QIF_END || ty == G_LIF || ty == G_LIF_CORNER;
  const bool ue = ty == G_QIF_END;
  // slots the kind does not use repeat the item's plain first operand
  P.a = kAlt ? ghost_cells(A, __ldg(A->a + i), P.la) : pa;
  P.b = !ub ? pa : kAlt ? ghost_cells(A, __ldg(A->b + i), P.lb) : __ldg(G.b + i);
  P.c = !uc ? pa : kAlt ? ghost_cells(A, __ldg(A->c + i), P.lc) : __ldg(G.c + i);
  P.d = ue ? __ldg(G.d + i) : pa;            // parent cells: never restricted
  P.e = ue ? __ldg(G.e + i) : pa;
  P.g = T(0);
  if (ty == G_DIRICHLET) P.g = T(8.0 / 3.0) * __ldg(bcg + __ldg(G.e + i));
  else if (ty == G_NEUMANN) P.g = (__ldg(G.b + i) ? hy : hx) * __ldg(bcg + __ldg(G.e + i));
  return P;
}

// a corner's face rule from its record; x: the record's last word
template <class T, bool kAlt>
__device__ __forceinline__ GhostPrep<T> rule_prep(const GhostRule *R, const T *bcg, T hx, T hy, int sh, int &x) {
  const int4 *p = reinterpret_cast<const int4 *>(R);
  const int4 u = __ldg(p), v = __ldg(p + 1), w = __ldg(p + 2);
  GhostPrep<T> P;
  P.ty = (int8_t)u.x;
  P.dst = 0;
  P.la = kAlt ? v.z : 0;
  P.lb = kAlt ? v.w : 0;
  P.lc = kAlt ? w.x : 0;
  P.a = u.y + (P.la ? sh : 0);
  P.b = u.z + (P.lb ? sh : 0);
  P.c = u.w + (P.lc ? sh : 0);
  P.d = v.x;
  P.e = v.y;
  x = w.w;
  P.g = T(0);
  if (P.ty == G_DIRICHLET) P.g = T(8.0 / 3.0) * __ldg(bcg + w.y);
  else if (P.ty == G_NEUMANN) P.g = (w.z ? hy : hx) * __ldg(bcg + w.y);
  return P;
}

// an item as a fill kernel holds it across its programmatic-launch wait: a
// physical corner also holds its two face rules
template <class T>
struct GhostPre {
  GhostPrep<T> P, P1, P2;      // corner: P.c (P.lc) is the interior operand
};
template <class T, bool kAlt = false>
__device__ __forceinline__ GhostPre<T> ghost_pre(const GhostItems &G, int i, int8_t ty, int dst, const T *bcg, T hx,
                                                 T hy, const GhostAlt *A = nullptr) {
  GhostPre<T> X;
  if (ty == G_PHYS_CORNER) {
    const CornerRec *R = (kAlt ? A->corner : G.corner) + __ldg(G.d + i);
    const int sh = kAlt ? A->sh : 0;
    X.P.ty = ty;
    X.P.dst = dst;
    X.P1 = rule_prep<T, kAlt>(&R->r[0], bcg, hx, hy, sh, X.P.c);
    X.P2 = rule_prep<T, kAlt>(&R->r[1], bcg, hx, hy, sh, X.P.lc);
    if (!kAlt) X.P.lc = 0;
    if (X.P.lc) X.P.c += sh;
  } else {
    X.P = ghost_prep<T, kAlt>(G, i, ty, dst, bcg, hx, hy, A);
  }
  return X;
}

// a solution operand's cells: one, or (fused fills only) the four whose
// restriction it is
template <class T, bool kCG, bool kAlt>
struct GhostCells {
  T v[kAlt ? 4 : 1];
  __device__ __forceinline__ void load(const T *Q, int i, int ld) {
    v[0] = ld_sol<kCG>(Q + i);
    if (kAlt && ld) {
      v[kAlt ? 1 : 0] = ld_sol<kCG>(Q + i + 1);
      v[kAlt ? 2 : 0] = ld_sol<kCG>(Q + i + ld);
      v[kAlt ? 3 : 0] = ld_sol<kCG>(Q + i + ld + 1);
    }
  }
  __device__ __forceinline__ T value(int ld) const {
    if constexpr (kAlt) {
      const T r = T(0.25) * (((v[0] + v[1]) + v[2]) + v[3]);
      return ld ? r : v[0];
    }
    return v[0];
  }
};

// a ghost's value from its operands and boundary part (every kind but the
// ring refresh and the physical corner)
template <class T>
__device__ __forceinline__ T ghost_formula(int ty, T qa, T qb, T qc, T qd, T qe, T g) {
  const T c23 = T(2.0 / 3.0), c13 = T(1.0 / 3.0);
  switch (ty) {
    case G_LIF_CORNER: return c23 * qc + c13 * qa;
    case G_DIRICHLET: return (g - 2 * qa) + c13 * qb;
    case G_NEUMANN: return qa + g;
    default: return rule_value<T>(ty, qa, qb, qc, qd, qe);   // COPY, QIF, QIF_END, LIF
  }
}

// the same without a branch per kind, for the few lanes of a corner's warp
// that hold rules of different kinds: sums of two or three products by
// constants (by 1 where a kind has none, which is exact)
template <class T>
__device__ __forceinline__ T ghost_formula_flat(int ty, T qa, T qb, T qc, T qd, T qe, T g) {
  const T A1 = T(-1.0 / 5.0), A2 = T(2.0 / 3.0), A3 = T(8.0 / 15.0);
  const T B1 = T(5.0 / 32.0), B2 = T(15.0 / 16.0), B3 = T(-3.0 / 32.0);
  const T c23 = T(2.0 / 3.0), c13 = T(1.0 / 3.0);
  if (ty == G_QIF_END) qc = (B1 * qc + B2 * qd) + B3 * qe;
  T x = qa, y = qb, z = qc, cx = A1, cy = A2, cz = A3;       // QIF, QIF_END
  if (ty == G_LIF) { x = qc; y = qa; z = qb; cx = cy = c23; cz = -c13; }
  else if (ty == G_LIF_CORNER) { x = qc; y = qa; cx = c23; cy = c13; }
  else if (ty == G_DIRICHLET) { x = g; y = qa; z = qb; cx = 1; cy = -2; cz = c13; }
  else if (ty == G_NEUMANN) { y = g; cx = cy = 1; }
  const T two = cx * x + cy * y, three = two + cz * z;
  return ty == G_COPY ? qa : (ty == G_LIF_CORNER || ty == G_NEUMANN) ? two : three;
}

// the operands of a prepared item that is not a ring refresh or a corner,
// all requested before the first is used, and its value
template <class T, bool kCG, bool kAlt>
struct GhostVals {
  GhostCells<T, kCG, kAlt> a, b, c;
  T d, e;
  __device__ __forceinline__ void load(const GhostPrep<T> &P, const T *Q) {
    a.load(Q, P.a, P.la);
    b.load(Q, P.b, P.lb);
    c.load(Q, P.c, P.lc);
    d = ld_sol<kCG>(Q + P.d);
    e = ld_sol<kCG>(Q + P.e);
  }
  template <bool kFlat = false>
  __device__ __forceinline__ T value(const GhostPrep<T> &P) const {
    T qa = a.v[0], qb = b.v[0], qc = c.v[0];
    if (kAlt && (P.la | P.lb | P.lc)) {      // the three restrictions side by side
      qa = a.value(P.la);
      qb = b.value(P.lb);
      qc = c.value(P.lc);
    }
    return kFlat ? ghost_formula_flat<T>(P.ty, qa, qb, qc, d, e, P.g) : ghost_formula<T>(P.ty, qa, qb, qc, d, e, P.g);
  }
};

// A level's own fill where the level lives at Q + sh: operands inside the
// level's range [lo, lo + n) of Q and the ghosts move by sh, parent cells
// (and a ring refresh's) do not.  kZero: parent cells hold 0 (k_restrict_fill).
struct GhostHome {
  int lo, n, sh;
};
template <class T, bool kZero>
__device__ __forceinline__ void ghost_apply_home(const GhostPre<T> &X, T *Q, T *QC, const GhostHome &M, bool zero) {
  auto op = [&](int j) -> T {
    if ((unsigned)(j - M.lo) < (unsigned)M.n) return Q[j + M.sh];
    return kZero && zero ? T(0) : Q[j];
  };
  if (X.P.ty == G_RING) {
    QC[X.P.dst] = Q[X.P.a];
    return;
  }
  // a corner: (face ghost 1 + face ghost 2) - interior, the face ghosts
  // evaluated by their own final rules (ebFillGhosts.m:84-89 reads them after
  // stage 3)
  if (X.P.ty == G_PHYS_CORNER) {
    const GhostPrep<T> &R = X.P1, &S = X.P2;
    const T ra = op(R.a), rb = op(R.b), rc = op(R.c), rd = op(R.d), re = op(R.e);
    const T sa = op(S.a), sb = op(S.b), sc = op(S.c), sd = op(S.d), se = op(S.e), in = op(X.P.c);
    Q[X.P.dst + M.sh] = (ghost_formula_flat<T>(R.ty, ra, rb, rc, rd, re, R.g) +
                         ghost_formula_flat<T>(S.ty, sa, sb, sc, sd, se, S.g)) - in;
    return;
  }
  const GhostPrep<T> &R = X.P;
  Q[R.dst + M.sh] = ghost_formula<T>(R.ty, op(R.a), op(R.b), op(R.c), op(R.d), op(R.e), R.g);
}

template <class T, bool kCG = false, bool kAlt = false>
__device__ __forceinline__ void ghost_apply(const GhostPre<T> &X, T *Q, T *QC) {
  if (X.P.ty == G_RING) {
    QC[X.P.dst] = ld_sol<kCG>(Q + X.P.a);
    return;
  }
  GhostVals<T, kCG, kAlt> V;
  if (X.P.ty == G_PHYS_CORNER) {
    GhostVals<T, kCG, kAlt> W;
    GhostCells<T, kCG, kAlt> C;
    V.load(X.P1, Q);
    W.load(X.P2, Q);
    C.load(Q, X.P.c, X.P.lc);
    Q[X.P.dst] = (V.template value<true>(X.P1) + W.template value<true>(X.P2)) - C.value(X.P.lc);
    return;
  }
  V.load(X.P, Q);
  Q[X.P.dst] = V.value(X.P);
}

// kT threads per block: kBlock, or 64 on a level whose kBlock grid leaves
// SMs idle
template <class T, int kT = kBlock>
__global__ void __launch_bounds__(kT) k_ghost(GhostItems G, int off, int n, T *__restrict__ Q, T *__restrict__ QC,
                                              const T *__restrict__ bcg, double hx_, double hy_,
                                              const int *__restrict__ active, const int *__restrict__ inst_nlev,
                                              int need, GhostHome M) {
  const int t = blockIdx.x * kT + threadIdx.x;
  const int i = off + t;
  // a converged instance of a batch stays frozen; a fill that follows the
  // restriction from level `need` skips the instances without that level
  // (their own V-cycle starts below it)
  const int inst = (t < n && G.inst) ? G.inst[i] : -1;
  const bool skip = t >= n || (inst >= 0 && (!active[inst] || inst_nlev[inst] < need));
  GhostPre<T> X;
  if (!skip) X = ghost_pre<T>(G, i, G.type[i], G.dst[i], bcg, T(hx_), T(hy_));
  chain_wait();
  if (skip) return;
  ghost_apply_home<T, false>(X, Q, QC, M, false);
}

// Ghost fills of several levels in one launch: span s holds the items
// [off[s], off[s] + beg[s+1] - beg[s]) of a level with cell sizes hx[s],
// hy[s], and launch item t belongs to the span with beg[s] <= t < beg[s+1].
// The host groups levels none of which reads a ghost cell that another level
// of the launch writes.
constexpr int kMaxSpans = 16;
struct GhostSpans {
  int off[kMaxSpans], beg[kMaxSpans + 1];
  double hx[kMaxSpans], hy[kMaxSpans];
  int n;
};

template <class T, int kT = kBlock>
__global__ void __launch_bounds__(kT) k_ghost_spans(GhostItems G, GhostSpans S, T *__restrict__ Q,
                                                    T *__restrict__ QC, const T *__restrict__ bcg,
                                                    const int *__restrict__ active) {
  const int t = blockIdx.x * kT + threadIdx.x;
  int off = S.off[0], b = 0, tot = 0;
  double hx = S.hx[0], hy = S.hy[0];
#pragma unroll
  for (int j = 1; j <= kMaxSpans; ++j) {
    if (j == S.n) tot = S.beg[j];
    if (j < kMaxSpans && j < S.n && t >= S.beg[j]) {
      off = S.off[j];
      b = S.beg[j];
      hx = S.hx[j];
      hy = S.hy[j];
    }
  }
  const bool in = t < tot;
  const int i = off + (t - b);
  const int inst = (in && G.inst) ? G.inst[i] : -1;
  const bool skip = !in || (inst >= 0 && !active[inst]);
  GhostPre<T> X;
  if (!skip) X = ghost_pre<T>(G, i, G.type[i], G.dst[i], bcg, T(hx), T(hy));
  chain_wait();
  if (skip) return;
  ghost_apply<T>(X, Q, QC);
}

// ---------------------------------------------------------------------------
// relax2d (EllipticBSAM/src/ebKernels.m:37-95): one colour of the red-black
// Gauss-Seidel sweep over all patches of a level, one thread per cell of
// the colour.  The colour cells of each patch are cut into chunks of
// kChunk that never straddle two patches; a chunk record carries everything
// a thread needs about its patch, so one load precedes the data loads.
// Partial physical ghosts ((8/3)g + (1/3)u_2 Dirichlet, h g Neumann) are
// formed in registers, the u_1 coupling being folded into InvDiagS.  The
// reference refills every ghost after each colour (ebRelaxLevel.m:36); with
// `fresh` set, a boundary thread instead evaluates its neighbour ghost's
// rule (stored inline per perimeter cell): every rule of an internal face
// reads only cells of the other colour (final after the previous pass),
// parent cells, or the reading cell itself (pre-update), so the value equals
// the refilled ghost bit for bit.  The first pass of a relaxation reads the
// ghosts as the last fill left them, as the reference does.
constexpr int kChunk = 64;

struct RelaxChunk {           // host record (packing of the operands)
  int q_off, c_off, dew_off, dns_off;
  int bcg_off, pe_off, mx, my;
  int par0, s0, n, inst;     // first colour-cell index in the patch, cells in the chunk, instance
  int bc[4];
};

// the chunk as the smoother kernels read it: three 16-byte words (three
// vector loads, ten registers); flags holds the W, E, S, N boundary codes in
// 2-bit fields and par0 in bit 8
struct __align__(16) RelaxChunkD {
  int q_off, c_off, bcg_off, pe_off;
  int mx, my, s0, n;
  int inst, flags, pad0, pad1;
};

// how a smoother chunk learns that its instance is frozen: kActNone, one
// instance (always live while a V-cycle runs); kActChunk, the per-chunk flag
// array k_solve_step keeps (a batch's instances' chunks are contiguous
// per level)
enum { kActNone = 0, kActChunk = 1 };

__device__ __forceinline__ int chunk_bc(int flags, int side) { return (flags >> (2 * side)) & 3; }
__device__ __forceinline__ int chunk_par0(int flags) { return (flags >> 8) & 1; }

// one ghost rule, inline (perimeter table): 32 bytes, two vector loads.  The
// operand slots a rule does not use repeat its first operand (set at
// upload), so all five can be read whatever the rule's kind.
struct __align__(16) Rule {
  int type, a, b, c, d, e, pad0, pad1;
};

// Every operand is requested before the rule's kind is looked at: the lanes
// of a warp that evaluate different kinds of rules then wait for one round of
// loads together, instead of one dependent round per kind in turn (the
// divergent branches would otherwise serialise their load latencies).
template <class T, bool kCG = false>
__device__ __forceinline__ T eval_inline(const Rule &R, const T *Q) {
  const T qa = ld_sol<kCG>(Q + R.a), qb = ld_sol<kCG>(Q + R.b), qc = ld_sol<kCG>(Q + R.c);
  const T qd = ld_sol<kCG>(Q + R.d), qe = ld_sol<kCG>(Q + R.e);
  return rule_value<T>(R.type, qa, qb, qc, qd, qe);
}

// The smoother's operands per chunk and colour, packed at upload: for chunk
// ch and colour m, five rows of kChunk values -- dE, dW, dN, dS (pre-scaled
// by 1/h^2 on power-of-two levels) and InvDiagS -- one per colour cell of
// the chunk, so a warp reads each operand as one contiguous row instead of
// every other value of the reference's arrays.
constexpr int kPackRows = 5;

// a static table row (never written while kernels run) brought into L1
// before the programmatic-launch wait; the read after the wait then hits L1
// without holding the row in registers across the wait
template <class R>
__device__ __forceinline__ void prefetch_l1(const R *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
  asm volatile("prefetch.global.L1 [%0];" ::"l"((const char *)(p + 1) - 1));
}

// Builds the packed operands of one level's chunks on the device from the
// reference-layout DeW, DnS and InvDiagS (one thread per chunk, colour and
// slot; slots past a chunk's cell count are zero).  `scale` multiplies the
// face coefficients by the exact 1/h^2 of a power-of-two level (ix, iy), the
// same product the relaxation's pre-scaled form relies on.
__global__ void __launch_bounds__(kBlock) k_pack(const RelaxChunk *__restrict__ ch, int nch,
                                                 const double *__restrict__ DeW, const double *__restrict__ DnS,
                                                 const double *__restrict__ ID, double ix, double iy, int scale,
                                                 double *__restrict__ pack) {
  const int64_t w = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  if (w >= (int64_t)nch * 2 * kChunk) return;
  const int c = (int)(w / (2 * kChunk)), m = (int)((w / kChunk) & 1), t = (int)(w % kChunk);
  const RelaxChunk R = ch[c];
  double *o = pack + ((size_t)c * 2 + m) * (kPackRows * kChunk) + t;
  if (t >= R.n) {
#pragma unroll
    for (int r = 0; r < kPackRows; ++r) o[r * kChunk] = 0.0;
    return;
  }
  const int s = R.s0 + t, half = R.mx >> 1;
  const int lj = s / half;
  const int li = 2 * (s - lj * half) + ((m + lj + R.par0) & 1);
  double e = DeW[R.dew_off + (li + 1) + lj * (R.mx + 1)], wv = DeW[R.dew_off + li + lj * (R.mx + 1)];
  double n = DnS[R.dns_off + li + (lj + 1) * R.mx], sv = DnS[R.dns_off + li + lj * R.mx];
  if (scale) {
    e = e * ix;
    wv = wv * ix;
    n = n * iy;
    sv = sv * iy;
  }
  o[0] = e;
  o[kChunk] = wv;
  o[2 * kChunk] = n;
  o[3 * kChunk] = sv;
  o[4 * kChunk] = ID[R.c_off + li + lj * R.mx];
}

// One colour-cell update in three stages, so that a persistent block can
// overlap them across chunk groups (k_relax_p): issue (the chunk record, its
// frozen flag and the packed operands), derive (the cell's position, its
// boundary data and ghost rules, all static), update (solution loads, ghost
// values, the candidate and its store).  relax_cell runs the three in order.
template <class T>
struct CellState {
  RelaxChunkD R;
  T dE, dW, dN, dS, idg, gx, gy;
  int q_off, c, cc, ldq, code, rx, ry;   // code: kx | ky << 2 | sx << 4 | sy << 5
  bool live;
};

// the chunk record, its frozen flag and the packed operands are indexed by
// the chunk alone: record and flag are requested together, the operands (a
// chunk's pack rows hold kChunk entries whatever its cell count) as soon as
// the small, cached flag says the chunk is live, so they are in flight with
// the record and a frozen chunk reads nothing else
template <class T>
__device__ __forceinline__ void cell_issue(const RelaxChunkD *__restrict__ chunks, int nchunks,
                                           const T *__restrict__ pack, int m, const uint8_t *__restrict__ cact,
                                           int amode, int ch, int tc, CellState<T> &S) {
  const bool okc = ch < nchunks;
  S.live = okc;
  S.dE = S.dW = S.dN = S.dS = S.idg = T(0);
  if (okc) {
    S.R = chunks[ch];
    if (amode == kActChunk) S.live = cact[ch] != 0;
  }
  if (S.live) {
    const T *__restrict__ pk = pack + (size_t)(ch * 2 + m) * (kPackRows * kChunk) + tc;
    S.dE = __ldg(pk);
    S.dW = __ldg(pk + kChunk);
    S.dN = __ldg(pk + 2 * kChunk);
    S.dS = __ldg(pk + 3 * kChunk);
    S.idg = __ldg(pk + 4 * kChunk);
  }
}

template <class T>
__device__ __forceinline__ void cell_derive(const FieldsT<T> &f, const Rule *__restrict__ perim, int m, int fresh,
                                            int tc, CellState<T> &S) {
  if (!S.live || tc >= S.R.n) {
    S.live = false;
    return;
  }
  const RelaxChunkD &R = S.R;
  const int s = R.s0 + tc;
  const int mx = R.mx, my = R.my, half = mx >> 1;
  const int lj = s / half;
  const int li = 2 * (s - lj * half) + ((m + lj + chunk_par0(R.flags)) & 1);
  S.ldq = mx + 2;
  S.c = (li + 1) + (lj + 1) * S.ldq;
  S.cc = R.c_off + li + lj * mx;
  S.q_off = R.q_off;
  // static boundary data and ghost rules; a cell touches at most one x side
  // (W or E) and one y side (S or N): kind 0 interior neighbour, 1
  // Dirichlet, 2 Neumann, 3 ghost rule
  const T *__restrict__ g4 = f.bcg + R.bcg_off;
  int kx = 0, ky = 0, sx = 0, sy = 0;       // sx: 0 west 1 east; sy: 0 south 1 north
  S.gx = S.gy = T(0);
  S.rx = S.ry = 0;                          // ghost rule indices (perimeter table)
  if (li == 0 || li == mx - 1) {
    sx = (li == 0) ? 0 : 1;
    const int bc = chunk_bc(R.flags, sx);   // a shift, not an indexed (local-memory) array
    if (bc) { kx = bc; S.gx = __ldg(g4 + sx * my + lj); }
    else if (fresh) { kx = 3; S.rx = R.pe_off + sx * my + lj; prefetch_l1(perim + S.rx); }
  }
  if (lj == 0 || lj == my - 1) {
    sy = (lj == 0) ? 0 : 1;
    const int bc = chunk_bc(R.flags, 2 + sy);
    if (bc) { ky = bc; S.gy = __ldg(g4 + 2 * my + sy * mx + li); }
    else if (fresh) { ky = 3; S.ry = R.pe_off + 2 * my + sy * mx + li; prefetch_l1(perim + S.ry); }
  }
  S.code = kx | (ky << 2) | (sx << 4) | (sy << 5);
}

template <class T, bool kPow2, bool kCG>
__device__ __forceinline__ void cell_update(const LevelD &L, const FieldsT<T> &f, const Rule *__restrict__ perim,
                                            T omega, int unit_omega, const CellState<T> &S) {
  if (!S.live) return;
  const T c83 = T(8.0 / 3.0), c13 = T(1.0 / 3.0);
  const auto H = level_h(L, T(0));
  const int c = S.c, ldq = S.ldq;
  const int kx = S.code & 3, ky = (S.code >> 2) & 3, sx = (S.code >> 4) & 1, sy = (S.code >> 5) & 1;
  T *__restrict__ Q = f.Q + S.q_off;
  T qe = ld_sol<kCG>(Q + c + 1), qw = ld_sol<kCG>(Q + c - 1), qn = ld_sol<kCG>(Q + c + ldq), qs = ld_sol<kCG>(Q + c - ldq);
  T t = f.F[S.cc];
  // the operands of the neighbour ghost's rule are requested with the
  // solution loads, before any value is formed, so lanes with different kinds
  // of ghosts wait for a single round of loads.  A lane holds one rule's
  // operands: a patch-corner cell with rules on both sides (x and y) forms
  // its y-side ghost in a second round.
  const bool rx = kx == 3, ry = ky == 3;
  T o0 = T(0), o1 = T(0), o2 = T(0), o3 = T(0), o4 = T(0);
  int rt = 0;
  if (rx || ry) {
    const Rule R = perim[rx ? S.rx : S.ry];
    rt = R.type;
    o0 = ld_sol<kCG>(f.Q + R.a); o1 = ld_sol<kCG>(f.Q + R.b); o2 = ld_sol<kCG>(f.Q + R.c);
    o3 = ld_sol<kCG>(f.Q + R.d); o4 = ld_sol<kCG>(f.Q + R.e);
  }
  // a partial Dirichlet ghost reads the interior neighbour across the cell,
  // which is the opposite neighbour already loaded
  if (kx > 0) {
    T v;
    if (kx == 1) v = c83 * S.gx + c13 * (sx ? qw : qe);
    else if (kx == 2) v = H.hx * S.gx;
    else v = rule_value<T>(rt, o0, o1, o2, o3, o4);
    if (sx) qe = v; else qw = v;
  }
  if (ky > 0) {
    T v;
    if (ky == 1) v = c83 * S.gy + c13 * (sy ? qs : qn);
    else if (ky == 2) v = H.hy * S.gy;
    else if (rx) v = eval_inline<T, kCG>(perim[S.ry], f.Q);
    else v = rule_value<T>(rt, o0, o1, o2, o3, o4);
    if (sy) qn = v; else qs = v;
  }
  // kPow2: the coefficients arrive pre-scaled by the exact 1/h^2 (a power of
  // two), and (q D) 2^-k == q (D 2^-k) in floating point, so one product
  // per neighbour gives the reference's (q D)/h^2 bit for bit
  if (kPow2) {
    t = t + qe * S.dE;
    t = t + qw * S.dW;
    t = t + qn * S.dN;
    t = t + qs * S.dS;
  } else {
    T d[4] = {qe * S.dE, qw * S.dW, qn * S.dN, qs * S.dS};
    div_group<2, 4, false>(d, H.dx, H.dy);
    t = (((t + d[0]) + d[1]) + d[2]) + d[3];
  }
  t = t * S.idg;
  if (unit_omega) Q[c] = t;
  else Q[c] = omega * t + (1 - omega) * ld_sol<kCG>(Q + c);
}

// one colour-cell update of chunk ch (thread tc of the chunk); kChain: the
// grid kernel's programmatic-launch wait sits between the static stages and
// the first read of the solution
template <class T, bool kPow2, bool kChain, bool kCG = false>
__device__ __forceinline__ void relax_cell(const LevelD &L, const RelaxChunkD *__restrict__ chunks, int nchunks,
                                           const FieldsT<T> &f, const T *__restrict__ pack,
                                           const Rule *__restrict__ perim, int m, T omega, int unit_omega, int fresh,
                                           const uint8_t *__restrict__ cact, int amode, int ch, int tc) {
  CellState<T> S;
  cell_issue<T>(chunks, nchunks, pack, m, cact, amode, ch, tc, S);
  cell_derive<T>(f, perim, m, fresh, tc, S);
  if (kChain) chain_wait();
  cell_update<T, kPow2, kCG>(L, f, perim, omega, unit_omega, S);
}

// Persistent form of one colour pass: a grid of resident blocks walks the
// level's chunk groups (kBlock / kChunk chunks each) with a grid stride;
// while a block updates one group it has the next group's chunk records and
// operands in flight, and derives that group's static data after the
// update.  The arithmetic of every update is relax_cell's.
template <class T, bool kPow2>
__global__ void __launch_bounds__(kBlock) k_relax_p(LevelD L, const RelaxChunkD *__restrict__ chunks, int nchunks,
                                                    FieldsT<T> f, const T *__restrict__ pack,
                                                    const Rule *__restrict__ perim, int m, T omega, int unit_omega,
                                                    int fresh, const uint8_t *__restrict__ cact, int amode) {
  constexpr int cpb = kBlock / kChunk;
  const int sub = threadIdx.x / kChunk, tc = threadIdx.x & (kChunk - 1);
  const int ngroups = (nchunks + cpb - 1) / cpb;
  int g = blockIdx.x;
  CellState<T> cur, nxt;
  cell_issue<T>(chunks, nchunks, pack, m, cact, amode, g * cpb + sub, tc, cur);
  cell_derive<T>(f, perim, m, fresh, tc, cur);
  chain_wait();
  while (g < ngroups) {
    const int gn = g + (int)gridDim.x;
    cell_issue<T>(chunks, nchunks, pack, m, cact, amode, gn * cpb + sub, tc, nxt);
    cell_update<T, kPow2, false>(L, f, perim, omega, unit_omega, cur);
    cell_derive<T>(f, perim, m, fresh, tc, nxt);
    cur = nxt;
    g = gn;
  }
}

// Coarsened smoother: each thread updates kN colour cells of its chunk
// (cells t, t + kChunk/kN, ...), in three phases -- static loads of every
// cell, then the solution loads of every cell, then every update -- so the
// loads of a thread's cells are in flight together.  Within a colour pass no
// cell reads another cell of its colour (a ghost rule reads cells of the
// other colour, parent cells or the reading cell itself, before its update),
// so loading all before storing any changes nothing: the arithmetic of each
// update is relax_cell's.
template <class T, bool kPow2, int kN>
__global__ void __launch_bounds__(kBlock) k_relax_n(LevelD L, const RelaxChunkD *__restrict__ chunks, int nchunks,
                                                    FieldsT<T> f, const T *__restrict__ pack,
                                                    const Rule *__restrict__ perim, int m, T omega, int unit_omega,
                                                    int fresh, const uint8_t *__restrict__ cact, int amode) {
  constexpr int tpc = kChunk / kN;                    // threads per chunk
  const int ch = blockIdx.x * (kBlock / tpc) + threadIdx.x / tpc;
  const int t0 = threadIdx.x % tpc;
  // chunk record and packed operands requested together (as relax_cell)
  const bool okc = ch < nchunks;
  RelaxChunkD R;
  bool live = okc;
  T dE[kN], dW[kN], dN[kN], dS[kN], idg[kN], gx[kN], gy[kN];
  if (okc) {
    R = chunks[ch];
    if (amode == kActChunk) live = cact[ch] != 0;
  }
  if (live) {
    const T *__restrict__ pk0 = pack + (size_t)(ch * 2 + m) * (kPackRows * kChunk) + t0;
#pragma unroll
    for (int u = 0; u < kN; ++u) {
      const T *__restrict__ pk = pk0 + u * tpc;
      dE[u] = __ldg(pk);
      dW[u] = __ldg(pk + kChunk);
      dN[u] = __ldg(pk + 2 * kChunk);
      dS[u] = __ldg(pk + 3 * kChunk);
      idg[u] = __ldg(pk + 4 * kChunk);
    }
  }
  if (!live || t0 >= R.n) {
    chain_wait();
    return;
  }
  const int mx = R.mx, my = R.my, half = mx >> 1, ldq = mx + 2;
  const T *__restrict__ g4 = f.bcg + R.bcg_off;
  bool on[kN];
  int c[kN], cc[kN], code[kN], rxi[kN], ryi[kN];    // code: kx | ky << 2 | sx << 4 | sy << 5
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    const int tc = t0 + u * tpc;
    on[u] = tc < R.n;
    const int s = R.s0 + (on[u] ? tc : 0);
    const int lj = s / half;
    const int li = 2 * (s - lj * half) + ((m + lj + chunk_par0(R.flags)) & 1);
    c[u] = (li + 1) + (lj + 1) * ldq;
    cc[u] = R.c_off + li + lj * mx;
    int kx = 0, ky = 0, sx = 0, sy = 0;
    gx[u] = 0;
    gy[u] = 0;
    rxi[u] = 0;
    ryi[u] = 0;
    if (li == 0 || li == mx - 1) {
      sx = (li == 0) ? 0 : 1;
      const int bc = chunk_bc(R.flags, sx);
      if (bc) { kx = bc; gx[u] = __ldg(g4 + sx * my + lj); }
      else if (fresh) { kx = 3; rxi[u] = R.pe_off + sx * my + lj; prefetch_l1(perim + rxi[u]); }
    }
    if (lj == 0 || lj == my - 1) {
      sy = (lj == 0) ? 0 : 1;
      const int bc = chunk_bc(R.flags, 2 + sy);
      if (bc) { ky = bc; gy[u] = __ldg(g4 + 2 * my + sy * mx + li); }
      else if (fresh) { ky = 3; ryi[u] = R.pe_off + 2 * my + sy * mx + li; prefetch_l1(perim + ryi[u]); }
    }
    code[u] = kx | (ky << 2) | (sx << 4) | (sy << 5);
  }
  chain_wait();
  const T c83 = T(8.0 / 3.0), c13 = T(1.0 / 3.0);
  const auto H = level_h(L, T(0));
  T *__restrict__ Q = f.Q + R.q_off;
  T qe[kN], qw[kN], qn[kN], qs[kN], fv[kN], qc[kN];
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    const int cu = c[u];
    qe[u] = Q[cu + 1];
    qw[u] = Q[cu - 1];
    qn[u] = Q[cu + ldq];
    qs[u] = Q[cu - ldq];
    qc[u] = unit_omega ? T(0) : Q[cu];
    fv[u] = f.F[cc[u]];
  }
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    const int kx = code[u] & 3, ky = (code[u] >> 2) & 3, sx = (code[u] >> 4) & 1, sy = (code[u] >> 5) & 1;
    const int cu = c[u];
    if (kx > 0) {
      T v;
      if (kx == 1) v = c83 * gx[u] + c13 * Q[sx ? cu - 1 : cu + 1];
      else if (kx == 2) v = H.hx * gx[u];
      else v = eval_inline<T>(perim[rxi[u]], f.Q);
      if (sx) qe[u] = v; else qw[u] = v;
    }
    if (ky > 0) {
      T v;
      if (ky == 1) v = c83 * gy[u] + c13 * Q[sy ? cu - ldq : cu + ldq];
      else if (ky == 2) v = H.hy * gy[u];
      else v = eval_inline<T>(perim[ryi[u]], f.Q);
      if (sy) qn[u] = v; else qs[u] = v;
    }
  }
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    if (!on[u]) continue;
    T t = fv[u];
    if (kPow2) {
      t = t + qe[u] * dE[u];
      t = t + qw[u] * dW[u];
      t = t + qn[u] * dN[u];
      t = t + qs[u] * dS[u];
    } else {
      t = t + div_c<false>(qe[u] * dE[u], H.dx);
      t = t + div_c<false>(qw[u] * dW[u], H.dx);
      t = t + div_c<false>(qn[u] * dN[u], H.dy);
      t = t + div_c<false>(qs[u] * dS[u], H.dy);
    }
    t = t * idg[u];
    if (unit_omega) Q[c[u]] = t;
    else Q[c[u]] = omega * t + (1 - omega) * qc[u];
  }
}

// One colour pass, one thread per colour cell.  The ghosts that a pass forms
// from rules are few (a coarse-fine side's cells), but nearly every warp holds
// one, and a warp pays for a rule's FP64 operations whatever the number of
// its lanes that want them.  So the lanes put their rules on the block's list
// before the programmatic-launch wait, the block's first threads evaluate it
// together after the wait, and the updates read the values from shared
// memory; a side that copies a sibling's cell reads that cell as its
// neighbour.  The arithmetic is relax_cell's.  Starfish, FP64, us per pass:
// 114,756 cells 3.97 -> 3.22, 379,536 cells 7.25 -> 5.90 (FP64 work alone 3.2;
// the rest is the rules', the launch's and the loads').
//
// kT threads per block: kBlock, or fewer on a level whose kBlock grid would
// leave SMs idle -- an SM issues about two FP64 operations per clock, so a
// block's FP64 work is spread over more SMs.
// kInt: four of the five products on the integer pipe (mul_int_pipe)
template <class T, bool kPow2, int kT = kBlock, bool kInt = false>
__global__ void __launch_bounds__(kT, (sizeof(T) == 4 ? 8 : 5) * (kBlock / kT))
    k_relax(LevelD L, const RelaxChunkD *__restrict__ chunks, int nchunks, FieldsT<T> f, const T *__restrict__ pack,
            const Rule *__restrict__ perim, int m, T omega, int unit_omega, int fresh,
            const uint8_t *__restrict__ cact, int amode) {
  if constexpr (sizeof(T) == 4) {            // little arithmetic: each lane evaluates its own rule (2.74 against 3.08 us)
    relax_cell<T, kPow2, true>(L, chunks, nchunks, f, pack, perim, m, omega, unit_omega, fresh, cact, amode,
                               blockIdx.x * (kT / kChunk) + threadIdx.x / kChunk, threadIdx.x & (kChunk - 1));
    return;
  }
  constexpr int kJobs = kT / 2;              // rules beyond these are evaluated by their own lanes
  __shared__ int4 s_ab[kJobs];               // type, a, b, c
  __shared__ int2 s_de[kJobs];
  __shared__ T s_val[kJobs];
  __shared__ int s_n;
  const int t = threadIdx.x, tc = t & (kChunk - 1);
  if (t == 0) s_n = 0;
  CellState<T> S;
  cell_issue<T>(chunks, nchunks, pack, m, cact, amode, blockIdx.x * (kT / kChunk) + t / kChunk, tc, S);
  const bool live = S.live && tc < S.R.n;
  const T c83 = T(8.0 / 3.0), c13 = T(1.0 / 3.0);
  const auto H = level_h(L, T(0));
  int c = 0, ne = 0, nw = 0, nn = 0, ns = 0, cc = 0, code = 0, jx = -1, jy = -1, rx = 0, ry = 0;
  T gx = T(0), gy = T(0);
  if (fresh) __syncthreads();
  if (live) {
    const RelaxChunkD &R = S.R;
    const int s = R.s0 + tc, mx = R.mx, my = R.my, half = mx >> 1, ldq = mx + 2;
    const int lj = s / half;
    const int li = 2 * (s - lj * half) + ((m + lj + chunk_par0(R.flags)) & 1);
    c = R.q_off + (li + 1) + (lj + 1) * ldq;
    cc = R.c_off + li + lj * mx;
    ne = c + 1;
    nw = c - 1;
    nn = c + ldq;
    ns = c - ldq;
    // a cell touches at most one x side and one y side.  code: physical kind
    // (1 Dirichlet, 2 Neumann) of the x side in bits 0-1, of the y side in
    // 2-3; bit 4: the x side is east, bit 5: the y side is north
    const T *__restrict__ g4 = f.bcg + R.bcg_off;
    auto rule = [&](int pe, int &nb, int &job) {
      const int4 r0 = __ldg(reinterpret_cast<const int4 *>(perim + pe));
      if (r0.x == G_COPY) {
        nb = r0.y;
        return;
      }
      job = atomicAdd(&s_n, 1);
      if (job < kJobs) {
        s_ab[job] = r0;
        s_de[job] = __ldg(reinterpret_cast<const int2 *>(perim + pe) + 2);
      }
    };
    if (li == 0 || li == mx - 1) {
      const int e = li != 0, bc = chunk_bc(R.flags, e), at = e * my + lj;
      code |= bc | (e << 4);
      if (bc) gx = bc == 1 ? c83 * __ldg(g4 + at) : H.hx * __ldg(g4 + at);
      else if (fresh) rule(rx = R.pe_off + at, e ? ne : nw, jx);
    }
    if (lj == 0 || lj == my - 1) {
      const int e = lj != 0, bc = chunk_bc(R.flags, 2 + e), at = 2 * my + e * mx + li;
      code |= (bc << 2) | (e << 5);
      if (bc) gy = bc == 1 ? c83 * __ldg(g4 + at) : H.hy * __ldg(g4 + at);
      else if (fresh) rule(ry = R.pe_off + at, e ? nn : ns, jy);
    }
  }
  if (fresh) __syncthreads();
  chain_wait();
  const T *Q = f.Q;
  T qe = T(0), qw = T(0), qn = T(0), qs = T(0), v = T(0);
  if (live) {
    qe = Q[ne];
    qw = Q[nw];
    qn = Q[nn];
    qs = Q[ns];
    v = f.F[cc];
  }
  if (fresh) {
    const int n = s_n;
    if (n > 0) {
      if (t < min(n, kJobs)) {
        const int4 r = s_ab[t];
        const int2 de = s_de[t];
        s_val[t] = rule_value<T>(r.x, Q[r.y], Q[r.z], Q[r.w], Q[de.x], Q[de.y]);
      }
      __syncthreads();
      if (jx >= 0) {
        const T g = jx < kJobs ? s_val[jx] : eval_inline<T>(perim[rx], Q);
        if (code & 16) qe = g; else qw = g;
      }
      if (jy >= 0) {
        const T g = jy < kJobs ? s_val[jy] : eval_inline<T>(perim[ry], Q);
        if (code & 32) qn = g; else qs = g;
      }
    }
  }
  if (!live) return;
  if (code & 15) {
    // a partial Dirichlet ghost reads the neighbour across the cell
    const int kx = code & 3, ky = (code >> 2) & 3;
    if (kx) {
      const T g = kx == 1 ? gx + c13 * ((code & 16) ? qw : qe) : gx;
      if (code & 16) qe = g; else qw = g;
    }
    if (ky) {
      const T g = ky == 1 ? gy + c13 * ((code & 32) ? qs : qn) : gy;
      if (code & 32) qn = g; else qs = g;
    }
  }
  if (kPow2) {
    v = v + mul_on<kInt>(qe, S.dE);
    v = v + mul_on<kInt>(qw, S.dW);
    v = v + mul_on<kInt>(qn, S.dN);
    v = v + mul_on<kInt>(qs, S.dS);
  } else {
    T d[4] = {mul_on<kInt>(qe, S.dE), mul_on<kInt>(qw, S.dW), mul_on<kInt>(qn, S.dN), mul_on<kInt>(qs, S.dS)};
    div_group<2, 4, kInt>(d, H.dx, H.dy);
    v = (((v + d[0]) + d[1]) + d[2]) + d[3];
  }
  v = v * S.idg;
  if (unit_omega) f.Q[c] = v;
  else f.Q[c] = omega * v + (1 - omega) * f.Q[c];
}
// A small level's whole relaxation in one launch: one thread-block cluster
// runs every colour pass of the `nsweeps` sweeps over all the level's chunks
// (cluster-strided), with a cluster barrier (release / acquire) between
// passes, then the level's ghost fill (launch_fill's items).  Each pass and
// the fill compute exactly what the separate launches compute -- the same
// relax_cell and ghost_apply code -- with the solution read from L2.  One
// cluster holds every block, so the barrier orders the whole level; no
// thread leaves the loop early, so every barrier is reached by all.
constexpr int kClusterBlock = 1024;

template <class T, bool kPow2>
__global__ void __launch_bounds__(kClusterBlock, 1)
    k_relax_cluster(LevelD L, const RelaxChunkD *__restrict__ chunks, int nchunks, FieldsT<T> f,
                    const T *__restrict__ pack, const Rule *__restrict__ perim, T omega, int unit_omega, int nsweeps,
                    int first_fresh, const uint8_t *__restrict__ cact, int amode, GhostItems G, int g_off, int g_n,
                    double hx_, double hy_) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int nth = (int)cl.num_blocks() * kClusterBlock;
  const int tid = (int)cl.block_rank() * kClusterBlock + threadIdx.x;
  chain_wait();
  const int nitems = nchunks * kChunk;
  for (int s = 0; s < nsweeps; ++s)
    for (int m = 0; m < 2; ++m) {
      const int fresh = (first_fresh || s > 0 || m > 0) ? 1 : 0;
      for (int w = tid; w < nitems; w += nth)
        relax_cell<T, kPow2, false, true>(L, chunks, nchunks, f, pack, perim, m, omega, unit_omega, fresh, cact,
                                          amode, w / kChunk, w % kChunk);
      cl.sync();
    }
  for (int t = tid; t < g_n; t += nth) {
    const int i = g_off + t;
    const int inst = G.inst ? G.inst[i] : -1;
    if (inst >= 0 && !f.active[inst]) continue;
    ghost_apply<T, true>(ghost_pre<T>(G, i, G.type[i], G.dst[i], f.bcg, T(hx_), T(hy_)), f.Q, f.QC);
  }
}


// A small level's relaxation with its solution in distributed shared
// memory.  One thread-block cluster copies the level's Q range [q0, q0 + qn)
// into the shared memory of its CTAs (CTA r holds elements [r S, (r + 1) S),
// S = 2^shift), runs every colour pass of the `nsweeps` sweeps with the
// neighbour and ghost-rule loads and the stores going to the owning CTA's
// shared memory, a cluster barrier between passes, then the level's ghost
// fill (g_n > 0), and copies the range back.  Each thread owns one chunk
// slot (the same colour-cell position of both colours) and loads its static
// data once, before the passes: the packed operands, boundary data, force,
// and its ghost rule with the rule's parent-cell operands (cells outside the
// range do not change during the relaxation), so a pass waits only for the
// shared-memory loads of the solution.  The arithmetic of every update and
// ghost is relax_cell's and ghost_apply's, so the results are the chained
// passes' bit for bit.  The host uses it on levels with at most one colour
// cell per thread and colour; the dynamic shared memory is the slice and
// ten values per thread (the rules' parent-cell operands).
constexpr int kDsmBlock = 512;   // threads per CTA of k_relax_dsm

template <class T>
struct DsmRange {
  int q0, qn, shift;
  uint32_t base;          // shared-window address of this CTA's slice
};

template <class T>
__device__ __forceinline__ uint32_t dsm_addr(const DsmRange<T> &D, int rel) {
  const uint32_t la = D.base + (uint32_t)(rel & ((1 << D.shift) - 1)) * (uint32_t)sizeof(T);
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(la), "r"((uint32_t)rel >> D.shift));
  return ra;
}
__device__ __forceinline__ double dsm_ld(uint32_t a, double) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float dsm_ld(uint32_t a, float) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void dsm_st(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void dsm_st(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// a solution value: from the cluster's copy inside the range, else from
// global memory (static while the kernel runs)
template <class T>
__device__ __forceinline__ T dsm_sol(const DsmRange<T> &D, const T *Q, int n) {
  const int rel = n - D.q0;
  if ((unsigned)rel < (unsigned)D.qn) return dsm_ld(dsm_addr(D, rel), T(0));
  return __ldg(Q + n);
}

template <class T>
__device__ __forceinline__ T dsm_rule(const DsmRange<T> &D, const Rule &R, const T *Q) {
  const T qa = dsm_sol(D, Q, R.a), qb = dsm_sol(D, Q, R.b), qc = dsm_sol(D, Q, R.c);
  const T qd = dsm_sol(D, Q, R.d), qe = dsm_sol(D, Q, R.e);
  return rule_value<T>(R.type, qa, qb, qc, qd, qe);
}

// one colour cell's static data for k_relax_dsm; its ghost rule's operands
// outside the range (static) wait in the CTA's shared memory at `ov`
template <class T>
struct DsmCell {
  T dE, dW, dN, dS, idg, gx, gy, fv;
  uint32_t oa[5];        // per rule operand: its shared-window address (inside the range) or global index
  int c, ldq, code, cc, rx, ry, rtype, omask;   // c relative to q0; omask bit i: operand i inside the range
  bool live;
};

// the static part, before the programmatic-launch wait: the cell's packed
// operands and boundary data, and its ghost rule -- kind, and per operand
// the shared-window address (inside the range, mask bit set) or the global
// index whose value the bind loads
template <class T>
__device__ __forceinline__ void dsm_cell_static(const RelaxChunkD *__restrict__ chunks, int nchunks,
                                                const T *__restrict__ pack, const FieldsT<T> &f,
                                                const Rule *__restrict__ perim, const uint8_t *__restrict__ cact,
                                                int amode, int ch, int tc, int m, const DsmRange<T> &D,
                                                DsmCell<T> &X) {
  CellState<T> S;
  cell_issue<T>(chunks, nchunks, pack, m, cact, amode, ch, tc, S);
  cell_derive<T>(f, perim, m, 1, tc, S);
  X.live = S.live;
  X.dE = S.dE; X.dW = S.dW; X.dN = S.dN; X.dS = S.dS; X.idg = S.idg; X.gx = S.gx; X.gy = S.gy;
  X.c = S.q_off + S.c - D.q0;
  X.ldq = S.ldq;
  X.code = S.code;
  X.cc = S.cc;
  X.rx = S.rx;
  X.ry = S.ry;
  X.rtype = 0;
  X.omask = 0;
  const int kx = X.code & 3, ky = (X.code >> 2) & 3;
  if (X.live && (kx == 3 || ky == 3)) {
    const Rule R = perim[kx == 3 ? X.rx : X.ry];
    X.rtype = R.type;
    const int op[5] = {R.a, R.b, R.c, R.d, R.e};
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int rel = op[i] - D.q0;
      if ((unsigned)rel < (unsigned)D.qn) {
        X.omask |= 1 << i;
        X.oa[i] = dsm_addr(D, rel);
      } else {
        X.oa[i] = (uint32_t)op[i];
      }
    }
  }
}

// the dynamic part of the set-up, after the wait: the force and the values
// of the rule's operands outside the range (into ov)
template <class T>
__device__ __forceinline__ void dsm_cell_bind(const FieldsT<T> &f, T *ov, DsmCell<T> &X) {
  if (!X.live) return;
  X.fv = f.F[X.cc];
  const int kx = X.code & 3, ky = (X.code >> 2) & 3;
  if (kx == 3 || ky == 3) {
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (!((X.omask >> i) & 1)) ov[i] = f.Q[(int)X.oa[i]];
  }
}

// cell_update from the static data and the cluster's copy of the solution
template <class T, bool kPow2>
__device__ __forceinline__ void dsm_cell_update(const LevelD &L, const FieldsT<T> &f, const Rule *__restrict__ perim,
                                                T omega, int unit_omega, int fresh, const DsmCell<T> &X,
                                                const T *ov, const DsmRange<T> &D) {
  if (!X.live) return;
  const T c83 = T(8.0 / 3.0), c13 = T(1.0 / 3.0);
  const auto H = level_h(L, T(0));
  const int ldq = X.ldq, c = X.c;
  int kx = X.code & 3, ky = (X.code >> 2) & 3;
  const int sx = (X.code >> 4) & 1, sy = (X.code >> 5) & 1;
  if (!fresh) {               // the stored ghosts, as the last fill left them
    if (kx == 3) kx = 0;
    if (ky == 3) ky = 0;
  }
  T qe = dsm_ld(dsm_addr(D, c + 1), T(0)), qw = dsm_ld(dsm_addr(D, c - 1), T(0));
  T qn = dsm_ld(dsm_addr(D, c + ldq), T(0)), qs = dsm_ld(dsm_addr(D, c - ldq), T(0));
  T t = X.fv;
  const bool rx = kx == 3, ry = ky == 3;
  T o[5];
#pragma unroll
  for (int i = 0; i < 5; ++i)
    o[i] = (rx || ry) ? (((X.omask >> i) & 1) ? dsm_ld(X.oa[i], T(0)) : ov[i]) : T(0);
  if (kx > 0) {
    T v;
    if (kx == 1) v = c83 * X.gx + c13 * (sx ? qw : qe);
    else if (kx == 2) v = H.hx * X.gx;
    else v = rule_value<T>(X.rtype, o[0], o[1], o[2], o[3], o[4]);
    if (sx) qe = v; else qw = v;
  }
  if (ky > 0) {
    T v;
    if (ky == 1) v = c83 * X.gy + c13 * (sy ? qs : qn);
    else if (ky == 2) v = H.hy * X.gy;
    else if (rx) v = dsm_rule<T>(D, perim[X.ry], f.Q);
    else v = rule_value<T>(X.rtype, o[0], o[1], o[2], o[3], o[4]);
    if (sy) qn = v; else qs = v;
  }
  if (kPow2) {
    t = t + qe * X.dE;
    t = t + qw * X.dW;
    t = t + qn * X.dN;
    t = t + qs * X.dS;
  } else {
    t = t + div_c<false>(qe * X.dE, H.dx);
    t = t + div_c<false>(qw * X.dW, H.dx);
    t = t + div_c<false>(qn * X.dN, H.dy);
    t = t + div_c<false>(qs * X.dS, H.dy);
  }
  t = t * X.idg;
  const uint32_t ac = dsm_addr(D, c);
  if (unit_omega) dsm_st(ac, t);
  else dsm_st(ac, omega * t + (1 - omega) * dsm_ld(ac, T(0)));
}

// one ghost rule's value from the cluster's copy
template <class T>
__device__ __forceinline__ T ghost_eval_dsm(const GhostItems &G, int i, const FieldsT<T> &f, T hx, T hy,
                                            const DsmRange<T> &D) {
  const GhostPrep<T> P = ghost_prep<T>(G, i, G.type[i], 0, f.bcg, hx, hy);
  const T qa = dsm_sol(D, f.Q, P.a), qb = dsm_sol(D, f.Q, P.b), qc = dsm_sol(D, f.Q, P.c);
  const T qd = dsm_sol(D, f.Q, P.d), qe = dsm_sol(D, f.Q, P.e);
  return ghost_formula<T>(P.ty, qa, qb, qc, qd, qe, P.g);
}

template <class T, bool kPow2>
__global__ void __launch_bounds__(kDsmBlock, 1)
    k_relax_dsm(LevelD L, const RelaxChunkD *__restrict__ chunks, int nchunks, FieldsT<T> f,
                const T *__restrict__ pack, const Rule *__restrict__ perim, T omega, int unit_omega, int nsweeps,
                int first_fresh, const uint8_t *__restrict__ cact, int amode, GhostItems G, int g_off, int g_n,
                double hx_, double hy_, int q0, int qn, int shift) {
  namespace cg = cooperative_groups;
  constexpr int kB = kDsmBlock;
  extern __shared__ __align__(16) unsigned char dsm_raw[];
  T *slice = reinterpret_cast<T *>(dsm_raw);
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), r = (int)cl.block_rank();
  const int S = 1 << shift;
  const DsmRange<T> D{q0, qn, shift, (uint32_t)__cvta_generic_to_shared(slice)};
  // this thread's chunk slot: CTA r takes a contiguous run of chunks
  const int cpc = (nchunks + C - 1) / C;
  const int w = r * cpc * kChunk + (int)threadIdx.x;
  const bool mine = (int)threadIdx.x < cpc * kChunk && w < nchunks * kChunk;
  // parent-cell operands of this thread's two rules, after the slice
  T *ov0 = slice + S + 10 * (int)threadIdx.x, *ov1 = ov0 + 5;
  DsmCell<T> X0, X1;
  X0.live = X1.live = false;
  if (mine) {
    dsm_cell_static<T>(chunks, nchunks, pack, f, perim, cact, amode, w / kChunk, w % kChunk, 0, D, X0);
    dsm_cell_static<T>(chunks, nchunks, pack, f, perim, cact, amode, w / kChunk, w % kChunk, 1, D, X1);
  }
  chain_wait();
  const int e0 = r * S, e1 = min(qn, e0 + S);
  for (int e = e0 + (int)threadIdx.x; e < e1; e += kB) slice[e - e0] = f.Q[q0 + e];
  dsm_cell_bind<T>(f, ov0, X0);
  dsm_cell_bind<T>(f, ov1, X1);
  cl.sync();
  for (int s = 0; s < nsweeps; ++s) {
    dsm_cell_update<T, kPow2>(L, f, perim, omega, unit_omega, (first_fresh || s > 0) ? 1 : 0, X0, ov0, D);
    cl.sync();
    dsm_cell_update<T, kPow2>(L, f, perim, omega, unit_omega, 1, X1, ov1, D);
    cl.sync();
  }
  if (g_n > 0) {
    const int nth = C * kB, tid = r * kB + (int)threadIdx.x;
    const T hx = T(hx_), hy = T(hy_);
    for (int t = tid; t < g_n; t += nth) {
      const int i = g_off + t;
      const int inst = G.inst ? G.inst[i] : -1;
      if (inst >= 0 && !f.active[inst]) continue;
      const int8_t ty = G.type[i];
      const int dst = G.dst[i];
      if (ty == G_RING) {
        f.QC[dst] = dsm_sol(D, f.Q, G.a[i]);
        continue;
      }
      T v;
      if (ty == G_PHYS_CORNER) {
        const T v1 = ghost_eval_dsm<T>(G, G.a[i], f, hx, hy, D);
        const T v2 = ghost_eval_dsm<T>(G, G.b[i], f, hx, hy, D);
        v = (v1 + v2) - dsm_sol(D, f.Q, G.c[i]);
      } else {
        v = ghost_eval_dsm<T>(G, i, f, hx, hy, D);
      }
      dsm_st(dsm_addr(D, dst - q0), v);
    }
    cl.sync();
  }
  for (int e = e0 + (int)threadIdx.x; e < e1; e += kB) f.Q[q0 + e] = slice[e - e0];
}

// ---------------------------------------------------------------------------
// restrict2 (ebKernels.m:98-102) of each patch interior into its QC interior
// and, for 'restrict' (ebTransfer.m:10-33), into the parent's Q over the
// footprint.  One thread per coarse cell.
template <class T>
__device__ __forceinline__ T restrict_cell(const T *Q, int ldq, int ci, int cj) {
  const int c = (2 * ci + 1) + (2 * cj + 1) * ldq;
  return T(0.25) * (((Q[c] + Q[c + 1]) + Q[c + ldq]) + Q[c + ldq + 1]);
}

// one coarse cell of the restriction; kChain: the grid kernel's
// programmatic-launch wait sits between the static loads and the solution
// (every early exit executes it too)
template <class T, bool kChain>
__device__ __forceinline__ void restrict_item(const LevelD &L, const Decomp &D, const FieldsT<T> &f, int to_parent,
                                              int g) {
  if (g >= D.n) {
    if (kChain) chain_wait();
    return;
  }
  const int p = find_patch(D, g / kBlock, g);
  const PatchD &P = L.patches[p];
  if (!f.active[P.inst]) {
    if (kChain) chain_wait();
    return;
  }
  const int cmx = P.mx >> 1, q_off = P.q_off, ldq = P.mx + 2, qc_off = P.qc_off;
  const int s = g - __ldg(D.beg + p);
  const int cj = s / cmx, ci = s - cj * cmx;
  const int dst = to_parent ? __ldg(f.fp + 2 * (P.fp_off + s)) : 0;
  if (kChain) chain_wait();
  const T R = restrict_cell<T>(f.Q + q_off + f.lsh, ldq, ci, cj);
  f.QC[qc_off + (ci + 1) + (cj + 1) * (cmx + 2)] = R;
  if (to_parent) f.Q[dst] = R;
}

// kT threads per block: kBlock, or 64 on a level whose kBlock grid leaves
// SMs idle
template <class T, int kT = kBlock>
__global__ void __launch_bounds__(kT) k_restrict(LevelD L, Decomp D, FieldsT<T> f, int to_parent) {
  restrict_item<T, true>(L, D, f, to_parent, blockIdx.x * kT + threadIdx.x);
}

// The restriction of level k into QC and the parent (ebTransfer.m:10-33)
// and the ghost fill of the parent level that follows it (ebVcycle.m:27,
// ebTransfer.m:73-79) in one launch: blocks [0, nb_r) restrict, the rest
// fill level k-1 with the fused operands of GhostAlt (a fill operand under
// level k's footprint is restricted by the item itself), so no item reads a
// value another item of the launch writes.
//
// Optionally (f_n > 0) the launch also runs level k's own ghost fill that
// precedes the restriction (the closing fill of its pre-smoothing, or of the
// finest level's post-smoothing before the fill-down): blocks
// [nb_r, nb_r + nb_f) run those items as k_ghost does, its ring items only
// with f_ring.  The host allows it on a level whose fill reads no cell the
// restriction or the parent's fill writes, and whose ghost cells the
// parent's fill does not read.  In the FP32 correction cycle it runs on
// every level in the zero-parent form (f_zero): the correction starts at 0
// and level k-1 is first written by this very launch, so every parent-level
// operand of level k's pre-smoothing fill is 0, which the items use instead
// of reading cells the launch may be writing.
//
// Bound by latency: a launch was as long as the warp of its physical corners,
// whose two face rules were looked up one after the other and evaluated kind
// by kind (a ragged level's parent fill 6.2 us, every other warp done in 1.6);
// with CornerRec, ghost_formula_flat and the operands' restrictions side by
// side 4.2 us; FP64 levels of 1,000 to 6,000 cells 3.0-3.7 -> 2.5-3.1.  Three
// 256-thread blocks per SM: the operands of a fused fill would take 98
// registers and hold back the restriction's warps (batch of 64 20.3 ms, with
// 80 registers 19.5).
template <class T, int kT = kBlock>
__global__ void __launch_bounds__(kT, kT == kBlock ? 3 : 1) k_restrict_fill(LevelD L, Decomp D, FieldsT<T> f, int to_parent, int nb_r,
                                                     GhostItems G, GhostAlt A, int g_off, int g_n, double hx_,
                                                     double hy_, const int *__restrict__ active,
                                                     const int *__restrict__ inst_nlev, int need, int f_off, int f_n,
                                                     int nb_f, int f_ring, double fhx, double fhy, GhostHome M,
                                                     int f_zero) {
  if ((int)blockIdx.x < nb_r) {
    restrict_item<T, true>(L, D, f, to_parent, blockIdx.x * kT + threadIdx.x);
    return;
  }
  if ((int)blockIdx.x < nb_r + nb_f) {
    const int t = ((int)blockIdx.x - nb_r) * kT + threadIdx.x;
    const int i = f_off + t;
    const int inst = (t < f_n && G.inst) ? G.inst[i] : -1;
    const int8_t ty = t < f_n ? G.type[i] : G_COPY;
    const bool skip = t >= f_n || (inst >= 0 && !active[inst]) || (ty == G_RING && !f_ring);
    GhostPre<T> X;
    if (!skip) X = ghost_pre<T>(G, i, ty, G.dst[i], f.bcg, T(fhx), T(fhy));
    chain_wait();
    if (skip) return;
    ghost_apply_home<T, true>(X, f.Q, f.QC, M, f_zero != 0);
    return;
  }
  const int t = ((int)blockIdx.x - nb_r - nb_f) * kT + threadIdx.x;
  const int i = g_off + t;
  const int inst = (t < g_n && G.inst) ? G.inst[i] : -1;
  const bool skip = t >= g_n || (inst >= 0 && (!active[inst] || inst_nlev[inst] < need));
  GhostPre<T> X;
  if (!skip) X = ghost_pre<T, true>(G, i, G.type[i], G.dst[i], f.bcg, T(hx_), T(hy_), &A);
  chain_wait();
  if (skip) return;
  ghost_apply<T, false, true>(X, f.Q, f.QC);
}
// ---------------------------------------------------------------------------
// ebFaceCorrections (ebFaceCorrections.m:18-61): the correction of one coarse
// face.  Its operands' indices are resolved at upload: the fine cells either
// side of the two fine faces (a - b), the coarse values where the reference's
// QC holds them -- the outer (ring) cell in the parent's Q, the inner cell in
// QC's interior (`qc_inner` false) or recomputed as the restriction of its
// four fine cells (`qc_inner` true: the residual's refresh,
// ebCompResidual.m:32-38) -- and the three diffusivities.  The arithmetic is
// FP64 for either value type (the reflux of the mixed form stays FP64).
struct __align__(16) CorrRec {
  int a1, b1, a2, b2;          // fine cells (Q)
  int out, qc, in, ldq;        // parent's cell (Q), QC cell, first inner fine cell (Q) and its row stride
  int c1, c2, cf, yface;       // DeW or DnS twice, interface D; 1: a y face
};

// a record and its diffusivities, held across a programmatic-launch wait
struct CorrPre {
  CorrRec r;
  double d1, d2, cf;
};
template <class T>
__device__ __forceinline__ CorrPre corr_pre(const CorrRec *__restrict__ rec, const FieldsT<T> &f) {
  CorrPre X;
  const int4 *p = reinterpret_cast<const int4 *>(rec);
  const int4 u = __ldg(p), v = __ldg(p + 1), w = __ldg(p + 2);
  X.r = CorrRec{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w, w.x, w.y, w.z, w.w};
  const T *D = X.r.yface ? f.DnS : f.DeW;
  X.d1 = dbl(__ldg(D + X.r.c1));
  X.d2 = dbl(__ldg(D + X.r.c2));
  X.cf = dbl(__ldg(f.cfd + X.r.cf));
  return X;
}
template <bool kPow2, class T>
__device__ __forceinline__ double corr_value(const CorrPre &X, const FieldsT<T> &f, const LevelD &Lc, bool qc_inner) {
  const CorrRec &r = X.r;
  const T *Q = f.Q + f.lsh;
  const double out = dbl(f.Q[r.out]);
  double in;
  if (qc_inner) {
    const T *q = Q + r.in;
    in = dbl(T(0.25) * (((q[0] + q[1]) + q[r.ldq]) + q[r.ldq + 1]));
  } else {
    in = dbl(f.QC[r.qc]);
  }
  const double v = (X.d1 * (dbl(Q[r.a1]) - dbl(Q[r.b1])) + X.d2 * (dbl(Q[r.a2]) - dbl(Q[r.b2]))) + X.cf * (out - in);
  return div_c<kPow2>(v, r.yface ? Lc.dy : Lc.dx);
}

// gather-form corrections of one target coarse cell: contributions in the
// reference's order (fine patch ascending, faces W, E, S, N)
struct CorrCSR {
  const int *cell, *patch, *beg;
  const CorrRec *rec;
};

// a target's contributions, the first two (nearly all targets have no more)
// read before the programmatic-launch wait: with item, patch and index
// arithmetic after it the coarse loads of a 4-level hierarchy of 64^2 patches
// took 4.5-5 us each, now 3.4-4
struct CorrTarget {
  int beg, end;
  CorrPre x0, x1;
};
template <class T>
__device__ __forceinline__ CorrTarget corr_target(const CorrCSR &C, int t, const FieldsT<T> &f) {
  CorrTarget X;
  X.beg = __ldg(C.beg + t);
  X.end = __ldg(C.beg + t + 1);
  if (X.beg < X.end) X.x0 = corr_pre<T>(C.rec + X.beg, f);
  if (X.beg + 1 < X.end) X.x1 = corr_pre<T>(C.rec + X.beg + 1, f);
  return X;
}
template <bool kPow2, class T>
__device__ __forceinline__ double add_corrections(double v, const CorrTarget &X, const CorrCSR &C, const LevelD &Lc,
                                                  const FieldsT<T> &f, bool qc_inner) {
  if (X.beg >= X.end) return v;
  v = v + corr_value<kPow2>(X.x0, f, Lc, qc_inner);
  if (X.beg + 1 < X.end) v = v + corr_value<kPow2>(X.x1, f, Lc, qc_inner);
  for (int i = X.beg + 2; i < X.end; ++i) v = v + corr_value<kPow2>(corr_pre<T>(C.rec + i, f), f, Lc, qc_inner);
  return v;
}

// ---------------------------------------------------------------------------
// FAS coarse load of level k (ebVcycle.m:28-29): one launch with three block
// ranges --
//   [0, nb_ring)            QC ring <- parent Q      (ebTransfer.m:35-55)
//   [nb_ring, +D.nblocks)   F_parent = restrict2(F - op(Q)) + op_c(QC, parent
//                           coefficients) over the footprint (ebCoarseLoad.m:17-32,
//                           ebParentCoeffs.m), the four fine residuals summed in
//                           restrict2 order (1,1), (2,1), (1,2), (2,2)
//   [.., +nb_tgt)           F_target = F_target + corrections (ebCoarseLoad.m:37-45)
// QC ring values are read from the parent's Q through the window table, so
// the three ranges are independent.
// the three item kinds of the coarse load (kChain as restrict_item)
template <class T, bool kChain>
__device__ __forceinline__ void load_ring_item(const FieldsT<T> &f, const int *__restrict__ ring,
                                               const int *__restrict__ ring_inst, int ring_off, int n_ring, int t) {
  int src = 0, dst = 0;
  bool on = t < n_ring && (!ring_inst || f.active[__ldg(ring_inst + ring_off + t)]);
  if (on) {
    src = __ldg(ring + 2 * (ring_off + t));
    dst = __ldg(ring + 2 * (ring_off + t) + 1);
  }
  if (kChain) chain_wait();
  if (on) f.QC[dst] = f.Q[src];
}

template <class T, bool kPow2, bool kInt, bool kChain>
__device__ __forceinline__ void load_fp_item(const LevelD &L, const LevelD &Lc, const Decomp &D, const FieldsT<T> &f,
                                             int g) {
  if (g >= D.n) {
    if (kChain) chain_wait();
    return;
  }
  const int p = find_patch(D, g / kBlock, g);
  const PatchD &P = L.patches[p];
  if (!f.active[P.inst]) {
    if (kChain) chain_wait();
    return;
  }
  const int mx = P.mx, cmx = mx >> 1, cmy = P.my >> 1, ldq = mx + 2;
  const int s = g - __ldg(D.beg + p);
  const int cj = s / cmx, ci = s - cj * cmx;
  const int q_off = P.q_off, c_off = P.c_off, qc_off = P.qc_off;
  // static operands: the 2 x 3 x-faces and 3 x 2 y-faces of the four fine
  // cells, their reaction coefficients, and the coarse operator's
  const T *DeW = f.DeW + P.dew_off + 2 * ci + 2 * cj * (mx + 1), *DnS = f.DnS + P.dns_off + 2 * ci + 2 * cj * mx;
  const T *CC = f.CC + c_off + 2 * ci + 2 * cj * mx;
  double dx[6], dy[6], cf[4];
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    dx[t] = dbl(__ldg(DeW + t % 3 + (t / 3) * (mx + 1)));
    dy[t] = dbl(__ldg(DnS + t % 2 + (t / 2) * mx));
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) cf[t] = dbl(__ldg(CC + (t & 1) + (t >> 1) * mx));
  const int ldc = cmx + 2;
  const int *win = f.win + P.win_off;
  const int w = (ci + 1) + (cj + 1) * ldc;
  // ring neighbours of the coarse operator come from the parent's Q
  const int se = (ci == cmx - 1) ? __ldg(win + w + 1) : -1;
  const int sw = (ci == 0) ? __ldg(win + w - 1) : -1;
  const int sn = (cj == cmy - 1) ? __ldg(win + w + ldc) : -1;
  const int ss = (cj == 0) ? __ldg(win + w - ldc) : -1;
  const T *PDeW = f.pcoef + P.pc_off;
  const T *PDnS = PDeW + (cmx + 1) * cmy;
  const T *PCC = PDnS + cmx * (cmy + 1);
  double px[2] = {dbl(__ldg(PDeW + ci + cj * (cmx + 1))), dbl(__ldg(PDeW + (ci + 1) + cj * (cmx + 1)))};
  double py[2] = {dbl(__ldg(PDnS + ci + cj * cmx)), dbl(__ldg(PDnS + ci + (cj + 1) * cmx))};
  const double pC = dbl(__ldg(PCC + s));
  const int dst = __ldg(f.fp + 2 * (P.fp_off + s) + 1);
  if (kPow2) {
    if (faces_in(dx, L.dx) && faces_in(dy, L.dy) && faces_in(px, Lc.dx) && faces_in(py, Lc.dy)) {
      scale_faces(dx, L.dx, true);
      scale_faces(dy, L.dy, true);
      scale_faces(px, Lc.dx, true);
      scale_faces(py, Lc.dy, true);
    } else {
      scale_faces(dx, L.dx, false);
      scale_faces(dy, L.dy, false);
      scale_faces(px, Lc.dx, false);
      scale_faces(py, Lc.dy, false);
    }
  }
  if (kChain) chain_wait();
  // the four fine cells and their eight neighbours: v[j][i], corners unused
  const T *Qp = f.Q + q_off + f.lsh + 2 * ci + 2 * cj * ldq;
  double v[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[j][i] = (i == 0 || i == 3) && (j == 0 || j == 3) ? 0.0 : dbl(Qp[i + j * ldq]);
  // each face's flux once: the neighbour across it forms the same one
  double fx[2][3], fy[3][2], rf[4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      fx[j][i] = mul_on<kInt>(dx[3 * j + i], v[j + 1][i + 1] - v[j + 1][i]);
      fy[i][j] = mul_on<kInt>(dy[2 * i + j], v[i + 1][j + 1] - v[i][j + 1]);
    }
  const T *Fp = f.F + c_off + 2 * ci + 2 * cj * mx;
  double dd[8];                // the four cells' flux differences
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int i = t & 1, j = t >> 1;
    dd[t] = -(fx[j][i + 1] - fx[j][i]);
    dd[4 + t] = fy[j + 1][i] - fy[j][i];
  }
  if (!kPow2) div_group<4, 8, kInt>(dd, L.dx, L.dy);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int i = t & 1, j = t >> 1;
    rf[t] = dbl(Fp[i + j * mx]) - ((dd[t] - dd[4 + t]) + mul_on<kInt>(cf[t], v[j + 1][i + 1]));
  }
  const double rr = 0.25 * (((rf[0] + rf[1]) + rf[2]) + rf[3]);
  const T *QC = f.QC + qc_off;
  const double q = dbl(QC[w]);
  const double qe = dbl(se >= 0 ? f.Q[se] : QC[w + 1]);
  const double qw = dbl(sw >= 0 ? f.Q[sw] : QC[w - 1]);
  const double qn = dbl(sn >= 0 ? f.Q[sn] : QC[w + ldc]);
  const double qs = dbl(ss >= 0 ? f.Q[ss] : QC[w - ldc]);
  const double lc = op_flux<kPow2>(px[1] * (qe - q), px[0] * (q - qw), py[1] * (qn - q), py[0] * (q - qs), pC, q, Lc);
  f.F[dst] = T(rr + lc);
}

// The same with a footprint cell on four lanes, one fine cell each, which
// also form one flux each of the coarse operator, for levels whose launch
// waits for one thread's 84 to 110 operations (a warp's FP64 operation takes
// its SM 19 cycles whatever else waits) and for that much straight-line code:
// 40 to 50 operations here.  A level of 1,000 to 6,000 cells 3.4 to 4.0 us ->
// 2.2 to 3.0, ragged (with divisions) mixed 6.6 -> 4.7.
template <class T, bool kPow2, bool kChain>
__device__ __forceinline__ void load_fp_quad(const LevelD &L, const LevelD &Lc, const Decomp &D, const FieldsT<T> &f,
                                             int g4) {
  const int g = g4 >> 2, t = g4 & 3;
  if (g >= D.n) {
    if (kChain) chain_wait();
    return;
  }
  const int p = find_patch(D, g / kBlock, g);
  const PatchD &P = L.patches[p];
  if (!f.active[P.inst]) {
    if (kChain) chain_wait();
    return;
  }
  const int mx = P.mx, cmx = mx >> 1, cmy = P.my >> 1, ldq = mx + 2;
  const int s = g - __ldg(D.beg + p);
  const int cj = s / cmx, ci = s - cj * cmx;
  const int li = 2 * ci + (t & 1), lj = 2 * cj + (t >> 1), cell = P.c_off + li + lj * mx;
  const T *DeW = f.DeW + P.dew_off + li + lj * (mx + 1), *DnS = f.DnS + P.dns_off + li + lj * mx;
  double dx[2] = {dbl(__ldg(DeW + 1)), dbl(__ldg(DeW))}, dy[2] = {dbl(__ldg(DnS + mx)), dbl(__ldg(DnS))};
  const double cf = dbl(__ldg(f.CC + cell));
  // the lane's face of the coarse cell, E W N S: its neighbour, ring cells
  // from the parent's Q
  const int ldc = cmx + 2, w = (ci + 1) + (cj + 1) * ldc, step = (t & 1 ? -1 : 1) * (t < 2 ? 1 : ldc);
  const bool edge = t == 0 ? ci == cmx - 1 : t == 1 ? ci == 0 : t == 2 ? cj == cmy - 1 : cj == 0;
  const T *nb = edge ? f.Q + __ldg(f.win + P.win_off + w + step) : f.QC + P.qc_off + w + step;
  const T *PDeW = f.pcoef + P.pc_off, *PDnS = PDeW + (cmx + 1) * cmy, *PCC = PDnS + cmx * (cmy + 1);
  double pd[1] = {dbl(__ldg(t < 2 ? PDeW + ci + (t == 0) + cj * (cmx + 1) : PDnS + ci + (cj + (t == 2)) * cmx))};
  const double pC = dbl(__ldg(PCC + s));
  const int dst = __ldg(f.fp + 2 * (P.fp_off + s) + 1);
  if (kPow2) {
    const DivC &Dp = t < 2 ? Lc.dx : Lc.dy;
    scale_faces(dx, L.dx, faces_in(dx, L.dx));
    scale_faces(dy, L.dy, faces_in(dy, L.dy));
    scale_faces(pd, Dp, faces_in(pd, Dp));
  }
  if (kChain) chain_wait();
  const T *Q = f.Q + P.q_off + f.lsh + (li + 1) + (lj + 1) * ldq;
  const double v = dbl(Q[0]), ve = dbl(Q[1]), vw = dbl(Q[-1]), vn = dbl(Q[ldq]), vs = dbl(Q[-ldq]);
  const double F = dbl(f.F[cell]), q = dbl(f.QC[P.qc_off + w]), qb = dbl(*nb);
  const double fl = pd[0] * ((t & 1) ? q - qb : qb - q);
  const double rf = F - op_flux<kPow2>(dx[0] * (ve - v), dx[1] * (v - vw), dy[0] * (vn - v), dy[1] * (v - vs), cf, v, L);
  const unsigned quad = 0xfu << (threadIdx.x & 28);
  auto from = [&](double x, int l) { return __shfl_sync(quad, x, l, 4); };
  const double rr = 0.25 * (((from(rf, 0) + from(rf, 1)) + from(rf, 2)) + from(rf, 3));
  const double lc = op_flux<kPow2>(from(fl, 0), from(fl, 1), from(fl, 2), from(fl, 3), pC, q, Lc);
  if (t == 0) f.F[dst] = T(rr + lc);
}

template <class T, bool kPow2, bool kChain>
__device__ __forceinline__ void load_corr_item(const LevelD &L, const LevelD &Lc, const FieldsT<T> &f, const CorrCSR &C,
                                               int n_tgt, int t) {
  const bool on = t < n_tgt && f.active[Lc.patches[C.patch[t]].inst];
  const int cell = on ? C.cell[t] : 0;
  CorrTarget X;
  double base = 0.0;
  if (on) {
    X = corr_target<T>(C, t, f);
    if (sizeof(T) == sizeof(double)) base = f.FTrue[cell];
  }
  if (kChain) chain_wait();
  if (!on) return;
  // FP64: the target's F before its corrections is FTrue (the value the
  // reference's per-cycle reset F = FTrue leaves there), so the V-cycle does
  // not depend on a reset of F before it; the correction cycle of the mixed
  // form adds to its own right-hand side
  if (sizeof(T) != sizeof(double)) base = dbl(f.F[cell]);
  f.F[cell] = T(add_corrections<kPow2, T>(base, X, C, Lc, f, false));
}

// kT threads per block (kBlock, or 64 on a level whose kBlock grid leaves
// SMs idle: a footprint cell is 45 to 85 FP64 operations, and an SM issues
// about two per clock); the decomposition's per-block patch table is kBlock-based
template <class T, bool kPow2, bool kInt, int kT = kBlock, bool kQuad = false>
__global__ void __launch_bounds__(kT) k_load(LevelD L, LevelD Lc, Decomp D, FieldsT<T> f, const int *__restrict__ ring,
                                             const int *__restrict__ ring_inst, int ring_off, int n_ring, CorrCSR C,
                                             int n_tgt) {
  const int nb_ring = (n_ring + kT - 1) / kT;
  const int nb_fp = ((kQuad ? 4 : 1) * D.n + kT - 1) / kT;
  int b = blockIdx.x;
  if (b < nb_ring) {
    load_ring_item<T, true>(f, ring, ring_inst, ring_off, n_ring, b * kT + threadIdx.x);
    return;
  }
  b -= nb_ring;
  if (b < nb_fp) {
    if constexpr (kQuad) load_fp_quad<T, kPow2, true>(L, Lc, D, f, b * kT + threadIdx.x);
    else load_fp_item<T, kPow2, kInt, true>(L, Lc, D, f, b * kT + threadIdx.x);
    return;
  }
  b -= nb_fp;
  load_corr_item<T, kPow2, true>(L, Lc, f, C, n_tgt, b * kT + threadIdx.x);
}

// ---------------------------------------------------------------------------
// prolongBilin (ebKernels.m:105-123) of the parent window: 'correct'
// (ebTransfer.m:57-71) adds P(W - QC) to the interior; mode 0 writes P(W)
// (new-level initial guess, ebAddLevel.m:26-31).  One thread per coarse cell
// writes its four fine cells.
//
// The FP64 form is bound by the FP64 pipe: 32 operations a coarse cell.
// Levels large enough to keep the pipe busy (kInt) form the five products and
// the four sixteenths on the integer pipe: 1,048,576 fine cells 18.2 us ->
// 15.3, 379,536 in patches 8.5 -> 7.5.  (Threads of two or four coarse cells
// that share their differences took 13.2 us on the former, but 4.7 to 8
// instead of 3.3 on small levels.)
template <class T, bool kChain, bool kInt>
__device__ __forceinline__ void prolong_item(const LevelD &L, const Decomp &D, const FieldsT<T> &f, int correct,
                                             int g) {
  if (g >= D.n) {
    if (kChain) chain_wait();
    return;
  }
  const int p = find_patch(D, g / kBlock, g);
  const PatchD &P = L.patches[p];
  if (!f.active[P.inst]) {   // frozen instance, or an instance whose level k is not new
    if (kChain) chain_wait();
    return;
  }
  const int cm = P.mx >> 1;
  const int s = g - __ldg(D.beg + p);
  const int b = s / cm, a = s - b * cm;
  const int ldw = cm + 2;
  const int *win = f.win + P.win_off;
  int src[3][3];
#pragma unroll
  for (int dj = 0; dj < 3; ++dj)
#pragma unroll
    for (int di = 0; di < 3; ++di) src[dj][di] = __ldg(win + (a + di) + (b + dj) * ldw);
  const int qc_off = P.qc_off, q_off = P.q_off, ldq = P.mx + 2;
  if (kChain) chain_wait();
  const T *QC = f.QC + qc_off;
  T E[3][3];
#pragma unroll
  for (int dj = 0; dj < 3; ++dj)
#pragma unroll
    for (int di = 0; di < 3; ++di) {
      const int w = (a + di) + (b + dj) * ldw;
      const T wv = f.Q[src[dj][di]];
      E[dj][di] = correct ? wv - QC[w] : wv;
    }
  const T c9 = times<9, kInt>(E[1][1]);
  const T w = c9 + times<3, kInt>(E[1][0]), e = c9 + times<3, kInt>(E[1][2]);
  const T s3 = times<3, kInt>(E[0][1]), n3 = times<3, kInt>(E[2][1]);
  const T f11 = sixteenth<kInt>((w + s3) + E[0][0]);
  const T f21 = sixteenth<kInt>((e + s3) + E[0][2]);
  const T f12 = sixteenth<kInt>((w + n3) + E[2][0]);
  const T f22 = sixteenth<kInt>((e + n3) + E[2][2]);
  T *Q = f.Q + q_off + f.lsh;
  const int c = (2 * a + 1) + (2 * b + 1) * ldq;
  if (correct) {
    Q[c] = Q[c] + f11;
    Q[c + 1] = Q[c + 1] + f21;
    Q[c + ldq] = Q[c + ldq] + f12;
    Q[c + ldq + 1] = Q[c + ldq + 1] + f22;
  } else {
    Q[c] = f11;
    Q[c + 1] = f21;
    Q[c + ldq] = f12;
    Q[c + ldq + 1] = f22;
  }
}

// The same with a coarse cell on four lanes, one fine cell each (13
// operations and 4 differences instead of 32 and 9), for levels below 131,072
// cells: solve of a ragged hierarchy whose levels reach 42,000 cells 2.54 ->
// 2.46 ms, disc 1.265 -> 1.235, starfish mixed 2.31 -> 2.26.
template <class T>
__device__ __forceinline__ void prolong_quad(const LevelD &L, const Decomp &D, const FieldsT<T> &f, int correct,
                                             int g4) {
  const int g = g4 >> 2, t = g4 & 3;
  if (g >= D.n) {
    chain_wait();
    return;
  }
  const int p = find_patch(D, g / kBlock, g);
  const PatchD &P = L.patches[p];
  if (!f.active[P.inst]) {
    chain_wait();
    return;
  }
  const int cm = P.mx >> 1, s = g - __ldg(D.beg + p);
  const int b = s / cm, a = s - b * cm, ldw = cm + 2;
  const int w = (a + 1) + (b + 1) * ldw, dx = t & 1 ? 1 : -1, dy = t & 2 ? ldw : -ldw;
  const int *win = f.win + P.win_off + w;
  const int sC = __ldg(win), sX = __ldg(win + dx), sY = __ldg(win + dy), sD = __ldg(win + dx + dy);
  const T *QC = f.QC + P.qc_off + w;
  T *q = f.Q + P.q_off + f.lsh + (2 * a + 1 + (t & 1)) + (2 * b + 1 + (t >> 1)) * (P.mx + 2);
  chain_wait();
  T C = f.Q[sC], X = f.Q[sX], Y = f.Q[sY], E = f.Q[sD];
  if (correct) {
    C = C - QC[0];
    X = X - QC[dx];
    Y = Y - QC[dy];
    E = E - QC[dx + dy];
  }
  const T v = (((9 * C + 3 * X) + 3 * Y) + E) / 16;
  *q = correct ? *q + v : v;
}

// kT threads per block: kBlock, or 64 on a level whose kBlock grid leaves
// SMs idle
template <class T, bool kInt, int kT = kBlock, bool kQuad = false>
__global__ void __launch_bounds__(kT) k_prolong(LevelD L, Decomp D, FieldsT<T> f, int correct) {
  if constexpr (kQuad) prolong_quad<T>(L, D, f, correct, blockIdx.x * kT + threadIdx.x);
  else prolong_item<T, true, kInt>(L, D, f, correct, blockIdx.x * kT + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Coarsest solve (ebCoarsest.m:79-91): u = Ainv (F + bcRhs), one warp per
// row; lane l sums columns l, l+32, ... in order, then a halving tree.
struct CoarsestD {
  int c_off, q_off, n1, N, inst, pad;
  long long ainv_off, rhs_off;
};

// bcRhs null: a homogeneous problem (the correction cycle of the mixed
// form), whose F is FP32 while the solve itself stays FP64.
//
// One hierarchy: one row per block, which spreads the rows' FP64 work over
// as many SMs as there are rows.
template <class T>
__global__ void __launch_bounds__(32) k_coarsest(const double *__restrict__ Ainv, const double *__restrict__ bcRhs,
                                                 const CoarsestD *__restrict__ cd, FieldsT<T> f) {
  const CoarsestD D = cd[0];
  const int row = blockIdx.x, lane = threadIdx.x, N = D.N;
  if (row >= N || !f.active[D.inst]) {
    chain_wait();
    return;
  }
  const double *a = Ainv + D.ainv_off + (size_t)row * N;
  const double *rhs = bcRhs ? bcRhs + D.rhs_off : nullptr;
  constexpr int kPre = 8;   // inverse entries held in registers (N <= 256)
  double av[kPre], bv[kPre];
#pragma unroll
  for (int i = 0; i < kPre; ++i) {
    const int c = lane + 32 * i;
    av[i] = c < N ? __ldg(a + c) : 0.0;
    bv[i] = (c < N && rhs) ? __ldg(rhs + c) : 0.0;
  }
  chain_wait();
  const T *F = f.F + D.c_off;
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < kPre; ++i) {
    const int c = lane + 32 * i;
    if (c < N) s = s + av[i] * (dbl(F[c]) + bv[i]);
  }
  for (int c = lane + 32 * kPre; c < N; c += 32) s = s + a[c] * (dbl(F[c]) + (rhs ? rhs[c] : 0.0));
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const double o = __shfl_down_sync(0xffffffffu, s, off);
    if (lane < off) s = s + o;
  }
  if (lane == 0) {
    const int i = row % D.n1, j = row / D.n1;
    f.Q[D.q_off + (i + 1) + (j + 1) * (D.n1 + 2)] = T(s);
  }
}

// A batch (blockIdx.y: instance): bound by the FP64 pipe, where a warp per
// row costs 29 operations (8 of F + bcRhs, 8 products, 8 sums, 5 of the
// tree).  A block of kBRows rows forms F + bcRhs once in shared memory, the
// products go to the integer pipe (the same bits, mul_int_pipe), and a warp
// holds four rows, whose trees share the halves that a tree leaves idle: 10
// operations a row, each sum in the order above.  64 instances of 256 rows
// 32 us -> 17.
constexpr int kBWarps = 4, kBRows = 4 * kBWarps, kBCols = 256;
template <class T>
__global__ void __launch_bounds__(32 * kBWarps, 7) k_coarsest_batch(const double *__restrict__ Ainv,
                                                                 const double *__restrict__ bcRhs,
                                                                 const CoarsestD *__restrict__ cd, FieldsT<T> f) {
  __shared__ double v[kBCols];
  const CoarsestD D = cd[blockIdx.y];
  const int lane = threadIdx.x & 31, N = D.N;
  const int b0 = blockIdx.x * kBRows, row0 = b0 + (int)(threadIdx.x >> 5) * 4;
  if (b0 >= N || !f.active[D.inst]) {
    chain_wait();
    return;
  }
  const double *rhs = bcRhs ? bcRhs + D.rhs_off : nullptr;
  const double *a = Ainv + D.ainv_off;
  // a ring of four columns per lane and row (more would leave the grid two
  // waves of blocks)
  constexpr int kRing = 4;
  double av[4][kRing];
  auto load = [&](int slot, int c) {
#pragma unroll
    for (int q = 0; q < 4; ++q) av[q][slot] = c < N ? __ldg(a + (size_t)min(row0 + q, N - 1) * N + c) : 0.0;
  };
#pragma unroll
  for (int i = 0; i < kRing; ++i) load(i, lane + 32 * i);
  chain_wait();
  const T *F = f.F + D.c_off;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c0 = 0; c0 < N; c0 += kBCols) {
    if (c0) __syncthreads();                 // the last columns' readers
    for (int c = threadIdx.x; c < kBCols && c0 + c < N; c += 32 * kBWarps)
      v[c] = dbl(F[c0 + c]) + (rhs ? __ldg(rhs + c0 + c) : 0.0);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kBCols / 32; ++i) {
      const int c = lane + 32 * i;
      if (c0 + c < N) {
        const double x = v[c];
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = s[q] + mul_int_pipe(av[q][i % kRing], x);
        load(i % kRing, c0 + c + 32 * kRing);
      }
    }
  }
  // halving trees: lanes l < off add lane l + off; the second of a pair of
  // trees runs in the lanes that the first has given up
  auto pair = [&](double x, double y, int off) -> double {
    const bool up = lane & off;
    const double mine = up ? y : x, sent = up ? x : y;
    return mine + __shfl_xor_sync(0xffffffffu, sent, off);
  };
  const double t0 = pair(s[0], s[1], 16), t1 = pair(s[2], s[3], 16);
  double t = pair(t0, t1, 8);
#pragma unroll
  for (int off = 4; off >= 1; off >>= 1) t = t + __shfl_xor_sync(0xffffffffu, t, off);
  // rows 0, 1 of the pair in lanes 0, 16; rows 2, 3 in lanes 8, 24
  const int q = (lane >> 4) + ((lane >> 3) & 1) * 2, row = row0 + q;
  if ((lane & 7) == 0 && row < N) {
    const int i = row % D.n1, j = row / D.n1;
    f.Q[D.q_off + (i + 1) + (j + 1) * (D.n1 + 2)] = T(t);
  }
}

// ---------------------------------------------------------------------------
// Composite residual (ebCompResidual.m:15-85) of every level >= root, for one
// hierarchy or every instance of a batch, in one launch.  The work is a list
// of warp tasks of up to 32 items of ONE patch (or of one instance's
// correction targets), so every warp belongs to one instance:
//   kind 0  r = FTrue - op(Q) on visible cells of a patch in the norms,
//           correction targets excluded while the corrections are on; an item
//           is kResRows cells of one column, whose inner y fluxes are formed
//           once, or on small hierarchies a single cell
//   kind 1  r at correction targets of a level, corrections added in order,
//           the coarse values taken as the refreshed QC holds them
// and, in a launch of their own (k_qc_refresh), tasks of up to 128 items:
//   kind 2  QC ring refresh of a patch (ebCompResidual.m:25)
//   kind 3  QC interior refresh of a patch (ebCompResidual.m:32-38)
// Inside a solve only the max-norms are needed (kL2 false): a warp reduces
// them into its instance's two accumulators with a max on their bit patterns
// (non-negative doubles order like integers); the source's norm does not
// change between V-cycles and is only formed before the first one.  A report
// (kL2) also reduces the squares, into one slot per task, for
// k_residual_final.  Max-norms are order-free, so linf and rel do not depend
// on the task layout.
//
// Bound by the FP64 pipe and latency: about 13 operations per cell (19 with
// every flux formed twice, the scaling by 1/h^2 on the FP64 pipe and the
// squares): starfish 34 us -> 16 us per iteration, its floor at the
// measured FP64 rate 10 us.
struct ResAcc {
  double out[5];        // linf, l2, fnorm, rel, ncell
};

struct ResTask {
  int kind, level, a, b, n, slot, inst, pad;   // a: patch / CSR level / ring start; b: first item
};

struct LevelX {
  LevelD L;
  CorrCSR C;            // corrections contributed by this (fine) level
  int ct_n, pad;
};

// max of non-negative doubles on the integer pipe (their bit patterns order
// like the values; the FP64 pipe of GB300 is the scarce one).  A NaN loses,
// as in fmax and the reference's max: its pattern ranks below zero here.
__device__ __forceinline__ double pmax(double a, double b) {
  constexpr long long kInf = 0x7FF0000000000000LL;
  long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  x = x > kInf ? -1 : x;
  y = y > kInf ? -1 : y;
  const long long m = x > y ? x : y;
  return __longlong_as_double(m < 0 ? 0 : m);
}

constexpr int kResRowsMax = 4;

// kT threads per block (kBlock, or 64 where the kBlock grid would leave
// SMs with unequal shares of the FP64 work; 14 of those per SM, with 72
// registers: with the 80 to 96 it takes by itself the starfish's 13.9 blocks
// per SM ran in two rounds, the second half empty, 16.5 us; 12 or 16 per SM no
// faster, solve 2.99 -> 2.96 ms, 1024^2 24.8 -> 24.7 for 60 V-cycles)
template <bool kL2, bool kPow2, bool kInt, int kT = kBlock, int kResRows = kResRowsMax>
__global__ void __launch_bounds__(kT, kT == 64 && kResRows == kResRowsMax ? 14 : 1) k_residual(const LevelX *__restrict__ X, const PatchD *__restrict__ patches,
                                                 const ResTask *__restrict__ tasks, int ntask, Fields f, double *slots,
                                                 int nslots, unsigned long long *norms, int want_fn, int mass_corr,
                                                 float *__restrict__ rout) {
  const int w = blockIdx.x * (kT / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  // a frozen instance's residual is neither reported nor needed, so its
  // warps only wait
  if (w >= ntask || !f.active[tasks[w].inst]) {
    chain_wait();
    return;
  }
  const ResTask T = tasks[w];
  double li = 0, sq = 0, fn = 0;
  const LevelX &Xk = X[T.level];
  auto take = [&](double r, double ft) {
    li = pmax(li, fabs(r));
    if (kL2) sq = sq + r * r;
    if (kL2 || want_fn) fn = pmax(fn, fabs(ft));
  };
  if (T.kind == 0) {
    const PatchD &P = patches[T.a];
    const int mx = P.mx, my = P.my, ldq = mx + 2;
    const int i = T.b + min(lane, T.n - 1);
    const int g = i / mx, lx = i - g * mx, lj0 = g * kResRows;
    const int rows = lane < T.n ? min(kResRows, my - lj0) : 0;
    const double *DeW = f.DeW + P.dew_off + lx + lj0 * (mx + 1), *DnS = f.DnS + P.dns_off + lx + lj0 * mx;
    const int cc = P.c_off + lx + lj0 * mx;
    // static operands before the programmatic-launch wait
    double dE[kResRows], dW[kResRows], dN[kResRows + 1], cf[kResRows], ft[kResRows];
    uint8_t fl[kResRows];
    dN[0] = __ldg(DnS);
#pragma unroll
    for (int u = 0; u < kResRows; ++u) {
      const int v = u < rows ? u : 0;
      dE[u] = __ldg(DeW + 1 + v * (mx + 1));
      dW[u] = __ldg(DeW + v * (mx + 1));
      dN[u + 1] = __ldg(DnS + (v + 1) * mx);
      cf[u] = __ldg(f.CC + cc + v * mx);
      ft[u] = __ldg(f.FTrue + cc + v * mx);
      fl[u] = __ldg(f.flags + cc + v * mx);
    }
    if (kPow2) {
      const DivC &Dx = Xk.L.dx, &Dy = Xk.L.dy;
      if (__all_sync(0xffffffffu, faces_in(dE, Dx) && faces_in(dW, Dx) && faces_in(dN, Dy))) {
        scale_faces(dE, Dx, true);
        scale_faces(dW, Dx, true);
        scale_faces(dN, Dy, true);
      } else {
        scale_faces(dE, Dx, false);
        scale_faces(dW, Dx, false);
        scale_faces(dN, Dy, false);
      }
    }
    chain_wait();
    const double *Q = f.Q + P.q_off + (lx + 1) + (lj0 + 1) * ldq;
    double q = Q[0], fs = mul_on<kInt>(dN[0], q - Q[-ldq]);
#pragma unroll
    for (int u = 0; u < kResRows; ++u) {
      if (u >= rows) break;
      const double *Qu = Q + u * ldq;
      const double qn = Qu[ldq];
      const double feE = mul_on<kInt>(dE[u], Qu[1] - q), feW = mul_on<kInt>(dW[u], q - Qu[-1]);
      const double fnN = mul_on<kInt>(dN[u + 1], qn - q);
      if (!((fl[u] & 1) || (mass_corr && (fl[u] & 2)))) {
        const double r = ft[u] - op_flux<kPow2, kInt>(feE, feW, fnN, fs, cf[u], q, Xk.L);
        take(r, ft[u]);
        if (rout) rout[cc + u * mx] = (float)r;
      }
      q = qn;
      fs = fnN;
    }
  } else {   // targets of this level, corrections from the level above
    const LevelX &Xf = X[T.level + 1];
    const bool on = mass_corr && lane < T.n;
    CorrTarget Y;
    int cell = 0, c = 0, ldq = 0;
    double dE = 0, dW = 0, dN = 0, dS = 0, cf = 0, ft = 0;
    bool vis = false;
    if (on) {
      const int g = T.b + lane;
      cell = __ldg(Xf.C.cell + g);
      const PatchD &Pc = Xk.L.patches[__ldg(Xf.C.patch + g)];
      const int s = cell - Pc.c_off, mx = Pc.mx;
      const int lj = s / mx, lx = s - lj * mx;
      ldq = mx + 2;
      c = Pc.q_off + (lx + 1) + (lj + 1) * ldq;
      const double *DeW = f.DeW + Pc.dew_off + lx + lj * (mx + 1), *DnS = f.DnS + Pc.dns_off + lx + lj * mx;
      dE = __ldg(DeW + 1);
      dW = __ldg(DeW);
      dN = __ldg(DnS + mx);
      dS = __ldg(DnS);
      cf = __ldg(f.CC + cell);
      ft = __ldg(f.FTrue + cell);
      vis = !(__ldg(f.flags + cell) & 1);
      Y = corr_target<double>(Xf.C, g, f);
    }
    chain_wait();
    if (on) {                // corrections off: kind 0 took these cells, and zeros go to the task's slot
      const double *Q = f.Q + c;
      double r = ft - op_pre<kPow2>(Q[0], Q[1], Q[-1], Q[ldq], Q[-ldq], dE, dW, dN, dS, cf, Xk.L);
      r = add_corrections<kPow2>(r, Y, Xf.C, Xk.L, f, true);
      if (rout) rout[cell] = (float)r;
      if (vis) take(r, ft);
    }
  }
  if (!kL2 && !norms) return;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    li = pmax(li, __shfl_down_sync(0xffffffffu, li, off));
    if (kL2 || want_fn) fn = pmax(fn, __shfl_down_sync(0xffffffffu, fn, off));
    if (kL2) sq = sq + __shfl_down_sync(0xffffffffu, sq, off);
  }
  if (lane) return;
  if (kL2) {
    slots[T.slot] = li;
    slots[nslots + T.slot] = sq;
    slots[2 * nslots + T.slot] = fn;
  } else {
    // most warps find a larger value there already and leave it
    unsigned long long *a = norms + 2 * T.inst;
    const unsigned long long l = (unsigned long long)__double_as_longlong(li);
    if (l > __ldcg(a)) atomicMax(a, l);
    if (want_fn) atomicMax(a + 1, (unsigned long long)__double_as_longlong(fn));
  }
}

// The refresh of QC's ring and interior that the reference's residual makes
// (ebCompResidual.m:25,32-38), a function of Q alone: no kernel reads a QC
// cell between a residual and the next restriction and ring gather, so a
// solve runs it once, after its last V-cycle.
__global__ void __launch_bounds__(kBlock) k_qc_refresh(const PatchD *__restrict__ patches,
                                                       const ResTask *__restrict__ tasks, int ntask, Fields f,
                                                       const int *__restrict__ ring) {
  const int w = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (w >= ntask) return;
  const ResTask T = tasks[w];
  if (T.kind == 2) {
    for (int e = lane; e < T.n; e += 32) {
      const int i = T.a + e;
      f.QC[__ldg(ring + 2 * i + 1)] = f.Q[__ldg(ring + 2 * i)];
    }
    return;
  }
  const PatchD &P = patches[T.a];
  const int cmx = P.mx >> 1;
  for (int e = lane; e < T.n; e += 32) {
    const int s = T.b + e;
    const int cj = s / cmx, ci = s - cj * cmx;
    f.QC[P.qc_off + (ci + 1) + (cj + 1) * (cmx + 2)] = restrict_cell(f.Q + P.q_off, P.mx + 2, ci, cj);
  }
}

// per instance: the slot ranges of its residual tasks, level by level
struct InstRes {
  int range0, range1;   // into the (slot0, slot1, level area) range table
  int max_vcycles, pad;
  double rel_tol, ncell;
};

struct SlotRange {
  int s0, s1;
  double area;
};

// The end of a solve's residual: per instance rel = linf / max(fnorm,
// realmin), the history and the stop test (ebSolveCycles.m:17-46: an instance
// stays active while it < MaxVCycles and rel > RelTol), then the condition of
// the solve loop's WHILE node (and of `c1`, with ncond 2): 1 while any
// instance iterates.  mode 0 is the residual before the first V-cycle; mode 1
// follows a V-cycle of the instances active during it.  One block, a thread
// per instance: the former pair of kernels (a tree over one slot per task,
// then the condition) and the turn of the loop took 21 us of a starfish
// iteration, now 7, six of them the loop's own.
constexpr int kStep = 256;
__global__ void __launch_bounds__(kStep) k_solve_step(const InstRes *__restrict__ ir, int ninst,
                                                      unsigned long long *norms, ResAcc *acc, int *active, int *iters,
                                                      double *hist, int hist_stride, int mode,
                                                      const int *__restrict__ crange, int nlev, uint8_t *cact,
                                                      cudaGraphConditionalHandle c0, cudaGraphConditionalHandle c1,
                                                      int ncond) {
  chain_wait();
  int any = 0;
  for (int i = threadIdx.x; i < ninst; i += kStep) {
    if (mode != 0 && !active[i]) continue;
    const InstRes R = ir[i];
    const double linf = __longlong_as_double((long long)norms[2 * i]);
    double fnorm = __longlong_as_double((long long)norms[2 * i + 1]);
    norms[2 * i] = 0;
    fnorm = fnorm > 2.2250738585072014e-308 ? fnorm : 2.2250738585072014e-308;
    const double rel = linf / fnorm;
    ResAcc &A = acc[i];
    A.out[0] = linf;
    A.out[2] = fnorm;
    A.out[3] = rel;
    A.out[4] = R.ncell;
    const int it = mode == 0 ? 0 : iters[i] + 1;
    iters[i] = it;
    if (it < hist_stride) hist[(size_t)i * hist_stride + it] = linf;
    const int a = (it < R.max_vcycles && rel > R.rel_tol) ? 1 : 0;
    active[i] = a;
    any |= a;
    // the smoother's per-chunk copy of the flag, over the instance's chunk
    // range of every level (crange: [inst][level] begin, end)
    if (cact && (mode == 0 || !a))
      for (int k = 0; k < nlev; ++k)
        for (int c = crange[2 * (i * nlev + k)]; c < crange[2 * (i * nlev + k) + 1]; ++c) cact[c] = (uint8_t)a;
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0 && ncond > 0) {
    cudaGraphSetConditional(c0, any ? 1u : 0u);
    if (ncond > 1) cudaGraphSetConditional(c1, any ? 1u : 0u);
  }
}

// A residual report of every instance (one block per instance): max-norms
// over its slots, L2 per level from that level's slots in a fixed tree order
// weighted by the cell area, rel = linf / max(fnorm, realmin).
constexpr int kFinal = 512, kFinalRanges = 8;
__global__ void __launch_bounds__(kFinal) k_residual_final(const InstRes *__restrict__ ir,
                                                          const SlotRange *__restrict__ ranges, const double *slots,
                                                          int nslots, ResAcc *acc) {
  chain_wait();
  const int inst = blockIdx.x, t = threadIdx.x;
  const InstRes R = ir[inst];
  double li = 0, fn = 0, l2sq = 0;
  // up to kFinalRanges levels' trees side by side, the last five steps of
  // each in a warp of its own (a report of a starfish 73 us through the call
  // with one level after the other, 65 side by side)
  __shared__ double s_p[kFinalRanges][kFinal], s_a[kFinal], s_b[kFinal], s_l2[kFinalRanges];
  for (int r0 = R.range0; r0 < R.range1; r0 += kFinalRanges) {
    const int nr = min(kFinalRanges, R.range1 - r0);
    for (int r = 0; r < nr; ++r) {
      const int s0 = ranges[r0 + r].s0, s1 = ranges[r0 + r].s1;
      double p = 0;
      for (int i = s0 + t; i < s1; i += kFinal) {
        p = p + slots[nslots + i];
        li = pmax(li, slots[i]);
        fn = pmax(fn, slots[2 * nslots + i]);
      }
      s_p[r][t] = p;
    }
    __syncthreads();
    for (int off = kFinal / 2; off >= 32; off >>= 1) {
      for (int i = t; i < nr * off; i += kFinal) {
        double *q = s_p[i / off] + (i & (off - 1));
        q[0] = q[0] + q[off];
      }
      __syncthreads();
    }
    for (int r = t >> 5; r < nr; r += kFinal / 32) {
      double p = s_p[r][t & 31];
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) p = p + __shfl_down_sync(0xffffffffu, p, off);
      if ((t & 31) == 0) s_l2[r] = p;
    }
    __syncthreads();
    for (int r = 0; r < nr; ++r) l2sq = l2sq + s_l2[r] * ranges[r0 + r].area;
    __syncthreads();
  }
  s_a[t] = li;
  s_b[t] = fn;
  __syncthreads();
  for (int off = kFinal / 2; off >= 1; off >>= 1) {
    if (t < off) {
      s_a[t] = pmax(s_a[t], s_a[t + off]);
      s_b[t] = pmax(s_b[t], s_b[t + off]);
    }
    __syncthreads();
  }
  if (t) return;
  const double linf = s_a[0], fnorm = s_b[0] > 2.2250738585072014e-308 ? s_b[0] : 2.2250738585072014e-308;
  ResAcc &A = acc[inst];
  A.out[0] = linf;
  A.out[1] = sqrt(l2sq);
  A.out[2] = fnorm;
  A.out[3] = linf / fnorm;
  A.out[4] = R.ncell;
}

// ---------------------------------------------------------------------------
// FP64 issue-rate probe (bsam_fp64_rate): eight independent x = x*a + b
// chains per thread, each a separate multiply and add (the library is built
// without contraction), so 16 FP64 operations per iteration.
constexpr int kFp64RateOps = 16;
__global__ void __launch_bounds__(kBlock) k_fp64_rate(double *out, int iters, double a, double b) {
  double x[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) x[u] = 1.0 + 1e-3 * u + 1e-9 * threadIdx.x;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = x[u] * a + b;
  }
  double s = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) s = s + x[u];
  out[blockIdx.x * kBlock + threadIdx.x] = s;
}

// ---------------------------------------------------------------------------
// Force reset F = FTrue (ebSolveCycles.m:30-34) of the active instances of a
// batch, one thread per cell over every patch of every level (a single
// hierarchy copies the whole array instead).
__global__ void __launch_bounds__(kBlock) k_freset(Decomp D, const PatchD *__restrict__ patches, Fields f) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) {
    chain_wait();
    return;
  }
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = patches[p];
  if (!f.active[P.inst]) {
    chain_wait();
    return;
  }
  const int cc = P.c_off + (g - __ldg(D.beg + p));
  const double v = __ldg(f.FTrue + cc);
  chain_wait();
  f.F[cc] = v;
}

// ---------------------------------------------------------------------------
// Defect correction of the mixed form: Q += E (FP64 += FP32) on the interior
// cells of every patch of the active instances.
__global__ void __launch_bounds__(kBlock) k_update(Decomp D, const PatchD *__restrict__ patches, double *Q,
                                                   const float *__restrict__ E, const int *__restrict__ active) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) {
    chain_wait();
    return;
  }
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = patches[p];
  if (!active[P.inst]) {
    chain_wait();
    return;
  }
  const int s = g - __ldg(D.beg + p);
  const int lj = s / P.mx, lx = s - lj * P.mx;
  const int qi = P.q_off + (lx + 1) + (lj + 1) * (P.mx + 2);
  chain_wait();
  Q[qi] = Q[qi] + (double)E[qi];
}

// Mixed form: Q += E of the correction cycle (k_update) and the restriction
// of the finest level k (k_restrict) in one launch, where the consistency
// step starts with that plain restriction: blocks [0, nb_r) restrict level
// k, each item adding E to its four fine cells first (k_update's sum) and
// restricting the sums (restrict_cell's order); the other blocks add E to
// the cells of the levels below k that no finer level covers.  A covered
// cell is rewritten by a restriction before anything reads it, and the ones
// this launch's restriction writes must not be touched here, so skipping
// them gives the values of k_update then k_restrict.
template <int kT = kBlock>
__global__ void __launch_bounds__(kT) k_restrict_update(LevelD L, Decomp D, Fields f, const float *__restrict__ E,
                                                       int nb_r, Decomp Du, const PatchD *__restrict__ patches) {
  if ((int)blockIdx.x < nb_r) {
    const int g = blockIdx.x * kT + threadIdx.x;
    if (g >= D.n) {
      chain_wait();
      return;
    }
    const int p = find_patch(D, g / kBlock, g);
    const PatchD &P = L.patches[p];
    if (!f.active[P.inst]) {
      chain_wait();
      return;
    }
    const int cmx = P.mx >> 1, ldq = P.mx + 2;
    const int s = g - __ldg(D.beg + p);
    const int cj = s / cmx, ci = s - cj * cmx;
    const int dst = __ldg(f.fp + 2 * (P.fp_off + s));
    chain_wait();
    double *Q = f.Q + P.q_off;
    const float *e = E + P.q_off;
    const int c = (2 * ci + 1) + (2 * cj + 1) * ldq;
    const double q0 = Q[c] + (double)e[c], q1 = Q[c + 1] + (double)e[c + 1];
    const double q2 = Q[c + ldq] + (double)e[c + ldq], q3 = Q[c + ldq + 1] + (double)e[c + ldq + 1];
    Q[c] = q0;
    Q[c + 1] = q1;
    Q[c + ldq] = q2;
    Q[c + ldq + 1] = q3;
    const double R = 0.25 * (((q0 + q1) + q2) + q3);
    f.QC[P.qc_off + (ci + 1) + (cj + 1) * (cmx + 2)] = R;
    f.Q[dst] = R;
    return;
  }
  const int g = ((int)blockIdx.x - nb_r) * kT + threadIdx.x;
  if (g >= Du.n) {
    chain_wait();
    return;
  }
  const int p = find_patch(Du, g / kBlock, g);
  const PatchD &P = patches[p];
  const int s = g - __ldg(Du.beg + p);
  if (!f.active[P.inst] || (__ldg(f.flags + P.c_off + s) & 1)) {
    chain_wait();
    return;
  }
  const int lj = s / P.mx, lx = s - lj * P.mx;
  const int qi = P.q_off + (lx + 1) + (lj + 1) * (P.mx + 2);
  chain_wait();
  f.Q[qi] = f.Q[qi] + (double)E[qi];
}

// Parabolic driver on the device.  k_history: Uoo = Uo, Uo = interior of Q
// (ebpSolve.m:52-56); with rotate 0 only Uo = interior of Q (the new
// hierarchy's Uo after a regrid, ebpRegrid.m:49).  k_prhs: FTrue of the step
// on the cells of levels at or above the root (ebpRhs.m:25-47): BE f + Uo/Dt,
// BDF2 f + (2 Uo - 0.5 Uoo)/Dt, in that operation order; f null is f = 0.
__global__ void __launch_bounds__(kBlock) k_history(Decomp D, const PatchD *__restrict__ patches, const double *Q,
                                                    double *Uo, double *Uoo, int rotate) {
  chain_wait();
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) return;
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = patches[p];
  const int s = g - __ldg(D.beg + p);
  const int lj = s / P.mx, lx = s - lj * P.mx;
  const int cc = P.c_off + s;
  if (rotate) Uoo[cc] = Uo[cc];
  Uo[cc] = Q[P.q_off + (lx + 1) + (lj + 1) * (P.mx + 2)];
}

// The BDF2 history Uoo of one level of a regridded hierarchy
// (ebpRegrid.m:62-137, transferLevel): where a patch of the old hierarchy
// on the same level covers the cell (src_old >= 0, an index into the old
// hierarchy's cells) its old value is copied; elsewhere the value is the
// conservative-linear prolongation of the new parent level's (already
// transferred) history over the patch footprint (conslinInterior +
// parentFootprint: central slopes inside the footprint, one-sided at its
// edges, none along a footprint one coarse cell wide), in the reference's
// operation order.  The footprint's parent cells come from the footprint
// table (second entry per coarse cell); the root level copies every cell.
__global__ void __launch_bounds__(kBlock) k_uoo_transfer(LevelD L, Decomp D, const int *__restrict__ fp,
                                                         const int *__restrict__ src_old,
                                                         const double *__restrict__ uoo_old, double *uoo) {
  chain_wait();
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) return;
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = L.patches[p];
  const int s = g - __ldg(D.beg + p);
  const int c = P.c_off + s;
  const int so = src_old[c];
  if (so >= 0) {
    uoo[c] = uoo_old[so];
    return;
  }
  const int mx = P.mx, lj = s / mx, li = s - lj * mx;
  const int cmx = mx >> 1, cmy = P.my >> 1, ci = li >> 1, cj = lj >> 1;
  const int *pc = fp + 2 * P.fp_off + 1;      // parent cell of footprint cell t at pc[2 t]
  auto at = [&](int a, int b) { return uoo[pc[2 * (a + b * cmx)]]; };
  const double v = at(ci, cj);
  double sx = 0, sy = 0;
  if (cmx > 1) sx = ci == 0 ? at(1, cj) - v : (ci == cmx - 1 ? v - at(ci - 1, cj) : (at(ci + 1, cj) - at(ci - 1, cj)) / 2);
  if (cmy > 1) sy = cj == 0 ? at(ci, 1) - v : (cj == cmy - 1 ? v - at(ci, cj - 1) : (at(ci, cj + 1) - at(ci, cj - 1)) / 2);
  const double a = (li & 1) ? v + sx / 4 : v - sx / 4;
  uoo[c] = (lj & 1) ? a + sy / 4 : a - sy / 4;
}

__global__ void __launch_bounds__(kBlock) k_prhs(Decomp D, const PatchD *__restrict__ patches, double *FTrue,
                                                 const double *__restrict__ fsrc, const double *__restrict__ Uo,
                                                 const double *__restrict__ Uoo, double dt, int bdf2) {
  chain_wait_static();
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) return;
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = patches[p];
  if (!(P.pflags & 1)) return;               // below the root
  const int cc = P.c_off + (g - __ldg(D.beg + p));
  const double f = fsrc ? fsrc[cc] : 0.0;
  FTrue[cc] = bdf2 ? f + (2 * Uo[cc] - 0.5 * Uoo[cc]) / dt : f + Uo[cc] / dt;
}

// ---------------------------------------------------------------------------
// Tagging indicators on the device (ebTagCluster.m:50-59 'ulap',
// ebRte.m:14-41 'rte'), on the finest level's index space (n0 x n1, stored
// i-major: index i * n1 + j).  Only the final mask goes to the host, where
// Berger-Rigoutsos clustering runs.  The arithmetic is the host
// restatement's, in its order, so the masks are identical.
__global__ void __launch_bounds__(kBlock) k_tag_ulap(LevelD L, Decomp D, const double *__restrict__ Q, double thr,
                                                     uint8_t *T, uint8_t *cover, int n1) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) return;
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = L.patches[p];
  const int s = g - __ldg(D.beg + p);
  const int lj = s / P.mx, li = s - lj * P.mx;
  const int ldq = P.mx + 2;
  const double *q = Q + P.q_off + (li + 1) + (lj + 1) * ldq;
  const double sdx = (q[1] - 2 * q[0]) + q[-1];
  const double sdy = (q[ldq] - 2 * q[0]) + q[-ldq];
  const double v = sqrt(sdx * sdx + sdy * sdy);
  const size_t o = (size_t)(P.ilo - 1 + li) * n1 + (P.jlo - 1 + lj);
  cover[o] = 1;
  if (v > thr) T[o] = 1;
}

// relative truncation error: |op_2h(R u) - R(op_h u)| per coarse cell,
// spread to its four fine cells
__global__ void __launch_bounds__(kBlock) k_tag_rte(LevelD L, Decomp D, Fields f, double thr, uint8_t *T,
                                                    uint8_t *cover, int n1) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= D.n) return;
  const int p = find_patch(D, blockIdx.x, g);
  const PatchD &P = L.patches[p];
  const int mx = P.mx, my = P.my, cmx = mx >> 1, cmy = my >> 1, ldq = mx + 2;
  const int s = g - __ldg(D.beg + p);
  const int cj = s / cmx, ci = s - cj * cmx;
  const double *Q = f.Q + P.q_off, *DeW = f.DeW + P.dew_off, *DnS = f.DnS + P.dns_off, *CC = f.CC + P.c_off;
  double Lf[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int li = 2 * ci + (t & 1), lj = 2 * cj + (t >> 1);
    Lf[t] = op_cell_r(Q, ldq, DeW, DnS, CC[li + lj * mx], mx, li, lj, L);
  }
  const double RL = 0.25 * (((Lf[0] + Lf[1]) + Lf[2]) + Lf[3]);
  // the restricted solution and its ghost frame (pair averages of fine ghosts)
  const double rc = restrict_cell(Q, ldq, ci, cj);
  const double re = ci + 1 < cmx ? restrict_cell(Q, ldq, ci + 1, cj)
                                 : 0.5 * (Q[(mx + 1) + (2 * cj + 1) * ldq] + Q[(mx + 1) + (2 * cj + 2) * ldq]);
  const double rw = ci > 0 ? restrict_cell(Q, ldq, ci - 1, cj) : 0.5 * (Q[(2 * cj + 1) * ldq] + Q[(2 * cj + 2) * ldq]);
  const double rn = cj + 1 < cmy ? restrict_cell(Q, ldq, ci, cj + 1)
                                 : 0.5 * (Q[(2 * ci + 1) + (my + 1) * ldq] + Q[(2 * ci + 2) + (my + 1) * ldq]);
  const double rs = cj > 0 ? restrict_cell(Q, ldq, ci, cj - 1) : 0.5 * (Q[2 * ci + 1] + Q[2 * ci + 2]);
  // averaged coarse coefficients
  const double cE = 0.5 * (DeW[(2 * ci + 2) + (2 * cj) * (mx + 1)] + DeW[(2 * ci + 2) + (2 * cj + 1) * (mx + 1)]);
  const double cW = 0.5 * (DeW[(2 * ci) + (2 * cj) * (mx + 1)] + DeW[(2 * ci) + (2 * cj + 1) * (mx + 1)]);
  const double cN = 0.5 * (DnS[(2 * ci) + (2 * cj + 2) * mx] + DnS[(2 * ci + 1) + (2 * cj + 2) * mx]);
  const double cS = 0.5 * (DnS[(2 * ci) + (2 * cj) * mx] + DnS[(2 * ci + 1) + (2 * cj) * mx]);
  const double cC = 0.25 * (((CC[2 * ci + 2 * cj * mx] + CC[2 * ci + 1 + 2 * cj * mx]) + CC[2 * ci + (2 * cj + 1) * mx]) +
                            CC[2 * ci + 1 + (2 * cj + 1) * mx]);
  const double H2x = (2 * L.hx) * (2 * L.hx), H2y = (2 * L.hy) * (2 * L.hy);
  const double feE = cE * (re - rc), feW = cW * (rc - rw), fnN = cN * (rn - rc), fnS = cS * (rc - rs);
  const double tau = ((-(feE - feW)) / H2x - (fnN - fnS) / H2y + cC * rc) - RL;
  const bool tag = fabs(tau) > thr;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int li = 2 * ci + (t & 1), lj = 2 * cj + (t >> 1);
    const size_t o = (size_t)(P.ilo - 1 + li) * n1 + (P.jlo - 1 + lj);
    cover[o] = 1;
    if (tag) T[o] = 1;
  }
}

// dilate by b cells (outside the index space counts as untagged), then keep
// what the 8-eroded patch cover allows (outside counts as covered)
__global__ void __launch_bounds__(kBlock) k_tag_buffer(const uint8_t *__restrict__ T, const uint8_t *__restrict__ cover,
                                                       uint8_t *out, int n0, int n1, int b) {
  const long long g = (long long)blockIdx.x * kBlock + threadIdx.x;
  if (g >= (long long)n0 * n1) return;
  const int i = (int)(g / n1), j = (int)(g - (long long)i * n1);
  bool t = false;
  for (int dx = -b; dx <= b && !t; ++dx)
    for (int dy = -b; dy <= b; ++dy) {
      const int ii = i + dx, jj = j + dy;
      if (ii >= 0 && ii < n0 && jj >= 0 && jj < n1 && T[(size_t)ii * n1 + jj]) {
        t = true;
        break;
      }
    }
  bool a = true;
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy) {
      const int ii = i + dx, jj = j + dy;
      if (ii >= 0 && ii < n0 && jj >= 0 && jj < n1 && !cover[(size_t)ii * n1 + jj]) a = false;
    }
  out[g] = (t && a) ? 1 : 0;
}

// the same for four cells of a row per thread, as bytes of a word: n1 a
// multiple of four and b at most four.  The rows' words are combined first
// (or of the tags, and of the cover), then the bytes beside a cell: 9 words
// per row and a few shifts instead of 34 bytes per cell (b = 2); the tags of
// 1024 x 1024 cells 156 us through the call -> 131
__global__ void __launch_bounds__(kBlock) k_tag_buffer4(const uint32_t *__restrict__ T, const uint32_t *__restrict__ cover,
                                                        uint32_t *out, int n0, int w, int b) {
  const long long g = (long long)blockIdx.x * kBlock + threadIdx.x;
  if (g >= (long long)n0 * w) return;
  const int i = (int)(g / w), j = (int)(g - (long long)i * w);
  // tags and covers hold 0 or 1 per byte; outside: untagged, covered
  uint32_t tl = 0, tc = 0, tr = 0, al = 0x01010101u, ac = 0x01010101u, ar = 0x01010101u;
  for (int ii = max(i - b, 0); ii <= min(i + b, n0 - 1); ++ii) {
    const uint32_t *r = T + (size_t)ii * w + j;
    tc |= r[0];
    if (j > 0) tl |= r[-1];
    if (j + 1 < w) tr |= r[1];
  }
#pragma unroll
  for (int d = -1; d <= 1; ++d) {
    const int ii = i + d;
    if (ii < 0 || ii >= n0) continue;
    const uint32_t *r = cover + (size_t)ii * w + j;
    ac &= r[0];
    if (j > 0) al &= r[-1];
    if (j + 1 < w) ar &= r[1];
  }
  uint32_t t = tc;
#pragma unroll
  for (int d = 1; d <= 4; ++d)               // the byte d to the right, d to the left
    if (d <= b) t |= __funnelshift_rc(tc, tr, 8 * d) | __funnelshift_lc(tl, tc, 8 * d);
  const uint32_t a = ac & __funnelshift_r(ac, ar, 8) & __funnelshift_l(al, ac, 8);
  out[g] = t & a;
}

// FP32 copy of an FP64 array (coefficient copies of the mixed form)
__global__ void __launch_bounds__(kBlock) k_to_f32(const double *__restrict__ a, float *__restrict__ b, long long n) {
  chain_wait_static();
  for (long long i = blockIdx.x * (long long)kBlock + threadIdx.x; i < n; i += (long long)gridDim.x * kBlock)
    b[i] = (float)a[i];
}

// ---------------------------------------------------------------------------
// Composite sums over visible cells, per-block partials of two quantities:
// sum(u) and the number of cells (ebCompositeMean.m), or sum(C u - FTrue) and
// sum(|FTrue|) (ebMassCheck.m lhs).  Several levels in one launch, the blocks
// of each as a launch of its own would have them; a launch per level, each
// with all four sums, made the mean of a starfish 62 us through the call and its
// mass check 77, one launch of two sums 30 and 47.
constexpr int kMaxSums = 16;
struct SumSpans {
  int n, b0[kMaxSums + 1];     // first block per level
  const PatchD *patches[kMaxSums];
  Decomp D[kMaxSums];
};
template <bool kMass>
__global__ void __launch_bounds__(kBlock) k_sums(const __grid_constant__ SumSpans S, Fields f, double *partials) {
  int l = 0;
  while ((int)blockIdx.x >= S.b0[l + 1]) ++l;
  const Decomp &D = S.D[l];
  const int b = blockIdx.x - S.b0[l], g = b * kBlock + threadIdx.x, t = threadIdx.x;
  double x = 0, y = 0;
  if (g < D.n) {
    const int p = find_patch(D, b, g);
    const PatchD &P = S.patches[l][p];
    const int s = g - __ldg(D.beg + p);
    const int lj = s / P.mx, lx = s - lj * P.mx;
    const int cc = P.c_off + s;
    if (!(f.flags[cc] & 1)) {
      const double u = f.Q[P.q_off + (lx + 1) + (lj + 1) * (P.mx + 2)];
      x = kMass ? f.CC[cc] * u - f.FTrue[cc] : u;
      y = kMass ? fabs(f.FTrue[cc]) : 1.0;
    }
  }
  // halving tree: thread t < off adds thread t + off
  __shared__ double sh[2][kBlock];
  sh[0][t] = x;
  sh[1][t] = y;
  __syncthreads();
#pragma unroll
  for (int off = kBlock / 2; off >= 32; off >>= 1) {
    if (t < 2 * off) {         // the second sum's threads follow the first's
      double *r = sh[t / off];
      r[t & (off - 1)] = r[t & (off - 1)] + r[(t & (off - 1)) + off];
    }
    __syncthreads();
  }
  if (t >= 64) return;
  double v = sh[t >> 5][t & 31];
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, off);
  if ((t & 31) == 0) partials[2 * blockIdx.x + (t >> 5)] = v;
}

// Boundary flux terms of the mass balance (ebMassCheck.m:30-60), one per
// uncovered physical face: D (u_ghost - u_interior) / h.  The whole solution
// and its coefficients went to the host for them before (13 MB of a starfish;
// the check 0.36 -> 0.08 ms).
struct FluxFace {
  int ghost, in, coef, yface;
  double h;
};
__global__ void __launch_bounds__(kBlock) k_flux_terms(const FluxFace *__restrict__ faces, int n,
                                                       const double *__restrict__ Q, const double *__restrict__ DeW,
                                                       const double *__restrict__ DnS, double *__restrict__ out) {
  const int i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  const FluxFace f = faces[i];
  out[i] = (f.yface ? DnS : DeW)[f.coef] * (Q[f.ghost] - Q[f.in]) / f.h;
}

}  // namespace bsam
