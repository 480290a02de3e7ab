// tile.cuh -- the smoother's tile form: up to kTilePasses colour passes of a
// level's red-black Gauss-Seidel (EllipticBSAM/src/ebRelaxLevel.m:28-38,
// relax2d of ebKernels.m:37-95) in one launch, without any exchange between
// blocks.
//
// A tile is a rectangle of one patch.  Its block loads the tile's cells and
// the surrounding cells of the level that the passes depend on (the tile's
// window: a rectangle of the level's index space, reaching into sibling
// patches) into shared memory, runs the passes there -- the halo cells'
// updates are repeated by every block that needs them -- and writes its own
// cells.  Source and destination are different copies of the level, so no
// block reads what another one writes: the pre-smoothing moves a level from
// the solution array to its second copy, the restriction, coarse load and
// prolongation-correction of that level work on the second copy (FieldsT's
// lsh), and the post-smoothing moves it back.
//
// What each update needs is found once per hierarchy, on the device
// (k_tile_build): a cell is needed after pass p if it is a tile cell, or a
// pass later than p updates a needed cell from it.  Inside the level a
// neighbour across a patch face is the sibling's cell itself (the COPY
// rules' operand, which the build checks), so no copied ghost is read;
// coarse-fine and physical sides are evaluated by the reading cell with
// relax_cell's arithmetic, their constant parts (parent cells, boundary
// data) formed once per launch.  Every update's operations and their order
// are relax_cell's: the results are the chained passes' bit for bit.
#pragma once
#include <climits>

#include "kernels.cuh"

namespace bsam {

constexpr int kTilePasses = 6;             // most passes of one launch
constexpr int kTileGroups = 3;             // pairs of passes
static_assert(kTilePasses == 2 * kTileGroups, "");
constexpr int kTileMax = 32;               // largest tile side
constexpr int kTileHalo = 2 * kTilePasses; // widest margin: a coarse-fine rule reads two cells along its face
constexpr int kTileWin = (kTileMax + 2 * kTileHalo) * (kTileMax + 2 * kTileHalo);
constexpr int kTileT = 256;                // threads of a tile's block
constexpr int kTileNear = 1024;            // patches a window may touch
constexpr int kTileFaces = 1024;           // cells of a window with a physical or coarse-fine side

struct __align__(16) TileD {
  int patch, i0, j0, w;        // level-local patch, first interior cell, size
  int h, pa, pb, inst;         // level-local patches of the tile's instance: [pa, pb)
  int wx, wy, mx, my;          // window size, and the tile's place in it
  int wq_off, pad0, pad1, pad2;   // first entry of the window's cell table
};

// the updates of a tile: entries [ent, ent + nA[2]) are cells of the last
// pass's colour, the first nA[g] of them needed g pairs of passes before the
// end, then nB[2] of the other colour in the same order
struct __align__(16) TileTab {
  int ent, face, nf, pad;
  int nA[kTileGroups], x0;     // x0 .. y1 (counting): the needed cells' bounds in the widest window
  int nB[kTileGroups], y0;
  int fA[kTileGroups], x1;     // the special ones' TileFaces, counted in the same way
  int fB[kTileGroups], y1;
};

// an update: window position | flags << 16 (bit 15: has a TileFace, index in
// bits 0..9), packed operands' and force's index
struct __align__(16) TileEnt {
  uint32_t sf;
  int pack, cell, pad;
};
constexpr uint32_t kTileSpecial = 0x8000u << 16;

// a physical or coarse-fine side: kind 0 none, 1 Dirichlet, 2 Neumann, else
// 8 + GhostType; bit 7: the west / south side.  a, b: window positions of
// the rule's operands on the level, c, d, e: its parent cells (physical: c
// the boundary datum), g: the ghost cell.
struct TileSide {
  uint16_t kind, a, b, pad;
  int c, d, e, g;
};
struct __align__(16) TileFace {
  TileSide s[2];               // x side, y side
};

// ---------------------------------------------------------------------------
// Build of the tables, one block per tile.  kEmit false counts the updates
// and finds the window's bounds (tab), true writes.  A tile the form cannot
// take (a rule operand off the level's index space, a table larger than its
// bound) raises *bad and the level keeps its other forms.
struct TileBuild {
  const PatchD *patches;       // the level's patches
  const Rule *perim;
  const TileD *tiles;
  const int *chunk0;           // level-local first chunk per patch
  TileTab *tab;
  int q_lo, q_hi;
  int *wq;                     // per window cell: its Q index, or -1 where it is not needed
  TileEnt *ent;
  TileFace *face;
  int *bad;
};

constexpr int kTileBuildT = 256;

template <bool kEmit>
__global__ void __launch_bounds__(kTileBuildT) k_tile_build(TileBuild B) {
  __shared__ uint16_t s_near[kTileNear];
  __shared__ uint16_t s_own[kTileWin];
  __shared__ int8_t s_need[kTileWin];
  __shared__ int s_n, s_bad, s_base, s_warp[kTileBuildT / 32], s_lo[2], s_hi[2];
  const int t = threadIdx.x;
  const TileD td = B.tiles[blockIdx.x];
  constexpr int mA = 1;                    // every launch ends with the second colour
  const int W = td.wx * td.wy;
  const PatchD &P0 = B.patches[td.patch];
  const int I0 = P0.ilo + td.i0 - td.mx, J0 = P0.jlo + td.j0 - td.my;
  if (t == 0) {
    s_n = s_bad = 0;
    s_lo[0] = s_lo[1] = INT_MAX;
    s_hi[0] = s_hi[1] = -1;
  }
  __syncthreads();
  // patches that meet the window
  for (int p = td.pa + t; p < td.pb; p += kTileBuildT) {
    const PatchD &P = B.patches[p];
    if (P.ilo < I0 + td.wx && P.ilo + P.mx > I0 && P.jlo < J0 + td.wy && P.jlo + P.my > J0) {
      const int k = atomicAdd(&s_n, 1);
      if (k < kTileNear) s_near[k] = (uint16_t)(p - td.pa);
      else s_bad = 1;
    }
  }
  __syncthreads();
  const int nn = min(s_n, kTileNear);
  auto patch_of = [&](int c) -> const PatchD & { return B.patches[td.pa + s_near[s_own[c]]]; };
  for (int c = t; c < W; c += kTileBuildT) {
    const int I = I0 + c % td.wx, J = J0 + c / td.wx;
    int o = 0xFFFF;
    for (int k = 0; k < nn; ++k) {
      const PatchD &P = B.patches[td.pa + s_near[k]];
      if (I >= P.ilo && I < P.ilo + P.mx && J >= P.jlo && J < P.jlo + P.my) {
        o = k;
        break;
      }
    }
    s_own[c] = (uint16_t)o;
    const int x = c % td.wx - td.mx, y = c / td.wx - td.my;
    const bool in = x >= 0 && x < td.w && y >= 0 && y < td.h;
    s_need[c] = in && o != 0xFFFF ? (int8_t)kTilePasses : (int8_t)-1;
    if (in && (o == 0xFFFF || s_near[o] != (uint16_t)(td.patch - td.pa))) s_bad = 1;
  }
  __syncthreads();
  auto local = [&](int c, const PatchD &P, int &li, int &lj) {
    li = I0 + c % td.wx - P.ilo;
    lj = J0 + c / td.wx - P.jlo;
  };
  auto qidx = [&](int c) {
    const PatchD &P = patch_of(c);
    int li, lj;
    local(c, P, li, lj);
    return P.q_off + (li + 1) + (lj + 1) * (P.mx + 2);
  };
  auto colour = [&](int c) {
    const PatchD &P = patch_of(c);
    int li, lj;
    local(c, P, li, lj);
    return (li + lj + P.par0) & 1;
  };
  // the window position of a Q index inside patch P's interior, or -1
  auto win_of = [&](const PatchD &P, int q) {
    const int loc = q - P.q_off, ld = P.mx + 2;
    if (loc < 0 || loc >= ld * (P.my + 2)) return -1;
    const int li = loc % ld - 1, lj = loc / ld - 1;
    if (li < 0 || li >= P.mx || lj < 0 || lj >= P.my) return -1;
    const int x = P.ilo + li - I0, y = P.jlo + lj - J0;
    return x >= 0 && x < td.wx && y >= 0 && y < td.wy ? x + y * td.wx : -1;
  };
  // the rule of the internal face `side` (0 W, 1 E, 2 S, 3 N) of cell (li, lj)
  auto rule_of = [&](const PatchD &P, int side, int li, int lj) -> const Rule & {
    return B.perim[P.pe_off + (side < 2 ? side * P.my + lj : 2 * P.my + (side - 2) * P.mx + li)];
  };
  const int dpos[4] = {-1, 1, -td.wx, td.wx};
  // needed cells, from the last pass backwards
  for (int p = kTilePasses; p >= 1; --p) {
    const int m = (kTilePasses - p) & 1 ? 1 - mA : mA;
    for (int c = t; c < W; c += kTileBuildT) {
      if (s_need[c] < p || colour(c) != m) continue;
      const PatchD &P = patch_of(c);
      int li, lj;
      local(c, P, li, lj);
      auto mark = [&](int w) {
        if (w < 0) s_bad = 1;
        else if (s_need[w] < p - 1) s_need[w] = (int8_t)(p - 1);
      };
      for (int side = 0; side < 4; ++side) {
        const bool at = side == 0 ? li == 0 : side == 1 ? li == P.mx - 1 : side == 2 ? lj == 0 : lj == P.my - 1;
        const int x = c % td.wx + (side == 0 ? -1 : side == 1), y = c / td.wx + (side == 2 ? -1 : side == 3);
        const int nb = x >= 0 && x < td.wx && y >= 0 && y < td.wy ? c + dpos[side] : -1;
        if (!at) {
          mark(nb);
          continue;
        }
        if (P.bc[side]) continue;
        const Rule &R = rule_of(P, side, li, lj);
        if (R.type == G_COPY) {
          if (nb < 0 || s_own[nb] == 0xFFFF || qidx(nb) != R.a) s_bad = 1;
          else mark(nb);
          continue;
        }
        mark(win_of(P, R.a));
        mark(win_of(P, R.b));
        // parent operands: constant during the relaxation only off the level
        const int op[3] = {R.c, R.type == G_QIF_END ? R.d : R.c, R.type == G_QIF_END ? R.e : R.c};
        for (int k = 0; k < 3; ++k)
          if (op[k] >= B.q_lo && op[k] < B.q_hi) s_bad = 1;
      }
    }
    __syncthreads();
  }
  if (kEmit) {
    for (int c = t; c < W; c += kTileBuildT) B.wq[td.wq_off + c] = s_need[c] >= 0 && s_own[c] != 0xFFFF ? qidx(c) : -1;
  } else {
    for (int c = t; c < W; c += kTileBuildT)
      if (s_need[c] >= 0) {
        atomicMin(&s_lo[0], c % td.wx);
        atomicMax(&s_hi[0], c % td.wx);
        atomicMin(&s_lo[1], c / td.wx);
        atomicMax(&s_hi[1], c / td.wx);
      }
  }
  // classes in order: per colour (the last pass's first) and group of needed
  // passes, plain and special entries, alternating so that special entries of
  // neighbouring groups meet
  const TileTab tb = B.tab[blockIdx.x];
  if (t == 0) s_base = 0;
  __syncthreads();
  int count[4 * kTileGroups + 1], faces[4 * kTileGroups + 1], nface = 0;
  for (int cls = 0; cls < 4 * kTileGroups; ++cls) {
    const int begin = s_base;
    count[cls] = begin;
    faces[cls] = nface;
    const int ccol = cls < 2 * kTileGroups ? mA : 1 - mA, cg = (cls % (2 * kTileGroups)) >> 1;
    const bool csp = ((cls & 1) ^ (cg & 1)) != 0;
    for (int c0 = 0; c0 < W; c0 += kTileBuildT) {
      const int c = c0 + t;
      bool in = false;
      int li = 0, lj = 0;
      if (c < W && s_own[c] != 0xFFFF && s_need[c] >= 1) {
        const PatchD &P = patch_of(c);
        local(c, P, li, lj);
        bool sp = false;
        for (int side = 0; side < 4; ++side) {
          const bool at = side == 0 ? li == 0 : side == 1 ? li == P.mx - 1 : side == 2 ? lj == 0 : lj == P.my - 1;
          if (at && (P.bc[side] || rule_of(P, side, li, lj).type != G_COPY)) sp = true;
        }
        // the last pass that updates the cell (its colour's at or below its
        // need), as a group: pairs of passes before the end
        const int m = (li + lj + P.par0) & 1;
        const int last = m == mA ? s_need[c] & ~1 : (s_need[c] - 1) | 1;
        const bool upd = m == mA ? last >= 2 : s_need[c] >= 1;
        const int g = m == mA ? (kTilePasses - last) >> 1 : (kTilePasses - 1 - min(last, kTilePasses - 1)) >> 1;
        in = upd && m == ccol && g == cg && sp == csp;
        const int x = c % td.wx, y = c / td.wx;   // an update reads all four neighbours' places
        if (in && (x == 0 || x == td.wx - 1 || y == 0 || y == td.wy - 1)) s_bad = 1;
      }
      const unsigned bal = __ballot_sync(0xffffffffu, in);
      if ((t & 31) == 0) s_warp[t >> 5] = __popc(bal);
      __syncthreads();
      int at = s_base + __popc(bal & ((1u << (t & 31)) - 1)), tot = 0;
      for (int k = 0; k < kTileBuildT / 32; ++k) {
        if (k < (t >> 5)) at += s_warp[k];
        tot += s_warp[k];
      }
      if (kEmit && in) {
        const int pl = td.pa + s_near[s_own[c]];
        const PatchD &P = B.patches[pl];
        const int fi = nface + (at - begin), s = (li >> 1) + lj * (P.mx >> 1);
        TileEnt e;
        e.sf = (uint32_t)c | (csp ? kTileSpecial | ((uint32_t)fi << 16) : 0u);
        e.pack = ((B.chunk0[pl] + s / kChunk) * 2 + ccol) * (kPackRows * kChunk) + s % kChunk;
        e.cell = P.c_off + li + lj * P.mx;
        e.pad = 0;
        B.ent[tb.ent + at] = e;
        if (csp) {
          TileFace F;
          for (int ax = 0; ax < 2; ++ax) {
            TileSide S{0, 0, 0, 0, 0, 0, 0, 0};
            const int pos = ax == 0 ? li : lj, n = ax == 0 ? P.mx : P.my;
            if (pos == 0 || pos == n - 1) {
              const int hi = pos == 0 ? 0 : 1, side = 2 * ax + hi;
              if (P.bc[side]) {
                S.kind = (uint16_t)P.bc[side];
                S.a = (uint16_t)(c + (ax == 0 ? 1 : td.wx) * (hi ? -1 : 1));   // the neighbour across the cell
                S.c = P.bcg_off + (ax == 0 ? hi * P.my + lj : 2 * P.my + hi * P.mx + li);
              } else {
                const Rule &R = rule_of(P, side, li, lj);
                if (R.type != G_COPY) {
                  const int step = ax == 0 ? 1 : P.mx + 2;
                  S.kind = (uint16_t)(8 + R.type);
                  S.a = (uint16_t)win_of(P, R.a);
                  S.b = (uint16_t)win_of(P, R.b);
                  S.c = R.c;
                  S.d = R.d;
                  S.e = R.e;
                  S.g = P.q_off + (li + 1) + (lj + 1) * (P.mx + 2) + (hi ? step : -step);
                }
              }
              if (S.kind && !hi) S.kind |= 0x80;
            }
            F.s[ax] = S;
          }
          B.face[tb.face + fi] = F;
        }
      }
      __syncthreads();
      if (t == 0) s_base += tot;
      __syncthreads();
    }
    if (csp) nface += s_base - begin;
  }
  count[4 * kTileGroups] = s_base;
  faces[4 * kTileGroups] = nface;
  if (t == 0) {
    if (nface > kTileFaces) s_bad = 1;
    if (s_bad) *B.bad = 1;
    if (!kEmit) {
      TileTab o{};
      o.nf = nface;
      for (int g = 0; g < kTileGroups; ++g) {
        o.nA[g] = count[2 * g + 2];
        o.nB[g] = count[2 * kTileGroups + 2 * g + 2] - count[2 * kTileGroups];
        o.fA[g] = faces[2 * g + 2];
        o.fB[g] = faces[2 * kTileGroups + 2 * g + 2] - faces[2 * kTileGroups];
      }
      o.x0 = s_lo[0];
      o.x1 = s_hi[0];
      o.y0 = s_lo[1];
      o.y1 = s_hi[1];
      B.tab[blockIdx.x] = o;
    }
  }
}

// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// shared memory of a launch: window, six operand rows of `cap` entries,
// four values per special entry, then the entries' codes, the window's Q
// indices and the special entries' side codes
template <class T>
__host__ __device__ inline size_t tile_smem(int win, int cap, int nf) {
  return sizeof(T) * ((size_t)win + 6 * (size_t)cap + 4 * (size_t)nf) +
         sizeof(uint32_t) * ((size_t)cap + win + 4 * (size_t)nf);
}

// `passes` colour passes of a level (an even number, the last one of the
// second colour) from src to dst, two copies of the level's cells; nothing
// else of either array is read or written, but with `stored` the first pass
// reads the coarse-fine ghosts stored in src, as the last fill left them.
// Five blocks per SM for FP32: left alone the compiler holds it to 32
// registers, with its loads one after the other (114,756 cells 1.71 us a pass,
// with 40 registers 1.70, with 48 1.54).  FP64 takes what it wants (ragged
// solve 2.64 ms with 70 to 88 registers or with 85, 2.68 with 64, 2.73 with 48).
template <class T, bool kPow2>
__global__ void __launch_bounds__(kTileT, sizeof(T) == 4 ? 5 : 1)
    k_relax_tile(LevelD L, const TileD *__restrict__ tiles, const TileTab *__restrict__ tab,
                 const int *__restrict__ wq, const TileEnt *__restrict__ ent, const TileFace *__restrict__ face,
                 FieldsT<T> f, const T *src, T *dst, const T *__restrict__ pack, int passes, int stored, T omega,
                 int unit_omega, int win_cap, int cap, int nf_cap) {
  extern __shared__ __align__(16) unsigned char tile_raw[];
  const int t = threadIdx.x;
  const TileD td = tiles[blockIdx.x];
  const TileTab tb = tab[blockIdx.x];
  if (!f.active[td.inst]) {
    chain_wait();
    return;
  }
  T *win = reinterpret_cast<T *>(tile_raw);
  T *op = win + win_cap;                      // rows dE dW dN dS InvDiagS F
  T *fst = op + 6 * cap;                      // special sides: constant part, ghost
  uint32_t *code = reinterpret_cast<uint32_t *>(fst + 4 * nf_cap);
  int *wqs = reinterpret_cast<int *>(code + cap);
  uint32_t *fk = reinterpret_cast<uint32_t *>(wqs + win_cap);
  const int W = td.wx * td.wy, wx = td.wx, nA = tb.nA[kTileGroups - 1], n = nA + tb.nB[kTileGroups - 1];
  // static tables and operands, before the programmatic-launch wait
  for (int c = t; c < W; c += kTileT) wqs[c] = wq[td.wq_off + c];
  for (int e = t; e < n; e += kTileT) {
    const TileEnt E = ent[tb.ent + e];
    const T *pk = pack + E.pack;
#pragma unroll
    for (int r = 0; r < kPackRows; ++r) cp_async(op + r * cap + e, pk + r * kChunk);
    code[e] = E.sf;
    *reinterpret_cast<int *>(op + kPackRows * cap + e) = E.cell;   // the force replaces it below
  }
  TileSide S0{};
  for (int i = t; i < 2 * tb.nf; i += kTileT) {
    const TileSide S = face[tb.face + (i >> 1)].s[i & 1];
    fk[2 * i] = (uint32_t)S.kind | ((uint32_t)S.a << 16);
    fk[2 * i + 1] = S.b;
    if (i == t) S0 = S;
  }
  chain_wait();
  // the window, the force and the special sides' parent values
  for (int c = t; c < W; c += kTileT) {
    const int q = wqs[c];
    if (q >= 0) cp_async(win + c, src + q);
  }
  for (int e = t; e < n; e += kTileT) {
    T *o = op + kPackRows * cap + e;
    cp_async(o, f.F + *reinterpret_cast<int *>(o));
  }
  const T A1 = T(-1.0 / 5.0), A2 = T(2.0 / 3.0), A3 = T(8.0 / 15.0);
  const T B1 = T(5.0 / 32.0), B2 = T(15.0 / 16.0), B3 = T(-3.0 / 32.0);
  const T c23 = T(2.0 / 3.0), c13 = T(1.0 / 3.0), c83 = T(8.0 / 3.0);
  const auto H = level_h(L, T(0));
  for (int i = t; i < 2 * tb.nf; i += kTileT) {
    if (i != t) S0 = face[tb.face + (i >> 1)].s[i & 1];
    const int k = S0.kind & 0x7f;
    if (k == 0) continue;
    T v;
    if (k == 1) v = c83 * f.bcg[S0.c];
    else if (k == 2) v = ((i & 1) ? H.hy : H.hx) * f.bcg[S0.c];
    else {
      if (stored) cp_async(fst + 2 * nf_cap + i, src + S0.g);
      const T qc = f.Q[S0.c];
      if (k == 8 + G_QIF) v = A3 * qc;
      else if (k == 8 + G_QIF_END) v = A3 * ((B1 * qc + B2 * f.Q[S0.d]) + B3 * f.Q[S0.e]);
      else v = c23 * qc;
    }
    fst[i] = v;
    if (k == 2) fst[2 * nf_cap + i] = v;
  }
  cp_async_wait();
  __syncthreads();
  // the ghost of special side i, which is neither a Neumann side (constant)
  // nor takes the stored ghost
  auto side = [&](int i) -> T {
    const uint32_t ka = fk[2 * i];
    const int k = ka & 0x7f;
    const T s = fst[i], qa = win[ka >> 16];
    if (k == 1) return s + c13 * qa;
    const T qb = win[fk[2 * i + 1]];
    return k == 8 + G_LIF ? (s + c23 * qa) - c13 * qb : (A1 * qa + A2 * qb) + s;
  };
  // an update
  auto update = [&](int e) {
    const uint32_t sf = code[e];
    const int c = sf & 0xffff;
    T qe = win[c + 1], qw = win[c - 1], qn = win[c + wx], qs = win[c - wx];
    T v = op[kPackRows * cap + e];
    if (sf & kTileSpecial) {
      const int fi = (sf >> 16) & (kTileFaces - 1);
#pragma unroll
      for (int ax = 0; ax < 2; ++ax) {
        const int i = 2 * fi + ax;
        const uint32_t ka = fk[2 * i];
        const int k = ka & 0x7f;
        if (k == 0) continue;
        const bool lo = (ka & 0x80) != 0;
        const T g = fst[2 * nf_cap + i];
        if (ax == 0) { if (lo) qw = g; else qe = g; }
        else { if (lo) qs = g; else qn = g; }
      }
    }
    const T dE = op[e], dW = op[cap + e], dN = op[2 * cap + e], dS = op[3 * cap + e];
    if constexpr (kPow2) {
      v = v + qe * dE;
      v = v + qw * dW;
      v = v + qn * dN;
      v = v + qs * dS;
    } else {
      T d[4] = {qe * dE, qw * dW, qn * dN, qs * dS};
      div_group<2, 4, false>(d, H.dx, H.dy);
      v = (((v + d[0]) + d[1]) + d[2]) + d[3];
    }
    v = v * op[4 * cap + e];
    if (unit_omega) win[c] = v;
    else win[c] = omega * v + (1 - omega) * win[c];
  };
#pragma unroll 1
  for (int p = kTilePasses - passes + 1; p <= kTilePasses; ++p) {
    const bool a = ((kTilePasses - p) & 1) == 0;
    const int g = (kTilePasses - p) >> 1;
    const int e0 = a ? 0 : nA;
    const int e1 = e0 + (g == 0 ? (a ? tb.nA[0] : tb.nB[0]) : g == 1 ? (a ? tb.nA[1] : tb.nB[1]) : (a ? tb.nA[2] : tb.nB[2]));
    const bool first = stored && p == kTilePasses - passes + 1;
    // the pass's special sides first, by the block's first threads together:
    // in the updates both axes' rules stood one after the other in front of
    // the chain of every warp with a special cell (5,200 to 5,800 cells in
    // patches 1.88 us a pass -> 1.54, 33,668 cells 2.40 -> 2.22; FP32 the same)
    const int f0 = a ? 0 : tb.fA[kTileGroups - 1];
    const int f1 = f0 + (g == 0 ? (a ? tb.fA[0] : tb.fB[0]) : g == 1 ? (a ? tb.fA[1] : tb.fB[1]) : (a ? tb.fA[2] : tb.fB[2]));
    if (f1 > f0) {
      for (int i = 2 * f0 + t; i < 2 * f1; i += kTileT) {
        const int k = fk[2 * i] & 0x7f;
        if (k != 0 && k != 2 && !(first && k != 1)) fst[2 * nf_cap + i] = side(i);
      }
      __syncthreads();
    }
    for (int e = e0 + t; e < e1; e += kTileT) update(e);
    __syncthreads();
  }
  for (int i = t; i < td.w * td.h; i += kTileT) {
    const int y = i / td.w, c = (td.mx + i - y * td.w) + (td.my + y) * wx;
    dst[wqs[c]] = win[c];
  }
}

}  // namespace bsam
