// step.cuh -- one whole time step of a two-dimensional grid (the x-sweep and
// the y-sweep of cliffs_main.f:317-345) in one kernel.
//
// A sweep per launch moves the state through memory twice a step: 72 bytes a
// cell, and each cell's window is loaded, classified and converted once per
// sweep.  Here a block takes a tile of 64 columns x 30 rows (StepLarge; smaller
// ones on smaller grids) with one halo row on each side (the y-sweep's), brings
// it into shared memory with tensor-map copies, sweeps its rows in place, then
// its columns out of the swept tile straight to the other copy of the state: 44
// bytes a cell, the max-wave fold included.
//
// Both sweeps march: a thread owns two lines of a sweep (two rows half a window
// apart in the x phase, two adjacent columns in the y phase) over 8 cells (4 in
// the smaller tiles) and carries the last cell and the last face's flux along,
// so that every celerity is computed 10/8 and every face flux 9/8 times a cell
// (6/4 and 5/4 in fast_kernel).  The two lines are the two halves of packed FP32 operations
// (add/sub/mul/fma.rn.f32x2): the same roundings as march.cuh's scalar ones,
// at half the issue slots.
//
// Classification.  As in sweep.cuh, a cell takes the plain update when it is
// interior and it and its neighbours are wet and subcritical; every other cell
// is left out of the thread's stores and, unless it is dry land at rest, put
// on the block's list, which its warps finish after the phase: by shore_cell
// where no cell is flooded, else by all the rules (general_cell), a warp's
// cells of the second kind together.
// The x phase's listed cells are evaluated on the step's input, in the window
// or, where the rows are swept in place, in global memory; the y phase's on the
// x-swept tile.  Tiles with a coast in them take longest and go first.
//
// Measured (us per step, replayed from graphs, against a launch per sweep;
// the same state bits): 4320 x 2160 sphere 88 from 144; 2048 x 2048 shelf 44.3
// from 68.6; 1500 x 1500 28.4 from 41.0; 1201 x 903 stretched 20.9 from 29.3;
// 1003 x 777 15.3 from 21.8; 600 x 600 11.5 from 18.4; 256 x 256 9.1 from 15.1.
// On the shelf 209 thread instructions a cell (400 in the two sweeps), 39 bytes
// a cell to and from DRAM, 16 warps an SM at 128 registers and 0.53
// instructions an SM sub-core and cycle while it is busy: what bounds it is the
// latency of the march and of the window's copies.  A small grid's step is the
// time of its slowest block: on 256 x 256 (64 threads an SM) 0.95 us for the
// window, 1.5 for the x phase, 1.8 for a coast's listed cells, 1.2 for the y
// phase and 1.2 to 3.5 for its listed cells; the code of the listed cells is
// cold in every launch, which is about a quarter of that.
//
// Tried on the shelf, from 46.5 us: the same march on one line a thread in
// scalar operations (64 registers, 32 warps) issued 271 instructions a cell at
// 0.70 and took 50.6; 96 registers and 5 blocks an SM 50.8 (spills); tiles of
// 32 columns 48.9; the max-wave update on the outputs, in the y phase, 49.5;
// later windows prefetched into L2 46.6.
#pragma once
#include "staged.cuh"

namespace cliffs {

// A tile of W columns, in a window of ROWS rows with HALO of them on each side
// (the y-sweep of a plain cell reads one, the full rules three); a thread of
// either phase marches SEG cells of two lines.  INPLACE: the rows are swept in
// place; else into fields of their own, so that the x phase's listed cells find
// their input in the window.
template <int W_, int ROWS_, int HALO_, int SEG_, bool INPLACE_>
struct StepTile {
  static constexpr int W = W_, Rows = ROWS_, Halo = HALO_, Seg = SEG_;
  static constexpr bool InPlace = INPLACE_;
  static constexpr int R = Rows - 2 * Halo;  // rows of the tile
  static constexpr int Part = (R + 3) / 4;   // rows of a thread of the y phase
  static constexpr int Pair = Rows / 2;      // rows between the two lines of an x thread
  static constexpr int Threads = Pair * (W / Seg);
  static constexpr int Blocks = 512 / Threads;  // per SM: 128 registers a thread
  // columns of the window: one 16-byte chunk on the left, two on the right (the
  // second unused): rows of an odd number of 16-byte chunks, so that the x
  // phase's accesses (2 rows x 4 segments a quarter warp) spread over the banks
  static constexpr int Win = W + 12;
  static constexpr int Field = Rows * Win;             // floats of one field of the window
  static constexpr int Out = InPlace ? 0 : 3 * Field;  // from a field of the input to the swept one
  static constexpr int Floats = (InPlace ? 4 : 7) * Field;
  static constexpr uint32_t Bytes = 4u * Field * 4u;   // of the window's copies
  static_assert(W / Seg == 8 && Threads == 2 * W, "8 segments of a row, 4 parts of a column pair");
};
using StepLarge = StepTile<64, 32, 1, 8, true>;
using StepSmall = StepTile<32, 16, 1, 4, false>;
using StepTiny = StepTile<32, 16, 3, 4, false>;

struct StepMaps {
  CUtensorMap dep, srf, xu, yv;  // the input copy's fields, a Win x Rows box
};

// ---- two FP32 lanes in a 64-bit register ---------------------------------------

using f2 = unsigned long long;

__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float lo2(f2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(f2 a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// A product that a sum takes in, as a fused operation with a zero of the sign
// that leaves every product as it is: a packed product and the packed sum after
// it come out of the compiler as one operation, and the sum's operand is to be
// rounded.  nz is a pair of -0 that the compiler does not see.
__device__ __forceinline__ f2 mulr2(f2 a, f2 b, f2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f2 both(float a) { return pk(a, a); }
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The constants of packed operations on one axis, each in both halves.  A
// phase reads them once from shared memory into registers, in a way that the
// compiler cannot repeat: made of scalars or read from the kernel's
// parameters they cost two moves at every use.  Signs are chosen so that one
// of dt and -dt, and of dtx and -dtx, is enough.
struct PairConst {
  f2 g, gcrough, mdt;   // gravity, its product with the friction coefficient, -dt
  f2 half, quarter, nz;  // 1/2, 1/4, -0 (mulr2)
  f2 inv, ndtx, ndfpm;  // a uniform axis: 1/dx, -dt/(2 dx), 0
};

__device__ __forceinline__ f2 ld_const(const f2* p) {
  f2 r;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r) : "r"(smem_u32(p)));
  return r;
}
__device__ __forceinline__ PairConst load_const(const PairConst* p) {
  PairConst k;
  k.g = ld_const(&p->g);
  k.gcrough = ld_const(&p->gcrough);
  k.mdt = ld_const(&p->mdt);
  k.half = ld_const(&p->half);
  k.quarter = ld_const(&p->quarter);
  k.nz = ld_const(&p->nz);
  k.inv = ld_const(&p->inv);
  k.ndtx = ld_const(&p->ndtx);
  k.ndfpm = ld_const(&p->ndfpm);
  return k;
}

struct PairPair {
  PairConst x, y;
};

struct StepCtl {
  unsigned long long wait_ns;  // limit of the window's wait
  unsigned extra;              // bytes it waits for beyond its copies: 0, except in the timeout self-test
  int flip;                    // last to first: bands, or a batch's tiles without a coast
  int coast;                   // a batch's tiles with one, at the front of the order
};

// rsqrtf for arguments that are not subnormal (celerities: g * max(H, ground);
// speeds: max(., 1e-30); depths of wet cells): the same value without its
// scaling of subnormal arguments.
__device__ __forceinline__ float rsq(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// A cell of both lines as the march sees it.
struct Cell2 {
  f2 u, v, c, e;     // normal and tangential velocity, celerity, eta
  f2 cc;             // friction (cliffs.f:204); not set on halo cells
  float s[2], H[2];  // surface state, total depth
};

// Geometry kinds of an axis: uniform spacing alone; uniform spacing with a row
// factor (x) or a metric term (y), as on a sphere; spacing from the table, with
// either.
enum { GEO_SCL = 1, GEO_DFPM = 2, GEO_FLAT = 0, GEO_METRIC = GEO_SCL, GEO_TABLE = GEO_SCL | GEO_DFPM };

// Geometry of one position on both lines.
struct Geo2 {
  f2 inv;    // 1/dx of the face on the cell's right
  f2 ndtx;   // -dt/(fm+fp) of the cell
  f2 ndfpm;  // fm - fp of the cell
  f2 scl8;   // 8 times the metric term of the cell
};

// What the march carries from cell to cell: the last cell, the tangential
// velocity of the one before, and the last face's scaled fluxes.
struct March {
  Cell2 j;
  f2 va;      // tangential velocity of the cell before j
  f2 qP, qQ;  // FP/dx, FQ/dx of the face on j's left
  f2 nqv;     // (v_a - v_j)/dx there
};

// HALO: a cell that is only a neighbour.
template <bool HALO = false>
__device__ __forceinline__ Cell2 make_cell2(const Phys<float>& p, const PairConst& K, float d0, float d1, float s0,
                                            float s1, float u0, float u1, float v0, float v1) {
  Cell2 n;
  n.s[0] = s0;
  n.s[1] = s1;
  n.H[0] = add_rn(s0, fmaxf(d0, 0.f));
  n.H[1] = add_rn(s1, fmaxf(d1, 0.f));
  n.e = pk(sub_rn(s0, fminf(d0, 0.f)), sub_rn(s1, fminf(d1, 0.f)));
  const f2 x = mul2(pk(fmaxf(n.H[0], p.ground), fmaxf(n.H[1], p.ground)), K.g);
  n.c = mulr2(x, pk(rsq(lo2(x)), rsq(hi2(x))), K.nz);
  n.u = pk(u0, u1);
  n.v = pk(v0, v1);
  n.cc = 0ull;
  if (!HALO) {
    const f2 w = fma2(n.u, n.u, mul2(n.v, n.v));
    const f2 r = pk(rsq(n.H[0]), rsq(n.H[1]));
    const f2 sp = mul2(w, pk(rsq(fmaxf(lo2(w), 1e-30f)), rsq(fmaxf(hi2(w), 1e-30f))));
    n.cc = mulr2(mul2(mul2(n.u, K.gcrough), sp), mul2(mul2(r, r), r), K.nz);
  }
  return n;
}

// The scaled fluxes of the face between j and the next cell b (face_flux).
__device__ __forceinline__ void face2(const Cell2& j, const Cell2& b, const PairConst& K, f2 inv, f2& qP, f2& qQ) {
  const f2 U = add2(j.u, b.u), C = add2(j.c, b.c), du = sub2(b.u, j.u), dc = sub2(b.c, j.c);
  const f2 gde = mulr2(sub2(b.e, j.e), K.g, K.nz);
  const f2 Udc = mulr2(U, dc, K.nz);
  const f2 FP = fma2(mul2(add2(U, C), K.half), du, add2(gde, Udc));
  const f2 FQ = fma2(mul2(sub2(U, C), K.half), du, sub2(gde, Udc));
  qP = mulr2(FP, inv, K.nz);
  qQ = mulr2(FQ, inv, K.nz);
}

// The plain update (interior_update<float, false, SPH>) of the march's cell j,
// with the fluxes qP, qQ of its right face and the next cell's tangential
// velocity vb: new surface state, velocities and celerity of both lines.
template <int G>
__device__ __forceinline__ void update2(const March& m, f2 vb, f2 qP, f2 qQ, const Geo2& g, float ginv,
                                        const PairConst& K, float (&os)[2], f2& ou, f2& ov, f2& cn) {
  const f2 u = m.j.u, v = m.j.v, c = m.j.c;
  const f2 ejP = add2(u, c), ejQ = sub2(u, c);
  f2 QsP = mul2(add2(qP, m.qP), K.half);
  f2 QsQ = mul2(add2(qQ, m.qQ), K.half);
  QsP = fma2(mul2(ejP, g.ndtx), sub2(qP, m.qP), QsP);
  QsQ = fma2(mul2(ejQ, g.ndtx), sub2(qQ, m.qQ), QsQ);
  f2 qcP = add2(QsP, m.j.cc), qcQ = add2(QsQ, m.j.cc);
  if (G & GEO_SCL) {
    // 8 c u scl: the factor 8 is exact wherever it stands
    const f2 sphr = mulr2(mul2(c, u), g.scl8, K.nz);
    qcP = sub2(qcP, sphr);
    qcQ = add2(qcQ, sphr);
  }
  const f2 dP = mulr2(qcP, K.mdt, K.nz), dQ = mulr2(qcQ, K.mdt, K.nz);
  const f2 Qv = fma2(sub2(vb, v), g.inv, m.nqv);
  const f2 nx = (G & GEO_DFPM) ? fma2(u, K.mdt, g.ndfpm) : mul2(u, K.mdt);  // -(u dt + fp - fm)
  const f2 vx = fma2(Qv, nx, sub2(vb, m.va));
  ov = fma2(mul2(u, g.ndtx), vx, v);
  const f2 dc = mul2(sub2(dP, dQ), K.quarter);
  cn = add2(c, dc);
  ou = fma2(add2(dP, dQ), K.half, u);
  // state_step of a wet cell that stays wet (cn > 0: the caller checks)
  const f2 t = mul2(dc, add2(add2(c, c), dc));
  os[0] = fma_rn(lo2(t), ginv, m.j.s[0]);
  os[1] = fma_rn(hi2(t), ginv, m.j.s[1]);
}

// The sign bit set where a cell is wet, and where it is supercritical.
__device__ __forceinline__ unsigned wet_sign(float H, const Phys<float>& p) {
  return __float_as_uint(sub_rn(p.ground, H));
}
__device__ __forceinline__ unsigned sup_sign(float u, float c) { return __float_as_uint(sub_rn(c, fabsf(u))); }
// A bit mask that takes in a sign bit: the newest cell at bit 0.
__device__ __forceinline__ unsigned take_sign(unsigned mask, unsigned x) { return __funnelshift_l(x, mask, 1); }

// ---- the cells that need the full rules ------------------------------------------

// The value of line cell o where no flooding is in play: the cell and its two
// neighbours are each either wet or stay land, so the cell becomes new land
// (whatever its neighbours do), or takes its edge rule or the interior update
// with mirror images in place of land neighbours (general_cell without its
// flooding and limiter, which act on flooded cells only).  w: the raw cells
// o-2 .. o+2; the outer two matter only to a wet cell, beside a land
// neighbour.  Returns false when general_cell has to decide: the cell or a
// neighbour of it is flooded, or a remainder of water or velocity lies on land
// with no wet cell in reach.
__device__ __forceinline__ bool shore_cell(const RawCell<float>* w, int o, int n, const LineCtx<float>& C,
                                           const Geo<float>& g, const Phys<float>& p, OutCell<float>& out) {
  float H[5], E[5];
  bool wet[5];
  bool anywet = false;
#pragma unroll
  for (int t = 0; t < 5; ++t) {
    H[t] = depth_of(w[t].s, w[t].d);
    E[t] = eta_of(w[t].s, w[t].d);
    wet[t] = w[t].present && H[t] > p.ground;
    anywet |= wet[t];
  }
  bool flooded = false;
#pragma unroll
  for (int t = 1; t <= 3; ++t) {
    const bool fr = wet[t - 1] && w[t - 1].u >= 0.f && E[t - 1] + w[t].d > p.ground;
    const bool fl = wet[t + 1] && w[t + 1].u <= 0.f && E[t + 1] + w[t].d > p.ground;
    flooded |= w[t].present && !wet[t] && (t == 2 || wet[2]) && (fr || fl);
  }
  if (flooded) return false;
  if (!wet[2]) {
    if (!anywet && !(H[2] == 0.f && w[2].u == 0.f && w[2].v == 0.f)) return false;
    out = OutCell<float>{state_from_depth(0.f, w[2].d), 0.f, 0.f};
    return true;
  }
  CellState<float> f[3];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const RawCell<float>& r = w[t + 1];
    const float h = H[t + 1];
    f[t] = CellState<float>{r.u, fsqrt_pos(p.g * (h > p.ground ? h : p.ground)), E[t + 1], r.d, r.v, h};
  }
  const CellState<float>& j = f[1];
  if (o == 1 || o == n) {
    out = OutCell<float>{w[2].s, w[2].u, w[2].v};
    const EdgeVals<float>& e = o == 1 ? C.eL : C.eR;
    if (!(o == 1 ? wet[3] : wet[1]) || !(e.eta + j.d > p.ground)) return true;
    float cn;
    if (o == 1)
      edge_left(j, f[2], e, C.inv_dx1, C.scl1, p, cn, out.u, out.v, out.s);
    else
      edge_right(f[0], j, e, C.inv_dxn1, C.scln, p, cn, out.u, out.v, out.s);
    return true;
  }
  const CellState<float> mir{-j.u, j.c, j.e, j.d, j.v, j.H};
  const CellState<float> a = wet[1] ? f[0] : mir, b = wet[3] ? f[2] : mir;
  float FPl, FQl, FPr, FQr, cn;
  face_flux(a.u, a.c, a.e, j.u, j.c, j.e, p, FPl, FQl);
  face_flux(j.u, j.c, j.e, b.u, b.c, b.e, p, FPr, FQr);
  out = interior_update(a, j, b, FPl, FQl, FPr, FQr, g, p, &cn);
  return true;
}

// All the rules on the step's input in global memory.
__device__ __noinline__ OutCell<float> step_x_general(const SweepArgs& X, int L, int i) {
  return general_value<0, false>(X, L, i);
}

// A cell's value, unless all the rules have to decide (ok false).
struct XValue {
  OutCell<float> out;
  bool ok;
};

// The constants of row L that the rules at and beside cell i need.
__device__ __forceinline__ LineCtx<float> x_line(const SweepArgs& X, int L, int i, float& alpha, float& ialpha) {
  alpha = ialpha = 1.f;
  if (X.lscale) {
    const float2 a = __ldg(X.lscale + (L - 1));
    alpha = a.x;
    ialpha = a.y;
  }
  LineCtx<float> C;
  C.n = X.n;
  C.eL = i == 1 ? edge_vals(X, L, 0) : EdgeVals<float>{0.f, 0.f, 0.f};
  C.eR = i == X.n ? edge_vals(X, L, 1) : EdgeVals<float>{0.f, 0.f, 0.f};
  C.inv_dx1 = X.inv_dx1 * ialpha;
  C.inv_dxn1 = X.inv_dxn1 * ialpha;
  C.scl1 = C.scln = 0.f;
  return C;
}

// The x-swept value of grid cell (row L, column i), 1-based, from the step's
// input in global memory, where no flooding is in play.
__device__ __noinline__ XValue step_x_shore(const SweepArgs& X, int L, int i) {
  const int n = X.n;
  XValue r;
  RawCell<float> w[5];
#pragma unroll
  for (int t = 0; t < 5; ++t) {
    const int k = i - 2 + t;
    w[t] = RawCell<float>{0.f, 0.f, 0.f, 0.f, false};
    if (k >= 1 && k <= n) {
      const size_t q = cidx<0>(L, k, X.pitch);
      w[t] = RawCell<float>{__ldg(X.dep + q), ld_state<false>(X.srf + q), ld_state<false>(X.xu + q),
                            ld_state<false>(X.yv + q), true};
    }
  }
  r.out = OutCell<float>{w[2].s, w[2].u, w[2].v};
  r.ok = true;
  if (L < X.lo || L > X.hi) return r;  // a row that is not swept
  float alpha, ialpha;
  const LineCtx<float> C = x_line(X, L, i, alpha, ialpha);
  r.ok = shore_cell(w, i, n, C, geo_at(X, i, alpha, ialpha), X.ph, r.out);
  return r;
}

// The same by whichever rules it takes.
__device__ __forceinline__ OutCell<float> step_x_value(const SweepArgs& X, int L, int i) {
  const XValue r = step_x_shore(X, L, i);
  return r.ok ? r.out : step_x_general(X, L, i);
}

// Whether the x-swept cell (row L, column i) is wet.  A dry cell between dry
// neighbours stays dry without an evaluation.
__device__ __forceinline__ bool step_x_wet(const SweepArgs& X, int L, int i) {
  float d[3], s[3];
#pragma unroll
  for (int t = 0; t < 3; ++t) {  // all loads at once; at a line's end the end twice
    const size_t q = cidx<0>(L, min(max(i - 1 + t, 1), X.n), X.pitch);
    d[t] = __ldg(X.dep + q);
    s[t] = ld_state<false>(X.srf + q);
  }
  bool any = false;
#pragma unroll
  for (int t = 0; t < 3; ++t) any |= depth_of(s[t], d[t]) > X.ph.ground;
  return any && depth_of(step_x_value(X, L, i).s, d[1]) > X.ph.ground;
}

// The constants of column L that the rules at and beside cell o need.
__device__ __forceinline__ LineCtx<float> y_line(const SweepArgs& Y, int L, int o) {
  LineCtx<float> C;
  C.n = Y.n;
  C.wet = true;
  C.eL = o == 1 ? edge_vals(Y, L, 0) : EdgeVals<float>{0.f, 0.f, 0.f};
  C.eR = o == Y.n ? edge_vals(Y, L, 1) : EdgeVals<float>{0.f, 0.f, 0.f};
  C.inv_dx1 = Y.inv_dx1;
  C.inv_dxn1 = Y.inv_dxn1;
  C.scl1 = Y.scl ? Y.scl[0] : 0.f;
  C.scln = Y.scl ? Y.scl[Y.n - 1] : 0.f;
  return C;
}

// Cell `at` of the window sm, column k of the grid, as the x-sweep reads it.
template <class T>
__device__ __forceinline__ RawCell<float> step_x_raw(const float* sm, int at, int k, int n) {
  const float* f = sm + at;
  return RawCell<float>{f[0], f[T::Field], f[2 * T::Field], f[3 * T::Field], k >= 1 && k <= n};
}

// The tile cell (t, c) of the x phase from the step's input in the window,
// where no flooding is in play.
template <class T>
__device__ __noinline__ XValue step_x_window_shore(const SweepArgs& X, const float* sm, int rb, int c0, int t, int c) {
  const int L = rb + t, i = c0 + c + 1, n = X.n;
  RawCell<float> w[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) w[q] = step_x_raw<T>(sm, t * T::Win + 2 + c + q, i - 2 + q, n);
  float alpha, ialpha;
  const LineCtx<float> C = x_line(X, L, i, alpha, ialpha);
  XValue r;
  r.ok = shore_cell(w, i, n, C, geo_at(X, i, alpha, ialpha), X.ph, r.out);
  return r;
}

// And by all the rules.
template <class T>
__device__ __noinline__ OutCell<float> step_x_window_full(const SweepArgs& X, const float* sm, int rb, int c0, int t,
                                                          int c) {
  const int L = rb + t, i = c0 + c + 1, n = X.n;
  RawCell<float> w[7];
  bool anywet = false;
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    w[q] = step_x_raw<T>(sm, t * T::Win + 1 + c + q, i - 3 + q, n);
    anywet |= w[q].present && depth_of(w[q].s, w[q].d) > X.ph.ground;
  }
  if (!anywet) return step_x_general(X, L, i);  // does the row hold a wet cell elsewhere?
  float alpha, ialpha;
  LineCtx<float> C = x_line(X, L, i, alpha, ialpha);
  C.wet = anywet;
  Geo<float> g[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) g[q] = geo_at(X, i - 1 + q, alpha, ialpha);
  return general_cell(w, i, C, g, X.ph);
}

// The x-swept cell (row k, column L) outside the window: swept again from the
// step's input.
__device__ __noinline__ RawCell<float> step_y_outside(const SweepArgs& X, int k, int L) {
  const OutCell<float> x = step_x_value(X, k, L);
  return RawCell<float>{__ldg(X.dep + cidx<0>(k, L, X.pitch)), x.s, x.v, x.u, true};
}

// The x-swept cell (t, c) of the window sm, as the y-sweep reads it.
template <class T>
__device__ __forceinline__ RawCell<float> step_y_raw(const float* sm, int t, int c) {
  const float* f = sm + t * T::Win + 4 + c;
  return RawCell<float>{f[0], f[T::Field + T::Out], f[3 * T::Field + T::Out], f[2 * T::Field + T::Out], true};
}

struct YValue {
  OutCell<float> out;
  bool scan;  // the column's wet scan has to decide
};

// The y-swept value of tile cell (t, c) (row rb + t, column c0 + c + 1, 1-based)
// from the x-swept window sm, unless a flooded cell, a remainder on land or a
// cell outside the window has a say in it.
template <class T>
__device__ __noinline__ XValue step_y_shore(const SweepArgs& Y, const float* sm, int rb, int c0, int t, int c) {
  const int o = rb + t, L = c0 + c + 1, n = Y.n;
  const float ground = Y.ph.ground;
  RawCell<float> w[5];
  bool have[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const int k = o - 2 + q, tt = t - 2 + q;
    w[q] = RawCell<float>{0.f, 0.f, 0.f, 0.f, false};
    have[q] = k < 1 || k > n || (tt >= 0 && tt < T::Rows);
    if (k >= 1 && k <= n && have[q]) w[q] = step_y_raw<T>(sm, tt, c);
  }
  XValue r;
  r.out = OutCell<float>{0.f, 0.f, 0.f};
  // a cell two rows away and outside the window matters to a wet cell beside a
  // land neighbour, and to a remainder on land
  const bool rest = w[2].u == 0.f && w[2].v == 0.f && depth_of(w[2].s, w[2].d) == 0.f;
  r.ok = false;
  if (!have[0] && !rest && !(depth_of(w[1].s, w[1].d) > ground)) return r;
  if (!have[4] && !rest && !(depth_of(w[3].s, w[3].d) > ground)) return r;
  const LineCtx<float> C = y_line(Y, L, o);
  r.ok = shore_cell(w, o, n, C, geo_at(Y, o, 1.f, 1.f), Y.ph, r.out);
  return r;
}

// The same by all the rules, from cells o-3 .. o+3.  pair: by two lanes, for cells
// in the tile's first and last rows: at most two of the cells lie outside the
// window, on one side of it, and each lane sweeps one of them again (one lane
// sweeping both, the few blocks with a flooded cell there ended 4 to 9 us after
// the others and held up the step).  Both lanes have the value.  The whole warp
// calls it, with the same `pair`; on: the lane (its pair) has a cell.
template <class T>
__device__ __noinline__ YValue step_y_full(const SweepArgs& X, const SweepArgs& Y, const float* sm, int rb, int c0,
                                           bool pair, bool on, int t, int c) {
  static_assert(T::Halo >= 1 && (T::Halo >= 3 || T::R >= 4), "at most two cells outside");
  const int o = rb + t, L = c0 + c + 1, n = Y.n, odd = (int)(threadIdx.x & 1);
  const float ground = Y.ph.ground;
  // above the window: rows t - 3, t - 2; below: t + 2, t + 3
  const bool above = t < 3;
  RawCell<float> mine{0.f, 0.f, 0.f, 0.f, false};
  if (T::Halo < 3 && pair) {
    const int tt = above ? t - 3 + odd : t + 2 + odd, k = rb + tt;
    if (on && (tt < 0 || tt >= T::Rows) && k >= 1 && k <= n) mine = step_y_outside(X, k, L);
    __syncwarp();
  }
  LineCtx<float> C = y_line(Y, L, o);
  Geo<float> g[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) g[q] = geo_at(Y, o - 1 + q, 1.f, 1.f);
  RawCell<float> w[7];
#pragma unroll
  for (int q = 0; q < 7; ++q) {
    const int k = o - 3 + q, tt = t - 3 + q;
    w[q] = RawCell<float>{0.f, 0.f, 0.f, 0.f, false};
    if (k >= 1 && k <= n && tt >= 0 && tt < T::Rows) w[q] = step_y_raw<T>(sm, tt, c);
  }
  if (T::Halo < 3 && pair) {
    RawCell<float> its;
    its.d = __shfl_xor_sync(0xffffffffu, mine.d, 1);
    its.s = __shfl_xor_sync(0xffffffffu, mine.s, 1);
    its.u = __shfl_xor_sync(0xffffffffu, mine.u, 1);
    its.v = __shfl_xor_sync(0xffffffffu, mine.v, 1);
    its.present = __shfl_xor_sync(0xffffffffu, (int)mine.present, 1);
    const RawCell<float> first = odd ? its : mine, second = odd ? mine : its;
    if (above && first.present) w[0] = first;
    if (above && second.present) w[1] = second;
    if (!above && first.present) w[5] = first;
    if (!above && second.present) w[6] = second;
  }
  bool anywet = false;
#pragma unroll
  for (int q = 0; q < 7; ++q) anywet |= w[q].present && depth_of(w[q].s, w[q].d) > ground;
  YValue r;
  r.out = OutCell<float>{w[3].s, w[3].u, w[3].v};
  r.scan = false;
  if (!on) return r;
  const bool rest = w[3].u == 0.f && w[3].v == 0.f && depth_of(w[3].s, w[3].d) == 0.f;
  if (!anywet && !rest) {  // whether its column holds a wet cell elsewhere decides (cliffs.f:113)
    // in the window first (rows outside the grid hold no water): a beach that a wave
    // has left has such cells in every step, and the one block that looked through
    // its column took a 600 x 600 step from 14.5 to 20.5 us
#pragma unroll 4
    for (int tt = 0; tt < T::Rows; ++tt) {
      const RawCell<float> x = step_y_raw<T>(sm, tt, c);
      anywet |= depth_of(x.s, x.d) > ground;
    }
    if (!anywet) {
      r.scan = true;
      return r;
    }
  }
  C.wet = anywet;
  r.out = general_cell(w, o, C, g, Y.ph);
  return r;
}

__device__ __forceinline__ void courant_status(const SweepArgs& A, float cour) {
  if (__any_sync(0xffffffffu, cour > 0.5f)) {
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(2.f * cour));
    if ((threadIdx.x & 31) == 0) {
      atomicOr(A.status, ST_CFL);
      atomicMax(A.status + 1, m);
    }
  }
}

// ---- the x phase ------------------------------------------------------------------

// Numbers that lanes of a warp leave behind, to be taken 16 or 32 at a time by
// lanes next to each other.  The whole warp calls each of the functions.
struct WarpQueue {
  uint16_t* q;     // 64 places in shared memory
  unsigned n = 0;  // how many are taken

  __device__ __forceinline__ void push(bool want, unsigned v) {  // n <= 32
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (want) q[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = (uint16_t)v;
    n += __popc(m);
    __syncwarp();
  }
  __device__ __forceinline__ bool peek(unsigned k, unsigned& v) const {  // the k-th
    v = k < n ? q[k] : 0u;
    return k < n;
  }
  __device__ __forceinline__ void take(WarpQueue& o) {  // all of o, at most 32
    if ((threadIdx.x & 31) < o.n) q[n + (threadIdx.x & 31)] = o.q[threadIdx.x & 31];
    n += o.n;
    o.n = 0u;
    __syncwarp();
  }
  __device__ __forceinline__ void pop(unsigned k) {  // the first k, or all
    const unsigned left = n > k ? n - k : 0u, lane = threadIdx.x & 31;
    const uint16_t v = lane < left ? q[k + lane] : (uint16_t)0;
    __syncwarp();
    if (lane < left) q[lane] = v;
    n = left;
    __syncwarp();
  }
};

// Appends the entries first + (bits of mask) to the block's list.
__device__ __forceinline__ void list_push(unsigned mask, unsigned first, uint16_t* s_list, unsigned* s_n) {
  if (!mask) return;
  unsigned at = atomicAdd(s_n, (unsigned)__popc(mask));
  for (; mask; mask &= mask - 1u) s_list[at++] = (uint16_t)(first + (unsigned)(__ffs(mask) - 1));
}

// Land at rest between dry cells: a cell that stays as it is.  near: the wet
// bits of the cell and its neighbours.
__device__ __forceinline__ bool at_rest(unsigned near, float H, float u, float v) {
  return (near & 7u) == 0u && H == 0.f && u == 0.f && v == 0.f;
}

template <class T, int GX>
__device__ __forceinline__ void step_x_phase(const SweepArgs& X, const PairConst* sK, float* sm, int rb, int c0,
                                             uint16_t* s_list, unsigned* s_n, bool& bad) {
  const Phys<float> p = X.ph;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a quarter warp takes 4 segments of 2 neighbouring rows; the warp, all
  // segments of its rows
  const int q4 = lane >> 3;
  const int seg = (lane & 3) | (q4 & 1) * 4;
  const int tA = warp * 4 + (q4 >> 1) * 2 + ((lane >> 2) & 1), tB = tA + T::Pair;
  const int n = X.n, k0 = c0 + T::Seg * seg + 1;
  float* rowA = sm + tA * T::Win + 4 + T::Seg * seg;
  float* rowB = rowA + T::Pair * T::Win;
  // the halo cells, before a neighbouring segment's results replace them
  float hl[8], hr[8];
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    hl[2 * f] = rowA[f * T::Field - 1];
    hl[2 * f + 1] = rowB[f * T::Field - 1];
    hr[2 * f] = rowA[f * T::Field + T::Seg];
    hr[2 * f + 1] = rowB[f * T::Field + T::Seg];
  }
  if (T::InPlace) __syncwarp();
  const int LA = rb + tA, LB = rb + tB;  // 1-based rows
  const bool swA = LA >= X.lo && LA <= X.hi && k0 <= n, swB = LB >= X.lo && LB <= X.hi && k0 <= n;
  float cour = 0.f;
  if (swA || swB) {
    const PairConst K = load_const(sK);
    f2 al = 0ull, ial = 0ull;  // row factors
    Geo2 g{K.inv, K.ndtx, 0ull, 0ull};
    if (GX != GEO_FLAT) {
      float2 a = make_float2(1.f, 1.f), b = a;
      if (X.lscale) {
        a = __ldg(X.lscale + min(max(LA, X.lo), X.hi) - 1);
        b = __ldg(X.lscale + min(max(LB, X.lo), X.hi) - 1);
      }
      al = pk(a.x, b.x);
      ial = pk(a.y, b.y);
      g.inv = mul2(K.inv, ial);
      g.ndtx = mul2(K.ndtx, ial);
    }
    // sign bits of the cells taken in, the newest at bit 0
    unsigned wetA = 0u, wetB = 0u, okA = 0u, okB = 0u;
    unsigned restA = 0u, restB = 0u;  // listed cells: cell i at bit i
    float cmA = 0.f, cmB = 0.f;       // the largest |u| + c of each line (times dt/(fm+fp) with GEO_TABLE)
    f2 chk = 0ull;                    // 0 * results: NaN when one is not finite
    // every cell of the segment interior, on swept rows
    const bool inner = swA && swB && k0 >= 2 && k0 + T::Seg - 1 <= n - 1;
    March m;
    auto flags = [&](const Cell2& c) {
      const unsigned a = wet_sign(c.H[0], p), b = wet_sign(c.H[1], p);
      wetA = take_sign(wetA, a);
      wetB = take_sign(wetB, b);
      okA = take_sign(okA, a & ~sup_sign(lo2(c.u), lo2(c.c)));
      okB = take_sign(okB, b & ~sup_sign(hi2(c.u), hi2(c.c)));
    };
    // the scaled fluxes of the face between m.j and the cell b at position k
    auto face = [&](const Cell2& b, int k, f2& inv, f2& qP, f2& qQ) {
      inv = g.inv;
      if (GX == GEO_TABLE) {
        // 1/dx(k-1): the table's left spacing of k or right spacing of k-1
        // (the ends of the line have no entry)
        const float x = k >= 2 && k <= n - 1 ? __ldg(X.geo + (k - 1)).x : (k == n ? __ldg(X.geo + (n - 2)).y : 0.f);
        inv = mul2(both(x), ial);
      }
      face2(m.j, b, K, inv, qP, qQ);
    };
    auto take = [&](const Cell2& b, f2 inv, f2 qP, f2 qQ) {
      m.nqv = mul2(sub2(m.j.v, b.v), inv);
      m.qP = qP;
      m.qQ = qQ;
      m.va = m.j.v;
      m.j = b;
    };
    // finishes cell i = m.j, with cell i + 1, and goes on to that one
    auto advance = [&](const Cell2& b, int i) {
      f2 inv, qP, qQ;
      face(b, k0 + i + 1, inv, qP, qQ);
      Geo2 gk = g;
      if (GX == GEO_TABLE) {
        const float4 q = __ldg(X.geo + (min(k0 + i, n) - 1));
        gk.inv = inv;
        gk.ndtx = mul2(both(-q.z), ial);
        gk.ndfpm = mul2(both(-q.w), al);
      }
      float os[2];
      f2 ou, ov, cn;
      update2<GX & GEO_DFPM>(m, b.v, qP, qQ, gk, p.ginv, K, os, ou, ov, cn);
      flags(b);
      float *const fA = rowA + T::Out + i, *const fB = rowB + T::Out + i;
      if ((okA & okB & 7u) == 7u && inner && fminf(lo2(cn), hi2(cn)) > 0.f) {
        fA[T::Field] = os[0];
        fA[2 * T::Field] = lo2(ou);
        fA[3 * T::Field] = lo2(ov);
        fB[T::Field] = os[1];
        fB[2 * T::Field] = hi2(ou);
        fB[3 * T::Field] = hi2(ov);
        chk = fma2(pk(os[0], os[1]), 0ull, fma2(ou, 0ull, fma2(ov, 0ull, chk)));
      } else {
        const int k = k0 + i;
        const bool in = k >= 2 && k <= n - 1;
        const bool pA = in && swA && (okA & 7u) == 7u && lo2(cn) > 0.f;
        const bool pB = in && swB && (okB & 7u) == 7u && hi2(cn) > 0.f;
        // rows that are not swept and land at rest keep their input, which
        // is in place or copied; the others are listed
        const bool kA = !swA || at_rest(wetA, m.j.H[0], lo2(m.j.u), lo2(m.j.v));
        const bool kB = !swB || at_rest(wetB, m.j.H[1], hi2(m.j.u), hi2(m.j.v));
        const bool wA = pA || (!T::InPlace && kA), wB = pB || (!T::InPlace && kB);
        const float s0 = pA ? os[0] : m.j.s[0], u0 = pA ? lo2(ou) : lo2(m.j.u), v0 = pA ? lo2(ov) : lo2(m.j.v);
        const float s1 = pB ? os[1] : m.j.s[1], u1 = pB ? hi2(ou) : hi2(m.j.u), v1 = pB ? hi2(ov) : hi2(m.j.v);
        if (wA) {
          fA[T::Field] = s0;
          fA[2 * T::Field] = u0;
          fA[3 * T::Field] = v0;
        }
        if (wB) {
          fB[T::Field] = s1;
          fB[2 * T::Field] = u1;
          fB[3 * T::Field] = v1;
        }
        // a finite sum of the results (0 where none is)
        const float z = (pA ? s0 + u0 + v0 : 0.f) * 0.f + (pB ? s1 + u1 + v1 : 0.f) * 0.f;
        bad = bad || z != z;
        if (k <= n) {
          restA |= (pA || kA ? 0u : 1u) << i;
          restB |= (pB || kB ? 0u : 1u) << i;
        }
      }
      float a = add_rn(fabsf(lo2(m.j.u)), lo2(m.j.c)), c = add_rn(fabsf(hi2(m.j.u)), hi2(m.j.c));
      if (GX == GEO_TABLE) {
        a *= -lo2(gk.ndtx);
        c *= -hi2(gk.ndtx);
      }
      cmA = fmaxf(cmA, a);
      cmB = fmaxf(cmB, c);
      take(b, inv, qP, qQ);
    };
    // Cells i and i + 1 of both rows at once.  The next cell is made ready
    // while one is finished: its square roots do not depend on the march, and
    // hide the latency of the chain from face to update.
    struct Two {
      float2 d[2], s[2], u[2], v[2];
    };
    auto load = [&](int i) {
      Two t;
      t.d[0] = *reinterpret_cast<const float2*>(rowA + i);
      t.d[1] = *reinterpret_cast<const float2*>(rowB + i);
      t.s[0] = *reinterpret_cast<const float2*>(rowA + T::Field + i);
      t.s[1] = *reinterpret_cast<const float2*>(rowB + T::Field + i);
      t.u[0] = *reinterpret_cast<const float2*>(rowA + 2 * T::Field + i);
      t.u[1] = *reinterpret_cast<const float2*>(rowB + 2 * T::Field + i);
      t.v[0] = *reinterpret_cast<const float2*>(rowA + 3 * T::Field + i);
      t.v[1] = *reinterpret_cast<const float2*>(rowB + 3 * T::Field + i);
      return t;
    };
    auto first = [&](const Two& t) {
      return make_cell2(p, K, t.d[0].x, t.d[1].x, t.s[0].x, t.s[1].x, t.u[0].x, t.u[1].x, t.v[0].x, t.v[1].x);
    };
    auto second = [&](const Two& t) {
      return make_cell2(p, K, t.d[0].y, t.d[1].y, t.s[0].y, t.s[1].y, t.u[0].y, t.u[1].y, t.v[0].y, t.v[1].y);
    };
    Cell2 b;  // the cell after m.j
    {
      m.j = make_cell2<true>(p, K, hl[0], hl[1], hl[2], hl[3], hl[4], hl[5], hl[6], hl[7]);
      flags(m.j);
      const Two t = load(0);
      const Cell2 j = first(t);
      b = second(t);
      f2 inv, qP, qQ;
      face(j, k0, inv, qP, qQ);
      flags(j);
      take(j, inv, qP, qQ);
    }
#pragma unroll 1
    for (int i = 0; i < T::Seg - 2; i += 2) {
      const Two t = load(i + 2);
      const Cell2 c = first(t);
      advance(b, i);
      b = second(t);
      advance(c, i + 1);
    }
    const Cell2 h = make_cell2<true>(p, K, hr[0], hr[1], hr[2], hr[3], hr[4], hr[5], hr[6], hr[7]);
    advance(b, T::Seg - 2);
    advance(h, T::Seg - 1);
    bad = bad || (swA && lo2(chk) != lo2(chk)) || (swB && hi2(chk) != hi2(chk));
    list_push(restA, tA * T::W + T::Seg * seg, s_list, s_n);
    list_push(restB, tB * T::W + T::Seg * seg, s_list, s_n);
    if (GX != GEO_TABLE) {
      cmA *= -lo2(g.ndtx);
      cmB *= -hi2(g.ndtx);
    }
    cour = fmaxf(swA ? cmA : 0.f, swB ? cmB : 0.f);
  } else if (!T::InPlace) {
#pragma unroll
    for (int f = 1; f < 4; ++f)
#pragma unroll
      for (int i = 0; i < T::Seg; ++i) {
        rowA[f * T::Field + T::Out + i] = rowA[f * T::Field + i];
        rowB[f * T::Field + T::Out + i] = rowB[f * T::Field + i];
      }
  }
  courant_status(X, cour);
}

// ---- the y phase ------------------------------------------------------------------

template <class T, int GY>
__device__ __forceinline__ void step_y_phase(const SweepArgs& Y, const PairConst* sK, const float* sm, int rb, int c0,
                                             uint16_t* s_list, unsigned* s_n, bool& bad) {
  const Phys<float> p = Y.ph;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = T::W == 64 ? warp : 2 * warp + (lane >> 4);  // of four, Part rows each
  const int c = 2 * (T::W == 64 ? lane : lane & 15), L = c0 + c + 1, n = Y.n;
  const int t0 = T::Halo + T::Part * part;
  const int rows = min(min(T::Part, T::R - T::Part * part), n - (rb + t0) + 1);  // output rows of this thread
  float cour = 0.f;
  if (rows > 0 && L <= Y.nlines) {
    const PairConst K = load_const(sK);
    const bool sw0 = L >= Y.lo && L <= Y.hi, sw1 = L + 1 >= Y.lo && L + 1 <= Y.hi;
    // every cell interior, on swept columns
    const bool inner = sw0 && sw1 && rb + t0 >= 2 && rb + t0 + rows - 1 <= n - 1;
    unsigned rest = 0u;  // listed cells: bit 2i + k, row t0 + i and column c + k
    const float* at = sm + (t0 - 1) * T::Win + 4 + c;
    auto load = [&](const float* f) {
      const float2 d = *reinterpret_cast<const float2*>(f);
      const float2 s = *reinterpret_cast<const float2*>(f + T::Field + T::Out);
      const float2 x = *reinterpret_cast<const float2*>(f + 2 * T::Field + T::Out);
      const float2 y = *reinterpret_cast<const float2*>(f + 3 * T::Field + T::Out);
      return make_cell2(p, K, d.x, d.y, s.x, s.y, y.x, y.y, x.x, x.y);
    };
    Cell2 b;  // the cell after m.j, made ready while m.j is finished
    const Geo2 g{K.inv, K.ndtx, 0ull, 0ull};
    March m;
    // wet cells, and wet subcritical ones, of either column, the newest at bit 0
    unsigned wet0 = 0u, wet1 = 0u, ok0 = 0u, ok1 = 0u;
    auto flags = [&](const Cell2& b) {
      const unsigned a0 = wet_sign(b.H[0], p), a1 = wet_sign(b.H[1], p);
      wet0 = take_sign(wet0, a0);
      wet1 = take_sign(wet1, a1);
      ok0 = take_sign(ok0, a0 & ~sup_sign(lo2(b.u), lo2(b.c)));
      ok1 = take_sign(ok1, a1 & ~sup_sign(hi2(b.u), hi2(b.c)));
    };
    float cm0 = 0.f, cm1 = 0.f;
    f2 chk = 0ull;
    auto face = [&](const Cell2& b, int k, f2& inv, f2& qP, f2& qQ) {  // between rows k - 1 and k
      inv = g.inv;
      if (GY == GEO_TABLE) {
        const float x = k >= 2 && k <= n - 1 ? __ldg(Y.geo + (k - 1)).x : (k == n ? __ldg(Y.geo + (n - 2)).y : 0.f);
        inv = both(x);
      }
      face2(m.j, b, K, inv, qP, qQ);
    };
    auto take = [&](const Cell2& b, f2 inv, f2 qP, f2 qQ) {
      m.nqv = mul2(sub2(m.j.v, b.v), inv);
      m.qP = qP;
      m.qQ = qQ;
      m.va = m.j.v;
      m.j = b;
    };
    m.j = load(at);
    m.va = 0ull;
    flags(m.j);
    {
      const Cell2 j = load(at + T::Win);
      b = load(at + 2 * T::Win);
      f2 inv, qP, qQ;
      face(j, rb + t0, inv, qP, qQ);
      take(j, inv, qP, qQ);
      flags(j);
    }
    at += 2 * T::Win;
    // byte offset of the output pair (a field is below 4 GB)
    uint32_t q = ((uint32_t)(rb + t0 - 1) * (uint32_t)Y.pitch + (uint32_t)(L - 1)) * 4u;
    char *const ps = reinterpret_cast<char*>(Y.srf_o), *const px = reinterpret_cast<char*>(Y.xu_o),
               *const py = reinterpret_cast<char*>(Y.yv_o);
#pragma unroll 2
    for (int i = 0; i < rows; ++i, q += 4u * (uint32_t)Y.pitch) {
      const int o = rb + t0 + i;  // the row finished here
      at += T::Win;
      // past the window's last row in a tile's last round: not used, within
      // the block's shared memory
      const Cell2 next = load(at);
      f2 inv, qP, qQ;
      face(b, o + 1, inv, qP, qQ);
      Geo2 gk = g;
      if (GY == GEO_TABLE) {
        const float4 t = __ldg(Y.geo + (o - 1));
        gk.inv = inv;
        gk.ndtx = both(-t.z);
        gk.ndfpm = both(-t.w);
      }
      if (GY & GEO_SCL) gk.scl8 = both(Y.scl ? 8.f * __ldg(Y.scl + (o - 1)) : 0.f);
      float os[2];
      f2 ou, ov, cn;
      update2<GY>(m, b.v, qP, qQ, gk, p.ginv, K, os, ou, ov, cn);
      flags(b);
      if ((ok0 & ok1 & 7u) == 7u && inner && fminf(lo2(cn), hi2(cn)) > 0.f) {
        *reinterpret_cast<float2*>(ps + q) = make_float2(os[0], os[1]);
        *reinterpret_cast<f2*>(px + q) = ov;
        *reinterpret_cast<f2*>(py + q) = ou;
        chk = fma2(pk(os[0], os[1]), 0ull, fma2(ou, 0ull, fma2(ov, 0ull, chk)));
      } else {
        // plain cells take their results; columns that are not swept and land
        // at rest keep their x-swept values; the others are listed
        const bool in = o >= 2 && o <= n - 1;
        const bool p0 = in && sw0 && (ok0 & 7u) == 7u && lo2(cn) > 0.f;
        const bool p1 = in && sw1 && (ok1 & 7u) == 7u && hi2(cn) > 0.f;
        const bool k0 = !sw0 || at_rest(wet0, m.j.H[0], lo2(m.j.u), lo2(m.j.v));
        const bool k1 = !sw1 || at_rest(wet1, m.j.H[1], hi2(m.j.u), hi2(m.j.v));
        const float s0 = p0 ? os[0] : m.j.s[0], x0 = p0 ? lo2(ov) : lo2(m.j.v), y0 = p0 ? lo2(ou) : lo2(m.j.u);
        const float s1 = p1 ? os[1] : m.j.s[1], x1 = p1 ? hi2(ov) : hi2(m.j.v), y1 = p1 ? hi2(ou) : hi2(m.j.u);
        const bool w0 = p0 || k0, w1 = (p1 || k1) && L + 1 <= Y.nlines;
        if (w0) {
          *reinterpret_cast<float*>(ps + q) = s0;
          *reinterpret_cast<float*>(px + q) = x0;
          *reinterpret_cast<float*>(py + q) = y0;
        }
        if (w1) {
          *reinterpret_cast<float*>(ps + q + 4) = s1;
          *reinterpret_cast<float*>(px + q + 4) = x1;
          *reinterpret_cast<float*>(py + q + 4) = y1;
        }
        const float z = (w0 ? s0 + x0 + y0 : 0.f) * 0.f + (w1 ? s1 + x1 + y1 : 0.f) * 0.f;
        bad = bad || z != z;
        rest |= ((p0 || k0 ? 0u : 1u) | (p1 || k1 ? 0u : 2u)) << (2 * i);
      }
      float a0 = add_rn(fabsf(lo2(m.j.u)), lo2(m.j.c)), a1 = add_rn(fabsf(hi2(m.j.u)), hi2(m.j.c));
      if (GY == GEO_TABLE) {
        a0 *= -lo2(gk.ndtx);
        a1 *= -lo2(gk.ndtx);
      }
      cm0 = fmaxf(cm0, a0);
      cm1 = fmaxf(cm1, a1);
      take(b, inv, qP, qQ);
      b = next;
    }
    if (rest) {
      unsigned w = atomicAdd(s_n, (unsigned)__popc(rest));
      for (; rest; rest &= rest - 1u) {
        const int b = __ffs(rest) - 1;
        s_list[w++] = (uint16_t)((t0 + (b >> 1)) * T::W + c + (b & 1));
      }
    }
    cour = fmaxf(sw0 ? cm0 : 0.f, sw1 ? cm1 : 0.f);
    if (GY != GEO_TABLE) cour *= -lo2(g.ndtx);
    bad = bad || lo2(chk) != lo2(chk) || hi2(chk) != hi2(chk);
  }
  courant_status(Y, cour);
}

// ---- the step ---------------------------------------------------------------------

template <class T>
struct StepShared {
  // dep, srf, xu, yv (and the swept srf, xu, yv): [row + Halo - r0][col + 4 - c0]
  __align__(128) float win[T::Floats];
  uint16_t list[T::Rows * T::W];             // listed cells: window row * W + tile column
  uint16_t queue[T::Threads / 32][2][64];    // places in the list that wait for all the rules (WarpQueue)
  unsigned n[2];                             // listed cells, x phase and y phase
  unsigned scans[2];                         // the columns (a bit each) of the y phase that need the wet scan
  PairConst k[2];                            // x and y axis
  __align__(8) uint64_t bar;
};

// The max-wave fold of the step's input (cliffs_main.f:347-355) over the rows
// of the window that the calling warp sweeps: loads issued before the wait for
// the window's copies.
template <class T>
struct Fold {
  static constexpr int N = T::W / 16;
  float4 h[N], v[N];
};

// Fold item k of a lane: window row and tile column (a float4).
template <class T>
__device__ __forceinline__ void fold_item(int k, int& t, int& c) {
  constexpr int kVecs = T::W / 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = (32 * k + lane) / kVecs;  // of the warp's 8 rows
  t = warp * 4 + r % 4 + (r / 4) * T::Pair;
  c = (lane % kVecs) * 4;
}

template <class T>
__device__ __forceinline__ bool fold_cell(const SweepArgs& X, int rb, int c0, int t, int c, size_t& q) {
  const int row = rb + t - 1;  // 0-based
  q = (size_t)row * (size_t)X.pitch + (size_t)(c0 + c);
  return t >= T::Halo && t < T::Halo + T::R && row < X.nlines && c0 + c < X.n;
}

// ---- the listed cells -------------------------------------------------------------

// A warp takes its share of a phase's list: the cells where no flooding is in play
// (most of a coast) at once, the others gathered so that the warp's lanes go
// through all the rules together.  A warp of both kinds pays for both: taken as
// they came, a sea floor of random depths, a third of it land, took 560 us a step
// at 2048 x 2048 and 51 at 600 x 600, 262 and 32 this way (a launch per sweep 259
// and 46).  Gathered by the block after a barrier, 256 x 256 with one beach took
// 9.9 us, 9.0 by warps (9.5 as they came).

// The cells of a list that a warp takes at a time.  In the smaller tiles, whose
// slowest block is the step's time, a short list is shared evenly (1003 x 777 with a
// rough coast 18.3 us a step, 19.4 by full turns); in large tiles fewer warps take
// full turns, and other blocks the rest (2048 x 2048 44.3, 44.5 shared; a batch of 24
// grids 74.6, 75.2).
template <class T>
__device__ __forceinline__ unsigned list_share(unsigned n) {
  constexpr unsigned kWarps = T::Threads / 32;
  return T::InPlace ? 32u : min((n + kWarps - 1) / kWarps, 32u);
}

// The x phase's, into the window; true if a value is not finite.  The whole block
// calls it.
template <class T>
__device__ __forceinline__ bool step_x_list(const SweepArgs& X, int rb, int c0, StepShared<T>& S) {
  const int tid = threadIdx.x;
  const unsigned lane = tid & 31, cx = S.n[0];
  bool bad = false;
  const auto put = [&](int t, int c, const OutCell<float>& r) {
    float* f = S.win + T::Out + t * T::Win + 4 + c;
    f[T::Field] = r.s;
    f[2 * T::Field] = r.u;
    f[3 * T::Field] = r.v;
    bad = bad || !isfinite(r.s + r.u + r.v);
  };
  WarpQueue Q{S.queue[tid >> 5][0]};
  const unsigned share = list_share<T>(cx), round = share * (T::Threads / 32);
  for (unsigned base = share * (unsigned)(tid >> 5);; base += round) {
    const unsigned i = base + lane;
    bool hard = false;
    if (lane < share && i < cx) {
      const int t = S.list[i] / T::W, c = S.list[i] % T::W;
      const XValue r = T::InPlace ? step_x_shore(X, rb + t, c0 + c + 1)
                                  : step_x_window_shore<T>(X, S.win, rb, c0, t, c);
      hard = !r.ok;
      if (r.ok) put(t, c, r.out);
    }
    Q.push(hard, i);
    const bool last = base + round >= cx;
    if (Q.n >= 32 || (Q.n && last)) {
      unsigned at;
      if (Q.peek(lane, at)) {
        const int t = S.list[at] / T::W, c = S.list[at] % T::W;
        put(t, c, T::InPlace ? step_x_general(X, rb + t, c0 + c + 1)
                             : step_x_window_full<T>(X, S.win, rb, c0, t, c));
      }
      Q.pop(32);
    }
    if (last && !Q.n) break;
  }
  __syncthreads();
  return bad;
}

// Remainders on land with no water in the window's part of their column, marked in
// the list: zeroed when the x-swept column holds a wet cell anywhere, else left as
// they are.  The block looks through each of their columns once, together: a 512 x
// 512 grid with a quarter of such land 0.61 ms a step, 2.1 with a look for each cell
// (0.50 a launch per sweep).
template <class T>
__device__ __noinline__ bool step_y_scan(const SweepArgs& X, const SweepArgs& Y, int rb, int c0, StepShared<T>& S) {
  const int tid = threadIdx.x;
  bool bad = false;
  unsigned wet[2] = {0u, 0u};
#pragma unroll
  for (int h = 0; h < 2; ++h)
    for (unsigned m = S.scans[h]; m; m &= m - 1u) {
      const int b = __ffs(m) - 1;
      bool any = false;
      for (int j = 0; j < Y.n && !any; j += T::Threads)
        any = __syncthreads_or(j + tid < Y.n && step_x_wet(X, j + tid + 1, c0 + 32 * h + b + 1));
      if (any) wet[h] |= 1u << b;
    }
  for (unsigned i = tid; i < S.n[1]; i += T::Threads) {
    const unsigned ent = S.list[i];
    if (!(ent & 0x8000u)) continue;
    const int t = (int)(ent & 0x7fffu) / T::W, c = (int)(ent & 0x7fffu) % T::W;
    const float* f = S.win + t * T::Win + 4 + c;
    const size_t q = (size_t)(rb + t - 1) * (size_t)Y.pitch + (size_t)(c0 + c);
    const bool z = (c < 32 ? wet[0] >> c : wet[1] >> (c - 32)) & 1u;
    const float s = z ? state_from_depth(0.f, f[0]) : f[T::Field + T::Out];
    const float u = z ? 0.f : f[2 * T::Field + T::Out], v = z ? 0.f : f[3 * T::Field + T::Out];
    Y.srf_o[q] = s;
    Y.xu_o[q] = u;
    Y.yv_o[q] = v;
    bad = bad || !isfinite(s + u + v);
  }
  return bad;
}

// The y phase's, to the output fields.
template <class T>
__device__ __forceinline__ bool step_y_list(const SweepArgs& X, const SweepArgs& Y, int rb, int c0, StepShared<T>& S) {
  const int tid = threadIdx.x;
  const unsigned lane = tid & 31, cy = S.n[1];
  bool bad = false;
  const auto store = [&](int t, int c, const OutCell<float>& r) {
    const size_t q = (size_t)(rb + t - 1) * (size_t)Y.pitch + (size_t)(c0 + c);
    Y.srf_o[q] = r.s;
    Y.xu_o[q] = r.v;
    Y.yv_o[q] = r.u;
    bad = bad || !isfinite(r.s + r.u + r.v);
  };
  // cells with all the rules' rows in the window, and those in the first and last
  // rows, a pair of lanes each; a few of both kinds go by pairs together (apart,
  // the one block of a 1003 x 777 grid with both took 21.1 us a step for its 19.1)
  WarpQueue Q{S.queue[tid >> 5][0]}, E{S.queue[tid >> 5][1]};
  const unsigned share = list_share<T>(cy), round = share * (T::Threads / 32);
  for (unsigned base = share * (unsigned)(tid >> 5);; base += round) {
    const unsigned i = base + lane;
    bool hard = false, end = false;
    if (lane < share && i < cy) {
      const int t = S.list[i] / T::W, c = S.list[i] % T::W;
      const XValue r = step_y_shore<T>(Y, S.win, rb, c0, t, c);
      hard = !r.ok;
      end = T::Halo < 3 && (t < 3 || t >= T::Rows - 3);
      if (r.ok) store(t, c, r.out);
    }
    const bool last = base + round >= cy;
    Q.push(hard && !end, i);
    if (T::Halo < 3) {
      E.push(hard && end, i);
      if (last && E.n && Q.n + E.n <= 16) E.take(Q);
    }
    for (;;) {
      const bool pair = E.n >= 16 || (last && E.n);
      if (!pair && !(Q.n >= 32 || (last && Q.n))) break;
      unsigned at;
      const bool on = pair ? E.peek(lane >> 1, at) : Q.peek(lane, at);
      const unsigned ent = on ? S.list[at] : (unsigned)(T::Halo * T::W);
      const int t = (int)ent / T::W, c = (int)ent % T::W;
      const YValue r = step_y_full<T>(X, Y, S.win, rb, c0, pair, on, t, c);
      if (on && !(pair && (lane & 1))) {
        if (r.scan) {
          S.list[at] = (uint16_t)(ent | 0x8000u);
          atomicOr(&S.scans[c >> 5], 1u << (c & 31));
        } else {
          store(t, c, r.out);
        }
      }
      if (pair)
        E.pop(16);
      else
        Q.pop(32);
    }
    if (last) break;
  }
  __syncthreads();
  if (S.scans[0] | S.scans[1]) bad |= step_y_scan<T>(X, Y, rb, c0, S);
  return bad;
}

// The two out of line.
template <class T>
__device__ __noinline__ bool step_x_list_apart(const SweepArgs& X, int rb, int c0, StepShared<T>& S) {
  return step_x_list<T>(X, rb, c0, S);
}
template <class T>
__device__ __noinline__ bool step_y_list_apart(const SweepArgs& X, const SweepArgs& Y, int rb, int c0,
                                               StepShared<T>& S) {
  return step_y_list<T>(X, Y, rb, c0, S);
}

template <class T, int GX, int GY>
__device__ __forceinline__ void step_tile(const SweepArgs& X, const SweepArgs& Y, const StepMaps& M, int r0, int c0,
                                          const StepCtl& C, StepShared<T>& S) {
  const int tid = threadIdx.x;
  const int rb = r0 + 1 - T::Halo;  // the 1-based row of window row 0
  if (tid == 0) {
    mbar_expect_tx(&S.bar, T::Bytes + C.extra);
    tma_load_2d(S.win, &M.dep, &S.bar, c0 - 4, rb - 1);
    tma_load_2d(S.win + T::Field, &M.srf, &S.bar, c0 - 4, rb - 1);
    tma_load_2d(S.win + 2 * T::Field, &M.xu, &S.bar, c0 - 4, rb - 1);
    tma_load_2d(S.win + 3 * T::Field, &M.yv, &S.bar, c0 - 4, rb - 1);
  }
  Fold<T> F;
#pragma unroll
  for (int k = 0; k < Fold<T>::N; ++k) {
    int t, c;
    size_t q;
    fold_item<T>(k, t, c);
    F.h[k] = F.v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (fold_cell<T>(X, rb, c0, t, c, q)) {
      F.h[k] = ld_state4<false>(X.hmax_in + q);
      F.v[k] = ld_state4<false>(X.velmax_in + q);
    }
  }
  const bool ok = mbar_wait_ns(&S.bar, 0u, C.wait_ns);
  if (__syncthreads_or(!ok)) {
    if (tid == 0) {
      atomicOr(X.status, ST_STALL);
      mbar_wait_ns(&S.bar, 0u, C.wait_ns);  // the copies in flight, before the block's memory goes
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < Fold<T>::N; ++k) {
    int t, c;
    size_t q;
    fold_item<T>(k, t, c);
    if (!fold_cell<T>(X, rb, c0, t, c, q)) continue;
    const float* f = S.win + t * T::Win + 4 + c;
    const float4 d = *reinterpret_cast<const float4*>(f), s = *reinterpret_cast<const float4*>(f + T::Field);
    const float4 x = *reinterpret_cast<const float4*>(f + 2 * T::Field);
    const float4 y = *reinterpret_cast<const float4*>(f + 3 * T::Field);
    F.h[k].x = fmaxf(F.h[k].x, eta_of(s.x, d.x));
    F.h[k].y = fmaxf(F.h[k].y, eta_of(s.y, d.y));
    F.h[k].z = fmaxf(F.h[k].z, eta_of(s.z, d.z));
    F.h[k].w = fmaxf(F.h[k].w, eta_of(s.w, d.w));
    F.v[k].x = fmaxf(F.v[k].x, fma_rn(x.x, x.x, mul_rn(y.x, y.x)));
    F.v[k].y = fmaxf(F.v[k].y, fma_rn(x.y, x.y, mul_rn(y.y, y.y)));
    F.v[k].z = fmaxf(F.v[k].z, fma_rn(x.z, x.z, mul_rn(y.z, y.z)));
    F.v[k].w = fmaxf(F.v[k].w, fma_rn(x.w, x.w, mul_rn(y.w, y.w)));
    *reinterpret_cast<float4*>(X.hmax_in + q) = F.h[k];
    *reinterpret_cast<float4*>(X.velmax_in + q) = F.v[k];
  }
  __syncwarp();  // the warp's rows are read before they are swept in place
  bool bad = false;
  step_x_phase<T, GX>(X, &S.k[0], S.win, rb, c0, S.list, &S.n[0], bad);
  __syncthreads();
  // The lists of large tiles with more than flat geometry are out of line: inline,
  // they take registers that the phases want (4320 x 2160 sphere 91.9 us a step,
  // 88.9 out of line; a flat 2048 x 2048 44.8 and 45.4, 256 x 256 9.0 and 9.5).
  constexpr bool kApart = T::InPlace && GX != GEO_FLAT;
  if (S.n[0]) bad |= kApart ? step_x_list_apart<T>(X, rb, c0, S) : step_x_list<T>(X, rb, c0, S);
  step_y_phase<T, GY>(Y, &S.k[1], S.win, rb, c0, S.list, &S.n[1], bad);
  __syncthreads();
  if (S.n[1]) bad |= kApart ? step_y_list_apart<T>(X, Y, rb, c0, S) : step_y_list<T>(X, Y, rb, c0, S);
  if (bad) atomicOr(X.status, ST_NAN);
}

// The order of a grid's tiles: those that hold a coast first, as their listed
// cells make them last longer (a step ends with its slowest block, which is to
// start early); the others band by band, every other step last to first: a
// step starts on the rows that the one before it wrote last, which are still
// in L2.  So there are two orders of a grid's tiles, one behind the other, for the
// steps from either copy of the state.  The coast is that of the depth at the
// context's creation: the order changes no result.

// Whether the tile of T at column x0, row y0 (0-based), or a cell beside it, holds
// land and sea.  The whole block calls it.
template <class T>
__device__ __forceinline__ bool coast_tile(int nx, int ny, int pitch, const float* __restrict__ dep, int x0, int y0) {
  bool land = false, sea = false;
  for (int i = threadIdx.x; i < (T::W + 2) * (T::R + 2); i += blockDim.x) {
    const int x = x0 - 1 + i % (T::W + 2), y = y0 - 1 + i / (T::W + 2);
    if (x < 0 || x >= nx || y < 0 || y >= ny) continue;
    const bool l = dep[(size_t)y * pitch + x] < 0.f;
    land = land || l;
    sea = sea || !l;
  }
  land = __syncthreads_or(land);
  sea = __syncthreads_or(sea);
  return land && sea;
}

// A block of 128 threads a tile: its flag, and in the block that finishes last the
// order of them all by put(place, tile, all): the tiles with a flag (all of them), then
// the others, each in their order.  done: 0 before the launch.
template <class Put>
__device__ __forceinline__ void order_tiles(bool coast, uint8_t* flags, unsigned* done, Put put) {
  __shared__ int s_warp[4];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, tiles = (int)gridDim.x;
  if (tid == 0) {
    flags[blockIdx.x] = coast;
    __threadfence();
    s_last = atomicAdd(done, 1u) == (unsigned)tiles - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int per = (tiles + 127) / 128, lo = min(tid * per, tiles), hi = min(lo + per, tiles);
  int mine = 0;
  for (int i = lo; i < hi; ++i) mine += __ldcg(flags + i);
  int upto = mine;  // of the warp's lanes so far
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const int v = __shfl_up_sync(0xffffffffu, upto, d);
    if (lane >= d) upto += v;
  }
  if (lane == 31) s_warp[tid >> 5] = upto;
  __syncthreads();
  int before = upto - mine, all = 0;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    if (w < tid >> 5) before += s_warp[w];
    all += s_warp[w];
  }
  int a = before, b = all + lo - before;
  for (int i = lo; i < hi; ++i) {
    const bool first = __ldcg(flags + i) != 0;
    const int place = first ? a++ : b++;
    put(place, i, all);
  }
}

// The orders of a grid's tiles (gridDim.x of them) for the steps from either copy.
template <class T>
__global__ void __launch_bounds__(128) k_tile_order(int nx, int ny, int pitch, const float* __restrict__ dep,
                                                    uint8_t* flags, unsigned* done, int* order) {
  const int across = (nx + T::W - 1) / T::W;
  const bool coast = coast_tile<T>(nx, ny, pitch, dep, (int)blockIdx.x % across * T::W, (int)blockIdx.x / across * T::R);
  const int tiles = (int)gridDim.x;
  order_tiles(coast, flags, done, [&](int place, int tile, int all) {
    order[place] = tile;
    order[tiles + (place < all ? place : tiles - 1 - (place - all))] = tile;
  });
}

// ORDERED: a one-dimensional grid, the tiles from the order; else a grid of
// tiles, by bands.
template <class T, int GX, int GY, bool ORDERED>
__global__ void __launch_bounds__(T::Threads, T::Blocks)
    step_kernel(const __grid_constant__ SweepArgs X, const __grid_constant__ SweepArgs Y,
                const __grid_constant__ StepMaps M, const StepCtl C, const __grid_constant__ PairPair K,
                const int* __restrict__ order) {
  __shared__ StepShared<T> S;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    mbar_init(&S.bar, 1);
    S.n[0] = S.n[1] = S.scans[0] = S.scans[1] = 0u;
    S.k[0] = K.x;
    S.k[1] = K.y;
    fence_mbar_init();
  }
  int bx, by;
  if (ORDERED) {  // written once, before the context's first launch: read ahead
    const int gx = (X.n + T::W - 1) / T::W;
    const int tile = __ldg(order + blockIdx.x);
    bx = tile % gx;
    by = tile / gx;
  } else {
    bx = (int)blockIdx.x;
    by = C.flip ? (int)(gridDim.y - 1 - blockIdx.y) : (int)blockIdx.y;
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  step_tile<T, GX, GY>(X, Y, M, by * T::R, bx * T::W, C, S);
}

// One whole step of many grids (batch.cuh): a block per tile of the list of
// all scenarios' tiles (coasts first, as above), the scenario's arguments
// staged in shared memory and its tensor maps read from device memory.  24
// scenarios of 256 to 768 nodes a side (6.8 M cells), a run of 64 steps with
// its uploads and maxima: 6.7 ms, from 12.2 with a launch per sweep phase.
struct StepArgs {
  SweepArgs X, Y;
  PairPair K;
  StepMaps M;
};

struct BatchStep {
  const StepArgs* args;  // per scenario, for the state copy that the step reads
  const int4* order;     // scenario, first row and first column of each tile
};

// The order of a batch's tiles, from the scenarios' own order `list`, and the number
// of those with a coast.  One order for both copies: its entries are 16 bytes and come
// from L2 at each block's start, with nothing to hide them (24 scenarios of 256 to 768
// nodes a side: 75.1 us a step with two, 74.7 with one).
template <class T>
__global__ void __launch_bounds__(128) k_batch_order(const StepArgs* __restrict__ args, const int4* __restrict__ list,
                                                     uint8_t* flags, unsigned* done, int4* order, int* count) {
  const int4 at = list[blockIdx.x];
  const SweepArgs& X = args[at.x].X;
  const bool coast = coast_tile<T>(X.n, X.nlines, X.pitch, X.dep, at.z, at.y);
  order_tiles(coast, flags, done, [&](int place, int tile, int all) {
    order[place] = list[tile];
    if (tile == 0) *count = all;
  });
}

template <class T, int GX, int GY>
__global__ void __launch_bounds__(T::Threads, T::Blocks) batch_step_kernel(const BatchStep B, const StepCtl C) {
  __shared__ StepShared<T> S;
  __shared__ SweepArgs sA[2];
  const int tid = threadIdx.x;
  const int id = (int)blockIdx.x;
  const int4 at = __ldg(B.order + (C.flip && id >= C.coast ? (int)gridDim.x - 1 - (id - C.coast) : id));
  const StepArgs* A = B.args + at.x;
  static_assert(sizeof(SweepArgs) % 8 == 0 && sizeof(PairPair) % 8 == 0, "copied in 8-byte words");
  const auto copy = [&](void* to, const void* from, int bytes) {
    for (int w = tid; w < bytes / 8; w += T::Threads)
      reinterpret_cast<unsigned long long*>(to)[w] = __ldg(reinterpret_cast<const unsigned long long*>(from) + w);
  };
  copy(&sA[0], &A->X, sizeof(SweepArgs));
  copy(&sA[1], &A->Y, sizeof(SweepArgs));
  copy(S.k, &A->K, sizeof(PairPair));
  if (tid == 0) {
    mbar_init(&S.bar, 1);
    S.n[0] = S.n[1] = S.scans[0] = S.scans[1] = 0u;
    fence_mbar_init();
  }
  __syncthreads();
  step_tile<T, GX, GY>(sA[0], sA[1], A->M, at.y, at.z, C, S);
}

}  // namespace cliffs
