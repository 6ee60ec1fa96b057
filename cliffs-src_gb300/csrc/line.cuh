// line.cuh -- many steps of a one-dimensional grid (one line: a channel, a
// beach transect) in one launch.
//
// A step of such a grid is one sweep of a few thousand cells.  With a launch
// per sweep it costs the launch and the latency of a cold kernel, 6 us, where
// the arithmetic takes a fraction of one.  Here a cluster of up to 8 blocks
// holds the line in shared memory, a thread per cell, and steps it as often as
// the call asks for: a step ends with the cluster's barrier, after each block
// has written its outermost three cells into its neighbours' shared memory.
//
// All cells take the same straight path: the rules of general_cell (march.cuh)
// in the phases the reference has them, with block barriers between,
//   flood    cells flooded from a neighbour, and the effective state
//            (cliffs.f:74-111, 122)
//   update   the interior update against the neighbours' effective state or
//            the mirror image, or the edge rule (cliffs.f:137-262, 287-329)
//   limit    the shoreline angle limiter of a newly flooded cell, against its
//            neighbour's update (cliffs.f:264-285); only in a step in which a
//            block has one
// instead of a common fast path and a long rare one: on one line the rare path
// of the shore would be every step's critical path.  A block computes two
// cells of each neighbour again, so that only the state crosses blocks.
//
// Results are the bits of the sweep kernels' (the same functions on the same
// values).  2000 cells: 1.0 us a step, from 6.0 with a launch per sweep,
// replayed from graphs; bound by the latency of the three barriers and of the
// chain between them.
#pragma once
#include <cooperative_groups.h>

#include "sweep.cuh"

namespace cliffs {

constexpr int kLineCluster = 8;   // blocks of a cluster at most (the portable size)
constexpr int kLineBlock = 256;   // threads that a block is meant to have
constexpr int kLineMax = 960;     // and has at most (its shared memory stays under 48 KB)
constexpr int kLineHalo = 3;      // cells of the state on each side (general_cell's window)
constexpr int kLineAgain = 2;     // cells on each side computed again
constexpr int kLineCells = kLineMax - 2 * kLineAgain;  // cells of a block at most

struct LineShared {
  float4 raw[2][kLineMax + 2];  // u, v, eta, H; [parity of the step][cell + kLineHalo]
  float4 eff[kLineMax];         // effective u, v, celerity, eta; [cell + kLineAgain]; in a
                                // limited step then the new celerity and normal velocity
  uint8_t wet[kLineMax];        // wet or flooded
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A: the arguments of the grid's sweep, in place (A.srf_o, A.xu_o, A.yv_o are
// A.srf, A.xu, A.yv); DIR 0: the line is row 1, DIR 1: column 1.  The other
// lines (a grid two cells wide) are passive: only their place in the max-wave
// fields is taken, once.  m: cells of a block (the last one's may be fewer).
template <int DIR, bool SPH>
__global__ void __launch_bounds__(kLineMax) line_kernel(const __grid_constant__ SweepArgs A, const int m,
                                                        const int steps) {
  namespace cg = cooperative_groups;
  __shared__ LineShared S;
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), blocks = (int)cl.num_blocks();
  const int n = A.n, base = rank * m, mine = min(m, n - base);  // cells base .. base + mine - 1, 0-based
  const int t = (int)threadIdx.x, i = t - kLineAgain;           // cell of the block
  const int k = base + i + 1;                                   // its position, 1-based
  const bool here = i < mine + kLineAgain && k >= 1 && k <= n, own = i >= 0 && i < mine;
  const Phys<float> p = A.ph;
  auto cell = [&](int pos, int line) { return cidx<DIR>(line, pos, A.pitch); };
  auto raw_of = [&](float s, float d, float u, float v) { return make_float4(u, v, eta_of(s, d), depth_of(s, d)); };
  auto ld_raw = [&](int pos) {
    if (pos < 1 || pos > n) return make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t q = cell(pos, 1);
    const float x = A.xu[q], y = A.yv[q];
    return raw_of(A.srf[q], A.dep[q], DIR == 0 ? x : y, DIR == 0 ? y : x);
  };
  // the line's state, halo included, and this cell's constants
  for (int c = t - kLineHalo; c < mine + kLineHalo; c += (int)blockDim.x) S.raw[0][c + kLineHalo] = S.raw[1][c + kLineHalo] = ld_raw(base + c + 1);
  float d = 0.f, dl = 0.f, dr = 0.f, s = 0.f, u = 0.f, v = 0.f, hm = 0.f, vm = 0.f;
  Geo<float> g{0.f, 0.f, 0.f, 0.f, 0.f};
  LineCtx<float> C;
  C.n = n;
  C.eL = C.eR = EdgeVals<float>{0.f, 0.f, 0.f};
  float alpha = 1.f, ialpha = 1.f;
  if (DIR == 0 && A.lscale) {
    alpha = A.lscale[0].x;
    ialpha = A.lscale[0].y;
  }
  C.inv_dx1 = A.inv_dx1 * ialpha;
  C.inv_dxn1 = A.inv_dxn1 * ialpha;
  C.scl1 = SPH ? A.scl[0] : 0.f;
  C.scln = SPH ? A.scl[n - 1] : 0.f;
  bool bad = false;
  float dtx = 0.f;  // of the Courant check: the ends of a uniform line have the line's
  if (here) {
    const size_t q = cell(k, 1);
    d = A.dep[q];
    dl = k > 1 ? A.dep[cell(k - 1, 1)] : 0.f;
    dr = k < n ? A.dep[cell(k + 1, 1)] : 0.f;
    g = geo_at(A, k, alpha, ialpha);
    dtx = A.geo_uniform ? A.geo0.z * ialpha : A.geo[k - 1].z * ialpha;
    s = A.srf[q];
    u = DIR == 0 ? A.xu[q] : A.yv[q];
    v = DIR == 0 ? A.yv[q] : A.xu[q];
    if (own) {
      hm = A.hmax[q];
      vm = A.velmax[q];
      for (int line = 2; line <= A.nlines; ++line) {  // the passive lines' state and maxima
        const size_t w = cell(k, line);
        const float x = A.xu[w], y = A.yv[w];
        A.hmax[w] = fmaxf(A.hmax[w], eta_of(A.srf[w], A.dep[w]));
        A.velmax[w] = fmaxf(A.velmax[w], fma_rn(x, x, mul_rn(y, y)));
        bad = bad || !isfinite(A.srf[w] + x + y);
      }
    }
  }
  float cour = 0.f;
  cluster_barrier();  // every block has its part of the line
  for (int step = 0; step < steps; ++step) {
    const float4* raw = S.raw[step & 1];
    float4* next = S.raw[(step + 1) & 1];
    // ---- flood
    const float4 l = raw[t], j = raw[t + 1], r = raw[t + 2];  // cells i - 1, i, i + 1 (kLineHalo - kLineAgain = 1)
    const bool land = !here || j.w <= p.ground;
    const bool lwet = here && k > 1 && !(l.w <= p.ground), rwet = here && k < n && !(r.w <= p.ground);
    const bool Rf = here && land && lwet && l.x >= 0.f && (l.z + d > p.ground);
    const bool Lf = here && land && !Rf && rwet && r.x <= 0.f && (r.z + d > p.ground);
    const bool ew = here && (!land || Rf || Lf);
    CellState<float> f;
    if (Rf || Lf)
      f = CellState<float>{Rf ? l.x : r.x, p.celmin, p.ground - d, d, Rf ? l.y : r.y, p.ground};
    else
      f = CellState<float>{j.x, fsqrt_pos(p.g * (j.w > p.ground ? j.w : p.ground)), j.z, d, j.y, j.w};
    S.eff[t] = make_float4(f.u, f.v, f.c, f.e);
    S.wet[t] = ew;
    if (own) cour = fmaxf(cour, (fabsf(j.x) + fsqrt_pos(p.g * fmaxf(j.w, p.ground))) * dtx);
    __syncthreads();
    // ---- update
    const int tl = max(t - 1, 0), tr = min(t + 1, (int)blockDim.x - 1);
    const float4 a4 = S.eff[tl], b4 = S.eff[tr];
    const bool ewl = S.wet[tl] != 0, ewr = S.wet[tr] != 0;
    const CellState<float> fa{a4.x, a4.z, a4.w, dl, a4.y, 0.f}, fb{b4.x, b4.z, b4.w, dr, b4.y, 0.f};
    OutCell<float> o{s, j.x, j.y};
    float cO = f.c;
    if (k == 1 || k == n) {
      if (Rf || Lf) o.s = state_from_depth(p.ground, d);
      o.u = f.u;
      o.v = f.v;
      float cn, un, vn, sn;
      if (ew && k == 1 && ewr && C.eL.eta + d > p.ground) {
        edge_left(f, fb, C.eL, C.inv_dx1, C.scl1, p, cn, un, vn, sn);
        o = OutCell<float>{sn, un, vn};
      } else if (ew && k == n && k > 1 && ewl && C.eR.eta + d > p.ground) {
        edge_right(fa, f, C.eR, C.inv_dxn1, C.scln, p, cn, un, vn, sn);
        o = OutCell<float>{sn, un, vn};
      }
    } else {
      const CellState<float> mir{-f.u, f.c, f.e, f.d, f.v, f.H};
      const CellState<float> a = ewl ? fa : mir, b = ewr ? fb : mir;
      float FPl, FQl, FPr, FQr;
      face_flux(a.u, a.c, a.e, f.u, f.c, f.e, p, FPl, FQl);
      face_flux(f.u, f.c, f.e, b.u, b.c, b.e, p, FPr, FQr);
      o = interior_update<float, true, SPH>(a, f, b, FPl, FQl, FPr, FQr, g, p, &cO);
    }
    // ---- limit
    const bool inner = k >= 2 && k <= n - 1;
    const bool limL = ew && inner && Lf && !ewl, limR = ew && inner && !limL && Rf && !ewr;
    if (__syncthreads_or(limL || limR)) {
      // the new celerity and velocity of interior cells, the effective ones of the line's ends
      S.eff[t] = inner ? make_float4(cO, o.u, 0.f, 0.f) : make_float4(f.c, f.u, 0.f, 0.f);
      __syncthreads();
      if (limL || limR) {
        const float4 nb = S.eff[limL ? tr : tl];
        if (p.sqr2 * cO > nb.x) {
          cO = nb.x / p.sqr2;
          o.s = state_from_c(cO, d, p);
        }
        if (limL ? o.u < nb.y : o.u > nb.y) o.u = nb.y;
      }
    }
    if (own) {
      if (!ew) {  // new land, or a line without water, which is left alone (cliffs.f:113-122)
        bool wet = lwet || rwet || (j.w == 0.f && j.x == 0.f && j.y == 0.f);
        for (int b = 0; b < blocks && !wet; ++b) {
          // a remainder with no wet cell beside it: every block's cells, which
          // stay as they are until the step's end
          const int at = (rank + b) % blocks;
          const float4* other = cl.map_shared_rank(&S.raw[step & 1][0], at);
          const int cells = min(m, n - at * m);
          for (int c = 0; c < cells && !wet; ++c) wet = !(other[c + kLineHalo].w <= p.ground);
        }
        if (wet) o = OutCell<float>{state_from_depth(0.f, d), 0.f, 0.f};
        else o = OutCell<float>{s, j.x, j.y};
      }
      s = o.s;
      u = o.u;
      v = o.v;
      const float4 q = raw_of(s, d, u, v);
      next[i + kLineHalo] = q;
      if (i < kLineHalo && rank > 0) cl.map_shared_rank(next, rank - 1)[m + i + kLineHalo] = q;
      if (i >= mine - kLineHalo && rank + 1 < blocks) cl.map_shared_rank(next, rank + 1)[i - mine + kLineHalo] = q;
      bad = bad || !isfinite(s + u + v);
      hm = fmaxf(hm, q.z);
      vm = fmaxf(vm, DIR == 0 ? fma_rn(u, u, mul_rn(v, v)) : fma_rn(v, v, mul_rn(u, u)));
    }
    cluster_barrier();
  }
  if (own) {
    const size_t q = cell(k, 1);
    A.srf_o[q] = s;
    A.xu_o[q] = DIR == 0 ? u : v;
    A.yv_o[q] = DIR == 0 ? v : u;
    A.hmax[q] = hm;
    A.velmax[q] = vm;
  }
  if (bad) atomicOr(A.status, ST_NAN);
  if (cour > 0.5f) {
    atomicOr(A.status, ST_CFL);
    atomicMax(A.status + 1, __float_as_uint(2.f * cour));
  }
}

}  // namespace cliffs
