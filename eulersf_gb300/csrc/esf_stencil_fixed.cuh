// The FP64 pressure stencil on integers (esf_fixed.cuh). Included by
// esf_solver.cu inside namespace esf after pressure_stencil, whose modes and
// arguments it shares.
//
// A warp owns 32 cell columns (30 of them its output, one halo column a side)
// and RY output rows, and marches along z over a chunk of cz layers with
// everything in registers: the previous layer's values, the node rows' products
// of the layer below, and row by row the sums; neighbours along x come by
// shuffle. The next layer's inputs are on their way into shared memory
// (cp.async, zero-filled outside the grid, each lane reading back only what it
// fetched) while a layer is computed; there is no barrier.
//   cell row:  P = v(k-1) + v(k), Q = v(k-1) - v(k); with the next column's P', Q':
//              P - P', P + P', Q + Q'
//   node row (between two cell rows):  J^T v = ((P-P') + (P-P')+, (P+P') - (P+P')+,
//              (Q+Q') + (Q+Q')+), times 1/m; A, B, C = with the layer below's
//   cell:      (A + C - B) + (C - A - B)' of the lower node row plus
//              (A + C + B) + (C - A + B)' of the upper (' of the column before)
//
// Bound: instruction issue (161x127x190 UPDATE: 89 M warp instructions, 0.61 a
// cycle and scheduler, its three or four warps waiting on their own chains; DRAM
// at a fifth). Measured against pressure_stencil<double>, whose bound is the FP64
// pipe: product 32^3 18.6 -> 8.5 us, 64^3 28.8 -> 18.7, 128^3 158 -> 66,
// 161x127x190 343 -> 109, 256^3 1154 -> 404; solve iteration (phase A included)
// 33 -> 20, 53 -> 36, 254 -> 125, 499 -> 207, 1748 -> 755 us. Error of a
// product against extended precision 4.7e-17 of the norm, the rounding of the
// result; a plain FP64 evaluation has 1.7e-16.
#pragma once

constexpr int FX_T = 128;              // threads a block: four warps, stacked along y
constexpr int FX_W = FX_T / 32, FX_COLS = 30;
constexpr long long FX_MAX_BLOCKS = 16384;  // the static solve's partial sums; ESF_MAX_PARTIALS is more
// values a lane fetches for a layer: the stencil's input rows (UPDATE: r, Ap
// and 1/diag), the node rows' 1/m, and for UPDATE the own rows' x and d
template <int MODE, int RY>
__host__ __device__ constexpr int fx_slots() {
  return (MODE == S_UPDATE ? 3 : 1) * (RY + 2) + (RY + 1) + (MODE == S_UPDATE ? 2 * RY : 0);
}
template <int MODE, int RY>
__host__ __device__ constexpr int fx_smem() {
  return 2 * fx_slots<MODE, RY>() * FX_T * 8;
}
// 8 bytes from global to shared memory, or zeros
__device__ __forceinline__ void fetch8(double* dst, const double* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 8 : 0)
               : "memory");
}

__device__ __forceinline__ Fix shfl_down(Fix a) {
  return Fix{__shfl_down_sync(0xffffffffu, a.l0, 1), __shfl_down_sync(0xffffffffu, a.l1, 1),
             __shfl_down_sync(0xffffffffu, a.l2, 1)};
}
__device__ __forceinline__ Fix shfl_up(Fix a) {
  return Fix{__shfl_up_sync(0xffffffffu, a.l0, 1), __shfl_up_sync(0xffffffffu, a.l1, 1),
             __shfl_up_sync(0xffffffffu, a.l2, 1)};
}

__device__ __forceinline__ double shfl_down(double a) { return __shfl_down_sync(0xffffffffu, a, 1); }
__device__ __forceinline__ double shfl_up(double a) { return __shfl_up_sync(0xffffffffu, a, 1); }

// A warp's layer as fixed_finish reads it: the rows' values, the node rows' 1/m.
template <int MODE, int RY>
struct FixedLayer {
  double v[RY + 2], m[RY + 1];
  __device__ __forceinline__ void load(const GridDev& g, const StencilArgs<double>& a, double alpha, int cx, int y0,
                                       int kk, int last) {
    const bool layer = kk >= 0 && kk < g.cZ && kk <= last, col = cx >= 0 && cx < g.cX;
#pragma unroll
    for (int j = 0; j < RY + 2; j++) {
      const int y = y0 - 1 + j;
      const long long c = cx + (long long)y * g.cX + (long long)kk * g.cslab;
      v[j] = 0.0;
      if (layer && col && y >= 0 && y < g.cY)
        v[j] = MODE == S_UPDATE ? upd_r(a.r[c], alpha, a.Ap[c], a.invd[c]) : a.in[c];
    }
#pragma unroll
    for (int j = 0; j < RY + 1; j++) {
      const int y = y0 + j;
      const bool in = col && cx < g.cX - 1 && y > 0 && y < g.Y - 1 && kk > 0 && kk < g.Z - 1 && kk <= last;
      m[j] = in ? a.minv[cx + 1 + (long long)y * g.X + (long long)kk * g.slab] : 0.0;
    }
  }
};
// Which of a warp's cells lose bits on integers that FP64 keeps: those whose
// largest product of a value and a factor lies below 2^(top - FIX_SPARE).
template <int RY>
struct FixedReach {
  int ev[RY + 2], en[RY + 1];  // of the layer before: values' places, products'
  __device__ __forceinline__ FixedReach() {
#pragma unroll
    for (int j = 0; j < RY + 2; j++) ev[j] = FIX_NOWHERE;
#pragma unroll
    for (int j = 0; j < RY + 1; j++) en[j] = FIX_NOWHERE;
  }
  // the next layer; bit j: this lane's cell of row j, layer kk - 1
  template <int MODE>
  __device__ __forceinline__ unsigned next(const FixedLayer<MODE, RY>& l, int top) {
    int pair = FIX_NOWHERE, pn = FIX_NOWHERE;  // of the row before
    unsigned loses = 0;
#pragma unroll
    for (int j = 0; j < RY + 2; j++) {
      const int e = fixed_place(l.v[j]), two = max(ev[j], e);
      ev[j] = e;
      int at = max(pair, two);
      pair = two;
      if (j == 0) continue;
      at = max(at, __shfl_down_sync(0xffffffffu, at, 1)) + fixed_place(l.m[j - 1]);
      const int nodes = max(en[j - 1], at);
      en[j - 1] = at;
      int best = max(pn, nodes);
      pn = nodes;
      if (j == 1) continue;
      best = max(best, __shfl_up_sync(0xffffffffu, best, 1));
      if (best > FIX_NOWHERE / 2 && best < top - FIX_SPARE) loses |= 1u << (j - 2);
    }
    return loses;
  }
};
// The warp's cells again in FP64: those that lose bits on integers (FixedReach),
// or `all`, for values that fit no scale (NaN, infinities, negative 1/m, the ends
// of the exponent range). The others' results stay, as do their shares of acc, but
// for CHECK, whose whole sum it forms. Apart from the kernel, whose registers it
// would cost; the march on integers only watches whether any warp needs it, which
// is 3 % of a product or an iteration (256^3 400 -> 411 us, 161x127x190 202 -> 207,
// 64^3 34.2 -> 35.1). A product of 256^3 cells takes 412 us, 1107 with values of
// 1e-12 around a one in every 16^3 cells, 563 with values that fall by e^40 along
// z, 686 with a NaN in every 16^3 cells (pressure_stencil<double> 1160 each); an
// iteration at 161x127x190 from a right-hand side of one cell 485 (499).
template <int MODE, int RY>
__device__ __noinline__ double fixed_finish(const GridDev& g, const StencilArgs<double>& a, double alpha, int top,
                                            bool all, int y0, int z0, int z1, double acc, unsigned* hx) {
  const int lane = threadIdx.x & 31, cx = blockIdx.x * FX_COLS + lane - 1;
  const bool own = cx >= 0 && cx < g.cX && lane >= 1 && lane <= FX_COLS;
  unsigned mine = 0;  // own rows
#pragma unroll
  for (int j = 0; j < RY; j++) mine |= own && y0 + j < g.cY ? 1u << j : 0u;
  FixedLayer<MODE, RY> l, n;
  if (MODE == S_APPLY && !all) {  // the layers that have any (a solve's reads cost more than the march saves)
    FixedReach<RY> reach;
    int first = INT_MAX, last = -1;
    n.load(g, a, alpha, cx, y0, z0 - 1, z1);
    for (int kk = z0 - 1; kk <= z1; kk++) {
      l = n;
      n.load(g, a, alpha, cx, y0, kk + 1, z1);
      if (reach.next(l, top) & mine && kk > z0) {
        first = min(first, kk - 1);
        last = kk - 1;
      }
    }
    z0 = __reduce_min_sync(0xffffffffu, first);
    z1 = __reduce_max_sync(0xffffffffu, last) + 1;
    if (z0 >= z1) return acc;
  }
  if (MODE == S_CHECK) acc = 0.0;
  FixedReach<RY> reach;
  double own_value[RY] = {};  // of the layer before
  double prev[RY + 2] = {}, mpx[RY + 1] = {}, mpy[RY + 1] = {}, mpz[RY + 1] = {};
  n.load(g, a, alpha, cx, y0, z0 - 1, z1);
  for (int kk = z0 - 1; kk <= z1; kk++) {
    l = n;
    n.load(g, a, alpha, cx, y0, kk + 1, z1);
    const unsigned loses = (all ? ~0u : reach.next(l, top)) & mine;
    double dp, xp, xq, vp = 0.0;  // as in the march on integers
#pragma unroll
    for (int j = 0; j < RY + 2; j++) {
      const double old = prev[j], P = old + l.v[j], Q = old - l.v[j];
      prev[j] = l.v[j];
      if (kk < z0) continue;
      const double pn = shfl_down(P), qn = shfl_down(Q);
      const double dp1 = P - pn, xp1 = P + pn, xq1 = Q + qn;
      if (j > 0) {
        const double m = l.m[j - 1];
        const double mx = (dp + dp1) * m, my = (xp - xp1) * m, mz = (xq + xq1) * m;
        if (kk > z0) {
          const double A = mpx[j - 1] + mx, B = mpy[j - 1] + my, C = mz - mpz[j - 1];
          const double CA = C - A, AC = A + C;
          const double up = shfl_up(CA + B), um = shfl_up(CA - B);
          if (j > 1) {
            const double o = (vp + up) + (AC + B);
            const long long c = cx + (long long)(y0 + j - 2) * g.cX + (long long)(kk - 1) * g.cslab;
            const bool it = loses >> (j - 2) & 1u;
            if (MODE == S_APPLY) {
              if (it) a.out[c] = o;
            } else if (MODE == S_UPDATE) {
              if (it) {
                acc += own_value[j - 2] * (o - a.out[c]);
                a.out[c] = o;
              }
            } else if (MODE == S_CHECK) {
              const double e = mine >> (j - 2) & 1u ? o - a.b[c] : 0.0;
              acc += e * e;
            } else if (MODE == S_RESID_INIT) {
              if (it) {
                const double rn = (a.b[c] - o) * a.invd[c];
                a.r[c] = rn;
                *hx = max(*hx, fixed_mag(rn));
              }
            }
          }
          vp = (AC - B) + um;
        }
        mpx[j - 1] = mx;
        mpy[j - 1] = my;
        mpz[j - 1] = mz;
      }
      dp = dp1;
      xp = xp1;
      xq = xq1;
    }
#pragma unroll
    for (int j = 0; j < RY; j++) own_value[j] = l.v[j + 1];
  }
  return acc;
}

// The bound of v = r - alpha Ap/diag from the largest |r| and |Ap/diag|, as a
// high word (fixed_mag); what lies below the scale's range gets its lowest.
__device__ __forceinline__ unsigned fixed_bound(unsigned hr, unsigned hq, double alpha) {
  const double b = from_words(hr, ~0u) + fabs(alpha) * from_words(hq, ~0u);
  return fixed_mag(b * 1.0000001);
}
// blocks an SM holds: the products' scan wants the registers, the solves' modes fit four
template <int MODE>
constexpr int FX_RESIDENT = MODE == S_APPLY ? 3 : 4;
template <int MODE, int RY>
__global__ void __launch_bounds__(FX_T, FX_RESIDENT<MODE>) pressure_stencil_fixed(const __grid_constant__ GridDev g,
                                                                                      const __grid_constant__ StencilArgs<double> a,
                                                                                      int cz) {
  extern __shared__ double ring[];  // [2][slots][FX_T]
  if (MODE != S_APPLY && a.st->done) return;
  constexpr int SLOTS = fx_slots<MODE, RY>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cx = blockIdx.x * FX_COLS + lane - 1;  // this lane's cell column; its node column is cx + 1
  const int y0 = (blockIdx.y * FX_W + warp) * RY;
  const int z0 = blockIdx.z * cz, z1 = min(z0 + cz, g.cZ);
  const bool col = cx >= 0 && cx < g.cX;
  const bool own = col && lane >= 1 && lane <= FX_COLS;
  const bool nodeCol = cx >= 0 && cx < g.cX - 1;
  const double alpha = MODE == S_UPDATE ? a.st->alpha : 0.0;
  double acc = 0.0;
  unsigned hx = 0;  // UPDATE: largest new x; RESID_INIT: largest r
  // how far down the values reach: the least over the cells of the largest in the
  // three rows around it (high words less one; all zero: none). A cell that loses
  // bits has small ones only around it, in its own column or one beside it.
  unsigned least = ~0u;
  const int rows = min(RY, g.cY - y0);
  auto cell = [&](int y, int z) { return cx + (long long)y * g.cX + (long long)z * g.cslab; };
  auto node = [&](int y, int z) { return cx + 1 + (long long)y * g.X + (long long)z * g.slab; };
  if (y0 < g.cY) {
    unsigned hv, hm, lm;  // bounds of v and 1/m; the least 1/m's high word less one
    if (MODE == S_APPLY) {  // this warp's own values
      hv = hm = 0;
      lm = ~0u;
      // (four layers' loads in flight: one layer at a time the scan took as long
      // as the march)
      for (int z = z0 - 1; z <= z1; z += 4) {
        double v[4][RY + 2], m[4][RY + 1];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int j = 0; j < RY + 2; j++) {
            const int y = y0 - 1 + j, zk = z + k;
            v[k][j] = col && y >= 0 && y < g.cY && zk >= 0 && zk < g.cZ && zk <= z1 ? a.in[cell(y, zk)] : 0.0;
            if (j > 0) m[k][j - 1] = nodeCol && y > 0 && y < g.Y - 1 && zk > 0 && zk <= z1 && zk < g.Z - 1 ? a.minv[node(y, zk)] : 0.0;
          }
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int j = 0; j < RY + 2; j++) {
            const unsigned h = fixed_mag1(v[k][j]);
            hv = max(hv, h);
            if (j > 0) {
              if (j > 1 && j - 2 < rows) least = min(least, max(max(h, fixed_mag1(v[k][j - 1])), fixed_mag1(v[k][j - 2])) - 1u);
              const unsigned w = hi_word(m[k][j - 1]) | (lo_word(m[k][j - 1]) ? 1u : 0u);
              hm = max(hm, w);
              lm = min(lm, w - 1u);
            }
          }
      }
      hv = __reduce_max_sync(0xffffffffu, hv);
      hm = __reduce_max_sync(0xffffffffu, hm);
      lm = __reduce_min_sync(0xffffffffu, lm);
    } else {
      hm = a.st->hm;
      lm = ~a.st->lm;
      hv = MODE == S_UPDATE ? a.st->hv : a.st->hx;
    }
    const int Em = fixed_exp(hm), Ev = fixed_scale(hv, hm);
    const bool ok = fixed_ok(hv, hm);
    if (MODE == S_APPLY && (!ok || fixed_low(hv, hm))) {
      fixed_finish<MODE, RY>(g, a, alpha, 0, true, y0, z0, z1, 0.0, nullptr);
      return;
    }
    // (in a solve, a scale that does not fit is a value on its way to infinity,
    // or NaN: the sums say so)
    if (!ok) acc = from_words(0x7ff80000u, 0u);
    Fix prev[RY + 2], mpx[RY + 1], mpy[RY + 1], mpz[RY + 1];
    double vo[RY];  // UPDATE: v of the own rows, layer kk - 1
#pragma unroll
    for (int j = 0; j < RY + 2; j++) prev[j] = Fix{0, 0, 0};
#pragma unroll
    for (int j = 0; j < RY + 1; j++) mpx[j] = mpy[j] = mpz[j] = Fix{0, 0, 0};
#pragma unroll
    for (int j = 0; j < RY; j++) vo[j] = 0.0;
    auto fetch = [&](int kk) {
      double* q = ring + ((kk & 1) * SLOTS) * FX_T + threadIdx.x;
      const bool layer = kk >= 0 && kk < g.cZ;
      int slot = 0;
#pragma unroll
      for (int j = 0; j < RY + 2; j++) {
        const int y = y0 - 1 + j;
        const bool in = layer && col && y >= 0 && y < g.cY;
        const long long c = in ? cell(y, kk) : 0;
        if (MODE == S_UPDATE) {
          fetch8(q + FX_T * slot++, a.r + c, in);
          fetch8(q + FX_T * slot++, a.Ap + c, in);
          fetch8(q + FX_T * slot++, a.invd + c, in);
        } else {
          fetch8(q + FX_T * slot++, a.in + c, in);
        }
      }
#pragma unroll
      for (int j = 0; j < RY + 1; j++) {
        const int ny = y0 + j;
        const bool in = nodeCol && ny > 0 && ny < g.Y - 1 && kk > 0 && kk < g.Z - 1;
        fetch8(q + FX_T * slot++, a.minv + (in ? node(ny, kk) : 0), in);
      }
      if (MODE == S_UPDATE)
#pragma unroll
        for (int j = 0; j < RY; j++) {
          const bool in = own && y0 + j < g.cY && kk >= z0 && kk < z1;
          const long long c = in ? cell(y0 + j, kk) : 0;
          fetch8(q + FX_T * slot++, a.x + c, in);
          fetch8(q + FX_T * slot++, a.d + c, in);
        }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (ok) fetch(z0 - 1);
    for (int kk = z0 - 1; kk <= z1 && ok; kk++) {
      if (kk < z1) {
        fetch(kk + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      const double* q = ring + ((kk & 1) * SLOTS) * FX_T + threadIdx.x;
      constexpr int IN = (MODE == S_UPDATE ? 3 : 1), M0 = IN * (RY + 2), X0 = M0 + RY + 1;
      double v[RY + 2];
#pragma unroll
      for (int j = 0; j < RY + 2; j++)
        v[j] = MODE == S_UPDATE
                   ? upd_r(q[FX_T * (3 * j)], alpha, q[FX_T * (3 * j + 1)], q[FX_T * (3 * j + 2)])
                   : q[FX_T * j];
      if (MODE != S_APPLY)
#pragma unroll
        for (int j = 2; j < RY + 2; j++)
          if (j - 2 < rows) least = min(least, max(max(fixed_mag(v[j - 2]), fixed_mag(v[j - 1])), fixed_mag(v[j])) - 1u);
      if (MODE == S_UPDATE && kk >= z0 && kk < z1) {
#pragma unroll
        for (int j = 0; j < RY; j++)
          if (own && y0 + j < g.cY) {
            const double xn = q[FX_T * (X0 + 2 * j)] + alpha * q[FX_T * (X0 + 2 * j + 1)];
            a.x[cell(y0 + j, kk)] = xn;
            hx = max(hx, fixed_mag(xn));
          }
      }
      Fix dp, xp, xq, vp = Fix{0, 0, 0};  // of the cell row before; a + c - b of the node row before
#pragma unroll
      for (int j = 0; j < RY + 2; j++) {
        const Fix f = fixed_from(v[j], Ev);
        const Fix P = prev[j] + f, Q = prev[j] - f;
        prev[j] = f;
        if (kk < z0) continue;
        const Fix pn = shfl_down(P), qn = shfl_down(Q);
        const Fix dp1 = P - pn, xp1 = P + pn, xq1 = Q + qn;
        if (j > 0) {
          const NodeFactor m = factor_from(q[FX_T * (M0 + j - 1)], Em);
          const Fix mx = fixed_mul(dp + dp1, m), my = fixed_mul(xp - xp1, m), mz = fixed_mul(xq + xq1, m);
          if (kk > z0) {
            const Fix A = mpx[j - 1] + mx, B = mpy[j - 1] + my, C = mz - mpz[j - 1];
            const Fix CA = C - A, AC = A + C;
            const Fix up = shfl_up(CA + B), um = shfl_up(CA - B);
            if (j > 1) {  // output cell row y0 + j - 2, layer kk - 1
              const double o = fixed_to((vp + up) + (AC + B), Ev + Em);
              if (own && y0 + j - 2 < g.cY) {
                const long long c = cell(y0 + j - 2, kk - 1);
                if (MODE == S_APPLY) {
                  a.out[c] = o;
                } else if (MODE == S_UPDATE) {
                  a.out[c] = o;
                  acc += vo[j - 2] * o;
                } else if (MODE == S_CHECK) {
                  const double e = o - a.b[c];
                  acc += e * e;
                } else if (MODE == S_RESID_INIT) {
                  const double bb = a.b[c], rn = (bb - o) * a.invd[c];
                  a.r[c] = rn;
                  hx = max(hx, fixed_mag(rn));
                  acc += bb * bb;
                }
              }
            }
            vp = (AC - B) + um;
          }
          mpx[j - 1] = mx;
          mpy[j - 1] = my;
          mpz[j - 1] = mz;
        }
        dp = dp1;
        xp = xp1;
        xq = xq1;
      }
      if (MODE == S_UPDATE)
#pragma unroll
        for (int j = 0; j < RY; j++) vo[j] = v[j + 1];
    }
    least = __reduce_min_sync(0xffffffffu, least);
    if (ok && least != ~0u && Ev - fixed_exp(least + 1u) + (Em - fixed_exp(lm + 1u)) > FIX_SPARE) {
      unsigned h = hx;
      acc = fixed_finish<MODE, RY>(g, a, alpha, Ev + Em, false, y0, z0, z1, acc, &h);
      hx = h;
    }
  }
  if (MODE == S_APPLY) return;
  if (MODE == S_UPDATE || MODE == S_RESID_INIT) block_max(hx, MODE == S_UPDATE ? &a.st->hx : &a.st->hr);
  const double bs = block_sum<FX_T>(acc);
  const int nblocks = gridDim.x * gridDim.y * gridDim.z;
  double total;
  PcrState L, *const st = &L;
  if (last_block_state<FX_T, 1>(bs, a.partial, a.st, nblocks, &total, st)) {
    if (MODE == S_UPDATE) {
      finish_update(st, total);
    } else if (MODE == S_CHECK) {
      finish_check(st, total);
    } else if (MODE == S_RESID_INIT) {
      st->bnorm2 = total;
      st->hv = fixed_bound(st->hr, 0u, 0.0);
      st->hr = 0;
    }
    *a.st = L;
  }
}

// Bounds a fixed-point solve starts from: the largest |x|, and the largest 1/m
// of the interior nodes (a negative one's sign bit makes it the largest); and the
// complement of their least 1/m's word less one (0: all are zero). The words are
// zero before.
__global__ void __launch_bounds__(256) fixed_bounds(GridDev g, const double* x, const double* minv, unsigned* hx,
                                                    unsigned* hm, unsigned* lm) {
  unsigned mx = 0, mm = 0, ml = 0;
  const long long stride = (long long)gridDim.x * 256;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < g.R; i += stride) mx = max(mx, fixed_mag(x[i]));
  for (long long n = blockIdx.x * 256LL + threadIdx.x; n < g.T; n += stride) {
    const int i = (int)(n % g.X), j = (int)((n / g.X) % g.Y), k = (int)(n / g.slab);
    if (i > 0 && j > 0 && k > 0 && i < g.X - 1 && j < g.Y - 1 && k < g.Z - 1) {
      const unsigned w = hi_word(minv[n]) | (lo_word(minv[n]) ? 1u : 0u);
      mm = max(mm, w);
      ml = max(ml, ~(w - 1u));
    }
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  mm = __reduce_max_sync(0xffffffffu, mm);
  ml = __reduce_max_sync(0xffffffffu, ml);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(hx, mx);
    atomicMax(hm, mm);
    atomicMax(lm, ml);
  }
}

// Launch shape: rows a warp and z-chunk depth, the ones of least cost in a model
// of what was measured. A block marches cz + 2 layers, and half of one is its
// start and end. An SM holds three blocks of a product's kernel, four of a
// solve's, so each of its schedulers as many of their warps: a warp alone issues
// every 4.5 cycles, two hardly disturb each other, three share half an issue a
// cycle (cost of a layer 4.5, 4.7, 6 and 7.5); more blocks run in waves. Products
// take two rows a warp or four (1.65 times the instructions of two), solves two:
// with four an iteration took 65 us for 61 at 96^3, 212 for 201 at 161x127x190,
// 745 for 733 at 256^3. Against fixed numbers of warps by size, an iteration took
// 41 for 53 us at 80^3, 121 for 130 at 128^3, 44 for 63 at 32x33x300; 64^3 the same
// (these before the watch for cells that lose bits, which costs each 3 %).
struct FixedShape {
  int ry, cz;
  dim3 grid;
};
static FixedShape fixed_shape(const GridDev& g, bool solve) {
  FixedShape best{};
  double least = 0;
  const long long gx = (g.cX + FX_COLS - 1) / FX_COLS;
  const int resident = solve ? FX_RESIDENT<S_UPDATE> : FX_RESIDENT<S_APPLY>;
  const double layer[5] = {0.0, 4.5, 4.7, 6.0, 7.5};
  for (int ry = 2; ry <= (solve ? 2 : 4); ry += 2) {
    const long long gy = (g.cY + FX_W * ry - 1) / (FX_W * ry), gxy = gx * gy;
    // the most chunks that a number of blocks an SM leaves room for
    const int last = (int)((gxy + 151) / 152) + 5 * resident;
    for (int k = 1; k <= last; k += k < resident ? 1 : resident) {
      long long n = 152LL * k / gxy;
      if (n < 1) n = 1;
      if (n > g.cZ) n = g.cZ;
      const int cz = (int)((g.cZ + n - 1) / n), gz = (g.cZ + cz - 1) / cz;
      const int per = (int)((gxy * gz + 151) / 152);
      const double cost = (cz + 2.5) * ((per / resident) * layer[resident] + layer[per % resident]) *
                          (ry == 2 ? 1.0 : 1.65);
      if (!best.ry || cost < least) {
        least = cost;
        best.ry = ry;
        best.cz = cz;
        best.grid = dim3((unsigned)gx, (unsigned)gy, (unsigned)gz);
      }
      if (n == g.cZ) break;
    }
  }
  return best;
}
template <int MODE, int RY>
static void launch_fixed_rows(const GridDev& g, const StencilArgs<double>& a, const FixedShape& s, cudaStream_t st) {
  constexpr int smem = fx_smem<MODE, RY>();
  static const cudaError_t attr = cudaFuncSetAttribute(pressure_stencil_fixed<MODE, RY>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  (void)attr;  // a refusal shows as the launch's error
  ESF_COUNTED pressure_stencil_fixed<MODE, RY><<<s.grid, FX_T, smem, st>>>(g, a, s.cz);
}
template <int MODE>
static void launch_fixed(const GridDev& g, const StencilArgs<double>& a, const FixedShape& s, cudaStream_t st) {
  if constexpr (MODE == S_APPLY) {
    if (s.ry == 4) {
      launch_fixed_rows<MODE, 4>(g, a, s, st);
      return;
    }
  }
  launch_fixed_rows<MODE, 2>(g, a, s, st);
}
// Whether a grid's FP64 products and solves use it. It is the faster one at
// every size and shape measured, a product and a solve iteration in us: 8^3 7.5
// and 17 against 18.1 and 31, 20^3 7.5 and 19 against 18.6 and 33; 3x200x200 cells
// (x y z) 37 and 60 against 107 and 156, 200x3x200 17 and 32 against 35 and 61,
// 200x200x3 14 and 28 against 23 and 42; 32x33x300 29 and 45 against 41 and 83. Below
// 8192 cells, where a step is its launches, FP64 in pressure_stencil's order
// stays, whose results to the last bit whole steps on such grids are compared
// by. More blocks than the sums have room for stay too.
static bool fixed_pays(const GridDev& g, bool solve, FixedShape* s) {
  if (g.R < 8192) return false;
  *s = fixed_shape(g, solve);
  return (long long)s->grid.x * s->grid.y * s->grid.z <= FX_MAX_BLOCKS && s->grid.y <= 65535 && s->grid.z <= 65535;
}
