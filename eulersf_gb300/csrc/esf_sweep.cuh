// The Gauss-Seidel sweeps of the coupled step: sweepPhi (the Eikonal distance
// of computeSDF) and sweepOnePass (the velocity extension). Included by
// esf_kernels.cuh inside namespace esf (esf_step.cu, compiled -fmad=false).
//
// Node (i,j,k) of a pass reads its three upwind neighbours as updated in the
// same pass, so every order in which each node comes after its three upwind
// neighbours gives the sequential loop's result bit for bit.
#pragma once

// solveDistance (DEFOR_SOLID_3D.cpp:369-394), in the reference's steps.
__device__ __forceinline__ void solve_distance(double p, double q, double r, double* v) {
  // std::min / std::max semantics: (b < a) ? b : a
  double ds[3];
  double mqr = (r < q) ? r : q, Mqr = (q < r) ? r : q;
  ds[0] = (mqr < p) ? mqr : p;
  ds[2] = (p < Mqr) ? Mqr : p;
  ds[1] = p + q + r - ds[0] - ds[2];
  double b[3], c[3];
  b[0] = ds[0];
  c[0] = ds[0] * ds[0] - 1.0f;
  for (int x = 1; x < 3; x++) {
    b[x] = ds[x] + b[x - 1];
    c[x] = ds[x] * ds[x] + c[x - 1];
  }
  int i = 2;
  double discrim = b[i] * b[i] - (double)(i + 1) * c[i];
  double nd = (b[i] + sqrt(discrim)) / (double)(i + 1);
  while ((discrim < 0.0f || nd < ds[i]) && i != -1) {
    i--;
    if (i < 0) break;
    discrim = b[i] * b[i] - (double)(i + 1) * c[i];
    if (discrim > 0.0f) nd = (b[i] + sqrt(discrim)) / (double)(i + 1);
  }
  if (nd < *v) *v = nd;
}

// x / 3 rounded to nearest, without a division: the quotient by the rounded
// reciprocal, corrected by its exact remainder (Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", 2004).
__device__ __forceinline__ double third(double x) {
  const double y = 1.0 / 3.0;
  const double q = x * y;
  return __fma_rn(__fma_rn(-3.0, q, x), y, q);
}

// a < b by their bits, for numbers (no NaN) that are not both negative unless they
// are the same: phi is -1/2 at nodes with mass and positive elsewhere, as the root
// of sum over ds_i < t of (t - ds_i)^2 = 1 lies at least 1/sqrt(3) above the least
// ds_i. 15 cycles, where an FP64 comparison and a select on it take 104.
__device__ __forceinline__ bool less_bits(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
// x to 24 bits, towards zero, as a float, 0 below 2^-126, by its bits (a conversion is an FP64
// operation); for numbers below 2^128.
__device__ __forceinline__ float near_float(double x) {
  const int hi = __double2hiint(x), m = hi & 0x7fffffff;
  const int e = m - (896 << 20);
  return __int_as_float((hi & 0x80000000) | (e > 0 ? (e << 3) | (int)((unsigned)__double2loint(x) >> 29) : 0));
}

// sqrt(x), x not negative
__device__ __forceinline__ double root(double x) {
  if ((unsigned)(__double2hiint(x) - (963 << 20)) >= (120u << 20)) return sqrt(x);  // not in 2^-60 .. 2^60
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(leading_float(x)));
  return root_from(x, y);
}

// The same update, with the FP64 work that cannot change its outcome left
// out. GB300 takes an FP64 instruction from a warp every 63 cycles, so their
// number is most of a node's time (27 here at first with sqrt() and the quotient
// by FMAs, 2740 cycles a node of a lone chain; 20 now, 2150), so:
//  * a node whose value v already lies below the new distance keeps it. The
//    new distance is the root of sum over ds_i < t of (t - ds_i)^2 = 1, whose
//    left side grows with t: where it is below `skipBelow` (0.99) at t = v,
//    the root is above v. FP32 copies decide it; their rounding moves the sum
//    by at most 4e-3 for distances up to 4096, and callers with larger ones
//    pass skipBelow = 0, which skips nothing;
//  * the reference tries the three-, two- and one-neighbour root in turn and
//    takes the first that is not below its largest neighbour. The i-neighbour
//    root lies below ds_i exactly where sum over j < i of (ds_i - ds_j)^2 > 1:
//    where FP32 shows that by a margin, the root is not formed. (At i = 1 the
//    reference keeps the last root where the discriminant is exactly 0, at
//    (ds_1 - ds_0)^2 = 2: a band around that, and any start with a
//    discriminant that is not positive, takes the reference's own steps.)
// Every value it returns is solve_distance's, bit for bit. Returns whether v
// changed.
__device__ __forceinline__ bool solve_distance_fast(double p, double q, double r, double& v, float fp, float fq,
                                                    float fr, float fv, float skipBelow) {
  const float tp = fmaxf(fv - fp, 0.0f), tq = fmaxf(fv - fq, 0.0f), tr = fmaxf(fv - fr, 0.0f);
  if (__fmaf_rn(tp, tp, __fmaf_rn(tq, tq, tr * tr)) < skipBelow) return false;
  const bool rq = less_bits(r, q);
  const double mqr = rq ? r : q, Mqr = rq ? q : r;  // (equal ones are the same)
  const double ds0 = less_bits(mqr, p) ? mqr : p, ds2 = less_bits(p, Mqr) ? Mqr : p;
  const double ds1 = p + q + r - ds0 - ds2;
  const float lo = fminf(fminf(fp, fq), fr), hi = fmaxf(fmaxf(fp, fq), fr), mid = fp + fq + fr - lo - hi;
  const float e1 = mid - lo, e2 = hi - lo, e21 = hi - mid;
  int i = 2;
  if (skipBelow > 0.0f && __fmaf_rn(e2, e2, e21 * e21) > 1.01f)
    i = (e1 * e1 > 1.01f && fabsf(__fmaf_rn(e1, e1, -2.0f)) > 0.02f) ? 0 : 1;
  const double c0 = ds0 * ds0 - 1.0;
  const double b1 = ds1 + ds0, c1 = ds1 * ds1 + c0;
  const double b2 = ds2 + b1, c2 = ds2 * ds2 + c1;
  auto positive = [](double d) { return __double_as_longlong(d) > 0; };  // (a difference: no NaN, no -0)
  auto negative = [](double d) { return __double2hiint(d) < 0; };
  // lanes of all i take the one path: K and the operands are selected, not the
  // results (1 c and 2 c are exact, t / 2 as well)
  bool nan = true, first = true;  // nd is NaN until a discriminant is not negative
  double nd = 0.0;
  for (;;) {
    const double b = i == 2 ? b2 : i == 1 ? b1 : ds0, c = i == 2 ? c2 : i == 1 ? c1 : c0;
    const double k = i == 2 ? 3.0 : i == 1 ? 2.0 : 1.0;
    const double discrim = b * b - k * c;
    if (first && i < 2 && !positive(discrim)) {
      i = 2;
      continue;
    }
    if (first ? !negative(discrim) : positive(discrim)) {
      const double t = b + root(discrim);
      if ((unsigned)(__double2hiint(t) - (100 << 20)) < (1900u << 20))
        nd = i == 2 ? third_of(t) : i == 1 ? half_of(t) : t;
      else  // (not a positive normal number)
        nd = i == 2 ? third(t) : i == 1 ? t * 0.5 : t;
      nan = false;
    }
    first = false;
    if (!negative(discrim) && (nan || !less_bits(nd, i == 2 ? ds2 : i == 1 ? ds1 : ds0))) break;
    if (--i < 0) break;
  }
  if (nan || !less_bits(nd, v)) return false;
  v = nd;
  return true;
}

// One pass: first index in sweep order, direction and count per axis.
struct Sweep {
  int i0, j0, k0;   // first index in sweep order
  int di, dj, dk;   // +1 / -1
  int ni, nj, nk;   // counts
};

// ---------------------------------------------- velocity extension (a19)
// DEFOR_SOLID_3D::sweepOnePass (DEFOR_SOLID_3D.cpp:457-519). Its
// solvableX/Y/Z flags live for the whole pass and, once cleared, stay
// cleared: a node sees a flag cleared iff some node at or before it in loop
// order triggered it. Triggers depend on phi and mass only (constant during
// the extension), so the first trigger rank of each flag is found by a min
// reduction before the passes run.

// First trigger rank of the three pass-long flags of sweepOnePass, by
// atomicMin over all nodes of the pass (ranks: long long loop order), for the
// eight directions (one grid row each).
struct Sweep8 {
  Sweep d[8];
};
__global__ void k_sweep_vec_ranks(GridDev g, const double* ph, const double* ms, const Sweep8 all,
                                  unsigned long long* ranks) {
  __shared__ unsigned long long sm[3];
  const Sweep w = all.d[blockIdx.y];
  ranks += 3 * blockIdx.y;
  if (threadIdx.x < 3) sm[threadIdx.x] = ~0ull;
  __syncthreads();
  unsigned long long r0 = ~0ull, r1 = ~0ull, r2 = ~0ull;
  const long long nij = (long long)w.ni * w.nj, total = nij * w.nk;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    int a = (int)(t % w.ni), b = (int)((t / w.ni) % w.nj), c = (int)(t / nij);
    int i = w.i0 + a * w.di, j = w.j0 + b * w.dj, k = w.k0 + c * w.dk;
    long long n = nidx(g, i, j, k);
    if (ms[n] != 0) continue;
    double pn = ph[n];
    double dp = pn - ph[nidx(g, i - w.di, j, k)], dpn = pn - ph[nidx(g, i + w.di, j, k)];
    if (dp < 0 && dpn >= 0) continue;
    if (dp < 0 && dpn < 0 && (unsigned long long)t < r0) r0 = t;
    double dq = pn - ph[nidx(g, i, j - w.dj, k)], dqn = pn - ph[nidx(g, i, j + w.dj, k)];
    if (dq < 0 && dqn >= 0) continue;
    if (dq < 0 && dqn < 0 && (unsigned long long)t < r1) r1 = t;
    double dr = pn - ph[nidx(g, i, j, k - w.dk)], drn = pn - ph[nidx(g, i, j, k + w.dk)];
    if (dr < 0 && drn >= 0) continue;
    if (dr < 0 && drn < 0 && (unsigned long long)t < r2) r2 = t;
  }
  // one shared-memory and one global atomic per block and flag
  if (r0 != ~0ull) atomicMin(&sm[0], r0);
  if (r1 != ~0ull) atomicMin(&sm[1], r1);
  if (r2 != ~0ull) atomicMin(&sm[2], r2);
  __syncthreads();
  if (threadIdx.x < 3 && sm[threadIdx.x] != ~0ull) atomicMin(&ranks[threadIdx.x], sm[threadIdx.x]);
}

// Blend weights of the eight directions' passes: (alpha, beta) of each node
// in loop order, or SWEEP_KEEP in alpha's place where the pass leaves the node
// as it is. Which nodes those are, and the weights, depend on phi, the mass
// and the flags only, which the four rounds of the extension do not change:
// formed once a direction instead of once a pass, and off the passes' critical
// path (two divisions a node). A pass leaves a node where phi falls away from
// the sweep on some axis, which is everywhere but in about one octant of the
// box; its bounds go to dims[8][6] (first and last a, b, c; the host presets
// INT_MAX and -1).
constexpr unsigned long long SWEEP_KEEP = 0x7ff4000000000001ull;  // a signalling NaN: no arithmetic gives it
__global__ void __launch_bounds__(KT) k_sweep_vec_weights(GridDev g, const double* ph, const double* ms,
                                                          const Sweep8 all, const unsigned long long* ranks,
                                                          double2* wt, int* dims) {
  __shared__ int sd[6];
  if (threadIdx.x < 6) sd[threadIdx.x] = threadIdx.x % 2 ? -1 : INT_MAX;
  __syncthreads();
  const Sweep w = all.d[blockIdx.y];
  ranks += 3 * blockIdx.y;
  dims += 6 * blockIdx.y;
  const unsigned long long rx = ranks[0], ry = ranks[1], rz = ranks[2];
  const long long nij = (long long)w.ni * w.nj, total = nij * w.nk;
  wt += blockIdx.y * total;
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {-1, -1, -1};
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int p[3] = {(int)(t % w.ni), (int)((t / w.ni) % w.nj), (int)(t / nij)};
    const int i = w.i0 + p[0] * w.di, j = w.j0 + p[1] * w.dj, k = w.k0 + p[2] * w.dk;
    const long long n = nidx(g, i, j, k);
    double2 out = make_double2(__longlong_as_double((long long)SWEEP_KEEP), 0.0);
    if (ms[n] == 0) {
      const double pn = ph[n];
      double dp = pn - ph[nidx(g, i - w.di, j, k)], dpn = pn - ph[nidx(g, i + w.di, j, k)];
      bool skip = dp < 0 && dpn >= 0;
      double dq = 0, dqn = 0, dr = 0, drn = 0;
      if (!skip) {
        dq = pn - ph[nidx(g, i, j - w.dj, k)];
        dqn = pn - ph[nidx(g, i, j + w.dj, k)];
        skip = dq < 0 && dqn >= 0;
      }
      if (!skip) {
        dr = pn - ph[nidx(g, i, j, k - w.dk)];
        drn = pn - ph[nidx(g, i, j, k + w.dk)];
        skip = dr < 0 && drn >= 0;
      }
      if (!skip) {
        if ((unsigned long long)t >= rx) dp = 0;
        if ((unsigned long long)t >= ry) dq = 0;
        if ((unsigned long long)t >= rz) dr = 0;
        if (dp + dq + dr < 1e-3) {
          out = make_double2(0.333, 0.333);
        } else {
          out = make_double2(dp / (dp + dq + dr), dq / (dp + dq + dr));
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
          lo[q] = min(lo[q], p[q]);
          hi[q] = max(hi[q], p[q]);
        }
      }
    }
    wt[t] = out;
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    lo[q] = __reduce_min_sync(0xffffffffu, lo[q]);
    hi[q] = __reduce_max_sync(0xffffffffu, hi[q]);
    if ((threadIdx.x & 31) == 0 && hi[q] >= 0) {
      atomicMin(&sd[2 * q], lo[q]);
      atomicMax(&sd[2 * q + 1], hi[q]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 6 && sd[1] >= 0) {
    if (threadIdx.x % 2) atomicMax(&dims[threadIdx.x], sd[threadIdx.x]);
    else atomicMin(&dims[threadIdx.x], sd[threadIdx.x]);
  }
}

// A direction's work list: the nodes its passes change, and the nodes those
// read from upwind that it does not change (copies), by level a + b + c + 1
// (nodes of one level do not depend on one another). off[dir][levels + 1]:
// first entry of each level (counts while they are made); cur[dir][levels]:
// the fill's cursors. `entry` starts at the direction's first entry, first[dir].
struct SweepEntry {
  double alpha, beta, gamma;  // gamma = 1 - alpha - beta
  int node;
  int col;  // (b - b0) + (c - c0) nb in the octant's plane; ~col for a copy
};
struct SweepLists {
  int* off;
  int* cur;
  int* count;  // [8] entries of a direction
  SweepEntry* entry;
  int levels;  // ni + nj + nk - 1
};
// COUNT: off[level + 1] += 1 for each entry; otherwise the entries (in no
// particular order within a level). One grid row a direction; the nodes of the
// pass and those one before its first on each axis.
template <bool COUNT>
__global__ void __launch_bounds__(KT) k_sweep_vec_list(GridDev g, const Sweep8 all, const double2* wt,
                                                       const int* dims, SweepLists L) {
  const Sweep w = all.d[blockIdx.y];
  const int* dd = dims + 6 * blockIdx.y;
  if (dd[1] < 0) return;
  int* off = L.off + (long long)blockIdx.y * (L.levels + 1);
  int* cur = L.cur + (long long)blockIdx.y * L.levels;
  const long long nij = (long long)w.ni * w.nj;
  wt += blockIdx.y * nij * w.nk;
  const int b0 = dd[2] - 1, c0 = dd[4] - 1, nb = dd[3] - b0 + 1;
  // the octant and its upwind neighbours
  const int ea = dd[1] - dd[0] + 2, eb = nb, ec = dd[5] - c0 + 1;
  const long long total = (long long)ea * eb * ec;
  auto keeps = [&](long long t) {
    return (unsigned long long)__double_as_longlong(wt[t].x) == SWEEP_KEEP;
  };
  SweepEntry* entry = L.entry;
  if (!COUNT)
    for (int d = 0; d < (int)blockIdx.y; d++) entry += L.count[d];
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int a = dd[0] - 1 + (int)(t % ea), b = b0 + (int)((t / ea) % eb), c = c0 + (int)(t / ((long long)ea * eb));
    const long long p = a + (long long)b * w.ni + c * nij;  // loop place
    const bool change = a >= 0 && b >= 0 && c >= 0 && !keeps(p);
    // a copy: some downwind neighbour reads it (those lie inside the octant's
    // bounds or change nothing)
    const bool copy = !change && ((b >= 0 && c >= 0 && a < dd[1] && !keeps(p + 1)) ||
                                  (a >= 0 && c >= 0 && b < dd[3] && !keeps(p + w.ni)) ||
                                  (a >= 0 && b >= 0 && c < dd[5] && !keeps(p + nij)));
    if (!change && !copy) continue;
    const int level = a + b + c + 1;
    if (COUNT) {
      atomicAdd(&off[level + 1], 1);
    } else {
      SweepEntry e;
      e.alpha = e.beta = e.gamma = 0.0;
      if (change) {
        e.alpha = wt[p].x;
        e.beta = wt[p].y;
        e.gamma = 1 - e.alpha - e.beta;
      }
      e.node = (int)nidx(g, w.i0 + a * w.di, w.j0 + b * w.dj, w.k0 + c * w.dk);
      const int col = (b - b0) + (c - c0) * nb;
      e.col = change ? col : ~col;
      entry[atomicAdd(&cur[level], 1)] = e;
    }
  }
}
// Counts to first entries, one block per direction.
__global__ void __launch_bounds__(KT) k_sweep_vec_scan(SweepLists L) {
  __shared__ int sh[KT];
  int* off = L.off + (long long)blockIdx.x * (L.levels + 1);
  int* cur = L.cur + (long long)blockIdx.x * L.levels;
  int carry = 0;
  for (int l0 = 1; l0 <= L.levels; l0 += KT) {
    const int l = l0 + threadIdx.x;
    const int v = l <= L.levels ? off[l] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < KT; o <<= 1) {
      const int u = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += u;
      __syncthreads();
    }
    if (l <= L.levels) {
      off[l] = carry + sh[threadIdx.x];
      cur[l - 1] = carry + sh[threadIdx.x] - v;
    }
    carry += sh[KT - 1];
    __syncthreads();
  }
  if (threadIdx.x == 0) L.count[blockIdx.x] = carry;
}

// extendVectorField (DEFOR_SOLID_3D.cpp:566-574): four rounds of the eight
// directions' passes (sweepOnePass, DEFOR_SOLID_3D.cpp:457-519) and the face
// copies of sweepVectorField (:544-563), all in one launch. The three
// components of the velocity do not depend on one another, so block e runs
// component e from beginning to end and nothing crosses an SM. A pass walks the
// levels of its direction's list with one barrier each; the values a level
// reads were written in the level before to a shared-memory plane over the
// octant's (b, c) columns (one plane for even levels, one for odd). Entries
// are loaded two levels ahead and a copy's value one, so the chain of a level
// is three shared-memory reads, the blend and the barrier.
// What bounds it is the FP64 pipe of one SM (five instructions an entry, three
// products and two sums, at two lanes a cycle) and that chain, about 0.3 us a
// level: so entries are packed: one thread to a column, idle lanes included, took
// 134 us a pass against 118 us for lists read through L2 and 85 us here, at 64^3.
// Measured a step: tiles over the whole box 9.8 ms at 64^3 and 13.2 at 128^3, over
// the octant 7.0 and 9.6, this 2.7 and 5.6; larger octants: extend_velocity.
constexpr int EXTEND_THREADS = 1024;
__global__ void __launch_bounds__(EXTEND_THREADS) k_extend_field(GridDev g, double* f, const double* ms, Box ex,
                                                                 const Sweep8 all, const int* __restrict__ dims,
                                                                 SweepLists L, int planeCols) {
  extern __shared__ double plane[];  // 2 x planeCols, then the eight directions' off
  int* const off8 = reinterpret_cast<int*>(plane + 2 * planeCols);
  double* const v = f + blockIdx.x;  // this block's component
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int t = tid; t < 8 * (L.levels + 1); t += nt) off8[t] = L.off[t];
  __syncthreads();
  for (int round = 0; round < 4; round++) {
    const SweepEntry* list = L.entry;
    for (int dir = 0; dir < 8; dir++) {
      const int* off = off8 + dir * (L.levels + 1);
      const int* dd = dims + 6 * dir;
      const SweepEntry* E = list;
      list += off[L.levels];
      if (dd[1] < 0) continue;  // the pass changes nothing
      const int nb = dd[3] - dd[2] + 2;
      const int first = dd[0] + dd[2] + dd[4], last = dd[1] + dd[3] + dd[5] + 1;
      auto load = [&](int l, SweepEntry& e) {
        e.col = INT_MIN;
        if (l <= last) {
          const int i = off[l] + tid;
          if (i < off[l + 1]) {
            const double2* p = reinterpret_cast<const double2*>(E + i);
            const double2 x = __ldg(p), y = __ldg(p + 1);
            e.alpha = x.x;
            e.beta = x.y;
            e.gamma = y.x;
            e.node = __double2loint(y.y);
            e.col = __double2hiint(y.y);
          }
        }
      };
      auto old_value = [&](const SweepEntry& e) { return e.col < 0 && e.col != INT_MIN ? v[3 * e.node] : 0.0; };
      auto apply = [&](const SweepEntry& e, double old, const double* P, double* Q) {
        if (e.col >= 0) {
          const double x = (e.alpha * P[e.col] + e.beta * P[e.col - 1]) + e.gamma * P[e.col - nb];
          Q[e.col] = x;
          v[3 * e.node] = x;
        } else if (e.col != INT_MIN) {
          Q[~e.col] = old;
        }
      };
      SweepEntry e0, e1, e2;
      load(first, e0);
      load(first + 1, e1);
      double o0 = old_value(e0);
      for (int l = first; l <= last; l++) {
        load(l + 2, e2);
        const double o1 = old_value(e1);
        const double* P = plane + ((l + 1) & 1) * planeCols;
        double* Q = plane + (l & 1) * planeCols;
        apply(e0, o0, P, Q);
        for (int i = off[l] + tid + nt; i < off[l + 1]; i += nt) {
          const SweepEntry e = E[i];
          apply(e, old_value(e), P, Q);
        }
        __syncthreads();
        e0 = e1;
        e1 = e2;
        o0 = o1;
      }
    }
    // faces, one axis after the other, in the order z, y, x
    for (int axis = 2; axis >= 0; axis--) {
      const int s0 = axis == 0 ? 1 : 0, s1 = axis == 2 ? 1 : 2;
      const int n0 = ex.hi[s0] - ex.lo[s0], n1 = ex.hi[s1] - ex.lo[s1];
      const long long corner = nidx(g, ex.lo[0], ex.lo[1], ex.lo[2]);
      for (int t = tid; t < n0 * n1; t += nt) {
        const long long A = corner + (t % n0) * (axis == 0 ? (long long)g.X : 1ll) +
                            (t / n0) * (axis == 2 ? (long long)g.X : g.slab);
        const long long sa = axis == 0 ? 1 : axis == 1 ? (long long)g.X : g.slab;
        const long long Z = A + (ex.hi[axis] - ex.lo[axis] - 1) * sa;
        if (ms[A] == 0) v[3 * A] = v[3 * (A + sa)];
        if (ms[Z] == 0) v[3 * Z] = v[3 * (Z - sa)];
      }
      __syncthreads();
    }
  }
}

// The passes of larger octants as a wavefront of tiles: the octant's nodes (w is
// its sweep: its first node and its sides) are cut into tiles of ST^3, and launch
// P runs every tile (I, J, K) with I + J + K = P, whose three upwind tiles ran in
// launch P - 1: some 15 us, 22 planes of a chain of shared-memory reads each. At
// 256^3 a step of it took 22 ms for a ball of 113 nodes across, 31 for 154, 49 for
// 215 (the wave 57, 80 and 117, tiles over the whole box 31, 44 and 70). A block copies its tile and the upwind layer of each axis into
// shared memory and walks the tile's planes a' + b' + c' = q there, a barrier a
// plane. Weights in loop order: the octant's node (0, 0, 0) at wt[first], rows of
// ni, planes of nij.
constexpr int ST = 8, SP = ST + 1;  // tile edge; with the upwind layer
constexpr int TILE_THREADS = ST * ST * ST;
// launches of a pass over the octant of these bounds (k_sweep_vec_weights)
inline int sweep_tile_launches(const int* q) {
  return (q[1] - q[0]) / ST + (q[3] - q[2]) / ST + (q[5] - q[4]) / ST + 1;
}
__global__ void __launch_bounds__(TILE_THREADS) k_sweep_vec_tile(GridDev g, double* f, Sweep w, const double2* wt,
                                                                 long long first, int ni, long long nij, int P) {
  __shared__ double sv[3 * SP * SP * SP];
  __shared__ double2 sw[TILE_THREADS];
  const int nti = (w.ni + ST - 1) / ST, ntj = (w.nj + ST - 1) / ST, ntk = (w.nk + ST - 1) / ST;
  const int I = blockIdx.x % nti, J = blockIdx.x / nti, K = P - I - J;
  if (J >= ntj || K < 0 || K >= ntk) return;
  const int a0 = I * ST, b0 = J * ST, c0 = K * ST;
  const int na = min(ST, w.ni - a0), nb = min(ST, w.nj - b0), nc = min(ST, w.nk - c0);
  // local -1 .. n-1 on each axis (local -1 of the first tile is the node before
  // the octant's first, inside the box)
  for (int t = threadIdx.x; t < SP * SP * SP; t += TILE_THREADS) {
    const int la = t % SP - 1, lb = (t / SP) % SP - 1, lc = t / (SP * SP) - 1;
    if (la >= na || lb >= nb || lc >= nc) continue;
    const long long n = nidx(g, w.i0 + (a0 + la) * w.di, w.j0 + (b0 + lb) * w.dj, w.k0 + (c0 + lc) * w.dk);
#pragma unroll
    for (int q = 0; q < 3; q++) sv[3 * t + q] = f[3 * n + q];
  }
  const int ta = threadIdx.x % ST, tb = (threadIdx.x / ST) % ST, tc = threadIdx.x / (ST * ST);
  const bool in = ta < na && tb < nb && tc < nc;
  sw[threadIdx.x] = in ? wt[first + (a0 + ta) + (long long)(b0 + tb) * ni + (c0 + tc) * nij]
                       : make_double2(__longlong_as_double((long long)SWEEP_KEEP), 0.0);
  auto keeps = [&](int u) { return (unsigned long long)__double_as_longlong(sw[u].x) == SWEEP_KEEP; };
  __syncthreads();
  for (int q = 0; q <= (na - 1) + (nb - 1) + (nc - 1); q++) {
    const int lc = q - ta - tb;  // (the first ST^2 threads)
    if (threadIdx.x < ST * ST && lc >= 0 && lc < ST) {
      const int u = ta + tb * ST + lc * ST * ST;
      if (!keeps(u)) {
        const int s = (ta + 1) + (tb + 1) * SP + (lc + 1) * SP * SP;
        const int sa = s - 1, sb = s - SP, sc = s - SP * SP;  // upwind in a, b, c
        const double alpha = sw[u].x, beta = sw[u].y;
#pragma unroll
        for (int e = 0; e < 3; e++)
          sv[3 * s + e] = (alpha * sv[3 * sa + e] + beta * sv[3 * sb + e]) + (1 - alpha - beta) * sv[3 * sc + e];
      }
    }
    __syncthreads();
  }
  if (!in || keeps(threadIdx.x)) return;
  const int s = (ta + 1) + (tb + 1) * SP + (tc + 1) * SP * SP;
  const long long n = nidx(g, w.i0 + (a0 + ta) * w.di, w.j0 + (b0 + tb) * w.dj, w.k0 + (c0 + tc) * w.dk);
#pragma unroll
  for (int e = 0; e < 3; e++) f[3 * n + e] = sv[3 * s + e];
}

// ------------------------------------------------------------- the march
// A pass as a systolic march of warps. The pass's (b, c) columns (y and z in
// sweep order) are cut into patches of 8 x 4; one warp owns a patch and
// marches along a (x in sweep order), lane (b', c') at node a = q - b' - c' of
// its column in step q, so its three upwind values are its own last value and
// the last values of the lanes b' - 1 and c' - 1 (shuffles). The values that
// leave a patch at its downwind faces go through mailboxes in global memory
// which the host fills with SWEEP_EMPTY before the pass: a value is its own
// arrival flag, so neither side fences, and the reader loads a batch of
// MARCH_BATCH steps ahead and polls again only where it came too early. (A patch
// trails its neighbour by a batch and the value's way: batches of 4, 3, 2 and 1
// gave 5.1, 4.65, 4.35 and 4.0 ms a phase at 64^3, 7.6, 6.9, 6.4 and 5.9 at 128^3.)
// What bounds a pass is the chain of steps: a patch trails its b neighbour by
// 8 steps and its c neighbour by 4, plus the ~1 us a value takes through L2,
// and then has n of its own. The warps are spread over all SMs, one or a few
// each, so their FP64 instructions (63 cycles each a warp) do not queue. Warps
// claim patches from a ticket counter in an order in which each patch comes
// after those it reads from, so a pass makes progress with any number of
// warps resident and needs no cooperative launch. Waits are bounded
// (MARCH_WAIT_LIMIT polls): a warp that gives up sets *err and stops waiting,
// as does every warp that sees *err, so the launch ends; the host reports it.
// Measured (mesh, SDF and particle phase of a step, GB300): 11.3 ms with the
// wave and 6.5 with the march at 64^3, 16.1 and 9.5 at 128^3; 5.1 and 7.6 with
// comparisons on the numbers' bits and the root and the third of esf_root.cuh, 4.0
// and 5.9 in batches of one step. What is left is the chain of FP64 instructions,
// 2150 cycles a step where lanes update, and the mailboxes' way. A version with
// progress counters (release and acquire every batch of 4) took 8.3 ms at 64^3.
constexpr int MARCH_B = 8, MARCH_C = 4, MARCH_BATCH = 1;
constexpr int MARCH_SKEW = (MARCH_B - 1) + (MARCH_C - 1);
constexpr unsigned MARCH_WAIT_LIMIT = 1u << 22;
constexpr unsigned long long SWEEP_EMPTY = ~0ull;  // a NaN no arithmetic gives
inline int march_rows(int n, int tile) { return (n + tile - 1) / tile; }
inline int march_patches(const Sweep& w) { return march_rows(w.nj, MARCH_B) * march_rows(w.nk, MARCH_C); }
// values in a pass's mailboxes: the b faces of all patches, then their c faces
inline size_t march_mail(const Sweep& w) {
  return (size_t)w.ni * ((size_t)(march_rows(w.nj, MARCH_B) - 1) * w.nk + (size_t)(march_rows(w.nk, MARCH_C) - 1) * w.nj);
}

__device__ __forceinline__ double mail_load(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
// (the high word alone tells: a NaN that would look empty goes as another one)
__device__ __forceinline__ void mail_store(double* p, double v) {
  int hi = __double2hiint(v);
  hi = hi == -1 ? 0x7ff80000 : hi;
  v = __hiloint2double(hi, __double2loint(v));
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool mail_empty(double v) { return __double2hiint(v) == -1; }

// A pass's seeds: the nodes that would change with the field as it is before
// the pass. A node changes in a pass only if it is a seed or an upwind
// neighbour of it changed in the pass, so everything a pass changes lies
// downstream of its seeds on every axis: their least a, b and c (words 0-2 of
// `state`, preset to 0x7f7f7f7f) bound the box the pass has to march over, and
// a pass without seeds changes nothing. (The second eight passes of a step
// change values by rounding only, in about one octant: 32^3 of the 59^3 nodes
// around the 64^3 scene's ball.) Word 3
// of `state` is the march's ticket, which this kernel zeroes.
constexpr int PHI_PASS_WORDS = 32, PHI_NO_SEED = 0x7f7f7f7f;
__global__ void __launch_bounds__(KT) k_sweep_seeds(GridDev g, const double* __restrict__ ph,
                                                    const double* __restrict__ ms, Sweep w, int* state,
                                                    float skipBelow) {
  __shared__ int lo[3];
  if (threadIdx.x < 3) lo[threadIdx.x] = PHI_NO_SEED;
  __syncthreads();
  int m[3] = {PHI_NO_SEED, PHI_NO_SEED, PHI_NO_SEED};
  const long long nij = (long long)w.ni * w.nj, total = nij * w.nk;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(t % w.ni), b = (int)((t / w.ni) % w.nj), c = (int)(t / nij);
    const long long n = nidx(g, w.i0 + a * w.di, w.j0 + b * w.dj, w.k0 + c * w.dk);
    if (ms[n] != 0) continue;
    const double p = ph[n - w.di], q = ph[n - (long long)w.dj * g.X], r = ph[n - w.dk * g.slab];
    double v = ph[n];
    if (solve_distance_fast(p, q, r, v, near_float(p), near_float(q), near_float(r), near_float(v), skipBelow)) {
      m[0] = min(m[0], a);
      m[1] = min(m[1], b);
      m[2] = min(m[2], c);
    }
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    m[q] = __reduce_min_sync(0xffffffffu, m[q]);
    if ((threadIdx.x & 31) == 0 && m[q] != PHI_NO_SEED) atomicMin(&lo[q], m[q]);
  }
  __syncthreads();
  if (threadIdx.x < 3 && lo[threadIdx.x] != PHI_NO_SEED) atomicMin(&state[threadIdx.x], lo[threadIdx.x]);
  if (blockIdx.x == 0 && threadIdx.x == 0) state[3] = 0;
}

// The distance update of sweepPhi (DEFOR_SOLID_3D.cpp:397-455) on phi, at the
// nodes without solid mass.
// Lanes outside the pass (before its first node, after its last, beyond its
// last column) load from clamped places and only their effects are masked: a
// version that branched around each load ran four times the instructions.
// (Offsets fit 32 bits: a scene has fewer than 2^28 nodes.)
__global__ void __launch_bounds__(32) k_sweep_march(GridDev g, double* f, const double* __restrict__ ms, Sweep w,
                                                    int* state, double* mail, int* err, float skipBelow) {
  constexpr int D = MARCH_BATCH;
  // the box downstream of the seeds
  if (state[0] == PHI_NO_SEED) return;
  w.i0 += state[0] * w.di;
  w.j0 += state[1] * w.dj;
  w.k0 += state[2] * w.dk;
  w.ni -= state[0];
  w.nj -= state[1];
  w.nk -= state[2];
  const int lane = threadIdx.x, lb = lane & (MARCH_B - 1), lc = lane / MARCH_B, skew = lb + lc;
  const int nJ = (w.nj + MARCH_B - 1) / MARCH_B, nK = (w.nk + MARCH_C - 1) / MARCH_C;
  const int steps = w.ni + MARCH_SKEW, last = w.ni - 1;
  const int X = g.X, slab = (int)g.slab;
  double* const mailC = mail + (size_t)w.ni * (nJ - 1) * w.nk;
  bool dead = false;
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(state + 3, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= nJ * nK) return;
    const int J = t % nJ, K = t / nJ;
    const int b = min(J * MARCH_B + lb, w.nj - 1), c = min(K * MARCH_C + lc, w.nk - 1);
    const bool active = J * MARCH_B + lb < w.nj && K * MARCH_C + lc < w.nk;
    const int base = w.i0 + (w.j0 + b * w.dj) * X + (w.k0 + c * w.dk) * slab;  // node a = 0 of the column
    // the upwind values from outside the patch: a mailbox, or the field itself
    // upwind of the pass's first row (constant); other lanes load their own
    // first node's and ignore it
    const bool needB = lb == 0, needC = lc == 0;
    const bool waitB = active && needB && J > 0, waitC = active && needC && K > 0;
    const double* const srcB = waitB ? mail + ((J - 1) * w.nk + c) * w.ni : f + (needB ? base - w.dj * X : base);
    const double* const srcC = waitC ? mailC + ((K - 1) * w.nj + b) * w.ni : f + (needC ? base - w.dk * slab : base);
    const int incB = needB ? (waitB ? 1 : w.di) : 0, incC = needC ? (waitC ? 1 : w.di) : 0;
    const bool sendB = active && lb == MARCH_B - 1 && J < nJ - 1, sendC = active && lc == MARCH_C - 1 && K < nK - 1;
    double* const outB = sendB ? mail + (J * w.nk + c) * w.ni : mail;
    double* const outC = sendC ? mailC + (K * w.nj + b) * w.ni : mail;
    double val = f[base - w.di];
    float fval = near_float(val);
    // the own values, mass and upwind values from outside of D steps, loaded
    // one batch ahead
    double nov[D], nms[D], nub[D], nuc[D];
    auto fetch = [&](int q0) {
#pragma unroll
      for (int s = 0; s < D; s++) {
        const int a = min(max(q0 + s - skew, 0), last);
        const int n = base + a * w.di;
        nub[s] = mail_load(srcB + a * incB);
        nuc[s] = mail_load(srcC + a * incC);
        nov[s] = f[n];
        nms[s] = ms[n];
      }
    };
    fetch(0);
    for (int q0 = 0; q0 < steps; q0 += D) {
      double ov[D], ub[D], uc[D];
      float fo[D];
      bool om[D];
#pragma unroll
      for (int s = 0; s < D; s++) {
        ov[s] = nov[s];
        fo[s] = near_float(nov[s]);
        om[s] = (__double2hiint(nms[s]) & 0x7fffffff) | __double2loint(nms[s]);
        ub[s] = nub[s];
        uc[s] = nuc[s];
      }
      auto missing = [&] {
        bool m = false;
#pragma unroll
        for (int s = 0; s < D; s++) {
          const int a = q0 + s - skew;
          m = m || (((waitB && mail_empty(ub[s])) || (waitC && mail_empty(uc[s]))) && a >= 0 && a <= last);
        }
        return m;
      };
      // values that had not arrived when they were loaded: poll
      unsigned it = 0;
      while (__any_sync(0xffffffffu, missing()) && !dead) {
#pragma unroll
        for (int s = 0; s < D; s++) {
          const int a = min(max(q0 + s - skew, 0), last);
          ub[s] = mail_load(srcB + a * incB);
          uc[s] = mail_load(srcC + a * incC);
        }
        if ((++it & 1023u) == 0 && (it >= MARCH_WAIT_LIMIT || __any_sync(0xffffffffu, *(volatile int*)err))) {
          dead = true;
          if (lane == 0) *(volatile int*)err = 1;
        }
      }
      if (q0 + D < steps) fetch(q0 + D);
#pragma unroll
      for (int s = 0; s < D; s++) {
        const int a = q0 + s - skew;
        const bool in = active && a >= 0 && a <= last;
        const int ac = min(max(a, 0), last);
        double vb = __shfl_up_sync(0xffffffffu, val, 1), vc = __shfl_up_sync(0xffffffffu, val, MARCH_B);
        float fb = __shfl_up_sync(0xffffffffu, fval, 1), fc = __shfl_up_sync(0xffffffffu, fval, MARCH_B);
        vb = needB ? ub[s] : vb;
        vc = needC ? uc[s] : vc;
        fb = needB ? near_float(vb) : fb;
        fc = needC ? near_float(vc) : fc;
        double v = ov[s];
        if (in && !om[s] && solve_distance_fast(val, vb, vc, v, fval, fb, fc, fo[s], skipBelow))
          f[base + ac * w.di] = v;
        val = in ? v : val;
        fval = near_float(val);
        if (sendB && in) mail_store(outB + ac, val);
        if (sendC && in) mail_store(outC + ac, val);
      }
    }
  }
}

constexpr int SWEEP_THREADS = 128;  // blocks of the wave kernel
// A whole sweep pass in one cooperative launch: the blocks walk the pass's
// hyperplanes a + b + c = p in order, each plane split over all threads, with
// a grid-wide barrier between planes. Values written in this pass by other
// blocks are read through L2 (ld.cg); the barrier is one growing counter in
// global memory, its wait bounded (a block that gives up sets *err and
// carries on, so the launch always ends; the host reports it).
// Same per-node operations as k_sweep_march, each node after its three
// upwind neighbours, so the same bits. Only ESF_SWEEP=wave runs it, as the
// independent schedule the march is compared against: a plane costs it 3.6 to
// 4.3 us (barrier, L2 round trips, the square-root chain), and a pass has 3n.
constexpr unsigned WAVE_WAIT_LIMIT = 1u << 22;
// Arrival p of every block: a release add on a counter that only grows (the
// host zeroes it before the launch), then acquire loads until it reaches
// (p + 1) x blocks.
__device__ __forceinline__ void wave_barrier(unsigned* count, unsigned target, int* err) {
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned cur;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(cur) : "l"(count) : "memory");
    cur += 1;
    unsigned it = 0;
    while (cur < target && ++it < WAVE_WAIT_LIMIT)
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(count) : "memory");
    if (cur < target) *err = 1;
  }
  __syncthreads();
}
template <bool VEC>
__global__ void __launch_bounds__(SWEEP_THREADS) k_sweep_wave(GridDev g, double* f, double* ph,
                                                              const double* ms, Sweep w,
                                                              const unsigned long long* ranks,
                                                              unsigned* bar, int* err) {
  const long long nij = (long long)w.ni * w.nj;
  const int planes = w.ni + w.nj + w.nk - 2;
  unsigned long long rx = 0, ry = 0, rz = 0;
  if (VEC) {
    rx = ranks[0];
    ry = ranks[1];
    rz = ranks[2];
  }
  for (int p = 0; p < planes; p++) {
    for (long long t = blockIdx.x * (long long)SWEEP_THREADS + threadIdx.x; t < nij;
         t += (long long)gridDim.x * SWEEP_THREADS) {
      const int a = (int)(t % w.ni), b = (int)(t / w.ni);
      const int c = p - a - b;
      if (c < 0 || c >= w.nk) continue;
      const int i = w.i0 + a * w.di, j = w.j0 + b * w.dj, k = w.k0 + c * w.dk;
      const long long n = nidx(g, i, j, k);
      if (ms[n] != 0) continue;
      const long long ea = nidx(g, i - w.di, j, k), eb = nidx(g, i, j - w.dj, k), ec = nidx(g, i, j, k - w.dk);
      if (!VEC) {
        double v = __ldcg(ph + n);
        solve_distance(__ldcg(ph + ea), __ldcg(ph + eb), __ldcg(ph + ec), &v);
        ph[n] = v;
        continue;
      }
      const unsigned long long rank = (unsigned long long)(a + (long long)b * w.ni + (long long)c * nij);
      const double pn = ph[n];
      double dp = pn - ph[ea], dpn = pn - ph[nidx(g, i + w.di, j, k)];
      if (dp < 0 && dpn >= 0) continue;
      double dq = pn - ph[eb], dqn = pn - ph[nidx(g, i, j + w.dj, k)];
      if (dq < 0 && dqn >= 0) continue;
      double dr = pn - ph[ec], drn = pn - ph[nidx(g, i, j, k + w.dk)];
      if (dr < 0 && drn >= 0) continue;
      if (rank >= rx) dp = 0;
      if (rank >= ry) dq = 0;
      if (rank >= rz) dr = 0;
      double alpha, beta;
      if (dp + dq + dr < 1e-3) {
        alpha = 0.333;
        beta = 0.333;
      } else {
        alpha = dp / (dp + dq + dr);
        beta = dq / (dp + dq + dr);
      }
#pragma unroll
      for (int e = 0; e < 3; e++)
        f[3 * n + e] = (alpha * __ldcg(f + 3 * ea + e) + beta * __ldcg(f + 3 * eb + e)) +
                       (1 - alpha - beta) * __ldcg(f + 3 * ec + e);
    }
    wave_barrier(bar, (unsigned)(p + 1) * gridDim.x, err);
  }
}
