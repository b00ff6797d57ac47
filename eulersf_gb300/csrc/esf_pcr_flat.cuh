// Loops of the one-pass FP32 iteration (esf_pcr_fused.cuh) for grids whose chunks
// are at most FL_L layers deep and whose blocks can all be resident at once: up
// to FL_CHUNK iterations in one cooperative launch of the same blocks, with the
// same sums and bits. Included by esf_solver.cu inside namespace esf after
// esf_pcr_fused.cuh.
//
// On such a grid a pass is a chain of latencies, so the loop shortens the chain:
//  * all layers of a block are in shared memory at once, and FL_G groups of 256
//    threads work on them side by side, where fused_pass marches layer by layer;
//  * x, d and 1/diag stay in registers and m^-1 in shared memory from one pass
//    to the next; r, t and q go through memory, because the neighbours read them,
//    and come back in three copies (one box a vector), which are on their way
//    while the sums are folded: they need no scalar of the new pass;
//  * a grid barrier, after which every block folds the sums for itself, a warp a
//    sum.
//
//   (a) group by layer: r' at tile and halo into V; own layers: x, d, q, r
//   (b) group by own layer: the two node layers around it, their sums A, B, C
//   (c) s', t' of the own layer, and what the sums are formed from
//   (d) group by sum: over the layers in fused_pass's order
// Bound: latencies (128 blocks at 64^3, one an SM; its 12 words a row are 2 us of
// L2). An iteration against a launch of fused_pass each: 12.4 -> 7.1 us at 32^3,
// 12.4 -> 7.7 at 64^3, in double-float 14.3 -> 8.4 and 15.1 -> 9.4 (8.2 at 64^3
// with the sums by eight warps in turn; 8.1 with one thread for barrier and
// copies). At 64^3 it is some 16000 cycles: (a) to (d) a third, block sums, folds
// and scalars, whose FP64 instructions take 63 cycles each, two fifths, the
// barrier a fifth. fused_pass itself in a loop gave 12.0 at 64^3, 21.2 for 19.0 at 96^3, 26.7 for 24.7 at
// 128^3: the launches in a graph cost a microsecond, the barrier as much.
#pragma once

constexpr int FL_L = 4, FL_G = 4;        // own layers of a block at most, groups
constexpr int FL_H = FL_L + 2;           // layers with the halo
constexpr int FL_CHUNK = 32;
// r, t, q: boxes 72 x 10 x 6 at (x0 - 4, y0 - 1, z0 - 1); m^-1: 68 x 9 x 5 at
// (x0, y0, z0); zeros outside the grid. (A thread issues a copy in some 150
// cycles: boxes of one layer took 5300 a pass.)
struct FlatMaps {
  CUtensorMap r[2], t[2], q[2], m;
};
constexpr int FL_RB = FL_H * TMA_HALO_BYTES, FL_MB = (FL_L + 1) * TMA_NODE_BYTES;
constexpr int FL_VP = TW_PP * HY;        // V of a layer, laid out as sP
constexpr int FL_NP = TW_NP * NYN;
constexpr int FL_SP = 8 * 33 + 4;        // a sum's values, warp w's at 33 w
constexpr int FL_OFF_R = 0, FL_OFF_M = 3 * FL_RB, FL_OFF_V = FL_OFF_M + (FL_MB + 127) / 128 * 128,
              FL_OFF_K = FL_OFF_V + FL_H * FL_VP * 4, FL_OFF_S = FL_OFF_K + 10 * NT * FL_L * 4,
              FL_OFF_T = FL_OFF_S + FU_SUMS * FL_SP * 4, FL_OFF_BAR = FL_OFF_T + FU_SUMS * 8, FL_SMEM = FL_OFF_BAR + 16;
static_assert(FL_RB % 128 == 0 && FL_OFF_M % 128 == 0 && FL_OFF_V % 16 == 0 && FL_OFF_K % 16 == 0 &&
                  FL_OFF_T % 16 == 0, "layout");
// (b) writes A, B, C over r, t and q, which (a) is done with
static_assert(FL_L * 3 * FL_NP * 4 <= FL_OFF_M, "overlay");

// Arrival of all blocks at the next pass: polls of the counter they add to, bounded.
__device__ __forceinline__ bool flat_wait(PcrState* st, unsigned target) {
  unsigned cur, it = 0, bad = 0;
  do {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(&st->ticket[2]) : "memory");
    if ((++it & 1023u) == 0) {
      bad = *(volatile unsigned*)&st->failed;
      if (it >= FU_LOOP_WAIT) bad = *(volatile unsigned*)&st->failed = 1;
    }
  } while ((int)(cur - target) < 0 && !bad);
  return !bad;
}
// block_sum's tree over 256 values by one warp: value(w, i) is lane i's of warp w.
template <typename F>
__device__ __forceinline__ double flat_tree(F value) {
  const int lane = threadIdx.x & 31, w = lane & 7, i = lane >> 3;
  double t[8];
#pragma unroll
  for (int k = 0; k < 8; k++) t[k] = value(w, i + 4 * k);
#pragma unroll
  for (int h = 4; h > 0; h /= 2)
#pragma unroll
    for (int k = 0; k < h; k++) t[k] += t[k + h];
  double r = t[0];
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}
// the first four warps, one on each of the SM's schedulers
__device__ __forceinline__ void flat_sync4() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <bool X64>
__global__ void __launch_bounds__(FL_G* NT, 1)
    pcr_loop_flat(GridDev g, const __grid_constant__ FlatMaps tm, FusedPtrs p, const float* invd, float* edf,
                  float* ddf, double* partial, PcrState* st, int cz, int budget) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ PcrState L;
  __shared__ int go, arrived;
  static_assert(FL_G == FL_L && FL_G == FU_SUMS, "a group for each own layer and each sum");
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem + FL_OFF_BAR);
  float* sV = reinterpret_cast<float*>(smem + FL_OFF_V);
  float* sK = reinterpret_cast<float*>(smem + FL_OFF_K);  // [layer][10][NT]
  float* sS = reinterpret_cast<float*>(smem + FL_OFF_S);  // [sum][FL_SP]
  double* sT = reinterpret_cast<double*>(smem + FL_OFF_T);  // [sum]
  float* sN = reinterpret_cast<float*>(smem + FL_OFF_R);  // [layer][A, B, C]
  const int nb = gridDim.x * gridDim.y * gridDim.z;
  const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const int x0 = blockIdx.x * TXW, y0 = blockIdx.y * TY, z0 = blockIdx.z * cz;
  const int layers = min(cz, g.cZ - z0);  // 1 .. FL_L

  const int grp = threadIdx.x / NT, tid = threadIdx.x % NT;
  const int lane = tid & 31, w = tid >> 5;
  const int cx = 2 * lane;
  const int cgx = x0 + cx, cgy = y0 + w;
  const bool cin = cgx < g.cX && cgy < g.cY;  // cX is a multiple of 4
  const bool own = cin && grp < layers;
  const long long oc = cgx + (long long)cgy * g.cX + (long long)(z0 + grp) * g.cslab;

  if (threadIdx.x == 0) L = *st;
  __syncthreads();
  if (L.done || L.failed) return;
  const unsigned base = L.ticket[0];
  auto fetch = [&](int set) {  // by one thread
    asm volatile("fence.proxy.async;" ::: "memory");  // (what the blocks wrote before the barrier)
    mbar_expect_tx(&bar[0], 3 * FL_RB);
    tma_load_3d(smem + FL_OFF_R, set ? &tm.r[1] : &tm.r[0], x0 - 4, y0 - 1, z0 - 1, &bar[0]);
    tma_load_3d(smem + FL_OFF_R + FL_RB, set ? &tm.t[1] : &tm.t[0], x0 - 4, y0 - 1, z0 - 1, &bar[0]);
    tma_load_3d(smem + FL_OFF_R + 2 * FL_RB, set ? &tm.q[1] : &tm.q[0], x0 - 4, y0 - 1, z0 - 1, &bar[0]);
  };
  if (threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fetch(L.pp & 1);
    mbar_expect_tx(&bar[1], FL_MB);
    tma_load_3d(smem + FL_OFF_M, &tm.m, x0, y0, z0, &bar[1]);
  }
  // x and d of the own pair (X64: e and d in double-float)
  float4 xs = make_float4(0.f, 0.f, 0.f, 0.f), ds = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 iv = make_float2(0.f, 0.f);
  if (own) {
    iv = *reinterpret_cast<const float2*>(invd + oc);
    if constexpr (X64) {
      xs = *reinterpret_cast<const float4*>(edf + 2 * oc);
      ds = *reinterpret_cast<const float4*>(ddf + 2 * oc);
    } else {
      const float2 a = *reinterpret_cast<const float2*>(p.x + oc), b = *reinterpret_cast<const float2*>(p.d + oc);
      xs.x = a.x;
      xs.y = a.y;
      ds.x = b.x;
      ds.y = b.y;
    }
  }
  __syncthreads();
  bool ok = mbar_wait(&bar[1], 0);

  const bool hasE = tid < TW_RING, hasN = tid < TW_NODE_EXTRA;
  int eh = 0, ey = 0;
  if (tid < TW_HX) {
    eh = tid;
  } else if (tid < 2 * TW_HX) {
    eh = tid - TW_HX;
    ey = HY - 1;
  } else {
    const int e = tid - 2 * TW_HX;
    ey = 1 + (e >> 1);
    eh = (e & 1) ? TW_HX - 1 : 0;
  }
  const int bM = (cx + 4) + (w + 1) * TMA_HW, pM = (cx + 2) + (w + 1) * TW_PP;
  const int bE = (eh + 3) + ey * TMA_HW, pE = (eh + 1) + ey * TW_PP;
  const int enx = tid < TY ? TW_NX - 1 : tid - TY, eny = tid < TY ? tid : NYN - 1;
  const int aN = cx + w * TW_NP;

  int pass = 0;
  bool failed = false;  // (the same in all threads)
  for (;; pass++) {
    const bool stop = pass == budget || L.done || L.iter >= L.maxIt;  // the same in every block
    ok = mbar_wait(&bar[0], pass & 1) && ok;
    if (stop) break;
    const int pout = (L.pp & 1) ^ 1;
    const bool rb = X64 && L.rebase;
    const float alpha = rb ? 0.0f : (float)L.alpha, beta = (float)L.beta;
    float* rOut = pout ? p.r[1] : p.r[0];
    float* qOut = pout ? p.q[1] : p.q[0];
    float* tOut = pout ? p.t[1] : p.t[0];
    // (a) r' = r - alpha (t + beta q)
    float2 vo = make_float2(0.f, 0.f), qo = vo;
    auto layer_in = [&](int h, bool mine, bool tile, bool ring) {
      const float* R = reinterpret_cast<const float*>(smem + FL_OFF_R + h * TMA_HALO_BYTES);
      const float *Tt = R + FL_RB / 4, *Qq = R + 2 * (FL_RB / 4);
      if (ring && hasE) sV[h * FL_VP + pE] = __fmaf_rn(-alpha, __fmaf_rn(beta, Qq[bE], Tt[bE]), R[bE]);
      if (!tile) return;
      const float2 r2 = *reinterpret_cast<const float2*>(R + bM);
      const float2 t2 = *reinterpret_cast<const float2*>(Tt + bM);
      const float2 q2 = *reinterpret_cast<const float2*>(Qq + bM);
      const float qn0 = rb ? q2.x : __fmaf_rn(beta, q2.x, t2.x), qn1 = rb ? q2.y : __fmaf_rn(beta, q2.y, t2.y);
      const float v0 = __fmaf_rn(-alpha, qn0, r2.x), v1 = __fmaf_rn(-alpha, qn1, r2.y);
      *reinterpret_cast<float2*>(sV + h * FL_VP + pM) = make_float2(v0, v1);
      if (!mine) return;
      if constexpr (X64) {
        const float2 dn0 = rb ? make_float2(ds.x, ds.y) : df_axpy(beta, make_float2(ds.x, ds.y), r2.x);
        const float2 dn1 = rb ? make_float2(ds.z, ds.w) : df_axpy(beta, make_float2(ds.z, ds.w), r2.y);
        const float2 en0 = df_add_scaled(make_float2(xs.x, xs.y), alpha, dn0);
        const float2 en1 = df_add_scaled(make_float2(xs.z, xs.w), alpha, dn1);
        ds = make_float4(dn0.x, dn0.y, dn1.x, dn1.y);
        xs = make_float4(en0.x, en0.y, en1.x, en1.y);
      } else {
        ds.x = __fmaf_rn(beta, ds.x, r2.x);
        ds.y = __fmaf_rn(beta, ds.y, r2.y);
        xs.x = __fmaf_rn(alpha, ds.x, xs.x);
        xs.y = __fmaf_rn(alpha, ds.y, xs.y);
      }
      *reinterpret_cast<float2*>(rOut + oc) = make_float2(v0, v1);
      *reinterpret_cast<float2*>(qOut + oc) = make_float2(qn0, qn1);
      vo = make_float2(v0, v1);
      qo = make_float2(qn0, qn1);
    };
    if (grp < layers) layer_in(grp + 1, own, true, true);
    // the layers around: tile and ring to a group each
    layer_in(grp < 2 ? 0 : layers + 1, false, grp & 1, !(grp & 1));
    failed = __syncthreads_or(!ok);
    if (failed) break;

    // (b) J^T r' scaled by m^-1 on the node layers below and above the own layer
    if (grp < layers) {
      float* sA = sN + grp * 3 * FL_NP;
      float *sB = sA + FL_NP, *sC = sB + FL_NP;
      {
        const float* V = sV + grp * FL_VP + (cx + 1) + w * TW_PP;
        float v[3][6];
#pragma unroll
        for (int k = 0; k < 3; k++) {
          const float* q = V + k * FL_VP;
          const float2 a = *reinterpret_cast<const float2*>(q + 1), b = *reinterpret_cast<const float2*>(q + 1 + TW_PP);
          v[k][0] = q[0];
          v[k][1] = a.x;
          v[k][2] = a.y;
          v[k][3] = q[TW_PP];
          v[k][4] = b.x;
          v[k][5] = b.y;
        }
        float mp[6];
#pragma unroll
        for (int n = 0; n < 2; n++) {
          const float* M = reinterpret_cast<const float*>(smem + FL_OFF_M + (grp + n) * TMA_NODE_BYTES);
          const float2 mi = *reinterpret_cast<const float2*>(M + cx + w * TMA_NW);
          float P[6], Q[6];
#pragma unroll
          for (int k = 0; k < 6; k++) {
            P[k] = v[n][k] + v[n + 1][k];
            Q[k] = v[n][k] - v[n + 1][k];
          }
          const float ab1 = P[1] + P[4];
          // (products rounded before they are added, as fused_pass has them)
          const float mx0 = __fmul_rn((P[0] + P[3]) - ab1, mi.x);
          const float my0 = __fmul_rn((P[0] + P[1]) - (P[3] + P[4]), mi.x);
          const float mz0 = __fmul_rn((Q[0] + Q[1]) + (Q[3] + Q[4]), mi.x);
          const float mx1 = __fmul_rn(ab1 - (P[2] + P[5]), mi.y);
          const float my1 = __fmul_rn((P[1] + P[2]) - (P[4] + P[5]), mi.y);
          const float mz1 = __fmul_rn((Q[1] + Q[2]) + (Q[4] + Q[5]), mi.y);
          if (n == 1) {
            *reinterpret_cast<float2*>(sA + aN) = make_float2(mp[0] + mx0, mp[1] + mx1);
            *reinterpret_cast<float2*>(sB + aN) = make_float2(mp[2] + my0, mp[3] + my1);
            *reinterpret_cast<float2*>(sC + aN) = make_float2(mz0 - mp[4], mz1 - mp[5]);
          }
          mp[0] = mx0; mp[1] = mx1; mp[2] = my0;
          mp[3] = my1; mp[4] = mz0; mp[5] = mz1;
        }
      }
      if (hasN) {
        const float* V = sV + grp * FL_VP + (enx + 1) + eny * TW_PP;
        const int aNE = enx + eny * TW_NP;
        float mpx = 0, mpy = 0, mpz = 0;
#pragma unroll
        for (int n = 0; n < 2; n++) {
          const float *lo = V + n * FL_VP, *hi = lo + FL_VP;
          const float mi =
              reinterpret_cast<const float*>(smem + FL_OFF_M + (grp + n) * TMA_NODE_BYTES)[enx + eny * TMA_NW];
          const float P00 = lo[0] + hi[0], P10 = lo[1] + hi[1], P01 = lo[TW_PP] + hi[TW_PP],
                      P11 = lo[TW_PP + 1] + hi[TW_PP + 1];
          const float Q00 = lo[0] - hi[0], Q10 = lo[1] - hi[1], Q01 = lo[TW_PP] - hi[TW_PP],
                      Q11 = lo[TW_PP + 1] - hi[TW_PP + 1];
          const float mx = __fmul_rn((P00 + P01) - (P10 + P11), mi);
          const float my = __fmul_rn((P00 + P10) - (P01 + P11), mi);
          const float mz = __fmul_rn((Q00 + Q10) + (Q01 + Q11), mi);
          if (n == 1) {
            sA[aNE] = mpx + mx;
            sB[aNE] = mpy + my;
            sC[aNE] = mz - mpz;
          }
          mpx = mx; mpy = my; mpz = mz;
        }
      }
    }
    __syncthreads();

    // (c) s' and t' = s'/diag
    if (own) {
      const float* sA = sN + grp * 3 * FL_NP;
      const float *sB = sA + FL_NP, *sC = sB + FL_NP;
      const float2 A01 = *reinterpret_cast<const float2*>(sA + aN);
      const float A2 = sA[aN + 2];
      const float2 B01 = *reinterpret_cast<const float2*>(sA + aN + TW_NP);
      const float B2 = sA[aN + 2 + TW_NP];
      const float2 c01 = *reinterpret_cast<const float2*>(sB + aN);
      const float c2 = sB[aN + 2];
      const float2 e01 = *reinterpret_cast<const float2*>(sB + aN + TW_NP);
      const float e2 = sB[aN + 2 + TW_NP];
      const float2 f01 = *reinterpret_cast<const float2*>(sC + aN);
      const float f2 = sC[aN + 2];
      const float2 g01 = *reinterpret_cast<const float2*>(sC + aN + TW_NP);
      const float g2 = sC[aN + 2 + TW_NP];
      const float mid = A01.y + B01.y;
      const float xp0 = mid - (A01.x + B01.x);
      const float yp0 = (e01.x + e01.y) - (c01.x + c01.y);
      const float zp0 = (f01.x + f01.y) + (g01.x + g01.y);
      const float xp1 = (A2 + B2) - mid;
      const float yp1 = (e01.y + e2) - (c01.y + c2);
      const float zp1 = (f01.y + f2) + (g01.y + g2);
      const float o0 = xp0 + yp0 + zp0, o1 = xp1 + yp1 + zp1;
      const float t0 = __fmul_rn(iv.x, o0), t1 = __fmul_rn(iv.y, o1);
      *reinterpret_cast<float2*>(tOut + oc) = make_float2(t0, t1);
      float* q = sK + grp * 10 * NT + tid;
      q[0] = vo.x;
      q[NT] = vo.y;
      q[2 * NT] = t0;
      q[3 * NT] = t1;
      q[4 * NT] = qo.x;
      q[5 * NT] = qo.y;
      q[6 * NT] = iv.x;
      q[7 * NT] = iv.y;
      q[8 * NT] = o0;
      q[9 * NT] = o1;
    }
    __syncthreads();

    // (d) (r', s'), (s', t'), (s', q), (Ap, q)
    float sum = 0;
    if (cin) {
      const float* q = sK + 2 * grp * NT + tid;
      for (int l = 0; l < layers; l++, q += 10 * NT) {
        const float a0 = q[0], a1 = q[NT];
        if (grp == 3) {
          // (quotients in the expressions that fused_pass has: formed earlier they
          // round differently)
          const float q0 = q[-2 * NT], q1 = q[-NT];
          if (a0 > 0.0f) sum += __fdividef(q0 * q0, a0);
          if (a1 > 0.0f) sum += __fdividef(q1 * q1, a1);
        } else {
          const float* o = sK + (10 * l + 8) * NT + tid;
          sum += a0 * o[0] + a1 * o[NT];
        }
      }
    }
    sS[grp * FL_SP + w * 33 + lane] = sum;
    __syncthreads();
    // a warp a sum, on schedulers of their own; a fifth fetches
    const unsigned target = base + (unsigned)(pass + 1) * nb;
    if (threadIdx.x < 128) {
      const int h = threadIdx.x >> 5;
      // (a block can be a pass ahead of another's fold)
      double* part = partial + ((pass & 1) * FU_SUMS + h) * nb;
      const float* mine = sS + h * FL_SP;
      const double ps = flat_tree([&](int a, int i) { return widen(mine[a * 33 + i]); });
      if (lane == 0) __stcg(part + bid, ps);
      flat_sync4();
      bool here = false;  // thread 0's: all sums are there
      if (threadIdx.x == 0) {
        asm volatile("red.add.release.gpu.global.u32 [%0], 1;" ::"l"(&st->ticket[2]) : "memory");
        here = flat_wait(st, target);  // (one poller: four in each block were slower)
        go = here;
      }
      flat_sync4();
      const double total =
          flat_tree([&](int a, int i) { return a * 32 + i < nb ? __ldcg(part + a * 32 + i) : 0.0; });
      if (lane == 0) sT[h] = total;
      flat_sync4();
      if (threadIdx.x == 0 && here) finish_fused(&L, sT[0], sT[1], sT[2], sT[3]);  // (not of sums that may be missing)
    } else if (threadIdx.x == 128) {
      arrived = flat_wait(st, target);
      if (arrived) fetch(pout);
    }
    __syncthreads();
    if (!go || !arrived) {
      if (arrived) mbar_wait(&bar[0], (pass + 1) & 1);
      failed = true;
      break;
    }
  }
  // a block that gave up on a copy or on the others has no x and d to store: the
  // solve has failed, whatever the others' sums say, and they give up too
  if (__syncthreads_or(failed || !ok)) {
    if (threadIdx.x == 0) *(volatile unsigned*)&st->failed = 1;
    return;
  }
  if (own) {
    if constexpr (X64) {
      *reinterpret_cast<float4*>(edf + 2 * oc) = xs;
      *reinterpret_cast<float4*>(ddf + 2 * oc) = ds;
    } else {
      *reinterpret_cast<float2*>(p.x + oc) = make_float2(xs.x, xs.y);
      *reinterpret_cast<float2*>(p.d + oc) = make_float2(ds.x, ds.y);
    }
  }
  if (bid == 0 && threadIdx.x == 0) {
    if (L.iter >= L.maxIt) L.done = 1;
    L.ticket[0] = L.ticket[2] = base + (unsigned)pass * nb;
    for (unsigned k = 0; k < sizeof(PcrState) / 4; k++)
      if (k != offsetof(PcrState, failed) / 4)
        reinterpret_cast<unsigned*>(st)[k] = reinterpret_cast<const unsigned*>(&L)[k];
  }
}
