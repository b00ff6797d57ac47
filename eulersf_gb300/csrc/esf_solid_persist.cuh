// The solid system's PCR solve as one persistent kernel: all iterations of
// solid_pcr_graph's loop (the reference's assembled solvePCR,
// CONJUGATE_RESIDUAL.inl:194-276, or an FP32 inner solve of a refinement) in
// one cooperative launch, with a grid barrier where the graph has a kernel
// boundary. Included by esf_solver.cu inside namespace esf.
//
// A solid of a few thousand nodes has 1-3 us of work an iteration; as three or
// four kernels it took 48 us (FP64, 64^3 scene: the block rows of 4.5 thousand
// nodes on 18 SMs) and 26 us (FP32 matrix-free, 128^3 scene), nearly all of it
// launches, last-block folds and the serial chain of one thread a row. Here an
// iteration is three barriers (~1.3 us each): d and Ap with Ap.Ap/diag; x and
// r with the operator; the operator's sums with r.s. The FP32 matrix-free
// operator forms the new r where it reads it (the same FMA chain as at its
// owner, so the same bits) and needs no pass of its own for it.
// Measured an iteration: FP64 48 -> 18 us (64^3 scene), 50 -> 39 (128^3);
// FP32 matrix-free 26 -> 15 (64^3), 26 -> 17 (128^3). What is left: the
// barriers, two folds at 2 to 2.5 us (FP64 additions, 63 cycles each, and a
// division, 640), and in FP64 the block rows' 324 FP64 instructions a warp.
//
// Both paths give the same bits: the sums keep the graph kernels' virtual
// blocks of VT threads, their order within a thread and a block, and the fold
// in block order. A row pass (one row a thread) deals its warps of 32 rows out
// over all blocks and leaves one sum a warp, from which every block forms the
// virtual blocks' sums and folds them.
#pragma once

template <typename T>
struct SolidPersist {
  long long S;
  const T *blocks, *invd, *b;
  const int* nbr;
  T *x, *r, *d, *Ap, *s;
  double* partial;
  PcrState* st;
  unsigned* bar;  // [0] arrivals (zeroed before the launch), [1] a barrier gave up
  int vb;         // virtual blocks of the vector passes
  SolidMF mf;
  float* share;
  const float* damped;
};
// partial sums of a pass: one region each
constexpr int PERSIST_FOLD = 2048;
constexpr long long PERSIST_MAX_ROWS = 65536;
static_assert(4 * PERSIST_FOLD <= ESF_MAX_PARTIALS, "regions of the partial sums");
static_assert(PERSIST_FOLD >= 152 * 8 && PERSIST_MAX_ROWS <= 32 * PERSIST_FOLD &&
                  PERSIST_MAX_ROWS <= 152 * 8 * VT,
              "vec_blocks' virtual blocks and the rows' warps fit a region, and a row pass has one row a thread");
constexpr unsigned PERSIST_WAIT_LIMIT = 1u << 22;

// Arrival of every block at the next barrier: a release add on a counter that
// only grows, then acquire loads. False in every block once one gave up.
__device__ __forceinline__ bool persist_sync(unsigned* bar, unsigned& target) {
  __shared__ int ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned cur, it = 0, bad = 0;
    asm volatile("red.add.release.gpu.global.u32 [%0], 1;" ::"l"(bar) : "memory");
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(bar) : "memory");
      if ((++it & 1023u) == 0) {
        bad = *(volatile unsigned*)(bar + 1);
        if (it >= PERSIST_WAIT_LIMIT) bad = *(volatile unsigned*)(bar + 1) = 1;
      }
    } while (cur < target && !bad);
    ok = !bad;
  }
  __syncthreads();
  return ok;
}
// The sum of a row pass in every block, in fold_partials' order (thread 0's
// value): n warp sums, eight to a virtual block, added up as
// block_sum's second stage adds them.
__device__ __forceinline__ double persist_fold_rows(const double* sums, int n) {
  double acc = 0;
  for (int v = threadIdx.x; 8 * v < n; v += VT) {
    double w[8];
#pragma unroll
    for (int k = 0; k < 8; k++) w[k] = 8 * v + k < n ? __ldcg(sums + 8 * v + k) : 0.0;
    acc += ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
  }
  return block_sum<VT>(acc);
}
// a warp's sum in block_sum's first stage (lane 0's value)
__device__ __forceinline__ double warp_tree(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Component c of block row a times `in`, summed in the assembled order over
// the neighbours that exist. All loads of nine blocks are issued before the
// first is used (an absent neighbour's from place 0, its term dropped by a
// select): with a branch around each block a row was a chain of 27 x 2 L2
// round trips, 27 us.
template <typename T>
__device__ __forceinline__ T spmv_component(const T* __restrict__ blocks, const int* __restrict__ nbr, const T* in,
                                            long long a, int c) {
  const int* nb = nbr + nbr_at(a, 0);
  const T* B0 = blocks + blk_at(a, 0) + 96 * c;
  int m[27];
#pragma unroll
  for (int j = 0; j < 27; j++) m[j] = __ldg(nb + 32 * j);
  T y = 0;
#pragma unroll
  for (int j0 = 0; j0 < 27; j0 += 9) {
    T v[9][3], B[9][3];
#pragma unroll
    for (int j = 0; j < 9; j++) {
      const T* x = in + 3 * (long long)max(m[j0 + j], 0);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        v[j][k] = x[k];
        B[j][k] = __ldg(B0 + 32 * (9 * (j0 + j) + k));
      }
    }
#pragma unroll
    for (int j = 0; j < 9; j++) {
      T t = y;
      t += B[j][0] * v[j][0] + B[j][1] * v[j][1] + B[j][2] * v[j][2];
      y = m[j0 + j] >= 0 ? t : y;
    }
  }
  return y;
}

// (FP32 solves, which a server runs for many scenes at once, leave half of an
// SM's registers to other streams' kernels)
template <typename T, bool MATRIX_FREE>
__global__ void __launch_bounds__(VT, std::is_same<T, float>::value ? 2 : 1) solid_pcr_persistent(SolidPersist<T> a, int budget) {
  __shared__ T sy[2][3][32];
  __shared__ PcrState L;  // every block's copy of the state; block 0's goes back
  const int tid = threadIdx.x, G = gridDim.x;
  const long long n = 3 * a.S;
  const int slices = (int)((a.S + 31) / 32);
  double *pv = a.partial, *ps = pv + PERSIST_FOLD, *pc = ps + PERSIST_FOLD, *pz = pc + PERSIST_FOLD;
  unsigned target = 0;
  bool ok = true;
  if (tid == 0) L = *a.st;
  __syncthreads();
  if (L.done) return;

  const int lane = tid & 31, warp = tid >> 5;
  // body(i, accumulator) for each element of the vectors, in the graph
  // kernels' virtual blocks, and their sums to `sums` (may be null)
  // (four virtual blocks at a time, a warp for each one's sum: a block that had
  // three of them one after another, 1000 cycles a sum, kept all others waiting)
  auto for_vec = [&](double* sums, auto zero, auto&& body) {
    typedef BlockTree<VT> B;
    __shared__ double values[4][B::WORDS];
    for (int v0 = blockIdx.x; v0 < a.vb; v0 += 4 * G) {
      if (sums) __syncthreads();
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int v = v0 + k * G;
        if (v >= a.vb) break;
        auto acc = zero;
        for (long long i = v * (long long)VT + tid; i < n; i += (long long)a.vb * VT) body(i, acc);
        if (sums) B::put(values[k], (double)acc);
      }
      if (!sums) continue;
      __syncthreads();
      const int v = v0 + warp * G;
      if (warp < 4 && v < a.vb) {
        const double bs = B::sum(values[warp]);
        if (lane == 0) sums[v] = bs;
      }
    }
  };
  // body(row, accumulator) for each row, its warps of 32 rows dealt out over all
  // blocks, and their sums to `sums`
  auto for_rows = [&](double* sums, auto zero, auto&& body) {
    for (int sl = warp * G + blockIdx.x; sl < slices; sl += 8 * G) {
      const long long row = 32LL * sl + lane;
      auto acc = zero;
      if (row < a.S) body(row, acc);
      const double w = warp_tree((double)acc);
      if (lane == 0) sums[sl] = w;
    }
  };
  // body(row, y = (A in)(row), accumulator) for each row of the blocks. With
  // few rows three warps take 32 of them, one a component, and meet in shared
  // memory (a warp alone is 1000 instructions at ten cycles each); where every
  // block has more than two warps of rows the warps take rows alone.
  auto for_block_rows = [&](const T* in, double* sums, auto zero, auto&& body) {
    if (slices > 2 * G) {
      for_rows(sums, zero, [&](long long row, auto& acc) {
        T y[3];
#pragma unroll
        for (int c = 0; c < 3; c++) y[c] = spmv_component(a.blocks, a.nbr, in, row, c);
        body(row, y, acc);
      });
      return;
    }
    const int unit = warp / 3, sl = unit * G + blockIdx.x;
    const long long row = 32LL * sl + lane;
    const bool mine = warp < 6 && sl < slices && row < a.S;
    if (mine) sy[unit][warp % 3][lane] = spmv_component(a.blocks, a.nbr, in, row, warp % 3);
    __syncthreads();
    if (warp < 6 && warp % 3 == 0 && sl < slices) {
      auto acc = zero;
      if (mine) {
        const T y[3] = {sy[unit][0][lane], sy[unit][1][lane], sy[unit][2][lane]};
        body(row, y, acc);
      }
      const double w = warp_tree((double)acc);
      if (lane == 0) sums[sl] = w;
    }
  };
  // s = A r, partial r.s (MATRIX_FREE: r first takes its update by alpha)
  auto apply = [&](T alpha, bool update) {
    if constexpr (MATRIX_FREE) {
      auto next = [&](long long i) { return upd_r(a.r[i], alpha, a.Ap[i], __ldg(a.invd + i)); };
      for (long long t = blockIdx.x * (long long)VT + tid; t < a.mf.nc; t += (long long)G * VT)
        mf_cell(a.mf, t, next, a.share);
      if (!persist_sync(a.bar, target)) return false;
      for_rows(ps, 0.0f, [&](long long row, float& accT) {
        float y[3];
        mf_node(a.mf, row, a.share, y);
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const long long i = 3 * row + c;
          const float in = next(i);
          if (update) {
            a.r[i] = in;
            a.x[i] = a.x[i] + alpha * a.d[i];
          }
          y[c] += __ldg(a.damped + i) * in;
          a.s[i] = y[c];
          accT += in * y[c];
        }
      });
    } else {
      for_block_rows(a.r, ps, (T)0, [&](long long row, const T* y, T& accT) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const long long i = 3 * row + c;
          a.s[i] = y[c];
          accT += a.r[i] * y[c];
        }
      });
    }
    if (!persist_sync(a.bar, target)) return false;
    const double total = persist_fold_rows(ps, slices);
    if (tid == 0) finish_update(&L, total);
    __syncthreads();
    return true;
  };

  if (L.setup) {  // r = b/diag, ||b||^2; x = d = Ap = 0; s = A r
    for_vec(pz, 0.0, [&](long long i, double& acc) {
      const T bv = a.b[i];
      a.x[i] = 0;
      a.r[i] = bv * a.invd[i];
      a.d[i] = 0;
      a.Ap[i] = 0;
      acc += (double)bv * (double)bv;
    });
    ok = persist_sync(a.bar, target);
    const double total = fold_partials<VT>(pz, a.vb);
    if (tid == 0) L.bnorm2 = total;
    __syncthreads();
    ok = ok && apply((T)0, false);
  }
  for (int it = 0; ok && it < budget && !L.done; it++) {
    if (L.iter >= L.maxIt) {
      __syncthreads();
      if (tid == 0) L.done = 1;
      __syncthreads();
      break;
    }
    // d = beta d + r; Ap = beta Ap + s; Ap . Ap/diag
    const T beta = (T)L.beta;
    for_vec(pv, (T)0, [&](long long i, T& acc) {
      const T iv = a.invd[i];
      const T dn = beta * a.d[i] + a.r[i];
      const T an = beta * a.Ap[i] + a.s[i];
      a.d[i] = dn;
      a.Ap[i] = an;
      acc += an * (an * iv);
    });
    ok = persist_sync(a.bar, target);
    if (!ok) break;
    const double total = fold_partials<VT>(pv, a.vb);
    if (tid == 0) {
      L.alpha = (fabs(total) > 0.0) ? L.delta / total : total;
      if (!(total == total)) {
        L.status = ESF_ERR_NUMERIC;
        L.done = 1;
      }
    }
    __syncthreads();
    if (L.done) break;
    const T alpha = (T)L.alpha;
    if constexpr (!MATRIX_FREE) {  // x += alpha d; r -= alpha Ap/diag
      for_vec(nullptr, 0, [&](long long i, int&) {
        a.x[i] = a.x[i] + alpha * a.d[i];
        a.r[i] = upd_r(a.r[i], alpha, a.Ap[i], a.invd[i]);
      });
      ok = persist_sync(a.bar, target);
      if (!ok) break;
    }
    // (a check after this update reads the iteration before finish_update moves it)
    const bool check = !L.inner && L.iter > 0 && L.iter % 5 == 0;
    ok = apply(alpha, true);
    if constexpr (!MATRIX_FREE) {
      if (ok && check && !L.done) {  // ||A x - b||^2 against eps ||b||
        for_block_rows(a.x, pc, 0.0, [&](long long row, const T* y, double& acc) {
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double t = (double)y[c] - (double)a.b[3 * row + c];
            acc += t * t;
          }
        });
        ok = persist_sync(a.bar, target);
        const double res = persist_fold_rows(pc, slices);
        if (tid == 0) {
          L.resid2 = res;
          if (sqrt(res) < L.eps * sqrt(L.bnorm2)) {
            L.converged = 1;
            L.done = 1;
          } else {
            L.iter++;
          }
          if (!(res == res)) {
            L.status = ESF_ERR_NUMERIC;
            L.done = 1;
          }
        }
        __syncthreads();
      }
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    if (!ok) {
      L.status = ESF_ERR_CUDA;
      L.done = 1;
    }
    *a.st = L;
  }
}

// Rows (solid nodes) up to which a solve runs persistent: beyond, one block an
// SM holds the memory system back more than the launches cost. Measured solid
// solve of a step, graph against persistent: 9.3 and 7.6 ms (FP64), 5.4 and 5.1
// (FP32) at 65 thousand rows; 18.2 and 21.2, 8.9 and 9.5 at 139 thousand.
// ESF_SOLID_SOLVE=graph keeps the graphs for any size, for comparison.
static long long persist_rows() {
  const char* e = getenv("ESF_SOLID_SOLVE");
  return e && strcmp(e, "graph") == 0 ? 0 : PERSIST_MAX_ROWS;
}

template <typename T>
static esf_status solid_pcr_persist(SolidPersist<T> p, bool mf, PcrState* hst, cudaStream_t st, PcrState* out) {
  int dev = 0, sms = 0;
  ESF_CUDA(cudaGetDevice(&dev));
  ESF_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const void* kernel = (const void*)solid_pcr_persistent<T, false>;
  if constexpr (std::is_same<T, float>::value)
    if (mf) kernel = (const void*)solid_pcr_persistent<float, true>;
  // one block an SM leaves room for the kernels of other scenes' streams, and
  // 64 unknowns a block spread a small solid's rows over many SMs; a
  // launch takes at most kBudget iterations, so that it ends in milliseconds
  constexpr int kBudget = 512;
  const int blocks = (int)std::min<long long>(sms, (3 * p.S + 63) / 64);
  int budget = kBudget;
  do {
    ESF_CUDA(cudaMemsetAsync(p.bar, 0, 2 * sizeof(unsigned), st));
    void* args[] = {&p, &budget};
    note_launch();
    ESF_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(VT), args, 0, st));
    ESF_CUDA(cudaMemcpyAsync(hst, p.st, sizeof(PcrState), cudaMemcpyDeviceToHost, st));
    ESF_CUDA(cudaStreamSynchronize(st));
    *out = hst[0];
  } while (!out->done);
  if (out->status == ESF_ERR_CUDA) {
    set_error("solid solve: a grid barrier timed out");
    return ESF_ERR_CUDA;
  }
  return ESF_OK;
}
