// Decoupling of every compressed box of a level in one launch
// (SkelFactorization::decouple, skel_factorization.cpp:55-91), and the dense
// assembly of the top-level skeleton matrix (skel_factorization.cpp:116-122).
//
// Per box, in pivot order [s; r] of the ID:
//   K_BN     = K(act, act) - (accumulated Schur updates of compressed boxes
//              below, restricted to the active dofs)
//   K_r_sn   = K_rs - T^T K_ss
//   X_rr     = (K_rr - T^T K_sr) - K_r_sn T
//   K_sn_r   = K_sr - K_ss T
//   X_rr^-1  by Gauss-Jordan elimination with partial pivoting (kept: the
//            solve sweeps multiply by it instead of solving with LU factors)
//   U        = X_rr^{-1} K_r_sn,  L = K_sn_r X_rr^{-1}   (GEMMs)
//   L       += (K_sn_r - L X_rr) X_rr^{-1}   (reference mode: a product with
//            the inverse from the right leaves a residual of cond(X_rr) eps,
//            where the reference's triangular solves leave eps; on the
//            4,096-node circle at id_tol 1e-13 the solution's error against
//            the analytic one is 1e-12 without this correction, 1e-14 with
//            it.  A preconditioner does not need it)
//   acc      = update(s, s) + L K_r_sn      (what the ancestors subtract)
// The reference re-searches every compressed descendant's skeleton inside
// the parent's index list (skel_factorization.cpp:246-294); here each box
// passes up one accumulated update on its skeleton, addressed through
// per-position block ids built on the host, so assembly is a direct lookup.
#include "ki_blockla.cuh"
#include "ki_kernels.h"

namespace kib {

namespace {

constexpr int kDecThreads = 256;
constexpr size_t kDecSmemMax = 227 * 1024;

__device__ __forceinline__ double upd_lookup(const int* bid, const int* bpos,
                                             const UpdBlock* blocks, int a, int b) {
  const int ia = bid[a];
  if (ia < 0 || ia != bid[b]) return 0.0;
  const UpdBlock blk = blocks[ia];
  return blk.acc[bpos[a] + static_cast<long long>(blk.size) * bpos[b]];
}

// Leading dimension of a matrix in shared memory whose DMMA fragments are
// read in place: 4 mod 8 doubles, so the four inner indices (or rows) of a
// half-warp's fragment, a stride apart, start 4 or 12 banks of 16 apart and
// its four consecutive entries fill the gaps: no two lanes share a bank.
__host__ __device__ inline int frag_ld(int n) { return n + ((4 - n % 8) + 8) % 8; }

// The CTA's product op(A) op(B) (m x n, inner kk) on the FP64 tensor cores,
// the operands in shared memory with a frag_ld stride (X_rr of L's
// correction: in global memory); out(i, j, v) receives every entry.  A warp computes 16 x 16 blocks (2 x 2 DMMA blocks)
// straight from the operands: no staging, no barriers.
template <bool TA, bool TB, class Out>
__device__ __forceinline__ void cta_mma(const double* A, int lda, const double* B, int ldb, int m,
                                        int n, int kk, Out out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr = lane >> 2, fk = lane & 3;
  const int tm = (m + 15) / 16, tn = (n + 15) / 16;
  for (int t = warp; t < tm * tn; t += kDecThreads / 32) {
    const int i0 = t % tm * 16, j0 = t / tm * 16;
    // (rows and columns past the edge repeat the last: never stored)
    const double *pa[2], *pb[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = min(i0 + 8 * h + fr, m - 1), j = min(j0 + 8 * h + fr, n - 1);
      pa[h] = TA ? A + static_cast<size_t>(lda) * i : A + i;
      pb[h] = TB ? B + j : B + static_cast<size_t>(ldb) * j;
    }
    double acc[2][2][2] = {};
#pragma unroll 4
    for (int l0 = 0; l0 < kk; l0 += 4) {
      const int l = l0 + fk;
      double fa[2], fb[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        fa[h] = l < kk ? pa[h][TA ? l : lda * l] : 0.0;
        fb[h] = l < kk ? pb[h][TB ? ldb * l : l] : 0.0;
      }
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int y = 0; y < 2; y++) dmma_8x8x4(acc[x][y][0], acc[x][y][1], fa[x], fb[y]);
    }
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < 2; y++)
#pragma unroll
        for (int v = 0; v < 2; v++) {
          const int i = i0 + 8 * x + fr, j = j0 + 8 * y + 2 * fk + v;
          if (i < m && j < n) out(i, j, acc[x][y][v]);
        }
  }
}

// Gauss-Jordan inversion of the r x r matrix X (shared memory, stride ld) by
// the CTA's 8 warps with the matrix in registers: warp w owns the columns
// c % 8 == w, its lanes the rows (lane + 32 s in slot s), a thread CW x RS
// entries.  Partial pivoting, rows never exchanged: step j eliminates column
// j with row p_j (the largest |x(i, j)| among the rows not yet pivots, the
// first on ties; a NaN counts as 0).  The owner warp of column j finds p_j
// and publishes the column (double-buffered by step parity), one barrier, and
// every warp updates its columns: row p_j's entries come by shuffle from the
// lane that holds them.  In place the result B holds X^{-1}(j, q) =
// B(p_j, p^{-1}(q)); it is stored to X in X^{-1}'s own order.  pr, pi: p and
// p^{-1}.  Returns nonzero when a pivot was 0, infinite or NaN.
// A step moves the pivot column through shared memory once; with the matrix
// there (a thread per row segment) it moved 24 bytes per entry and step:
// 6,000 against 900 cycles a step for r = 70 with the SM shared.
template <int CW, int RS>
__device__ __forceinline__ int cta_gj_regs(double* X, int ld, int r, double* colj, int* sp, int* pr,
                                           int* pi) {
  constexpr int RP = 32 * RS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double x[CW][RS];
#pragma unroll
  for (int u = 0; u < CW; u++) {
    const int c = u * 8 + warp;
#pragma unroll
    for (int s = 0; s < RS; s++) {
      const int i = lane + 32 * s;
      x[u][s] = c < r && i < r ? X[i + static_cast<size_t>(ld) * c] : 0.0;
    }
  }
  unsigned used = 0;  // slots whose row has been a pivot
  int info = 0;
  for (int j = 0; j < r; j++) {
    double* cj = colj + (j & 1) * RP;
    if ((j & 7) == warp) {
      // (comparing columns, not u: with an equality on u the compiler indexes
      // the register array by it and puts it in local memory)
      double y[RS];
#pragma unroll
      for (int u = 0; u < CW; u++)
        if (u * 8 + warp == j) {
#pragma unroll
          for (int s = 0; s < RS; s++) y[s] = x[u][s];
        }
      unsigned long long key = 0;
      int idx = 0x7fffffff;
#pragma unroll
      for (int s = 0; s < RS; s++) {
        const int i = lane + 32 * s;
        double v = fabs(y[s]);
        if (v != v) v = 0.0;
        const unsigned long long k = static_cast<unsigned long long>(__double_as_longlong(v));
        if (i < r && !(used >> s & 1) && (idx == 0x7fffffff || k > key)) {
          key = k;
          idx = i;
        }
        cj[i] = y[s];
      }
      unsigned long long gk;
      int p;
      warp_argmax_bits(key, idx, &gk, &p);
      if (lane == 0) {
        sp[j & 1] = p;
        pr[j] = p;
        pi[p] = j;
      }
    }
    __syncthreads();
    const int p = sp[j & 1];
    const double piv = cj[p];
    if (!(fabs(piv) > 0.0) || isinf(piv)) info = 1;  // (0, NaN or infinite)
    const double inv = 1.0 / piv;
    double f[RS];
#pragma unroll
    for (int s = 0; s < RS; s++) f[s] = lane + 32 * s == p ? 0.0 : cj[lane + 32 * s];
#pragma unroll
    for (int s = 0; s < RS; s++) {
      const int t = p - 32 * s;
      if (static_cast<unsigned>(t) < 32u) {  // the slot of row p
#pragma unroll
        for (int u = 0; u < CW; u++) {
          const double q = __shfl_sync(0xffffffffu, x[u][s], t) * inv;
#pragma unroll
          for (int h = 0; h < RS; h++) x[u][h] = fma(-f[h], q, x[u][h]);
          if (lane == t) x[u][s] = q;
        }
        if (lane == t) used |= 1u << s;
      }
    }
    if ((j & 7) == warp) {
#pragma unroll
      for (int u = 0; u < CW; u++)
        if (u * 8 + warp == j) {
#pragma unroll
          for (int s = 0; s < RS; s++) x[u][s] = lane + 32 * s == p ? inv : -f[s] * inv;
        }
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < CW; u++) {
    const int c = u * 8 + warp;
    if (c < r) {
      double* col = X + static_cast<size_t>(ld) * pr[c];
#pragma unroll
      for (int s = 0; s < RS; s++) {
        const int i = lane + 32 * s;
        if (i < r) col[pi[i]] = x[u][s];
      }
    }
  }
  __syncthreads();
  return info;
}

// Shared memory of a box: K_BN (in place K_r_sn, K_sn_r, X_rr and its
// inverse), T and later L (tl: unless they stay in global memory), the pivot
// column twice, pivots, per-dof ints.
struct DecLayout {
  int ldn, ldk;
  size_t tl, colj, ints, bytes;  // offsets in doubles, total bytes
};
__host__ __device__ inline DecLayout dec_layout(int n, int k, bool tl) {
  DecLayout d;
  const int r = n - k;
  d.ldn = frag_ld(n);
  d.ldk = tl ? frag_ld(k) : k;
  d.tl = static_cast<size_t>(n) * d.ldn;
  const size_t t = tl ? static_cast<size_t>(d.ldk) * r : 0, nodes = 8 * static_cast<size_t>(n);
  d.colj = d.tl + (((t > nodes ? t : nodes) + 1) & ~static_cast<size_t>(1));
  d.ints = d.colj + 2 * 160;
  d.bytes = sizeof(double) * d.ints + sizeof(int) * (5 * static_cast<size_t>(n) + 4);
  return d;
}

// FAST: entries by contracted arithmetic (a preconditioner's, whose sketched
// IDs use it too: on stars and circles of 1,024 to 32,768 nodes their rms
// error against 64-bit significands is 0.57 to 0.92 of that of the reference's
// order of roundings, for every kernel and distance); else the reference's
// bits, and L corrected.  TL: T is
// copied to shared memory, where L takes its place; else, for boxes whose
// K_BN leaves no room for it (149 dofs and more, by rank), the products read
// T, and L as it is made, in global memory (from L1: a warp's fragment is
// eight runs of four entries).  Sent through decouple_large instead, as the
// only alternative, such boxes cost 17 launches each: 16,384-node star, 160
// dofs a leaf, 4.65 ms against 2.96 ms, 200 a leaf 7.26 against 5.44 ms.
template <int CW, int RS, int MINB, bool FAST, bool TL>
__global__ void __launch_bounds__(kDecThreads, MINB) decouple_kernel(DecParams P) {
  extern __shared__ __align__(16) double dsm[];
  const DecTask tk = P.tasks[blockIdx.x];
  const int n = tk.n, k = tk.k, r = n - k;
  const DecLayout lay = dec_layout(n, k, TL);
  const int ldn = lay.ldn, ldk = lay.ldk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* K = dsm;
  const double* T = TL ? dsm + lay.tl : tk.T;
  double* L = TL ? dsm + lay.tl : tk.L;
  double* colj = dsm + lay.colj;
  int* prow = reinterpret_cast<int*>(dsm + lay.ints);  // n
  int* pinv = prow + n;                                 // n
  int* dof = pinv + n;                                  // n, pivot order; likewise:
  int* sbid = dof + n;                                  // n
  int* sbpos = sbid + n;                                // n
  int* sp = sbpos + n;                                  // 2

  // ---- K_BN in pivot order: a lane keeps its row's node record and block,
  // the columns' records pass by broadcast, four at a time (their update
  // entries are loads from global memory)
  Node* nd = reinterpret_cast<Node*>(dsm + lay.tl);
  const int sh = P.pde == kStokes ? 1 : 0;
  for (int a = threadIdx.x; a < n; a += kDecThreads) {
    const int pa = tk.perm[a], d = tk.act[pa];
    dof[a] = d;
    nd[a] = P.nodes[d >> sh];
    sbid[a] = tk.bid[pa];
    sbpos[a] = tk.bpos[pa];
  }
  __syncthreads();
  {
    const int rb = (n + 31) / 32, nch = (8 + rb - 1) / rb;
    for (int w = warp; w < rb * nch; w += kDecThreads / 32) {
      const int a = 32 * (w % rb) + lane, ch = w / rb;
      const bool in = a < n;
      const int aa = in ? a : n - 1;
      const Node na = nd[aa];
      const int da = dof[aa], ba = sbid[aa], pa = sbpos[aa];
      const double* acc = ba >= 0 ? tk.blocks[ba].acc + pa : nullptr;
      const int size = ba >= 0 ? tk.blocks[ba].size : 0;
      const int b1 = (ch + 1) * n / nch;
      for (int b0 = ch * n / nch; b0 < b1; b0 += 4) {
        double up[4], v[4];
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int b = min(b0 + h, b1 - 1);
          up[h] = ba >= 0 && sbid[b] == ba ? acc[static_cast<size_t>(size) * sbpos[b]] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 4; h++) {
          const int b = min(b0 + h, b1 - 1);
          v[h] = pair_entry<FAST>(P.pde, na, da, nd[b], dof[b]) - up[h];
        }
#pragma unroll
        for (int h = 0; h < 4; h++)
          if (in && b0 + h < b1) K[a + static_cast<size_t>(ldn) * (b0 + h)] = v[h];
      }
    }
  }
  __syncthreads();
  if (TL) {
    for (int c = warp; c < r; c += kDecThreads / 32)
      for (int l = lane; l < k; l += 32)
        L[l + static_cast<size_t>(ldk) * c] = tk.T[l + static_cast<size_t>(k) * c];
    __syncthreads();
  }
  double* Kss = K;
  double* Krs = K + k;
  double* Ksr = K + static_cast<size_t>(ldn) * k;
  double* Krr = Ksr + k;
  auto minus = [&](double* C) {
    return [C, ldn](int i, int j, double v) { C[i + static_cast<size_t>(ldn) * j] -= v; };
  };
  // K_r_sn = K_rs - T^T K_ss,  X = (K_rr - T^T K_sr) - K_r_sn T,  K_sn_r =
  // K_sr - K_ss T, each in place (an entry is read as C only by the thread
  // that replaces it)
  cta_mma<true, false>(T, ldk, Kss, ldn, r, k, k, minus(Krs));
  cta_mma<true, false>(T, ldk, Ksr, ldn, r, r, k, minus(Krr));
  __syncthreads();
  cta_mma<false, false>(Krs, ldn, T, ldk, r, r, k, minus(Krr));
  cta_mma<false, false>(Kss, ldn, T, ldk, k, r, k, minus(Ksr));
  __syncthreads();
  auto store_x = [&]() {
    for (int c = warp; c < r; c += kDecThreads / 32)
      for (int i = lane; i < r; i += 32)
        tk.X[i + static_cast<size_t>(r) * c] = Krr[i + static_cast<size_t>(ldn) * c];
  };
  // (L's correction needs X_rr itself: until then it waits in the place of
  // its inverse)
  if (!FAST) store_x();
  const int info = cta_gj_regs<CW, RS>(Krr, ldn, r, colj, sp, prow, pinv);
  if (info && threadIdx.x == 0) atomicExch(P.status, 1);
  for (int j = threadIdx.x; j < r; j += kDecThreads) tk.piv[j] = prow[j];
  if (FAST) store_x();
  // U = X^{-1} K_r_sn,  L = K_sn_r X^{-1}  (TL: in T's place)
  cta_mma<false, false>(Krr, ldn, Krs, ldn, r, k, r, [&](int i, int j, double v) {
    tk.U[i + static_cast<size_t>(r) * j] = v;
  });
  cta_mma<false, false>(Ksr, ldn, Krr, ldn, k, r, r, [&](int i, int j, double v) {
    L[i + static_cast<size_t>(ldk) * j] = v;
  });
  __syncthreads();
  if (!FAST) {
    cta_mma<false, false>(L, ldk, tk.X, r, k, r, r, minus(Ksr));
    __syncthreads();
    store_x();
    cta_mma<false, false>(Ksr, ldn, Krr, ldn, k, r, r, [&](int i, int j, double v) {
      L[i + static_cast<size_t>(ldk) * j] += v;
    });
    __syncthreads();
  }
  if (TL)
    for (int c = warp; c < r; c += kDecThreads / 32)
      for (int l = lane; l < k; l += 32)
        tk.L[l + static_cast<size_t>(k) * c] = L[l + static_cast<size_t>(ldk) * c];
  // acc = update(s, s) + L K_r_sn
  cta_mma<false, false>(L, ldk, Krs, ldn, k, k, r, [&](int i, int j, double v) {
    const int bi = sbid[i];
    double up = 0.0;
    if (bi >= 0 && bi == sbid[j])
      up = tk.blocks[bi].acc[sbpos[i] + static_cast<size_t>(tk.blocks[bi].size) * sbpos[j]];
    tk.acc[i + static_cast<size_t>(k) * j] = v + up;
  });
}

__global__ void assemble_top_kernel(int pde, const Node* nodes, const int* dofs, int n,
                                    const int* bid, const int* bpos, const UpdBlock* blocks,
                                    double* out, int ld) {
  const long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (e >= static_cast<long long>(n) * n) return;
  const int a = static_cast<int>(e % n), b = static_cast<int>(e / n);
  out[a + static_cast<long long>(ld) * b] =
      boundary_entry(pde, nodes, dofs[a], dofs[b]) - upd_lookup(bid, bpos, blocks, a, b);
}

__global__ void assemble_perm_kernel(int pde, const Node* nodes, const int* act, const int* perm,
                                     int n, const int* bid, const int* bpos,
                                     const UpdBlock* blocks, double* K) {
  const long long e = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (e >= static_cast<long long>(n) * n) return;
  const int a = static_cast<int>(e % n), b = static_cast<int>(e / n);
  const int pa = perm[a], pb = perm[b];
  K[e] = boundary_entry(pde, nodes, act[pa], act[pb]) - upd_lookup(bid, bpos, blocks, pa, pb);
}

__global__ void identity_kernel(double* y, int r) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < r * r) y[e] = (e % r == e / r) ? 1.0 : 0.0;
}

__global__ void acc_finish_kernel(double* acc, int k, const int* perm, const int* bid,
                                  const int* bpos, const UpdBlock* blocks) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= k * k) return;
  const int i = e % k, j = e / k;
  acc[e] = upd_lookup(bid, bpos, blocks, perm[i], perm[j]) - acc[e];
}

}  // namespace

// K_BN (n x n), the LU's flags, and X_rr in reference mode
size_t decouple_large_scratch(int n, int k, bool fast) {
  const size_t r = static_cast<size_t>(n) - k;
  return static_cast<size_t>(n) * n + kLuSyncInts + (fast ? 0 : r * r);
}

cudaError_t decouple_large(const DecTask& tk, int pde, const Node* nodes, int* status, bool fast,
                           cudaStream_t s) {
  const int n = tk.n, k = tk.k, r = n - k;
  const long long nn = static_cast<long long>(n) * n;
  count_launches(2);
  assemble_perm_kernel<<<static_cast<int>((nn + 255) / 256), 256, 0, s>>>(
      pde, nodes, tk.act, tk.perm, n, tk.bid, tk.bpos, tk.blocks, tk.K);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const double* K = tk.K;
  const double* Kss = K;
  const double* Krs_in = K + k;
  const double* Ksr = K + static_cast<long long>(n) * k;
  const double* Krr = K + k + static_cast<long long>(n) * k;
  // K_r_sn in U, K_sn_r in L, X = (K_rr - T^T K_sr) - K_r_sn T
  if ((e = launch_gemm_sub(tk.U, r, Krs_in, n, tk.T, k, true, Kss, n, false, r, k, k, s))) return e;
  if ((e = launch_gemm_sub(tk.L, k, Ksr, n, Kss, n, false, tk.T, k, false, k, r, k, s))) return e;
  if ((e = launch_gemm_sub(tk.X, r, Krr, n, tk.T, k, true, Ksr, n, false, r, r, k, s))) return e;
  if ((e = launch_gemm_sub(tk.X, r, tk.X, r, tk.U, r, false, tk.T, k, false, r, r, k, s))) return e;
  // X^{-1}: LU, then the solve of X Y = I (one CTA per column), into X
  // through the K scratch (K is no longer needed); K_r_sn and K_sn_r are
  // kept behind it (r^2 + 2 k r <= n^2)
  double* Y = tk.K;
  double* Krsn = Y + static_cast<long long>(r) * r;
  double* Ksnr = Krsn + static_cast<long long>(r) * k;
  if ((e = cudaMemcpyAsync(Krsn, tk.U, sizeof(double) * r * k, cudaMemcpyDeviceToDevice, s)))
    return e;
  if ((e = cudaMemcpyAsync(Ksnr, tk.L, sizeof(double) * r * k, cudaMemcpyDeviceToDevice, s)))
    return e;
  double* X0 = tk.K + nn + kLuSyncInts;  // X_rr, for L's correction
  if (!fast && (e = cudaMemcpyAsync(X0, tk.X, sizeof(double) * r * r, cudaMemcpyDeviceToDevice, s)))
    return e;
  if ((e = dense_lu(tk.X, r, r, tk.piv, status, s, reinterpret_cast<int*>(tk.K + nn)))) return e;
  count_launches(1);
  identity_kernel<<<(r * r + 255) / 256, 256, 0, s>>>(Y, r);
  if ((e = cudaGetLastError())) return e;
  if ((e = dense_lu_solve(tk.X, r, r, tk.piv, Y, r, r, s))) return e;
  if ((e = cudaMemcpyAsync(tk.X, Y, sizeof(double) * r * r, cudaMemcpyDeviceToDevice, s))) return e;
  // U = X^{-1} K_r_sn, L = K_sn_r X^{-1}, acc = update + L K_r_sn
  if ((e = launch_gemm_tiled(tk.U, r, nullptr, 0, tk.X, r, false, Krsn, r, false, r, k, r, 1.0,
                             s)))
    return e;
  if ((e = launch_gemm_tiled(tk.L, k, nullptr, 0, Ksnr, k, false, tk.X, r, false, k, r, r, 1.0,
                             s)))
    return e;
  if (!fast) {
    if ((e = launch_gemm_sub(Ksnr, k, Ksnr, k, tk.L, k, false, X0, r, false, k, r, r, s)))
      return e;
    if ((e = launch_gemm_tiled(tk.L, k, tk.L, k, Ksnr, k, false, tk.X, r, false, k, r, r, 1.0, s)))
      return e;
  }
  if ((e = launch_gemm_sub(tk.acc, k, nullptr, 0, tk.L, k, false, Krsn, r, false, k, k, r, s)))
    return e;
  acc_finish_kernel<<<(k * k + 255) / 256, 256, 0, s>>>(tk.acc, k, tk.perm, tk.bid, tk.bpos,
                                                         tk.blocks);
  return cudaGetLastError();
}

namespace {
// The register tile of X_rr's inversion by r, and the CTAs of it an SM's
// registers hold (without TL: its shared memory holds one).
template <int CW, int RS, int MINB, bool FAST, bool TL>
cudaError_t launch_class(const DecParams& p, size_t smem, cudaStream_t s) {
  const cudaError_t e = raise_func_attr(
      reinterpret_cast<const void*>(&decouple_kernel<CW, RS, MINB, FAST, TL>),
      cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  count_launches(1);
  decouple_kernel<CW, RS, MINB, FAST, TL><<<p.ntasks, kDecThreads, smem, s>>>(p);
  return cudaGetLastError();
}
template <bool FAST>
cudaError_t launch_any(const DecParams& p, int cls, size_t smem, cudaStream_t s) {
  switch (cls) {
    case 0: return launch_class<8, 2, 3, FAST, true>(p, smem, s);
    case 1: return launch_class<12, 3, 2, FAST, true>(p, smem, s);
    case 2: return launch_class<20, 5, 1, FAST, true>(p, smem, s);
    case 3: return launch_class<8, 2, 1, FAST, false>(p, smem, s);
    case 4: return launch_class<12, 3, 1, FAST, false>(p, smem, s);
    case 5: return launch_class<20, 5, 1, FAST, false>(p, smem, s);
    default: return cudaErrorInvalidValue;
  }
}
}  // namespace

int decouple_class(int n, int k) {
  const int r = n - k, tile = r <= 64 ? 0 : r <= 96 ? 1 : r <= 160 ? 2 : -1;
  if (tile < 0) return -1;
  if (dec_layout(n, k, true).bytes <= kDecSmemMax) return tile;
  return dec_layout(n, k, false).bytes <= kDecSmemMax ? 3 + tile : -1;
}

size_t decouple_smem_bytes(int n, int k) {
  return dec_layout(n, k, decouple_class(n, k) < 3).bytes;
}

cudaError_t launch_decouple(const DecParams& p, int cls, bool fast, size_t smem, cudaStream_t s) {
  if (p.ntasks == 0) return cudaSuccess;
  return fast ? launch_any<true>(p, cls, smem, s) : launch_any<false>(p, cls, smem, s);
}

cudaError_t launch_assemble_top(int pde, const Node* nodes, const int* dofs, int n,
                                const int* bid, const int* bpos, const UpdBlock* blocks,
                                double* out, int ld, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const long long total = static_cast<long long>(n) * n;
  const int threads = 256;
  const int grid = static_cast<int>((total + threads - 1) / threads);
  count_launches(1);
  assemble_top_kernel<<<grid, threads, 0, s>>>(pde, nodes, dofs, n, bid, bpos, blocks, out,
                                                ld);
  return cudaGetLastError();
}

}  // namespace kib
