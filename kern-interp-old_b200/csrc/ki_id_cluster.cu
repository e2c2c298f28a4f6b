// Interpolative decomposition of every box of one quadtree level in one
// launch, each box on chip: fused ID-matrix generation, column-pivoted
// Householder QR with the reference's rank rule, and T = R11^{-1} R12.
//
// Reference semantics (paths relative to the reference repository):
//   * ID matrix rows: Kernel::get_id_mat, kernel.cpp:153-235 (proxy circle
//     of radius 1.5 side with 128 points; levels 1-2 use all other boxes).
//   * Pivoting and Householder steps: LAPACK dgeqp3/dlaqp2 as called by
//     ki_Mat::id (ki_mat.cpp:502-541): first-maximum column pivot on the
//     partial column norms, dlarfg reflector (beta = -sign(alpha) |x|), the
//     norm downdate with recomputation when it loses accuracy (tol3z).
//   * Rank: first i >= 1 with |R_ii| < tol |R_00|; none => 0 (no compression).
//   * T = R11^{-1} R12 by column back substitution (dtrtrs).
// The factorization stops at the rank: R_ii never changes after step i and
// T only needs R's first k rows, so steps k..n-1 of dgeqp3 are skipped.  The
// skeleton (pivots 0..k-1, in order) is unchanged by this; the redundant
// columns come out in their order at step k instead of dgeqp3's later pivot
// order, which only permutes the redundant set inside the box.
//
// Layout.  A box is owned by a cluster of G CTAs and its rows are dealt
// round-robin (row r to CTA r % G), every CTA holding its rows of all n
// columns.  A pivot step is then: every CTA, on its own rows, one pass over
// the trailing columns; one exchange of n partial sums; and the rest of the
// step (reflector, R row, norms, next pivot) computed by every CTA alike
// from the same numbers in the same order, so the CTAs need no second
// exchange and stay in step.  With the columns dealt instead, every CTA had
// to read the whole pivot column from its owner each step, fifteen readers
// of one SM's shared memory in a 16-CTA cluster.
//
// What bounds it is shared memory.  A step applies the previous reflector
// to the trailing columns and takes their products with the next pivot
// column in ONE pass (a column's products with an unscaled reflector need
// no norm first: v = [1; x / (alpha - beta)]), each warp carrying four
// columns (eight in the short variant) past one load of the two vectors: 20
// to 24 bytes of shared memory per matrix element and step, where an update
// pass after a product pass, a column at a time, took 40.  The column norms
// LAPACK downdates are summed afresh in the same pass for a quarter of the
// columns each step (FP64 arithmetic is not the bound), so its tol3z
// recomputation, which would need another exchange, all but never runs.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "ki_blockla.cuh"
#include "ki_kernels.h"

namespace cg = cooperative_groups;

namespace kib {

namespace {

constexpr int kOcThreads = 512;  // 16 warps per CTA
constexpr int kOcWarps = kOcThreads / 32;

// 32-bit integer hash (the "lowbias32" finalizer published by C. Wellons):
// the sketch takes its row choice from the low bits and its sign from the
// top bit.
__device__ __forceinline__ unsigned sketch_hash(unsigned x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

// ------------------------------------------------------------ generation
// Entries are made by pairs of rows that share a node pair: near row r of
// the ID matrix is K(row, column), row I + r is K(column, row), and the two
// have the same |r|^2 (and, in fast arithmetic, one reciprocal); proxy point
// q's rows, as targets and as sources, likewise.  FAST: contracted, Newton
// reciprocals; else every operation of pair_entry / proxy_entry_node in
// their order (a negated difference changes no bit of the products), so the
// entries keep the reference's bits.  A near row is never a node of the box
// (coincident nodes are refused before any ID), so there is no diagonal case
// here, whose branch would keep the entries of several columns apart.

// Stokes, row dof component rc of node rn, both dofs of column node cn:
// e0, e1 = K(row, col x / y), e2, e3 = K(col x / y, row).
template <bool FAST>
__device__ __forceinline__ void stokes_near2(const Node& rn, int rc, const Node& cn, double* e) {
  using M = EM<FAST>;
  const double r0 = M::sub(rn.x, cn.x), r1 = M::sub(rn.y, cn.y);
  const double rr = M::add(M::mul(r0, r0), M::mul(r1, r1));
  const double nc = M::mul(M::mul(cn.w, KI_INV_PI), M::add(M::mul(r0, cn.nx), M::mul(r1, cn.ny)));
  const double nr =
      M::mul(M::mul(rn.w, KI_INV_PI), M::add(M::mul(-r0, rn.nx), M::mul(-r1, rn.ny)));
  double pc, pr;
  if (FAST) {
    const double inv = nr_rcp(rr), i2 = inv * inv;
    pc = nc * i2;
    pr = nr * i2;
  } else {
    const double d = M::mul(rr, rr);
    pc = M::div(nc, d);
    pr = M::div(nr, d);
  }
  const double rt = rc ? r1 : r0, n_r = rc ? rn.ny : rn.nx;
  const double pt = M::mul(pc, rt), wt = M::mul(cn.w, n_r);
  e[0] = M::add(M::mul(pt, r0), M::mul(wt, cn.nx));
  e[1] = M::add(M::mul(pt, r1), M::mul(wt, cn.ny));
  e[2] = M::add(M::mul(M::mul(pr, r0), rt), M::mul(M::mul(rn.w, cn.nx), n_r));
  e[3] = M::add(M::mul(M::mul(pr, r1), rt), M::mul(M::mul(rn.w, cn.ny), n_r));
}

// A Laplace or Laplace-Neumann entry for r = target - source, not the diagonal.
template <bool FAST, int PDE>
__device__ __forceinline__ double laplace_off(double r0, double r1, double rr, double inv,
                                              double sw, double sn0, double sn1, double tn0,
                                              double tn1) {
  using M = EM<FAST>;
  const double d = PDE == kLaplace ? M::add(M::mul(r0, sn0), M::mul(r1, sn1))
                                   : M::add(M::mul(r0, tn0), M::mul(r1, tn1));
  const double num = M::mul(M::mul(PDE == kLaplace ? -sw : sw, KI_INV_2PI), d);
  const double q = FAST ? num * inv : M::div(num, rr);
  return PDE == kLaplace ? q : M::add(sw, q);
}

// One column dof (component cc): e0 = K(row, col), e1 = K(col, row).
template <bool FAST, int PDE>
__device__ __forceinline__ void near1(const Node& rn, int rdof, const Node& cn, int cdof,
                                      double* e) {
  using M = EM<FAST>;
  if constexpr (PDE != kStokes) {
    const double r0 = M::sub(rn.x, cn.x), r1 = M::sub(rn.y, cn.y);
    const double rr = M::add(M::mul(r0, r0), M::mul(r1, r1));
    const double inv = FAST ? nr_rcp(rr) : 0.0;
    e[0] = laplace_off<FAST, PDE>(r0, r1, rr, inv, cn.w, cn.nx, cn.ny, rn.nx, rn.ny);
    e[1] = laplace_off<FAST, PDE>(-r0, -r1, rr, inv, rn.w, rn.nx, rn.ny, cn.nx, cn.ny);
    return;
  }
  const int rc = rdof & 1, cc = cdof & 1;
  const double r0 = M::sub(rn.x, cn.x), r1 = M::sub(rn.y, cn.y);
  const double rr = M::add(M::mul(r0, r0), M::mul(r1, r1));
  const double nc = M::mul(M::mul(cn.w, KI_INV_PI), M::add(M::mul(r0, cn.nx), M::mul(r1, cn.ny)));
  const double nr =
      M::mul(M::mul(rn.w, KI_INV_PI), M::add(M::mul(-r0, rn.nx), M::mul(-r1, rn.ny)));
  double pc, pr;
  if (FAST) {
    const double inv = nr_rcp(rr), i2 = inv * inv;
    pc = nc * i2;
    pr = nr * i2;
  } else {
    const double d = M::mul(rr, rr);
    pc = M::div(nc, d);
    pr = M::div(nr, d);
  }
  const double rt = rc ? r1 : r0, rs = cc ? r1 : r0;
  const double n_r = rc ? rn.ny : rn.nx, n_c = cc ? cn.ny : cn.nx;
  e[0] = M::add(M::mul(M::mul(pc, rt), rs), M::mul(M::mul(cn.w, n_r), n_c));
  e[1] = M::add(M::mul(M::mul(pr, rs), rt), M::mul(M::mul(rn.w, n_c), n_r));
}

// A proxy point (px, py) with direction (tn0, tn1), component pc, weight pw:
// as target (e0, e1 for the node's dofs) and as source (e2, e3).
template <bool FAST>
__device__ __forceinline__ void stokes_proxy2(double px, double py, double tn0, double tn1, int pc,
                                              double pw, const Node& cn, double* e) {
  using M = EM<FAST>;
  const double r0 = M::sub(px, cn.x), r1 = M::sub(py, cn.y);
  const double rr = M::add(M::mul(r0, r0), M::mul(r1, r1));
  const double n1 = M::mul(M::mul(cn.w, KI_INV_PI), M::add(M::mul(r0, cn.nx), M::mul(r1, cn.ny)));
  const double n2 = M::mul(M::mul(-pw, KI_INV_PI), M::add(M::mul(r0, tn0), M::mul(r1, tn1)));
  double p1, p2;
  if (FAST) {
    const double inv = nr_rcp(rr), i2 = inv * inv;
    p1 = n1 * i2;
    p2 = n2 * i2;
  } else {
    const double d = M::mul(rr, rr);
    p1 = M::div(n1, d);
    p2 = M::div(n2, d);
  }
  const double rc = pc ? r1 : r0, tnc = pc ? tn1 : tn0;
  const double a = M::mul(p1, rc), wt = M::mul(cn.w, tnc), b = M::mul(p2, rc);
  e[0] = M::add(M::mul(a, r0), M::mul(wt, cn.nx));
  e[1] = M::add(M::mul(a, r1), M::mul(wt, cn.ny));
  e[2] = M::add(M::mul(b, r0), M::mul(M::mul(pw, cn.nx), tnc));
  e[3] = M::add(M::mul(b, r1), M::mul(M::mul(pw, cn.ny), tnc));
}

// One column dof: e0 the proxy point as target, e1 as source.
template <bool FAST, int PDE>
__device__ __forceinline__ void proxy1(double px, double py, double tn0, double tn1,
                                       int pc, double pw, const Node& cn, int cdof, double* e) {
  using M = EM<FAST>;
  const double r0 = M::sub(px, cn.x), r1 = M::sub(py, cn.y);
  if constexpr (PDE != kStokes) {
    const double rr = M::add(M::mul(r0, r0), M::mul(r1, r1));
    const double inv = FAST ? nr_rcp(rr) : 0.0;
    e[0] = laplace_off<FAST, PDE>(r0, r1, rr, inv, cn.w, cn.nx, cn.ny, tn0, tn1);
    e[1] = laplace_off<FAST, PDE>(-r0, -r1, rr, inv, pw, tn0, tn1, cn.nx, cn.ny);
    return;
  }
  const double rr = M::add(M::mul(r0, r0), M::mul(r1, r1));
  const double n1 = M::mul(M::mul(cn.w, KI_INV_PI), M::add(M::mul(r0, cn.nx), M::mul(r1, cn.ny)));
  const double n2 = M::mul(M::mul(-pw, KI_INV_PI), M::add(M::mul(r0, tn0), M::mul(r1, tn1)));
  double p1, p2;
  if (FAST) {
    const double inv = nr_rcp(rr), i2 = inv * inv;
    p1 = n1 * i2;
    p2 = n2 * i2;
  } else {
    const double d = M::mul(rr, rr);
    p1 = M::div(n1, d);
    p2 = M::div(n2, d);
  }
  const double rc = pc ? r1 : r0, tnc = pc ? tn1 : tn0;
  const double rs = (cdof & 1) ? r1 : r0, sns = (cdof & 1) ? cn.ny : cn.nx;
  e[0] = M::add(M::mul(M::mul(p1, rc), rs), M::mul(M::mul(cn.w, tnc), sns));
  e[1] = M::add(M::mul(M::mul(p2, rc), rs), M::mul(M::mul(pw, sns), tnc));
}

// Generates one CTA's share of a box's ID matrix, or of its row sketch (SK),
// into colp(t)[local row].  Near rows and proxy points are dealt to the
// CTAs round-robin, a CTA's rows in four runs: its near rows as targets, the
// same as sources (oc_near(I, G) rows each), its proxy points as targets, as
// sources; the order of rows changes neither the pivots nor T.  Rows past a
// run's and past the last up to the stride ldl are zero.  SK: Y = S A, every
// 32 rows of a run landing on a run of consecutive sketch rows (mod mg, the
// CTA's own) from a hashed start, each row with a hashed sign: a sparse sign
// embedding whose lanes meet only when the run wraps past mg < 32 rows, where
// they take turns; a column is only touched by its warp, so the result is
// deterministic.  ex: scratch for the columns' node records (9 n + 2
// doubles, 16-byte aligned); si[3], si[4]: scratch.  Ends without a barrier.
template <bool SK, int NW, class ColFn>
__device__ __forceinline__ void oc_generate(const IdParams& P, const IdTask& tk, int mg, int ldl,
                                            int g, int G, double* ex, int* si, ColFn colp) {
  const int n = tk.n, I = tk.n_row, pde = P.pde;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int* act = P.act + tk.act_off;
  const int* rowd = P.rowdofs + tk.row_off;
  const Node* nodes = P.nodes;
  const int sh = pde == kStokes ? 1 : 0;
  Node* cn = reinterpret_cast<Node*>(ex);  // the columns' node records, dofs, work units
  int* cdof = reinterpret_cast<int*>(cn + n);
  int* unit = cdof + n;  // first columns of the work units
  const int Ic = (I + G - 1) / G, Ig = (I - g + G - 1) / G;  // near rows of a CTA, of this one
  const int Pg = tk.proxy / (2 * G);                         // proxy rows (of each kind)
  const int nb = (Ig + 31) / 32, pb = (Pg + 31) / 32;        // 32-row blocks of one kind
  for (int t = threadIdx.x; t < n; t += 32 * NW) {
    const int cd = act[t];
    cdof[t] = cd;
    cn[t] = nodes[cd >> sh];
  }
  if (SK) {
    for (int t = warp; t < n; t += NW)
      for (int r = lane; r < ldl; r += 32) colp(t)[r] = 0.0;
  } else {
    for (int t = threadIdx.x; t < n; t += 32 * NW) {
      double* col = colp(t);
      for (int r = Ig; r < Ic; r++) col[r] = col[Ic + r] = 0.0;
      for (int r = mg; r < ldl; r++) col[r] = 0.0;
    }
  }
  __syncthreads();
  // work units: the columns that are the two dofs of one Stokes node, first,
  // then the others
  if (warp == 0) {
    int cnt = 0;
    for (int pass = 0; pass < 2; pass++) {
      for (int base = 0; base < n; base += 32) {
        const int t = base + lane;
        bool start = t < n, two = false;
        if (start && pde == kStokes) {
          const int cd = cdof[t];
          start = !((cd & 1) && t > 0 && cdof[t - 1] == cd - 1);
          two = !(cd & 1) && t + 1 < n && cdof[t + 1] == cd + 1;
        }
        start = start && two == (pass == 0);
        const unsigned bal = __ballot_sync(0xffffffffu, start);
        if (start) unit[cnt + __popc(bal & ((1u << lane) - 1u))] = t;
        cnt += __popc(bal);
      }
      if (lane == 0) si[3 + pass] = cnt;
    }
  }
  __syncthreads();
  const int npair = si[3], nunits = si[4];
  // blocks [0, nb): near rows, [nb, nb + pb): proxy points; a sketched
  // column belongs to one warp, an exact block's columns are split so that
  // every warp has work
  const int nblk = nb + pb;
  const int nch = SK ? NW : nblk >= NW ? 1 : min(nunits, (NW + nblk - 1) / max(nblk, 1));
  const int jobs = SK ? NW * nblk : nblk * nch;
  // a block's row record: its index and node are two dependent loads from
  // global memory, so the next block's are on their way during this one
  auto row_dof = [&](int w) -> int {
    const int q = 32 * (SK ? w / NW : w % max(nblk, 1)) + lane;
    return w < jobs && q < Ig && q < 32 * nb ? rowd[g + G * q] : 0;
  };
  int next_dof = row_dof(warp);
  Node next_row = nodes[next_dof >> sh];
  for (int w = warp; w < jobs; w += NW) {
    const int blk = SK ? w / NW : w % nblk;
    const int u0 = SK ? warp : (w / nblk) * nunits / nch;
    const int u1 = SK ? nunits : (w / nblk + 1) * nunits / nch;
    const bool near = blk < nb;
    const int q = 32 * (near ? blk : blk - nb) + lane;  // this lane's row of the CTA's
    const bool valid = q < (near ? Ig : Pg);
    const Node rn = next_row;
    const int rdof = next_dof;
    next_dof = row_dof(w + NW);
    next_row = nodes[next_dof >> sh];
    int pc = 0;
    double px = 0, py = 0, tn0 = 0, tn1 = 0;
    if (!near) {
      // proxy rows of one kind: point (row >> sh), component row & 1
      const int row = g + G * q, pt = (pde == kStokes ? row >> 1 : row) << (SK ? tk.pshift : 0);
      pc = row & 1;
      if (valid) {
        tn0 = P.proxy_dir[pt];
        tn1 = P.proxy_dir[kNumProxy + pt];
        px = EM<SK>::add(tk.cx, EM<SK>::mul(tk.rad, tn0));
        py = EM<SK>::add(tk.cy, EM<SK>::mul(tk.rad, tn1));
      }
    }
    int i0, i1;  // rows of the slab for the two kinds
    double s0 = 1.0, s1 = 1.0;
    if (SK) {
      const unsigned h = static_cast<unsigned>(2 * blk);
      i0 = (static_cast<int>(sketch_hash(h ^ 0x9e3779b9u) % static_cast<unsigned>(mg)) + lane) % mg;
      i1 = (static_cast<int>(sketch_hash((h + 1) ^ 0x9e3779b9u) % static_cast<unsigned>(mg)) +
            lane) % mg;
      const unsigned id = (static_cast<unsigned>(g) << 20) + 64u * blk + lane;
      s0 = (sketch_hash(id) & 0x80000000u) ? -1.0 : 1.0;
      s1 = (sketch_hash(id + 32u) & 0x80000000u) ? -1.0 : 1.0;
    } else {
      i0 = near ? q : 2 * Ic + q;
      i1 = near ? Ic + q : 2 * Ic + Pg + q;
    }
    // K units at a time (independent chains of about 300 cycles each: with
    // 8 or 16 warps an SM one at a time waits on latency), TWO columns each
    constexpr int step = SK ? NW : 1;
    auto units = [&](auto kc, auto twoc, auto pdec, auto nearc, int u, int end) {
      constexpr int K = decltype(kc)::value, NE = decltype(twoc)::value ? 4 : 2;
      constexpr int PDE = decltype(pdec)::value;
      constexpr bool NEAR = decltype(nearc)::value;
      double e[K][NE];
      double* col[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int t = unit[u + step * k < end ? u + step * k : u];  // (a repeat is not stored)
        col[k] = colp(t);
        const Node& c = cn[t];
        if constexpr (NE == 4 && NEAR) {
          stokes_near2<SK>(rn, rdof & 1, c, e[k]);
        } else if constexpr (NE == 4) {
          stokes_proxy2<SK>(px, py, tn0, tn1, pc, tk.pw, c, e[k]);
        } else if constexpr (NEAR) {
          near1<SK, PDE>(rn, rdof, c, cdof[t], e[k]);
        } else {
          proxy1<SK, PDE>(px, py, tn0, tn1, pc, tk.pw, c, cdof[t], e[k]);
        }
      }
      // (the second column of a pair: the next one, not spilled apart)
      if constexpr (SK) {
        for (int l0 = 0; l0 < 32; l0 += mg) {
          const bool turn = valid && lane >= l0 && lane < l0 + mg;
#pragma unroll
          for (int half = 0; half < 2; half++) {
            const int at = half ? i1 : i0;
            const double sg = half ? s1 : s0;
            if (turn) {
#pragma unroll
              for (int k = 0; k < K; k++) {
                if (u + step * k >= end) break;
                col[k][at] = fma(sg, e[k][half * NE / 2], col[k][at]);
                if (NE == 4) col[k][ldl + at] = fma(sg, e[k][half * NE / 2 + 1], col[k][ldl + at]);
              }
            }
            __syncwarp();
          }
        }
      } else if (valid) {
#pragma unroll
        for (int k = 0; k < K; k++) {
          if (u + step * k >= end) break;
          col[k][i0] = e[k][0];
          col[k][i1] = e[k][NE / 2];
          if (NE == 4) {
            double* col1 = colp(unit[u + step * k] + 1);
            col1[i0] = e[k][1];
            col1[i1] = e[k][3];
          }
        }
      }
    };
    auto columns = [&](auto pdec, auto nearc) {
      const int up = min(u1, npair);
      int u = u0;
      if constexpr (decltype(pdec)::value == kStokes) {
        for (; u < up; u += 2 * step)
          units(std::integral_constant<int, 2>{}, std::true_type{}, pdec, nearc, u, up);
        // (this warp's first single-column unit)
        u = u0 < npair ? u0 + (npair - u0 + step - 1) / step * step : u0;
      }
      for (; u < u1; u += 4 * step)
        units(std::integral_constant<int, 4>{}, std::false_type{}, pdec, nearc, u, u1);
    };
    auto rows = [&](auto pdec) {
      if (near) {
        columns(pdec, std::true_type{});
      } else {
        columns(pdec, std::false_type{});
      }
    };
    if (pde == kStokes) {
      rows(std::integral_constant<int, kStokes>{});
    } else if (pde == kLaplace) {
      rows(std::integral_constant<int, kLaplace>{});
    } else {
      rows(std::integral_constant<int, kLaplaceNeumann>{});
    }
  }
}

// ------------------------------------------------------------ layout
// Doubles and ints of one CTA's shared memory, the same in every CTA of the
// cluster (peers write into each other's sums at the same offsets):
//   slab   nres x ldl   this CTA's rows of the resident columns
//   cb     2 x ldl      pivot column of this step and of the last (unscaled)
//   ex     partial sums from every CTA (two steps' worth when G > 1), row i
//          of the matrix from its owner; the generation's column records
//          before that
//   rdiag, tws, vn1, vn2, slot keys, ints
constexpr int kNormWindow = 4;  // columns whose norm a step sums afresh: one unit in four

__host__ __device__ inline int oc_rows(int m, int G) { return (m + G - 1) / G; }
// Column stride: even (16-byte loads of row pairs) and 2 mod 4, so the
// threads that read one row across columns meet two to a bank at worst (a
// multiple of 16 doubles would put them all on one).
__host__ __device__ inline int oc_stride(int m, int G) {
  const int r = (oc_rows(m, G) + 1) & ~1;
  return r % 4 ? r : r + 2;
}
// R's rows in the workspace, an even count: the spilled columns behind them
// are read as 16-byte pairs, and so is the next box's share.
__host__ __device__ inline long long oc_rows_doubles(int mn, int n) {
  return (static_cast<long long>(mn) * n + 1) & ~1LL;
}
__host__ __device__ inline int oc_part(int n) { return (n + n / kNormWindow + 9) & ~1; }
__host__ __device__ inline size_t oc_ex_doubles(int n, int G) {
  const size_t ne = (static_cast<size_t>(n) + 1) & ~static_cast<size_t>(1);
  const size_t ex = G > 1 ? static_cast<size_t>(2 * G + 1) * oc_part(n) + 3 * ne : oc_part(n);
  const size_t gen = 9 * static_cast<size_t>(n) + 2;  // a Node and two ints per column
  return ((ex > gen ? ex : gen) + 1) & ~static_cast<size_t>(1);
}
__host__ __device__ inline size_t oc_fixed_bytes(int m, int n, int G) {
  const int mn = m < n ? m : n;
  return sizeof(double) * (2 * static_cast<size_t>(oc_stride(m, G)) + oc_ex_doubles(n, G) + mn +
                           3 * static_cast<size_t>(n) + kOcWarps + 4) +
         sizeof(int) * (5 * static_cast<size_t>(n) + kOcWarps + 8);
}

__device__ __forceinline__ double oc_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One unit of the pass of step i: C columns by L lanes (lane gl of the
// group takes rows r0 + 2 gl, + 2 L, ...).  Column u: x <- x - tw[u] cp (the
// last reflector), S[u] += x c with c = ap - twp cp the new pivot column
// below row i (rows from lo on; 0 above), and with NORM N[u] += x^2 over the
// same rows.  The result goes to dst (col, but for a column that moves).
template <int L, int C, bool NORM>
__device__ __forceinline__ void oc_pass(double* const (&col)[C], double* const (&dst)[C],
                                        const double (&tw)[C],
                                        const bool (&on)[C], const double* cprev,
                                        const double* ap, double twp, int r0, int lo, int mend,
                                        int gl, double (&S)[C], double (&N)[C]) {
#pragma unroll
  for (int u = 0; u < C; u++) S[u] = N[u] = 0.0;
#pragma unroll 2
  for (int r = r0 + 2 * gl; r < mend; r += 2 * L) {
    const double2 cp = *reinterpret_cast<const double2*>(cprev + r);
    const double2 av = *reinterpret_cast<const double2*>(ap + r);
    const double c0 = r >= lo ? fma(-twp, cp.x, av.x) : 0.0;
    const double c1 = r + 1 >= lo ? fma(-twp, cp.y, av.y) : 0.0;
    double2 x[C];
#pragma unroll
    for (int u = 0; u < C; u++)
      if (on[u]) x[u] = *reinterpret_cast<const double2*>(col[u] + r);
#pragma unroll
    for (int u = 0; u < C; u++)
      if (on[u]) {
        x[u].x = fma(-tw[u], cp.x, x[u].x);
        x[u].y = fma(-tw[u], cp.y, x[u].y);
        *reinterpret_cast<double2*>(dst[u] + r) = x[u];
        S[u] = fma(x[u].x, c0, S[u]);
        S[u] = fma(x[u].y, c1, S[u]);
        if (NORM) {
          if (r >= lo) N[u] = fma(x[u].x, x[u].x, N[u]);
          if (r + 1 >= lo) N[u] = fma(x[u].y, x[u].y, N[u]);
        }
      }
  }
}

// Sums C values per lane over the L lanes of a group, halving the values
// with the lanes: afterwards lane gl holds the total of value (gl / (L /
// C)), i.e. L / C lanes hold each.
template <int L, int C>
__device__ __forceinline__ double oc_group_sum(const double (&v)[C], int gl) {
  if constexpr (C == 1) {
    double t = v[0];
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  } else {
    double h[C / 2];
    const bool up = (gl & (L / 2)) != 0;
#pragma unroll
    for (int u = 0; u < C / 2; u++) {
      const double keep = up ? v[u + C / 2] : v[u];
      const double send = up ? v[u] : v[u + C / 2];
      h[u] = keep + __shfl_xor_sync(0xffffffffu, send, L / 2);
    }
    return oc_group_sum<L / 2, C / 2>(h, gl);
  }
}

// T = R11^{-1} R12 by the CTA, dtrsm's column sweep, CT redundant columns at
// a time in a warp's registers (lane l holding rows l, l + 32, ... of up to
// 32 KR), so one load of R11's column serves CT of them and their shuffles
// overlap.  Redundant columns are dealt to the CTAs, then the warps.  rcp:
// the reciprocals of R's diagonal; rcol(q): column q of R11 (rows < q); R(l,
// j): row l of R in matrix column j.
template <int KR, int CT, int NW, class ColFn, class RowFn>
__device__ __forceinline__ void oc_tsolve_regs(int k, int n, int g, int G, const int* pos2col,
                                               const double* rcp, double* T, ColFn rcol, RowFn R) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mine = (n - k - g + G - 1) / G;  // this CTA's redundant columns
  for (int c0 = warp * CT; c0 < mine; c0 += NW * CT) {
    double x[CT][KR];
#pragma unroll
    for (int c = 0; c < CT; c++) {
      const int j = pos2col[k + g + G * min(c0 + c, mine - 1)];
#pragma unroll
      for (int u = 0; u < KR; u++) {
        const int l = lane + 32 * u;
        x[c][u] = l < k ? R(l, j) : 0.0;
      }
    }
    // rows q in [32 u, 32 u + 32) sit in slot u: the slot loop outside
    // (unrolled), so every register index is a constant
#pragma unroll
    for (int u = KR - 1; u >= 0; u--) {
#pragma unroll 2
      for (int q = min(k, 32 * u + 32) - 1; q >= 32 * u; q--) {
        const double* rq = rcol(q);
        const double rc = rcp[q];
        double r[KR];
#pragma unroll
        for (int v = 0; v <= u; v++) r[v] = lane + 32 * v < q ? rq[lane + 32 * v] : 0.0;
#pragma unroll
        for (int c = 0; c < CT; c++) {
          const double xq = __shfl_sync(0xffffffffu, x[c][u], q & 31) * rc;
#pragma unroll
          for (int v = 0; v <= u; v++) x[c][v] = fma(-xq, r[v], x[c][v]);
          if (lane == (q & 31)) x[c][u] = xq;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < CT; c++)
      if (c0 + c < mine) {
        double* Tp = T + static_cast<long long>(g + G * (c0 + c)) * k;
#pragma unroll
        for (int u = 0; u < KR; u++) {
          const int l = lane + 32 * u;
          if (l < k) Tp[l] = x[c][u];
        }
      }
  }
}

// ... by rank; ranks past 256, and an R11 without rcol (fast false), sweep in
// the output itself.
template <int NW, class ColFn, class RowFn>
__device__ __forceinline__ void oc_tsolve(int k, int n, int g, int G, const int* pos2col,
                                          const double* rcp, double* T, bool fast, ColFn rcol,
                                          RowFn R) {
  if (fast && k <= 32) return oc_tsolve_regs<1, 4, NW>(k, n, g, G, pos2col, rcp, T, rcol, R);
  if (fast && k <= 64) return oc_tsolve_regs<2, 4, NW>(k, n, g, G, pos2col, rcp, T, rcol, R);
  if (fast && k <= 128) return oc_tsolve_regs<4, 2, NW>(k, n, g, G, pos2col, rcp, T, rcol, R);
  if (fast && k <= 256) return oc_tsolve_regs<8, 1, NW>(k, n, g, G, pos2col, rcp, T, rcol, R);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q0 = k + g + G * warp; q0 < n; q0 += G * NW) {
    const int j = pos2col[q0];
    double* Tp = T + static_cast<long long>(q0 - k) * k;
    for (int l = lane; l < k; l += 32) Tp[l] = R(l, j);
    __syncwarp();
    for (int q = k - 1; q >= 0; q--) {
      const double bq = Tp[q];
      __syncwarp();
      const double xq = bq * rcp[q];
      const int jq = pos2col[q];
      if (lane == 0) Tp[q] = xq;
      for (int l = lane; l < q; l += 32) Tp[l] -= xq * R(l, jq);
      __syncwarp();
    }
  }
}

// Pivot key of a squared partial norm; 0 when it is not a positive number.
// Norms that rounding cannot tell apart count as equal, so the first of
// them is taken as LAPACK takes the first of equal ones: a column's entries
// err by about eps |A|, its squared norm relatively by 2 eps |A| / norm, so
// the key drops 4 bits plus half the bits the squared norm has lost since
// the start (e0: exponent of the largest): columns whose squares differ by
// less than 4e-15, late in a box at id_tol 1e-10 by less than 3e-5, both
// about 16 times their rounding error.  Tied columns are then usually, not
// always, taken by position: two on either side of a step of the key are
// not.  Against the CPU restatement of LAPACK's steps, 24 eight-hole Stokes
// domains (16,384 dofs, 13,272 boxes, id_tol 1e-10): 30 boxes in 5 domains
// differ, with the exact comparison 33 in 4 (equally spaced nodes on the
// holes tie); ellipses and stars (6,957 boxes): none by either.  Sketched
// boxes, and id_kernel with its boxes past shared memory, compare exactly.
__device__ __forceinline__ unsigned long long oc_cand_key(double v, int e0, bool sketched) {
  if (!(v > 0.0)) return 0ull;
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  if (sketched) return u;
  const int sh = min(46, 4 + max(0, (e0 - static_cast<int>(u >> 52)) >> 1));
  return (u + (1ull << (sh - 1))) >> sh << sh;
}

// ------------------------------------------------------ register tiles
// The pivoted QR with the matrix in registers: warp w of a CTA's NW owns the
// columns j % NW == w, its lanes the CTA's rows (local row lane + 32 s in
// slot s), so a thread holds CW x RS entries for the whole factorization
// and a pivot step moves only the pivot column through shared memory.  A step:
//   1. every warp: products of its columns with the pivot column c (rows
//      > i), |c|^2 and the norms of a quarter of its columns, in one warp
//      sum; G > 1: these partial sums to every CTA, one cluster barrier;
//   2. every warp: the reflector u = [alpha - beta; c] from the same sums in
//      the same order, its columns' update x -= u (u.x) / (beta (beta -
//      alpha)), norms, candidate for the next pivot; a CTA barrier;
//   3. the owner warp writes the next pivot column; a CTA barrier.
// What bounds a step is its chain (warp sums, a square root, a division, two
// barriers) and, for the larger tiles, instruction issue; few warps with
// many columns each keep the per-warp part of that small.
// Against the former slab in shared memory with columns dealt to the CTAs:
// 602 x 48, 8 boxes, 167 us -> 82 us; 976 x 58, 10 boxes, 262 us -> 121 us;
// 384 x 81, 311 us -> 181 us.
template <int V>
struct TileSum {  // warp sums of V values: lane holds the total of value lane / H
  static constexpr int P2 = V <= 1 ? 1 : V <= 2 ? 2 : V <= 4 ? 4 : V <= 8 ? 8 : V <= 16 ? 16 : 32;
  static constexpr int H = 32 / P2;
  static __device__ __forceinline__ double sum(const double (&v)[V]) {
    double w[P2];
#pragma unroll
    for (int u = 0; u < P2; u++) w[u] = u < V ? v[u] : 0.0;
    return oc_group_sum<32, P2>(w, threadIdx.x & 31);
  }
};

// One CTA's sums of a step: a product per column, the window's norms, |c|^2
// (an even count: copied in 16-byte pairs).
__host__ __device__ inline int tile_part(int n, int NW, int CW) {
  return (n + (CW + kNormWindow - 1) / kNormWindow * NW + 2) & ~1;
}
// The exchange area: this CTA's sums and row i, every CTA's for two steps.
__host__ __device__ inline size_t tile_ex_doubles(int n, int G, int NW, int CW) {
  const size_t ne = (static_cast<size_t>(n) + 1) & ~static_cast<size_t>(1);
  const size_t ex = G > 1 ? (2 * static_cast<size_t>(G) + 1) * tile_part(n, NW, CW) + 3 * ne : 0;
  const size_t gen = 9 * static_cast<size_t>(n) + 2;
  return ((ex > gen ? ex : gen) + 1) & ~static_cast<size_t>(1);
}
// Shared memory of a tile CTA: the generated slab (later R's rows), the
// pivot column, the exchange area, per-warp scratch, rdiag, reciprocals,
// keys, ints.
__host__ __device__ inline size_t tile_smem_bytes(int m, int n, int G, int NW, int CW, int RS) {
  return sizeof(double) * (static_cast<size_t>(n) * oc_stride(m, G) + 32 * RS +
                           tile_ex_doubles(n, G, NW, CW) + 2 * NW * CW + 2 * n + NW + 4) +
         sizeof(int) * (2 * static_cast<size_t>(n) + NW + 8);
}

template <int NW, int CW, int RS, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) id_tile_kernel(IdParams P, int lg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G = 1 << lg;  // CTAs of the cluster
  const int task = blockIdx.x >> lg;
  const int g = blockIdx.x & (G - 1);  // (a cluster's blocks are consecutive)
  const IdTask tk = P.tasks[task];
  const bool sk = tk.sk > 0;
  const int n = tk.n;
  const int m = sk ? tk.sk : id_padded_rows(tk.n_row, tk.proxy, G);  // rows over the cluster
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mn = min(sk ? m : tk.m, n), ldl = oc_stride(m, G);
  const int mg = (m - g + G - 1) >> lg;  // this CTA's rows
  const int ps = tile_part(n, NW, CW);
  constexpr int NS = (CW + kNormWindow - 1) / kNormWindow;
  using Sum = TileSum<CW + NS + 1>;
  constexpr int H = Sum::H;

  double* slab = reinterpret_cast<double*>(smem_raw);
  double* cs = slab + static_cast<size_t>(n) * ldl;  // 32 RS: pivot column, rows > i
  double* ex = cs + 32 * RS;
  double* part = ex;                       // G > 1: [2][G][ps]
  double* loc = ex + 2 * G * ps;           // this CTA's, ps
  double* rowi = loc + ps;                 // [2][ne] row i, then this CTA's copy
  const int ne = (n + 1) & ~1;
  double* loci = rowi + 2 * ne;
  double* wa = ex + tile_ex_doubles(n, G, NW, CW) + warp * 2 * CW;  // the warp's row i
  double* wc = wa + CW;                                             // ... coefficients
  double* rdiag = ex + tile_ex_doubles(n, G, NW, CW) + 2 * NW * CW;  // n
  double* rcp = rdiag + n;                                           // n
  unsigned long long* skey = reinterpret_cast<unsigned long long*>(rcp + n);  // NW
  double* hh = reinterpret_cast<double*>(skey + NW);  // [0] alpha (G = 1), [1] |tol R_00|
  int* sidx = reinterpret_cast<int*>(hh + 4);         // NW
  int* si = sidx + NW;  // [2] rank once found, [3, 4] units, [5] last step with a lost norm + 1
  int* pos2col = si + 8;                              // n
  int* col2pos = pos2col + n;                         // n
  double* Rg = P.work + tk.a_off;                     // G > 1: R's columns, [n][mn]
  auto barrier = [&]() {
    if (G > 1) {
      cg::this_cluster().sync();
    } else {
      __syncthreads();
    }
  };

  for (int t = threadIdx.x; t < n; t += 32 * NW) pos2col[t] = col2pos[t] = t;
  if (threadIdx.x == 0) si[2] = si[5] = 0;
  {
    auto colp = [&](int j) -> double* { return slab + static_cast<size_t>(j) * ldl; };
    if (sk) {
      oc_generate<true, NW>(P, tk, mg, ldl, g, G, ex, si, colp);
    } else {
      oc_generate<false, NW>(P, tk, mg, ldl, g, G, ex, si, colp);
    }
  }
  barrier();  // (every CTA done with its column records: the sums take their place)

  // the warp's columns u NW + warp into registers
  double x[CW][RS];
#pragma unroll
  for (int u = 0; u < CW; u++) {
    const int j = u * NW + warp;
#pragma unroll
    for (int s = 0; s < RS; s++) {
      const int lr = lane + 32 * s;
      x[u][s] = j < n && lr < mg ? slab[static_cast<size_t>(j) * ldl + lr] : 0.0;
    }
  }
  // this lane's column in the per-column work of the warp
  const int v = lane / H, sub = lane & (H - 1);
  const int jv = v < CW ? v * NW + warp : n;
  bool live = jv < n;           // a column, not yet a pivot
  double vn1 = 0.0, vn2 = 0.0;  // its squared partial norm, ... when last summed

  auto publish = [&](unsigned long long key, int idx) {
    unsigned long long wk;
    int wi;
    warp_argmax_bits(key, idx, &wk, &wi);
    if (lane == 0) {
      skey[warp] = wk;
      sidx[warp] = wi;
    }
  };
  auto chosen = [&]() -> int {
    unsigned long long wk;
    int wi;
    warp_argmax_bits(lane < NW ? skey[lane] : 0ull, lane < NW ? sidx[lane] : 0x7fffffff, &wk, &wi);
    return wi;
  };
  int e0 = 0;
  auto candidate = [&]() {
    publish(live ? oc_cand_key(vn1, e0, sk) : 0ull,
            live ? col2pos[jv] << 16 | jv : 0x7fffffff);
  };
  // the sums W of this CTA's rows (and its row i, where it owns it) to every
  // CTA's part b; a cluster barrier
  auto exchange = [&](double t, int b, bool row) {
    if (v < CW) {
      if (jv < n && sub == 0) loc[jv] = t;
    } else if (v < CW + NS) {
      if (sub == 0) loc[n + (v - CW) * NW + warp] = t;
    } else if (v == CW + NS && warp == 0 && sub == 0) {
      loc[n + NS * NW] = t;
    }
    if (row && lane < CW && lane * NW + warp < n) loci[lane * NW + warp] = wa[lane];
    __syncthreads();
    const double2* src = reinterpret_cast<const double2*>(loc);
    for (int gg = warp; gg < G; gg += NW) {
      double2* dst = reinterpret_cast<double2*>(
          cg::this_cluster().map_shared_rank(part + (b * G + g) * ps, gg));
      for (int e = lane; 2 * e < ps; e += 32) dst[e] = src[e];
      if (row) {
        double2* rd =
            reinterpret_cast<double2*>(cg::this_cluster().map_shared_rank(rowi + b * ne, gg));
        for (int e = lane; 2 * e < ne; e += 32) rd[e] = reinterpret_cast<const double2*>(loci)[e];
      }
    }
    cg::this_cluster().sync();
  };
  // sum over the CTAs of entry e of their parts, by the H lanes of a column
  auto total = [&](int e, int b) -> double {
    double t = 0.0;
    for (int q = sub; q < G; q += H) t += part[(b * G + q) * ps + e];
#pragma unroll
    for (int o = H / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  };
  // the columns' squared norms over the rows >= lo of this CTA, all CTAs'
  auto norms = [&](int lo, int b) -> double {
    double W[CW + NS + 1];
#pragma unroll
    for (int u = 0; u < CW + NS + 1; u++) W[u] = 0.0;
#pragma unroll
    for (int s = 0; s < RS; s++)
      if (lane + 32 * s >= lo) {
#pragma unroll
        for (int u = 0; u < CW; u++) W[u] = fma(x[u][s], x[u][s], W[u]);
      }
    const double t = Sum::sum(W);
    if (G == 1) return t;
    exchange(t, b, false);
    return total(jv < n ? jv : 0, b);
  };
  vn1 = vn2 = norms(0, 1);
  candidate();
  __syncthreads();
  int pick = chosen();
  e0 = static_cast<int>(
      __reduce_max_sync(0xffffffffu, lane < NW ? static_cast<unsigned>(skey[lane] >> 52) : 0u));

  const double tol3z = sqrt(0.5 * 2.220446049250313e-16);
  int rank = 0;
  for (int i = 0; i < mn; i++) {
    const int b = i & 1;
    const int p = pick & 0xffff, ppos = pick >> 16;
    const bool iown = (i & (G - 1)) == g;
    const int iloc = i >> lg;
    const int lo = (i - g + G) >> lg;  // this CTA's rows <= i
    // ---- 3. the pivot column (of the step's rows > i) by its warp.  (The
    // column is compared, not u, and rows likewise below: knowing u == p / NW
    // the compiler would index the registers by it and spill them all.)
#pragma unroll
    for (int u = 0; u < CW; u++)
      if (u * NW + warp == p) {
#pragma unroll
        for (int s = 0; s < RS; s++) {
          const int lr = lane + 32 * s;
          cs[lr] = lr >= lo ? x[u][s] : 0.0;
          if (G == 1 && lr == i) hh[0] = x[u][s];
        }
      }
    if (threadIdx.x == 32 * ((p + 1) % NW)) {  // (a thread of another warp)
      const int ci = pos2col[i];
      pos2col[i] = p;
      pos2col[ppos] = ci;
      col2pos[ci] = ppos;
      col2pos[p] = i;
    }
    __syncthreads();
    if (jv == p) live = false;

    // ---- 1. products, norms of a quarter of the columns, row i
    double W[CW + NS + 1];
#pragma unroll
    for (int u = 0; u < CW + NS + 1; u++) W[u] = 0.0;
#pragma unroll
    for (int s = 0; s < RS; s++) {
      const double c = cs[lane + 32 * s];
      W[CW + NS] = fma(c, c, W[CW + NS]);
#pragma unroll
      for (int u = 0; u < CW; u++) W[u] = fma(x[u][s], c, W[u]);
    }
#pragma unroll
    for (int w = 0; w < kNormWindow; w++)
      if (w < CW && ((i - w) & (kNormWindow - 1)) == 0) {
#pragma unroll
        for (int s = 0; s < RS; s++)
          if (lane + 32 * s >= lo) {
#pragma unroll
            for (int u = w; u < CW; u += kNormWindow)
              W[CW + u / kNormWindow] = fma(x[u][s], x[u][s], W[CW + u / kNormWindow]);
          }
      }
    if (iown) {
#pragma unroll
      for (int s = 0; s < RS; s++)
        if (lane + 32 * s == iloc) {
#pragma unroll
          for (int u = 0; u < CW; u++) wa[u] = x[u][s];
        }
      __syncwarp();
    }
    double t = Sum::sum(W), a, Nv, xs, alpha;
    if (G > 1) {
      exchange(t, b, iown);
      t = total(jv < n ? jv : 0, b);
      Nv = total(n + (v < CW ? v / kNormWindow : 0) * NW + warp, b);
      xs = 0.0;
      for (int q = 0; q < G; q++) xs += part[(b * G + q) * ps + n + NS * NW];
      a = jv < n ? rowi[b * ne + jv] : 0.0;
      alpha = rowi[b * ne + p];
    } else {
      Nv = __shfl_sync(0xffffffffu, t, (CW + (v < CW ? v / kNormWindow : 0)) * H);
      xs = __shfl_sync(0xffffffffu, t, (CW + NS) * H);
      a = v < CW ? wa[v] : 0.0;
      alpha = hh[0];
    }

    // ---- 2. reflector, update, norms, candidate
    double beta = alpha, amb = 0.0, kappa = 0.0;
    if (xs != 0.0) {
      const double tt = fma(alpha, alpha, xs), rt = sqrt(tt);
      beta = -copysign(rt, alpha);
      amb = alpha - beta;
      kappa = 1.0 / fma(fabs(alpha), rt, tt);  // 1 / (beta (beta - alpha))
    }
    const double coef = live ? fma(amb, a, t) * kappa : 0.0;
    if (v < CW && sub == 0) wc[v] = coef;
    __syncwarp();
    if (threadIdx.x == 0) {
      rdiag[i] = beta;
      if (i == 0) {
        hh[1] = fabs(P.tol * beta);
      } else if (fabs(beta) < hh[1]) {
        si[2] = i;
      }
    }
    {
      double cf[CW];
#pragma unroll
      for (int u = 0; u < CW; u++) cf[u] = wc[u];
#pragma unroll
      for (int s = 0; s < RS; s++) {
        const double c = cs[lane + 32 * s];
#pragma unroll
        for (int u = 0; u < CW; u++) x[u][s] = fma(-cf[u], c, x[u][s]);
      }
    }
    bool flagged = false;
    if (live) {
      // row i of R, and the squared norm below it: dlaqp2's downdate, vn1 (1
      // - (r / vn1)^2)^(1/2) with its test against vn2, in squares; from the
      // window's fresh sum where there is one
      const double r = fma(-coef, amb, a);
      if (sub == 0) {
        if (G == 1) {
          slab[static_cast<size_t>(jv) * ldl + i] = r;
        } else if (iown) {
          Rg[static_cast<long long>(jv) * mn + i] = r;
        }
      }
      double base = vn1;
      if (v % kNormWindow == i % kNormWindow) base = vn2 = fma(a, a, Nv);
      double nv = base;
      if (base != 0.0) {
        nv = fma(-r, r, base);
        flagged = nv <= tol3z * vn2;
      }
      vn1 = nv;
      if (flagged) si[5] = i + 1;
    }
    candidate();
    __syncthreads();
    if (si[2] != 0) {
      rank = si[2];
      break;
    }
    if (i + 1 == mn) break;
    if (si[5] == i + 1) {
      // norms whose downdate lost its accuracy, summed anew; rare, as every
      // column's norm is renewed each fourth step
      const double f = norms(lo, b ^ 1);
      if (flagged) vn1 = vn2 = f;
      __syncthreads();  // (the keys and the mark read by nobody any more)
      candidate();
      barrier();  // (and no peer's next sums before these are read)
    }
    pick = chosen();
  }

  // a sketch shorter than n + 16 rows certifies a rank only well below its
  // row count; otherwise the box is reported (-1) for the full sketch
  if (sk && m < n + 16 && (rank == 0 || rank > m - 16)) rank = -1;
  if (g == 0) {
    if (threadIdx.x == 0) P.rank[task] = rank;
    for (int q = threadIdx.x; q < n; q += 32 * NW) P.perm[tk.perm_off + q] = pos2col[q];
  }
  const int k = rank;
  barrier();  // (R's rows complete; no peer writes here any more)
  if (k <= 0) return;
  // R11's columns: in the slab for G = 1; else gathered, packed, from the
  // workspace
  const bool staged =
      G > 1 && static_cast<size_t>(k) * (k - 1) / 2 <= static_cast<size_t>(rdiag - slab);
  if (staged)
    for (int q = warp; q < k; q += NW) {
      const double* col = Rg + static_cast<long long>(pos2col[q]) * mn;
      for (int l = lane; l < q; l += 32) slab[static_cast<size_t>(q) * (q - 1) / 2 + l] = col[l];
    }
  for (int q = threadIdx.x; q < k; q += 32 * NW) rcp[q] = 1.0 / rdiag[q];
  __syncthreads();
  oc_tsolve<NW>(
      k, n, g, G, pos2col, rcp, P.tout + tk.t_off, G == 1 || staged,
      [&](int q) -> const double* {
        return G > 1 ? slab + static_cast<size_t>(q) * (q - 1) / 2
                     : slab + static_cast<size_t>(pos2col[q]) * ldl;
      },
      [&](int l, int j) -> double {
        return G > 1 ? Rg[static_cast<long long>(j) * mn + l]
                     : slab[static_cast<size_t>(j) * ldl + l];
      });
}

// The tiles: warps, columns of a warp, row slots of a lane (NW CW columns, 32
// RS rows of a CTA), CTAs that share an SM.  A box takes the one with the
// fewest entries that holds it.
struct TileShape {
  int nw, cw, rs, minb;
};
constexpr TileShape kTiles[] = {{8, 8, 2, 3}, {8, 16, 2, 2}, {8, 4, 8, 2},  {8, 8, 4, 2},
                                {16, 8, 3, 1}, {16, 8, 5, 1}, {8, 4, 18, 1}, {8, 8, 9, 1},
                                {16, 12, 3, 1}, {16, 20, 2, 1}};
constexpr int kNumTiles = sizeof(kTiles) / sizeof(kTiles[0]);

template <int T>
cudaError_t launch_tile(const IdParams& p, int G, cudaStream_t s) {
  constexpr TileShape ts = kTiles[T];
  const size_t smem = static_cast<size_t>(p.onchip_smem);
  if (smem == 0 || smem > 227 * 1024) return cudaErrorInvalidValue;
  const void* fn = reinterpret_cast<const void*>(&id_tile_kernel<ts.nw, ts.cw, ts.rs, ts.minb>);
  cudaError_t e = raise_func_attr(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  if (G > 8) {
    e = raise_func_attr(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G * p.ntasks);
  cfg.blockDim = dim3(32 * ts.nw);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = G;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = G > 1 ? 1 : 0;
  int lg = 0;
  while ((1 << lg) < G) lg++;
  return cudaLaunchKernelEx(&cfg, id_tile_kernel<ts.nw, ts.cw, ts.rs, ts.minb>, p, lg);
}

template <int T = 0>
cudaError_t launch_tile_any(int t, const IdParams& p, int G, cudaStream_t s) {
  if constexpr (T < kNumTiles) {
    if (t == T) return launch_tile<T>(p, G, s);
    return launch_tile_any<T + 1>(t, p, G, s);
  }
  return cudaErrorInvalidValue;
}

// SK: the working matrix is the sk x n row sketch of a preconditioner-mode
// box.  SPILL: a box too large for a cluster's shared
// memory keeps its columns from tk.nres on in global memory (L2), each CTA
// its own rows of them.
template <int G, bool SK, bool SPILL>
__global__ void __launch_bounds__(kOcThreads, 1) id_cluster_kernel(IdParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int task = blockIdx.x / G;
  int g = 0;
  if constexpr (G > 1) g = static_cast<int>(cg::this_cluster().block_rank());
  const IdTask tk = P.tasks[task];
  const int n = tk.n;
  const int m = SK ? tk.sk : id_padded_rows(tk.n_row, tk.proxy, G);  // rows over the cluster
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mn = min(SK ? m : tk.m, n), ldl = oc_stride(m, G);
  const int mg = (m - g + G - 1) / G;  // this CTA's rows
  const int mend = (oc_rows(m, G) + 1) & ~1;
  const int nres = SPILL ? tk.nres : n;
  const int ps = oc_part(n);

  double* slab = reinterpret_cast<double*>(smem_raw);
  double* cb = slab + static_cast<size_t>(nres) * ldl;
  double* ex = cb + 2 * ldl;
  const int ne = (n + 1) & ~1;
  double* part = ex;                              // [2][G][ps] (G > 1)
  double* loc = G > 1 ? ex + 2 * G * ps : ex;     // this CTA's sums, ps
  double* rowi = loc + ps;                        // [2][ne] row i, then this CTA's copy (G > 1)
  double* loci = rowi + 2 * ne;
  double* rdiag = ex + oc_ex_doubles(n, G);       // mn
  double* tws = rdiag + mn;                       // n: last reflector's coefficient per column
  double* vn1 = tws + n;                          // n: squared partial norms
  double* vn2 = vn1 + n;                          // n: ... when last summed
  unsigned long long* skey = reinterpret_cast<unsigned long long*>(vn2 + n);  // kOcWarps
  double* hh = reinterpret_cast<double*>(skey + kOcWarps);  // [0] alpha (G = 1), [1] |tol R_00|
  int* sidx = reinterpret_cast<int*>(hh + 4);     // kOcWarps
  int* si = sidx + kOcWarps;  // [2] rank once found, [3] units, [6] next spilled column, [7] slot
  int* pos2col = si + 8;                          // n
  int* col2pos = pos2col + n;                     // n
  int* own = col2pos + n;                         // n: the trailing columns
  int* col2own = own + n;                         // n
  int* slot = col2own + n;                        // n: a column's place (spilled ones past nres)
  // R's rows when they are spread over a cluster, then the spilled columns
  double* Rg = P.work + tk.a_off;                 // [mn][n]
  double* spill = nullptr;
  if constexpr (SPILL)
    spill = Rg + oc_rows_doubles(mn, n) + static_cast<long long>(g) * (n - nres) * ldl;
  auto place = [&](int q) -> double* {
    if constexpr (SPILL) {
      if (q >= nres) return spill + static_cast<long long>(q - nres) * ldl;
    }
    return slab + static_cast<size_t>(q) * ldl;
  };
  // A pivot's place in shared memory is free a step later; the next spilled
  // column moves there as that step's pass updates it, so that the passes
  // through L2 shrink with every step (1400 x 422: 3.57 ms -> 3.39 ms).
  auto colp = [&](int j) -> double* { return place(SPILL ? slot[j] : j); };
  auto barrier = [&]() {
    if constexpr (G > 1) {
      cg::this_cluster().sync();
    } else {
      __syncthreads();
    }
  };
  // this CTA's sums loc (and its row i, loci, where it owns it) to every
  // CTA's part b, row by row in 16-byte stores (scattered 8-byte ones took
  // 2,000 to 6,000 cycles a step), then a cluster barrier; G = 1: loc itself
  auto exchange = [&](int b, bool row) {
    __syncthreads();
    if constexpr (G > 1) {
      const double2* src = reinterpret_cast<const double2*>(loc);
      for (int gg = warp; gg < G; gg += kOcWarps) {
        double2* dst = reinterpret_cast<double2*>(
            cg::this_cluster().map_shared_rank(part + (b * G + g) * ps, gg));
        for (int e = lane; 2 * e < ps; e += 32) dst[e] = src[e];
        if (row) {
          double2* rd =
              reinterpret_cast<double2*>(cg::this_cluster().map_shared_rank(rowi + b * ne, gg));
          for (int e = lane; 2 * e < ne; e += 32) rd[e] = reinterpret_cast<const double2*>(loci)[e];
        }
      }
      cg::this_cluster().sync();
    }
  };
  auto total = [&](int e, int b) -> double {
    if constexpr (G == 1) return loc[e];
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < G; q++) t += part[(b * G + q) * ps + e];
    return t;
  };

  // ---- generation of this CTA's rows of every column
  for (int t = threadIdx.x; t < n; t += kOcThreads) {
    pos2col[t] = col2pos[t] = own[t] = col2own[t] = slot[t] = t;
    tws[t] = 0.0;
  }
  for (int e = threadIdx.x; e < 2 * ldl; e += kOcThreads) cb[e] = 0.0;
  if (threadIdx.x == 0) {
    si[2] = 0;
    si[6] = nres;
    si[7] = -1;
  }
  oc_generate<SK, kOcWarps>(P, tk, mg, ldl, g, G, ex, si, place);
  barrier();  // (every CTA done with its column records: the sums take their place)
  // ---- initial norms
  for (int t = warp; t < n; t += kOcWarps) {
    const double* col = colp(t);
    double ss = 0.0;
    for (int r = 2 * lane; r < mend; r += 64) {
      const double2 x = *reinterpret_cast<const double2*>(col + r);
      ss += x.x * x.x + x.y * x.y;
    }
    ss = oc_warp_sum(ss);
    if (lane == 0) loc[t] = ss;
  }
  exchange(1, false);

  // Best candidate (largest squared norm, then smallest position) of every
  // thread's (key, position << 16 | column); publish() before a CTA barrier,
  // chosen() after it.  A norm that is not a positive number has key 0.
  auto publish = [&](unsigned long long key, int idx) {
    unsigned long long wk;
    int wi;
    warp_argmax_bits(key, idx, &wk, &wi);
    if (lane == 0) {
      skey[warp] = wk;
      sidx[warp] = wi;
    }
  };
  auto chosen = [&](int nw) -> int {
    unsigned long long wk;
    int wi;
    warp_argmax_bits(lane < nw ? skey[lane] : 0ull, lane < nw ? sidx[lane] : 0x7fffffff, &wk, &wi);
    return wi;
  };
  int e0 = 0;  // exponent of the largest initial norm
  auto cand_key = [&](double v) { return oc_cand_key(v, e0, SK); };
  auto better_cand = [](unsigned long long k, int ix, unsigned long long bk, int bi) {
    return k > bk || (k == bk && ix < bi);
  };
  // candidates from the norms of the trailing columns own[0 .. cnt)
  auto candidates = [&](int cnt) {
    unsigned long long key = 0;
    int idx = 0x7fffffff;
    for (int q = threadIdx.x; q < cnt; q += kOcThreads) {
      const int j = own[q];
      const unsigned long long k = cand_key(vn1[j]);
      const int ix = col2pos[j] << 16 | j;
      if (better_cand(k, ix, key, idx)) {
        key = k;
        idx = ix;
      }
    }
    publish(key, idx);
  };
  for (int t = threadIdx.x; t < n; t += kOcThreads) {
    vn1[t] = vn2[t] = total(t, 1);
  }
  candidates(n);  // (each thread reads back its own norms)
  __syncthreads();
  int pick = chosen(kOcWarps);
  e0 = static_cast<int>(cand_key(vn1[pick & 0xffff]) >> 52);

  const double tol3z = sqrt(0.5 * 2.220446049250313e-16);
  // lanes per column and columns per group: a warp carries four columns
  // past 64 rows at a time, or, where this CTA's rows are few, eight
  // columns past 16 (fewer shuffles per column)
  const bool tall = !SK && mend > 192;
  const int lp = tall ? 2 : 3, per = 1 << lp;  // columns of a unit
  int rank = 0;
  for (int i = 0; i < mn; i++) {
    const int b = G > 1 ? (i & 1) : 0;
    const double* ri = rowi + b * ne;
    const int p = pick & 0xffff, ppos = pick >> 16;
    const int cnt = n - i - 1;  // trailing columns without the pivot
    // the pivot's place in the list goes to the last column (the list itself
    // changes under the pass; place qs is not read meanwhile)
    const int qs = col2own[p], last = own[cnt];
    auto list = [&](int q) { return q == qs ? last : own[q]; };
    if (threadIdx.x == kOcThreads - 1) {
      const int ci = pos2col[i];
      pos2col[i] = p;
      pos2col[ppos] = ci;
      col2pos[ci] = ppos;
      col2pos[p] = i;
      own[qs] = last;
      col2own[last] = qs;
    }
    const int below = i > g ? (i - g + G - 1) / G : 0;  // this CTA's rows < i
    const int r0 = below & ~1;
    const bool iown = i % G == g;
    const int lo = below + (iown ? 1 : 0), iloc = i / G;
    const double* cprev = cb + ((i + 1) & 1) * ldl;
    double* cnew = cb + (i & 1) * ldl;
    const double* ap = colp(p);
    const double twp = tws[p];
    int mv = -1;  // the column that moves to the free place to
    double* to = nullptr;
    if constexpr (SPILL) {
      if (si[7] >= 0) {
        to = place(si[7]);
        // (col2pos changes under this for the pivot and the column it trades
        // places with, which stays at i or past it)
        for (int j = si[6]; j < n && mv < 0; j++)
          if (j != p && col2pos[j] >= i) mv = j;
      }
    }
    const int nunit = (cnt + per - 1) >> lp;
    for (int u = warp; u <= nunit; u += kOcWarps) {
      if (u == nunit) {
        // the pivot column itself, kept for the next step's update, its
        // norm below row i and its row i
        double xs = 0.0;
        for (int r = r0 + 2 * lane; r < mend; r += 64) {
          const double2 cp = *reinterpret_cast<const double2*>(cprev + r);
          const double2 av = *reinterpret_cast<const double2*>(ap + r);
          double2 c;
          c.x = r >= lo ? fma(-twp, cp.x, av.x) : 0.0;
          c.y = r + 1 >= lo ? fma(-twp, cp.y, av.y) : 0.0;
          *reinterpret_cast<double2*>(cnew + r) = c;
          xs += c.x * c.x + c.y * c.y;
        }
        xs = oc_warp_sum(xs);
        if (lane == 0) {
          loc[p] = xs;
          if (iown) {
            const double alpha = fma(-twp, cprev[iloc], ap[iloc]);
            if constexpr (G > 1) {
              loci[p] = alpha;
            } else {
              hh[0] = alpha;
            }
          }
        }
        continue;
      }
      const bool norm = u % kNormWindow == i % kNormWindow;
      const int wslot = n + (u / kNormWindow << lp);  // the unit's window sums
      auto unit_pass = [&](auto lc, auto cc) {
        constexpr int L = decltype(lc)::value, C = decltype(cc)::value;
        const int gl = lane & (L - 1), q0 = (u << lp) + lane / L * C;
        double *col[C], *dst[C];
        double tw[C], S[C], N[C];
        bool on[C];
#pragma unroll
        for (int v = 0; v < C; v++) {
          on[v] = q0 + v < cnt;
          const int j = on[v] ? list(q0 + v) : p;
          col[v] = colp(j);
          dst[v] = SPILL && j == mv ? to : col[v];
          tw[v] = tws[j];
        }
        if (norm) {
          oc_pass<L, C, true>(col, dst, tw, on, cprev, ap, twp, r0, lo, mend, gl, S, N);
        } else {
          oc_pass<L, C, false>(col, dst, tw, on, cprev, ap, twp, r0, lo, mend, gl, S, N);
        }
        const double s = oc_group_sum<L, C>(S, gl);
        const double nn = norm ? oc_group_sum<L, C>(N, gl) : 0.0;
        // L / C lanes hold column v's sums
        constexpr int H = L / C;
        const int v = gl / H, sub = gl & (H - 1);
        __syncwarp();
        if (q0 + v < cnt && sub == 0) {
          const int j = list(q0 + v);
          loc[j] = s;
          if (norm) loc[wslot + lane / L * C + v] = nn;
          if (G > 1 && iown) loci[j] = (SPILL && j == mv ? to : colp(j))[iloc];
        }
      };
      if constexpr (!SK) {
        if (tall) {
          unit_pass(std::integral_constant<int, 32>{}, std::integral_constant<int, 4>{});
          continue;
        }
      }
      unit_pass(std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{});
    }
    exchange(b, iown);
    if constexpr (SPILL) {
      if (threadIdx.x == kOcThreads - 1) {  // (nobody reads these before the next barrier)
        if (mv >= 0) {
          slot[mv] = si[7];
          si[6] = mv + 1;
        }
        si[7] = slot[p] < nres ? slot[p] : -1;
      }
    }

    // ---- reflector, row i of R, norms and the next pivot: the same in
    // every CTA
    bool flagged = false;
    unsigned long long key = 0;
    int idx = 0x7fffffff;
    if (warp * 32 < cnt || warp == 0) {
      const double xs = total(p, b);
      const double alpha = G > 1 ? ri[p] : hh[0];
      double beta = alpha, amb = 0.0, kappa = 0.0;
      if (xs != 0.0) {
        const double tt = fma(alpha, alpha, xs), rt = sqrt(tt);
        beta = -copysign(rt, alpha);
        amb = alpha - beta;
        kappa = 1.0 / fma(fabs(alpha), rt, tt);  // 1 / (beta (beta - alpha))
      }
      if (threadIdx.x == 0) {
        rdiag[i] = beta;
        if (i == 0) {
          hh[1] = fabs(P.tol * beta);
        } else if (fabs(beta) < hh[1]) {
          si[2] = i;
        }
      }
      for (int q = threadIdx.x; q < cnt; q += kOcThreads) {
        const int j = own[q];
        const double S = total(j, b);
        const double a = G > 1 ? ri[j] : slab[static_cast<size_t>(j) * ldl + i];
        const double tw = fma(amb, a, S) * kappa;  // the column takes off tw [amb; c]
        const double r = fma(-tw, amb, a);
        tws[j] = tw;
        if constexpr (G > 1) {
          if (iown) Rg[static_cast<long long>(i) * n + j] = r;
        } else {
          slab[static_cast<size_t>(j) * ldl + i] = r;
        }
        // squared norm below row i: dlaqp2's downdate, vn1 (1 - (r /
        // vn1)^2)^(1/2) with its test against vn2, in squares; from the
        // window's fresh sum where there is one
        double base = vn1[j];
        if ((q >> lp) % kNormWindow == i % kNormWindow) {
          const int w = n + ((q >> lp) / kNormWindow << lp) + (q & (per - 1));
          base = fma(a, a, total(w, b));
          vn2[j] = base;
        }
        double nv = base;
        if (base != 0.0) {
          nv = fma(-r, r, base);
          if (nv <= tol3z * vn2[j]) {
            flagged = true;
            nv = -1.0;
          }
        }
        vn1[j] = nv;
        const unsigned long long k = cand_key(nv);
        const int ix = col2pos[j] << 16 | j;
        if (better_cand(k, ix, key, idx)) {
          key = k;
          idx = ix;
        }
      }
    }
    publish(key, idx);
    const int any = __syncthreads_or(flagged);
    if (si[2] != 0) {
      rank = si[2];
      break;
    }
    if (i + 1 == mn) break;
    if (any) {
      // norms whose downdate lost its accuracy, summed anew (with the
      // pending reflector applied on the way); rare, as the window renews
      // every column's norm about every fourth step
      for (int q = warp; q < cnt; q += kOcWarps) {
        const int j = own[q];
        if (!(vn1[j] < 0.0)) continue;
        const double* col = colp(j);
        const double tw = tws[j];
        double ss = 0.0;
        for (int r = lo + lane; r < mend; r += 32) {
          const double x = fma(-tw, cnew[r], col[r]);
          ss += x * x;
        }
        ss = oc_warp_sum(ss);
        if (lane == 0) loc[j] = ss;
      }
      exchange(b ^ (G > 1 ? 1 : 0), false);
      for (int q = threadIdx.x; q < cnt; q += kOcThreads) {
        const int j = own[q];
        if (vn1[j] < 0.0) vn1[j] = vn2[j] = total(j, b ^ (G > 1 ? 1 : 0));
      }
      candidates(cnt);
      barrier();  // (and no peer's next sums before these are read)
    }
    pick = chosen(kOcWarps);
  }
  // R's rows are complete and no peer writes here any more
  barrier();

  // a sketch shorter than n + 16 rows certifies a rank only well below its
  // row count; otherwise the box is reported (-1) for the full sketch
  if (SK && m < n + 16 && (rank == 0 || rank > m - 16)) rank = -1;
  if (g == 0) {
    if (threadIdx.x == 0) P.rank[task] = rank;
    for (int q = threadIdx.x; q < n; q += kOcThreads) P.perm[tk.perm_off + q] = pos2col[q];
  }
  const int k = rank;
  if (k <= 0) return;

  // ---- T = R11^{-1} R12: a warp per redundant column (dtrsm column sweep).
  // R11's columns: in place for G = 1; else gathered, packed, into the
  // shared memory the matrix has left (if they fit).
  double* T = P.tout + tk.t_off;
  double* U = slab;
  const bool staged =
      G > 1 && static_cast<size_t>(k) * (k - 1) / 2 <= static_cast<size_t>(rdiag - slab);
  if (staged)
    for (int q = warp; q < k; q += kOcWarps) {
      const int j = pos2col[q];
      for (int l = lane; l < q; l += 32)
        U[static_cast<size_t>(q) * (q - 1) / 2 + l] = Rg[static_cast<long long>(l) * n + j];
    }
  // reciprocals of R's diagonal, off the substitutions' dependent chains
  for (int q = threadIdx.x; q < k; q += kOcThreads) vn2[q] = 1.0 / rdiag[q];
  __syncthreads();
  oc_tsolve<kOcWarps>(
      k, n, g, G, pos2col, vn2, T, G == 1 || staged,
      [&](int q) -> const double* {
        return G > 1 ? U + static_cast<size_t>(q) * (q - 1) / 2
                     : slab + static_cast<size_t>(pos2col[q]) * ldl;
      },
      [&](int l, int j) -> double {
        return G > 1 ? Rg[static_cast<long long>(l) * n + j]
                     : slab[static_cast<size_t>(j) * ldl + l];
      });
}

template <int G, bool SK, bool SPILL>
cudaError_t launch_cluster(const IdParams& p, cudaStream_t s) {
  const size_t smem = static_cast<size_t>(p.onchip_smem);
  if (smem == 0 || smem > 227 * 1024) return cudaErrorInvalidValue;
  const void* fn = reinterpret_cast<const void*>(&id_cluster_kernel<G, SK, SPILL>);
  cudaError_t e = raise_func_attr(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  if (G > 8) {
    e = raise_func_attr(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G * p.ntasks);
  cfg.blockDim = dim3(kOcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  int na = 0;
  if (G > 1) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = G;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    na = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, id_cluster_kernel<G, SK, SPILL>, p);
}

template <int G>
int cluster_fits(size_t smem) {
  const void* fn = reinterpret_cast<const void*>(&id_cluster_kernel<G, false, false>);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3(kOcThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = G;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  cudaError_t e = raise_func_attr(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem));
  if (e == cudaSuccess && G > 8)
    e = raise_func_attr(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveClusters(&clusters, id_cluster_kernel<G, false, false>, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return clusters > 0 ? 1 : 0;
}

}  // namespace

size_t id_onchip_smem_bytes(int m, int n, int G, int nres) {
  return oc_fixed_bytes(m, n, G) +
         sizeof(double) * static_cast<size_t>(nres) * oc_stride(m, G);
}

int id_resident_columns(int m, int n, int G) {
  const size_t fixed = oc_fixed_bytes(m, n, G), cap = 227 * 1024;
  if (fixed >= cap || n >= 32768) return 0;
  const size_t c = (cap - fixed) / (sizeof(double) * oc_stride(m, G));
  return static_cast<int>(std::min<size_t>(c, n));
}

long long id_workspace_doubles(int m, int n, int G, int nres) {
  if (G == 1) return 0;
  return oc_rows_doubles(std::min(m, n), n) +
         static_cast<long long>(G) * (n - nres) * oc_stride(m, G);
}

int id_tile(int m, int n, int G) {
  if (n >= 32768) return -1;
  int best = -1;
  auto entries = [](int t) { return kTiles[t].nw * kTiles[t].cw * kTiles[t].rs; };
  for (int t = 0; t < kNumTiles; t++) {
    const TileShape& ts = kTiles[t];
    if (n <= ts.nw * ts.cw && oc_rows(m, G) <= 32 * ts.rs &&
        tile_smem_bytes(m, n, G, ts.nw, ts.cw, ts.rs) <= 227 * 1024 &&
        (best < 0 || entries(t) < entries(best)))
      best = t;
  }
  return best;
}

size_t id_group_smem_bytes(int group, int m, int n, int nres) {
  if (group < kTile) return id_onchip_smem_bytes(m, n, group % 100, nres);
  const TileShape& ts = kTiles[(group - kTile) / 100];
  return tile_smem_bytes(m, n, group % 100, ts.nw, ts.cw, ts.rs);
}

cudaError_t launch_id_cluster(const IdParams& p, int group, cudaStream_t s) {
  if (group >= kTile) return launch_tile_any((group - kTile) / 100, p, group % 100, s);
  switch (group) {
    case kOnChip + 1: return launch_cluster<1, false, false>(p, s);
    case kOnChip + 2: return launch_cluster<2, false, false>(p, s);
    case kOnChip + 4: return launch_cluster<4, false, false>(p, s);
    case kOnChip + 8: return launch_cluster<8, false, false>(p, s);
    case kOnChip + 16: return launch_cluster<16, false, false>(p, s);
    case kSketched + 1: return launch_cluster<1, true, false>(p, s);
    case kSketched + 2: return launch_cluster<2, true, false>(p, s);
    case kSketched + 8: return launch_cluster<8, true, false>(p, s);
    case kSketched + 16: return launch_cluster<16, true, false>(p, s);
    case kSpilled + 8: return launch_cluster<8, false, true>(p, s);
    case kSpilled + 16: return launch_cluster<16, false, true>(p, s);
    default: return cudaErrorInvalidValue;
  }
}

int id_cluster_fits(int G) {
  switch (G) {
    case 1: return 1;
    case 2: return cluster_fits<2>(227 * 1024);
    case 4: return cluster_fits<4>(227 * 1024);
    case 8: return cluster_fits<8>(227 * 1024);
    case 16: return cluster_fits<16>(227 * 1024);
    default: return 0;
  }
}

}  // namespace kib
