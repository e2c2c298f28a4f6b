// The solution on a set of domain points, as boundary_integral_solve
// computes it (linear_solve.cpp:142-180): out = K_domain mu + U_forward alpha
// with the forward kernel (kernel.cpp:337-357) and the hole border columns
// (linear_solve.cpp:18-64), then zero wherever Boundary::is_in_domain says
// the point lies outside the domain.
//
// The reference forms K_domain as a dense |targets| x N matrix (16 GB for a
// 350^2 grid on 16,384 nodes) and multiplies it.  Here each thread owns one
// or two targets and sweeps the source nodes staged in shared memory, forming the
// entries on the fly (FP64, reciprocal by a refined hardware estimate, so the
// sums agree with the exact entries to FP64 rounding); the sources are split
// across CTAs when there are too few targets to fill the GPU, and a finish
// kernel adds the split sums in a fixed order, the border term and the mask.
//
// Domain tests (kept apart from the sums so they are exact):
//   * nodes: CubicBoundary::is_in_domain (cubic_boundary.cpp:182-230), the
//     test of every node-defined boundary: outside when within 1e-2 of any
//     node, when the crossing count of the outer curve is even, or when a
//     hole's crossing count is +1 modulo 2 (C remainder semantics: a count
//     of -1 does not exclude).  A crossing is counted for the edge from node
//     i to the next node of its curve when node i lies right of the point
//     and the edge's end heights straddle it.
//   * disk: Circle / Annulus / Donut::is_in_domain (circle.cpp:34-42,
//     annulus.cpp:66-79, donut.cpp:67-80): outside when |x - c| + 1e-2 > R or
//     |x - hole center| - 1e-2 < hole radius for any hole.
#include "ki_kernels.h"

namespace kib {

namespace {

constexpr int kDomThreads = 256;
constexpr double kDomainEps = 1e-2;  // cubic_boundary.cpp:185, circle.cpp:37

// Per-source values staged in shared memory, as in the operator product:
//   Laplace:          a = -(w / 2 pi) mu (n_x, n_y)
//   Laplace-Neumann:  a0 = (w / 2 pi) mu        (forward entry (w/2pi) log|r|)
//   Stokes:           a = (w / pi) (n_x, n_y), density (mu_0, mu_1)
// A thread owns H targets of a block's 256 (two, 128 apart, where the blocks
// fill the GPU), as in the operator product: bound by the FP64 pipe.  live,
// if given, is the number of points inside the domain and their list: the
// others are zero in the result and no sum is formed for them (blocks past
// the number return at once).  350^2 points of a star's bounding square on
// its 16,384 nodes, test and sums: 1.94 ms -> 0.76 ms, the sums about five
// sixths of it.
template <int PDE, int H>
__global__ void __launch_bounds__(kDomThreads / H)
    domain_partial_kernel(const Node* __restrict__ nodes, int np, int nt,
                          const double* __restrict__ tg, const int* __restrict__ live,
                          const double* __restrict__ mu, int chunk, long long stride,
                          double* __restrict__ part) {
  const int count = live ? live[0] : nt;
  if (blockIdx.x * kDomThreads >= count) return;
  constexpr int T = kDomThreads / H;
  __shared__ SourceArray<(H > 1), kDomThreads> spos, samp, sden;
  int t[H];
  double tx[H], ty[H], y0[H], y1[H];
#pragma unroll
  for (int h = 0; h < H; h++) {
    const int i = blockIdx.x * kDomThreads + threadIdx.x + h * T;
    t[h] = i < count ? (live ? live[1 + i] : i) : -1;
    tx[h] = t[h] >= 0 ? tg[2 * t[h]] : 0.0;
    ty[h] = t[h] >= 0 ? tg[2 * t[h] + 1] : 0.0;
    y0[h] = y1[h] = 0.0;
  }
  const int s0 = blockIdx.y * chunk;
  const int s1 = min(np, s0 + chunk);
  for (int base = s0; base < s1; base += kDomThreads) {
    __syncthreads();
#pragma unroll
    for (int h = 0; h < H; h++) {
      const int k = threadIdx.x + h * T, j = base + k;
      if (j < s1) {
        const Node s = nodes[j];
        spos.put(k, s.x, s.y);
        if (PDE == kLaplace) {
          const double c = -s.w * KI_INV_2PI * mu[j];
          samp.put(k, c * s.nx, c * s.ny);
        } else if (PDE == kLaplaceNeumann) {
          samp.put(k, s.w * KI_INV_2PI * mu[j], 0.0);
        } else {
          const double c = s.w * KI_INV_PI;
          samp.put(k, c * s.nx, c * s.ny);
          sden.put(k, mu[2 * j], mu[2 * j + 1]);
        }
      } else {
        // padding: a far source of zero strength (|r|^2 stays inside the
        // range of the reciprocal estimate; every numerator is zero)
        spos.put(k, 1e15, 1e15);
        samp.put(k, 0.0, 0.0);
        sden.put(k, 0.0, 0.0);
      }
    }
    __syncthreads();
    const int cnt = min(kDomThreads, (s1 - base + 3) & ~3);  // (the padding past it is not summed)
#pragma unroll 1
    for (int q4 = 0; q4 < cnt; q4 += 4) {
#pragma unroll
      for (int q = q4; q < q4 + 4; q++) {
        const double2 p = spos.get(q), a = samp.get(q);
        const double2 d = PDE == kStokes ? sden.get(q) : make_double2(0.0, 0.0);
#pragma unroll
        for (int h = 0; h < H; h++) {
          if (PDE == kLaplaceNeumann) {
            const double r0 = tx[h] - p.x, r1 = ty[h] - p.y;
            y0[h] += a.x * (0.5 * log(r0 * r0 + r1 * r1));
          } else {
            pair_sum<PDE>(tx[h], ty[h], 0.0, 0.0, p.x, p.y, a.x, a.y, d.x, d.y, y0[h], y1[h]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < H; h++) {
    if (t[h] < 0) continue;
    if (PDE == kStokes) {
      part[stride * blockIdx.y + 2 * t[h]] = y0[h];
      part[stride * blockIdx.y + 2 * t[h] + 1] = y1[h];
    } else {
      part[stride * blockIdx.y + t[h]] = y0[h];
    }
  }
}

// CubicBoundary::is_in_domain, in two steps.
//
// curve_prep_kernel, one thread per node: the node's position, the height of
// the next node of its curve, and a code marking the last node of the outer
// curve (1) or of a hole (2), as structure-of-arrays; and per tile of 32
// consecutive nodes (one warp) the bounds a point must meet for the tile to
// matter: the nodes' box, the lowest and highest edge end, whether a curve
// ends in it.
//
// domain_mask_nodes_kernel, one warp per 32 targets, no block barriers: the
// warp walks the tiles in order, 32 at a time: a tile per lane, tested
// against the targets' bounding box, so that the walk waits for a load per
// 32 tiles and not for each; of the tiles left, one that no target of the
// warp can be within 1e-2 of (box distance) and that no target lies strictly
// between the tile's edge ends and left of its rightmost node contributes
// nothing and is skipped, unless it ends a curve.  Other tiles are staged in
// the warp's shared-memory slice and every lane runs the reference's tests
// on the 32 nodes.  mask[t] = 1 inside, 0 outside.
struct CurveTile {
  double bx0, bx1, by0, by1, ey0, ey1;
  int code, pad;
};

__global__ void curve_prep_kernel(const Node* __restrict__ nodes, int np,
                                  const double* __restrict__ holes, int nh,
                                  double* __restrict__ cx, double* __restrict__ cy,
                                  double* __restrict__ cyn, int* __restrict__ ccode,
                                  CurveTile* __restrict__ tiles) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int n_outer = np;
  for (int h = 0; h < nh; h++) n_outer -= static_cast<int>(holes[4 * h + 3]);
  double bx0 = NAN, bx1 = NAN, by0 = NAN, by1 = NAN, ey0 = NAN, ey1 = NAN;
  int code = 0;
  if (j < np) {
    int start = 0, end = n_outer;
    code = 1;
    if (j >= n_outer) {
      start = n_outer;
      code = 2;
      for (int h = 0; h < nh; h++) {
        end = start + static_cast<int>(holes[4 * h + 3]);
        if (j < end) break;
        start = end;
      }
    }
    const Node s = nodes[j];
    const double yn = nodes[j + 1 < end ? j + 1 : start].y;
    code = j == end - 1 ? code : 0;
    cx[j] = s.x;
    cy[j] = s.y;
    cyn[j] = yn;
    ccode[j] = code;
    bx0 = bx1 = s.x;
    by0 = by1 = s.y;
    ey0 = fmin(s.y, yn);
    ey1 = fmax(s.y, yn);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    bx0 = fmin(bx0, __shfl_xor_sync(0xffffffffu, bx0, o));
    bx1 = fmax(bx1, __shfl_xor_sync(0xffffffffu, bx1, o));
    by0 = fmin(by0, __shfl_xor_sync(0xffffffffu, by0, o));
    by1 = fmax(by1, __shfl_xor_sync(0xffffffffu, by1, o));
    ey0 = fmin(ey0, __shfl_xor_sync(0xffffffffu, ey0, o));
    ey1 = fmax(ey1, __shfl_xor_sync(0xffffffffu, ey1, o));
    code |= __shfl_xor_sync(0xffffffffu, code, o);
  }
  if (lane == 0 && j < np) tiles[j >> 5] = CurveTile{bx0, bx1, by0, by1, ey0, ey1, code, 0};
}

// Points inside the domain, listed for the sums (inside[0] counts them; the
// list's order varies, which no sum depends on).  All lanes of the warp.
__device__ __forceinline__ void list_inside(bool in, int t, int* __restrict__ inside) {
  if (!inside) return;
  const unsigned m = __ballot_sync(0xffffffffu, in);
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0 && m) at = atomicAdd(inside, __popc(m));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (in) inside[1 + at + __popc(m & ((1u << lane) - 1u))] = t;
}

constexpr int kMaskWarps = 8;
__global__ void __launch_bounds__(32 * kMaskWarps)
    domain_mask_nodes_kernel(const double* __restrict__ cx, const double* __restrict__ cy,
                             const double* __restrict__ cyn, const int* __restrict__ ccode,
                             const CurveTile* __restrict__ tiles, int np, int nt,
                             const double* __restrict__ tg, unsigned char* __restrict__ mask,
                             int* __restrict__ inside) {
  __shared__ double sx[kMaskWarps][32], sy[kMaskWarps][32], syn[kMaskWarps][32];
  __shared__ int scode[kMaskWarps][32];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int t = (blockIdx.x * kMaskWarps + wl) * 32 + lane;
  const bool live = t < nt;
  const double tx = live ? tg[2 * t] : 0.0, ty = live ? tg[2 * t + 1] : 0.0;
  int wind = 0;
  bool out = false;
  double near2 = INFINITY;
  const int ntiles = (np + 31) >> 5;
  // the live targets' bounding box
  double gx0 = live ? tx : INFINITY, gx1 = live ? tx : -INFINITY;
  double gy0 = live ? ty : INFINITY, gy1 = live ? ty : -INFINITY;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gx0 = fmin(gx0, __shfl_xor_sync(0xffffffffu, gx0, o));
    gx1 = fmax(gx1, __shfl_xor_sync(0xffffffffu, gx1, o));
    gy0 = fmin(gy0, __shfl_xor_sync(0xffffffffu, gy0, o));
    gy1 = fmax(gy1, __shfl_xor_sync(0xffffffffu, gy1, o));
  }
  unsigned todo = 0;
  for (int k = 0; k < ntiles; k++) {
    if ((k & 31) == 0) {
      bool take = false;
      if (k + lane < ntiles) {
        const CurveTile tl = tiles[k + lane];
        const double dx = fmax(fmax(tl.bx0 - gx1, gx0 - tl.bx1), 0.0);
        const double dy = fmax(fmax(tl.by0 - gy1, gy0 - tl.by1), 0.0);
        take = dx * dx + dy * dy < 1.0004e-4 ||
               (gy1 > tl.ey0 && gy0 < tl.ey1 && gx0 < tl.bx1) || tl.code != 0;
      }
      todo = __ballot_sync(0xffffffffu, take);
    }
    if (!todo) {
      k |= 31;  // (none of these 32)
      continue;
    }
    if (!(todo >> (k & 31) & 1)) continue;
    const CurveTile tl = tiles[k];  // (in L1 from the walk above)
    const double dx = fmax(fmax(tl.bx0 - tx, tx - tl.bx1), 0.0);
    const double dy = fmax(fmax(tl.by0 - ty, ty - tl.by1), 0.0);
    const bool near_box = dx * dx + dy * dy < 1.0004e-4;
    const bool cross = ty > tl.ey0 && ty < tl.ey1 && tx < tl.bx1;
    const bool any_near = __any_sync(0xffffffffu, live && near_box);
    const bool any_cross = __any_sync(0xffffffffu, live && cross);
    if (!any_near && !any_cross && tl.code == 0) continue;
    const int j = (k << 5) + lane;
    __syncwarp();
    if (j < np) {
      sx[wl][lane] = cx[j];
      sy[wl][lane] = cy[j];
      syn[wl][lane] = cyn[j];
      scode[wl][lane] = ccode[j];
    } else {
      // padding: left of every point (no crossing), infinitely far
      sx[wl][lane] = -INFINITY;
      sy[wl][lane] = 0.0;
      syn[wl][lane] = 0.0;
      scode[wl][lane] = 0;
    }
    __syncwarp();
    // the two tests apart, each only where a lane needs it.  Distances:
    // the root of the smallest square decides (sqrt rounds monotonically).
    if (any_near) {
#pragma unroll 8
      for (int q = 0; q < 32; q++) {
        const double ddx = subd(tx, sx[wl][q]), ddy = subd(ty, sy[wl][q]);
        const double d2 = add(mul(ddx, ddx), mul(ddy, ddy));
        near2 = d2 < near2 ? d2 : near2;
      }
    }
    if (!any_cross && tl.code == 0) continue;
#pragma unroll 8
    for (int q = 0; q < 32; q++) {
      const double py = sy[wl][q], pyn = syn[wl][q];
      const bool right = sx[wl][q] > tx;
      wind += right && py < ty && pyn > ty;
      wind -= right && py > ty && pyn < ty;
      const int cq = scode[wl][q];
      if (cq) {
        if (cq == 1 ? wind % 2 == 0 : wind % 2 == 1) out = true;
        wind = 0;
      }
    }
  }
  if (near2 < 1.0001e-4 && __dsqrt_rn(near2) < kDomainEps) out = true;
  if (live) mask[t] = out ? 0 : 1;
  list_inside(live && !out, t, inside);
}

// Circle / Annulus / Donut::is_in_domain with the disk (cx, cy, R).
__global__ void domain_mask_disk_kernel(double cx, double cy, double R,
                                        const double* __restrict__ holes, int nh, int nt,
                                        const double* __restrict__ tg,
                                        unsigned char* __restrict__ mask,
                                        int* __restrict__ inside) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = t < nt;
  const double tx = live ? tg[2 * t] : 0.0, ty = live ? tg[2 * t + 1] : 0.0;
  const double x = subd(tx, cx), y = subd(ty, cy);
  bool out = add(__dsqrt_rn(add(mul(x, x), mul(y, y))), kDomainEps) > R;
  for (int h = 0; h < nh && !out; h++) {
    const double rx = subd(tx, holes[4 * h]), ry = subd(ty, holes[4 * h + 1]);
    if (subd(__dsqrt_rn(add(mul(rx, rx), mul(ry, ry))), kDomainEps) < holes[4 * h + 2])
      out = true;
  }
  if (live) mask[t] = out ? 0 : 1;
  list_inside(live && !out, t, inside);
}

// Split sums in a fixed order, + U_forward alpha, masked.
__global__ void domain_finish_kernel(int pde, int nt, int splits, long long stride,
                                     const double* __restrict__ part,
                                     const double* __restrict__ tg, int nh,
                                     const double* __restrict__ holes,
                                     const double* __restrict__ alpha,
                                     const unsigned char* __restrict__ mask,
                                     double* __restrict__ out) {
  const int sd = pde == kStokes ? 2 : 1;
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= nt * sd) return;
  const int t = row / sd, comp = row % sd;
  if (mask && !mask[t]) {
    out[row] = 0.0;
    return;
  }
  double s = part[row];
  for (int k = 1; k < splits; k++) s += part[stride * k + row];
  if (alpha && pde != kLaplaceNeumann) {
    const double tx = tg[2 * t], ty = tg[2 * t + 1];
    for (int h = 0; h < nh; h++) {
      double u[3];
      border_u(pde, tx, ty, holes + 4 * h, comp, u);
      if (pde == kLaplace) {
        s += u[0] * alpha[h];
      } else {
        s += u[0] * alpha[3 * h] + u[1] * alpha[3 * h + 1] + u[2] * alpha[3 * h + 2];
      }
    }
  }
  out[row] = s;
}

}  // namespace

int domain_splits(int nt, int np, int num_sms) {
  // about 32 blocks per SM, of at least 512 sources each: blocks of points
  // outside the domain leave at once, and the last of the others to start
  // are a small part of an SM's work
  const int tiles = (nt + kDomThreads - 1) / kDomThreads;
  const int want = (32 * num_sms + tiles - 1) / tiles;
  return std::max(1, std::min(want, (np + 511) / 512));
}

size_t domain_mask_scratch_bytes(int np) {
  const size_t tiles = (static_cast<size_t>(np) + 31) / 32;
  return 3 * sizeof(double) * np + sizeof(int) * np + sizeof(CurveTile) * tiles + 256;
}

cudaError_t launch_domain_mask(int kind, const Node* nodes, int np, const double* holes, int nh,
                               const double* disk, int nt, const double* targets,
                               unsigned char* mask, int* inside, void* scratch,
                               cudaStream_t s) {
  if (nt == 0) return cudaSuccess;
  if (inside) {
    const cudaError_t e = cudaMemsetAsync(inside, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
  }
  if (kind == kDomainNodes) {
    // scratch: x, y, next y (np doubles each), tiles (16-byte aligned), codes
    double* cx = static_cast<double*>(scratch);
    double* cy = cx + np;
    double* cyn = cy + np;
    CurveTile* tiles = reinterpret_cast<CurveTile*>(cyn + np + (np & 1));
    int* ccode = reinterpret_cast<int*>(tiles + (np + 31) / 32);
    count_launches(2);
    curve_prep_kernel<<<(np + 255) / 256, 256, 0, s>>>(nodes, np, holes, nh, cx, cy, cyn, ccode,
                                                       tiles);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int per_block = 32 * kMaskWarps;
    domain_mask_nodes_kernel<<<(nt + per_block - 1) / per_block, per_block, 0, s>>>(
        cx, cy, cyn, ccode, tiles, np, nt, targets, mask, inside);
  } else {
    count_launches(1);
    const int grid = (nt + kDomThreads - 1) / kDomThreads;
    domain_mask_disk_kernel<<<grid, kDomThreads, 0, s>>>(disk[0], disk[1], disk[2], holes, nh,
                                                        nt, targets, mask, inside);
  }
  return cudaGetLastError();
}

namespace {
template <int H>
void launch_partial(int pde, dim3 grid, const Node* nodes, int np, int nt, const double* targets,
                    const int* inside, const double* mu, int chunk, long long rows, double* dst,
                    cudaStream_t s) {
  constexpr int T = kDomThreads / H;
  if (pde == kLaplace)
    domain_partial_kernel<kLaplace, H><<<grid, T, 0, s>>>(nodes, np, nt, targets, inside, mu,
                                                          chunk, rows, dst);
  else if (pde == kLaplaceNeumann)
    domain_partial_kernel<kLaplaceNeumann, H><<<grid, T, 0, s>>>(nodes, np, nt, targets, inside,
                                                                mu, chunk, rows, dst);
  else
    domain_partial_kernel<kStokes, H><<<grid, T, 0, s>>>(nodes, np, nt, targets, inside, mu,
                                                         chunk, rows, dst);
}
}  // namespace

cudaError_t launch_domain_eval(int pde, const Node* nodes, int np, int nt,
                               const double* targets, const double* mu, int nh,
                               const double* holes, const double* alpha,
                               const unsigned char* mask, const int* inside, int splits,
                               double* part, double* out, int num_sms, cudaStream_t s) {
  if (nt == 0) return cudaSuccess;
  const int sd = pde == kStokes ? 2 : 1;
  const long long rows = static_cast<long long>(nt) * sd;
  double* dst = splits > 1 ? part : out;
  // (whole tiles of sources: 700 in two chunks are three tiles, not four)
  const int chunk = ((np + splits - 1) / splits + kDomThreads - 1) / kDomThreads * kDomThreads;
  const dim3 grid((nt + kDomThreads - 1) / kDomThreads, splits);
  count_launches(2);
  if (sum_targets(static_cast<long long>(grid.x) * splits, num_sms, kDomainSingle) == 1) {
    launch_partial<1>(pde, grid, nodes, np, nt, targets, inside, mu, chunk, rows, dst, s);
  } else {
    launch_partial<2>(pde, grid, nodes, np, nt, targets, inside, mu, chunk, rows, dst, s);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  domain_finish_kernel<<<static_cast<int>((rows + 255) / 256), 256, 0, s>>>(
      pde, nt, splits, rows, dst, targets, nh, holes, alpha, mask, out);
  return cudaGetLastError();
}

}  // namespace kib
