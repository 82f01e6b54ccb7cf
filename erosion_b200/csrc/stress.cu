// Wall shear stress on the bodies (computeShearStress, stokesSolver.f:3002-3096)
// and velocity/pressure/vorticity at target points (computeQoiTargets,
// :3099-3323).
#include "state.h"
#include "cluster.cuh"
#include <cmath>

namespace eb {

// Offset of curve c's five boundary-value fields in the all-curves buffer.
__device__ __forceinline__ long long bd_all_off(const GeoDev& G, int c) {
  return c == 0 ? 0LL : 5LL * G.nout + 5LL * (c - 1) * G.n;
}

// Parts of the source curves of about as many nodes each: the first curve of part y, the
// one with N y / parts nodes or more before it.
__device__ __forceinline__ int part_first(const GeoDev& G, int y, int parts) {
  const long long at = (long long)G.N * y / parts;
  if (y == parts) return G.M + 1;
  return at == 0 ? 0 : at <= G.nout ? 1 : 1 + (int)((at - G.nout + G.n - 1) / G.n);
}

// Longest body curve that a warp takes by itself (k_bary_sum): a stage of the tile holds
// eight of them or more.  With eight warps sharing a curve's nodes the block sums after
// each of the three passes cost more than the nodes do: 20,000 targets (60,000) against
// 500 bodies of 8 nodes take 1.8 ms (4.2) by warps and 5.9 (14.5) shared, 1000 of 16 nodes
// 5.2 (13.1) and 13.4 (33.1), 500 of 32 nodes 4.9 (12.5) and 8.9 (22.2); 100 targets against
// the last 0.32 and 0.33.
constexpr int SHORT_CURVE = NEAR_TK / NEAR_W;

// Barycentric Stokes DLP with gradient of the source curves of part blockIdx.y
// of gridDim.y at 32 targets: CTA blockIdx.x takes targets 32 blockIdx.x.. of all
// ntar, or with bodies = 1 (the targets are the body nodes) 32 nodes of one body,
// skipping that body's curve.  Partial sums per part: out[(y*6 + q)*ntar + t] with
// q = ux, uy, u1x, u1y, u2x, u2y.  SHORT: the bodies' curves are staged many at a time and
// a warp takes every eighth.
template <bool SHORT>
__global__ void __launch_bounds__(NEAR_NT, 2)
k_bary_sum(GeoDev G, const double2* __restrict__ bd_all, const double2* __restrict__ txy, int bodies, int ntar,
           double* __restrict__ out) {
  __shared__ BaryTile T;
  const int per = bodies ? (G.n + NEAR_T - 1) / NEAR_T : 0, b = bodies ? blockIdx.x / per : -1;
  const int t0 = bodies ? b * G.n + NEAR_T * (blockIdx.x - b * per) : NEAR_T * blockIdx.x;
  const int t1 = bodies ? min((b + 1) * G.n, t0 + NEAR_T) : min(ntar, t0 + NEAR_T);
  const int t = t0 + (threadIdx.x & 31), wid = threadIdx.x >> 5;
  const bool act = t < t1;
  const double2 zt = txy[act ? t : t1 - 1];
  double a[6] = {0, 0, 0, 0, 0, 0};
  auto add = [&](const DLPVal& r) {
    a[0] += r.ux; a[1] += r.uy; a[2] += r.u1x; a[3] += r.u1y; a[4] += r.u2x; a[5] += r.u2y;
  };
  int c = part_first(G, blockIdx.y, gridDim.y);
  const int c1 = part_first(G, blockIdx.y + 1, gridDim.y);
  if constexpr (SHORT) {
    if (c == 0 && c1 > 0) {   // the wall by all warps; each holds the sum
      const DLPVal r = bary_eval<2>(T, G, 0, bd_all, zt, act);
      if (wid == 0) add(r);
      c = 1;
    }
    const int stage = NEAR_TK / G.n / NEAR_W * NEAR_W;   // bodies staged at a time
    for (; c < c1; c += stage) {
      const int k = min(stage, c1 - c);
      __syncthreads();
      if ((int)threadIdx.x < k * G.n) {
        const int e = threadIdx.x / G.n, j = threadIdx.x - e * G.n, g = curve_start(G, c) + (int)threadIdx.x;
        const double2 z = G.xy[g];
        const double2* __restrict__ bdc = bd_all + bd_all_off(G, c + e) + j;
        T.z[threadIdx.x] = z;
        T.dz[threadIdx.x] = G.dz[g];
        T.za[threadIdx.x] = cinv(csub(z, G.cen[c + e - 1]));
#pragma unroll
        for (int q = 0; q < 5; ++q) T.b[q][threadIdx.x] = bdc[q * G.n];
      }
      __syncthreads();
      for (int e = wid; e < k; e += NEAR_W)
        if (c + e != b + 1 || !bodies)
          add(bary_eval<2, 1, true>(T, G, c + e, bd_all + bd_all_off(G, c + e), zt, act, e * G.n));
    }
    __syncthreads();
    near_reduce(a, T.red);
  } else {
    for (; c < c1; ++c)
      if (c != b + 1 || !bodies) add(bary_eval<2>(T, G, c, bd_all + bd_all_off(G, c), zt, act));
  }
  if (act && threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < 6; ++q) out[((size_t)blockIdx.y * 6 + q) * ntar + t] = a[q];
  }
}

// Launches k_bary_sum for tasks CTAs of targets and the parts of the curves.
static void bary_sum(State& s, int tasks, int parts, const double2* bd_all, const double2* txy, int bodies, int ntar,
                     double* out) {
  const GeoDev G = s.geo();
  const dim3 grid(tasks, parts);
  if (G.M > 0 && G.n <= SHORT_CURVE)
    k_bary_sum<true><<<grid, NEAR_NT, 0, s.st>>>(G, bd_all, txy, bodies, ntar, out);
  else
    k_bary_sum<false><<<grid, NEAR_NT, 0, s.st>>>(G, bd_all, txy, bodies, ntar, out);
  EB_LAUNCH_CHECK();
}

// Self-interaction of each body for the deformation tensor: the odd-even
// trapezoid rule on the subtracted density (:2744-2833) plus the jump term
// from the spectral tangential derivative of sigma (:2933-2958).  CTA = 32
// nodes of a body, one per lane; its 8 warps split the body's sources in pairs
// of neighbours (one enters the rule, both the derivative) and meet in a fixed
// order.  out[3][n*M] = E11, E12, E22.  A chain of n/16 pairs a thread: 7.6 us
// at 37 bodies x 200 nodes and 66 us at 400 x 256 (a thread per node with all
// sources and a correctly rounded division: 27.8 and 79.2 us).
__global__ void __launch_bounds__(NEAR_NT)
k_stress_self(GeoDev G, const double* __restrict__ den, const double* __restrict__ dk, double* __restrict__ out) {
  __shared__ double2 ss[FAR_TS], xs[FAR_TS], ps[FAR_TS];
  __shared__ double ws[FAR_TS];
  __shared__ double red[NEAR_W / 2][5][32];
  const int n = G.n, per = (n + 31) / 32, b = blockIdx.x / per, nb = n * G.M;
  const int start = G.nout + b * n, wid = threadIdx.x >> 5;
  const int kk = 32 * (blockIdx.x - b * per) + (threadIdx.x & 31), k = min(kk, n - 1), g = start + k;
  const double2 x = G.xy[g];
  const double sxk = den[ix_of(G, g)], syk = den[iy_of(G, g)];
  const int odd = k & 1;
  double e[5] = {0, 0, 0, 0, 0};   // E11, E12, E22, d sigma/d theta
  for (int k0 = 0; k0 < n; k0 += FAR_TS) {
    __syncthreads();
    const int j = k0 + threadIdx.x;
    if (j < n) {
      const int gj = start + j;
      ss[threadIdx.x] = make_double2(den[ix_of(G, gj)], den[iy_of(G, gj)]);
      xs[threadIdx.x] = G.xy[gj];
      ps[threadIdx.x] = G.nrm[gj];
      ws[threadIdx.x] = G.w[gj];
    }
    __syncthreads();
    const int kt = min(FAR_TS, n - k0) / 2;   // pairs of neighbours (n is even)
    const int hi = kt * (wid + 1) / NEAR_W;
    for (int q = kt * wid / NEAR_W; q < hi; ++q) {
      const double2 s0 = ss[2 * q], s1 = ss[2 * q + 1];
      int m = k - (k0 + 2 * q);
      if (m < 0) m += n;
      const int m1 = m > 0 ? m - 1 : n - 1;
      const double d0 = __ldg(dk + m), d1 = __ldg(dk + m1);
      e[3] = fma(d0, s0.x, fma(d1, s1.x, e[3]));
      e[4] = fma(d0, s0.y, fma(d1, s1.y, e[4]));
      const int o = 2 * q + 1 - odd;   // the neighbour of the other parity
      const double2 p = ps[o], sj = odd ? s0 : s1;
      const double rx = x.x - xs[o].x, ry = x.y - xs[o].y;
      const double ir2 = rcp_raw64(fma(rx, rx, ry * ry));
      const double ir4 = ir2 * ir2 * ws[o];
      const double rdotn = fma(rx, p.x, ry * p.y), routn = fma(rx, p.y, ry * p.x);
      const double dsx = sj.x - sxk, dsy = sj.y - syk;
      const double rdots = fma(rx, dsx, ry * dsy), routs = fma(rx, dsy, ry * dsx);
      const double A = 2.0 * rdotn * rdots * ir4, C = 4.0 * A * ir2;
      e[0] += A + 2.0 * ir4 * rx * fma(rdots, p.x, rdotn * dsx) - C * rx * rx;
      e[1] += ir4 * fma(rdots, routn, rdotn * routs) - C * rx * ry;
      e[2] += A + 2.0 * ir4 * ry * fma(rdots, p.y, rdotn * dsy) - C * ry * ry;
    }
  }
  __syncthreads();
  near_reduce(e, red);
  if (threadIdx.x >= 32 || kk >= n) return;
  // jump: t = (-py, px) at the target, d(sigma)/ds . t
  const double spk = G.sp[g];
  const double2 nn = G.nrm[g];
  const double tx = -nn.y, ty = nn.x;
  const double dd = (e[3] / spk) * tx + (e[4] / spk) * ty;
  const int i = b * n + k;
  out[i] = e[0] + 0.5 * dd * (tx * tx - ty * ty);
  out[nb + i] = e[1] + 0.5 * dd * 2.0 * tx * ty;
  out[2 * nb + i] = e[2] + 0.5 * dd * (-tx * tx + ty * ty);
}

// Trapezoid deformation tensor of every other curve (deformation_on_boundary_trap,
// :2350-2384 for the wall and :2496-2543 for the bodies), as partial sums
// over the far-field tile splits.  out[(split*3 + q)*nb + i].
__global__ void __launch_bounds__(256)
k_stress_trap(GeoDev G, const double* __restrict__ den, const int4* __restrict__ tiles,
              const int* __restrict__ split_ptr, double* __restrict__ out) {
  __shared__ double2 sxy[FAR_TS], sn[FAR_TS], ss[FAR_TS];
  __shared__ double sw[FAR_TS];
  const int nb = G.n * G.M;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < nb;
  const int ic = act ? i : nb - 1;
  const int g = G.nout + ic;
  const int mycurve = 1 + ic / G.n;
  const double2 p = G.xy[g];
  double e11 = 0, e12 = 0, e22 = 0;
  const int split = blockIdx.y;
  for (int ti = split_ptr[split]; ti < split_ptr[split + 1]; ++ti) {
    const int4 T = tiles[ti];
    __syncthreads();
    if (threadIdx.x < T.y) {
      int gs = T.x + threadIdx.x;
      sxy[threadIdx.x] = G.xy[gs];
      sn[threadIdx.x] = G.nrm[gs];
      ss[threadIdx.x] = make_double2(den[ix_of(G, gs)], den[iy_of(G, gs)]);
      sw[threadIdx.x] = G.w[gs];
    }
    __syncthreads();
    if (T.z == mycurve) continue;
    double a11 = 0, a12 = 0, a22 = 0;
    for (int j = 0; j < T.y; ++j) {
      const double2 q = sxy[j], nn = sn[j], s = ss[j];
      double rx = p.x - q.x, ry = p.y - q.y;
      double rho2 = rx * rx + ry * ry;
      double ir2 = 1.0 / rho2, ir4 = ir2 * ir2, ir6 = ir4 * ir2;
      double rdotn = rx * nn.x + ry * nn.y;
      double routn = rx * nn.y + ry * nn.x;
      double rdotden = rx * s.x + ry * s.y;
      double routden = rx * s.y + ry * s.x;
      double wg = sw[j];
      a11 += 0.5 * (2.0 * rdotn * rdotden * ir4 + 2.0 * rdotden * ir4 * rx * nn.x + 2.0 * rdotn * ir4 * rx * s.x -
                    8.0 * rdotn * rdotden * ir6 * rx * rx) * wg;
      a12 += 0.5 * (rdotden * routn * ir4 + rdotn * routden * ir4 - 8.0 * rdotn * rdotden * rx * ry * ir6) * wg;
      a22 += 0.5 * (2.0 * rdotn * rdotden * ir4 + 2.0 * rdotden * ir4 * ry * nn.y + 2.0 * rdotn * ir4 * ry * s.y -
                    8.0 * rdotn * rdotden * ir6 * ry * ry) * wg;
    }
    e11 += a11; e12 += a12; e22 += a22;
  }
  if (act) {
    out[((size_t)split * 3 + 0) * nb + i] = e11;
    out[((size_t)split * 3 + 1) * nb + i] = e12;
    out[((size_t)split * 3 + 2) * nb + i] = e22;
  }
}

// ---- Shear stress with the trapezoid rule wherever it is exact to rounding.
// The reference evaluates every other curve's contribution to a body node by
// the barycentric formulas (deformation_on_boundary, :2707-2727 and
// :2893-2925).  Away from a source curve the trapezoid rule on the same
// density gives the same value up to its quadrature (aliasing) error, which
// for a density with content up to the Nyquist mode decays like
// exp(-pi d / h) with the distance d to the curve and its node spacing h:
// beyond d = STRESS_NEAR_H h it is below 1e-16 of the value.  So the
// barycentric evaluation runs only on the (body node, source curve) pairs
// within that distance, and the trapezoid rule (FP64) on all the others.
constexpr double STRESS_NEAR_H = 12.0;

// Per body node: min over wall nodes j of |x_i - x_j|^2 / h_j^2, with h_j the
// local wall spacing |z'_j| 2 pi / nout.  Wall nodes staged through shared
// memory in chunks.
__global__ void __launch_bounds__(256)
k_stress_wall_dist(GeoDev G, double* __restrict__ d2h) {
  __shared__ double2 sxy[256];
  __shared__ double sh2[256];
  const int nb = G.n * G.M;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const double2 p = G.xy[G.nout + (i < nb ? i : nb - 1)];
  const double hs = EB_TWOPI / G.nout;
  double best = 1e300;
  for (int j0 = 0; j0 < G.nout; j0 += 256) {
    __syncthreads();
    const int j = j0 + threadIdx.x;
    if (j < G.nout) {
      sxy[threadIdx.x] = G.xy[j];
      const double h = G.sp[j] * hs;
      sh2[threadIdx.x] = 1.0 / (h * h);
    }
    __syncthreads();
    const int jt = min(256, G.nout - j0);
    for (int k = 0; k < jt; ++k) {
      const double dx = p.x - sxy[k].x, dy = p.y - sxy[k].y;
      best = fmin(best, (dx * dx + dy * dy) * sh2[k]);
    }
  }
  if (i < nb) d2h[i] = best;
}

// Per body: radius of the smallest centroid-centred disc holding its nodes,
// and its node spacing (mean speed x 2 pi / n); per wall cluster (nwt of them, 8 to a
// CTA behind the bodies') the distance from its centre within which its nodes' near
// targets lie.  Clears the count of k_stress_wall's list.
__global__ void __launch_bounds__(256)
k_body_extent(GeoDev G, const int4* __restrict__ tiles, const double* __restrict__ rad, int nwt,
              double2* __restrict__ ext, int* __restrict__ wcount) {
  __shared__ double red[32];
  if (blockIdx.x == 0 && threadIdx.x == 0) *wcount = 0;
  if ((int)blockIdx.x >= G.M) {
    const int t = 8 * ((int)blockIdx.x - G.M) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= nwt) return;
    const int4 W = tiles[t];
    double hm = lane < W.y ? G.sp[W.x + lane] * (EB_TWOPI / G.nout) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) hm = fmax(hm, __shfl_xor_sync(0xffffffffu, hm, o));
    if (lane == 0) ext[G.M + t] = make_double2(rad[t] + STRESS_NEAR_H * hm, 0.0);
    return;
  }
  const int b = blockIdx.x;
  const double2 c = G.cen[b];
  double r = 0.0;
  for (int k = threadIdx.x; k < G.n; k += blockDim.x) {
    const double2 p = G.xy[G.nout + b * G.n + k];
    r = fmax(r, sqrt((p.x - c.x) * (p.x - c.x) + (p.y - c.y) * (p.y - c.y)));
  }
  // block max: within each warp, then across the warps
  for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(0xffffffffu, r, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x < 32) {
    r = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(0xffffffffu, r, o));
    if (threadIdx.x == 0) ext[b] = make_double2(r, G.rb[b] * EB_TWOPI / G.n);
  }
}

// Appends the lanes' nodes i with take set to the list of k_stress_wall (all lanes of a
// warp call it).
__device__ __forceinline__ void wall_list_add(bool take, int i, int* __restrict__ wcount, int* __restrict__ wlist) {
  const unsigned m = __ballot_sync(0xffffffffu, take);
  if (!m) return;
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(wcount, __popc(m));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (take) wlist[at + __popc(m & ((1u << lane) - 1u))] = i;
}

// Near mask of the stress: bit c of mask[i * mw + c/32] is set when body node
// i lies within STRESS_NEAR_H node spacings of source curve c (its own body
// excluded): for the wall from k_stress_wall_dist, for a body by its bounding
// disc.
__global__ void __launch_bounds__(256)
k_stress_near_mask(GeoDev G, const double* __restrict__ wall_d2h, const double2* __restrict__ ext, int mw,
                   unsigned* __restrict__ mask, int* __restrict__ wcount, int* __restrict__ wlist) {
  const int nb = G.n * G.M;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  wall_list_add(i < nb && wall_d2h[i] <= STRESS_NEAR_H * STRESS_NEAR_H, i, wcount, wlist);
  if (i >= nb) return;
  const int own = 1 + i / G.n;
  const double2 p = G.xy[G.nout + i];
  for (int w = 0; w < mw; ++w) {
    unsigned bits = 0u;
    for (int q = 0; q < 32; ++q) {
      const int c = 32 * w + q;
      if (c > G.M) break;
      bool near;
      if (c == 0) {
        near = wall_d2h[i] <= STRESS_NEAR_H * STRESS_NEAR_H;
      } else if (c == own) {
        near = false;
      } else {
        const double2 cc = G.cen[c - 1], e = ext[c - 1];
        const double R = e.x + STRESS_NEAR_H * e.y;
        const double dx = p.x - cc.x, dy = p.y - cc.y;
        near = dx * dx + dy * dy <= R * R;
      }
      if (near) bits |= 1u << q;
    }
    mask[(size_t)i * mw + w] = bits;
  }
}

// The mask of k_stress_near_mask with the clusters at hand: CTA = item (32 nodes
// of a body cluster, one per lane).  A curve or wall cluster is tested node by
// node only when its disc, widened by STRESS_NEAR_H of its spacings, reaches
// the disc of the item's cluster; the warps share the words of the mask and the
// wall's clusters, whose reach k_body_extent has left behind the bodies' extents.
// 4.8 us at 37 bodies x 200 nodes and 15 us at 400 x 256 (every warp measuring every
// wall cluster's spacing: 7.1 and 55 us; every node against every body and wall node:
// 35 and 334 us).
__global__ void __launch_bounds__(256)
k_stress_near_items(GeoDev G, const int2* __restrict__ items, const int4* __restrict__ tiles, int nwt,
                    const double2* __restrict__ cen, const double* __restrict__ rad, const double2* __restrict__ ext,
                    int mw, unsigned* __restrict__ mask, int* __restrict__ wcount, int* __restrict__ wlist) {
  __shared__ unsigned wall[8][32];
  const int2 it = items[blockIdx.x];
  const int4 T = tiles[it.x];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = min(it.y + lane, T.y - 1), i = T.x + k - G.nout, own = T.z;
  const double2 p = G.xy[T.x + k], ct = cen[it.x];
  const double rt = rad[it.x];
  const double hs = EB_TWOPI / G.nout;
  unsigned nearw = 0u;
  for (int t0 = 0; t0 < nwt; t0 += 256) {   // neighbouring clusters to different warps
    const int tl = t0 + 8 * lane + wid;
    bool cand = false;
    if (tl < nwt) {
      const double reach = rt + ext[G.M + tl].x;
      cand = cabs2(csub(ct, cen[tl])) <= reach * reach * 1.0001;
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, cand); todo; todo &= todo - 1u) {
      const int4 W = tiles[t0 + 8 * (__ffs(todo) - 1) + wid];
      const double hl = lane < W.y ? G.sp[W.x + lane] * hs : 0.0;
      const double2 xl = G.xy[W.x + min(lane, W.y - 1)];
      const double ih2 = 1.0 / (hl * hl);
      for (int j = 0; j < W.y; ++j) {
        const double wx = __shfl_sync(0xffffffffu, xl.x, j), wy = __shfl_sync(0xffffffffu, xl.y, j);
        const double w2 = __shfl_sync(0xffffffffu, ih2, j);
        const double dx = p.x - wx, dy = p.y - wy;
        if ((dx * dx + dy * dy) * w2 <= STRESS_NEAR_H * STRESS_NEAR_H) nearw = 1u;
      }
    }
  }
  wall[wid][lane] = nearw;
  __syncthreads();
  for (int w = wid; w < mw; w += 8) {
    const int c = 32 * w + lane;
    bool cand = false;
    double2 cc = make_double2(0, 0);
    double R = 0.0;
    if (c >= 1 && c <= G.M && c != own) {
      cc = G.cen[c - 1];
      const double2 e = ext[c - 1];
      R = e.x + STRESS_NEAR_H * e.y;
      const double reach = rt + R;
      cand = cabs2(csub(ct, cc)) <= reach * reach * 1.0001;
    }
    unsigned todo = __ballot_sync(0xffffffffu, cand), bits = 0u;
    while (todo) {
      const int q = __ffs(todo) - 1;
      todo &= todo - 1u;
      const double cx = __shfl_sync(0xffffffffu, cc.x, q), cy = __shfl_sync(0xffffffffu, cc.y, q);
      const double Rq = __shfl_sync(0xffffffffu, R, q);
      const double dx = p.x - cx, dy = p.y - cy;
      if (dx * dx + dy * dy <= Rq * Rq) bits |= 1u << q;
    }
    if (w == 0) {
      unsigned any = 0u;
#pragma unroll
      for (int v = 0; v < 8; ++v) any |= wall[v][lane];
      bits |= any;
      wall_list_add(any != 0u && it.y + lane < T.y, i, wcount, wlist);
    }
    if (it.y + lane < T.y) mask[(size_t)i * mw + w] = bits;
  }
}

// Barycentric Stokes DLP gradient of the near source bodies only: CTA =
// NEAR_T nodes of one body, one per lane of every warp; the CTA visits,
// in order, every body that is near for at least one of its nodes, and a
// node keeps the value only for the bodies near to it.  With 32 nodes a CTA
// visits fewer curves that only some of its nodes need than with 128, and the
// warps share each curve's nodes (bary_eval).  out[q * nb + i], q as
// k_bary_sum (one split).
__global__ void __launch_bounds__(NEAR_NT, 2)
k_bary_sum_near(GeoDev G, const double2* __restrict__ bd_all, const unsigned* __restrict__ mask, int mw,
                double* __restrict__ out) {
  __shared__ BaryTile T;
  const int nb = G.n * G.M;
  const int per = (G.n + NEAR_T - 1) / NEAR_T, b = blockIdx.x / per;
  const int k = NEAR_T * (blockIdx.x - b * per) + (threadIdx.x & 31);
  const bool act = k < G.n;
  const int t = b * G.n + k, tc = act ? t : b * G.n + G.n - 1;
  const double2 zt = G.xy[G.nout + tc];
  double a[6] = {0, 0, 0, 0, 0, 0};
  for (int w = 0; w < mw; ++w) {
    unsigned my = act ? mask[(size_t)tc * mw + w] : 0u;
    if (w == 0) my &= ~1u;   // the wall: k_stress_wall
    unsigned bits = __reduce_or_sync(0xffffffffu, my);   // the same in every warp
    while (bits) {
      const int q = __ffs(bits) - 1;
      bits &= bits - 1u;
      const int c = 32 * w + q;
      DLPVal r = bary_eval<2>(T, G, c, bd_all + bd_all_off(G, c), zt, act);
      if ((my >> q) & 1u) {
        a[0] += r.ux; a[1] += r.uy; a[2] += r.u1x; a[3] += r.u1y; a[4] += r.u2x; a[5] += r.u2y;
      }
    }
  }
  if (act && threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < 6; ++q) out[(size_t)q * nb + t] = a[q];
  }
}

// Adds the wall's to out of k_bary_sum_near, for the nodes near to it (wlist, *wcount of
// them in any order): a cluster of STRESS_CL CTAs takes 32 of them at a time, its CTAs
// 1/STRESS_CL of the wall's nodes each.  Bound by the FP64 pipe.  Within
// k_bary_sum_near a CTA near the wall had the whole wall in one chain, for a third of
// its lanes on average, and the chip was half idle: both together took 463 us at 400 bodies
// x 256 nodes and a wall of 4096 and 69 us at 37 x 200, this takes 235 and 16 us and the
// bodies' 88 and 47 us.
constexpr int STRESS_CL = 8;
__global__ void __cluster_dims__(STRESS_CL, 1, 1) __launch_bounds__(NEAR_NT, 2)
k_stress_wall(GeoDev G, const double2* __restrict__ bd_all, const int* __restrict__ wcount,
              const int* __restrict__ wlist, double* __restrict__ out) {
  __shared__ BaryTile T;
  const int nb = G.n * G.M, cnt = *wcount;
  for (int p0 = 32 * (blockIdx.x / STRESS_CL); p0 < cnt; p0 += 32 * (gridDim.x / STRESS_CL)) {
    const int p = p0 + (threadIdx.x & 31);
    const bool act = p < cnt;
    const int t = wlist[act ? p : cnt - 1];
    const DLPVal r = bary_eval<2, STRESS_CL>(T, G, 0, bd_all + bd_all_off(G, 0), G.xy[G.nout + t], act);
    if (act && threadIdx.x < 32 && blockIdx.x % STRESS_CL == 0) {
      const double v[6] = {r.ux, r.uy, r.u1x, r.u1y, r.u2x, r.u2y};
#pragma unroll
      for (int q = 0; q < 6; ++q) out[(size_t)q * nb + t] += v[q];
    }
  }
  cooperative_groups::this_cluster().sync();   // no CTA's shared memory goes before the others have read it
}

// Per body: the speed-weighted rigid part of its density, sigma_rigid(x) =
// (t1, t2) + t3 (-(y - yb), x - xb) with (xb, yb) the speed-weighted centroid
// (the split k_prep makes for the far field), as rig[5 b + (0..4)] = t1, t2,
// t3, xb, yb.
__global__ void __launch_bounds__(256)
k_stress_rigid(GeoDev G, const double* __restrict__ den, double* __restrict__ rig) {
  __shared__ double sh[32];
  const int b = blockIdx.x, start = G.nout + b * G.n;
  double a0 = 0, a1 = 0, s0 = 0, sxw = 0, syw = 0;
  for (int j = threadIdx.x; j < G.n; j += blockDim.x) {
    const int g = start + j;
    const double sp = G.sp[g];
    const double2 p = G.xy[g];
    a0 += den[ix_of(G, g)] * sp;
    a1 += den[iy_of(G, g)] * sp;
    s0 += sp;
    sxw += sp * p.x;
    syw += sp * p.y;
  }
  a0 = block_sum<256>(a0, sh);
  a1 = block_sum<256>(a1, sh);
  s0 = block_sum<256>(s0, sh);
  sxw = block_sum<256>(sxw, sh);
  syw = block_sum<256>(syw, sh);
  const double xb = sxw / s0, yb = syw / s0;
  double r0 = 0, r1 = 0;
  for (int j = threadIdx.x; j < G.n; j += blockDim.x) {
    const int g = start + j;
    const double sp = G.sp[g];
    const double2 p = G.xy[g];
    const double fx = -(p.y - yb), fy = p.x - xb;
    r0 += sp * (fx * den[ix_of(G, g)] + fy * den[iy_of(G, g)]);
    r1 += sp * (fx * fx + fy * fy);
  }
  r0 = block_sum<256>(r0, sh);
  r1 = block_sum<256>(r1, sh);
  if (threadIdx.x == 0) {
    rig[5 * b] = a0 / s0;
    rig[5 * b + 1] = a1 / s0;
    rig[5 * b + 2] = r1 > 0 ? r0 / r1 : 0.0;
    rig[5 * b + 3] = xb;
    rig[5 * b + 4] = yb;
  }
}

// Trapezoid deformation tensor of every other curve except the near ones
// (mask as k_stress_near_mask), as partial sums over the far-field tile
// splits: out[(split*3 + q)*nb + i].  The same terms as k_stress_trap, the
// density scaled by the weight when staged and the reciprocal by
// rcp_newton.  A source body's density enters without its rigid part
// (k_stress_rigid): a rigid-motion density has no exterior double layer, and
// at these distances the trapezoid rule's value for it is below 1e-16 of its
// size, while the rigid parts (large for the smallest bodies) would otherwise
// set the rounding error of the sum.
__global__ void __launch_bounds__(256)
k_stress_far(GeoDev G, const double* __restrict__ den, const int4* __restrict__ tiles,
             const int* __restrict__ split_ptr, const unsigned* __restrict__ mask, int mw,
             const double* __restrict__ rig, double* __restrict__ out) {
  __shared__ double4 sg[FAR_TS];   // x, y, nx, ny
  __shared__ double2 ss[FAR_TS];   // w sigma
  const int nb = G.n * G.M;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < nb;
  const int ic = act ? i : nb - 1;
  const int g = G.nout + ic;
  const int mycurve = 1 + ic / G.n;
  const double2 p = G.xy[g];
  double e11 = 0, e12 = 0, e22 = 0;
  const int split = blockIdx.y;
  for (int ti = split_ptr[split]; ti < split_ptr[split + 1]; ++ti) {
    const int4 T = tiles[ti];
    __syncthreads();
    for (int k = threadIdx.x; k < T.y; k += blockDim.x) {
      const int gs = T.x + k;
      const double2 q = G.xy[gs], nn = G.nrm[gs];
      const double wg = G.w[gs];
      sg[k] = make_double4(q.x, q.y, nn.x, nn.y);
      double sx = den[ix_of(G, gs)], sy = den[iy_of(G, gs)];
      if (T.z > 0) {
        const double* R = rig + 5 * (T.z - 1);
        sx -= R[0] - R[2] * (q.y - R[4]);
        sy -= R[1] + R[2] * (q.x - R[3]);
      }
      ss[k] = make_double2(sx * wg, sy * wg);
    }
    __syncthreads();
    if (T.z == mycurve || ((__ldg(mask + (size_t)ic * mw + (T.z >> 5)) >> (T.z & 31)) & 1u)) continue;
    double a11 = 0, a12 = 0, a22 = 0;
#pragma unroll 2
    for (int j = 0; j < T.y; ++j) {
      const double4 q = sg[j];
      const double2 sd = ss[j];
      const double rx = p.x - q.x, ry = p.y - q.y;
      const double inv = rcp_newton(fma(rx, rx, ry * ry));
      const double i4 = inv * inv;
      const double rdn = fma(rx, q.z, ry * q.w), rtn = fma(rx, q.w, ry * q.z);
      const double rds = fma(rx, sd.x, ry * sd.y), rts = fma(rx, sd.y, ry * sd.x);
      const double A = rdn * rds * i4;
      const double C = 4.0 * A * inv;
      a11 += A + i4 * rx * fma(rds, q.z, rdn * sd.x) - C * rx * rx;
      a22 += A + i4 * ry * fma(rds, q.w, rdn * sd.y) - C * ry * ry;
      a12 += 0.5 * i4 * fma(rds, rtn, rdn * rts) - C * rx * ry;
    }
    e11 += a11; e12 += a12; e22 += a22;
  }
  if (act) {
    out[((size_t)split * 3 + 0) * nb + i] = e11;
    out[((size_t)split * 3 + 1) * nb + i] = e12;
    out[((size_t)split * 3 + 2) * nb + i] = e22;
  }
}

// Deformation tensor assembly, stokeslet/rotlet gradients (:2964-2994; the
// trapezoid variant flips the sign of the rotlet's E22 term, :2604-2605),
// traction -2 E n and shear stress tau = f.(p_y, -p_x) (:3075-3092).
// part_b: barycentric partial sums (6 per split, NDER = 2 layout of
// k_bary_sum), part_t: trapezoid partial sums (3 per split, k_stress_trap and
// k_stress_far layout); either count may be zero.
__global__ void __launch_bounds__(256)
k_stress_final(GeoDev G, const double* __restrict__ den, const double* __restrict__ part_b, int nsplit_b,
               const double* __restrict__ part_t, int nsplit_t, int bary, const double* __restrict__ eself,
               double* __restrict__ tau, double* __restrict__ Eout) {
  __shared__ double4 sc[SR_CHUNK];
  __shared__ double sr[SR_CHUNK];
  const int nb = G.n * G.M;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool act = i < nb;
  const int ic = act ? i : nb - 1;
  double e11 = 0, e12 = 0, e22 = 0;
  for (int s = 0; s < nsplit_b; ++s) {
    const double* P = part_b + (size_t)s * 6 * nb;
    e11 += P[2 * (size_t)nb + ic];
    e12 += 0.5 * (P[3 * (size_t)nb + ic] + P[4 * (size_t)nb + ic]);
    e22 += P[5 * (size_t)nb + ic];
  }
  for (int s = 0; s < nsplit_t; ++s) {
    const double* P = part_t + (size_t)s * 3 * nb;
    e11 += P[ic];
    e12 += P[(size_t)nb + ic];
    e22 += P[2 * (size_t)nb + ic];
  }
  e11 += eself[ic];
  e12 += eself[nb + ic];
  e22 += eself[2 * nb + ic];
  const int g = G.nout + ic;
  const double2 p = G.xy[g];
  for (int b0 = 0; b0 < G.M; b0 += SR_CHUNK) {
    __syncthreads();
    for (int t = threadIdx.x; t < SR_CHUNK; t += blockDim.x) {
      int b = b0 + t;
      if (b < G.M) {
        double2 cc = G.cen[b];
        sc[t] = make_double4(cc.x, cc.y, den[ic_of(G, b, 0)], den[ic_of(G, b, 1)]);
        sr[t] = den[ic_of(G, b, 2)];
      }
    }
    __syncthreads();
    const int bt = min(SR_CHUNK, G.M - b0);
    for (int t = 0; t < bt; ++t) {
      const double4 q = sc[t];
      const double rot = sr[t];
      const double rx = p.x - q.x, ry = p.y - q.y;
      const double rho2 = rx * rx + ry * ry;
      const double rd = rx * q.z + ry * q.w;
      const double ir2 = 1.0 / rho2, ir4 = ir2 * ir2;
      e11 += 0.5 / EB_TWOPI * (rd * ir2 - 2 * rx * rx * rd * ir4);
      e12 -= 1.0 / EB_TWOPI * (rd * ir4 * rx * ry);
      e22 += 0.5 / EB_TWOPI * (rd * ir2 - 2 * ry * ry * rd * ir4);
      e11 -= 2.0 * rot * rx * ry * ir4;
      e12 += rot * (rx * rx - ry * ry) * ir4;
      if (bary) e22 += 2.0 * rot * rx * ry * ir4;
      else e22 -= 2.0 * rot * rx * ry * ir4;
    }
  }
  if (!act) return;
  const double2 nn = G.nrm[g];
  const double tx = -2.0 * e11 * nn.x - 2.0 * e12 * nn.y;
  const double ty = -2.0 * e12 * nn.x - 2.0 * e22 * nn.y;
  tau[i] = tx * nn.y - ty * nn.x;
  if (Eout) {
    Eout[i] = e11;
    Eout[nb + i] = e12;
    Eout[2 * nb + i] = e22;
  }
}

// The same assembly when the strain of the other curves comes by clusters:
// near: barycentric strain (layout of k_bary_sum_near); part: nslot slots of
// (E11, E12) per node, E22 = -E11; the stokeslets and rotlets of the bodies in
// the node's near list and its own are summed here, the others came with the
// expansions (sing = 0: all bodies are summed here).  COMBINE_G threads share a
// node.
__global__ void __launch_bounds__(256)
k_stress_assemble(GeoDev G, const double* __restrict__ den, ClView L, const int4* __restrict__ tiles, int sing,
                  const double* __restrict__ near, const double2* __restrict__ part, int nslot,
                  const double* __restrict__ eself, double* __restrict__ tau, double* __restrict__ Eout) {
  const int nb = G.n * G.M;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(tid / COMBINE_G), sub = (int)(tid % COMBINE_G);
  const bool act = i < nb;
  const int ic = act ? i : nb - 1, g = G.nout + ic;
  const double2 p = G.xy[g];
  double e11 = 0, e12 = 0, e22 = 0;
  for (int s = sub; s < nslot; s += COMBINE_G) {
    const double2 v = part[(size_t)s * G.N + g];
    e11 += v.x;
    e12 += v.y;
    e22 -= v.x;
  }
  auto singular = [&](int b) {
    const double2 c = G.cen[b];
    const double lx = den[ic_of(G, b, 0)], ly = den[ic_of(G, b, 1)], rot = den[ic_of(G, b, 2)];
    const double rx = p.x - c.x, ry = p.y - c.y;
    const double rd = rx * lx + ry * ly;
    const double ir2 = 1.0 / (rx * rx + ry * ry), ir4 = ir2 * ir2;
    e11 += 0.5 / EB_TWOPI * (rd * ir2 - 2 * rx * rx * rd * ir4) - 2.0 * rot * rx * ry * ir4;
    e12 += rot * (rx * rx - ry * ry) * ir4 - 1.0 / EB_TWOPI * (rd * ir4 * rx * ry);
    e22 += 0.5 / EB_TWOPI * (rd * ir2 - 2 * ry * ry * rd * ir4) + 2.0 * rot * rx * ry * ir4;
  };
  if (sing) {
    const int t = tile_of(G, g), own = tiles[t].z;
    const int2 c4 = L.ncnt[t];
    for (int e = c4.x - 1 + sub; e < c4.y; e += COMBINE_G)
      singular((e < c4.x ? own : tiles[L.near[(size_t)t * L.T + e]].z) - 1);
  } else {
    for (int b = sub; b < G.M; b += COMBINE_G) singular(b);
  }
  if (sub == 0) {
    e11 += near[2 * (size_t)nb + ic] + eself[ic];
    e12 += 0.5 * (near[3 * (size_t)nb + ic] + near[4 * (size_t)nb + ic]) + eself[nb + ic];
    e22 += near[5 * (size_t)nb + ic] + eself[2 * nb + ic];
  }
#pragma unroll
  for (int o = 1; o < COMBINE_G; o <<= 1) {
    e11 += __shfl_xor_sync(0xffffffffu, e11, o);
    e12 += __shfl_xor_sync(0xffffffffu, e12, o);
    e22 += __shfl_xor_sync(0xffffffffu, e22, o);
  }
  if (!act || sub != 0) return;
  const double2 nn = G.nrm[g];
  const double tx = -2.0 * e11 * nn.x - 2.0 * e12 * nn.y;
  const double ty = -2.0 * e12 * nn.x - 2.0 * e22 * nn.y;
  tau[i] = tx * nn.y - ty * nn.x;
  if (Eout) {
    Eout[i] = e11;
    Eout[nb + i] = e12;
    Eout[2 * nb + i] = e22;
  }
}

// Trapezoid pressure (always) and velocity/vorticity (VEL: ibary = 0) at targets
// from every node (:3170-3197, :3225-3255).  CTA = 32 targets, one per lane, and
// part blockIdx.y of the source tiles; its 8 warps split a tile's sources.
// out[(part*4 + q)*ntar + t], q = u, v, p, w.  Bound by the FP64 pipe: 3200
// targets and 7424 nodes 47 us (a thread per target, three divisions a pair,
// 132 us).
template <bool VEL>
__global__ void __launch_bounds__(256)
k_qoi_trap(GeoDev G, const double* __restrict__ den, const int4* __restrict__ tiles, int ntile, int ntar,
           const double2* __restrict__ txy, double* __restrict__ out) {
  __shared__ double4 sg[FAR_TS];   // x, y, nx, ny
  __shared__ double4 sd[FAR_TS];   // w sigma, w n.sigma
  __shared__ double red[NEAR_W / 2][4][32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, t = 32 * blockIdx.x + lane;
  const bool act = t < ntar;
  const double2 p = txy[act ? t : ntar - 1];
  double a[4] = {0, 0, 0, 0};
  int ti = (int)((long long)ntile * blockIdx.y / gridDim.y);
  const int te = (int)((long long)ntile * (blockIdx.y + 1) / gridDim.y);
  while (ti < te) {
    // consecutive tiles are consecutive nodes: take as many as fit
    const int g0 = tiles[ti].x;
    int len = 0;
    __syncthreads();
    while (ti < te && len + tiles[ti].y <= FAR_TS) len += tiles[ti++].y;
    if ((int)threadIdx.x < len) {
      const int g = g0 + threadIdx.x;
      const double2 q = G.xy[g], nn = G.nrm[g];
      const double wg = G.w[g], sx = wg * den[ix_of(G, g)], sy = wg * den[iy_of(G, g)];
      sg[threadIdx.x] = make_double4(q.x, q.y, nn.x, nn.y);
      sd[threadIdx.x] = make_double4(sx, sy, nn.x * sx + nn.y * sy, 0.0);
    }
    __syncthreads();
    const int kb = len * (wid + 1) / NEAR_W;
#pragma unroll 2
    for (int j = len * wid / NEAR_W; j < kb; ++j) {
      const double4 q = sg[j], s = sd[j];
      const double rx = p.x - q.x, ry = p.y - q.y;
      const double i2 = rcp_raw64(fma(rx, rx, ry * ry));
      const double rdn = fma(rx, q.z, ry * q.w), rds = fma(rx, s.x, ry * s.y);
      const double m = rdn * rds * i2 * i2;
      a[2] += fma(2.0, m, -s.z * i2);
      if (VEL) {
        const double rn = fma(-rx, q.w, ry * q.z), rs = fma(-rx, s.y, ry * s.x);
        a[0] = fma(m, rx, a[0]);
        a[1] = fma(m, ry, a[1]);
        a[3] = fma(fma(rds, rn, rdn * rs), i2 * i2, a[3]);
      }
    }
  }
  __syncthreads();
  near_reduce(a, red);
  if (act && wid == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) out[((size_t)blockIdx.y * 4 + q) * ntar + t] = a[q];
  }
}

// Nearest body node of 32 targets (one per lane), the first minimum in body-major
// order, among part blockIdx.y of the nodes: the warps split them, in order, and meet
// in order.  dist[part*ntar + t], idx[...].
__global__ void __launch_bounds__(256)
k_qoi_nearest(GeoDev G, int ntar, const double2* __restrict__ txy, double* __restrict__ dist, int* __restrict__ idx) {
  __shared__ double dm[NEAR_W][32];
  __shared__ int di[NEAR_W][32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, t = 32 * blockIdx.x + lane;
  const double2 p = txy[min(t, ntar - 1)];
  const long long nb = (long long)G.n * G.M, parts = (long long)NEAR_W * gridDim.y, w0 = (long long)NEAR_W * blockIdx.y + wid;
  double dmin = 1e10;
  int ind = 0;
  const int hi = (int)(nb * (w0 + 1) / parts);
#pragma unroll 4
  for (int i = (int)(nb * w0 / parts); i < hi; ++i) {
    const double2 q = G.xy[G.nout + i];
    const double d2 = (p.x - q.x) * (p.x - q.x) + (p.y - q.y) * (p.y - q.y);
    if (d2 < dmin) { dmin = d2; ind = i; }
  }
  dm[wid][lane] = dmin;
  di[wid][lane] = ind;
  __syncthreads();
  if (wid != 0 || t >= ntar) return;
  for (int w = 1; w < NEAR_W; ++w)
    if (dm[w][lane] < dmin) { dmin = dm[w][lane]; ind = di[w][lane]; }
  dist[(size_t)blockIdx.y * ntar + t] = dmin;
  idx[(size_t)blockIdx.y * ntar + t] = ind;
}

// Final assembly at targets: barycentric velocity and vorticity (:3199-3212,
// :3257-3270), stokeslets/rotlets (:3275-3298), and zeroing of targets that
// classifyPointsOld (:4420-4500) puts inside a body (:3301-3309): the nearest
// body node (npart candidates of k_qoi_nearest, in order) decides the side through the
// sign of (x_t - x_k).n_k.  CTA = 32 targets, one per lane; the warps split the
// bodies.  8 us at 3200 targets and 50 bodies (with the nearest nodes searched by the same
// 100 CTAs: 52 us).
__global__ void __launch_bounds__(256)
k_qoi_final(GeoDev G, const double* __restrict__ den, int ntar, const double2* __restrict__ txy,
            const double* __restrict__ ptrap, int ns1, const double* __restrict__ pbary, int ns2, int ibary,
            const double* __restrict__ dist, const int* __restrict__ idx, int npart, double* __restrict__ uo, double* __restrict__ vo, double* __restrict__ po, double* __restrict__ wo) {
  __shared__ double red[NEAR_W / 2][4][32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, t = 32 * blockIdx.x + lane;
  const bool act = t < ntar;
  const int tc = act ? t : ntar - 1;
  const double2 p = txy[tc];
  double a[4] = {0, 0, 0, 0};   // u, v, p, w
  for (int s = wid; s < ns1; s += NEAR_W)
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] += ptrap[((size_t)s * 4 + q) * ntar + tc];
  if (ibary)
    for (int s = wid; s < ns2; s += NEAR_W) {
      const double* P = pbary + (size_t)s * 6 * ntar;
      a[0] += P[tc];
      a[1] += P[(size_t)ntar + tc];
      a[3] += P[4 * (size_t)ntar + tc] - P[3 * (size_t)ntar + tc];
    }
  for (int b = wid; b < G.M; b += NEAR_W) {
    const double2 cc = G.cen[b];
    const double s1 = den[ic_of(G, b, 0)], s2 = den[ic_of(G, b, 1)], rot = den[ic_of(G, b, 2)];
    const double rx = p.x - cc.x, ry = p.y - cc.y;
    const double rho2 = rx * rx + ry * ry, rd = rx * s1 + ry * s2;
    const double ir = 1.0 / rho2, lg = log(rho2);
    a[0] += 0.5 / EB_TWOPI * (-0.5 * lg * s1 + rd * ir * rx) + rot * ry * ir;
    a[1] += 0.5 / EB_TWOPI * (-0.5 * lg * s2 + rd * ir * ry) - rot * rx * ir;
    a[2] += 1.0 / EB_TWOPI * rd * ir;
    a[3] += (ry * s1 - rx * s2) * ir / EB_TWOPI;
  }
  near_reduce(a, red);
  if (wid != 0 || !act) return;
  if (G.M > 0) {
    double dmin = dist[t];
    int ind = idx[t];
    for (int w = 1; w < npart; ++w) {
      const double d = dist[(size_t)w * ntar + t];
      if (d < dmin) { dmin = d; ind = idx[(size_t)w * ntar + t]; }
    }
    const double2 q = G.xy[G.nout + ind], nn = G.nrm[G.nout + ind];
    const double vdn = (p.x - q.x) * nn.x + (p.y - q.y) * nn.y;
    if (!(vdn < 0.0)) a[0] = a[1] = a[2] = a[3] = 0.0;
  }
  uo[t] = a[0];
  vo[t] = a[1];
  po[t] = a[2];
  wo[t] = a[3];
}

__global__ void k_pack(int n, const double* __restrict__ x, const double* __restrict__ y, double2* __restrict__ xy) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) xy[i] = make_double2(x[i], y[i]);
}

// ---------------------------------------------------------------------------
// Host side.

// Boundary values of all curves (wall first, then every body).
static void bdval_all(State& s, const double* d_den, DBuf<double2>& bd_all, cudaStream_t st) {
  const Problem& pr = s.pr;
  bd_all.ensure(5LL * pr.nout + 5LL * pr.n * pr.M);
  k_bdval<<<nblk(pr.nout, NEAR_T) + (unsigned)pr.M * nblk(pr.n, NEAR_T), NEAR_NT, 0, st>>>(
      s.geo(), d_den, nullptr, s.dker_wall.p, s.dker_body.p, bd_all.p);
  EB_LAUNCH_CHECK();
}

int eb_num_sms();

// ---------------------------------------------------------------------------
// Pressure on the body boundaries (computePressure, stokesSolver.f:4644-4885).
// Every pair: (2 (r.n)(r.s)/rho^4 - (n.s)/rho^2) w_j with the trapezoid weight
// w = speed (2pi/n_c)/pi.  Targets: body nodes; sources: every tile, split
// over blockIdx.y.  A target's own body uses odd-even quadrature: sources of
// the other index parity only, weight doubled, density minus its value at the
// target (:4728-4787).
__global__ void __launch_bounds__(256)
k_pressure_sum(GeoDev G, const double* __restrict__ den, const int4* __restrict__ tiles,
               const int* __restrict__ split_ptr, double* __restrict__ part) {
  __shared__ double4 sg[FAR_TS];
  __shared__ double2 sd[FAR_TS];
  __shared__ double sw[FAR_TS];
  __shared__ int sl[FAR_TS];
  const int nb = G.n * G.M;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int tc = t < nb ? t : nb - 1;
  const int g = G.nout + tc;
  const int b = tc / G.n, k = tc - b * G.n, curve = 1 + b;
  const double2 p = G.xy[g];
  const double sxk = den[ix_of(G, g)], syk = den[iy_of(G, g)];
  double acc = 0.0;
  const int split = blockIdx.y;
  for (int ti = split_ptr[split]; ti < split_ptr[split + 1]; ++ti) {
    const int4 T = tiles[ti];
    __syncthreads();
    for (int q = threadIdx.x; q < T.y; q += blockDim.x) {
      const int j = T.x + q;
      const double2 xy = G.xy[j], nn = G.nrm[j];
      sg[q] = make_double4(xy.x, xy.y, nn.x, nn.y);
      sd[q] = make_double2(den[ix_of(G, j)], den[iy_of(G, j)]);
      sw[q] = G.w[j];
      sl[q] = j - curve_start(G, T.z);   // index within its curve
    }
    __syncthreads();
    const bool own = T.z == curve;
    for (int q = 0; q < T.y; ++q) {
      if (own && ((sl[q] & 1) == (k & 1))) continue;
      const double4 sq = sg[q];
      const double2 dq = sd[q];
      const double sx = own ? dq.x - sxk : dq.x, sy = own ? dq.y - syk : dq.y;
      const double rx = p.x - sq.x, ry = p.y - sq.y;
      const double rho2 = rx * rx + ry * ry;
      const double rdn = rx * sq.z + ry * sq.w, rds = rx * sx + ry * sy, dn = sq.z * sx + sq.w * sy;
      const double v = (2.0 * rdn * rds / rho2 / rho2 - dn / rho2) * sw[q];
      acc += own ? 2.0 * v : v;
    }
  }
  if (t < nb) part[(size_t)split * nb + t] = acc;
}

// Split sums, the jump -(d sigma/ds . tangent) with the spectral derivative
// (the circulant d[m] of fourierDiff) and the stokeslet pressure
// (r . lambda)/(2 pi rho^2) of every body (:4829-4881); one thread per node.
__global__ void __launch_bounds__(256)
k_pressure_final(GeoDev G, const double* __restrict__ den, const double* __restrict__ part, int nsplit,
                 const double* __restrict__ dk, double* __restrict__ out) {
  const int nb = G.n * G.M;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nb) return;
  const int b = t / G.n, k = t - b * G.n, g = G.nout + t;
  double acc = 0.0;
  for (int q = 0; q < nsplit; ++q) acc += part[(size_t)q * nb + t];
  double dx = 0.0, dy = 0.0;
  for (int j = 0; j < G.n; ++j) {
    int m = k - j;
    if (m < 0) m += G.n;
    const double d = __ldg(dk + m);
    const int gj = G.nout + b * G.n + j;
    dx = fma(d, den[ix_of(G, gj)], dx);
    dy = fma(d, den[iy_of(G, gj)], dy);
  }
  const double2 nn = G.nrm[g];
  const double spd = G.sp[g];
  acc -= (dx / spd) * (-nn.y) + (dy / spd) * nn.x;
  const double2 p = G.xy[g];
  for (int s = 0; s < G.M; ++s) {
    const double2 c = G.cen[s];
    const double rx = p.x - c.x, ry = p.y - c.y;
    acc += (rx * den[ic_of(G, s, 0)] + ry * den[ic_of(G, s, 1)]) / (EB_TWOPI * (rx * rx + ry * ry));
  }
  out[t] = acc;
}

// Parts of the source curves for ntasks CTAs of targets: about four CTAs per SM.
static int source_splits(int ntasks, int ncurves) {
  return std::max(1, std::min((4 * eb_num_sms() + ntasks - 1) / std::max(ntasks, 1), ncurves));
}

// The same for k_bary_sum, two CTAs of which an SM holds: the parts, up to eight CTAs per
// SM, with the least time in whole waves of them.  3200 targets (100 CTAs) against 50
// x 128 + 1024 nodes: 11 parts (3.7 waves) 325 us, 6 (2.03 waves) 382 us.
static int bary_splits(int ntasks, int ncurves) {
  const long long slots = 2 * eb_num_sms();
  int best = 1;
  auto waves = [&](int p) { return ((long long)ntasks * p + slots - 1) / slots; };
  for (int p = 2; p <= ncurves && (long long)ntasks * p <= 4 * slots; ++p)
    if (waves(p) * best < waves(best) * p) best = p;
  return best;
}

void body_pressure(State& s, const double* d_den, double* d_p) {
  const Problem& pr = s.pr;
  const GeoDev G = s.geo();
  const int nb = pr.n * pr.M;
  if (nb == 0) return;
  static DBuf<double> part;
  part.ensure((size_t)s.nsplit * nb);
  k_pressure_sum<<<dim3(nblk(nb, 256), s.nsplit), 256, 0, s.st>>>(G, d_den, s.tiles.p, s.split_ptr.p, part.p);
  EB_LAUNCH_CHECK();
  k_pressure_final<<<nblk(nb, 256), 256, 0, s.st>>>(G, d_den, part.p, s.nsplit, s.dker_body.p, d_p);
  EB_LAUNCH_CHECK();
}

void shear_stress(State& s, const double* d_den, double* d_tau, double* d_E) {
  const Problem& pr = s.pr;
  const GeoDev G = s.geo();
  const int nb = pr.n * pr.M;
  if (nb == 0) return;
  static DBuf<double> eself, part;
  static DBuf<double2> bd_all;
  eself.ensure(3LL * nb);
  const int bary = pr.P.ibary == 1;
  // By clusters, a branch takes the bodies' own strain, the boundary values and the
  // barycentric sums, the library stream the near lists and the expansions: neither
  // half fills the chip with its last CTAs and its short launches.  A call at 400 bodies
  // x 256 nodes takes 1.80 ms, 2.05 with one after the other; at 37 x 200 0.33 and 0.41.
  const bool branch = bary && !pr.P.stress_all_bary && s.cl_ready;
  cudaStream_t side = s.st;
  if (branch) {
    ensure_branches(s);
    side = s.br[0];
    EB_CK(cudaEventRecord(s.ev_fork[0], s.st));
    EB_CK(cudaStreamWaitEvent(side, s.ev_fork[0], 0));
  }
  k_stress_self<<<pr.M * nblk(pr.n, 32), NEAR_NT, 0, side>>>(G, d_den, s.dker_body.p, eself.p);
  EB_LAUNCH_CHECK();
  if (bary && pr.P.stress_all_bary) {   // every pair barycentric, as the reference evaluates it
    bdval_all(s, d_den, bd_all, s.st);
    const int tasks = pr.M * (int)nblk(pr.n, NEAR_T), nsplit = bary_splits(tasks, pr.M + 1);
    part.ensure((size_t)nsplit * 6 * nb);
    bary_sum(s, tasks, nsplit, bd_all.p, s.xy.p + pr.nout, 1, nb, part.p);
    k_stress_final<<<nblk(nb, 256), 256, 0, s.st>>>(G, d_den, part.p, nsplit, nullptr, 0, 1, eself.p, d_tau, d_E);
    EB_LAUNCH_CHECK();
  } else if (bary) {   // barycentric near pairs, trapezoid elsewhere
    static DBuf<double> wall_d2h;
    static DBuf<double2> ext;
    static DBuf<unsigned> smask;
    static DBuf<double> pnear;
    const int mw = (pr.M + 1 + 31) / 32;
    static DBuf<int> wlist;   // the nodes near the wall, their count at [nb]
    wlist.ensure((size_t)nb + 1);
    const int nwt = s.cl_ready ? s.nwall_tiles : 0;
    k_body_extent<<<pr.M + nblk(nwt, 8), 256, 0, s.st>>>(G, s.tiles.p, s.cl_rad.p, nwt, ext.ensure(pr.M + nwt),
                                                         wlist.p + nb);
    EB_LAUNCH_CHECK();
    const unsigned wall_ctas =
        STRESS_CL * std::max(1u, std::min(nblk(nb, 32), (unsigned)(2 * eb_num_sms() / STRESS_CL)));
    smask.ensure((size_t)nb * mw);
    pnear.ensure(6LL * nb);
    bdval_all(s, d_den, bd_all, side);
    const unsigned near_ctas = pr.M * nblk(pr.n, NEAR_T);
    if (s.cl_ready) {
      const int2* items = s.items32.p + s.n_items32_wall;
      const int nit = s.n_items32 - s.n_items32_wall;
      k_stress_near_items<<<nit, 256, 0, s.st>>>(G, items, s.tiles.p, s.nwall_tiles, s.cl_cen.p, s.cl_rad.p, ext.p, mw,
                                                 smask.p, wlist.p + nb, wlist.p);
      EB_LAUNCH_CHECK();
      EB_CK(cudaEventRecord(s.ev_fork[1], s.st));
      EB_CK(cudaStreamWaitEvent(side, s.ev_fork[1], 0));
      k_bary_sum_near<<<near_ctas, NEAR_NT, 0, side>>>(G, bd_all.p, smask.p, mw, pnear.p);
      EB_LAUNCH_CHECK();
      k_stress_wall<<<wall_ctas, NEAR_NT, 0, side>>>(G, bd_all.p, wlist.p + nb, wlist.p, pnear.p);
      EB_LAUNCH_CHECK();
      EB_CK(cudaEventRecord(s.ev_join[0], side));
      // strengths without the bodies' rigid parts (see k_stress_rigid), the
      // near lists of this mask, their strain and that of the expansions
      ClLists& lists = s.cl_stress;
      k_prep<<<pr.M + nblk(pr.nout, 256), 256, 0, s.st>>>(G, d_den, s.ws.p, s.sq64.p, s.sq32.p, s.d_w.ensure(pr.ntot), s.sigdotn.p, 1);
      EB_LAUNCH_CHECK();
      build_lists(s, lists, s.nwall_tiles, smask.p, mw, pr.nout, s.cl_expand, true, nullptr);
      const ClView L = cl_view(s, lists);
      const int parts = near_parts(nit, eb_num_sms());
      s.partial.ensure((size_t)(parts + 1) * pr.N);
      k_cl_near64<true, true><<<dim3(nit, parts), 256, 0, s.st>>>(G, L, items, s.tiles.p, 0, s.sq64.p, smask.p, mw,
                                                                  pr.nout, s.partial.p);
      EB_LAUNCH_CHECK();
      if (s.cl_expand) {
        k_cl_form<CL_P / 8><<<s.ntile, 256, 0, s.st>>>(G, 0, s.tiles.p, s.cl_cen.p, s.cl_rad.p, s.sq64.p,
                                             s.cl_sing ? d_den : nullptr, s.cl_mp.p, s.cl_lam.p);
        EB_LAUNCH_CHECK();
        k_cl_shift_strain<<<s.ntile - s.nwall_tiles, 256, 0, s.st>>>(G, L, s.nwall_tiles, s.tiles.p, s.cl_mp.p,
                                                                     s.cl_lam.p, s.partial.p + (size_t)parts * pr.N);
        EB_LAUNCH_CHECK();
      }
      EB_CK(cudaStreamWaitEvent(s.st, s.ev_join[0], 0));
      k_stress_assemble<<<nblk((long long)nb * COMBINE_G, 256), 256, 0, s.st>>>(
          G, d_den, L, s.tiles.p, s.cl_sing, pnear.p, s.partial.p, parts + (s.cl_expand ? 1 : 0), eself.p, d_tau, d_E);
      EB_LAUNCH_CHECK();
      return;
    }
    k_stress_wall_dist<<<nblk(nb, 256), 256, 0, s.st>>>(G, wall_d2h.ensure(nb));
    EB_LAUNCH_CHECK();
    k_stress_near_mask<<<nblk(nb, 256), 256, 0, s.st>>>(G, wall_d2h.p, ext.p, mw, smask.p, wlist.p + nb, wlist.p);
    EB_LAUNCH_CHECK();
    k_bary_sum_near<<<near_ctas, NEAR_NT, 0, s.st>>>(G, bd_all.p, smask.p, mw, pnear.p);
    EB_LAUNCH_CHECK();
    k_stress_wall<<<wall_ctas, NEAR_NT, 0, s.st>>>(G, bd_all.p, wlist.p + nb, wlist.p, pnear.p);
    EB_LAUNCH_CHECK();
    const int nsplit = s.nsplit;
    part.ensure((size_t)nsplit * 3 * nb);
    static DBuf<double> rig;
    k_stress_rigid<<<pr.M, 256, 0, s.st>>>(G, d_den, rig.ensure(5LL * pr.M));
    EB_LAUNCH_CHECK();
    k_stress_far<<<dim3(nblk(nb, 256), nsplit), 256, 0, s.st>>>(G, d_den, s.tiles.p, s.split_ptr.p, smask.p, mw,
                                                                 rig.p, part.p);
    EB_LAUNCH_CHECK();
    k_stress_final<<<nblk(nb, 256), 256, 0, s.st>>>(G, d_den, pnear.p, 1, part.p, nsplit, 1, eself.p, d_tau, d_E);
    EB_LAUNCH_CHECK();
  } else {
    const int nsplit = s.nsplit;
    part.ensure((size_t)nsplit * 3 * nb);
    dim3 grid(nblk(nb, 256), nsplit);
    k_stress_trap<<<grid, 256, 0, s.st>>>(G, d_den, s.tiles.p, s.split_ptr.p, part.p);
    EB_LAUNCH_CHECK();
    k_stress_final<<<nblk(nb, 256), 256, 0, s.st>>>(G, d_den, nullptr, 0, part.p, nsplit, 0, eself.p, d_tau, d_E);
    EB_LAUNCH_CHECK();
  }
}

void qoi_targets(State& s, const double* d_den, long long ntar, const double* d_xt, const double* d_yt, double* d_u,
                 double* d_v, double* d_p, double* d_w) {
  const Problem& pr = s.pr;
  const GeoDev G = s.geo();
  if (ntar == 0) return;
  static DBuf<double2> txy, bd_all;
  static DBuf<double> ptrap, pbary;
  txy.ensure(ntar);
  k_pack<<<nblk(ntar, 256), 256, 0, s.st>>>((int)ntar, d_xt, d_yt, txy.p);
  EB_LAUNCH_CHECK();
  const int ibary = pr.P.ibary == 1, tasks = (int)nblk(ntar, NEAR_T);
  const int ns1 = source_splits(tasks, std::min(s.ntile, 16));
  ptrap.ensure((size_t)ns1 * 4 * ntar);
  // the trapezoid sums and the nearest nodes on a branch beside the barycentric sums: of
  // the call at 3200 targets, 50 x 128 + 1024 nodes 65 us
  ensure_branches(s);
  const cudaStream_t side = s.br[0];
  EB_CK(cudaEventRecord(s.ev_fork[0], s.st));
  EB_CK(cudaStreamWaitEvent(side, s.ev_fork[0], 0));
  int ns2 = 0;
  if (ibary) {
    bdval_all(s, d_den, bd_all, s.st);
    ns2 = bary_splits(tasks, pr.M + 1);
    pbary.ensure((size_t)ns2 * 6 * ntar);
    bary_sum(s, tasks, ns2, bd_all.p, txy.p, 0, (int)ntar, pbary.p);
    k_qoi_trap<false><<<dim3(tasks, ns1), 256, 0, side>>>(G, d_den, s.tiles.p, s.ntile, (int)ntar, txy.p, ptrap.p);
  } else {
    k_qoi_trap<true><<<dim3(tasks, ns1), 256, 0, side>>>(G, d_den, s.tiles.p, s.ntile, (int)ntar, txy.p, ptrap.p);
  }
  EB_LAUNCH_CHECK();
  const int parts = near_parts(tasks, eb_num_sms());
  static DBuf<double> ndist;
  static DBuf<int> nidx;
  k_qoi_nearest<<<dim3(tasks, parts), 256, 0, side>>>(G, (int)ntar, txy.p, ndist.ensure((size_t)parts * ntar),
                                                      nidx.ensure((size_t)parts * ntar));
  EB_LAUNCH_CHECK();
  EB_CK(cudaEventRecord(s.ev_join[0], side));
  EB_CK(cudaStreamWaitEvent(s.st, s.ev_join[0], 0));
  k_qoi_final<<<tasks, 256, 0, s.st>>>(G, d_den, (int)ntar, txy.p, ptrap.p, ns1, pbary.p, ns2, ibary, ndist.p, nidx.p,
                                       parts, d_u, d_v, d_p, d_w);
  EB_LAUNCH_CHECK();
}

}  // namespace eb

// ===========================================================================
// C ABI
using namespace eb;

namespace {

template <class F>
int guarded2(F&& f) {
  State& s = state();
  std::lock_guard<std::mutex> lk(s.mu);
  try {
    ensure_init(s);
    int rc = f(s);
    set_status(rc, "");
    return rc;
  } catch (const Error& e) {
    settle(s);
    set_status(e.code, e.what());
    return e.code;
  } catch (const std::exception& e) {
    settle(s);
    set_status(EROSION_CUDA_ERROR, e.what());
    return EROSION_CUDA_ERROR;
  }
}

Problem problem_of(const erosion_params* p, int64_t npts, int64_t nbods, int64_t nouter) {
  if (npts < 0 || nbods < 0 || nouter < 0 || npts > (1 << 24) || nbods > (1 << 24) || nouter > (1 << 26))
    throw Error(EROSION_BAD_INPUT, "negative or oversized sizes");
  Problem pr;
  if (p) pr.P = *p;
  else erosion_default_params(&pr.P);
  pr.n = (int)npts; pr.M = (int)nbods; pr.nout = (int)nouter;
  return pr;
}

void host_setup(State& s, const Problem& pr, const double* xx, const double* yy, const double* density) {
  size_t nb = (size_t)pr.n * pr.M;
  double* dx = s.d_xx.ensure(std::max<size_t>(nb, 1));
  double* dy = s.d_yy.ensure(std::max<size_t>(nb, 1));
  h2d(dx, xx, nb, s.st);
  h2d(dy, yy, nb, s.st);
  setup_problem(s, pr, dx, dy);
  double* dd = s.d_den.ensure(s.pr.ntot);
  h2d(dd, density, s.pr.ntot, s.st);
}

}  // namespace

extern "C" {

int erosion_shear_stress(const erosion_params* p, int64_t npts, int64_t nbods, int64_t nouter, const double* xx,
                         const double* yy, const double* density, double* tau, double* E) {
  return guarded2([&](State& s) {
    Problem pr = problem_of(p, npts, nbods, nouter);
    if (pr.M == 0) return EROSION_OK;
    host_setup(s, pr, xx, yy, density);
    const size_t nb = (size_t)s.pr.n * s.pr.M;
    static DBuf<double> dtau, dE;
    dtau.ensure(nb);
    if (E) dE.ensure(3 * nb);
    shear_stress(s, s.d_den.p, dtau.p, E ? dE.p : nullptr);
    d2h(tau, dtau.p, nb, s.st);
    if (E) d2h(E, dE.p, 3 * nb, s.st);
    EB_CK(cudaStreamSynchronize(s.st));
    return EROSION_OK;
  });
}

int erosion_shear_stress_device(const erosion_params* p, int64_t npts, int64_t nbods, int64_t nouter,
                                const double* d_xx, const double* d_yy, const double* d_density, double* d_tau) {
  return guarded2([&](State& s) {
    Problem pr = problem_of(p, npts, nbods, nouter);
    if (pr.M == 0) return EROSION_OK;
    setup_problem(s, pr, d_xx, d_yy);
    shear_stress(s, d_density, d_tau, nullptr);
    EB_CK(cudaStreamSynchronize(s.st));
    return EROSION_OK;
  });
}

int erosion_pressure(const erosion_params* p, int64_t npts, int64_t nbods, int64_t nouter, const double* xx,
                     const double* yy, const double* density, double* pressure) {
  return guarded2([&](State& s) {
    Problem pr = problem_of(p, npts, nbods, nouter);
    if (pr.M == 0) return EROSION_OK;
    host_setup(s, pr, xx, yy, density);
    const size_t nb = (size_t)s.pr.n * s.pr.M;
    static DBuf<double> dp;
    dp.ensure(nb);
    body_pressure(s, s.d_den.p, dp.p);
    d2h(pressure, dp.p, nb, s.st);
    EB_CK(cudaStreamSynchronize(s.st));
    return EROSION_OK;
  });
}

void computepressure_(const int64_t* npts, const int64_t* nbods, const int64_t* nouter, const double* xx,
                      const double* yy, const double* density, double* pressure) {
  erosion_pressure(nullptr, *npts, *nbods, *nouter, xx, yy, density, pressure);
}

void computeshearstress_(const int64_t* npts, const int64_t* nbods, const int64_t* nouter, const double* xx,
                         const double* yy, const double* density, const int64_t* ibary, double* tau) {
  erosion_params p;
  erosion_default_params(&p);
  p.ibary = (int32_t)*ibary;
  erosion_shear_stress(&p, *npts, *nbods, *nouter, xx, yy, density, tau, nullptr);
}

int erosion_qoi_targets(const erosion_params* p, int64_t npts, int64_t nbods, int64_t nouter, const double* xx,
                        const double* yy, const double* density, int64_t ntargets, const double* xtar,
                        const double* ytar, double* utar, double* vtar, double* ptar, double* vortar) {
  return guarded2([&](State& s) {
    Problem pr = problem_of(p, npts, nbods, nouter);
    if (ntargets < 0) throw Error(EROSION_BAD_INPUT, "negative target count");
    host_setup(s, pr, xx, yy, density);
    if (ntargets == 0) return EROSION_OK;
    static DBuf<double> buf;
    double* b = buf.ensure(6 * (size_t)ntargets);
    h2d(b, xtar, ntargets, s.st);
    h2d(b + ntargets, ytar, ntargets, s.st);
    qoi_targets(s, s.d_den.p, ntargets, b, b + ntargets, b + 2 * ntargets, b + 3 * ntargets, b + 4 * ntargets,
                b + 5 * ntargets);
    d2h(utar, b + 2 * ntargets, ntargets, s.st);
    d2h(vtar, b + 3 * ntargets, ntargets, s.st);
    d2h(ptar, b + 4 * ntargets, ntargets, s.st);
    d2h(vortar, b + 5 * ntargets, ntargets, s.st);
    EB_CK(cudaStreamSynchronize(s.st));
    return EROSION_OK;
  });
}

void computeqoitargets_(const int64_t* npts, const int64_t* nbods, const int64_t* nouter, const int64_t* ibary,
                        const double* xx, const double* yy, const double* density, const int64_t* ntargets,
                        const double* xtar, const double* ytar, double* utar, double* vtar, double* ptar,
                        double* vortar) {
  erosion_params p;
  erosion_default_params(&p);
  p.ibary = (int32_t)*ibary;
  erosion_qoi_targets(&p, *npts, *nbods, *nouter, xx, yy, density, *ntargets, xtar, ytar, utar, vtar, ptar, vortar);
}

}  // extern "C"
