// The far field by clusters.  A cluster is a far-field tile (an arc of 32 wall
// nodes, or up to 256 nodes of one body).  For every target cluster the source
// clusters fall into two lists: the separated ones act through their multipole
// expansion, shifted to a local expansion about the target cluster's centre
// and evaluated at its nodes; the others are summed pair by pair.
//
// In complex notation (z a target, s_j a source, n_j its normal and v_j its
// weighted strength as complex numbers) the double-layer sum is
//   u = sum_j (r.n)(r.v) r / |r|^4 = 1/4 [ phi - z conj(phi') + conj(chi) ],
//   phi(z) = sum A_j/(z - s_j),  A = n v,
//   chi(z) = sum B_j/(z - s_j) - A_j conj(s_j)/(z - s_j)^2,  B = 2 Re(n conj(v)),
// z and s_j measured from one common origin.  A and B follow from the pair
// tensor (n_x v_x, n_x v_y + n_y v_x, n_y v_y) that the direct sums read.  A
// body's stokeslet l and rotlet xi sit at the centre of its cluster (when the
// body is a single cluster) and add
//   phi: -2 q L log,  chi: -2 q conj(L) log + 2 q conj(L) + 4 i xi / (z - c),
// L = l_x + i l_y, q = 1/(4 pi); of the logarithm only log|.| is kept in the
// constants, where the imaginary parts of phi and conj(chi) cancel.
//
// About a source cluster's centre c with radius R the expansions are
//   phi = sum_k a_k (R/y)^k / y,  chi = sum_k x_k (R/y)^k / y,  y = z - c,
//   a_k = sum A t^k,  x_k = sum B t^k - k sum A conj(t) t^(k-1),  t = (s - c)/R,
// and taking chi to a target centre c + D adds conj(D)/R k a_(k-1) to x_k.  The
// local coefficients about that centre, w = (z - c - D)/R', are
//   alpha_l = (-R'/D)^l sum_k C(k + l, l) a_k (R/D)^k / D,
// a product of one real matrix of binomials with the scaled multipoles of all
// pairs: FP64 tensor-core work (mma m8n8k4).
//
// Accuracy.  Clusters are separated when R <= theta (|D| - R') and R' <= theta
// (|D| - R); phi's series then converge like theta^p.  The terms k a_(k-1) and, in
// the evaluation, phi' put a factor p / theta on the first one that is cut, so p
// terms carry pairs up to a theta whose cut is 5e-16 (FP64 rounding) of a source's
// field |A|/r, or of its strain |A|/r^2, measured over positions, directions and radii
// of the two clusters: 0.373 and 0.337 for CL_P = 40 (cl_class has the others').
// By theta^p alone (32 terms at 1/3, 8 at 1/81) the cut was 2e-14 to 9e-14 of the
// field and 1e-12 of the strain.
//
// Cost.  Per pair of clusters 4 multiply-adds per local and multipole term, 16 x 12 to
// 40 x 40 of them, and about as many operations around them, against 256 x 256 x ~18
// operations for the pairs of two bodies.
#pragma once
#include "state.h"
#include "kernels.cuh"

namespace {

constexpr int CL_P = 40;                 // terms of an expansion
constexpr int CL_MP = 3 * CL_P;          // multipole record of a cluster: a_k, x_k, k a_(k-1) / R
constexpr int CL_MAX_TILES = 4096;       // above this the lists (tiles^2 entries) are not built

// Nodes from which the separated clusters act through expansions; below, every
// cluster pair is summed directly.  Near lists, expansions and assembly with
// and without them, FP64 (mixed): 2304 nodes 24.8 and 20.5 us (30.4 and 19.1),
// 3072 nodes 29.2 and 28.7 us (34.7 and 27.3), 3584 nodes 32.0 and 33.5 us
// (36.2 and 32.5), 8704 nodes 54.7 and 140.6 us (47.4 and 89.2); the
// expansions are two launches more.
constexpr int kExpandNodes = 3200;

// The binomials in the order in which the lanes of cl_shift_run read them: c[lt][kt][lane]
// = C(k + l, l) for l = 8 lt + lane / 4, k = 4 kt + lane % 4.
struct BinomTable {
  double c[CL_P / 8][CL_P / 4][32];
  constexpr BinomTable() : c{} {
    double b[CL_P][CL_P] = {};
    for (int l = 0; l < CL_P; ++l)
      for (int k = 0; k < CL_P; ++k) {
        b[l][k] = (l == 0 || k == 0) ? 1.0 : b[l - 1][k] + b[l][k - 1];
        c[l / 8][k / 4][4 * (l % 8) + k % 4] = b[l][k];
      }
  }
};
__device__ const BinomTable kBinom{};

// Centre and radius of every cluster: the node mean (of a body that is one
// cluster the body's own centre, where its stokeslet and rotlet sit) and the
// largest distance of a node from it.  One warp per cluster.
__global__ void __launch_bounds__(128)
k_cl_geom(GeoDev G, int ntile, const int4* __restrict__ tiles, double2* __restrict__ cen, double* __restrict__ rad) {
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= ntile) return;
  const int4 T = tiles[t];
  double sx = 0.0, sy = 0.0;
  for (int k = lane; k < T.y; k += 32) {
    const double2 p = G.xy[T.x + k];
    sx += p.x;
    sy += p.y;
  }
  double2 c = make_double2(warp_sum(sx) / T.y, warp_sum(sy) / T.y);
  if (T.z > 0 && T.y == G.n) c = G.cen[T.z - 1];
  double r2 = 0.0;
  for (int k = lane; k < T.y; k += 32) {
    const double2 p = G.xy[T.x + k];
    r2 = fmax(r2, cabs2(csub(p, c)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if (lane == 0) {
    cen[t] = c;
    rad[t] = fmax(sqrt(r2), 1e-30);
  }
}

// Orders of the expansions.  A pair of separated clusters with theta = max(R/(|D| -
// R'), R'/(|D| - R)) takes the local x multipole terms that keep its cut below 5e-16:
//   terms            16 x 12   16 x 16   24 x 24   32 x 32   40 x 40
//   velocity, theta   0.036     0.085     0.195     0.293     0.373
//   strain, theta     0.0286    0.068     0.167     0.26      0.337
// The far list of a cluster is sorted by class of order; most pairs of a packing are
// far apart (400 bodies in the 2 x 1 channel: 90% need 16 terms), and the work of a pair
// goes with the product.  The last class pays: with 32 terms at most the near lists of 400
// bodies x 256 nodes take in 168 M pairs instead of 115 M.  Finer steps (8 x 12 at 0.0098,
// 24 x 20 at 0.14) changed the time of a mixed step by 0.2% at most.
constexpr int CL_NCLS = 5;

// Class of a pair at centre distance D: 0..4 of ascending order, CL_NCLS near.
// strain: for the derivative.
__device__ __forceinline__ int cl_class(double D, double rs, double rt, int strain) {
  constexpr double vel[CL_NCLS] = {0.036, 0.085, 0.195, 0.293, 0.373};
  constexpr double str[CL_NCLS] = {0.0286, 0.068, 0.167, 0.26, 0.337};
  const double a = D - rt, b = D - rs;
#pragma unroll
  for (int c = 0; c < CL_NCLS; ++c) {
    const double th = strain ? str[c] : vel[c];
    if (rs <= th * a && rt <= th * b) return c;
  }
  return CL_NCLS;
}

// The lists of target cluster blockIdx.x + tile0.  mask: bit c of node i's row
// (node index less mask0) marks the source curves that another rule evaluates
// at that node; a cluster pair with any marked node stays in the near list.
// expand = 0 puts every cluster there; strain: see cl_class.  A body's own clusters are in neither
// list (k_self64); the wall's are, its own pairs included.  pairs[0], pairs[1]
// += node pairs of the near lists with wall and with body sources, unmasked
// (nullptr: not counted).  With expand = 0, no mask and no count, cen, rad, far, lnd
// and fcls are not touched.
__global__ void __launch_bounds__(256)
k_cl_lists(GeoDev G, int ntile, int tile0, const int4* __restrict__ tiles, const double2* __restrict__ cen,
           const double* __restrict__ rad, const unsigned* __restrict__ mask, int mw, int mask0, int expand, int strain,
           int* __restrict__ near, int* __restrict__ far, double* __restrict__ lnd, int2* __restrict__ ncnt,
           int* __restrict__ fcls, unsigned long long* __restrict__ pairs) {
  extern __shared__ int marked[];   // marked nodes of this cluster per source curve
  constexpr int NC = CL_NCLS + 1;   // the near list is the last category
  __shared__ int tot[NC], wall[NC], at[NC], wcnt[8][NC];
  const int t = blockIdx.x + tile0;
  const int4 T = tiles[t];
  if (!expand && !mask && !pairs) {   // every cluster but the own body's, in order
    const int nwt = (G.nout + WALL_TS - 1) / WALL_TS, per = T.z > 0 ? (G.n + FAR_TS - 1) / FAR_TS : 0;
    const int a = T.z > 0 ? nwt + (T.z - 1) * per : ntile;
    for (int s = threadIdx.x; s < ntile - per; s += blockDim.x) near[(size_t)t * ntile + s] = s < a ? s : s + per;
    if (threadIdx.x == 0) ncnt[t] = make_int2(nwt, ntile - per);
    return;
  }
  const double2 ct = cen[t];
  const double rt = rad[t];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < NC) tot[threadIdx.x] = wall[threadIdx.x] = 0;
  if (mask)
    for (int c = threadIdx.x; c < 32 * mw; c += blockDim.x) marked[c] = 0;
  __syncthreads();
  if (mask) {
    for (int e = threadIdx.x; e < T.y * mw; e += blockDim.x) {
      const int w = e % mw;
      unsigned m = mask[(size_t)(T.x - mask0) * mw + e];
      while (m) {
        atomicAdd(&marked[32 * w + __ffs(m) - 1], 1);
        m &= m - 1;
      }
    }
    __syncthreads();
  }
  double D = 0.0;
  auto category = [&](int s) {
    if (s >= ntile) return -1;
    const int4 S = tiles[s];
    if (S.z > 0 && S.z == T.z) return -1;
    D = sqrt(cabs2(csub(ct, cen[s])));
    if (!expand || (mask && marked[S.z])) return CL_NCLS;
    return cl_class(D, rad[s], rt, strain);
  };
  // sizes
  unsigned long long pw = 0, pb = 0;
  for (int s0 = 0; s0 < ntile; s0 += 256) {
    const int s = s0 + threadIdx.x, c = category(s);
    const bool sw = s < ntile && tiles[s].z == 0;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const unsigned b = __ballot_sync(0xffffffffu, c == q), bw = __ballot_sync(0xffffffffu, c == q && sw);
      if (lane == 0 && b) atomicAdd(&tot[q], __popc(b));
      if (lane == 0 && bw) atomicAdd(&wall[q], __popc(bw));
    }
    if (c == CL_NCLS) {
      const int4 S = tiles[s];
      const unsigned long long p =
          (unsigned long long)(T.y - (mask ? marked[S.z] : 0)) * S.y - (s == t ? T.y : 0);
      if (S.z == 0) pw += p;
      else pb += p;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int o = 0;
    int* f = fcls + (size_t)t * (2 * CL_NCLS + 1);
    for (int q = 0; q < CL_NCLS; ++q) {
      at[q] = f[q] = o;
      f[CL_NCLS + 1 + q] = o + wall[q];
      o += tot[q];
    }
    f[CL_NCLS] = o;
    at[CL_NCLS] = 0;
    ncnt[t] = make_int2(wall[CL_NCLS], tot[CL_NCLS]);
  }
  // places: ascending within a category, so the wall's clusters come first
  for (int s0 = 0; s0 < ntile; s0 += 256) {
    const int s = s0 + threadIdx.x, c = category(s);
    unsigned mine = 0;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const unsigned b = __ballot_sync(0xffffffffu, c == q);
      if (c == q) mine = b;
      if (lane == 0) wcnt[wid][q] = __popc(b);
    }
    __syncthreads();
    if (c >= 0) {
      int o = at[c] + __popc(mine & ((1u << lane) - 1u));
      for (int w = 0; w < wid; ++w) o += wcnt[w][c];
      if (c == CL_NCLS) {
        near[(size_t)t * ntile + o] = s;
      } else {
        far[(size_t)t * ntile + o] = s;
        lnd[(size_t)t * ntile + o] = log(D);
      }
    }
    __syncthreads();
    if (threadIdx.x < NC)
      for (int w = 0; w < 8; ++w) at[threadIdx.x] += wcnt[w][threadIdx.x];
    __syncthreads();
  }
  if (!pairs) return;
  for (int o = 16; o > 0; o >>= 1) {
    pw += __shfl_xor_sync(0xffffffffu, pw, o);
    pb += __shfl_xor_sync(0xffffffffu, pb, o);
  }
  if (lane == 0 && pw) atomicAdd(pairs, pw);
  if (lane == 0 && pb) atomicAdd(pairs + 1, pb);
}

// The first 8 NP multipoles of cluster blockIdx.x + tile0: mp[t][0..39] = a_k, [40..79]
// = x_k, [80..119] = k a_(k-1) / R (entry 0: 2 q L of the stokeslet), lam[t] = -2 q L.
// den: the density the stokeslets and rotlets are read from (nullptr: none).
// Warp w sums the powers NP w .. NP w + NP - 1 over all nodes, a node per lane: 15
// complex products a node (NP = 5) instead of a chain of 40, then the lanes meet in a
// fixed tree.  Bound by latency (a few hundred FP64 operations per thread).
template <int NP>
__global__ void __launch_bounds__(256)
k_cl_form(GeoDev G, int tile0, const int4* __restrict__ tiles, const double2* __restrict__ cen,
          const double* __restrict__ rad, const double4* __restrict__ sq, const double* __restrict__ den,
          double2* __restrict__ mp, double2* __restrict__ lam) {
  __shared__ double2 sA[FAR_TS], sT[FAR_TS];
  __shared__ double sB[FAR_TS];
  __shared__ double2 ka[8 * NP], ke[8 * NP], kb[8 * NP];
  const int t = blockIdx.x + tile0;
  const int4 T = tiles[t];
  const double2 c = cen[t];
  const double R = rad[t], iR = 1.0 / R;
  for (int j = threadIdx.x; j < T.y; j += blockDim.x) {
    const double4 S = sq[T.x + j];
    sA[j] = make_double2(S.x - S.z, S.y);
    sB[j] = 2.0 * (S.x + S.z);
    sT[j] = cscale(csub(G.xy[T.x + j], c), iR);
  }
  __syncthreads();
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double a[NP][6];
#pragma unroll
  for (int q = 0; q < NP; ++q)
#pragma unroll
    for (int v = 0; v < 6; ++v) a[q][v] = 0.0;
  for (int j = lane; j < T.y; j += 32) {
    const double2 A = sA[j], tj = sT[j];
    const double B = sB[j];
    double2 p = make_double2(1.0, 0.0);   // t^(NP wid)
    double2 tp = tj;
#pragma unroll
    for (int q = 1; q < NP; ++q) tp = cmul(tp, tj);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      if ((wid >> b) & 1) p = cmul(p, tp);
      tp = cmul(tp, tp);
    }
    const double2 At = cmul(A, make_double2(tj.x, -tj.y));
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      cfma2(a[q][0], a[q][1], A, p);
      cfma2(a[q][2], a[q][3], At, p);
      a[q][4] = fma(B, p.x, a[q][4]);
      a[q][5] = fma(B, p.y, a[q][5]);
      p = cmul(p, tj);
    }
  }
#pragma unroll
  for (int q = 0; q < NP; ++q)
#pragma unroll
    for (int v = 0; v < 6; ++v) a[q][v] = warp_sum(a[q][v]);
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      ka[NP * wid + q] = make_double2(a[q][0], a[q][1]);
      ke[NP * wid + q] = make_double2(a[q][2], a[q][3]);
      kb[NP * wid + q] = make_double2(a[q][4], a[q][5]);
    }
  }
  __syncthreads();
  const int k = threadIdx.x;
  if (k >= 8 * NP) return;
  double2 x = kb[k], d = make_double2(0, 0);
  if (k > 0) {
    x = make_double2(fma(-(double)k, ke[k - 1].x, x.x), fma(-(double)k, ke[k - 1].y, x.y));
    d = cscale(ka[k - 1], k * iR);
  } else {
    double2 L = make_double2(0, 0);
    double xi = 0.0;
    if (den && T.z > 0 && T.y == G.n) {
      L = make_double2(den[ic_of(G, T.z - 1, 0)], den[ic_of(G, T.z - 1, 1)]);
      xi = den[ic_of(G, T.z - 1, 2)];
    }
    const double q2 = 1.0 / EB_TWOPI;   // 2 q
    x.y += 4.0 * xi;
    d = cscale(L, q2);
    lam[t] = cscale(L, -q2);
  }
  double2* o = mp + (size_t)t * CL_MP;
  o[k] = ka[k];
  o[CL_P + k] = x;
  o[2 * CL_P + k] = d;
}

// One FP64 tensor-core product: c (8 x 8) += a (8 x 4) b (4 x 8); a: row
// lane/4, column lane%4; b: row lane%4, column lane/4; c: row lane/4, columns
// 2 (lane%4) and the next.
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// The local expansion of the far list of cluster t: loc[0][l] = alpha_l,
// loc[1][l] = those of chi, valid for all threads on return.  Every warp takes
// two sources at a time; their phi and chi, real and imaginary, are the 8
// columns of the product with the binomials, which sit in shared memory in the
// order a lane reads them.  Each lane forms its own operand: its component of
// the scaled multipole of the order k it holds, the power of R/D by recurrence
// from k to k + 4.  The products stay in registers until they are scaled by
// (-R'/D)^l and added to the lane's sums, which the warps combine at the end in
// a fixed order.  Bound by the FP64 pipe, which the tensor-core products share:
// of ~450 operations per lane for two sources of 32 x 32 terms, 256 are products.
// The velocity at 400 bodies x 256 nodes takes 98 us, at 200 x 256 52 us, at
// 100 x 256 27 us (all pairs with 32 x 32 terms took 180 us at the first).
struct ClShared {
  double P[CL_P * CL_P];
  double2 red[8][CL_P][2];
  double2 loc[2][CL_P];
};

// The entries [i0, i1) of the far list with 8 LT local and 4 KT multipole terms; w: which of
// the eight warps this one is here.
template <int LT, int KT, int NL>
__device__ __forceinline__ void cl_shift_run(const ClView& L, int t, int i0, int i1, int w,
                                             const double2* __restrict__ mp, const double2* __restrict__ lam,
                                             const double* P, double (&ax)[NL], double (&ay)[NL]) {
  const int lane = threadIdx.x & 31;
  const double2 ct = L.cen[t];
  const double rt = L.rad[t];
  const int* __restrict__ far = L.far + (size_t)t * L.T;
  const double* __restrict__ lnd = L.lnd + (size_t)t * L.T;
  const int kq = lane & 3, bsrc = lane >> 4, bfn = (lane >> 3) & 1, bri = (lane >> 2) & 1;
  const int row = lane >> 2, csrc = (lane >> 1) & 1, cfn = lane & 1;
  for (int i = i0 + 2 * w; i < i1; i += 16) {
    const bool vb = i + bsrc < i1;
    const int s = far[min(i + bsrc, i1 - 1)];
    const double2 D = csub(ct, L.cen[s]);
    const double R = L.rad[s];
    const double id2 = rcp_raw64(cabs2(D));
    const double2 rho = make_double2(D.x * id2, -D.y * id2);   // 1/D
    const double2 q1 = cscale(rho, R), q2 = cmul(q1, q1), q4 = cmul(q2, q2);
    double2 g = vb ? rho : make_double2(0, 0);                 // (R/D)^k / D, k = kq
    if (kq & 1) g = cmul(g, q1);
    if (kq & 2) g = cmul(g, q2);
    const double2 kap = bfn ? make_double2(D.x, -D.y) : make_double2(0, 0);
    const double2* __restrict__ m = mp + (size_t)s * CL_MP;
    const double2* __restrict__ mb = m + bfn * CL_P;
    double c0[LT], c1[LT];
#pragma unroll
    for (int lt = 0; lt < LT; ++lt) c0[lt] = c1[lt] = 0.0;
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
      const int k = 4 * kt + kq;
      double2 y = mb[k];
      const double2 d = m[2 * CL_P + k];
      cfma2(y.x, y.y, kap, d);
      const double b = bri ? fma(y.x, g.y, y.y * g.x) : fma(y.x, g.x, -y.y * g.y);
#pragma unroll
      for (int lt = 0; lt < LT; ++lt) mma_f64(c0[lt], c1[lt], P[(lt * (CL_P / 4) + kt) * 32 + lane], b);
      if (kt + 1 < KT) g = cmul(g, q4);
    }
    // scale by (-R'/D)^l of the lane's own source
    const int from = csrc << 4;
    const double2 r1 = make_double2(__shfl_sync(0xffffffffu, rho.x, from), __shfl_sync(0xffffffffu, rho.y, from));
    const int sc = __shfl_sync(0xffffffffu, s, from);
    const bool vc = i + csrc < i1;
    const double2 p1 = cscale(r1, -rt), p2 = cmul(p1, p1), p4 = cmul(p2, p2), p8 = cmul(p4, p4);
    double2 pw = vc ? make_double2(1.0, 0.0) : make_double2(0, 0);
    if (row & 1) pw = cmul(pw, p1);
    if (row & 2) pw = cmul(pw, p2);
    if (row & 4) pw = cmul(pw, p4);
    double2 lm = lam[sc];
    if (cfn) lm.y = -lm.y;
    const double l0 = lnd[min(i + csrc, i1 - 1)] - cfn;
#pragma unroll
    for (int lt = 0; lt < LT; ++lt) {
      const int l = 8 * lt + row;
      const double f = l == 0 ? l0 : -1.0 / l;
      cfma2(ax[lt], ay[lt], make_double2(fma(lm.x, f, c0[lt]), fma(lm.y, f, c1[lt])), pw);
      if (lt + 1 < LT) pw = cmul(pw, p8);
    }
  }
}

// CL_WALL32: only the wall's clusters as sources, to single precision (a cut of 8e-8 of a
// source's field, an ulp being 1.2e-7): the preconditioner's coupling.
enum ClUse { CL_ALL, CL_WALL32 };

// Local terms that a use fills.
constexpr int cl_terms(int use) { return use == CL_WALL32 ? 24 : CL_P; }

template <int USE>
__device__ __forceinline__ void cl_shift(const ClView& L, int t, const double2* __restrict__ mp,
                                         const double2* __restrict__ lam, ClShared& sh) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = lane >> 2, csrc = (lane >> 1) & 1, cfn = lane & 1;
  constexpr int NL = cl_terms(USE) / 8;
  for (int e = threadIdx.x; e < NL * 8 * CL_P; e += blockDim.x) sh.P[e] = (&kBinom.c[0][0][0])[e];
  __syncthreads();
  double ax[NL] = {}, ay[NL] = {};
  const int* __restrict__ f = L.fcls + (size_t)t * (2 * CL_NCLS + 1);
  constexpr int E = USE == CL_WALL32 ? CL_NCLS + 1 : 1;   // ends of the wall's entries, or of all
  // pairs of the classes before: the warps go on in turn instead of from the first in
  // every class (a mixed step of 100 bodies 171 ms, 177; of 200 bodies 1.5% less)
  int at = 0;
#define EB_RUN(C, LT, KT)                                                                  \
  cl_shift_run<LT, KT>(L, t, f[C], f[C + E], (wid - at) & 7, mp, lam, sh.P, ax, ay);       \
  at += (f[C + E] - f[C] + 1) >> 1
  if constexpr (USE == CL_WALL32) {
    EB_RUN(0, 1, 2); EB_RUN(1, 1, 2); EB_RUN(2, 2, 3); EB_RUN(3, 2, 4); EB_RUN(4, 3, 5);
  } else {
    EB_RUN(0, 2, 3); EB_RUN(1, 2, 4); EB_RUN(2, 3, 6); EB_RUN(3, 4, 8); EB_RUN(4, 5, 10);
  }
#undef EB_RUN
#pragma unroll
  for (int lt = 0; lt < NL; ++lt) {
    ax[lt] += __shfl_xor_sync(0xffffffffu, ax[lt], 2);
    ay[lt] += __shfl_xor_sync(0xffffffffu, ay[lt], 2);
    if (csrc == 0) sh.red[wid][8 * lt + row][cfn] = make_double2(ax[lt], ay[lt]);
  }
  __syncthreads();
  if (threadIdx.x < 16 * NL) {
    const int l = threadIdx.x >> 1, fn = threadIdx.x & 1;
    double2 v = sh.red[0][l][fn];
#pragma unroll
    for (int w = 1; w < 8; ++w) v = cadd(v, sh.red[w][l][fn]);
    sh.loc[fn][l] = v;
  }
  __syncthreads();
}

// The separated sources' velocity at the nodes of cluster blockIdx.x + tile0.  MINB: CTAs
// an SM holds, 2 with 127 registers or 3 with 80 and a few spills (shift_ctas).
template <int USE, int MINB>
__global__ void __launch_bounds__(256, MINB)
k_cl_shift(GeoDev G, ClView L, int tile0, const int4* __restrict__ tiles, const double2* __restrict__ mp,
           const double2* __restrict__ lam, double2* __restrict__ out) {
  __shared__ ClShared sh;
  constexpr int TL = cl_terms(USE);
  const int t = blockIdx.x + tile0;
  const int4 T = tiles[t];
  cl_shift<USE>(L, t, mp, lam, sh);
  const double2 c = L.cen[t];
  const double iR = 1.0 / L.rad[t];
  for (int j = threadIdx.x; j < T.y; j += blockDim.x) {
    const double2 w = cscale(csub(G.xy[T.x + j], c), iR);
    double2 f = sh.loc[0][TL - 1], df = make_double2(0, 0), x = sh.loc[1][TL - 1];
#pragma unroll 4
    for (int l = TL - 2; l >= 0; --l) {
      df = cadd(cmul(df, w), f);
      f = cadd(cmul(f, w), sh.loc[0][l]);
      x = cadd(cmul(x, w), sh.loc[1][l]);
    }
    const double2 e = cmul(w, make_double2(df.x, -df.y));
    out[T.x + j] = make_double2(0.25 * (f.x - e.x + x.x), 0.25 * (f.y - e.y - x.y));
  }
}

// The separated sources' strain at the nodes of cluster blockIdx.x + tile0:
// du/d(conj z) = 1/4 [ -z conj(phi'') + conj(chi') ] = (E11 - E22)/2 + i E12, and
// the field is free of divergence (E22 = -E11).  out[i] = (E11, E12).
// 121 us at 400 bodies x 256 nodes, with the near lists' strain 530 us, where the
// trapezoid sum over every pair took 30.8 ms.
__global__ void __launch_bounds__(256, 2)
k_cl_shift_strain(GeoDev G, ClView L, int tile0, const int4* __restrict__ tiles, const double2* __restrict__ mp,
                  const double2* __restrict__ lam, double2* __restrict__ out) {
  __shared__ ClShared sh;
  const int t = blockIdx.x + tile0;
  const int4 T = tiles[t];
  cl_shift<CL_ALL>(L, t, mp, lam, sh);
  const double2 c = L.cen[t];
  const double iR = 1.0 / L.rad[t];
  for (int j = threadIdx.x; j < T.y; j += blockDim.x) {
    const double2 w = cscale(csub(G.xy[T.x + j], c), iR);
    double2 f = sh.loc[0][CL_P - 1], df = make_double2(0, 0), hf = make_double2(0, 0);   // phi, phi', phi''/2
    double2 x = sh.loc[1][CL_P - 1], dx = make_double2(0, 0);
#pragma unroll 4
    for (int l = CL_P - 2; l >= 0; --l) {
      hf = cadd(cmul(hf, w), df);
      df = cadd(cmul(df, w), f);
      f = cadd(cmul(f, w), sh.loc[0][l]);
      dx = cadd(cmul(dx, w), x);
      x = cadd(cmul(x, w), sh.loc[1][l]);
    }
    const double2 e = cmul(w, make_double2(2.0 * hf.x, -2.0 * hf.y));
    out[T.x + j] = make_double2(0.25 * iR * (dx.x - e.x), 0.25 * iR * (-dx.y - e.y));
  }
}

// ---------------------------------------------------------------------------
// The near lists, pair by pair.  CTA = item (target cluster, first node in
// it): up to 32 targets (FP64) or 64 (FP32, two per lane).  The CTA stages up to
// 256 sources of consecutive list entries at a time and its 8 warps split
// them, so that a cluster with few targets still fills 8 warps; the warps' sums
// meet in a fixed order.  blockIdx.y takes a contiguous part of every list into
// a slot of its own (out[part * N + i]): few items alone leave SMs idle and a
// CTA with a long chain of stages.  Bound by the FP64 (FP32) pipe as k_far64
// (k_far32), whose arithmetic and near masks they share, at thousands of items,
// by the latency of the stages at tens.
constexpr int CL_MAXE = 64;   // list entries whose tiles are read at a time

// STRAIN: instead of the velocity q r/rho^4, q = r^T S r, its strain
//   E11 = (h_x r_x - h_y r_y)/rho^4 - 2 q (r_x^2 - r_y^2)/rho^6,
//   E12 = (h_x r_y + h_y r_x)/rho^4 - 4 q r_x r_y/rho^6,   h = S r,  E22 = -E11.
// mask rows start at node mask0.
template <bool STRAIN, bool MASK>
__global__ void __launch_bounds__(256)
k_cl_near64(GeoDev G, ClView L, const int2* __restrict__ items, const int4* __restrict__ tiles, int wall_only,
            const double4* __restrict__ sq, const unsigned* __restrict__ mask, int mw, int mask0,
            double2* __restrict__ out) {
  __shared__ double4 sg[FAR_TS];
  __shared__ double sw[FAR_TS];
  __shared__ double red[NEAR_W / 2][2][32];
  __shared__ int4 ent[CL_MAXE];
  const int2 it = items[blockIdx.x];
  const int4 T = tiles[it.x];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool act = it.y + lane < T.y;
  const int i = T.x + (act ? it.y + lane : T.y - 1);
  const double2 p = G.xy[i];
  const int2 c4 = L.ncnt[it.x];
  const int nt = wall_only ? c4.x : c4.y;
  const int ne = (int)((long long)nt * (blockIdx.y + 1) / gridDim.y);
  const int* __restrict__ near = L.near + (size_t)it.x * L.T;
  double a[2] = {0.0, 0.0};
  int eb = 0, nb = 0;   // the entries held in ent: [eb, eb + nb)
  for (int e0 = (int)((long long)nt * blockIdx.y / gridDim.y); e0 < ne;) {
    __syncthreads();
    if (e0 >= eb + nb || (eb + nb < ne && e0 - eb > CL_MAXE / 2)) {   // refill
      eb = e0;
      nb = min(CL_MAXE, ne - e0);
      if ((int)threadIdx.x < nb) ent[threadIdx.x] = tiles[near[e0 + threadIdx.x]];
      __syncthreads();
    }
    // stage the entries from e0 that fit (the same walk in every thread)
    int m = 0, len = 0;
    while (e0 + m < eb + nb) {
      const int4 S = ent[e0 + m - eb];
      if (len + S.y > FAR_TS) break;
      if ((int)threadIdx.x >= len && (int)threadIdx.x < len + S.y) {
        const int g = S.x + (int)threadIdx.x - len;
        const double2 q = G.xy[g];
        const double4 s4 = sq[g];
        sg[threadIdx.x] = make_double4(q.x, q.y, s4.x, s4.y);
        sw[threadIdx.x] = s4.z;
      }
      len += S.y;
      ++m;
    }
    __syncthreads();
    const int ka = len * wid / NEAR_W, kb = len * (wid + 1) / NEAR_W;
    int at = 0;   // first staged source of entry e
    for (int e = e0 - eb; e < e0 - eb + m; ++e) {
      const int lo = max(ka, at), hi = min(kb, at + ent[e].y);
      at += ent[e].y;
      if (lo >= hi) continue;
      bool use = true;
      if (MASK) {
        const int c = ent[e].z;
        use = !((__ldg(mask + (size_t)(i - mask0) * mw + (c >> 5)) >> (c & 31)) & 1u);
        if (!__any_sync(0xffffffffu, use)) continue;
      }
      double tx = 0.0, ty = 0.0;
#pragma unroll 4
      for (int j = lo; j < hi; ++j) {
        const double4 s = sg[j];   // x, y, S_xx, 2 S_xy
        const double syy = sw[j];
        const double rx = p.x - s.x, ry = p.y - s.y;
        const double ry2 = ry * ry;
        const double rho2 = fma(rx, rx, ry2);
        const double inv = rcp_newton64<2>(rho2);   // 0 for a wall node on itself
        if constexpr (STRAIN) {
          const double sxy = 0.5 * s.w;
          const double hx = fma(sxy, ry, s.z * rx), hy = fma(sxy, rx, syy * ry);
          const double i4 = inv * inv, hr = hy * ry;
          const double d = 2.0 * fma(hx, rx, hr) * inv;   // 2 q/rho^2
          const double rxy = rx * ry;
          tx = fma(i4, fma(hx, rx, -hr) - d * fma(rx, rx, -ry2), tx);
          ty = fma(i4, fma(hx, ry, hy * rx) - 2.0 * d * rxy, ty);
        } else {
          const double tt = fma(s.w, ry, s.z * rx);
          const double qq = fma(tt, rx, syy * ry2);
          const double c = qq * inv * inv;
          tx = fma(c, rx, tx);
          ty = fma(c, ry, ty);
        }
      }
      if (use) { a[0] += tx; a[1] += ty; }
    }
    e0 += m;
  }
  __syncthreads();
  near_reduce(a, red);
  if (act && wid == 0) out[(size_t)blockIdx.y * G.N + i] = make_double2(a[0], a[1]);
}

// FP32 pair terms as k_far32's (chunks of F32_CHUNK sources summed in FP32 and
// added to FP64 accumulators); body sources [cnt.x, cnt.y) of the near list, or
// the wall's [0, cnt.x) with wall_only.
template <bool MASK>
__global__ void __launch_bounds__(256)
k_cl_near32(GeoDev G, ClView L, const int2* __restrict__ items, const int4* __restrict__ tiles, int wall_only,
            const float4* __restrict__ src, const float2* __restrict__ tgt, const double2* __restrict__ anchor,
            const double2* __restrict__ tile_c, const float4* __restrict__ sq32, const unsigned* __restrict__ mask,
            int mw, double2* __restrict__ out) {
  __shared__ float4 s_pos[F32_TS], s_q1[F32_TS];
  __shared__ float2 s_q2[F32_TS];
  __shared__ double red[NEAR_W / 2][4][32];
  __shared__ int4 ent[CL_MAXE];
  __shared__ double2 ecen[CL_MAXE];
  const int2 it = items[blockIdx.x];
  const int4 T = tiles[it.x];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k0 = it.y + lane, k1 = k0 + 32;
  const int i0 = T.x + min(k0, T.y - 1), i1 = T.x + min(k1, T.y - 1);
  const double2 an = anchor[i0];   // one cluster: one anchor
  const float2 o0 = tgt[i0], o1 = tgt[i1];
  const int2 c4 = L.ncnt[it.x];
  const int n0 = wall_only ? 0 : c4.x, nt = (wall_only ? c4.x : c4.y) - n0;
  const int ne = n0 + (int)((long long)nt * (blockIdx.y + 1) / gridDim.y);
  const int* __restrict__ near = L.near + (size_t)it.x * L.T;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  int eb = 0, nb = 0;   // the entries held in ent: [eb, eb + nb)
  for (int e0 = n0 + (int)((long long)nt * blockIdx.y / gridDim.y); e0 < ne;) {
    __syncthreads();
    if (e0 >= eb + nb || (eb + nb < ne && e0 - eb > CL_MAXE / 2)) {   // refill
      eb = e0;
      nb = min(CL_MAXE, ne - e0);
      if ((int)threadIdx.x < nb) {
        const int ti = near[e0 + threadIdx.x];
        ent[threadIdx.x] = tiles[ti];
        ecen[threadIdx.x] = tile_c[ti];
      }
      __syncthreads();
    }
    int m = 0, len = 0;   // entries and sources staged, every entry padded to whole chunks
    while (e0 + m < eb + nb) {
      const int4 S = ent[e0 + m - eb];
      const int pl = (S.y + F32_CHUNK - 1) / F32_CHUNK * F32_CHUNK;
      if (len + pl > F32_TS) break;
      const int k = (int)threadIdx.x - len;
      if (k >= 0 && k < pl) {
        if (k < S.y) {
          const float4 x = src[S.x + k], q = sq32[S.x + k];
          s_pos[threadIdx.x] = make_float4(-x.x, -x.x, -x.y, -x.y);
          s_q1[threadIdx.x] = make_float4(q.x, q.x, q.y, q.y);
          s_q2[threadIdx.x] = make_float2(q.z, q.z);
        } else {   // zero strength, far from every target: exactly zero terms
          s_pos[threadIdx.x] = make_float4(-1e4f, -1e4f, -1e4f, -1e4f);
          s_q1[threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
          s_q2[threadIdx.x] = make_float2(0.f, 0.f);
        }
      }
      len += pl;
      ++m;
    }
    __syncthreads();
    const int nch = len / F32_CHUNK;
    const int ca = nch * wid / NEAR_W, cb = nch * (wid + 1) / NEAR_W;
    int at = 0;   // first chunk of entry e
    for (int e = e0 - eb; e < e0 - eb + m; ++e) {
      const int nc = (ent[e].y + F32_CHUNK - 1) / F32_CHUNK;
      const int lo = max(ca, at), hi = min(cb, at + nc);
      at += nc;
      if (lo >= hi) continue;
      bool u0 = true, u1 = true;
      if (MASK) {
        const int c = ent[e].z;
        u0 = !((__ldg(mask + (size_t)i0 * mw + (c >> 5)) >> (c & 31)) & 1u);
        u1 = !((__ldg(mask + (size_t)i1 * mw + (c >> 5)) >> (c & 31)) & 1u);
        if (!__any_sync(0xffffffffu, u0 || u1)) continue;
      }
      const double2 cs = ecen[e];
      const float dx = (float)(an.x - cs.x), dy = (float)(an.y - cs.y);
      const float2 PX = make_float2(dx + o0.x, dx + o1.x), PY = make_float2(dy + o0.y, dy + o1.y);
      for (int c = lo; c < hi; ++c) {
        float2 TX = make_float2(0.f, 0.f), TY = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int j = c * F32_CHUNK; j < (c + 1) * F32_CHUNK; ++j) {
          const float4 A = s_pos[j], B = s_q1[j];
          const float2 qyy = s_q2[j];
          const float2 rx = __fadd2_rn(PX, make_float2(A.x, A.y));
          const float2 ry = __fadd2_rn(PY, make_float2(A.z, A.w));
          const float2 ry2 = __fmul2_rn(ry, ry);
          const float2 rho2 = __ffma2_rn(rx, rx, ry2);
          const float2 inv = make_float2(rcp_approx(rho2.x), rcp_approx(rho2.y));
          const float2 t = __ffma2_rn(make_float2(B.z, B.w), ry, __fmul2_rn(make_float2(B.x, B.y), rx));
          const float2 q = __ffma2_rn(t, rx, __fmul2_rn(qyy, ry2));
          const float2 cc = __fmul2_rn(__fmul2_rn(q, inv), inv);
          TX = __ffma2_rn(cc, rx, TX);
          TY = __ffma2_rn(cc, ry, TY);
        }
        if (u0) { a[0] += (double)TX.x; a[1] += (double)TY.x; }
        if (u1) { a[2] += (double)TX.y; a[3] += (double)TY.y; }
      }
    }
    e0 += m;
  }
  __syncthreads();
  near_reduce(a, red);
  if (wid == 0) {
    double2* o = out + (size_t)blockIdx.y * G.N;
    if (k0 < T.y) o[i0] = make_double2(a[0], a[1]);
    if (k1 < T.y) o[i1] = make_double2(a[2], a[3]);
  }
}

}  // namespace

// Host side.
namespace eb {

// CTAs per SM of k_cl_shift for that many clusters: two while all of them find a place, at
// 164, 264 and 294 clusters 27.0, 33.6 and 43.6 us (three: 32.5, 43.8, 49.3), then three, as
// the clusters past two an SM would make a wave of their own: at 328, 428, 528, 628 and 728
// clusters 50.2, 63.6, 97.8, 129.9 and 147.1 us (two: 55.0, 73.8, 99.9, 140.9, 165.7).
inline int shift_ctas(int ntile, int sms) { return ntile <= 2 * sms ? 2 : 3; }

static inline ClView cl_view(const State& s, const ClLists& L) {
  ClView v;
  v.T = s.ntile;
  v.cen = s.cl_cen.p;
  v.rad = s.cl_rad.p;
  v.near = L.near.p;
  v.far = L.far.p;
  v.ncnt = L.ncnt.p;
  v.fcls = L.fcls.p;
  v.lnd = L.lnd.p;
  return v;
}

// Lists of the target clusters from tile0 on (mask as k_cl_lists takes it).
// pairs: see k_cl_lists, or nullptr.
static inline void build_lists(State& s, ClLists& L, int tile0, const unsigned* mask, int mw, int mask0, bool expand,
                               bool strain, unsigned long long* pairs) {
  const size_t T = s.ntile;
  const size_t smem = mask ? 32 * (size_t)mw * sizeof(int) : 0;
  k_cl_lists<<<(unsigned)(T - tile0), 256, smem, s.st>>>(
      s.geo(), s.ntile, tile0, s.tiles.p, s.cl_cen.p, s.cl_rad.p, mask, mw, mask0, expand, strain, L.near.ensure(T * T),
      L.far.ensure(T * T), L.lnd.ensure(T * T), L.ncnt.ensure(T), L.fcls.ensure(T * (2 * CL_NCLS + 1)), pairs);
  EB_LAUNCH_CHECK();
}

}  // namespace eb
