// Set-up of one geometry's near field on the device: the reference's selection
// of the (target node, source curve) pairs that the barycentric formulas
// evaluate (stokesSolver.f:694-926), the checks of the input nodes, and the pair
// lists.  The tests are written with separately rounded operations
// (__dmul_rn, __dadd_rn), so that a node on the edge of a rule falls to the
// same side whatever the compiler contracts.  On the host (the coordinates
// read back, two powers per node, the pairs in vectors, ten uploads) this took
// 0.1 ms at 3 bodies x 64 nodes and 4.5 ms at 400 x 256; the four launches here
// take 14 us and 38 us, with one synchronisation.
#pragma once
#include "kernels.cuh"

namespace {

// What the host needs of it.
struct NearInfo {
  long long lw;                  // integer wall length scale (see k_near_head)
  long long pairs, wall_pairs;   // barycentric pairs, of which with the wall as source
  unsigned long long cl[2];      // node pairs of the near lists (k_cl_lists)
  int work;                      // CTAs of k_bary_list
  int tnext;                     // target slots handed out
  int flags;                     // 1 non-finite node, 2 degenerate wall, 4 node outside the wall
  int pad;
};

// The wall length scale 'lw' of matvec_DLP_fmmbary, an implicitly typed INTEGER
// there (:705-709): lw = (lw + |z'_k|) truncated at every node, then an integer
// division.  Truncating every |z'_k| gives the same sum unless a fraction is so
// close to 1 that the addition may round up, within half an ulp of the running sum (at
// most 1.2e-16 of it; the margin allows for nodes at 1/80 of the mean speed): the 1/256
// of the nodes around one is then summed in order (at the wall's flat sides |z'| is 1 to
// 1e-13).  Per body:
// near the wall (:711-730) or not, the |y| from which its nodes are, and the
// radius within which wall nodes are.
__global__ void __launch_bounds__(256)
k_near_head(GeoDev G, double bw, NearInfo* __restrict__ info, double2* __restrict__ reach, int* __restrict__ wflag,
            int* __restrict__ cnt, int* __restrict__ fill) {
  __shared__ long long part[256];   // truncated speeds of the threads' runs of nodes, summed up to each within its warp
  __shared__ long long wsum[8], lws;
  __shared__ unsigned edge[8];
  __shared__ int bad;
  if (threadIdx.x == 0) {
    bad = 0;
    info->pairs = info->wall_pairs = 0;
    info->cl[0] = info->cl[1] = 0;
    info->work = info->tnext = info->flags = 0;
  }
  __syncthreads();
  const int per = (G.nout + 255) / 256, k0 = min((int)threadIdx.x * per, G.nout), k1 = min(k0 + per, G.nout);
  long long s = 0;
  int e = 0;
  for (int k = k0; k < k1; ++k) {
    const double v = G.sp[k];
    if (!(v > 0.0) || !isfinite(v)) {
      bad = 1;
    } else if (v < 1e15) {
      const long long f = (long long)v;
      if (v - (double)f > 1.0 - (1e-9 + 1e-14 * G.nout * v)) e = 1;
      s += f;
    } else {
      e = 1;
    }
  }
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  long long inc = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  part[threadIdx.x] = inc;
  const unsigned eb = __ballot_sync(0xffffffffu, e);
  if (lane == 31) wsum[wid] = inc;
  if (lane == 0) edge[wid] = eb;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long more = 0, base = 0;   // more: what the runs with such a fraction add beyond their truncated speeds
    for (int w = 0; w < 8; ++w) {
      for (unsigned m = bad ? 0u : edge[w]; m; m &= m - 1u) {
        const int t = 32 * w + __ffs(m) - 1;
        long long lw = base + (t > 32 * w ? part[t - 1] : 0) + more;
        for (int k = t * per; k < min((t + 1) * per, G.nout); ++k) lw = (long long)((double)lw + G.sp[k]);
        more = lw - (base + part[t]);
      }
      base += wsum[w];
    }
    lws = (base + more) / G.nout;
    info->lw = lws;
    if (bad) info->flags = 2;
  }
  __syncthreads();
  const double step = __ddiv_rn(__dmul_rn(__dmul_rn(4.0, (double)lws), EB_TWOPI), (double)G.nout);
  for (int b = threadIdx.x; b < G.M; b += blockDim.x) {
    const double ay = fabs(G.cen[b].y), rb = G.rb[b];
    const double ylim = bw - __dadd_rn(rb, step);
    reach[b] = make_double2(ylim, __dadd_rn(bw - ay, __dmul_rn(2.0, rb)));
    wflag[b] = ay >= ylim;
  }
  for (int c = threadIdx.x; c <= G.M; c += blockDim.x) cnt[c] = fill[c] = 0;
}

__device__ __forceinline__ double dist2_rn(double2 a, double2 b) {
  const double dx = a.x - b.x, dy = a.y - b.y;
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
}

// Near mask (bit c of row i: node i's pair with source curve c is barycentric),
// the number of pairs of every source curve (cnt) and the slots of every target
// (tl[i] = first, count).  mode 0: no pairs; 1: the rules of matvec_DLP_fmmbary;
// 2: every pair of distinct curves (matvec_DLP_bary).  Also checks the nodes:
// finite, and bodies' strictly inside the superellipse wall.  CTA = item (32
// nodes of a cluster, one per lane); a curve is tested node by node only where
// its rule can reach the item; the 8 warps share the words of the mask.
__global__ void __launch_bounds__(256)
k_near_mask(GeoDev G, int mode, double wa, double wb, double order, const int2* __restrict__ items,
            const int4* __restrict__ tiles, const double2* __restrict__ cen, const double* __restrict__ rad,
            const double2* __restrict__ reach, const int* __restrict__ wflag, int mw, unsigned* __restrict__ mask,
            int2* __restrict__ tl, int* __restrict__ cnt, NearInfo* __restrict__ info) {
  __shared__ int tc[32];
  const int2 it = items[blockIdx.x];
  const int4 T = tiles[it.x];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, own = T.z;
  const bool act = it.y + lane < T.y;
  const int i = T.x + min(it.y + lane, T.y - 1);
  const double2 p = G.xy[i];
  if (threadIdx.x < 32) {
    tc[lane] = 0;
    int bad = 0;
    if (!isfinite(p.x) || !isfinite(p.y)) bad = 1;
    else if (own > 0 && !(pow(fabs(p.x) / wa, order) + pow(fabs(p.y) / wb, order) < 1.0)) bad = 4;
    if (bad) atomicOr(&info->flags, bad);
  }
  __syncthreads();
  if (mode == 0) return;
  const double2 ct = cen[it.x];
  const double rt = rad[it.x];
  double2 own_c = make_double2(0, 0);
  double own_r = 0.0;
  if (own > 0) { own_c = G.cen[own - 1]; own_r = G.rb[own - 1]; }
  for (int w = wid; w < mw; w += 8) {
    const int c = 32 * w + lane;
    bool cand = false;
    double2 cc = make_double2(0, 0);
    double lim = 0.0;   // the rule's radius squared about cc; c = 0: the |y| limit
    if (mode == 2) {
      cand = c <= G.M && c != own;
    } else if (c == 0) {
      cand = own > 0 && wflag[own - 1];
      if (cand) lim = reach[own - 1].x;
    } else if (c <= G.M && c != own) {
      cc = G.cen[c - 1];
      if (own == 0) {
        const double r = reach[c - 1].y, far = fabs(r) + rt;
        cand = wflag[c - 1] && cabs2(csub(cc, ct)) <= far * far * 1.0001;
        lim = __dmul_rn(r, r);
      } else {
        const double h = __dadd_rn(G.rb[c - 1], own_r);
        const double rs = __dadd_rn(h, __ddiv_rn(__dmul_rn(__dmul_rn(4.0, h), EB_TWOPI), (double)G.n));
        lim = __dmul_rn(rs, rs);
        cand = dist2_rn(cc, own_c) <= lim;
      }
    }
    unsigned todo = __ballot_sync(0xffffffffu, cand), bits = 0u;
    while (todo) {
      const int q = __ffs(todo) - 1;
      todo &= todo - 1u;
      const double2 cq = make_double2(__shfl_sync(0xffffffffu, cc.x, q), __shfl_sync(0xffffffffu, cc.y, q));
      const double lq = __shfl_sync(0xffffffffu, lim, q);
      bool hit = act;
      if (mode == 1) hit = act && (32 * w + q == 0 ? fabs(p.y) >= lq : dist2_rn(cq, p) <= lq);
      if (hit) bits |= 1u << q;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (lane == 0 && m) atomicAdd(&cnt[32 * w + q], __popc(m));
    }
    if (act) mask[(size_t)i * mw + w] = bits;
    if (bits) atomicAdd(&tc[lane], __popc(bits));
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int mine = act ? tc[lane] : 0;
  int at = mine;   // inclusive prefix
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += v;
  }
  int base = 0;
  if (lane == 31 && at) base = atomicAdd(&info->tnext, at);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (act) tl[i] = make_int2(base + at - mine, mine);
}

// Exclusive prefix sums of the pairs (ptr) and of the CTAs of k_bary_list (wptr)
// over the source curves, and the totals.  One CTA.
__global__ void __launch_bounds__(1024)
k_near_scan(int ncurves, int nout, const int* __restrict__ cnt, int* __restrict__ ptr, int* __restrict__ wptr,
            NearInfo* __restrict__ info) {
  __shared__ long long sp[1024];
  __shared__ int sw[1024];
  const int t = threadIdx.x, per = (ncurves + 1023) / 1024, c0 = min(t * per, ncurves), c1 = min(c0 + per, ncurves);
  long long p = 0;
  int w = 0;
  for (int c = c0; c < c1; ++c) {
    p += cnt[c];
    w += (cnt[c] + NEAR_T - 1) / NEAR_T;
  }
  sp[t] = p;
  sw[t] = w;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {   // inclusive scan
    const long long a = t >= o ? sp[t - o] : 0;
    const int b = t >= o ? sw[t - o] : 0;
    __syncthreads();
    sp[t] += a;
    sw[t] += b;
    __syncthreads();
  }
  long long pb = sp[t] - p;
  int wb = sw[t] - w;
  for (int c = c0; c < c1; ++c) {
    ptr[c] = (int)pb;
    wptr[c] = wb;
    pb += cnt[c];
    wb += (cnt[c] + NEAR_T - 1) / NEAR_T;
  }
  if (t == 1023) {
    info->pairs = sp[1023];
    info->work = sw[1023];
    info->wall_pairs = cnt[0];
  }
}

// The pairs: pair_tgt[q] of the slots ptr[c].. of source curve c, tpairs of every
// target in ascending source order, and the CTAs (curve, first, last) of
// k_bary_list.  Which slot of its curve a pair gets does not matter: a slot is
// evaluated by itself and read through tpairs.
__global__ void __launch_bounds__(256)
k_near_fill(int ncurves, const int2* __restrict__ items, const int4* __restrict__ tiles, int mw,
            const unsigned* __restrict__ mask, const int2* __restrict__ tl, const int* __restrict__ cnt,
            const int* __restrict__ ptr, const int* __restrict__ wptr, int* __restrict__ fill,
            int* __restrict__ pair_tgt, int* __restrict__ tpairs, int4* __restrict__ work) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncurves; c += gridDim.x * blockDim.x)
    for (int q = 0, w = wptr[c]; q < cnt[c]; q += NEAR_T, ++w)
      work[w] = make_int4(c, ptr[c] + q, ptr[c] + min(q + NEAR_T, cnt[c]), 0);
  const int2 it = items[blockIdx.x];
  const int4 T = tiles[it.x];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool act = it.y + lane < T.y;
  const int i = T.x + min(it.y + lane, T.y - 1);
  const unsigned below = (1u << lane) - 1u;
  for (int w = wid; w < mw; w += 8) {
    const unsigned bits = act ? mask[(size_t)i * mw + w] : 0u;
    unsigned any = __reduce_or_sync(0xffffffffu, bits);
    if (!any) continue;
    int at = tl[i].x;
    for (int v = 0; v < w; ++v) at += __popc(mask[(size_t)i * mw + v]);
    while (any) {
      const int q = __ffs(any) - 1, c = 32 * w + q;
      any &= any - 1u;
      const bool hit = (bits >> q) & 1u;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      int base = 0;
      if (lane == 0) base = atomicAdd(&fill[c], __popc(m));
      base = ptr[c] + __shfl_sync(0xffffffffu, base, 0);
      if (hit) {
        const int slot = base + __popc(m & below);
        pair_tgt[slot] = i;
        tpairs[at + __popc(bits & ((1u << q) - 1u))] = slot;
      }
    }
  }
}

}  // namespace
