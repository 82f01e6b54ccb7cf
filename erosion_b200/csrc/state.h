// Host-side state of the library: device buffers kept between calls, the
// current problem's geometry and near-field bookkeeping, and the status
// channel of the C ABI.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>
#include <cstdint>
#include <algorithm>
#include "erosion_b200.h"
#include "common.cuh"

namespace eb {

extern std::atomic<long long> g_launches;
extern thread_local long long t_launches;   // those of the calling thread

struct Error : std::runtime_error {
  int code;
  bool memory;   // the device had none left
  Error(int c, const std::string& m, bool oom = false) : std::runtime_error(m), code(c), memory(oom) {}
};

#define EB_CK(x)                                                                               \
  do {                                                                                         \
    cudaError_t e_ = (x);                                                                      \
    if (e_ != cudaSuccess)                                                                     \
      throw ::eb::Error(EROSION_CUDA_ERROR, std::string(#x) + ": " + cudaGetErrorString(e_),   \
                        e_ == cudaErrorMemoryAllocation);                                      \
  } while (0)

#define EB_LAUNCH_CHECK()  \
  do {                     \
    ++::eb::g_launches;    \
    ++::eb::t_launches;    \
    EB_CK(cudaGetLastError()); \
  } while (0)

// Grow-only device buffer.
template <class T>
struct DBuf {
  T* p = nullptr;
  size_t cap = 0;
  T* ensure(size_t n) {
    if (n > cap) {
      release();
      size_t m = std::max<size_t>(n, 1);
      EB_CK(cudaMalloc((void**)&p, m * sizeof(T)));
      cap = m;
    }
    return p;
  }
  // Grows keeping the first `keep` elements.
  T* grow_keep(size_t n, size_t keep, cudaStream_t st) {
    if (n <= cap) return p;
    T* q = nullptr;
    EB_CK(cudaMalloc((void**)&q, n * sizeof(T)));
    if (p && keep) EB_CK(cudaMemcpyAsync(q, p, keep * sizeof(T), cudaMemcpyDeviceToDevice, st));
    EB_CK(cudaStreamSynchronize(st));
    release();
    p = q;
    cap = n;
    return p;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
};

template <class T>
void h2d(T* d, const T* h, size_t n, cudaStream_t st) {
  if (n) EB_CK(cudaMemcpyAsync(d, h, n * sizeof(T), cudaMemcpyHostToDevice, st));
}
template <class T>
void d2h(T* h, const T* d, size_t n, cudaStream_t st) {
  if (n) EB_CK(cudaMemcpyAsync(h, d, n * sizeof(T), cudaMemcpyDeviceToHost, st));
}

inline unsigned nblk(long long n, int nt) { return (unsigned)((n + nt - 1) / nt); }

struct Problem {
  int n = 0, M = 0, nout = 0, N = 0;
  long long ntot = 0;
  erosion_params P{};
};

// Near-field bookkeeping of one geometry (near.cuh).
struct Near {
  long long lw = 0;
  bool rules = false;        // the near-wall rules were applied (wflag is valid)
  long long npairs = 0;
  int mw = 0;                // mask words per target
  int n_bary_work = 0;
  DBuf<int> cnt, ptr, wptr, fill, wflag;   // per source curve: pairs, offsets, counters; per body: near the wall
  DBuf<double2> reach;
  DBuf<int> pair_tgt, tpairs;
  DBuf<int2> tl;
  DBuf<int4> bary_work;
  DBuf<unsigned> mask;
  DBuf<unsigned char> info;  // NearInfo
};

// Near and far lists of the clusters (ClView in kernels.cuh).
struct ClLists {
  DBuf<int> near, far, fcls;
  DBuf<int2> ncnt;
  DBuf<double> lnd;
};

struct State {
  std::mutex mu;
  bool init = false;
  int device = -1;
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr, ef0 = nullptr, ef1 = nullptr, ew0 = nullptr, ew1 = nullptr;

  Problem pr;
  bool geo_valid = false;

  // spectral derivative kernels
  int dker_body_n = -1, dker_wall_n = -1;
  DBuf<double> dker_body, dker_wall;

  // geometry
  DBuf<double> wx, wy, sp, cur, w, rb;
  DBuf<double2> xy, nrm, dz, cen, d1tmp;

  Near near;

  // far field
  DBuf<int4> tiles;
  DBuf<int> split_ptr, split_ptr32, split_ptr64t, split_ptr64f, split_ptrw, split_tune;
  int lay_n = -1, lay_M = -1, lay_nout = -1;   // sizes that tiles, items and splits were built for
  int nsplit = 0, nsplit32 = 0, nsplit64t = 0, nsplit64f = 0, nsplitw = 0, ntile = 0;
  long long far64_pairs = 0, farw_pairs = 0;   // pairs per full FP64 / wall-source launch
  // far-field launch shapes: index into the candidate lists of kernels.cuh
  // (kind 0 FP64, 1 FP32), chosen by the autotuner or forced by the caller
  // (kind 0 accurate FP64, 1 FP32, 2 fast FP64)
  int far_shape[3] = {0, 0, 0};
  int force_shape[3] = {-1, -1, -1};
  int tuned_shape[3] = {-1, -1, -1};
  int tune_N = -1, tune_ntile = -1, tune_masked = -1;
  float tune_ms[3][8] = {};
  cudaEvent_t et0 = nullptr, et1 = nullptr;
  // mixed precision: FP32 geometry, strengths, self-curve tasks and sums
  DBuf<float4> src32;
  DBuf<float4> sq32;        // FP32 far-field source tensors (pair_tensor32)
  DBuf<float2> tgt32;
  DBuf<double2> tile_c, anchor;
  int pc_wsplit = 1;        // wall-tile splits of the preconditioner's coupling sum
  DBuf<double2> selfsum;    // k_self64: pairs within each body
  // far field by clusters (cluster.cuh)
  bool cl_ready = false;    // clusters exist for this problem
  bool cl_active = false;   // the operator sums by clusters, not by split tile ranges
  bool cl_expand = false;   // separated clusters act through expansions
  bool cl_sing = false;     // ... and carry the stokeslets and rotlets
  ClLists cl, cl_stress;    // lists of the operator's near mask and of the shear stress's
  DBuf<double2> cl_cen, cl_mp, cl_lam;
  DBuf<double> cl_rad;
  DBuf<int2> items32, items64;   // (tile, first node) of 32 and of 64 targets, wall first
  int n_items32 = 0, n_items64 = 0, n_items32_wall = 0, n_items64_wall = 0;
  int cl_parts64 = 1, cl_parts32 = 1;   // parts of the near lists (k_cl_near64, k_cl_near32)
  DBuf<double4> pc_sq64;    // wall pair tensors of the preconditioner's coupling sum
  long long far32_pairs = 0;
  // block Gauss-Seidel preconditioner
  bool pc_active = false;
  int nwall_tiles = 0;
  DBuf<float> pcB;          // M inverse blocks of (2n+3)^2
  DBuf<double> pc_z, pc_u;  // scratch vectors
  DBuf<double2> pc_tw;      // A_bw z_wall: pc_wsplit partial sums, N long each (body nodes after the wall's)
  DBuf<float4> pc_sq32;     // wall source tensors of the coupling sum (pair_tensor32 of w z_wall)
  DBuf<int> pc_split_ptr;   // its splits of the wall tiles
  // coarse correction (precond = 2): inverse of the completion fields' rigid
  // moments (3M x 3M, FP32), the constraint rows' 3 x 3 inverses (FP64),
  // coarse coordinates
  DBuf<float> cg_B;
  DBuf<double> cg_Cinv, cg_q, cg_cs, cg_cr;
  DBuf<int> cg_bad;
  bool cg_ready = false;
  DBuf<int> pc_bad;         // per body: 1 when its block had a zero pivot
  int pc_singular = 0;      // bodies left unpreconditioned
  bool pc_valid = false;    // pcB holds inverses of a (pc_M, pc_n) problem
  int pc_M = -1, pc_n = -1, pc_nout = -1, pc_age = 0;   // ... built pc_age set-ups ago
  double pc_setup_ms = 0.0; // device time of block assembly + inversion
  double setup_ms = 0.0;    // host wall time of the last setup_problem
  int far_kind = 0;   // kind of the far launch bracketed by ef0/ef1: 0 FP64, 1 FP32, 2 fast FP64

  // work buffers
  DBuf<double2> ws, partial, bd, pair_out;
  DBuf<double4> sq64;        // FP64 far-field source tensors (pair_tensor64)
  DBuf<double> sigdotn;
  DBuf<double> d_xx, d_yy, d_den, d_rhs, d_r, d_w;

  // Krylov
  DBuf<double> V, Z, part, hdev, ydev;
  // Arnoldi steps by captured graphs (gmres_cycle): the vector to apply the
  // operator to, its image, dot products, column count, and the branches of a step
  DBuf<double> k_cur, k_w, k_h1, k_h2, k_np;
  DBuf<int> k_count;
  cudaStream_t br[3] = {nullptr, nullptr, nullptr};
  cudaEvent_t ev_fork[2] = {nullptr, nullptr}, ev_join[3] = {nullptr, nullptr, nullptr}, ev_step[2] = {nullptr, nullptr};
  double* k_host = nullptr; // pinned: two slots of CGS_MAX + 2, a column of the Hessenberg matrix each
  bool forked = false;      // the operator's independent launches go to br
  struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    long long launches = 0;
    int bound = 0, prec = 0;
    bool stale = false;     // of an earlier set-up: to be updated before its next use
    const double *V = nullptr, *Z = nullptr, *part = nullptr;
  };
  std::vector<StepGraph> steps;
  long long captures = 0;         // graphs captured so far
  long long timed_far = 0, timed_farw = 0, timed_far32 = 0, timed_far64f = 0;   // launches with event times
  long long vcap = 0;   // vectors held by V
  long long zcap = 0;   // vectors held by Z (preconditioned basis, flexible GMRES)
  double* h_pinned = nullptr;
  size_t h_pinned_cap = 0;

  erosion_solve_stats stats{};
  bool farw_pending = false;  // ew0/ew1 bracket a wall-source FP64 launch not yet harvested
  bool far_pending = false;   // ef0/ef1 bracket a far-field launch not yet harvested

  GeoDev geo() const {
    GeoDev G;
    G.n = pr.n; G.M = pr.M; G.nout = pr.nout; G.N = pr.N; G.ntot = pr.ntot;
    G.xy = xy.p; G.nrm = nrm.p; G.sp = sp.p; G.cur = cur.p; G.w = w.p; G.dz = dz.p;
    G.cen = cen.p; G.rb = rb.p;
    return G;
  }
};

State& state();

// Sets v while it lives; the old value comes back however the scope is left.
template <class T>
struct Scoped {
  T& v;
  T old;
  Scoped(T& ref, T value) : v(ref), old(ref) { v = value; }
  ~Scoped() { v = old; }
  Scoped(const Scoped&) = delete;
  Scoped& operator=(const Scoped&) = delete;
};

// Runs f with the library stream of the state replaced by st.  A failed launch in f throws:
// the stream comes back with it, or the next call would run, and destroy_state end, a branch
// in its place.
template <class F>
void on_stream(State& s, cudaStream_t st, F&& f) {
  const Scoped<cudaStream_t> keep(s.st, st);
  f();
}

// Waits for what a failed call left in flight on the state's streams (its branches are
// joined by nothing, and the next call uses the same buffers), and clears the error that
// the call reports, which would otherwise be found by the next call's first launch.
void settle(State& s);
int eb_num_sms();
// Creates the branch streams and their events.
void ensure_branches(State& s);
// Parts of the near lists on a device of sms SMs: about four CTAs per SM from items
// CTAs, at most 8.
// 10 bodies x 128 nodes and 1024 wall nodes (72 items): 31.5 us in one part,
// 20.4 us in 5, 17.1 us in 8, 16.0 us in 12 (and 3 us more in larger assemblies);
// 100 x 256, FP32 (464 items): 39.8 us in one part, 33.7 us in 2, 33.3 us in 4.
inline int near_parts(int items, int sms) { return std::max(1, std::min(8, (4 * sms + items - 1) / items)); }
// Raises a kernel's dynamic shared-memory cap to the device's opt-in maximum
// (less the kernel's static shared memory).  Every caller sets the same value, so set-ups running concurrently on host
// threads (the ensemble) that need different sizes never lower the cap under
// each other's launches.
void allow_max_dynamic_smem(const void* fn);
// The outcome of the last entry-point call made by the calling thread,
// read back by erosion_last_status / erosion_last_error.  Thread-local, so it
// takes no lock and one thread's call never overwrites another's outcome.
void set_status(int code, const std::string& msg);
void ensure_init(State& s);
// Streams and events of a state on the current device (no-op when it has them), and
// their end; the buffers are release_state_buffers'.
void init_state(State& s, int device);
void destroy_state(State& s);

// Geometry + near lists + far-field tiles for (xx, yy) already on the device.
void setup_problem(State& s, const Problem& pr, const double* d_xx, const double* d_yy);
// vel = A den, device pointers.  prec 0: FP64 far field; 1: FP32 far field
// between distinct curves + FP64 self-curve sums.
void apply_operator(State& s, const double* d_den, double* d_vel, int prec = 0);
// apply_operator in parts, as a captured step launches it: k_prep (strengths), then
// far_field into s.partial (far_slots(s, prec) slots) beside the self and near sums of
// operator_post, then its assembly.
void operator_prep(State& s, const double* d_den, double* d_vel);
int far_slots(const State& s, int prec);
void operator_post(State& s, const double* d_den, double* d_vel, int nsplit, int* kp = nullptr);
// The captured Arnoldi steps: their end, and their invalidation (a set-up or a buffer
// they refer to changed).
void drop_steps(State& s);
void stale_steps(State& s);
void build_rhs(State& s, double* d_rhs);
// GMRES (SLATEC DGMRES semantics, CGS2 Arnoldi); returns EROSION_* status.
int gmres_solve(State& s, const double* d_b, double* d_x, bool x0_zero, long long maxl, double tol,
                long long* iters, double* est);
// Initial guess selection: candidates zero, the supplied d_x (have_x: the
// previous step's density) and, with learned and have_x, that density plus
// the network's predicted increment (d_hist: the encoded previous
// increment, or null); d_x receives the one with the smallest FP64
// residual.  Returns true when that is the zero vector.
bool choose_initial_guess(State& s, const double* d_b, double* d_x, bool have_x, bool learned,
                          const float* d_hist = nullptr);
// Adds the learned density increment of every body to d_den (the previous
// step's density; wall untouched), given the encoding of the previous
// increment d_hist (nbods x lw_out_width(), or null); false when no trained
// network exists.
bool lw_guess_increment(State& s, const float* d_hist, double* d_den);
// The learned part's density encoding (lw_out_width() floats per body) of
// d_den on the current geometry.
void lw_encode_current(State& s, const double* d_den, float* d_out);
int lw_out_width();
// Builds (or disables) the block preconditioner for the current geometry.
void setup_preconditioner(State& s);
// Copies the last set-up's figures (time, preconditioner state) into s.stats.
void record_setup_stats(State& s);
// z = P^{-1} v (device vectors of length ntot).
void apply_preconditioner(State& s, const double* v, double* z);
// The far field of a prepared density into the partial slots (kind 0 FP64, 1 mixed,
// 2 fast FP64), timed: its launches bracketed by events for the statistics.
void far_field(State& s, const double* d_den, int kind, bool timed);
double device_norm(State& s, const double* d_v, long long n);
// Adds the last far-field launch's event time to stats.ms_far (after a sync).
void harvest_far_timing(State& s);

void release_state_buffers(State& s);
// Bytes of device memory they take.
size_t state_bytes(State& s);
// Memory of the library's device.
size_t eb_device_bytes();
// Frees the ensemble solver's members (batch.cu).
void release_batch();

// Shear stress / targets (stress.cu)
void shear_stress(State& s, const double* d_den, double* d_tau, double* d_E);
// Pressure on the body boundaries (computePressure).
void body_pressure(State& s, const double* d_den, double* d_p);
void qoi_targets(State& s, const double* d_den, long long ntar, const double* d_xt, const double* d_yt,
                 double* d_u, double* d_v, double* d_p, double* d_w);

}  // namespace eb
