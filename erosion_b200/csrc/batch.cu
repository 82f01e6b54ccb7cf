// Ensemble solve: many independent geometries (different body counts, node
// counts per body and wall sizes) solved together.  Every geometry runs the
// single solve (gmres_solve: the same method, the same captured Arnoldi steps) on
// its own State, streams and buffers, the set-ups and then the solves on a pool of
// host threads, so that the GPU always has as many steps in flight as there are
// threads: small geometries fill it together, large ones follow each other.
//
// This takes the place of lockstep rounds (one far-field launch for all
// geometries between each geometry's two captured graphs, with a synchronisation
// per round), in which every geometry waited for the slowest one's kernels and the
// host: 12 geometries of 20-40 bodies x 128 nodes to 1e-11 took 440 ms in 422
// rounds, and 110 ms here.  The members' buffers and captured steps stay for the
// next call (allocating, capturing and freeing them took 100 ms and more of it), up to a
// share of the device's memory; those of more geometries than the next call has are
// freed by it, all of them by erosion_release.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <memory>
#include <vector>

#include "pool.h"
#include "state.h"

namespace eb {
namespace ensemble {

struct Member {
  State s;
  DBuf<double> x, b;
  long long iterations = 0, captures = 0;
  double residual = -1.0;
  int status = EROSION_OK;
};

struct Batch {
  std::vector<std::unique_ptr<Member>> m;
  cudaEvent_t a = nullptr, b = nullptr;
  erosion_batch_stats stats{};
};

Batch& batch() {
  static Batch B;
  return B;
}

void release_buffers(Member& mb) {
  settle(mb.s);
  release_state_buffers(mb.s);
  mb.x.release();
  mb.b.release();
}

void destroy_member(Member& mb) {
  release_buffers(mb);
  destroy_state(mb.s);
}

// What the members keep for the next call is bounded by this share of the device's memory
// (11 GB): the bases of many large geometries are freed when the call ends, those of 12
// geometries of 40 bodies x 128 nodes (1.5 GB) stay.
constexpr size_t kKeepShare = 16;

void trim(Batch& B) {
  size_t kept = 0;
  for (auto& mb : B.m) {
    kept += state_bytes(mb->s);
    if (kept > eb_device_bytes() / kKeepShare) {
      kept -= state_bytes(mb->s);
      release_buffers(*mb);
    }
  }
}

// Runs f for every geometry, in the order of `order`, on a pool of host threads.
template <class F>
void for_each(int device, const std::vector<int>& order, F&& f) {
  const int threads = (int)std::min(16u, std::max(1u, std::thread::hardware_concurrency()));
  on_pool(threads, order, [device] { EB_CK(cudaSetDevice(device)); }, f);
}

}  // namespace ensemble

using namespace ensemble;

void release_batch() {
  Batch& B = batch();
  for (auto& mb : B.m) destroy_member(*mb);
  B.m.clear();
}

}  // namespace eb

using namespace eb;
using namespace eb::ensemble;

extern "C" {

int erosion_solve_batch(const erosion_params* p, int32_t nbatch, const int64_t* npts, const int64_t* nbods,
                        const int64_t* nouter, const double* xx, const double* yy, double* density, int64_t* nits) {
  State& lib = state();
  std::lock_guard<std::mutex> lk(lib.mu);
  try {
    ensure_init(lib);
    if (nbatch <= 0 || !npts || !nbods || !nouter || !density || !nits)
      throw Error(EROSION_BAD_INPUT, "erosion_solve_batch: empty ensemble or null array");
    erosion_params P;
    if (p) P = *p;
    else erosion_default_params(&P);
    P.learned_guess = 0;
    P.true_residual = 0;
    Batch& B = batch();
    if (!B.a) { EB_CK(cudaEventCreate(&B.a)); EB_CK(cudaEventCreate(&B.b)); }
    B.stats = erosion_batch_stats{};
    while ((int)B.m.size() > nbatch) {
      destroy_member(*B.m.back());
      B.m.pop_back();
    }
    while ((int)B.m.size() < nbatch) B.m.push_back(std::make_unique<Member>());
    std::vector<size_t> node_offs(nbatch), den_offs(nbatch);
    std::vector<int> order(nbatch);
    std::vector<double> size(nbatch);
    {
      size_t node_off = 0, den_off = 0;
      for (int g = 0; g < nbatch; ++g) {
        if (npts[g] < 0 || nbods[g] < 0 || nouter[g] < 0) throw Error(EROSION_BAD_INPUT, "negative sizes");
        node_offs[g] = node_off;
        den_offs[g] = den_off;
        node_off += (size_t)npts[g] * nbods[g];
        den_off += 2 * (size_t)nouter[g] + 2 * (size_t)npts[g] * nbods[g] + 3 * (size_t)nbods[g];
        order[g] = g;
        size[g] = (double)nouter[g] + (double)npts[g] * nbods[g];
      }
    }
    // the largest geometries first: the pool ends together
    std::stable_sort(order.begin(), order.end(), [&](int i, int j) { return size[i] > size[j]; });
    cudaStream_t st = lib.st;
    EB_CK(cudaEventRecord(B.a, st));
    auto run = [&] {
      const auto t_setup = std::chrono::steady_clock::now();
      for_each(lib.device, order, [&](int g) {
        Member& mb = *B.m[g];
        State& s = mb.s;
        init_state(s, lib.device);
        s.pc_valid = false;   // the inverses it holds are of another call's geometry
        Problem pr;
        pr.P = P;
        pr.n = (int)npts[g]; pr.M = (int)nbods[g]; pr.nout = (int)nouter[g];
        const size_t nb = (size_t)pr.n * pr.M;
        double* dx = s.d_xx.ensure(std::max<size_t>(nb, 1));
        double* dy = s.d_yy.ensure(std::max<size_t>(nb, 1));
        h2d(dx, xx + node_offs[g], nb, s.st);
        h2d(dy, yy + node_offs[g], nb, s.st);
        setup_problem(s, pr, dx, dy);
        h2d(mb.x.ensure(s.pr.ntot), density + den_offs[g], (size_t)s.pr.ntot, s.st);
        build_rhs(s, mb.b.ensure(s.pr.ntot));
        if (device_norm(s, mb.b.p, s.pr.ntot) == 0.0)
          throw Error(EROSION_BAD_INPUT, "erosion_solve_batch: zero right-hand side");
      });
      B.stats.setup_host_ms =
          std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_setup).count();
      for_each(lib.device, order, [&](int g) {
        Member& mb = *B.m[g];
        State& s = mb.s;
        const long long n = s.pr.ntot, maxl = std::min<long long>(P.maxl > 0 ? P.maxl : 10, n);
        bool zero = true;
        for (long long i = 0; i < n && zero; ++i) zero = density[den_offs[g] + i] == 0.0;
        s.stats = erosion_solve_stats{};
        const long long c0 = s.captures;
        mb.status = gmres_solve(s, mb.b.p, mb.x.p, zero, maxl, P.tol, &mb.iterations, &mb.residual);
        mb.captures = s.captures - c0;
      });
    };
    bool kept = false;
    for (auto& mb : B.m) kept = kept || mb->s.V.p;
    try {
      run();
    } catch (const Error& e) {
      // buffers kept from another ensemble, whose large geometries had other places, may be
      // what the device has no room for: once more without them
      if (!e.memory || !kept) throw;
      for (auto& mb : B.m) release_buffers(*mb);
      run();
    }
    // handed over once every geometry has ended: a call that fails leaves the
    // caller's densities as they were (12 geometries 104.7 ms, each as it ended 105.1)
    for (int g = 0; g < nbatch; ++g) {
      State& s = B.m[g]->s;
      d2h(density + den_offs[g], B.m[g]->x.p, (size_t)s.pr.ntot, s.st);
      EB_CK(cudaStreamSynchronize(s.st));
    }
    EB_CK(cudaEventRecord(B.b, st));
    EB_CK(cudaEventSynchronize(B.b));
    float ms = 0;
    EB_CK(cudaEventElapsedTime(&ms, B.a, B.b));
    B.stats.ms_total = ms;
    B.stats.geometries = nbatch;
    int worst = EROSION_OK;
    for (int g = 0; g < nbatch; ++g) {
      const Member& mb = *B.m[g];
      const erosion_solve_stats& q = mb.s.stats;
      nits[g] = mb.iterations;
      B.stats.iterations += mb.iterations;
      B.stats.rounds = std::max<int64_t>(B.stats.rounds, mb.iterations);
      B.stats.graph_captures += mb.captures;
      const double p64 = P.precision == 0 ? (double)mb.s.far64_pairs : (double)mb.s.farw_pairs;
      const double p32 = P.precision == 0 ? 0.0 : (double)mb.s.far32_pairs;
      B.stats.pairs64_per_round += p64;
      B.stats.pairs32_per_round += p32;
      B.stats.pairs64_total += (double)mb.s.far64_pairs * (double)(q.matvecs - q.matvecs_fp32) +
                               (double)mb.s.farw_pairs * (double)q.matvecs_fp32;
      B.stats.pairs32_total += (double)mb.s.far32_pairs * (double)q.matvecs_fp32;
      if (mb.status != EROSION_OK && worst == EROSION_OK) worst = mb.status;
      B.stats.max_true_residual = std::max(B.stats.max_true_residual, mb.residual);
    }
    trim(B);
    set_status(worst, worst == EROSION_OK ? "" : "a geometry of the ensemble did not converge");
    return worst;
  } catch (const Error& e) {
    for (auto& mb : batch().m) settle(mb->s);
    trim(batch());
    set_status(e.code, e.what());
    return e.code;
  } catch (const std::exception& e) {
    for (auto& mb : batch().m) settle(mb->s);
    trim(batch());
    set_status(EROSION_CUDA_ERROR, e.what());
    return EROSION_CUDA_ERROR;
  }
}

void erosion_get_batch_stats(erosion_batch_stats* out) {
  if (out) *out = batch().stats;
}

}  // extern "C"
