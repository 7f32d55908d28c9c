// C ABI implementation (include/nrg_chem.h): handle, mechanism upload,
// host-layout gather/scatter, CUDA-graph capture and the launch autotuner.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <unistd.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif
#include <string>
#include <vector>

#include "../../include/nrg_chem.h"
#include "chem_device.cuh"
#include "chem_kernels.hpp"
#include "mechanism.hpp"
#include "surrogate.hpp"
#include "transport.hpp"
#include "diffusion.hpp"
#include "order.hpp"
#include "table.hpp"

using nrg::DevMech;
using nrg::LaunchCfg;
using nrg::StepArgs;

static thread_local std::string g_create_error;

struct nrg_chem {
  nrg::Mechanism mech;
  DevMech dm;   // tables over all species
  DevMech dmr;  // reaction lists over the reacting species (fast / mixed thread kernels)
  // generated mechanism-specialised code in use (0: tables): right-hand side and
  // iteration matrix over the reacting species, right-hand side over all (reference mode)
  int spec = 0, spec_full = 0;
  bool has_transport = false;
  nrg::DiffusivityArgs diff;  // pair tables of the loaded transport deck
  int device = 0;
  int num_sms = 148;
  cudaStream_t stream = nullptr;
  // host path: H2D and D2H copy streams and per-chunk events (copied in,
  // stepped, copied out), so that transfers and host work overlap the steps
  cudaStream_t copy_in = nullptr, copy_out = nullptr;
  // host path, surrogate mode: a second compute stream (odd chunks) and the
  // event that joins it back into the compute stream
  cudaStream_t stream2 = nullptr;
  cudaEvent_t ev_join = nullptr;
  cudaEvent_t ev_h2d[8] = {}, ev_step[8] = {}, ev_chunk[8] = {};
  int mode = NRG_MODE_FAST;
  LaunchCfg cfg;
  bool use_graph = true;
  double eps = 0.0;           // integrator tolerance override (0: the reference's EPS)
  double fallback_eps = 0.0;  // tolerance of the surrogate's FP64 fallback (0: eps)
  bool timing = false;
  cudaEvent_t ph[4] = {nullptr, nullptr, nullptr, nullptr};
  int* d_queue = nullptr;
  DevMech* d_mech = nullptr;  // global copy of the tables for kernels that stage them in shared memory
  unsigned long long* d_counters = nullptr;
  unsigned long long* h_counters = nullptr;  // pinned
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev_in = nullptr;
  // host-path staging
  size_t cap = 0;
  double *d_T = nullptr, *d_rho = nullptr, *d_Y = nullptr, *d_Yp = nullptr, *d_Yp2 = nullptr,
         *d_Ef = nullptr;
  int8_t* d_bc = nullptr;
  uint8_t* d_status = nullptr;
  double *h_T = nullptr, *h_rho = nullptr, *h_Y = nullptr, *h_Yp = nullptr, *h_Yp2 = nullptr,
         *h_Ef = nullptr;
  int8_t* h_bc = nullptr;
  uint8_t* h_status = nullptr;
  // temperature order of the plain integrator's cells (order.hpp)
  bool order_cells = true;
  long order_cap = 0;
  nrg::OrderScratch order;
  int *d_order_list = nullptr, *d_order_count = nullptr;
  // graph cache
  cudaGraphExec_t gexec = nullptr;
  // table of the table_approximated mode (nrg_chem_set_table / nrg_chem_load_table)
  double *d_tab_T = nullptr, *d_tab_Y = nullptr;
  int2* d_tab_idx = nullptr;  // bucket index of sorted nodes (nrg::TableIndex)
  nrg::TableIndex tab_idx;
  long tab_rows = 0;
  bool tab_sorted = false;
  // surrogate state (owned by surrogate.cu): the main network and a second
  // one for the flame's preheat band; the nrg_surrogate_* set-up calls act on
  // network sur_sel (nrg_surrogate_select)
  nrg::Surrogate* sur_net[nrg::kMaxNets] = {};
  int sur_sel = 0;
  std::string err;
};

namespace {

int fail(nrg_chem* h, int code, const std::string& msg) {
  if (h) h->err = msg;
  else g_create_error = msg;
  return code;
}

int cuda_fail(nrg_chem* h, cudaError_t e, const char* where) {
  return fail(h, NRG_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

#define CK(h, call)                                        \
  do {                                                     \
    cudaError_t e_ = (call);                               \
    if (e_ != cudaSuccess) return cuda_fail(h, e_, #call); \
  } while (0)

// Makes the handle's device current for the rest of an entry point and gives
// the calling thread its own current device back when the entry point
// returns, so a host code that drives several GPUs from one thread may call
// any handle at any time.
struct DeviceScope {
  int prev = -1;
  cudaError_t enter(int dev) {
    cudaError_t e = cudaGetDevice(&prev);
    if (e != cudaSuccess) {
      prev = -1;
      return e;
    }
    return prev == dev ? cudaSuccess : cudaSetDevice(dev);
  }
  ~DeviceScope() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};
#define ON_DEVICE(h)         \
  DeviceScope device_scope_; \
  CK(h, device_scope_.enter((h)->device))

// Gear coefficients EL(13,12), TQ(3,12) (ddcst.f90:35-106, MINT = 2).
void gear_coefficients(double* el, double* tq) {
  const int maxord = nrg::kMaxOrd;
  double fact[13];
  fact[0] = 1.0;
  for (int i = 2; i <= maxord; ++i) fact[i - 1] = (double)i * fact[i - 2];
  auto E = [&](int i, int j) -> double& { return el[(j - 1) * 13 + (i - 1)]; };
  auto Q = [&](int i, int j) -> double& { return tq[(j - 1) * 3 + (i - 1)]; };
  std::fill(el, el + 13 * 12, 0.0);
  std::fill(tq, tq + 3 * 12, 0.0);
  E(1, 1) = 1.0;
  E(2, 1) = 1.0;
  for (int j = 2; j <= maxord; ++j) {
    E(1, j) = fact[j - 1];
    for (int i = 2; i <= j; ++i) E(i, j) = (double)j * E(i, j - 1) + E(i - 1, j - 1);
    E(j + 1, j) = 1.0;
  }
  double sum = 1.0;
  for (int j = 2; j <= maxord; ++j) {
    sum = sum + 1.0 / (double)j;
    for (int i = 1; i <= j + 1; ++i) E(i, j) = E(i, j) / (fact[j - 1] * sum);
  }
  for (int j = 1; j <= maxord; ++j) {
    if (j > 1) Q(1, j) = 1.0 / fact[j - 2];
    Q(2, j) = (double)(j + 1) / E(1, j);
    Q(3, j) = (double)(j + 2) / E(1, j);
  }
}

// Atom counts of H, O, N from a species formula such as "H2O2".
void formula_elements(const std::string& name, double out[3]) {
  out[0] = out[1] = out[2] = 0.0;
  size_t i = 0;
  while (i < name.size()) {
    char c = name[i++];
    int idx = c == 'H' ? 0 : c == 'O' ? 1 : c == 'N' ? 2 : -1;
    int cnt = 0;
    while (i < name.size() && std::isdigit((unsigned char)name[i])) cnt = cnt * 10 + (name[i++] - '0');
    if (cnt == 0) cnt = 1;
    if (idx >= 0) out[idx] += cnt;
  }
}

std::string build_dev_mech(const nrg::Mechanism& m, DevMech* d) {
  const int N = m.n(), R = m.r();
  if (N > nrg::kMaxSpecies || R > nrg::kMaxReactions) return "mechanism larger than the compiled tables";
  std::memset(d, 0, sizeof(DevMech));
  d->N = N;
  d->R = R;
  for (int r = 0; r < R; ++r) {
    const nrg::Reaction& rx = m.reactions[r];
    d->type[r] = rx.type;
    d->nl[r] = rx.n_left;
    d->nr[r] = rx.n_right;
    for (int i = 0; i < 3; ++i) {
      d->left[r][i] = (i < rx.n_left) ? (rx.left[i] == N + 1 ? -1 : rx.left[i] - 1) : -1;
      d->right[r][i] = (i < rx.n_right) ? (rx.right[i] == N + 1 ? -1 : rx.right[i] - 1) : -1;
    }
    int u = 0;
    for (int k = 1; k <= N; ++k) {
      for (int i = 0; i < rx.n_left; ++i)
        if (rx.left[i] == k) { d->upd_k[r][u] = k - 1; d->upd_prod[r][u] = 0; ++u; }
      for (int i = 0; i < rx.n_right; ++i)
        if (rx.right[i] == k) { d->upd_k[r][u] = k - 1; d->upd_prod[r][u] = 1; ++u; }
    }
    d->nupd[r] = u;
    d->A[r] = rx.A;
    d->beta[r] = rx.beta;
    d->E[r] = rx.E;
    d->A_low[r] = rx.A_low;
    d->beta_low[r] = rx.beta_low;
    d->E_low[r] = rx.E_low;
    for (int q = 0; q < 4; ++q) d->troe[r][q] = rx.troe[q];
    d->dnu[r] = (double)(rx.n_right - rx.n_left);
    for (int uu = 0; uu < u; ++uu) {
      const int k = d->upd_k[r][uu];
      if (d->sp_n[k] >= nrg::kMaxSpecUpd) return "species appears in too many reactions";
      d->sp_list[d->sp_n[k]][k] = (r << 1) | (d->upd_prod[r][uu] ? 1 : 0);
      d->sp_n[k] += 1;
    }
    for (int k = 0; k < N; ++k) d->eff_t[k][r] = m.eff[(size_t)r * N + k];
  }
  for (int k = 0; k < N; ++k) {
    for (int s = 0; s < 2; ++s)
      for (int i = 0; i < 7; ++i) d->a[k][s][i] = m.a_coeffs[((size_t)k * 2 + s) * 7 + i];
    d->W[k] = m.molar_mass[k];
    if (d->W[k] == 0.0) return "zero molar mass for species " + m.species[k];
    d->invW[k] = 1.0 / d->W[k];
    d->h_ref[k] = nrg::specie_enthalpy(m, nrg::kTRef, k);
    double e[3];
    formula_elements(m.species[k], e);
    for (int q = 0; q < 3; ++q) d->elem[q][k] = e[q];
  }
  d->RM = R;
  for (int r = 0; r < R; ++r) d->m_of[r] = r;
  d->NI = N;
  for (int k = 0; k < N; ++k) d->full_of[k] = k;
  d->n_inert = 0;
  gear_coefficients(d->el, d->tq);
  for (int q = 1; q <= nrg::kMaxOrd; ++q)
    for (int i = 0; i < 3; ++i) {
      const double x = d->tq[(q - 1) * 3 + i];
      d->itq2[q][i] = x != 0.0 ? 1.0 / (x * x) : 0.0;
    }
  d->eps = 1.0e-9;
  d->ewt = 1.0e-4;
  d->hmax = (double)1.0E-7f;  // single-precision literal in the reference
  d->uround = DBL_EPSILON;
  d->sqrt_uround = std::sqrt(DBL_EPSILON);
  d->br = std::pow(DBL_EPSILON, 0.875);
  d->bl = std::pow(DBL_EPSILON, 0.75);
  d->bp = std::pow(DBL_EPSILON, -0.15);
  d->facmin = std::pow(DBL_EPSILON, 0.78);
  return "";
}

// Reorders the reactions so that those whose reactant and product lists equal
// an earlier one's come last (DevMech::RM, m_of).
void merge_equal_reactions(DevMech* d) {
  const DevMech in = *d;
  auto equal = [&](int a, int b) {
    return std::memcmp(in.left[a], in.left[b], sizeof in.left[a]) == 0 &&
           std::memcmp(in.right[a], in.right[b], sizeof in.right[a]) == 0;
  };
  std::vector<int> order, repeats, to(in.R);
  for (int r = 0; r < in.R; ++r) {
    int f = 0;
    while (!equal(f, r)) ++f;
    (f == r ? order : repeats).push_back(r);
    to[r] = f;
  }
  d->RM = (int)order.size();
  std::vector<int> pos(in.R);
  for (int q = 0; q < d->RM; ++q) pos[order[q]] = q;
  order.insert(order.end(), repeats.begin(), repeats.end());
  for (int q = 0; q < in.R; ++q) {
    const int r = order[q];
    d->m_of[q] = pos[to[r]];
    d->type[q] = in.type[r];
    d->nl[q] = in.nl[r];
    d->nr[q] = in.nr[r];
    std::memcpy(d->left[q], in.left[r], sizeof in.left[r]);
    std::memcpy(d->right[q], in.right[r], sizeof in.right[r]);
    d->nupd[q] = in.nupd[r];
    std::memcpy(d->upd_k[q], in.upd_k[r], sizeof in.upd_k[r]);
    std::memcpy(d->upd_prod[q], in.upd_prod[r], sizeof in.upd_prod[r]);
    d->A[q] = in.A[r];
    d->beta[q] = in.beta[r];
    d->E[q] = in.E[r];
    d->A_low[q] = in.A_low[r];
    d->beta_low[q] = in.beta_low[r];
    d->E_low[q] = in.E_low[r];
    std::memcpy(d->troe[q], in.troe[r], sizeof in.troe[r]);
    d->dnu[q] = in.dnu[r];
    for (int k = 0; k < in.N; ++k) d->eff_t[k][q] = in.eff_t[k][r];
  }
}

// Tables for the integrators that skip inert species: the reaction lists
// renumbered over the species that react (mechanism order kept).
void reduce_dev_mech(const DevMech& full, DevMech* d) {
  *d = full;
  bool reacts[nrg::kMaxSpecies] = {};
  for (int r = 0; r < full.R; ++r) {
    for (int i = 0; i < full.nl[r]; ++i)
      if (full.left[r][i] >= 0) reacts[full.left[r][i]] = true;
    for (int i = 0; i < full.nr[r]; ++i)
      if (full.right[r][i] >= 0) reacts[full.right[r][i]] = true;
  }
  int int_of[nrg::kMaxSpecies];
  d->NI = 0;
  d->n_inert = 0;
  for (int k = 0; k < full.N; ++k) {
    if (reacts[k]) {
      int_of[k] = d->NI;
      d->full_of[d->NI++] = k;
    } else {
      int_of[k] = -1;
      d->inert_of[d->n_inert++] = k;
    }
  }
  for (int r = 0; r < full.R; ++r) {
    for (int i = 0; i < 3; ++i) {
      if (d->left[r][i] >= 0) d->left[r][i] = int_of[d->left[r][i]];
      if (d->right[r][i] >= 0) d->right[r][i] = int_of[d->right[r][i]];
    }
    for (int u = 0; u < d->nupd[r]; ++u) d->upd_k[r][u] = int_of[d->upd_k[r][u]];
  }
  if (d->NI <= nrg::kMergeUpTo) merge_equal_reactions(d);
}

void free_staging(nrg_chem* h) {
  cudaFree(h->d_T); cudaFree(h->d_rho); cudaFree(h->d_Y); cudaFree(h->d_Yp); cudaFree(h->d_Yp2);
  cudaFree(h->d_Ef); cudaFree(h->d_bc); cudaFree(h->d_status);
  cudaFreeHost(h->h_T); cudaFreeHost(h->h_rho); cudaFreeHost(h->h_Y); cudaFreeHost(h->h_Yp);
  cudaFreeHost(h->h_Yp2); cudaFreeHost(h->h_Ef); cudaFreeHost(h->h_bc); cudaFreeHost(h->h_status);
  h->d_T = h->d_rho = h->d_Y = h->d_Yp = h->d_Yp2 = h->d_Ef = nullptr;
  h->h_T = h->h_rho = h->h_Y = h->h_Yp = h->h_Yp2 = h->h_Ef = nullptr;
  h->d_bc = h->h_bc = nullptr;
  h->d_status = h->h_status = nullptr;
  h->cap = 0;
}

// Host threads for the gather and scatter of the host path: started once per
// process and kept (a step runs up to 16 parallel loops; starting threads for
// each cost more than the loops' own work on small chunks).  run(nt, f) calls
// f(0..nt-1) on the workers and the calling thread and returns when all are
// done; calls from several host threads are serialised.  A child process
// made by fork() starts its own pool (the parent's workers do not exist
// there).  The pool is never destroyed: its workers wait on a condition
// variable until the process ends.
class HostPool {
 public:
  static HostPool& get() {
    static std::mutex mu;
    static HostPool* pool = nullptr;
    static pid_t owner = 0;
    std::lock_guard<std::mutex> lk(mu);
    if (!pool || owner != getpid()) {
      pool = new HostPool();
      owner = getpid();
    }
    return *pool;
  }
  long size() const { return (long)workers_.size() + 1; }
  void run(long nt, const std::function<void(long)>& f) {
    if (nt <= 0) return;
    std::lock_guard<std::mutex> run_lk(run_mu_);
    if (workers_.empty() || nt == 1) {
      for (long i = 0; i < nt; ++i) f(i);
      return;
    }
    {
      std::lock_guard<std::mutex> lk(mu_);
      job_ = &f;
      ntasks_ = nt;
      next_.store(0);
      busy_ = (long)workers_.size();
      ++gen_;
    }
    cv_.notify_all();
    work();
    std::unique_lock<std::mutex> lk(mu_);
    done_.wait(lk, [&] { return busy_ == 0; });
    job_ = nullptr;
  }

 private:
  HostPool() {
    const unsigned hw = std::thread::hardware_concurrency();
    const long nw = std::max(0L, std::min(31L, (long)hw - 1));
    for (long i = 0; i < nw; ++i) {
      workers_.emplace_back([this] {
        unsigned long long seen = 0;
        for (;;) {
          {
            std::unique_lock<std::mutex> lk(mu_);
            cv_.wait(lk, [&] { return gen_ != seen; });
            seen = gen_;
          }
          work();
          std::lock_guard<std::mutex> lk(mu_);
          if (--busy_ == 0) done_.notify_one();
        }
      });
      workers_.back().detach();
    }
  }
  void work() {
    for (;;) {
      const long i = next_.fetch_add(1);
      if (i >= ntasks_) break;
      (*job_)(i);
    }
  }
  std::mutex run_mu_, mu_;
  std::condition_variable cv_, done_;
  std::vector<std::thread> workers_;
  const std::function<void(long)>* job_ = nullptr;
  long ntasks_ = 0, busy_ = 0;
  std::atomic<long> next_{0};
  unsigned long long gen_ = 0;
};

// Runs f(i) for every i in [r0, r1) on the host's hardware threads
// (contiguous blocks of indices per task).  Each task ends with a store
// fence, so the streaming stores below are visible before the loop returns
// (and before a copy engine reads what they wrote).
template <class F>
void parallel_rows(long r0, long r1, F f) {
  const long n = r1 - r0;
  if (n <= 0) return;
  HostPool& pool = HostPool::get();
  const long T = std::min(pool.size(), n);
  pool.run(T, [&](long t) {
    for (long r = r0 + n * t / T; r < r0 + n * (t + 1) / T; ++r) f(r);
#if defined(__SSE2__)
    _mm_sfence();
#endif
  });
}

// The host path's gather and scatter are bound by host memory bandwidth.
// Destinations that are written whole go through streaming (non-temporal)
// stores: a plain store first reads the destination's cache line, a third
// more traffic on a copy.
inline void stream_copy(double* dst, const double* src, long n) {
#if defined(__SSE2__)
  long i = 0;
  if (n > 0 && ((uintptr_t)dst & 15) != 0) {
    dst[0] = src[0];
    i = 1;
  }
  for (; i + 1 < n; i += 2) _mm_stream_pd(dst + i, _mm_loadu_pd(src + i));
  if (i < n) dst[i] = src[i];
#else
  std::memcpy(dst, src, (size_t)n * 8);
#endif
}

// y2[i] = src[i] in the cells the step did not skip (the reference leaves
// Y_prod2 as it was in skipped cells); streaming stores where both cells of
// an aligned pair are written.
inline void masked_y_prod2(double* y2, const double* src, const uint8_t* st, long n) {
#if defined(__SSE2__)
  long i = 0;
  if (n > 0 && ((uintptr_t)y2 & 15) != 0) {
    if (st[0] != NRG_CELL_SKIPPED) y2[0] = src[0];
    i = 1;
  }
  for (; i + 1 < n; i += 2) {
    const bool a = st[i] != NRG_CELL_SKIPPED, b = st[i + 1] != NRG_CELL_SKIPPED;
    if (a && b) {
      _mm_stream_pd(y2 + i, _mm_loadu_pd(src + i));
    } else {
      if (a) y2[i] = src[i];
      if (b) y2[i + 1] = src[i + 1];
    }
  }
  if (i < n && st[i] != NRG_CELL_SKIPPED) y2[i] = src[i];
#else
  for (long i = 0; i < n; ++i)
    if (st[i] != NRG_CELL_SKIPPED) y2[i] = src[i];
#endif
}

// yp[i] = Y_prod2 W / dt (the two IEEE operations the kernels evaluate), 0 in
// skipped cells.
inline void stream_y_prod(double* yp, const double* y2, const uint8_t* st, long n, double W, double dt) {
  auto v = [&](long i) { return st[i] == NRG_CELL_SKIPPED ? 0.0 : y2[i] * W / dt; };
#if defined(__SSE2__)
  long i = 0;
  if (n > 0 && ((uintptr_t)yp & 15) != 0) {
    yp[0] = v(0);
    i = 1;
  }
  for (; i + 1 < n; i += 2) _mm_stream_pd(yp + i, _mm_set_pd(v(i + 1), v(i)));
  if (i < n) yp[i] = v(i);
#else
  for (long i = 0; i < n; ++i) yp[i] = v(i);
#endif
}

int ensure_staging(nrg_chem* h, size_t n) {
  if (n <= h->cap) return NRG_OK;
  free_staging(h);
  const size_t N = (size_t)h->mech.n();
  CK(h, cudaMalloc(&h->d_T, n * 8));
  CK(h, cudaMalloc(&h->d_rho, n * 8));
  CK(h, cudaMalloc(&h->d_Y, N * n * 8));
  CK(h, cudaMalloc(&h->d_Yp, N * n * 8));
  CK(h, cudaMalloc(&h->d_Yp2, N * n * 8));
  CK(h, cudaMalloc(&h->d_Ef, n * 8));
  CK(h, cudaMalloc(&h->d_bc, n));
  CK(h, cudaMalloc(&h->d_status, n));
  CK(h, cudaMallocHost(&h->h_T, n * 8));
  CK(h, cudaMallocHost(&h->h_rho, n * 8));
  CK(h, cudaMallocHost(&h->h_Y, N * n * 8));
  CK(h, cudaMallocHost(&h->h_Yp, N * n * 8));
  CK(h, cudaMallocHost(&h->h_Yp2, N * n * 8));
  CK(h, cudaMallocHost(&h->h_Ef, n * 8));
  CK(h, cudaMallocHost(&h->h_bc, n));
  CK(h, cudaMallocHost(&h->h_status, n));
  h->cap = n;
  return NRG_OK;
}

int jac_of(int mode) { return mode == NRG_MODE_REFERENCE ? 0 : 1; }
int spec_of(const nrg_chem* h) { return h->mode == NRG_MODE_REFERENCE ? h->spec_full : h->spec; }

// Enqueue the plain integrator (no surrogate) on stream s.
cudaError_t enqueue_integrator(nrg_chem* h, const StepArgs& a, const LaunchCfg& cfg, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  if (cfg.kernel != nrg::kKernelThreadGrid) {
    e = cudaMemsetAsync(h->d_queue, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
  }
  LaunchCfg c = cfg;
  if (c.kernel == nrg::kKernelThreadQueue && c.grid <= 0) c.grid = h->num_sms;
  StepArgs b = a;
  b.eps = a.eps > 0.0 ? a.eps : h->eps;
  b.lu_rolled = c.lu_rolled;
  // a whole field with one dt: its cells in temperature order (lanes of a
  // warp then take similar BDF paths); lists built by the caller and the
  // per-cell-dt training states keep their own order
  if (h->order_cells && a.cell_list == nullptr && a.dt_cells == nullptr && a.n > 0 && a.n <= h->order_cap) {
    e = nrg::order_cells_by_temperature(a.n, a.T, a.bc, nullptr, &h->order, h->d_order_list, h->d_order_count,
                                        nullptr, s);
    if (e != cudaSuccess) return e;
    b.cell_list = h->d_order_list;
    b.n_list = (int)a.n;
    b.n_list_dev = nullptr;
  }
  return nrg::launch_chem(h->mech.n(), h->dmr.NI, spec_of(h), h->mech.r(), jac_of(h->mode), h->mode == NRG_MODE_MIXED, b, c,
                          h->d_queue, h->d_counters, s);
}

// The surrogate's FP64 fallback: the plain integrator at the fallback
// tolerance on the rejected cells' list.
nrg::FallbackFn integrator_fallback(nrg_chem* h, cudaEvent_t* ph) {
  return [h, ph](const StepArgs& fa, cudaStream_t fs) {
    if (ph) cudaEventRecord(ph[2], fs);
    StepArgs fb = fa;
    fb.eps = h->fallback_eps;
    cudaError_t e = enqueue_integrator(h, fb, h->cfg, fs);
    if (ph) cudaEventRecord(ph[3], fs);
    return e;
  };
}

// The step's kernels on stream s, adding to the device counters; ph: the
// phase events (or nullptr).
cudaError_t enqueue_step_body(nrg_chem* h, const StepArgs& a, cudaStream_t s, cudaEvent_t* ph) {
  if (h->mode == NRG_MODE_TABLE) {
    const nrg::TableArgs t{h->tab_rows, h->d_tab_T, h->d_tab_Y, h->tab_sorted ? 1 : 0, h->d_tab_idx,
                           (int)h->tab_idx.lo.size(), h->tab_idx.t0, h->tab_idx.inv_w};
    if (ph) cudaEventRecord(ph[2], s);
    cudaError_t e = nrg::launch_table_step(h->mech.n(), a, t, h->d_counters, s);
    if (ph) cudaEventRecord(ph[3], s);
    return e;
  }
  if (h->mode == NRG_MODE_SURROGATE)
    return nrg::surrogate_step(h->sur_net, a, h->cfg, h->d_queue, h->d_counters, s, integrator_fallback(h, ph),
                               ph);
  if (ph) cudaEventRecord(ph[2], s);
  cudaError_t e2 = enqueue_integrator(h, a, h->cfg, s);
  if (ph) cudaEventRecord(ph[3], s);
  return e2;
}

cudaError_t enqueue_step(nrg_chem* h, const StepArgs& a, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(h->d_counters, 0, sizeof(unsigned long long) * 8, s);
  if (e != cudaSuccess) return e;
  return enqueue_step_body(h, a, s, h->timing ? h->ph : nullptr);
}

// Runs the step on stream s, through a CUDA graph when enabled.
// The kernels read the mechanism from per-translation-unit __constant__
// tables, one set per device.  Before a handle launches work, its tables are
// put in place if another handle (possibly another mechanism) put its own
// there last; the switch waits for the device to be idle, so calls of
// handles with different tables are serialised rather than overlapped.
std::mutex g_tables_mu;
const nrg_chem* g_tables_owner[64] = {};

cudaError_t use_tables(nrg_chem* h) {
  std::lock_guard<std::mutex> lock(g_tables_mu);
  const int d = h->device;
  if (d < 0 || d >= 64) return cudaErrorInvalidDevice;
  if (g_tables_owner[d] == h) return cudaSuccess;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return e;
  nrg::upload_mechanism(h->dm, h->dmr, h->stream);
  nrg::surrogate_upload_tables(h->dm, h->stream);
  e = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) g_tables_owner[d] = h;
  return e;
}

void release_tables(const nrg_chem* h) {
  std::lock_guard<std::mutex> lock(g_tables_mu);
  for (auto& o : g_tables_owner)
    if (o == h) o = nullptr;
}

// Tables in place, surrogate ready and its scratch sized for up to n cells.
// Scratch of the temperature order for fields of up to n cells (grow-only,
// reserved before any graph capture).
int ensure_order(nrg_chem* h, long n) {
  if (!h->order_cells || n <= h->order_cap || n > (long)INT_MAX) return NRG_OK;
  cudaFree(h->d_order_list);
  h->d_order_list = nullptr;
  h->order_cap = 0;
  const std::string e = nrg::order_reserve(&h->order, n);
  if (!e.empty()) return fail(h, NRG_ERR_CUDA, e);
  if (!h->d_order_count) CK(h, cudaMalloc(&h->d_order_count, sizeof(int)));
  CK(h, cudaMalloc(&h->d_order_list, sizeof(int) * (size_t)n));
  h->order_cap = n;
  return NRG_OK;
}

int step_prepare(nrg_chem* h, long n) {
  CK(h, use_tables(h));
  if (h->mode == NRG_MODE_TABLE && h->tab_rows < 1)
    return fail(h, NRG_ERR_STATE, "table mode selected but no table is loaded (nrg_chem_load_table)");
  int rc = ensure_order(h, n);
  if (rc) return rc;
  if (h->mode == NRG_MODE_SURROGATE) {
    if (!(h->mech.n() == 9 && h->mech.r() == 24))
      return fail(h, NRG_ERR_UNSUPPORTED, "the surrogate is built for the 9-species, 24-reaction mechanism");
    if (!nrg::surrogate_ready(h->sur_net[0]))
      return fail(h, NRG_ERR_STATE, "surrogate mode selected but no trained model is loaded");
    const std::string e = nrg::surrogate_reserve(h->sur_net[0], n);
    if (!e.empty()) return fail(h, NRG_ERR_CUDA, e);
  }
  return NRG_OK;
}

// After the step's work was queued on s between h->ev0 and h->ev1: waits for
// it, fills stats (may be NULL) and checks the surrogate's error word.
int step_finish(nrg_chem* h, cudaStream_t s, long n, nrg_chem_stats* stats, bool phases = true) {
  CK(h, cudaMemcpyAsync(h->h_counters, h->d_counters, sizeof(unsigned long long) * 8,
                        cudaMemcpyDeviceToHost, s));
  CK(h, cudaStreamSynchronize(s));
  if (stats) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, h->ev0, h->ev1);
    std::memset(stats, 0, sizeof(*stats));
    stats->cells = n;
    stats->cells_active = (long long)h->h_counters[0];
    stats->steps = (long long)h->h_counters[1];
    stats->rhs_evals = (long long)h->h_counters[2];
    stats->jacobians = (long long)h->h_counters[3];
    stats->solves = (long long)h->h_counters[4];
    stats->cells_bad = (long long)h->h_counters[5];
    stats->cells_surrogate = (long long)h->h_counters[6];
    stats->cells_fallback = (long long)h->h_counters[7];
    if (h->mode == NRG_MODE_SURROGATE) stats->cells_active += stats->cells_surrogate;
    stats->device_ms = ms;
    if (h->timing && phases) {
      float p = 0.f;
      if (h->mode == NRG_MODE_SURROGATE) {
        cudaEventElapsedTime(&p, h->ev0, h->ph[1]);  // features + MLP (ph[1] = gate start)
        stats->phase_ms[0] = p;
        cudaEventElapsedTime(&p, h->ph[1], h->ph[2]);
        stats->phase_ms[1] = p;
      }
      cudaEventElapsedTime(&p, h->ph[2], h->ph[3]);
      stats->phase_ms[2] = p;
    }
  }
  if (h->mode == NRG_MODE_SURROGATE) {
    std::string e;
    for (int i = 0; i < nrg::kMaxNets && e.empty(); ++i) e = nrg::surrogate_check(h->sur_net[i], s);
    if (!e.empty()) return fail(h, NRG_ERR_CUDA, e);
  }
  return NRG_OK;
}

int run_step(nrg_chem* h, const StepArgs& a, cudaStream_t s, nrg_chem_stats* stats) {
  int rc = step_prepare(h, a.n);
  if (rc) return rc;
  CK(h, cudaEventRecord(h->ev0, s));
  if (h->timing) {
    for (int i = 0; i < 4; ++i) CK(h, cudaEventRecord(h->ph[i], s));
  }
  if (h->use_graph && !h->timing) {
    cudaGraph_t g = nullptr;
    CK(h, cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = enqueue_step(h, a, s);
    cudaError_t e2 = cudaStreamEndCapture(s, &g);
    if (e != cudaSuccess) { if (g) cudaGraphDestroy(g); return cuda_fail(h, e, "enqueue_step"); }
    if (e2 != cudaSuccess) return cuda_fail(h, e2, "cudaStreamEndCapture");
    bool updated = false;
    if (h->gexec) {
      cudaGraphExecUpdateResultInfo info;
      updated = cudaGraphExecUpdate(h->gexec, g, &info) == cudaSuccess;
      if (!updated) {
        cudaGetLastError();
        cudaGraphExecDestroy(h->gexec);
        h->gexec = nullptr;
      }
    }
    if (!h->gexec) {
      e = cudaGraphInstantiate(&h->gexec, g, 0);
      if (e != cudaSuccess) { cudaGraphDestroy(g); return cuda_fail(h, e, "cudaGraphInstantiate"); }
    }
    cudaGraphDestroy(g);
    CK(h, cudaGraphLaunch(h->gexec, s));
  } else {
    cudaError_t e = enqueue_step(h, a, s);
    if (e != cudaSuccess) return cuda_fail(h, e, "enqueue_step");
  }
  CK(h, cudaEventRecord(h->ev1, s));
  return step_finish(h, s, a.n, stats);
}

}  // namespace

// ------------------------------------------------------------------ API
extern "C" int nrg_chem_create(const char* mechanism_path, const char* thermo_path,
                               const char* molar_masses_path, double default_enhanced_efficiencies,
                               int eact_units, nrg_chem** out) {
  if (!mechanism_path || !thermo_path || !molar_masses_path || !out)
    return fail(nullptr, NRG_ERR_ARG, "null argument to nrg_chem_create");
  if (eact_units < 0 || eact_units > 3) return fail(nullptr, NRG_ERR_ARG, "unknown eact_units");
  *out = nullptr;
  nrg_chem* h = new nrg_chem();
  std::string e = nrg::load_mechanism(mechanism_path, thermo_path, molar_masses_path,
                                      default_enhanced_efficiencies, (nrg::EactUnits)eact_units, &h->mech);
  if (!e.empty()) { delete h; return fail(nullptr, NRG_ERR_IO, e); }
  e = build_dev_mech(h->mech, &h->dm);
  if (!e.empty()) { delete h; return fail(nullptr, NRG_ERR_UNSUPPORTED, e); }
  if (!nrg::supported_mechanism(h->mech.n(), h->mech.r())) {
    std::string msg = "no compiled kernel for " + std::to_string(h->mech.n()) + " species / " +
                      std::to_string(h->mech.r()) + " reactions";
    delete h;
    return fail(nullptr, NRG_ERR_UNSUPPORTED, msg);
  }
  cudaError_t ce;
  if ((ce = cudaGetDevice(&h->device)) != cudaSuccess ||
      (ce = cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, h->device)) != cudaSuccess ||
      (ce = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking)) != cudaSuccess ||
      (ce = cudaMalloc(&h->d_queue, sizeof(int) * 4)) != cudaSuccess ||
      (ce = cudaMalloc(&h->d_mech, sizeof(DevMech))) != cudaSuccess ||
      (ce = cudaMemcpy(h->d_mech, &h->dm, sizeof(DevMech), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (ce = cudaMalloc(&h->d_counters, sizeof(unsigned long long) * 8)) != cudaSuccess ||
      (ce = cudaMallocHost(&h->h_counters, sizeof(unsigned long long) * 8)) != cudaSuccess ||
      (ce = cudaEventCreate(&h->ev0)) != cudaSuccess || (ce = cudaEventCreate(&h->ev1)) != cudaSuccess ||
      (ce = cudaEventCreateWithFlags(&h->ev_in, cudaEventDisableTiming)) != cudaSuccess ||
      (ce = cudaEventCreate(&h->ph[0])) != cudaSuccess || (ce = cudaEventCreate(&h->ph[1])) != cudaSuccess ||
      (ce = cudaEventCreate(&h->ph[2])) != cudaSuccess || (ce = cudaEventCreate(&h->ph[3])) != cudaSuccess) {
    std::string msg = std::string("CUDA initialisation failed: ") + cudaGetErrorString(ce);
    nrg_chem_destroy(h);
    return fail(nullptr, NRG_ERR_CUDA, msg);
  }
  reduce_dev_mech(h->dm, &h->dmr);
  h->spec = nrg::match_specialised(h->dmr);
  h->spec_full = nrg::match_specialised_full(h->dm);
  for (int i = 0; i < nrg::kMaxNets; ++i) h->sur_net[i] = nrg::surrogate_create(h->dm);
  if ((ce = use_tables(h)) != cudaSuccess) {
    std::string msg = std::string("mechanism upload failed: ") + cudaGetErrorString(ce);
    nrg_chem_destroy(h);
    return fail(nullptr, NRG_ERR_CUDA, msg);
  }
  h->cfg.kernel = nrg::kKernelThreadGrid;  // the fastest shape measured on the flame field
  h->cfg.block = 32;
  h->cfg.grid = 0;
  h->cfg.chunk = 1;
  *out = h;
  return NRG_OK;
}

extern "C" int nrg_chem_destroy(nrg_chem* h) {
  if (!h) return NRG_ERR_ARG;
  release_tables(h);
  DeviceScope device_scope;  // frees on the handle's device whatever device is current
  device_scope.enter(h->device);
  if (h->stream) cudaStreamSynchronize(h->stream);
  if (h->gexec) cudaGraphExecDestroy(h->gexec);
  for (int i = 0; i < nrg::kMaxNets; ++i) nrg::surrogate_destroy(h->sur_net[i]);
  cudaFree(h->d_tab_T);
  cudaFree(h->d_tab_Y);
  cudaFree(h->d_tab_idx);
  free_staging(h);
  cudaFree(h->d_queue);
  cudaFree(h->d_mech);
  cudaFree(h->d_counters);
  nrg::order_free(&h->order);
  cudaFree(h->d_order_list);
  cudaFree(h->d_order_count);
  cudaFreeHost(h->h_counters);
  if (h->ev0) cudaEventDestroy(h->ev0);
  if (h->ev1) cudaEventDestroy(h->ev1);
  if (h->ev_in) cudaEventDestroy(h->ev_in);
  for (int i = 0; i < 4; ++i)
    if (h->ph[i]) cudaEventDestroy(h->ph[i]);
  if (h->stream) cudaStreamDestroy(h->stream);
  if (h->copy_in) cudaStreamDestroy(h->copy_in);
  if (h->copy_out) cudaStreamDestroy(h->copy_out);
  if (h->stream2) cudaStreamDestroy(h->stream2);
  if (h->ev_join) cudaEventDestroy(h->ev_join);
  for (cudaEvent_t* arr : {h->ev_h2d, h->ev_step, h->ev_chunk})
    for (int i = 0; i < 8; ++i)
      if (arr[i]) cudaEventDestroy(arr[i]);
  delete h;
  return NRG_OK;
}

extern "C" int nrg_chem_set_mode(nrg_chem* h, int mode) {
  if (!h) return NRG_ERR_ARG;
  if (mode < NRG_MODE_REFERENCE || mode > NRG_MODE_TABLE) return fail(h, NRG_ERR_ARG, "unknown mode");
  h->mode = mode;
  return NRG_OK;
}

extern "C" int nrg_chem_set_specialised(nrg_chem* h, int enable) {
  if (!h) return NRG_ERR_ARG;
  const int id = nrg::match_specialised(h->dmr);  // full lists that match reduce to lists that match
  if (enable && id == 0)
    return fail(h, NRG_ERR_UNSUPPORTED, "the mechanism matches none of the generated specialised codes");
  h->spec = enable ? id : 0;
  h->spec_full = enable ? nrg::match_specialised_full(h->dm) : 0;
  return NRG_OK;
}

extern "C" int nrg_chem_set_launch(nrg_chem* h, int kernel, int block, int grid, int chunk) {
  if (!h) return NRG_ERR_ARG;
  const bool ok_kernel = kernel >= 0 && kernel <= 2;
  const bool ok_block = kernel == 2 ? (block == 128 || block == 256) : (block == 32 || block == 64);
  if (!ok_kernel || !ok_block || chunk < 1 || chunk > 64 || grid < 0)
    return fail(h, NRG_ERR_ARG,
                "launch shape out of range (kernel 0/1: block 32 or 64; kernel 2: block 128 or 256; chunk 1..64)");
  h->cfg.kernel = kernel;
  h->cfg.block = block;
  h->cfg.grid = grid;
  h->cfg.chunk = chunk;
  return NRG_OK;
}

extern "C" int nrg_chem_set_lu_form(nrg_chem* h, int rolled) {
  if (!h) return NRG_ERR_ARG;
  h->cfg.lu_rolled = rolled != 0;
  return NRG_OK;
}

extern "C" int nrg_chem_get_lu_form(nrg_chem* h, int* rolled) {
  if (!h || !rolled) return NRG_ERR_ARG;
  *rolled = h->cfg.lu_rolled;
  return NRG_OK;
}

extern "C" int nrg_chem_get_launch(nrg_chem* h, int* kernel, int* block, int* grid, int* chunk) {
  if (!h) return NRG_ERR_ARG;
  if (kernel) *kernel = h->cfg.kernel;
  if (block) *block = h->cfg.block;
  if (grid) *grid = h->cfg.grid;
  if (chunk) *chunk = h->cfg.chunk;
  return NRG_OK;
}

extern "C" int nrg_chem_set_graph(nrg_chem* h, int enable) {
  if (!h) return NRG_ERR_ARG;
  h->use_graph = enable != 0;
  return NRG_OK;
}

extern "C" int nrg_chem_set_cell_order(nrg_chem* h, int enable) {
  if (!h) return NRG_ERR_ARG;
  h->order_cells = enable != 0;
  if (h->sur_net[0]) nrg::surrogate_set_cell_order(h->sur_net[0], h->order_cells);
  return NRG_OK;
}

extern "C" int nrg_chem_set_eps(nrg_chem* h, double eps) {
  if (!h) return NRG_ERR_ARG;
  if (!(eps >= 0.0) || !(eps < 1.0)) return fail(h, NRG_ERR_ARG, "eps must be in [0, 1); 0 restores the reference's 1e-9");
  h->eps = eps;
  return NRG_OK;
}

extern "C" int nrg_chem_set_timing(nrg_chem* h, int enable) {
  if (!h) return NRG_ERR_ARG;
  h->timing = enable != 0;
  return NRG_OK;
}

extern "C" int nrg_chem_step_device(nrg_chem* h, double time_step, long n, long ld, const double* T,
                                    const double* rho, const double* Y, const signed char* bc,
                                    double* Y_prod, double* Y_prod2, double* E_f_prod, double* T_after,
                                    unsigned char* status, void* stream, nrg_chem_stats* stats) {
  if (!h) return NRG_ERR_ARG;
  if (n < 0 || ld < n) return fail(h, NRG_ERR_ARG, "need 0 <= n <= ld");
  if (!(time_step > 0.0) || !std::isfinite(time_step)) return fail(h, NRG_ERR_ARG, "time_step must be > 0");
  if (n > 0 && (!T || !rho || !Y || !Y_prod || !Y_prod2 || !E_f_prod))
    return fail(h, NRG_ERR_ARG, "null field pointer");
  if (n > 0x7fffffffL / 2) return fail(h, NRG_ERR_ARG, "too many cells for one call");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  StepArgs a;
  a.n = n;
  a.ld = ld;
  a.dt = time_step;
  a.T = T;
  a.rho = rho;
  a.Y = Y;
  a.bc = (const int8_t*)bc;
  a.Y_prod = Y_prod;
  a.Y_prod2 = Y_prod2;
  a.E_f_prod = E_f_prod;
  a.T_after = T_after;
  a.status = status;
  a.mxstep = 10000;
  a.mech = h->d_mech;
  a.dt_cells = nullptr;
  a.cell_list = nullptr;
  a.n_list = 0;
  a.n_list_dev = nullptr;
  if (n == 0) {
    if (stats) std::memset(stats, 0, sizeof(*stats));
    return NRG_OK;
  }
  // Work runs on the handle's own (capturable) stream, ordered after
  // everything already queued on the caller's stream (legacy default included).
  CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)stream));
  CK(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  return run_step(h, a, h->stream, stats);
}

extern "C" int nrg_chem_step(nrg_chem* h, double time_step, const nrg_field_desc* f, nrg_chem_stats* stats) {
  if (!h || !f) return NRG_ERR_ARG;
  ON_DEVICE(h);
  const int N = h->mech.n();
  long ext[3], cnt[3];
  for (int d = 0; d < 3; ++d) {
    ext[d] = (long)f->ub[d] - f->lb[d] + 1;
    if (ext[d] <= 0 || f->lo[d] < f->lb[d] || f->hi[d] > f->ub[d])
      return fail(h, NRG_ERR_ARG, "field bounds inconsistent (need lb <= lo, hi <= ub)");
    cnt[d] = f->hi[d] >= f->lo[d] ? (long)f->hi[d] - f->lo[d] + 1 : 0;
  }
  if (!f->T || !f->rho || !f->E_f_prod) return fail(h, NRG_ERR_ARG, "null T, rho or E_f_prod");
  for (int k = 0; k < N; ++k)
    if (!f->Y[k] || !f->Y_prod[k] || !f->Y_prod2[k]) return fail(h, NRG_ERR_ARG, "null species array");
  const long n = cnt[0] * cnt[1] * cnt[2];
  if (n == 0) {
    if (stats) std::memset(stats, 0, sizeof(*stats));
    return NRG_OK;
  }
  if (!(time_step > 0.0)) return fail(h, NRG_ERR_ARG, "time_step must be > 0");
  int rc = ensure_staging(h, (size_t)n);
  if (rc) return rc;
  if (!h->copy_in) {
    CK(h, cudaStreamCreateWithFlags(&h->copy_in, cudaStreamNonBlocking));
    CK(h, cudaStreamCreateWithFlags(&h->copy_out, cudaStreamNonBlocking));
    CK(h, cudaStreamCreateWithFlags(&h->stream2, cudaStreamNonBlocking));
    CK(h, cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming));
    for (cudaEvent_t* arr : {h->ev_h2d, h->ev_step, h->ev_chunk})
      for (int i = 0; i < 8; ++i) CK(h, cudaEventCreateWithFlags(&arr[i], cudaEventDisableTiming));
  }
  rc = step_prepare(h, n);
  if (rc) return rc;
  const bool sur = h->mode == NRG_MODE_SURROGATE, table = h->mode == NRG_MODE_TABLE;
  // The interior is handled as rows along i (contiguous in the reference's
  // column-major arrays), split into up to eight chunks of rows.  Per chunk
  // the host gathers on all its threads into pinned staging and copies in on
  // copy_in; the host gathers chunk p + 1 while chunk p is copied.
  // * integrator and table modes: each chunk is stepped as it arrives,
  //   copied out on copy_out and scattered while later chunks are stepped
  //   (on the 2048 x 2048 flame field this beats one launch over the whole
  //   field after the last chunk: 90 against 96 ms);
  // * surrogate mode: each chunk goes through the networks, the gate and
  //   the FP64 fallback of its rejected cells as it arrives, and is copied
  //   out and scattered while later chunks arrive (one fallback launch per
  //   chunk: 17.4 ms per flame step, against 19.7 ms with two fallbacks over
  //   half the field each and a packed read-back of the rejected cells);
  //   odd chunks run on a second stream with their own scratch, so that the
  //   chunks' tails of slow cells overlap (15.7 ms).
  // Every mode but the table writes Y_prod = Y_prod2 W / dt: only Y_prod2
  // crosses PCIe and the host rebuilds Y_prod with the same two operations.
  const bool derive_yp = !table;
  const long rowlen = cnt[0], nrow = cnt[1] * cnt[2];
  auto row_base = [&](long r) {
    const int j = f->lo[1] + (int)(r % cnt[1]), k = f->lo[2] + (int)(r / cnt[1]);
    return ((long)(k - f->lb[2]) * ext[1] + (j - f->lb[1])) * ext[0] + (f->lo[0] - f->lb[0]);
  };
  const int P = (int)std::min<long>(8, nrow);
  const size_t rb = (size_t)rowlen * 8;
  cudaStream_t s = h->stream, ci = h->copy_in, co = h->copy_out;
  auto chunk_cells = [&](int p, long* c0, long* nc) {
    const long r0 = nrow * p / P, r1 = nrow * (p + 1) / P;
    *c0 = r0 * rowlen;
    *nc = (r1 - r0) * rowlen;
  };
  auto args_of = [&](long c0, long nc) {
    StepArgs a;
    a.n = nc;
    a.ld = n;
    a.dt = time_step;
    a.T = h->d_T + c0;
    a.rho = h->d_rho + c0;
    a.Y = h->d_Y + c0;
    a.bc = h->d_bc + c0;
    a.Y_prod = h->d_Yp + c0;
    a.Y_prod2 = h->d_Yp2 + c0;
    a.E_f_prod = h->d_Ef + c0;
    a.T_after = nullptr;
    a.status = h->d_status + c0;
    a.mxstep = 10000;
    a.mech = h->d_mech;
    a.dt_cells = nullptr;
    a.cell_list = nullptr;
    a.n_list = 0;
    a.n_list_dev = nullptr;
    return a;
  };
  // chunk p's outputs back to the host once event `ready` has fired on s
  auto copy_out = [&](int p, cudaEvent_t ready) -> int {
    long c0, nc;
    chunk_cells(p, &c0, &nc);
    CK(h, cudaStreamWaitEvent(co, ready, 0));
    for (int sp = 0; sp < N; ++sp) {
      if (!derive_yp)
        CK(h, cudaMemcpyAsync(h->h_Yp + (size_t)sp * n + c0, h->d_Yp + (size_t)sp * n + c0, nc * 8,
                              cudaMemcpyDeviceToHost, co));
      CK(h, cudaMemcpyAsync(h->h_Yp2 + (size_t)sp * n + c0, h->d_Yp2 + (size_t)sp * n + c0, nc * 8,
                            cudaMemcpyDeviceToHost, co));
    }
    CK(h, cudaMemcpyAsync(h->h_Ef + c0, h->d_Ef + c0, nc * 8, cudaMemcpyDeviceToHost, co));
    CK(h, cudaMemcpyAsync(h->h_status + c0, h->d_status + c0, nc, cudaMemcpyDeviceToHost, co));
    CK(h, cudaEventRecord(h->ev_chunk[p], co));
    return NRG_OK;
  };
  using clk = std::chrono::steady_clock;
  auto ms_since = [](clk::time_point t0) { return std::chrono::duration<double, std::milli>(clk::now() - t0).count(); };
  const clk::time_point t_call = clk::now();
  double host_ms[2] = {0.0, 0.0};  // gather, scatter (with its waits for the chunks)
  CK(h, cudaMemsetAsync(h->d_counters, 0, sizeof(unsigned long long) * 8, s));
  CK(h, cudaEventRecord(h->ev0, s));
  // surrogate mode: even chunks on the compute stream, odd ones on a second
  // stream with their own scratch (lane 1), so that one chunk's networks,
  // gate and fallback fill the other's tail of slow cells.  The plain
  // integrator's queue kernels share a queue head, so only the grid kernel
  // takes part.
  const bool two_lanes = sur && P > 1 && nrg::surrogate_fused(h->sur_net[0]) &&
                         h->cfg.kernel == nrg::kKernelThreadGrid;
  if (two_lanes) {
    long max_nc = 0;
    for (int p = 0; p < P; ++p) {
      long a0, an;
      chunk_cells(p, &a0, &an);
      max_nc = std::max(max_nc, an);
    }
    const std::string le = nrg::surrogate_reserve_lane1(h->sur_net[0], max_nc);
    if (!le.empty()) return fail(h, NRG_ERR_CUDA, le);
    CK(h, cudaStreamWaitEvent(h->stream2, h->ev0, 0));  // after the counters are cleared
  }
  for (int p = 0; p < P; ++p) {
    long c0, nc;
    chunk_cells(p, &c0, &nc);
    const clk::time_point tg = clk::now();
    parallel_rows(nrow * p / P, nrow * (p + 1) / P, [&](long r) {
      const long L = row_base(r), c = r * rowlen;
      stream_copy(h->h_T + c, f->T + L, rowlen);
      stream_copy(h->h_rho + c, f->rho + L, rowlen);
      if (f->bc_markers)
        std::memcpy(h->h_bc + c, f->bc_markers + L, (size_t)rowlen);
      else
        std::memset(h->h_bc + c, 0, (size_t)rowlen);
      for (int sp = 0; sp < N; ++sp) stream_copy(h->h_Y + (size_t)sp * n + c, f->Y[sp] + L, rowlen);
    });
    host_ms[0] += ms_since(tg);
    CK(h, cudaMemcpyAsync(h->d_T + c0, h->h_T + c0, nc * 8, cudaMemcpyHostToDevice, ci));
    CK(h, cudaMemcpyAsync(h->d_rho + c0, h->h_rho + c0, nc * 8, cudaMemcpyHostToDevice, ci));
    CK(h, cudaMemcpyAsync(h->d_bc + c0, h->h_bc + c0, nc, cudaMemcpyHostToDevice, ci));
    for (int sp = 0; sp < N; ++sp)
      CK(h, cudaMemcpyAsync(h->d_Y + (size_t)sp * n + c0, h->h_Y + (size_t)sp * n + c0, nc * 8,
                            cudaMemcpyHostToDevice, ci));
    CK(h, cudaEventRecord(h->ev_h2d[p], ci));
    const int lane = two_lanes ? (p & 1) : 0;
    cudaStream_t sp = lane ? h->stream2 : s;
    CK(h, cudaStreamWaitEvent(sp, h->ev_h2d[p], 0));
    const cudaError_t e = sur ? nrg::surrogate_gate(h->sur_net, args_of(c0, nc), c0, h->d_counters, sp, nullptr, lane)
                              : enqueue_step_body(h, args_of(c0, nc), s, nullptr);
    if (e != cudaSuccess) return cuda_fail(h, e, sur ? "surrogate_gate" : "enqueue_step");
    if (sur) {
      // the chunk's rejected cells right after its gate, so that its outputs
      // are final when it is copied out
      const cudaError_t ef = nrg::surrogate_fallback(h->sur_net, args_of(c0, nc), c0, h->d_counters, sp,
                                                     integrator_fallback(h, nullptr), lane);
      if (ef != cudaSuccess) return cuda_fail(h, ef, "surrogate_fallback");
    }
    CK(h, cudaEventRecord(h->ev_step[p], sp));
    if ((rc = copy_out(p, h->ev_step[p]))) return rc;
  }
  if (two_lanes) {
    CK(h, cudaEventRecord(h->ev_join, h->stream2));
    CK(h, cudaStreamWaitEvent(s, h->ev_join, 0));
  }
  CK(h, cudaEventRecord(h->ev1, s));
  const double* W = h->mech.molar_mass.data();
  const clk::time_point ts = clk::now();
  for (int p = 0; p < P; ++p) {
    CK(h, cudaEventSynchronize(h->ev_chunk[p]));
    parallel_rows(nrow * p / P, nrow * (p + 1) / P, [&](long r) {
      const long L = row_base(r), c = r * rowlen;
      stream_copy(f->E_f_prod + L, h->h_Ef + c, rowlen);
      const uint8_t* stc = h->h_status + c;
      for (int sp = 0; sp < N; ++sp) {
        double* y2 = f->Y_prod2[sp] + L;
        const double* src = h->h_Yp2 + (size_t)sp * n + c;
        if (derive_yp) {
          stream_y_prod(f->Y_prod[sp] + L, src, stc, rowlen, W[sp], time_step);
          masked_y_prod2(y2, src, stc, rowlen);
        } else {
          std::memcpy(f->Y_prod[sp] + L, h->h_Yp + (size_t)sp * n + c, rb);
          for (long i = 0; i < rowlen; ++i)
            if (stc[i] != NRG_CELL_SKIPPED) y2[i] = src[i];
        }
      }
    });
  }
  host_ms[1] = ms_since(ts);
  rc = step_finish(h, s, n, stats, false);  // host times instead of the phase events
  if (rc == NRG_OK && stats && h->timing) {
    for (int i = 0; i < 2; ++i) stats->phase_ms[i] = host_ms[i];
    stats->phase_ms[3] = ms_since(t_call);
  }
  return rc;
}

extern "C" int nrg_chem_autotune(nrg_chem* h, double time_step, long n, long ld, const double* T,
                                 const double* rho, const double* Y, const signed char* bc, double* Y_prod,
                                 double* Y_prod2, double* E_f_prod, double* ms_best) {
  if (!h) return NRG_ERR_ARG;
  if (n <= 0 || ld < n || !T || !rho || !Y || !Y_prod || !Y_prod2 || !E_f_prod)
    return fail(h, NRG_ERR_ARG, "autotune needs device inputs with n > 0");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  if (int rc = ensure_order(h, n)) return rc;
  StepArgs a;
  a.n = n; a.ld = ld; a.dt = time_step; a.T = T; a.rho = rho; a.Y = Y; a.bc = (const int8_t*)bc;
  a.Y_prod = Y_prod; a.Y_prod2 = Y_prod2; a.E_f_prod = E_f_prod; a.T_after = nullptr; a.status = nullptr;
  a.mxstep = 10000;
  a.mech = h->d_mech;
  a.dt_cells = nullptr;
  a.cell_list = nullptr;
  a.n_list = 0;
  a.n_list_dev = nullptr;
  // candidate shapes: warp per cell (occupancy-derived persistent grid),
  // thread per cell from the work queue (1 or 2 blocks of 64 per SM, chunk 1
  // or 2) and thread per cell over the plain grid (32- or 64-thread blocks, LU
  // unrolled or as a loop).  The integrator in passes chooses its blocks and
  // has one LU form, so there the grid is one candidate, the caller's block and
  // LU form are kept for the kernels they matter to, and the queue's blocks
  // are the 2 or 4 of 64 that fit an SM.
  const bool passes = nrg::integrates_in_passes(jac_of(h->mode), h->dmr.NI);
  std::vector<LaunchCfg> cands;
  for (int block : {128, 256}) {
    LaunchCfg c;
    c.kernel = nrg::kKernelWarpQueue;
    c.block = block;
    c.grid = 0;
    c.chunk = 1;
    cands.push_back(c);
  }
  for (int half : {1, 2})
    for (int chunk : {1, 2}) {
      const int per_sm = passes ? 2 * half : half;
      LaunchCfg c;
      c.kernel = nrg::kKernelThreadQueue;
      c.block = 64;
      c.grid = per_sm * h->num_sms;
      c.chunk = chunk;
      cands.push_back(c);
    }
  if (passes) {
    LaunchCfg c;
    c.kernel = nrg::kKernelThreadGrid;
    cands.push_back(c);
    for (LaunchCfg& k : cands) {
      k.lu_rolled = h->cfg.lu_rolled;
      if (k.kernel != nrg::kKernelWarpQueue && h->cfg.kernel != nrg::kKernelWarpQueue) k.block = h->cfg.block;
    }
  } else {
    for (int block : {32, 64})
      for (int rolled : {0, 1}) {
        LaunchCfg c;
        c.kernel = nrg::kKernelThreadGrid;
        c.block = block;
        c.lu_rolled = rolled;
        cands.push_back(c);
      }
  }
  cudaStream_t s = h->stream;
  float best = 1e30f;
  LaunchCfg best_cfg = h->cfg;
  for (const LaunchCfg& c : cands) {
    // two launches per shape, the second one timed (the first pays for
    // the kernel's first-use set-up)
    for (int rep = 0; rep < 2; ++rep) {
      CK(h, cudaMemsetAsync(h->d_counters, 0, sizeof(unsigned long long) * 8, s));
      CK(h, cudaEventRecord(h->ev0, s));
      cudaError_t e = enqueue_integrator(h, a, c, s);
      if (e == cudaErrorNotSupported) {  // shape not compiled for this mechanism
        cudaGetLastError();
        CK(h, cudaStreamSynchronize(s));
        break;
      }
      if (e != cudaSuccess) return cuda_fail(h, e, "autotune launch");
      CK(h, cudaEventRecord(h->ev1, s));
      CK(h, cudaStreamSynchronize(s));
      float ms = 0.f;
      cudaEventElapsedTime(&ms, h->ev0, h->ev1);
      if (rep == 1 && ms < best) { best = ms; best_cfg = c; }
    }
  }
  h->cfg = best_cfg;
  if (ms_best) *ms_best = best;
  return NRG_OK;
}

extern "C" int nrg_chem_apply_state_device(nrg_chem* h, double time_step, long n, long ld, int dims,
                                           const double* rho, const double* Y_prod, const double* E_f_prod,
                                           const signed char* bc, double* Y, double* E_f, const double* v,
                                           double* T, double* p, double* gamma, double* cp_mass, double* h_s,
                                           double* h_full, double* v_s, double* mix_mol_mass,
                                           unsigned char* status, void* stream) {
  if (!h) return NRG_ERR_ARG;
  if (n < 0 || ld < n || dims < 0 || dims > 3 || (dims > 0 && !v) ||
      (n > 0 && (!rho || !Y || !E_f || !T || !p || !gamma)) || ((Y_prod || E_f_prod) && !(time_step > 0.0)))
    return fail(h, NRG_ERR_ARG, "bad arguments to nrg_chem_apply_state_device");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)stream));
  CK(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  nrg::ApplyStateArgs a{};
  a.n = n; a.ld = ld; a.dims = dims; a.dt = time_step; a.rho = rho; a.Y_prod = Y_prod; a.E_f_prod = E_f_prod;
  a.bc = (const int8_t*)bc; a.Y = Y; a.E_f = E_f; a.v = v; a.T = T; a.p = p; a.gamma = gamma;
  a.cp_mass = cp_mass; a.h_s = h_s; a.h_full = h_full; a.v_s = v_s; a.mix_mol_mass = mix_mol_mass;
  a.status = status;
  const cudaError_t e = nrg::launch_apply_state(h->mech.n(), a, h->stream);
  if (e != cudaSuccess) return cuda_fail(h, e, "state equation launch");
  CK(h, cudaStreamSynchronize(h->stream));
  return NRG_OK;
}

extern "C" int nrg_species_predictor_device(nrg_chem* h, double time_step, const nrg_grid_desc* grid,
                                            const double* const* v_f, const double* x_center, const signed char* bc,
                                            const double* Y_prod_diff, const double* Y_prod_chem,
                                            int n_particle_phases, const double* const* Y_prod_particles,
                                            double* rho, double* Y, double* rho_old, double* Y_old, double* rho_int,
                                            double* Y_int, void* stream) {
  if (!h) return NRG_ERR_ARG;
  nrg::PredictorArgs a;
  const int N = h->mech.n();
  bool ok = grid && N <= nrg::kPredictorMaxSpecies && v_f && rho && Y && rho_old && Y_old && rho_int && Y_int &&
            n_particle_phases >= 0 && n_particle_phases <= nrg::kPredictorMaxParticlePhases &&
            (n_particle_phases == 0 || Y_prod_particles) && std::isfinite(time_step) &&
            nrg::predictor_grid(a, grid->dims, grid->n) && grid->coord >= 0 && grid->coord <= 2 &&
            (grid->coord == 0 || x_center) && grid->dx > 0.0;
  if (ok) {
    for (int d = 0; d < grid->dims; ++d) ok = ok && v_f[d];
    for (int p = 0; p < n_particle_phases; ++p) ok = ok && Y_prod_particles[p];
    ok = ok && grid->ld >= a.e[0] * a.e[1] * a.e[2];
  }
  if (!ok) return fail(h, NRG_ERR_ARG, "bad arguments to nrg_species_predictor_device");
  a.coord = grid->coord;
  a.ld = (long)grid->ld;
  a.dx = grid->dx;
  a.inv_dx = 1.0 / grid->dx;
  a.dt = time_step;
  for (int s = 0; s < N; ++s) a.W[s] = h->dm.W[s];
  a.rho = rho; a.Y = Y;
  for (int d = 0; d < grid->dims; ++d) a.v_f[d] = v_f[d];
  a.x_center = x_center; a.bc = (const int8_t*)bc;
  a.Y_prod_diff = Y_prod_diff; a.Y_prod_chem = Y_prod_chem;
  a.n_part = n_particle_phases;
  for (int p = 0; p < n_particle_phases; ++p) a.Y_prod_part[p] = Y_prod_particles[p];
  a.rho_old = rho_old; a.Y_old = Y_old; a.rho_int = rho_int; a.Y_int = Y_int;
  a.rho_out = rho; a.Y_out = Y;
  ON_DEVICE(h);
  CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)stream));
  CK(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  const cudaError_t e = nrg::launch_species_predictor(N, a, h->stream);
  if (e == cudaErrorNotSupported) return fail(h, NRG_ERR_UNSUPPORTED, "no species predictor for this species count");
  if (e != cudaSuccess) return cuda_fail(h, e, "species predictor launch");
  CK(h, cudaStreamSynchronize(h->stream));
  return NRG_OK;
}

extern "C" int nrg_chem_load_transport(nrg_chem* h, const char* transport_path) {
  if (!h || !transport_path) return NRG_ERR_ARG;
  const int N = h->mech.n();
  if (N > nrg::kDiffMaxSpecies) return fail(h, NRG_ERR_UNSUPPORTED, "too many species for the diffusivity kernel");
  const std::string e = nrg::load_transport(transport_path, &h->mech);
  if (!e.empty()) return fail(h, NRG_ERR_IO, e);
  nrg::DiffusivityArgs& d = h->diff;
  d = nrg::DiffusivityArgs();
  d.N = N;
  for (int k = 0; k < N; ++k) d.W[k] = h->mech.molar_mass[k];
  int q = 0;
  double uniq[nrg::kDiffMaxPairs];
  for (int i = 0; i < N - 1; ++i)
    for (int j = i + 1; j < N; ++j, ++q) {
      const double eps_i = h->mech.well_depth[i], eps_j = h->mech.well_depth[j];
      const double bdc = h->mech.binary_diffusivity[(size_t)i * N + j];
      if (!(bdc > 0.0 && eps_i > 0.0 && eps_j > 0.0)) continue;
      d.ibdc[q] = 1.0 / bdc;
      const double sq = std::sqrt(eps_i * eps_j);
      int u = 0;
      while (u < d.n_uniq && uniq[u] != sq) ++u;
      if (u == d.n_uniq) {
        uniq[d.n_uniq++] = sq;
        d.uniq_isq[u] = 1.0 / sq;
        const long double c = 1.06036L * powl(sq / 1024.0L, 0.15610L);
        d.uniq_pow[u] = (double)c;
        d.uniq_pow_lo[u] = (double)(c - d.uniq_pow[u]);
      }
      d.pair_u[q] = (unsigned char)u;
    }
  h->has_transport = true;
  return NRG_OK;
}

extern "C" int nrg_mech_transport_tables(const char* mechanism_path, const char* thermo_path,
                                         const char* molar_masses_path, const char* transport_path,
                                         double* well_depth, double* collision_diameter,
                                         double* binary_diffusivity) {
  if (!mechanism_path || !thermo_path || !molar_masses_path || !transport_path)
    return fail(nullptr, NRG_ERR_ARG, "null path");
  nrg::Mechanism m;
  std::string e = nrg::load_mechanism(mechanism_path, thermo_path, molar_masses_path, 1.0, nrg::EactUnits::cal_mol, &m);
  if (e.empty()) e = nrg::load_transport(transport_path, &m);
  if (!e.empty()) return fail(nullptr, NRG_ERR_IO, e);
  const int N = m.n();
  for (int k = 0; k < N; ++k) {
    if (well_depth) well_depth[k] = m.well_depth[k];
    if (collision_diameter) collision_diameter[k] = m.collision_diameter[k];
  }
  if (binary_diffusivity)
    for (size_t i = 0; i < (size_t)N * N; ++i) binary_diffusivity[i] = m.binary_diffusivity[i];
  return NRG_OK;
}

extern "C" int nrg_mixture_diffusivity_device(nrg_chem* h, long n, long ld, const double* T, const double* p,
                                              const double* Y, const double* mix_mol_mass, const signed char* bc,
                                              double* D, void* stream) {
  if (!h) return NRG_ERR_ARG;
  if (!h->has_transport) return fail(h, NRG_ERR_STATE, "no transport deck loaded (nrg_chem_load_transport)");
  if (n < 0 || ld < n || (n > 0 && (!T || !p || !Y || !mix_mol_mass || !D)))
    return fail(h, NRG_ERR_ARG, "bad arguments to nrg_mixture_diffusivity_device");
  nrg::DiffusivityArgs a = h->diff;
  a.n = n; a.ld = ld; a.T = T; a.p = p; a.Y = Y; a.m_mix = mix_mol_mass; a.bc = (const int8_t*)bc; a.D = D;
  ON_DEVICE(h);
  CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)stream));
  CK(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  const cudaError_t e = nrg::launch_mixture_diffusivity(a, h->stream);
  if (e != cudaSuccess) return cuda_fail(h, e, "diffusivity launch");
  CK(h, cudaStreamSynchronize(h->stream));
  return NRG_OK;
}

extern "C" int nrg_chem_info(nrg_chem* h, int* n_species, int* n_reactions) {
  if (!h) return NRG_ERR_ARG;
  if (n_species) *n_species = h->mech.n();
  if (n_reactions) *n_reactions = h->mech.r();
  return NRG_OK;
}

static void fill_tables(const nrg::Mechanism& m, int* reaction_type, int* coeffs, double* arrhenius,
                        double* troe3, double* eff, double* a_coeffs, double* molar_mass) {
  const int N = m.n(), R = m.r();
  for (int r = 0; r < R; ++r) {
    const nrg::Reaction& rx = m.reactions[r];
    if (reaction_type) reaction_type[r] = rx.type;
    if (coeffs) {
      int* L = coeffs + (0 * R + r) * 4;
      int* P = coeffs + (1 * R + r) * 4;
      L[0] = rx.n_left; P[0] = rx.n_right;
      for (int i = 0; i < 3; ++i) { L[1 + i] = rx.left[i]; P[1 + i] = rx.right[i]; }
    }
    if (arrhenius) {
      double* A = arrhenius + r * 9;
      A[0] = rx.A; A[1] = rx.beta; A[2] = rx.E; A[3] = rx.A_low; A[4] = rx.beta_low; A[5] = rx.E_low;
      A[6] = rx.troe[0]; A[7] = rx.troe[1]; A[8] = rx.troe[2];
    }
    if (troe3) troe3[r] = rx.troe[3];
  }
  if (eff) std::memcpy(eff, m.eff.data(), sizeof(double) * (size_t)R * N);
  if (a_coeffs) std::memcpy(a_coeffs, m.a_coeffs.data(), sizeof(double) * (size_t)N * 14);
  if (molar_mass) std::memcpy(molar_mass, m.molar_mass.data(), sizeof(double) * (size_t)N);
}

extern "C" int nrg_chem_tables(nrg_chem* h, int* reaction_type, int* coeffs, double* arrhenius, double* troe3,
                               double* eff, double* a_coeffs, double* molar_mass) {
  if (!h) return NRG_ERR_ARG;
  fill_tables(h->mech, reaction_type, coeffs, arrhenius, troe3, eff, a_coeffs, molar_mass);
  return NRG_OK;
}

extern "C" int nrg_mech_tables(const char* mechanism_path, const char* thermo_path,
                               const char* molar_masses_path, double default_enhanced_efficiencies,
                               int eact_units, int* n_species, int* n_reactions, int* reaction_type,
                               int* coeffs, double* arrhenius, double* troe3, double* eff,
                               double* a_coeffs, double* molar_mass) {
  if (!mechanism_path || !thermo_path || !molar_masses_path)
    return fail(nullptr, NRG_ERR_ARG, "null path");
  if (eact_units < 0 || eact_units > 3) return fail(nullptr, NRG_ERR_ARG, "unknown eact_units");
  nrg::Mechanism m;
  std::string e = nrg::load_mechanism(mechanism_path, thermo_path, molar_masses_path,
                                      default_enhanced_efficiencies, (nrg::EactUnits)eact_units, &m);
  if (!e.empty()) return fail(nullptr, NRG_ERR_IO, e);
  if (n_species) *n_species = m.n();
  if (n_reactions) *n_reactions = m.r();
  fill_tables(m, reaction_type, coeffs, arrhenius, troe3, eff, a_coeffs, molar_mass);
  return NRG_OK;
}

extern "C" int nrg_chem_species_name(nrg_chem* h, int k, char* buf, int buflen) {
  if (!h || !buf || buflen <= 0 || k < 0 || k > h->mech.n()) return NRG_ERR_ARG;
  std::string s = k == h->mech.n() ? std::string("M") : h->mech.species[k];
  std::snprintf(buf, (size_t)buflen, "%s", s.c_str());
  return NRG_OK;
}

extern "C" const char* nrg_chem_last_error(nrg_chem* h) {
  return h ? h->err.c_str() : g_create_error.c_str();
}

extern "C" int nrg_selftest_bounded_wait(long long limit_ns, int* timed_out, double* waited_ms) {
  if (limit_ns <= 0 || limit_ns > 2000000000LL || !timed_out) return NRG_ERR_ARG;
  const std::string e = nrg::bounded_wait_probe((unsigned long long)limit_ns, timed_out, waited_ms);
  return e.empty() ? NRG_OK : fail(nullptr, NRG_ERR_CUDA, e);
}

extern "C" int nrg_fp64_peak_tflops(double* tflops) {
  if (!tflops) return NRG_ERR_ARG;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return NRG_ERR_CUDA;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double* out = nullptr;
  if (cudaMalloc(&out, 8) != cudaSuccess) return NRG_ERR_CUDA;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int blocks = sms * 8, threads = 256, iters = 4096;
  nrg::launch_fp64_peak(out, blocks, threads, 64, nullptr);  // warm-up
  cudaEventRecord(e0);
  nrg::launch_fp64_peak(out, blocks, threads, iters, nullptr);
  cudaEventRecord(e1);
  cudaError_t e = cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return NRG_ERR_CUDA;
  const double flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return NRG_OK;
}

// ---------------------------------------------------------------- table
extern "C" int nrg_table_read(const char* path, int n_species, long capacity, double* T_t, double* Y_t,
                              long* rows) {
  if (!path || !rows || n_species < 1 || n_species > NRG_MAX_SPECIES || (T_t && (!Y_t || capacity < 1)))
    return fail(nullptr, NRG_ERR_ARG, "bad arguments to nrg_table_read");
  nrg::ChemTable t;
  const std::string e = nrg::read_chem_table(path, n_species, &t);
  if (!e.empty()) return fail(nullptr, NRG_ERR_IO, e);
  *rows = t.rows;
  if (!T_t) return NRG_OK;
  if (capacity < t.rows) return fail(nullptr, NRG_ERR_ARG, "nrg_table_read: capacity below the table's rows");
  std::copy(t.T.begin(), t.T.end(), T_t);
  for (int k = 0; k < n_species; ++k)
    std::copy(t.Y.begin() + (size_t)k * t.rows, t.Y.begin() + (size_t)(k + 1) * t.rows, Y_t + (size_t)k * capacity);
  return NRG_OK;
}

extern "C" int nrg_table_write(const char* path, int n_species, const char* const* species_names,
                               const nrg_field_desc* f) {
  if (!path || !species_names || !f || !f->T || n_species < 1 || n_species > NRG_MAX_SPECIES)
    return fail(nullptr, NRG_ERR_ARG, "bad arguments to nrg_table_write");
  for (int k = 0; k < n_species; ++k)
    if (!f->Y_prod2[k] || !species_names[k]) return fail(nullptr, NRG_ERR_ARG, "null Y_prod2 array or species name");
  for (int d = 1; d < 3; ++d)
    if (f->lb[d] > 1 || f->ub[d] < 1)
      return fail(nullptr, NRG_ERR_ARG, "the table is written from the row j = 1, k = 1, which the arrays must hold");
  if (f->lo[0] < f->lb[0] || f->hi[0] > f->ub[0]) return fail(nullptr, NRG_ERR_ARG, "interior outside the arrays");
  const long e0 = (long)f->ub[0] - f->lb[0] + 1, e1 = (long)f->ub[1] - f->lb[1] + 1;
  const long row = ((long)(1 - f->lb[2]) * e1 + (1 - f->lb[1])) * e0;  // cells(lb0, 1, 1)
  auto at = [&](int i) { return row + (i - f->lb[0]); };
  // write_chemical_kinetics_table (chemical_kinetics_solver.f90:574-582):
  // first interior cell between 300.5 and 310 K, first cell of the largest T
  double max_T = 0.0;
  int first = 0, last = 0;
  for (int i = f->lo[0]; i <= f->hi[0]; ++i) {
    const double t = f->T[at(i)];
    if (t > 300.5 && t < 310.0 && first == 0) first = i;
    if (t > max_T) {
      last = i;
      max_T = t;
    }
  }
  if (first <= last && (first < f->lb[0] || last > f->ub[0]))
    return fail(nullptr, NRG_ERR_ARG, "the tabulated rows reach outside the arrays (no cell between 300.5 and 310 K)");
  std::vector<std::string> names;
  for (int k = 0; k < n_species; ++k) names.emplace_back(species_names[k]);
  const std::string e = nrg::write_chem_table(
      path, names, first, last, [&](int i) { return f->T[at(i)]; },
      [&](int k, int i) { return f->Y_prod2[k][at(i)]; });
  return e.empty() ? NRG_OK : fail(nullptr, NRG_ERR_IO, e);
}

extern "C" int nrg_chem_set_table(nrg_chem* h, long rows, const double* T_t, const double* Y_t) {
  if (!h) return NRG_ERR_ARG;
  if (rows < 1 || !T_t || !Y_t) return fail(h, NRG_ERR_ARG, "a table needs at least one row");
  ON_DEVICE(h);
  CK(h, cudaStreamSynchronize(h->stream));
  cudaFree(h->d_tab_T);
  cudaFree(h->d_tab_Y);
  cudaFree(h->d_tab_idx);
  h->d_tab_T = h->d_tab_Y = nullptr;
  h->d_tab_idx = nullptr;
  h->tab_idx = nrg::TableIndex();
  h->tab_rows = 0;
  const size_t N = (size_t)h->mech.n();
  CK(h, cudaMalloc(&h->d_tab_T, sizeof(double) * (size_t)rows));
  CK(h, cudaMalloc(&h->d_tab_Y, sizeof(double) * (size_t)rows * N));
  CK(h, cudaMemcpy(h->d_tab_T, T_t, sizeof(double) * (size_t)rows, cudaMemcpyHostToDevice));
  CK(h, cudaMemcpy(h->d_tab_Y, Y_t, sizeof(double) * (size_t)rows * N, cudaMemcpyHostToDevice));
  const std::vector<double> nodes(T_t, T_t + rows);
  h->tab_sorted = nrg::table_nodes_sorted(nodes);
  // Sorted nodes: a bucket index of 4,096 buckets (32 KB) narrows each
  // cell's bisection to the few nodes of its bucket.
  if (h->tab_sorted && nrg::build_table_index(nodes, 4096, &h->tab_idx)) {
    std::vector<int2> pairs(h->tab_idx.lo.size());
    for (size_t j = 0; j < pairs.size(); ++j) pairs[j] = make_int2(h->tab_idx.lo[j], h->tab_idx.hi[j]);
    CK(h, cudaMalloc(&h->d_tab_idx, sizeof(int2) * pairs.size()));
    CK(h, cudaMemcpy(h->d_tab_idx, pairs.data(), sizeof(int2) * pairs.size(), cudaMemcpyHostToDevice));
  } else {
    h->tab_idx = nrg::TableIndex();
  }
  h->tab_rows = rows;
  return NRG_OK;
}

extern "C" int nrg_chem_load_table(nrg_chem* h, const char* path) {
  if (!h || !path) return NRG_ERR_ARG;
  nrg::ChemTable t;
  const std::string e = nrg::read_chem_table(path, h->mech.n(), &t);
  if (!e.empty()) return fail(h, NRG_ERR_IO, e);
  return nrg_chem_set_table(h, t.rows, t.T.data(), t.Y.data());
}

// ------------------------------------------------------------- surrogate
namespace {
int order_after_legacy(nrg_chem* h) {
  CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)0));
  CK(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
  return NRG_OK;
}
int sfail(nrg_chem* h, const std::string& e) { return e.empty() ? NRG_OK : fail(h, NRG_ERR_CUDA, e); }
constexpr int kNormFloats = 4 * nrg::kMlpIn + nrg::kMlpOut + 4;
void norm_to_floats(const nrg::MlpNorm& m, float* f) {
  int k = 0;
  for (int j = 0; j < nrg::kMlpIn; ++j) f[k++] = m.x_mu[j];
  for (int j = 0; j < nrg::kMlpIn; ++j) f[k++] = m.x_sd[j];
  for (int j = 0; j < nrg::kMlpIn; ++j) f[k++] = m.x_min[j];
  for (int j = 0; j < nrg::kMlpIn; ++j) f[k++] = m.x_max[j];
  for (int j = 0; j < nrg::kMlpOut; ++j) f[k++] = m.y_sd[j];
  f[k++] = m.hull_margin;
  f[k++] = m.dt_pow;
  f[k++] = m.log_mask;
  f[k++] = m.log_eps;
}
nrg::MlpNorm floats_to_norm(const float* f) {
  nrg::MlpNorm m{};
  int k = 0;
  for (int j = 0; j < nrg::kMlpIn; ++j) m.x_mu[j] = f[k++];
  for (int j = 0; j < nrg::kMlpIn; ++j) m.x_sd[j] = f[k++];
  for (int j = 0; j < nrg::kMlpIn; ++j) m.x_min[j] = f[k++];
  for (int j = 0; j < nrg::kMlpIn; ++j) m.x_max[j] = f[k++];
  for (int j = 0; j < nrg::kMlpOut; ++j) m.y_sd[j] = f[k++];
  m.hull_margin = f[k++];
  m.dt_pow = f[k++];
  m.log_mask = f[k++];
  m.log_eps = f[k++];
  return m;
}
}  // namespace

extern "C" int nrg_surrogate_param_count(void) { return nrg::surrogate_param_count(); }

extern "C" int nrg_surrogate_select(nrg_chem* h, int net) {
  if (!h) return NRG_ERR_ARG;
  if (net < 0 || net >= nrg::kMaxNets) return fail(h, NRG_ERR_ARG, "network index must be 0 (main) to 7");
  h->sur_sel = net;
  return NRG_OK;
}
extern "C" int nrg_surrogate_norm_count(void) { return kNormFloats; }

extern "C" int nrg_surrogate_init(nrg_chem* h, unsigned long long seed) {
  if (!h) return NRG_ERR_ARG;
  ON_DEVICE(h);
  CK(h, use_tables(h));
  return sfail(h, nrg::surrogate_init(h->sur_net[h->sur_sel], seed, h->stream));
}

extern "C" int nrg_surrogate_get_params(nrg_chem* h, float* params) {
  if (!h || !params) return NRG_ERR_ARG;
  ON_DEVICE(h);
  return sfail(h, nrg::surrogate_get_params(h->sur_net[h->sur_sel], params, h->stream));
}

extern "C" int nrg_surrogate_set_params(nrg_chem* h, const float* params) {
  if (!h || !params) return NRG_ERR_ARG;
  ON_DEVICE(h);
  return sfail(h, nrg::surrogate_set_params(h->sur_net[h->sur_sel], params, h->stream));
}

extern "C" int nrg_surrogate_get_norm(nrg_chem* h, float* norm) {
  if (!h || !norm) return NRG_ERR_ARG;
  norm_to_floats(nrg::surrogate_get_norm(h->sur_net[h->sur_sel]), norm);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_norm(nrg_chem* h, const float* norm) {
  if (!h || !norm) return NRG_ERR_ARG;
  ON_DEVICE(h);
  return sfail(h, nrg::surrogate_set_norm(h->sur_net[h->sur_sel], floats_to_norm(norm)));
}

extern "C" int nrg_surrogate_prepare(nrg_chem* h, long n, long ld, double dt, const double* dt_cells,
                                     const double* T, const double* rho, const double* Y, const double* Y_prod,
                                     const double* T_after, const nrg_surrogate_opts* opts, void* x_bf16,
                                     float* y) {
  if (!h || n <= 0 || ld < n || !T || !rho || !Y || !Y_prod || !T_after || !opts || !x_bf16 || !y)
    return fail(h, NRG_ERR_ARG, "bad arguments to nrg_surrogate_prepare");
  if (!(opts->hull_margin >= 0.f) || !(opts->log_eps > 0.f) || (opts->log_mask >> 9))
    return fail(h, NRG_ERR_ARG, "bad nrg_surrogate_opts (hull_margin >= 0, log_eps > 0, log_mask < 512)");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  int rc = order_after_legacy(h);
  if (rc) return rc;
  const nrg::PrepareOpts o{opts->hull_margin, opts->dt_pow, opts->log_mask, opts->log_eps, opts->common_dY_scale};
  return sfail(h, nrg::surrogate_prepare(h->sur_net[h->sur_sel], n, ld, dt, dt_cells, T, rho, Y, Y_prod, T_after, o,
                                         (__nv_bfloat16*)x_bf16, y, h->stream));
}

extern "C" int nrg_surrogate_features(nrg_chem* h, long n, long ld, double dt, const double* dt_cells,
                                      const double* T, const double* rho, const double* Y, float* xraw,
                                      void* x_bf16) {
  if (!h || n < 0 || ld < n || (n > 0 && (!T || !rho || !Y))) return fail(h, NRG_ERR_ARG, "bad features args");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  int rc = order_after_legacy(h);
  if (rc) return rc;
  std::string e = nrg::surrogate_features(h->sur_net[h->sur_sel], n, ld, dt, dt_cells, T, rho, Y, xraw, (__nv_bfloat16*)x_bf16,
                                          h->stream);
  if (!e.empty()) return sfail(h, e);
  CK(h, cudaStreamSynchronize(h->stream));
  return NRG_OK;
}

extern "C" int nrg_surrogate_forward(nrg_chem* h, long n, const void* x_bf16, float* out) {
  if (!h || n <= 0 || !x_bf16 || !out) return fail(h, NRG_ERR_ARG, "bad forward args");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  int rc = order_after_legacy(h);
  if (rc) return rc;
  return sfail(h, nrg::surrogate_forward(h->sur_net[h->sur_sel], n, (const __nv_bfloat16*)x_bf16, out, h->stream));
}

extern "C" int nrg_surrogate_grad(nrg_chem* h, long n, const void* x_bf16, const float* y, float* grads_host,
                                  double* loss_host) {
  if (!h || n <= 0 || !x_bf16 || !y) return fail(h, NRG_ERR_ARG, "bad grad args");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  int rc = order_after_legacy(h);
  if (rc) return rc;
  return sfail(h, nrg::surrogate_grad(h->sur_net[h->sur_sel], n, (const __nv_bfloat16*)x_bf16, y, grads_host, loss_host, h->stream));
}

extern "C" int nrg_surrogate_train(nrg_chem* h, long n, const void* x_bf16, const float* y, int epochs, int batch,
                                   float lr, unsigned long long seed, float* loss_per_epoch) {
  if (!h || n <= 0 || !x_bf16 || !y || epochs <= 0 || !(lr > 0.f)) return fail(h, NRG_ERR_ARG, "bad train args");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  int rc = order_after_legacy(h);
  if (rc) return rc;
  return sfail(h, nrg::surrogate_train(h->sur_net[h->sur_sel], n, (const __nv_bfloat16*)x_bf16, y, epochs, batch, lr, seed,
                                       loss_per_epoch, h->stream));
}

extern "C" int nrg_surrogate_set_gate(nrg_chem* h, double elem_tol, double raw_elem_tol, double dT_tol,
                                      double dT_max) {
  if (!h || !(elem_tol >= 0) || !(raw_elem_tol >= 0) || !(dT_tol >= 0) || !(dT_max >= 0)) return NRG_ERR_ARG;
  nrg::surrogate_set_gate(h->sur_net[h->sur_sel], elem_tol, raw_elem_tol, dT_tol, dT_max);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_band(nrg_chem* h, double T_lo, double T_hi) {
  if (!h) return NRG_ERR_ARG;
  const bool unset = T_lo == 0.0 && T_hi == 0.0;
  if (!(T_lo == T_lo) || !(T_hi == T_hi)) return fail(h, NRG_ERR_ARG, "routing band bounds must be numbers");
  nrg::surrogate_set_band(h->sur_net[h->sur_sel], !unset, T_lo, T_hi);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_partner(nrg_chem* h, int partner, double agree_Y, double agree_T) {
  if (!h) return NRG_ERR_ARG;
  if (partner < -1 || partner >= nrg::kMaxNets || partner == h->sur_sel || !(agree_Y >= 0) || !(agree_T >= 0))
    return fail(h, NRG_ERR_ARG, "partner must be -1 or another network (0..7), agreement bounds >= 0");
  nrg::surrogate_set_partner(h->sur_net[h->sur_sel], partner, agree_Y, agree_T);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_fallback_eps(nrg_chem* h, double eps) {
  if (!h) return NRG_ERR_ARG;
  if (!(eps >= 0.0) || !(eps < 1.0)) return fail(h, NRG_ERR_ARG, "fallback eps must be in [0, 1)");
  h->fallback_eps = eps;
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_gate_band(nrg_chem* h, int band, double dt_max, double elem_tol,
                                           double raw_elem_tol, double dT_tol, double dT_max) {
  if (!h) return NRG_ERR_ARG;
  if (band < 1 || band >= nrg::kGateBands || !(dt_max >= 0.0) || !(elem_tol >= 0.0) || !(raw_elem_tol >= 0.0) ||
      !(dT_tol >= 0.0) || !(dT_max >= 0.0))
    return fail(h, NRG_ERR_ARG, "gate band must be 1..3 with non-negative bounds");
  nrg::surrogate_set_gate_band(h->sur_net[h->sur_sel], band, dt_max, elem_tol, raw_elem_tol, dT_tol, dT_max);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_dt_band(nrg_chem* h, double dt_lo, double dt_hi) {
  if (!h) return NRG_ERR_ARG;
  if (!(dt_lo >= 0.0) || !(dt_hi > dt_lo)) return fail(h, NRG_ERR_ARG, "step band needs 0 <= dt_lo < dt_hi");
  nrg::surrogate_set_dt_band(h->sur_net[h->sur_sel], dt_lo, dt_hi);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_gate_dt(nrg_chem* h, double dt_max) {
  if (!h || !(dt_max > 0)) return NRG_ERR_ARG;
  nrg::surrogate_set_gate_dt(h->sur_net[h->sur_sel], dt_max);
  return NRG_OK;
}

extern "C" int nrg_surrogate_set_inference(nrg_chem* h, int fused) {
  if (!h) return NRG_ERR_ARG;
  nrg::surrogate_set_fused(h->sur_net[0], fused != 0);
  return NRG_OK;
}

extern "C" int nrg_surrogate_infer(nrg_chem* h, long n, long ld, double dt, const double* dt_cells, const double* T,
                                   const double* rho, const double* Y, float* out) {
  if (!h || n < 0 || ld < n || (n > 0 && (!T || !rho || !Y || !out)) || (!(dt > 0.0) && !dt_cells))
    return fail(h, NRG_ERR_ARG, "bad arguments to nrg_surrogate_infer");
  ON_DEVICE(h);
  CK(h, use_tables(h));
  int rc = order_after_legacy(h);
  if (rc) return rc;
  StepArgs a{};
  a.n = n; a.ld = ld; a.dt = dt > 0.0 ? dt : 1.0; a.dt_cells = dt_cells; a.T = T; a.rho = rho; a.Y = Y;
  a.mech = h->d_mech;
  return sfail(h, nrg::surrogate_infer(h->sur_net[h->sur_sel], a, out, h->stream));
}

extern "C" int nrg_surrogate_enable(nrg_chem* h, int enable) {
  if (!h) return NRG_ERR_ARG;
  nrg::surrogate_set_ready(h->sur_net[h->sur_sel], enable != 0);
  return NRG_OK;
}

extern "C" int nrg_surrogate_save(nrg_chem* h, const char* path) {
  if (!h || !path) return NRG_ERR_ARG;
  const int P = nrg::surrogate_param_count();
  std::vector<float> p((size_t)P), nm(kNormFloats);
  int rc = nrg_surrogate_get_params(h, p.data());
  if (rc) return rc;
  norm_to_floats(nrg::surrogate_get_norm(h->sur_net[h->sur_sel]), nm.data());
  FILE* f = std::fopen(path, "wb");
  if (!f) return fail(h, NRG_ERR_IO, std::string("cannot write ") + path);
  const char magic[8] = {'N', 'R', 'G', 'S', 'U', 'R', '3', '\0'};
  bool ok = std::fwrite(magic, 1, 8, f) == 8 && std::fwrite(&P, 4, 1, f) == 1 &&
            std::fwrite(p.data(), 4, (size_t)P, f) == (size_t)P &&
            std::fwrite(nm.data(), 4, (size_t)kNormFloats, f) == (size_t)kNormFloats;
  ok = (std::fclose(f) == 0) && ok;
  return ok ? NRG_OK : fail(h, NRG_ERR_IO, std::string("short write to ") + path);
}

extern "C" int nrg_surrogate_load(nrg_chem* h, const char* path) {
  if (!h || !path) return NRG_ERR_ARG;
  FILE* f = std::fopen(path, "rb");
  if (!f) return fail(h, NRG_ERR_IO, std::string("cannot read ") + path);
  char magic[8];
  int P = 0;
  const int want = nrg::surrogate_param_count();
  std::vector<float> p((size_t)want), nm(kNormFloats);
  bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "NRGSUR3", 8) == 0 &&
            std::fread(&P, 4, 1, f) == 1 && P == want && std::fread(p.data(), 4, (size_t)P, f) == (size_t)P &&
            std::fread(nm.data(), 4, (size_t)kNormFloats, f) == (size_t)kNormFloats;
  std::fclose(f);
  if (!ok) return fail(h, NRG_ERR_IO, std::string("not a surrogate model file: ") + path);
  int rc = nrg_surrogate_set_params(h, p.data());
  if (rc) return rc;
  rc = nrg_surrogate_set_norm(h, nm.data());
  if (rc) return rc;
  nrg::surrogate_set_ready(h->sur_net[h->sur_sel], true);
  return NRG_OK;
}

extern "C" int nrg_chem_integrate(nrg_chem* h, long n, long ld, double dt, const double* dt_cells,
                                  const double* T, const double* rho, const double* Y, const signed char* bc,
                                  double* Y_prod, double* Y_prod2, double* E_f_prod, double* T_after,
                                  unsigned char* status, void* stream, nrg_chem_stats* stats) {
  if (!h) return NRG_ERR_ARG;
  const int saved = h->mode;
  if (h->mode == NRG_MODE_SURROGATE) h->mode = NRG_MODE_FAST;
  if (n < 0 || ld < n || (!(dt > 0.0) && !dt_cells)) { h->mode = saved; return fail(h, NRG_ERR_ARG, "bad integrate args"); }
  if (n > 0 && (!T || !rho || !Y || !Y_prod || !Y_prod2 || !E_f_prod)) {
    h->mode = saved;
    return fail(h, NRG_ERR_ARG, "null field pointer");
  }
  ON_DEVICE(h);
  CK(h, use_tables(h));
  StepArgs a{};
  a.n = n; a.ld = ld; a.dt = dt > 0.0 ? dt : 1.0; a.T = T; a.rho = rho; a.Y = Y; a.bc = (const int8_t*)bc;
  a.Y_prod = Y_prod; a.Y_prod2 = Y_prod2; a.E_f_prod = E_f_prod; a.T_after = T_after; a.status = status;
  a.mxstep = 10000; a.mech = h->d_mech; a.dt_cells = dt_cells; a.cell_list = nullptr; a.n_list = 0;
  a.n_list_dev = nullptr;
  int rc = NRG_OK;
  if (n == 0) {
    if (stats) std::memset(stats, 0, sizeof(*stats));
  } else {
    CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)stream));
    CK(h, cudaStreamWaitEvent(h->stream, h->ev_in, 0));
    rc = run_step(h, a, h->stream, stats);
  }
  h->mode = saved;
  return rc;
}

// ------------------------------------------------- no-allocation step
// nrg_chem_step_device_noalloc: the compacted FP64 integration (skip rule ->
// order-preserving list of active cells -> integrator over the list) with all
// of its scratch -- cell flags, per-block counts and offsets, the cell list,
// the work-queue head and the statistics counters -- in one file-scope device
// array instead of memory allocated by the library.  It serves callers that
// must not allocate device memory during a step.
namespace {

constexpr long kNaMaxCells = 1L << 20;  // 1,048,576 cells per call
constexpr int kNaBlock = 1024;
constexpr int kNaMaxBlocks = (int)(kNaMaxCells / kNaBlock);
constexpr size_t kNaOffQueue = 0;                    // int
constexpr size_t kNaOffNList = 4;                    // int
constexpr size_t kNaOffCounters = 64;                // 8 x unsigned long long
constexpr size_t kNaOffBlockCount = 256;             // kNaMaxBlocks x int
constexpr size_t kNaOffBlockOff = 256 + 4 * kNaMaxBlocks;
constexpr size_t kNaOffList = 256 + 8 * kNaMaxBlocks;  // kNaMaxCells x int (256-aligned)
constexpr size_t kNaOffFlag = kNaOffList + 4 * (size_t)kNaMaxCells;
constexpr size_t kNaBytes = kNaOffFlag + (size_t)kNaMaxCells;  // about 5.3 MB
static_assert(kNaOffList % 256 == 0, "cell list must stay 256-byte aligned");

}  // namespace

// Every GPU that loads the library holds this array until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

namespace {

std::mutex g_na_mutex;
unsigned char* g_na_addr[64] = {};  // device address of g_noalloc_scratch per device

// Set-up, once per device, with that device current: the array's name is only
// a host-side stand-in, so the kernels get the address the runtime reports.
unsigned char* noalloc_scratch(int dev, std::string* err) {
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (dev < 0 || dev >= 64) {
    *err = "device ordinal out of range for the no-allocation scratch table";
    return nullptr;
  }
  if (!g_na_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      *err = std::string("cudaGetSymbolAddress(no-allocation scratch): ") + cudaGetErrorString(e);
      return nullptr;
    }
    g_na_addr[dev] = static_cast<unsigned char*>(p);
  }
  return g_na_addr[dev];
}

__global__ void k_na_flag(StepArgs a, int n_species, unsigned char* flag) {
  for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < a.n; c += (long)gridDim.x * blockDim.x) {
    const double Tc = a.T[c];
    const bool active = nrg::reference_cell_active(Tc, a.bc, c);
    flag[c] = active ? 1 : 0;
    if (!active) nrg::write_skipped_cell(a, c, n_species, Tc);
  }
}

__global__ void k_na_count(long n, const unsigned char* flag, int* block_count) {
  const long i = (long)blockIdx.x * kNaBlock + threadIdx.x;
  const int cnt = __syncthreads_count(i < n ? (int)flag[i] : 0);
  if (threadIdx.x == 0) block_count[blockIdx.x] = cnt;
}

__global__ void k_na_scan(int nb, const int* block_count, int* block_off, int* total) {
  __shared__ int wsum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < nb; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < nb ? block_count[i] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
      int s = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      wsum[lane] = s;
    }
    __syncthreads();
    const int incl = x + (w > 0 ? wsum[w - 1] : 0);
    if (i < nb) block_off[i] = carry + incl - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry += incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void k_na_compact(long n, const unsigned char* flag, const int* block_off, int* list) {
  __shared__ int wcount[kNaBlock / 32];
  const long i = (long)blockIdx.x * kNaBlock + threadIdx.x;
  const int f = i < n ? (int)flag[i] : 0;
  const unsigned bal = __ballot_sync(0xffffffffu, f);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) wcount[w] = __popc(bal);
  __syncthreads();
  int before = 0;
  for (int q = 0; q < w; ++q) before += wcount[q];
  if (f) list[block_off[blockIdx.x] + before + __popc(bal & ((1u << lane) - 1u))] = (int)i;
}

}  // namespace

extern "C" int nrg_chem_step_device_noalloc(nrg_chem* h, double time_step, long n, long ld, const double* T,
                                            const double* rho, const double* Y, const signed char* bc,
                                            double* Y_prod, double* Y_prod2, double* E_f_prod, double* T_after,
                                            unsigned char* status, void* stream, nrg_chem_stats* stats) {
  if (!h) return NRG_ERR_ARG;
  if (n < 0 || ld < n) return fail(h, NRG_ERR_ARG, "need 0 <= n <= ld");
  if (n > kNaMaxCells)
    return fail(h, NRG_ERR_ARG,
                "nrg_chem_step_device_noalloc takes at most 1048576 cells per call (its scratch is a fixed "
                "device array); split the field or use nrg_chem_step_device");
  if (!(time_step > 0.0) || !std::isfinite(time_step)) return fail(h, NRG_ERR_ARG, "time_step must be > 0");
  if (n > 0 && (!T || !rho || !Y || !Y_prod || !Y_prod2 || !E_f_prod))
    return fail(h, NRG_ERR_ARG, "null field pointer");
  if (h->mode == NRG_MODE_SURROGATE || h->mode == NRG_MODE_TABLE)
    return fail(h, NRG_ERR_STATE,
                "the no-allocation step integrates (reference, fast or mixed mode); use nrg_chem_step_device");
  if (n == 0) {
    if (stats) std::memset(stats, 0, sizeof(*stats));
    return NRG_OK;
  }
  ON_DEVICE(h);
  CK(h, use_tables(h));
  std::string err;
  unsigned char* base = noalloc_scratch(h->device, &err);
  if (!base) return fail(h, NRG_ERR_CUDA, err);
  int* queue = reinterpret_cast<int*>(base + kNaOffQueue);
  int* n_list = reinterpret_cast<int*>(base + kNaOffNList);
  unsigned long long* counters = reinterpret_cast<unsigned long long*>(base + kNaOffCounters);
  int* block_count = reinterpret_cast<int*>(base + kNaOffBlockCount);
  int* block_off = reinterpret_cast<int*>(base + kNaOffBlockOff);
  int* list = reinterpret_cast<int*>(base + kNaOffList);
  unsigned char* flag = base + kNaOffFlag;

  cudaStream_t s = h->stream;
  CK(h, cudaEventRecord(h->ev_in, (cudaStream_t)stream));
  CK(h, cudaStreamWaitEvent(s, h->ev_in, 0));
  StepArgs a{};
  a.n = n;
  a.ld = ld;
  a.dt = time_step;
  a.T = T;
  a.rho = rho;
  a.Y = Y;
  a.bc = (const int8_t*)bc;
  a.Y_prod = Y_prod;
  a.Y_prod2 = Y_prod2;
  a.E_f_prod = E_f_prod;
  a.T_after = T_after;
  a.status = status;
  a.mxstep = 10000;
  a.mech = h->d_mech;
  a.dt_cells = nullptr;
  a.cell_list = nullptr;
  a.n_list = 0;
  a.n_list_dev = nullptr;
  const int nb = (int)((n + kNaBlock - 1) / kNaBlock);
  CK(h, cudaEventRecord(h->ev0, s));
  // queue head, list length and counters start at zero on every call
  CK(h, cudaMemsetAsync(base, 0, kNaOffBlockCount, s));
  k_na_flag<<<(unsigned)std::min<long>((n + 255) / 256, 148L * 16), 256, 0, s>>>(a, h->mech.n(), flag);
  k_na_count<<<nb, kNaBlock, 0, s>>>(n, flag, block_count);
  k_na_scan<<<1, 1024, 0, s>>>(nb, block_count, block_off, n_list);
  k_na_compact<<<nb, kNaBlock, 0, s>>>(n, flag, block_off, list);
  CK(h, cudaGetLastError());
  StepArgs fa = a;
  fa.cell_list = list;
  fa.n_list = (int)n;  // grid bound; the kernels read the device-side count
  fa.n_list_dev = n_list;
  LaunchCfg cfg = h->cfg;
  if (cfg.kernel == nrg::kKernelThreadQueue && cfg.grid <= 0) cfg.grid = h->num_sms;
  const cudaError_t le = nrg::launch_chem(h->mech.n(), h->dmr.NI, spec_of(h), h->mech.r(), jac_of(h->mode), h->mode == NRG_MODE_MIXED,
                                          fa, cfg, queue, counters, s);
  if (le != cudaSuccess) return cuda_fail(h, le, "no-allocation integrator launch");
  CK(h, cudaEventRecord(h->ev1, s));
  CK(h, cudaMemcpyAsync(h->h_counters, counters, sizeof(unsigned long long) * 8, cudaMemcpyDeviceToHost, s));
  CK(h, cudaStreamSynchronize(s));
  if (stats) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, h->ev0, h->ev1);
    std::memset(stats, 0, sizeof(*stats));
    stats->cells = n;
    stats->cells_active = (long long)h->h_counters[0];
    stats->steps = (long long)h->h_counters[1];
    stats->rhs_evals = (long long)h->h_counters[2];
    stats->jacobians = (long long)h->h_counters[3];
    stats->solves = (long long)h->h_counters[4];
    stats->cells_bad = (long long)h->h_counters[5];
    stats->device_ms = ms;
  }
  return NRG_OK;
}
