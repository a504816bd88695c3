// Batched TM runs and reverse sweeps on the chip (dn_resident2d.cuh, struct
// List): which CTA takes which bands of which grids, and the entry points.
#include <algorithm>
#include <climits>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

#include "dn_resident2d.cuh"
#include "dn_sample_dft.cuh"

namespace dn {

long long batch2d_inst_offset(const dn_batch2d* cfg, const dn_batch2d_inst* insts);

namespace res {
namespace {

// samples of one launch, and grids (their monitors' kernels take one per blockIdx.y);
// more go in further launches
constexpr long long GROUP_SAMPLE_BYTES = 1LL << 30;
constexpr int GROUP_GRIDS = 65535;

// The blob: Head | ListGrid[n_inst] | per group: start[n_cta + 1], jobs | (host
// and device copies are the same bytes).  Grids are in the table's order.
struct Group {
  int first, count;           // grids
  long long o_start, o_jobs;  // byte offsets
  long long mail_words, sample_bytes;
  long long max_cells;        // largest monitor
  double steps;               // of the longest list
};
constexpr int MAX_GROUPS = 256;
struct Head {
  int n_inst, n_cta, R, adjoint, n_groups, dtype;
  int curls, pad;  // curls: every grid has a curl record
  long long inst_offset, o_grids, bytes, ws_bytes;
  Group group[MAX_GROUPS];
};

struct Plan {
  Head h{};
  std::vector<ListGrid> grids;
  std::vector<std::vector<int>> start;
  std::vector<std::vector<ListJob>> jobs;
};

inline long long up16(long long x) { return (x + 15) / 16 * 16; }

// us per step of bands with R = 1, 2, 4 rows per warp (B200, FP32, 16 warps; FP64 goes
// by the same, unmeasured): run, recorded run, reverse sweep
constexpr double STEP_US[3][3] = {{0.82, 1.06, 1.66}, {1.0, 1.5, 4.0}, {1.4, 2.6, 0.0}};

// The CTAs by the steps they have been given, fewest first.
struct Loads {
  std::vector<std::pair<double, int>> v;
  explicit Loads(int n_cta) : v(n_cta) {
    for (int c = 0; c < n_cta; ++c) v[c] = {0.0, c};
  }
  // the next grid: its bands go to the CTAs that are free first, all of which are
  // then busy until it ends; give(band, cta)
  template <typename F>
  void add(int bands, int steps, const F& give) {
    const double end = v[bands - 1].first + steps;
    for (int b = 0; b < bands; ++b) {
      give(b, v[b].second);
      v[b].first = end;
    }
    const auto rest = v.begin() + bands;
    std::rotate(v.begin(), rest,
                std::upper_bound(rest, v.end(), std::pair<double, int>(end, INT_MAX)));
  }
};

// false: some grid does not fit, or the batch is not a TM one
bool make_plan(const dn_batch2d* cfg, const dn_batch2d_inst* insts, bool adjoint, Plan* P,
               int nsm = sm_count()) {
  const long long off = batch2d_inst_offset(cfg, insts);
  if (off < 0 || cfg->pol != DN_TM || nsm < 1) return false;
  const int n = cfg->n_inst, elem = cfg->dtype == DN_F32 ? 4 : 8, cols = 32 * 16 / elem;
  std::vector<int> order(n);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(),
                   [&](int a, int b) { return insts[a].n_steps > insts[b].n_steps; });
  auto grid_of = [&](const dn_batch2d_inst& I, int R) {
    ListGrid G{};
    G.strips = (I.W + cols - 1) / cols;
    G.groups = G.strips > MAX_WARPS
                   ? 0 : std::min(MAX_WARPS / G.strips, std::max(1, (I.H + R - 1) / R));
    G.bands = G.groups ? (I.H + G.groups * R - 1) / (G.groups * R) : 0;
    return G;
  };
  // The rows per warp with which the last CTA is done first: more rows are fewer and
  // slower turns (96 x 256^2, 2000 steps: 40 / 23 / 20 ms with R = 1 / 2 / 4; 12
  // recorded grids of 100^2 to 512^2: 3.9 / 3.2 / 3.9 ms, of 100^2 to 200^2 0.84 / 1.24 /
  // 3.3; their sweeps 5.5 / 5.3 and 1.3 / 2.2)
  bool record = false, curls = true;
  for (int b = 0; b < n; ++b) {
    record = record || insts[b].curl != nullptr;
    curls = curls && insts[b].curl != nullptr;
  }
  int R = 0;
  double best = 0.0;
  for (int r = 1; r <= (adjoint ? 2 : 4); r *= 2) {
    Loads loads(nsm);
    bool fits = true;
    for (int k = 0; k < n && fits; ++k) {
      const ListGrid G = grid_of(insts[order[k]], r);
      fits = G.groups > 0 && G.bands <= nsm;
      if (fits) loads.add(G.bands, insts[order[k]].n_steps, [](int, int) {});
    }
    if (!fits) continue;
    const double t = loads.v.back().first * STEP_US[adjoint ? 2 : record ? 1 : 0][r / 2];
    if (R == 0 || t < best) {
      best = t;
      R = r;
    }
  }
  if (R == 0) return false;
  Head& h = P->h;
  h.n_inst = n;
  h.n_cta = nsm;
  h.R = R;
  h.adjoint = adjoint;
  h.curls = curls;
  h.dtype = cfg->dtype;
  h.inst_offset = off;
  long long ws = 0;
  for (int k = 0; k < n;) {
    if (h.n_groups == MAX_GROUPS) return false;
    Group g{};
    g.first = k;
    long long mail = 0, sample = 0;
    Loads loads(nsm);
    std::vector<std::vector<ListJob>> lists(nsm);
    for (; k < n; ++k) {
      const dn_batch2d_inst& I = insts[order[k]];
      ListGrid G = grid_of(I, R);
      long long cells = 0, bytes = 0;
      if (I.mon_comp != DN_NONE) {
        cells = (long long)(I.mon_box.hi[1] - I.mon_box.lo[1]) *
                (I.mon_box.hi[2] - I.mon_box.lo[2]);
        G.stride = up16(cells * elem) / elem;
        bytes = G.stride * elem * I.n_steps;
      }
      if (bytes > GROUP_SAMPLE_BYTES) return false;
      if (k > g.first && (sample + bytes > GROUP_SAMPLE_BYTES || k - g.first == GROUP_GRIDS))
        break;
      G.mail = mail;
      G.sample = sample;
      mail += (long long)G.bands * 4 * G.strips * ROW_WORDS;
      sample += bytes;
      g.max_cells = std::max(g.max_cells, cells);
      P->grids.push_back(G);
      loads.add(G.bands, I.n_steps, [&](int b, int cta) { lists[cta].push_back({k, b}); });
    }
    g.count = k - g.first;
    g.mail_words = mail;
    g.sample_bytes = sample;
    g.steps = loads.v.back().first;
    ws = std::max(ws, mail * 8 + sample);
    std::vector<int> start(nsm + 1, 0);
    std::vector<ListJob> jobs;
    for (int c = 0; c < nsm; ++c) {
      jobs.insert(jobs.end(), lists[c].begin(), lists[c].end());
      start[c + 1] = (int)jobs.size();
    }
    P->start.push_back(start);
    P->jobs.push_back(jobs);
    h.group[h.n_groups++] = g;
  }
  long long at = up16(sizeof(Head));
  h.o_grids = at;
  at += up16((long long)n * sizeof(ListGrid));
  for (int g = 0; g < h.n_groups; ++g) {
    h.group[g].o_start = at;
    at += up16((nsm + 1) * sizeof(int));
    h.group[g].o_jobs = at;
    at += up16((long long)P->jobs[g].size() * sizeof(ListJob));
  }
  h.bytes = at;
  h.ws_bytes = ws;
  return true;
}

// f(), or `otherwise` where the host has no memory for a plan (no exception leaves a C
// entry)
template <typename R, typename F>
R with_memory(R otherwise, const F& f) {
  try {
    return f();
  } catch (const std::bad_alloc&) {
    return otherwise;
  }
}

// a batch as make_plan takes it; for a reverse sweep with all that the sweep reads and
// writes
bool valid(const dn_batch2d* cfg, const dn_batch2d_inst* insts, bool adjoint) {
  if (!cfg || !insts || batch2d_inst_offset(cfg, insts) < 0) return false;
  for (int b = 0; adjoint && b < cfg->n_inst; ++b) {
    const dn_batch2d_inst& I = insts[b];
    if (!I.curl || !I.grad) return false;
    for (int c = 0; c < 3; ++c)
      if (!I.lam[0][c] || !I.lam[1][c]) return false;
  }
  return true;
}

// running DFTs of a group's monitors, one grid per blockIdx.y
template <typename T>
__global__ void __launch_bounds__(DFT_WARPS * 32)
    k_list_dft(const dn_batch2d_inst* insts, const ListGrid* grids, unsigned char* samples,
               int first, const int* status) {
  if (status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0) return;
  const dn_batch2d_inst& I = insts[first + blockIdx.y];
  const ListGrid& G = grids[first + blockIdx.y];
  if (I.mon_comp == DN_NONE) return;
  const long long ncell = (long long)(I.mon_box.hi[1] - I.mon_box.lo[1]) *
                          (I.mon_box.hi[2] - I.mon_box.lo[2]);
  if (blockIdx.x * 32LL >= ncell) return;
  sample_dft<T>(reinterpret_cast<const T*>(samples + G.sample), G.stride, I.n_steps, ncell, I.phase,
                I.n_freq, I.acc);
}

// what a group's monitors add in the reverse sweep: before the first step straight
// into lambda, for the later ones a table; one grid per blockIdx.y
template <typename T>
__global__ void __launch_bounds__(256)
    k_list_adds(const dn_batch2d_inst* insts, const ListGrid* grids, unsigned char* samples,
                int first) {
  const dn_batch2d_inst& I = insts[first + blockIdx.y];
  const ListGrid& G = grids[first + blockIdx.y];
  if (I.mon_comp == DN_NONE || I.gmon == nullptr) return;
  const int bw = I.mon_box.hi[2] - I.mon_box.lo[2];
  const long long ncell = (long long)(I.mon_box.hi[1] - I.mon_box.lo[1]) * bw;
  T* table = reinterpret_cast<T*>(samples + G.sample);
  T* lam = static_cast<T*>(I.lam[I.n_steps & 1][0]);
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < ncell * I.n_steps;
       e += gridDim.x * 256LL) {
    const long long n = e / ncell, cell = e - n * ncell;
    const T v = add_of<T>(cell, ncell, I.n_steps - 1 - n, I.phase, I.n_freq, I.gmon);
    if (n == 0)
      lam[(I.mon_box.lo[1] + cell / bw) * I.pitch + I.mon_box.lo[2] + cell % bw] += v;
    else
      table[(n - 1) * G.stride + cell] = v;
  }
}

template <typename T>
int run_groups(const Head& h, bool record, unsigned char* table, unsigned char* blob,
               unsigned char* ws, int* status, cudaStream_t s) {
  const dn_batch2d_inst* insts = reinterpret_cast<const dn_batch2d_inst*>(table + h.inst_offset);
  const ListGrid* grids = reinterpret_cast<const ListGrid*>(blob + h.o_grids);
  for (int q = 0; q < h.n_groups; ++q) {
    const Group& g = h.group[q];
    List L{insts,
           grids,
           reinterpret_cast<const ListJob*>(blob + g.o_jobs),
           reinterpret_cast<const int*>(blob + g.o_start),
           reinterpret_cast<uint64_t*>(ws),
           ws + g.mail_words * 8,
           polls_of(g.steps)};
    DN_CUDA_CHECK(cudaMemsetAsync(ws, 0, (size_t)g.mail_words * 8, s));
    const unsigned cells = (unsigned)((g.max_cells + 31) / 32);
    if (h.adjoint && cells) {
      k_list_adds<T><<<dim3(64, g.count), 256, 0, s>>>(insts, grids, L.samples, g.first);
      DN_CUDA_CHECK(cudaGetLastError());
    }
    const int rc = run_resident_list<T>(L, h.adjoint, record, h.R, h.n_cta, status, s);
    if (rc != DN_OK) return rc;
    if (!h.adjoint && cells) {
      k_list_dft<T><<<dim3(cells, g.count), DFT_WARPS * 32, 0, s>>>(insts, grids, L.samples,
                                                                    g.first, status);
      DN_CUDA_CHECK(cudaGetLastError());
    }
  }
  return DN_OK;
}

}  // namespace
}  // namespace res
}  // namespace dn

extern "C" int64_t dn_batch2d_resident_bytes(const dn_batch2d* cfg, const dn_batch2d_inst* insts,
                                             int32_t adjoint) {
  if (!dn::res::valid(cfg, insts, adjoint != 0)) return -1;
  return dn::res::with_memory<int64_t>(0, [&]() -> int64_t {
    dn::res::Plan P;
    return dn::res::make_plan(cfg, insts, adjoint != 0, &P) ? P.h.bytes : 0;
  });
}

extern "C" int32_t dn_batch2d_resident_plan(const dn_batch2d* cfg, const dn_batch2d_inst* insts,
                                            int32_t adjoint, int32_t n_sm, dn_batch2d_plan* out) {
  if (!cfg || !insts || !out || n_sm < 0 || dn::batch2d_inst_offset(cfg, insts) < 0)
    return DN_EINVAL;
  *out = dn_batch2d_plan{};
  return dn::res::with_memory<int32_t>(DN_ENOMEM, [&]() -> int32_t {
    dn::res::Plan P;
    if (!dn::res::make_plan(cfg, insts, adjoint != 0, &P, n_sm > 0 ? n_sm : dn::sm_count()))
      return DN_OK;
    out->rows = P.h.R;
    out->launches = P.h.n_groups;
    for (int g = 0; g < P.h.n_groups; ++g) {
      const dn::res::Group& G = P.h.group[g];
      out->most_grids = std::max(out->most_grids, G.count);
      out->wait_polls = std::max<int64_t>(out->wait_polls, dn::res::polls_of(G.steps));
    }
    return DN_OK;
  });
}

extern "C" int32_t dn_batch2d_resident_pack(const dn_batch2d* cfg, const dn_batch2d_inst* insts,
                                            int32_t adjoint, void* host_plan, int64_t bytes,
                                            int64_t* ws_bytes) {
  if (!dn::res::valid(cfg, insts, adjoint != 0) || !host_plan || !ws_bytes) return DN_EINVAL;
  return dn::res::with_memory<int32_t>(DN_ENOMEM, [&]() -> int32_t {
    dn::res::Plan P;
    if (!dn::res::make_plan(cfg, insts, adjoint != 0, &P)) return DN_EUNSUPPORTED;
    if (bytes < P.h.bytes) return DN_EINVAL;
    unsigned char* b = static_cast<unsigned char*>(host_plan);
    std::memset(b, 0, (size_t)P.h.bytes);
    std::memcpy(b, &P.h, sizeof(P.h));
    std::memcpy(b + P.h.o_grids, P.grids.data(), P.grids.size() * sizeof(dn::res::ListGrid));
    for (int g = 0; g < P.h.n_groups; ++g) {
      std::memcpy(b + P.h.group[g].o_start, P.start[g].data(), P.start[g].size() * sizeof(int));
      std::memcpy(b + P.h.group[g].o_jobs, P.jobs[g].data(),
                  P.jobs[g].size() * sizeof(dn::res::ListJob));
    }
    *ws_bytes = P.h.ws_bytes;
    return DN_OK;
  });
}

extern "C" int32_t dn_batch2d_run_resident(const dn_batch2d* cfg, void* dev_table,
                                           const void* host_plan, void* dev_plan, void* ws,
                                           int64_t ws_bytes, int32_t record, int32_t* status,
                                           void* stream) {
  if (!cfg || !dev_table || !host_plan || !dev_plan ||
      ((reinterpret_cast<uintptr_t>(dev_table) | reinterpret_cast<uintptr_t>(dev_plan) |
        reinterpret_cast<uintptr_t>(ws)) & 15))
    return DN_EINVAL;
  const dn::res::Head& h = *static_cast<const dn::res::Head*>(host_plan);
  if (cfg->n_inst != h.n_inst || cfg->pol != DN_TM || cfg->dtype != h.dtype ||
      ws_bytes < h.ws_bytes || (h.ws_bytes && !ws) || (record && !h.adjoint && !h.curls))
    return DN_EINVAL;
  unsigned char *t = static_cast<unsigned char*>(dev_table),
                *b = static_cast<unsigned char*>(dev_plan), *w = static_cast<unsigned char*>(ws);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cfg->dtype == DN_F32)
    return dn::res::run_groups<float>(h, record != 0, t, b, w, status, s);
  if (cfg->dtype == DN_F64)
    return dn::res::run_groups<double>(h, record != 0, t, b, w, status, s);
  return DN_EINVAL;
}
