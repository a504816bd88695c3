// Resident 2-D runs (dn_resident2d.cuh): the choice of the work split, the
// workspace and the entry points.
#include <algorithm>

#include "dn_adjoint.cuh"
#include "dn_resident2d.cuh"
#include "dn_sample_dft.cuh"
#include "dn_strip.cuh"

namespace dn {
namespace res {
namespace {

// The work split of a grid, or none (R = 0) when it does not fit on the chip.
//
// A step costs what the busiest warp's block costs (rows per warp) plus the
// trip of a row to the next band.  Measured on B200, FP32 TM, us per step: one
// cluster (at most 16 bands) 0.41 (R = 1, 8 warps), 0.55 (R = 1, 16 warps),
// 0.45 / 0.48 / 0.76 (R = 2; 4 / 8 / 16 warps); bands over the whole chip 0.7 -
// 0.95 (R = 1), 1.0 - 1.2 (R = 2), 1.6 - 2.0 (R = 3), 1.9 - 2.2 (R = 4), where
// one launch per step takes 6.2 (256 x 256) to 8.3 (1024 x 1024).  So: a cluster
// where 16 bands hold the grid, else the fewest rows per warp for which one
// band per SM does.  (At 16 warps of two rows, about 192^2 to 256^2 in FP32, the
// cluster's 0.76 and the whole chip's 0.7 - 0.95 have not been compared on one grid;
// FP64 goes by the FP32 figures.)  The reverse sweep holds the FP64 gradient too: at most
// R = 3 (909 k cells in FP32).
constexpr int R_MAX = 4, R_MAX_ADJ = 3;
Split choose_split(int H, int W, int elem, int nsm, int r_max) {
  Split S{};
  const int cols = 32 * 16 / elem;
  const int strips = (W + cols - 1) / cols;
  auto fits = [&](int R, int bands) {
    const int groups = std::max(1, (H + bands * R - 1) / (bands * R));
    if (strips * groups > MAX_WARPS) return false;
    S = Split{R, strips, groups, (H + groups * R - 1) / (groups * R), 0};
    return true;
  };
  if (fits(1, 16) && S.strips * S.groups <= 8) return S.cluster = 1, S;
  if (fits(2, 16)) return S.cluster = 1, S;
  for (int R = 1; R <= r_max; ++R)
    if (fits(R, nsm)) return S;
  return Split{};
}

constexpr long long SAMPLE_BYTES = 64LL << 20;  // most workspace for samples
constexpr int MIN_STEPS = 8;  // shorter runs go launch by launch
constexpr int MIN_PIECE = 4 * MIN_STEPS;  // so do runs whose samples allow fewer steps per launch

// everything a run needs, or ok = false for the launch-by-launch path
struct Plan2d {
  bool ok;
  Split S;
  long long mail_bytes;    // the two mailboxes of every band
  long long sample_bytes;  // one step's samples of all monitors
  int piece;               // most steps per launch (whole run, or what the samples allow)
};

Plan2d make_plan2d(const dn_grid* g, const dn_source* src, const dn_monitor* mons, int n_mon,
                   int nsteps, bool adjoint, int nsm = sm_count()) {
  Plan2d P{};
  if (nsm < 1) return P;
  const int elem = g->dtype == DN_F32 ? 4 : 8;
  const int first = g->pol == DN_TM ? DN_EZ : DN_HZ;
  if (nsteps < MIN_STEPS || (g->pitch_y * elem) % 16 != 0) return P;
  if (src && src->component != DN_NONE && src->component != first) return P;
  // the TE update of these equations grows without bound (FP32 overflows within
  // ~130 steps): FP32 TE has no resident form (FDTDSolver2D takes dn_batch2d.cu's
  // cluster kernel for it where that is faster than a launch per step)
  if (g->pol == DN_TE && (adjoint || g->dtype == DN_F32)) return P;
  // what a monitor adds in the reverse sweep goes to lambda_Ez alone
  for (int m = 0; adjoint && m < n_mon; ++m)
    if (mons[m].component != first) return P;
  P.S = choose_split(g->H, g->W, elem, nsm, adjoint ? R_MAX_ADJ : R_MAX);
  if (P.S.R == 0) return P;
  P.mail_bytes = P.S.cluster ? 0 : (long long)P.S.bands * 4 * P.S.strips * ROW_WORDS * 8;
  P.piece = nsteps;
  for (int m = 0; m < n_mon; ++m)
    P.sample_bytes += (to_dev(mons[m].box).cells() * elem + 15) / 16 * 16;
  if (P.sample_bytes * nsteps > SAMPLE_BYTES) {
    P.piece = (int)(SAMPLE_BYTES / P.sample_bytes);
    if (P.piece < MIN_PIECE) return P;
  }
  P.ok = true;
  return P;
}

long long workspace_of(const Plan2d& P) {
  return P.ok ? P.mail_bytes + P.sample_bytes * P.piece : 0;
}

template <typename T>
int run2d_resident(const dn_grid* g, void* const fa[6], void* const fb[6], const void* ce,
                   const dn_cpml* cpml, const StepParams<T>& p, const dn_probe* probe,
                   const dn_curl_record* crec, int t0, int nsteps, int* status, cudaStream_t s,
                   const Plan2d& P, unsigned char* ws) {
  const bool tm = g->pol == DN_TM;
  const int comp[3] = {tm ? DN_EZ : DN_HZ, tm ? DN_HX : DN_EX, tm ? DN_HY : DN_EY};
  Job<T> J{};
  J.H = g->H;
  J.W = g->W;
  J.py = g->pitch_y;
  J.ce = static_cast<const T*>(ce);
  for (int a = 0; a < 2; ++a) {
    J.b[a] = cpml->b[1 + a];
    J.c[a] = cpml->c[1 + a];
    J.src_lo[a] = p.src.box.lo[1 + a];
    J.src_hi[a] = p.src.box.hi[1 + a];
  }
  J.dt = g->dt;
  J.dl = g->dl;
  J.src = p.src.comp >= 0;
  J.wave = p.src.wave;
  constexpr int VEC = 16 / (int)sizeof(T);
  const Pieces cut(nsteps, P.piece);
  for (int piece = 0; piece < cut.count; ++piece) {
    const int n = cut.begin(piece), k = cut.begin(piece + 1) - n;
    J.t0 = t0 + n;
    J.nsteps = k;
    for (int c = 0; c < 3; ++c) {
      void* const to = nsteps % 2 ? fb[comp[c]] : fa[comp[c]];
      J.in[c] = static_cast<const T*>(n == 0 ? fa[comp[c]] : to);
      J.out[c] = static_cast<T*>(to);
    }
    if (crec) {
      J.curl_stride = crec->step_stride;
      for (int c = 0; c < (tm ? 1 : 2); ++c)
        J.curl[c] = static_cast<T*>(crec->curl[tm ? 2 : c]) +
                    (long long)(t0 + n - crec->t0) * crec->step_stride;
    }
    SampleSet<T> set{};
    unsigned char* at = ws + P.mail_bytes;
    auto add = [&](int c, const BoxDev& b, T* buf, long long stride) {
      Samples<T>& q = set.s[set.n++];
      for (int a = 0; a < 2; ++a) {
        q.lo[a] = b.lo[1 + a];
        q.hi[a] = b.hi[1 + a];
      }
      q.comp = c == comp[0] ? 0 : c == comp[1] ? 1 : 2;
      q.vec = q.lo[1] % VEC == 0 && (q.hi[1] - q.lo[1]) % VEC == 0;
      q.buf = buf;
      q.step_stride = stride;
    };
    for (int m = 0; m < p.n_mon; ++m) {
      const long long stride = (p.mon[m].ncell * (long long)sizeof(T) + 15) / 16 * 16 / sizeof(T);
      add(p.mon[m].comp, p.mon[m].box, reinterpret_cast<T*>(at), stride);
      at += stride * sizeof(T) * k;
    }
    if (p.probe.comp >= 0) {
      BoxDev b{};
      for (int a = 0; a < 3; ++a) b.lo[a] = p.probe.pos[a], b.hi[a] = p.probe.pos[a] + 1;
      add(p.probe.comp, b, p.probe.out + t0 + n, 1);
      set.s[set.n - 1].vec = 0;
    }
    if (P.mail_bytes) DN_CUDA_CHECK(cudaMemsetAsync(ws, 0, P.mail_bytes, s));
    uint64_t* const mail = reinterpret_cast<uint64_t*>(ws);
    int rc = DN_EINVAL;
    if (tm)
      rc = run_resident<T, DN_TM>(J, set, P.S, mail, status, s);
    else if constexpr (sizeof(T) == 8)
      rc = run_resident<T, DN_TE>(J, set, P.S, mail, status, s);
    if (rc != DN_OK) return rc;
    for (int m = 0; m < p.n_mon; ++m) {
      const MonDev& M = p.mon[m];
      k_sample_dft<T><<<(unsigned)((M.ncell + 31) / 32), DFT_WARPS * 32, 0, s>>>(
          set.s[m].buf, set.s[m].step_stride, k, M.ncell,
          M.phase + (long long)(t0 + n) * M.nf * 2, M.nf, M.acc, status);
    }
    DN_CUDA_CHECK(cudaGetLastError());
  }
  return DN_OK;
}

// 16-byte rows: every array the polarisation uses, and the curl slots
template <typename T>
bool rows_ok(const dn_grid* g, void* const fa[6], void* const fb[6], const void* ce,
             const dn_curl_record* rec) {
  const int comps[2][3] = {{DN_EZ, DN_HX, DN_HY}, {DN_HZ, DN_EX, DN_EY}};
  const int tm = g->pol == DN_TM;
  if (!aligned16(ce)) return false;
  for (int c : comps[tm ? 0 : 1])
    if (!aligned16(fa[c]) || !aligned16(fb[c])) return false;
  if (rec) {
    if ((rec->step_stride * (long long)sizeof(T)) % 16 != 0) return false;
    if (tm ? !aligned16(rec->curl[2]) : !aligned16(rec->curl[0]) || !aligned16(rec->curl[1]))
      return false;
  }
  return true;
}

template <typename T>
int run_ws(const dn_grid* g, void* const fa[6], void* const fb[6], const void* ce,
           const dn_cpml* cpml, const dn_source* src, const dn_monitor* mons, int32_t n_mon,
           const dn_probe* probe, const dn_curl_record* rec, int32_t t0, int32_t nsteps,
           int32_t* status, cudaStream_t s, int32_t* final_in_b, void* ws, int64_t ws_bytes,
           bool* done) {
  *done = false;
  StepParams<T> p;
  const int rc = build_params<T>(false, g, fa, fb, ce, cpml, src, mons, n_mon, probe, status, &p);
  if (rc != DN_OK) return rc;
  if (t0 < 0 || !final_in_b || !steps_ok(src, mons, n_mon, probe, t0, (int64_t)t0 + nsteps))
    return DN_EINVAL;
  if (rec) {
    const bool tm = g->pol == DN_TM;
    if ((tm && !rec->curl[2]) || (!tm && (!rec->curl[0] || !rec->curl[1]))) return DN_EINVAL;
    if (rec->step_stride < (int64_t)g->H * g->pitch_y || rec->t0 < 0 || t0 < rec->t0 ||
        t0 + nsteps > rec->t0 + rec->nslots)
      return DN_EINVAL;
  }
  const Plan2d P = make_plan2d(g, src, mons, n_mon, nsteps, false);
  if (!P.ok || workspace_of(P) > ws_bytes || !aligned16(ws) || !rows_ok<T>(g, fa, fb, ce, rec))
    return DN_OK;
  *done = true;
  const int r2 = run2d_resident<T>(g, fa, fb, ce, cpml, p, probe, rec, t0, nsteps, status, s, P,
                                   static_cast<unsigned char*>(ws));
  if (r2 == DN_OK) *final_in_b = nsteps % 2;
  return r2;
}

// what the monitors add to lambda before reverse steps t, t-1, ..: out[n][cell] =
// sum_f g[f][cell] . phase[t - n][f]
template <typename T>
__global__ void __launch_bounds__(256)
    k_add_table(T* __restrict__ out, long long stride, int nsteps, int t, long long ncell,
                const double* __restrict__ phase, int nf, const double* __restrict__ g) {
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < ncell * nsteps;
       e += gridDim.x * 256LL) {
    const long long n = e / ncell, cell = e - n * ncell;
    out[n * stride + cell] = add_of<T>(cell, ncell, t - n, phase, nf, g);
  }
}

template <typename T>
int adjoint_ws(const dn_grid* g, void* const la[6], void* const lb[6], const void* ce,
               const dn_cpml* cpml, const dn_curl_record* curl, double* grad,
               const dn_monitor* mons, int32_t n_mon, int32_t t_end, int32_t nsteps,
               int32_t* status, cudaStream_t s, int32_t* final_in_b, unsigned char* ws,
               int64_t ws_bytes, bool* done) {
  *done = false;
  AdjParams<T> p;
  int rc = build_adj_params<T>(false, g, la, lb, ce, cpml, curl, grad, t_end, nsteps, status, &p);
  if (rc != DN_OK) return rc;
  if (!final_in_b || n_mon < 0 || n_mon > DN_MAX_MONITORS || (n_mon > 0 && !mons))
    return DN_EINVAL;
  if (!mons_steps_ok(mons, n_mon, (int64_t)t_end - nsteps, t_end)) return DN_EINVAL;
  for (int m = 0; m < n_mon; ++m)
    if (!box_ok(mons[m].box, 1, g->H, g->W) || mons[m].n_freq < 1 ||
        mons[m].n_freq > DN_MAX_FREQS || !mons[m].phase || !mons[m].acc)
      return DN_EINVAL;
  const Plan2d P = make_plan2d(g, nullptr, mons, n_mon, nsteps, true);
  const int comp[3] = {DN_EZ, DN_HX, DN_HY};
  if (!P.ok || workspace_of(P) > ws_bytes || !aligned16(ws) || !aligned16(ce) ||
      !aligned16(grad) || !aligned16(curl->curl[2]) ||
      (curl->step_stride * (long long)sizeof(T)) % 16 != 0)
    return DN_OK;
  for (int c : comp)
    if (!aligned16(la[c]) || !aligned16(lb[c])) return DN_OK;
  *done = true;
  AdjJob<T> J{};
  J.H = g->H;
  J.W = g->W;
  J.py = g->pitch_y;
  J.ce = static_cast<const T*>(ce);
  for (int a = 0; a < 2; ++a) {
    J.b[a] = cpml->b[1 + a];
    J.c[a] = cpml->c[1 + a];
  }
  J.dt = g->dt;
  J.dl = g->dl;
  J.grad = grad;
  J.curl_stride = curl->step_stride;
  constexpr int VEC = 16 / (int)sizeof(T);
  const Pieces cut(nsteps, P.piece);
  for (int piece = 0; piece < cut.count; ++piece) {
    const int n = cut.begin(piece), k = cut.begin(piece + 1) - n;
    const int t = t_end - 1 - n;  // the piece's first reverse step
    J.nsteps = k;
    J.curl = static_cast<const T*>(curl->curl[2]) + (long long)(t - curl->t0) * J.curl_stride;
    for (int c = 0; c < 3; ++c) {
      void* const to = nsteps % 2 ? lb[comp[c]] : la[comp[c]];
      p.in[comp[c]] = static_cast<const T*>(n == 0 ? la[comp[c]] : to);
      J.in[c] = p.in[comp[c]];
      J.out[c] = static_cast<T*>(to);
    }
    // the first step's share straight into lambda, the later ones as tables
    p.t = t;
    if ((rc = inject_monitors<T>(p, mons, n_mon, false, g->pol, s)) != DN_OK) return rc;
    SampleSet<T> set{};
    unsigned char* at = ws + P.mail_bytes;
    for (int m = 0; m < n_mon && k > 1; ++m) {
      const BoxDev b = to_dev(mons[m].box);
      const long long ncell = b.cells();
      Samples<T>& q = set.s[set.n++];
      for (int a = 0; a < 2; ++a) {
        q.lo[a] = b.lo[1 + a];
        q.hi[a] = b.hi[1 + a];
      }
      q.vec = q.lo[1] % VEC == 0 && (q.hi[1] - q.lo[1]) % VEC == 0;
      q.buf = reinterpret_cast<T*>(at);
      q.step_stride = (ncell * (long long)sizeof(T) + 15) / 16 * 16 / sizeof(T);
      at += q.step_stride * sizeof(T) * k;
      const long long blocks = (ncell * (k - 1) + 255) / 256;
      k_add_table<T><<<(unsigned)std::min(blocks, 148LL * 16), 256, 0, s>>>(
          q.buf, q.step_stride, k - 1, t - 1, ncell, mons[m].phase, mons[m].n_freq, mons[m].acc);
    }
    if (P.mail_bytes) DN_CUDA_CHECK(cudaMemsetAsync(ws, 0, P.mail_bytes, s));
    rc = run_resident_adjoint<T>(J, set, P.S, reinterpret_cast<uint64_t*>(ws), status, s);
    if (rc != DN_OK) return rc;
    DN_CUDA_CHECK(cudaGetLastError());
  }
  *final_in_b = nsteps % 2;
  return DN_OK;
}

}  // namespace
}  // namespace res
}  // namespace dn

extern "C" int32_t dn_fdtd2d_adjoint_ws(const dn_grid* g, void* const la[6], void* const lb[6],
                                        const void* ce, const dn_cpml* cpml,
                                        const dn_curl_record* curl, double* grad_ce,
                                        const dn_monitor* mons, int32_t n_mon, int32_t t_end,
                                        int32_t nsteps, int32_t* status, void* stream,
                                        int32_t* final_in_b, void* ws, int64_t ws_bytes) {
  if (!g) return DN_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned char* const w = static_cast<unsigned char*>(ws);
  if (nsteps >= dn::res::MIN_STEPS && (ws || ws_bytes == 0)) {
    bool done = false;
    int rc = DN_OK;
    if (g->dtype == DN_F32)
      rc = dn::res::adjoint_ws<float>(g, la, lb, ce, cpml, curl, grad_ce, mons, n_mon, t_end,
                                      nsteps, status, s, final_in_b, w, ws_bytes, &done);
    else if (g->dtype == DN_F64)
      rc = dn::res::adjoint_ws<double>(g, la, lb, ce, cpml, curl, grad_ce, mons, n_mon, t_end,
                                       nsteps, status, s, final_in_b, w, ws_bytes, &done);
    if (rc != DN_OK || done) return rc;
  }
  return dn_fdtd2d_adjoint(g, la, lb, ce, cpml, curl, grad_ce, mons, n_mon, t_end, nsteps, status,
                           stream, final_in_b);
}

extern "C" int64_t dn_fdtd2d_workspace_bytes(const dn_grid* g, const dn_source* src,
                                             const dn_monitor* mons, int32_t n_mon,
                                             int32_t nsteps) {
  if (!g || g->H < 1 || g->W < 1 || g->D != 1 || (g->dtype != DN_F32 && g->dtype != DN_F64) ||
      (g->pol != DN_TM && g->pol != DN_TE) || n_mon < 0 || n_mon > DN_MAX_MONITORS ||
      (n_mon > 0 && !mons))
    return -1;
  for (int m = 0; m < n_mon; ++m)
    if (!dn::box_ok(mons[m].box, 1, g->H, g->W)) return -1;
  return std::max(
      dn::res::workspace_of(dn::res::make_plan2d(g, src, mons, n_mon, nsteps, false)),
      dn::res::workspace_of(dn::res::make_plan2d(g, nullptr, mons, n_mon, nsteps, true)));
}

extern "C" int32_t dn_fdtd2d_resident_plan(const dn_grid* g, const dn_source* src,
                                           const dn_monitor* mons, int32_t n_mon, int32_t nsteps,
                                           int32_t adjoint, int32_t n_sm, dn_resident_plan* out) {
  if (!out || n_sm < 0 || nsteps < 0 ||
      dn_fdtd2d_workspace_bytes(g, src, mons, n_mon, nsteps) < 0)
    return DN_EINVAL;
  *out = dn_resident_plan{};
  const dn::res::Plan2d P =
      dn::res::make_plan2d(g, adjoint ? nullptr : src, mons, n_mon, nsteps, adjoint != 0,
                           n_sm > 0 ? n_sm : dn::sm_count());
  if (!P.ok) return DN_OK;
  out->rows = P.S.R;
  out->bands = P.S.bands;
  out->cluster = P.S.cluster;
  return dn::describe_pieces(nsteps, P.piece, out);
}

extern "C" int32_t dn_fdtd2d_run_ws(const dn_grid* g, void* const fa[6], void* const fb[6],
                                    const void* ce, const dn_cpml* cpml, const dn_source* src,
                                    const dn_monitor* mons, int32_t n_mon, const dn_probe* probe,
                                    const dn_curl_record* rec, int32_t t0, int32_t nsteps,
                                    int32_t* status, void* stream, int32_t* final_in_b, void* ws,
                                    int64_t ws_bytes) {
  if (!g) return DN_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (nsteps >= dn::res::MIN_STEPS && (ws || ws_bytes == 0)) {
    bool done = false;
    int rc = DN_OK;
    if (g->dtype == DN_F32)
      rc = dn::res::run_ws<float>(g, fa, fb, ce, cpml, src, mons, n_mon, probe, rec, t0, nsteps,
                                  status, s, final_in_b, ws, ws_bytes, &done);
    else if (g->dtype == DN_F64)
      rc = dn::res::run_ws<double>(g, fa, fb, ce, cpml, src, mons, n_mon, probe, rec, t0, nsteps,
                                   status, s, final_in_b, ws, ws_bytes, &done);
    if (rc != DN_OK || done) return rc;
  }
  return dn_fdtd2d_run(g, fa, fb, ce, cpml, src, mons, n_mon, probe, rec, t0, nsteps, status,
                       stream, final_in_b);
}
