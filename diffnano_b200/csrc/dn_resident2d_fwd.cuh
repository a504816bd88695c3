// The resident forward run (dn_resident2d.cuh), included by one source file per
// element type and polarisation.
#pragma once

#include "dn_resident2d_dev.cuh"

namespace dn {
namespace res {

// ---------------------------------------------------------------------------
// the run of one band
// ---------------------------------------------------------------------------
template <typename T, int POL, int R, int MAIL, bool REC, bool SMP, bool LISTED>
__device__ __forceinline__ void run_band(const Job<T>& J, const Split& S, int band,
                                         unsigned char* smem, uint64_t* mail, unsigned polls,
                                         int* status, const Samples<T>* smps, int n_smp) {
  using B = Block<T, R, MAIL, LISTED>;
  using L = typename B::L;
  constexpr int VEC = B::VEC;
  constexpr int COLS = B::COLS;
  using V = Pack<T>;
  using C = typename V::S;
  const int H = J.H, W = J.W;
  const long long py = J.py;
  const double idl = 1.0 / J.dl;
  const B K(H, W, S, band, smem, mail, polls, status);
  const int lane = K.lane, ia = K.ia, j0 = K.j0, jv = K.jv;
  const bool live = K.live, any = K.any, full = K.full;
  const bool first_row = K.first_row, last_row = K.last_row;
  const bool first_col = K.first_col, last_col = K.last_col;
  // cells just outside the grid that a warp holds (the row below H-1, the
  // column right of W-1) carry a copy of their neighbour's injected field, so
  // that the difference across the edge is 0
  const int ghost_row = live && last_row && ia + R > H ? H - ia : R;
  const int ghost_col = K.tail && jv + VEC > W ? W - jv : VEC;
  K.coefficients(J, S);

  // dt/eps in registers, or in shared memory where R rows of it would not fit
  constexpr bool CES = R >= 4;
  V f[R], a[R], b[R], ce[CES ? 1 : R];
  unsigned char* const ces = smem + L::CES + K.w * R * 512 + lane * 16;
  const long long o0 = (long long)ia * py + jv;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool ok = ia + r < H;
    f[r] = K.load(J.in[0], o0 + r * py, ok, W);
    a[r] = K.load(J.in[1], o0 + r * py, ok, W);
    b[r] = K.load(J.in[2], o0 + r * py, ok, W);
    const V c = K.load(J.ce, o0 + r * py, ok, W);
    if (CES)
      st16<T>(ces + r * 512, c);
    else
      ce[r < (CES ? 1 : R) ? r : 0] = c;
  }
  // the injected field of the rows above and below before the first step, and
  // this warp's copies of its neighbours' second fields
  // (a block at the grid's edge reads its own row there: no difference)
  V f_up = first_row ? f[0] : K.load(J.in[0], o0 - py, true, W);
  V f_dn = last_row ? f[R - 1] : K.load(J.in[0], o0 + R * py, true, W);
  V hb, hce;      // TM: Hy of row ia-1; TE: Ey of row ia+R and its dt/eps
  T ha[R], hca[R];  // TM: Hx of column j0-1; TE: Ex of column j0+COLS and its dt/eps
  const bool hb_ok = POL == DN_TM ? !first_row : !last_row;
  const long long hb_o = POL == DN_TM ? o0 - py : o0 + R * py;
  hb = K.load(J.in[2], hb_o, hb_ok, W);
  if (POL == DN_TE) hce = K.load(J.ce, hb_o, hb_ok, W);
  const int ha_j = POL == DN_TM ? j0 - 1 : j0 + COLS;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool ok = live && ia + r < H && (POL == DN_TM ? !first_col : !last_col);
    ha[r] = ld<T>(J.in[1], (long long)(ia + r) * py + ha_j, ok);
    if (POL == DN_TE) hca[r] = ld<T>(J.ce, (long long)(ia + r) * py + ha_j, ok);
  }
  const bool te_r = POL == DN_TE && !last_col;
  const T bxr = te_r ? static_cast<T>(J.b[1][j0 + COLS]) : T(1);
  const T gkr = te_r ? static_cast<T>((1.0 + J.c[1][j0 + COLS]) * idl) : T(0);

  unsigned src_rows = 0;
  if (J.src && live && j0 < J.src_hi[1] && j0 + COLS > J.src_lo[1]) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (ia + r >= J.src_lo[0] && ia + r < J.src_hi[0] && ia + r < H) src_rows |= 1u << r;
  }
  V src_cols = {};  // 1 on the source's columns
#pragma unroll
  for (int q = 0; q < VEC; ++q)
    src_cols.set(q, jv + q >= J.src_lo[1] && jv + q < J.src_hi[1] ? T(1) : T(0));
  T wv = src_rows ? __ldg(J.wave + J.t0) : T(0);  // the next step's source value

  // sampled boxes that meet this warp's block
  unsigned smp_mask = 0;
  for (int m = 0; SMP && m < n_smp; ++m)
    if (live && smps[m].lo[0] < ia + R && smps[m].hi[0] > ia && smps[m].lo[1] < j0 + COLS &&
        smps[m].hi[1] > j0)
      smp_mask |= 1u << m;

  const bool has_ghosts = ghost_row < R || (last_col && W % VEC != 0);
  auto ghosts = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int q = 1; q < VEC; ++q)
        f[r].set(q, q == ghost_col ? f[r].get(q - 1) : f[r].get(q));
      if (r > 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          f[r].p[h] = r == ghost_row ? f[r > 0 ? r - 1 : 0].p[h] : f[r].p[h];
      }
    }
  };
  // one step of the block's fields (parity of the published edge columns)
  auto coef_e = [&](int r) -> V { return CES ? ld16<T>(ces + r * 512) : ce[CES ? 0 : r]; };
  auto step = [&](int par, int n) {
    const T* const fl = K.l_edge + par * B::EDGE_P;
    const T* const fr = K.r_edge + par * B::EDGE_P;
    const V bx = ld16<T>(K.cc), hk = ld16<T>(K.cc + MAX_WARPS * 512);
    const V gk = ld16<T>(K.cc + 2 * MAX_WARPS * 512);
    if (POL == DN_TM) {
      hb = fmav<T>(hk, subv<T>(f[0], f_up), mulv<T>(bx, hb));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const V rc = ld16<T>(K.cf + 32 * r);
        const C by = rc.p[0], nck = rc.p[1];
        T right = __shfl_down_sync(ALL, f[r].get(0), 1);
        right = K.right_lane ? fr[r] : right;
        ha[r] = fma1(low(nck), f[r].get(0) - fl[r], mul1(low(by), ha[r]));
        a[r] = fmav<T>(nck, fwd_cols<T>(f[r], right), mulv<T>(a[r], by));
        b[r] = fmav<T>(hk, subv<T>(r + 1 < R ? f[r + 1 < R ? r + 1 : r] : f_dn, f[r]),
                       mulv<T>(bx, b[r]));
      }
      if (first_row) hb = b[0];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const C by = ld16<T>(K.cf + 32 * r).p[0], nyk = ld16<T>(K.cf + 32 * r + 16).p[0];
        T left = __shfl_up_sync(ALL, a[r].get(VEC - 1), 1);
        left = lane == 0 ? (first_col ? a[r].get(0) : ha[r]) : left;
        const V cz = fmav<T>(gk, subv<T>(b[r], r > 0 ? b[r > 0 ? r - 1 : 0] : hb),
                             mulv<T>(bwd_cols<T>(a[r], left), nyk));
        f[r] = fmav<T>(coef_e(r), cz, mulv<T>(mulv<T>(bx, by), f[r]));
        if (REC && any && ia + r < H)
          stv(J.curl[0] + (long long)n * J.curl_stride, o0 + r * py, vec_of<T>(cz), full, jv, W);
      }
    } else {
      const C byn = ld16<T>(K.cf + 32 * R).p[0], nykn = ld16<T>(K.cf + 32 * R + 16).p[0];
      hb = fmav<T>(hce, mulv<T>(subv<T>(f_dn, f[R - 1]), nykn), mulv<T>(hb, byn));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const C by = ld16<T>(K.cf + 32 * r).p[0], nyk = ld16<T>(K.cf + 32 * r + 16).p[0];
        T left = __shfl_up_sync(ALL, f[r].get(VEC - 1), 1);
        left = lane == 0 ? (first_col ? f[r].get(0) : fl[r]) : left;
        ha[r] = fma1(hca[r], mul1(gkr, fr[r] - f[r].get(VEC - 1)), mul1(bxr, ha[r]));
        const V cx = mulv<T>(gk, bwd_cols<T>(f[r], left));
        const V cy = mulv<T>(subv<T>(f[r], r > 0 ? f[r > 0 ? r - 1 : 0] : f_up), nyk);
        const V c = coef_e(r);
        a[r] = fmav<T>(c, cx, mulv<T>(bx, a[r]));
        b[r] = fmav<T>(c, cy, mulv<T>(b[r], by));
        if (REC && any && ia + r < H) {
          stv(J.curl[0] + (long long)n * J.curl_stride, o0 + r * py, vec_of<T>(cx), full, jv, W);
          stv(J.curl[1] + (long long)n * J.curl_stride, o0 + r * py, vec_of<T>(cy), full, jv, W);
        }
      }
      if (last_row) {
        hb = b[R - 1];
        // the row below H-1 inside the block
#pragma unroll
        for (int r = 1; r < R; ++r)
#pragma unroll
          for (int h = 0; h < 2; ++h) b[r].p[h] = r == ghost_row ? b[r - 1].p[h] : b[r].p[h];
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const V rc = ld16<T>(K.cf + 32 * r);
        const C by = rc.p[0], nck = rc.p[1];
        T right = __shfl_down_sync(ALL, a[r].get(0), 1);
        right = K.right_lane ? (last_col ? a[r].get(VEC - 1) : ha[r]) : right;
        V d = fwd_cols<T>(a[r], right);
#pragma unroll
        for (int q = 0; q + 1 < VEC; ++q)  // column W-1 inside the lane
          d.set(q, q + 1 == ghost_col ? T(0) : d.get(q));
        f[r] = fmav<T>(hk, subv<T>(r + 1 < R ? b[r + 1 < R ? r + 1 : r] : hb, b[r]),
                       fmav<T>(nck, d, mulv<T>(mulv<T>(bx, by), f[r])));
      }
    }
  };

  if (has_ghosts) ghosts();
  K.publish(0, f);
  __syncthreads();  // also: the coefficients are in place

  // step n, reading the buffers of parity PAR and filling the others; false
  // after the last step
  auto advance = [&](auto par_c, int n) -> bool {
    constexpr int PAR = decltype(par_c)::value;
    constexpr int NXT = PAR ^ 1;
    const int t = J.t0 + n;
    if (K.active) step(PAR, n);
    if (src_rows) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((src_rows >> r) & 1u) f[r] = fmav<T>(both(wv), src_cols, f[r]);
      if (n + 1 < J.nsteps) wv = __ldg(J.wave + t + 1);
    }
    const bool more = n + 1 < J.nsteps;
    if (more) {
      if (has_ghosts) ghosts();
      K.post(NXT, n, f);
      if (K.active) K.publish(NXT, f);
      __syncthreads();
    }
    if (SMP && smp_mask) {  // (while the rows are on their way)
#pragma unroll 1
      for (int m = 0; m < n_smp; ++m) {
        if (!((smp_mask >> m) & 1u)) continue;
        const Samples<T>& M = smps[m];
        const int bw = M.hi[1] - M.lo[1], k = jv - M.lo[1];
        T* const to = M.buf + (long long)n * M.step_stride + k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = ia + r - M.lo[0];
          if (i < 0 || ia + r >= M.hi[0]) continue;
          V x = f[r];
          if (M.comp != 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) x.p[h] = M.comp == 1 ? a[r].p[h] : b[r].p[h];
          }
          if (M.vec) {
            if (k >= 0 && k < bw) st16<T>(reinterpret_cast<unsigned char*>(to + i * bw), x);
          } else {
#pragma unroll
            for (int q = 0; q < VEC; ++q)
              if (k + q >= 0 && k + q < bw) to[i * bw + q] = x.get(q);
          }
        }
      }
    }
    if (!more) return false;
    return K.gather(NXT, n, f_up, f_dn);
  };
  using P0 = std::integral_constant<int, 0>;
  using P1 = std::integral_constant<int, 1>;
#pragma unroll 1
  for (int n = 0;; n += 2) {
    if (!advance(P0{}, n)) break;
    if (!advance(P1{}, n + 1)) break;
  }

  if (live && any) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (ia + r >= H) break;
      stv(J.out[0], o0 + r * py, vec_of<T>(f[r]), full, jv, W);
      stv(J.out[1], o0 + r * py, vec_of<T>(a[r]), full, jv, W);
      stv(J.out[2], o0 + r * py, vec_of<T>(b[r]), full, jv, W);
    }
  }
}

// ---------------------------------------------------------------------------
// one grid: every CTA of the launch is a band of it
// ---------------------------------------------------------------------------
template <typename T, int POL, int R, int MAIL, bool REC, bool SMP>
__global__ void __launch_bounds__(MAX_WARPS * 32, 1)
    k_resident2d(const __grid_constant__ Job<T> J, const __grid_constant__ SampleSet<T> smps,
                 const Split S, uint64_t* mail, int* status) {
  using L = Smem<T, R, MAIL == MAIL_CLUSTER>;
  extern __shared__ __align__(16) unsigned char r_smem[];
  if constexpr (MAIL == MAIL_CLUSTER) arm_mailboxes<L>(r_smem);
  // a previous launch that recorded an error turns this one into a no-op
  const bool skip = status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
  if (!skip && (int)blockIdx.x < S.bands)
    run_band<T, POL, R, MAIL, REC, SMP, false>(J, S, blockIdx.x, r_smem, mail, 0, status, smps.s,
                                               smps.n);
  if constexpr (MAIL == MAIL_CLUSTER) cg::this_cluster().sync();  // no row still under way
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <typename T, int POL, int R, int MAIL, bool REC, bool SMP>
int launch(const Job<T>& J, const SampleSet<T>& smps, const Split& S, uint64_t* mail, int* status,
           cudaStream_t s) {
  return launch_bands(k_resident2d<T, POL, R, MAIL, REC, SMP>, S,
                      Smem<T, R, MAIL == MAIL_CLUSTER>::BYTES, s, J, smps, S, mail, status);
}

template <typename T, int POL, int R, int MAIL>
int launch_rec(const Job<T>& J, const SampleSet<T>& smps, const Split& S, uint64_t* mail,
               int* status, cudaStream_t s) {
  if (J.curl[0] != nullptr)
    return launch<T, POL, R, MAIL, true, true>(J, smps, S, mail, status, s);
  return smps.n > 0 ? launch<T, POL, R, MAIL, false, true>(J, smps, S, mail, status, s)
                    : launch<T, POL, R, MAIL, false, false>(J, smps, S, mail, status, s);
}

template <typename T, int POL>
int run_resident(const Job<T>& J, const SampleSet<T>& smps, const Split& S, uint64_t* mail,
                 int* status, cudaStream_t s) {
  if (S.cluster)
    return S.R == 1   ? launch_rec<T, POL, 1, MAIL_CLUSTER>(J, smps, S, mail, status, s)
           : S.R == 2 ? launch_rec<T, POL, 2, MAIL_CLUSTER>(J, smps, S, mail, status, s)
                      : DN_EINVAL;
  return S.R == 1   ? launch_rec<T, POL, 1, MAIL_GLOBAL>(J, smps, S, mail, status, s)
         : S.R == 2 ? launch_rec<T, POL, 2, MAIL_GLOBAL>(J, smps, S, mail, status, s)
         : S.R == 3 ? launch_rec<T, POL, 3, MAIL_GLOBAL>(J, smps, S, mail, status, s)
         : S.R == 4 ? launch_rec<T, POL, 4, MAIL_GLOBAL>(J, smps, S, mail, status, s)
                    : DN_EINVAL;
}

}  // namespace res
}  // namespace dn

