// The resident reverse sweep of a TM run (dn_resident2d.cuh): the transpose of
// the forward step (dn_adjoint2d.cu has it term by term), a block of rows and
// columns per warp as in the forward run.  What neighbours need of each other is
// u = dt/eps lambda_Ez of one row above and below and one column left and right;
// lambda_Hy of the row above and lambda_Hx of the column to the left are copies
// that the warp updates itself.  The FP64 gradient of the block's cells stays in
// registers for the whole sweep (it was a read and a write of 8 bytes per cell and
// step), its sum is taken while the rows are on their way, and what the monitors add
// to lambda_Ez before a step comes as a table, computed for all steps at once.
//
// Bound by the same chain as the forward run (row received, block updated, row
// sent).  Measured on B200, 300 x 413 FP32, one monitor row at three wavelengths:
// 1.5 us per reverse step (1.2 without a monitor); before, two launches per step
// (injection 2.2 us and reverse step 5.2 us, and the gaps between them).
#pragma once

#include "dn_resident2d_dev.cuh"

namespace dn {
namespace res {

template <typename T, int R, int MAIL, bool LISTED>
__device__ __forceinline__ void sweep_band(const AdjJob<T>& J, const Split& S, int band,
                                           unsigned char* smem, uint64_t* mail, unsigned polls,
                                           int* status, const Samples<T>* adds, int n_add) {
  using B = Block<T, R, MAIL, LISTED>;
  using L = typename B::L;
  constexpr int VEC = B::VEC;
  constexpr int COLS = B::COLS;
  constexpr int CARR = MAX_WARPS * 512;  // bytes between the column arrays
  using V = Pack<T>;
  using C = typename V::S;
  const int H = J.H, W = J.W;
  const long long py = J.py;
  const B K(H, W, S, band, smem, mail, polls, status);
  const int lane = K.lane, ia = K.ia, j0 = K.j0, jv = K.jv;
  const bool live = K.live, any = K.any, full = K.full;
  const bool first_row = K.first_row, first_col = K.first_col, last_col = K.last_col;
  const bool corner = lane == 0 && first_col;  // the lane that holds column 0
  K.coefficients(J, S);

  // lambda_Ez, lambda_Hx, lambda_Hy, u = dt/eps lambda_Ez, gradient, this step's curl
  constexpr bool CES = R >= 3;  // dt/eps in shared memory
  V e[R], a[R], b[R], u[R], c[R], ce[CES ? 1 : R];
  double g[R][VEC];
  unsigned char* const ces = smem + L::CES + K.w * R * 512 + lane * 16;
  const long long o0 = (long long)ia * py + jv;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool ok = ia + r < H;
    const long long o = o0 + r * py;
    e[r] = K.load(J.in[0], o, ok, W);
    a[r] = K.load(J.in[1], o, ok, W);
    b[r] = K.load(J.in[2], o, ok, W);
    c[r] = K.load(J.curl, o, ok, W);
    const V x = K.load(J.ce, o, ok, W);
    u[r] = mulv<T>(x, e[r]);
    if (CES)
      st16<T>(ces + r * 512, x);
    else
      ce[r < (CES ? 1 : R) ? r : 0] = x;
    const Vec<double, VEC> gr =
        ldv<double, VEC, LD_PLAIN>(J.grad, o, ok && live && any, full, jv, W);
#pragma unroll
    for (int q = 0; q < VEC; ++q) g[r][q] = gr[q];
  }
  // u of the rows above and below (0 where the forward difference had no such
  // neighbour, or no weight on it), copies of the second fields
  V u_up = mulv<T>(K.load(J.ce, o0 - py, ia > 1, W), K.load(J.in[0], o0 - py, ia > 1, W));
  V u_dn = mulv<T>(K.load(J.ce, o0 + R * py, !K.last_row, W),
                   K.load(J.in[0], o0 + R * py, !K.last_row, W));
  V hb = K.load(J.in[2], o0 - py, !first_row, W);
  T ha[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    ha[r] = ld<T>(J.in[1], (long long)(ia + r) * py + j0 - 1, live && ia + r < H && !first_col);

  unsigned add_mask = 0;
  for (int m = 0; m < n_add; ++m)
    if (live && adds[m].lo[0] < ia + R && adds[m].hi[0] > ia && adds[m].lo[1] < j0 + COLS &&
        adds[m].hi[1] > j0)
      add_mask |= 1u << m;

  // The block's first monitor, when it adds to one row of the block in 16-byte pieces,
  // is read a step ahead into registers (read when it is added, it cost every step of
  // the grid 0.4 us).
  V pre{};
  int pre_m = -1;  // its index
  auto pre_row = [&](const Samples<T>& M) { return M.lo[0] > ia ? M.lo[0] - ia : 0; };
  auto fetch_add = [&](int n) {
    const Samples<T>& M = adds[pre_m];
    const long long row = (ia + pre_row(M) - M.lo[0]) * (long long)(M.hi[1] - M.lo[1]);
    ld16_where<T>(M.buf + n * M.step_stride + row + (jv - M.lo[1]),
                  n + 1 < J.nsteps && jv >= M.lo[1] && jv < M.hi[1], pre);
  };
  if (add_mask) {
    const Samples<T>& M = adds[__ffs(add_mask) - 1];
    const int hi = M.hi[0] < ia + R ? M.hi[0] - ia : R;
    // rows of the table on 16-byte boundaries (a step's are a multiple long)
    if (hi - pre_row(M) == 1 && M.lo[1] % VEC == 0 &&
        (M.hi[0] - M.lo[0] == 1 || (M.hi[1] - M.lo[1]) % VEC == 0)) {
      pre_m = __ffs(add_mask) - 1;
      add_mask &= add_mask - 1;
      fetch_add(0);
    }
  }

  auto coef_e = [&](int r) -> V { return CES ? ld16<T>(ces + r * 512) : ce[CES ? 0 : r]; };
  // Curl rows come from memory into L2 two steps before they are loaded, and into
  // registers one step before they are used (300 x 413, us per step: 1.67 when the
  // load was waited for on the spot, 1.31 without, 1.22 with the rows in L2 too).
  constexpr int CURL_AHEAD = 2;
  auto fetch_curl = [&](int n) {
    if (n >= J.nsteps || !live || !any) return;
    const T* const from = J.curl - (long long)n * J.curl_stride + o0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (ia + r < H) asm volatile("prefetch.global.L2 [%0];" ::"l"(from + r * py));
  };
  // the gradient's share of step n, and the curl of the step after it
  auto gradient = [&](int n) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int q = 0; q < VEC; ++q)
        g[r][q] = fma(static_cast<double>(e[r].get(q)), static_cast<double>(c[r].get(q)), g[r][q]);
    }
    if (n + 1 < J.nsteps) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        ld16_where<T>(J.curl - (long long)(n + 1) * J.curl_stride + o0 + r * py,
                      live && any && ia + r < H, c[r]);
    }
    fetch_curl(n + 1 + CURL_AHEAD);
  };
  auto step = [&](int par) {
    const T* const fl = K.l_edge + par * B::EDGE_P;
    const T* const fr = K.r_edge + par * B::EDGE_P;
    const V bx = ld16<T>(K.cc), hk = ld16<T>(K.cc + CARR);
    const V gk = ld16<T>(K.cc + 2 * CARR);
    // lambda_Hy' of row ia-1 and its vy
    V vy_up;
    {
      const V hp = fmav<T>(gk, subv<T>(u_up, u[0]), hb);
      vy_up = mulv<T>(hk, hp);
      hb = mulv<T>(bx, hp);
#pragma unroll
      for (int h = 0; h < 2; ++h) vy_up.p[h] = first_row ? C(0) : vy_up.p[h];
    }
    const V cm = ld16<T>(K.cc + 3 * CARR);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const V rc = ld16<T>(K.cf + 32 * r), rd = ld16<T>(K.cf + 32 * r + 16);
      const C by = rc.p[0], nck = rc.p[1], nyk = rd.p[0], last = rd.p[1];
      T right = __shfl_down_sync(ALL, u[r].get(0), 1);
      right = lane == 31 ? (last_col ? T(0) : fr[r]) : right;
      // u (0 in column 0) minus u of the next column
      V d = minus_next<T>(u[r], right);
      d.set(0, corner ? -u[r].get(1) : d.get(0));
      const V ap = fmav<T>(nyk, d, a[r]);
      const T hp = fma1(low(nyk), fl[r] - u[r].get(0), ha[r]);
      ha[r] = mul1(low(by), hp);
      const V vx = mulv<T>(mulv<T>(ap, nck), cm);  // minus vx
      T left = __shfl_up_sync(ALL, vx.get(VEC - 1), 1);
      left = lane == 0 ? (first_col ? T(0) : mul1(low(nck), hp)) : left;
      a[r] = mulv<T>(ap, by);
      // u (0 in row 0) minus u of the next row
      V own = u[r];
      if (r == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) own.p[h] = first_row ? C(0) : own.p[h];
      }
      const V bp = fmav<T>(gk, subv<T>(own, r + 1 < R ? u[r + 1 < R ? r + 1 : r] : u_dn), b[r]);
      b[r] = mulv<T>(bx, bp);
      const V vy = mulv<T>(mulv<T>(hk, bp), last);
      e[r] = subv<T>(subv<T>(mulv<T>(mulv<T>(bx, by), e[r]), bwd_cols<T>(vx, left)),
                     subv<T>(vy, vy_up));
      vy_up = vy;
    }
  };

  for (int n = 1; n <= CURL_AHEAD; ++n) fetch_curl(n);
  gradient(0);
  K.publish(0, u);
  __syncthreads();  // also: the coefficients are in place

  auto advance = [&](auto par_c, int n) -> bool {
    constexpr int PAR = decltype(par_c)::value;
    constexpr int NXT = PAR ^ 1;
    if (K.active) step(PAR);
    if (n + 1 == J.nsteps) return false;
    if (pre_m >= 0) {
      const Samples<T>& M = adds[pre_m];
      const int pr = pre_row(M), left = jv >= M.lo[1] ? M.hi[1] - jv : 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r != pr) continue;
        if (left >= VEC) {
          e[r] = addv<T>(e[r], pre);
        } else {
#pragma unroll
          for (int q = 0; q < VEC; ++q)
            if (q < left) e[r].set(q, e[r].get(q) + pre.get(q));
        }
      }
    }
    if (add_mask) {
#pragma unroll 1
      for (int m = 0; m < n_add; ++m) {
        if (!((add_mask >> m) & 1u)) continue;
        const Samples<T>& M = adds[m];
        const int bw = M.hi[1] - M.lo[1], k = jv - M.lo[1];
        const T* const from = M.buf + (long long)n * M.step_stride + k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int i = ia + r - M.lo[0];
          if (i < 0 || ia + r >= M.hi[0]) continue;
          if (M.vec) {
            if (k >= 0 && k < bw)
              e[r] = addv<T>(e[r], ld16<T>(reinterpret_cast<const unsigned char*>(from + i * bw)));
          } else {
#pragma unroll
            for (int q = 0; q < VEC; ++q)
              if (k + q >= 0 && k + q < bw) e[r].set(q, e[r].get(q) + from[i * bw + q]);
          }
        }
      }
    }
    if (K.active) {
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = mulv<T>(coef_e(r), e[r]);
      K.post(NXT, n, u);
      K.publish(NXT, u);
    }
    __syncthreads();
    if (K.active) gradient(n + 1);  // while the rows are on their way
    if (pre_m >= 0) fetch_add(n + 1);
    const bool go = K.gather(NXT, n, u_up, u_dn);
    if (ia <= 1) {  // row ia-1 = 0 has no weight on its own u; row -1 does not exist
#pragma unroll
      for (int h = 0; h < 2; ++h) u_up.p[h] = C(0);
    }
    if (K.last_row) {
#pragma unroll
      for (int h = 0; h < 2; ++h) u_dn.p[h] = C(0);
    }
    return go;
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
      const long long o = o0 + r * py;
      stv(J.out[0], o, vec_of<T>(e[r]), full, jv, W);
      stv(J.out[1], o, vec_of<T>(a[r]), full, jv, W);
      stv(J.out[2], o, vec_of<T>(b[r]), full, jv, W);
      Vec<double, VEC> gr;
#pragma unroll
      for (int q = 0; q < VEC; ++q) gr[q] = g[r][q];
      stv(J.grad, o, gr, full, jv, W);
    }
  }
}

template <typename T, int R, int MAIL>
__global__ void __launch_bounds__(MAX_WARPS * 32, 1)
    k_resident2d_adj(const __grid_constant__ AdjJob<T> J, const __grid_constant__ SampleSet<T> adds,
                     const Split S, uint64_t* mail, int* status) {
  using L = Smem<T, R, MAIL == MAIL_CLUSTER>;
  extern __shared__ __align__(16) unsigned char r_smem[];
  if constexpr (MAIL == MAIL_CLUSTER) arm_mailboxes<L>(r_smem);
  const bool skip = status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
  if (!skip && (int)blockIdx.x < S.bands)
    sweep_band<T, R, MAIL, false>(J, S, blockIdx.x, r_smem, mail, 0, status, adds.s, adds.n);
  if constexpr (MAIL == MAIL_CLUSTER) cg::this_cluster().sync();  // no row still under way
}

template <typename T>
int run_resident_adjoint(const AdjJob<T>& J, const SampleSet<T>& adds, const Split& S,
                         uint64_t* mail, int* status, cudaStream_t s) {
  auto go = [&](auto r_c, auto m_c) {
    constexpr int R = decltype(r_c)::value, MAIL = decltype(m_c)::value;
    return launch_bands(k_resident2d_adj<T, R, MAIL>, S, Smem<T, R, MAIL == MAIL_CLUSTER>::BYTES, s,
                        J, adds, S, mail, status);
  };
  using std::integral_constant;
  constexpr integral_constant<int, MAIL_CLUSTER> cl{};
  constexpr integral_constant<int, MAIL_GLOBAL> gl{};
  constexpr integral_constant<int, 1> r1{};
  constexpr integral_constant<int, 2> r2{};
  constexpr integral_constant<int, 3> r3{};
  if (S.cluster) return S.R == 1 ? go(r1, cl) : S.R == 2 ? go(r2, cl) : DN_EINVAL;
  return S.R == 1 ? go(r1, gl) : S.R == 2 ? go(r2, gl) : S.R == 3 ? go(r3, gl) : DN_EINVAL;
}

}  // namespace res
}  // namespace dn
