// Device code and launchers of the resident forward run (dn_resident2d.cuh);
// included by one source file per element type and polarisation.
#pragma once

#include <type_traits>

#include <cooperative_groups.h>

#include "dn_resident2d.cuh"

namespace dn {
namespace res {

namespace cg = cooperative_groups;

constexpr unsigned ALL = STRIP_FULL_MASK;
constexpr unsigned SPIN_LIMIT = 1u << 22;   // polls of one wait on a global mailbox
constexpr unsigned PROBE_LIMIT = 1u << 16;  // probes of one wait on an mbarrier ...
constexpr uint32_t PROBE_NS = 20000;        // ... each suspended for at most this long

// ---- a lane's 16 bytes ----------------------------------------------------------
// FP32: four columns in two register pairs, updated with the packed f32x2
// instructions (one issue slot for two columns, each half rounded as the scalar
// instruction rounds it); FP64: two columns, scalar instructions.
template <typename T>
struct Pack;
template <>
struct Pack<float> {
  using S = uint64_t;  // a scalar in both halves
  uint64_t p[2];
  __device__ __forceinline__ float get(int q) const {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p[q >> 1]));
    return (q & 1) ? hi : lo;
  }
  __device__ __forceinline__ void set(int q, float x) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p[q >> 1]));
    (q & 1) ? hi = x : lo = x;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p[q >> 1]) : "f"(lo), "f"(hi));
  }
};
template <>
struct Pack<double> {
  using S = double;
  double p[2];
  __device__ __forceinline__ double get(int q) const { return p[q]; }
  __device__ __forceinline__ void set(int q, double x) { p[q] = x; }
};
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t both(float x) { return pair(x, x); }
__device__ __forceinline__ double both(double x) { return x; }
__device__ __forceinline__ float low(uint64_t s) { return __uint_as_float((uint32_t)s); }
__device__ __forceinline__ double low(double s) { return s; }

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {  // a - b, rounded once
  return fma2(b, 0xbf800000bf800000ull, a);
}
__device__ __forceinline__ double mul2(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fma2(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double sub2(double a, double b) { return __dsub_rn(a, b); }

template <typename T>
__device__ __forceinline__ Pack<T> mulv(const Pack<T>& a, typename Pack<T>::S s) {
  return {{mul2(a.p[0], s), mul2(a.p[1], s)}};
}
template <typename T>
__device__ __forceinline__ Pack<T> mulv(const Pack<T>& a, const Pack<T>& b) {
  return {{mul2(a.p[0], b.p[0]), mul2(a.p[1], b.p[1])}};
}
template <typename T>
__device__ __forceinline__ Pack<T> subv(const Pack<T>& a, const Pack<T>& b) {
  return {{sub2(a.p[0], b.p[0]), sub2(a.p[1], b.p[1])}};
}
template <typename T>
__device__ __forceinline__ Pack<T> fmav(const Pack<T>& a, const Pack<T>& b, const Pack<T>& c) {
  return {{fma2(a.p[0], b.p[0], c.p[0]), fma2(a.p[1], b.p[1], c.p[1])}};
}
template <typename T>
__device__ __forceinline__ Pack<T> fmav(typename Pack<T>::S s, const Pack<T>& b,
                                        const Pack<T>& c) {
  return {{fma2(s, b.p[0], c.p[0]), fma2(s, b.p[1], c.p[1])}};
}
__device__ __forceinline__ float mul1(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul1(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma1(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma1(double a, double b, double c) { return __fma_rn(a, b, c); }

// differences of neighbouring columns: forward (x of the next column minus own;
// `next` = the column after the lane's last) and backward
template <typename T>
__device__ __forceinline__ Pack<T> fwd_cols(const Pack<T>& v, T next) {
  constexpr int VEC = 16 / (int)sizeof(T);
  T d[VEC];
#pragma unroll
  for (int q = 0; q < VEC; ++q) d[q] = (q + 1 < VEC ? v.get(q + 1 < VEC ? q + 1 : q) : next) - v.get(q);
  Pack<T> r;
  if constexpr (sizeof(T) == 4)
    r.p[0] = pair(d[0], d[1]), r.p[1] = pair(d[2], d[3]);
  else
    r.p[0] = d[0], r.p[1] = d[1];
  return r;
}
template <typename T>
__device__ __forceinline__ Pack<T> bwd_cols(const Pack<T>& v, T prev) {
  constexpr int VEC = 16 / (int)sizeof(T);
  T d[VEC];
#pragma unroll
  for (int q = 0; q < VEC; ++q) d[q] = v.get(q) - (q > 0 ? v.get(q > 0 ? q - 1 : 0) : prev);
  Pack<T> r;
  if constexpr (sizeof(T) == 4)
    r.p[0] = pair(d[0], d[1]), r.p[1] = pair(d[2], d[3]);
  else
    r.p[0] = d[0], r.p[1] = d[1];
  return r;
}

template <typename T>
__device__ __forceinline__ Pack<T> pack_of(const Vec<T, 16 / (int)sizeof(T)>& v) {
  Pack<T> r;
  if constexpr (sizeof(T) == 4)
    r.p[0] = pair(v[0], v[1]), r.p[1] = pair(v[2], v[3]);
  else
    r.p[0] = v[0], r.p[1] = v[1];
  return r;
}
template <typename T>
__device__ __forceinline__ Vec<T, 16 / (int)sizeof(T)> vec_of(const Pack<T>& p) {
  constexpr int VEC = 16 / (int)sizeof(T);
  Vec<T, VEC> v;
#pragma unroll
  for (int q = 0; q < VEC; ++q) v[q] = p.get(q);
  return v;
}
__device__ __forceinline__ uint64_t bits(uint64_t x) { return x; }
__device__ __forceinline__ uint64_t bits(double x) { return (uint64_t)__double_as_longlong(x); }
__device__ __forceinline__ void from_bits(uint64_t u, uint64_t& x) { x = u; }
__device__ __forceinline__ void from_bits(uint64_t u, double& x) {
  x = __longlong_as_double((long long)u);
}

// ---- rows between CTAs ---------------------------------------------------------
// global mailbox: 64-bit words (step tag | value), one row = 4 words per lane
template <typename T>
__device__ __forceinline__ void post_words(uint64_t* box, uint32_t tag, const Pack<T>& v) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint64_t u = bits(v.p[q >> 1]);
    const uint32_t w = (q & 1) ? (uint32_t)(u >> 32) : (uint32_t)u;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(box + q * 32),
                 "l"(((uint64_t)tag << 32) | w)
                 : "memory");
  }
}
// bounded wait for a row, or for two at once (TWO: both boxes are read in one
// round trip); false when it gave up or another CTA recorded an error
template <typename T, bool TWO>
__device__ __forceinline__ bool take_words(const uint64_t* a, const uint64_t* b, uint32_t tag,
                                           Pack<T>& va, Pack<T>& vb, const int* status) {
  constexpr int N = TWO ? 8 : 4;
  for (unsigned n = 0; n < SPIN_LIMIT; ++n) {
    uint64_t u[N];
    bool ok = true;
#pragma unroll
    for (int q = 0; q < N; ++q)
      asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
                   : "=l"(u[q])
                   : "l"((q < 4 ? a : b) + (q & 3) * 32)
                   : "memory");
#pragma unroll
    for (int q = 0; q < N; ++q) ok = ok && (uint32_t)(u[q] >> 32) == tag;
    if (__all_sync(ALL, ok)) {
      from_bits((u[1] << 32) | (uint32_t)u[0], va.p[0]);
      from_bits((u[3] << 32) | (uint32_t)u[2], va.p[1]);
      if (TWO) {
        from_bits((u[N - 3] << 32) | (uint32_t)u[N - 4], vb.p[0]);
        from_bits((u[N - 1] << 32) | (uint32_t)u[N - 2], vb.p[1]);
      }
      return true;
    }
    if ((n & 4095u) == 4095u && status && *reinterpret_cast<const volatile int*>(status) != 0)
      return false;
  }
  return false;
}

// shared-memory mailbox of a cluster neighbour: the lane's 16 bytes and their
// count on the receiving warp's mbarrier in one instruction
template <typename T>
__device__ __forceinline__ void post_async(uint32_t slot, uint32_t bar, const Pack<T>& v) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(
          slot),
      "l"(bits(v.p[0])), "l"(bits(v.p[1])), "r"(bar)
      : "memory");
}
__device__ __forceinline__ uint32_t map_cta(uint32_t addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// ---- shared memory of one CTA --------------------------------------------------
// row[parity][top/bottom][warp][COLS]      published rows
// inrow[up/down][parity][strip][COLS]      rows from the neighbour bands (cluster)
// colc[b_x, dt (1+c_x)/dl, (1+c_x)/dl][strip][COLS]
// coef[row] = (b_y, -dt (1+c_y)/dl, -(1+c_y)/dl), 8 bytes each (FP32: the value
//   in both halves), 32 bytes per row, row = 0 .. 16 R
// edge[parity][left/right][warp][R]        published edge columns
// bar[up/down][parity][strip]              mbarriers of inrow
// flag[2]                a wait ran out, by step parity
// ces[warp][R][COLS]  dt/eps, R >= 4
template <typename T, int R, bool CLUSTER>
struct Smem {
  static constexpr int VEC = 16 / (int)sizeof(T);
  static constexpr int COLS = 32 * VEC;
  static constexpr int ROW_BYTES = 512;  // COLS values
  static constexpr int ROWS = 0;
  static constexpr int INROW = ROWS + 4 * MAX_WARPS * ROW_BYTES;
  static constexpr int COLC = INROW + (CLUSTER ? 4 * MAX_WARPS * ROW_BYTES : 0);
  static constexpr int COEF = COLC + 3 * MAX_WARPS * ROW_BYTES;
  static constexpr int EDGE = COEF + (MAX_WARPS * R + 1) * 32;
  static constexpr int EDGE_PAR = 2 * MAX_WARPS * R * (int)sizeof(T);
  static constexpr int BAR = (EDGE + 2 * EDGE_PAR + 7) / 8 * 8;
  static constexpr int FLAG = (BAR + (CLUSTER ? 4 * MAX_WARPS * 8 : 0) + 15) / 16 * 16;
  static constexpr int CES = FLAG + 16;
  static constexpr int BYTES = CES + (R >= 4 ? MAX_WARPS * R * ROW_BYTES : 0);

  __host__ __device__ static constexpr int row(int par, int bottom, int w) {
    return ROWS + ((par * 2 + bottom) * MAX_WARPS + w) * ROW_BYTES;
  }
  __host__ __device__ static constexpr int inrow(int down, int par, int strip) {
    return INROW + ((down * 2 + par) * MAX_WARPS + strip) * ROW_BYTES;
  }
  __host__ __device__ static constexpr int edge(int par, int right, int w) {
    return EDGE + par * EDGE_PAR + (right * MAX_WARPS + w) * R * (int)sizeof(T);
  }
  __host__ __device__ static constexpr int bar(int down, int par, int strip) {
    return BAR + ((down * 2 + par) * MAX_WARPS + strip) * 8;
  }
};

template <typename T>
__device__ __forceinline__ Pack<T> ld16(const unsigned char* a) {
  const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(a);
  Pack<T> v;
  from_bits(x.x, v.p[0]);
  from_bits(x.y, v.p[1]);
  return v;
}
template <typename T>
__device__ __forceinline__ void st16(unsigned char* a, const Pack<T>& v) {
  *reinterpret_cast<ulonglong2*>(a) = make_ulonglong2(bits(v.p[0]), bits(v.p[1]));
}

// bounded wait for a phase of an mbarrier
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity) {
  for (unsigned n = 0; n < PROBE_LIMIT; ++n)
    if (mbar_try_wait_sleep(bar, parity, PROBE_NS)) return true;
  return false;
}

// ---------------------------------------------------------------------------
// the run of one band
// ---------------------------------------------------------------------------
template <typename T, int POL, int R, int MAIL, bool REC, bool SMP>
__device__ __forceinline__ void run_band(const Job<T>& J, const Split& S, int band, int nbands,
                                         unsigned char* smem, uint64_t* mail, int* status,
                                         const Samples<T>* smps, int n_smp) {
  constexpr bool CLUSTER = MAIL == MAIL_CLUSTER;
  using L = Smem<T, R, CLUSTER>;
  constexpr int VEC = L::VEC;
  constexpr int COLS = L::COLS;
  using V = Pack<T>;
  using C = typename V::S;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int strip = w % S.strips, group = w / S.strips;
  const int H = J.H, W = J.W;
  const long long py = J.py;
  const int ia0 = band * S.groups * R;
  const int ia = ia0 + group * R;
  const int j0 = strip * COLS, jv = j0 + lane * VEC;
  const bool live = ia < H;
  const bool any = jv < W, full = jv + VEC <= W;
  const double idl = 1.0 / J.dl;
  const bool first_row = ia == 0, last_row = ia + R >= H;
  const bool first_col = strip == 0, last_col = strip + 1 == S.strips;
  // rows from or to another CTA
  const bool band_up = live && !first_row && group == 0;
  const bool band_dn = live && !last_row && group + 1 == S.groups;
  const bool tail = any && jv + VEC >= W;  // the lane that holds column W-1
  // cells just outside the grid that a warp holds (the row below H-1, the
  // column right of W-1) carry a copy of their neighbour's injected field, so
  // that the difference across the edge is 0
  const int ghost_row = live && last_row && ia + R > H ? H - ia : R;
  const int ghost_col = tail && jv + VEC > W ? W - jv : VEC;

  // coefficients: row profiles of the band, column profiles of the strips
  C* coef = reinterpret_cast<C*>(smem + L::COEF);
  for (int e = threadIdx.x; e < S.groups * R + 1; e += blockDim.x) {
    const int i = ia0 + e;
    const double g = i < H ? 1.0 + J.c[0][i] : 1.0;
    coef[4 * e] = both(i < H ? static_cast<T>(J.b[0][i]) : T(1));
    coef[4 * e + 1] = both(static_cast<T>(-(J.dt * g * idl)));
    coef[4 * e + 2] = both(static_cast<T>(-(g * idl)));
  }
  T* colc = reinterpret_cast<T*>(smem + L::COLC);
  for (int j = threadIdx.x; j < S.strips * COLS; j += blockDim.x) {
    const double g = j < W ? 1.0 + J.c[1][j] : 1.0;
    colc[j] = j < W ? static_cast<T>(J.b[1][j]) : T(1);
    colc[MAX_WARPS * COLS + j] = static_cast<T>(J.dt * g * idl);
    colc[2 * MAX_WARPS * COLS + j] = static_cast<T>(g * idl);
  }

  // dt/eps in registers, or in shared memory where R rows of it would not fit
  constexpr bool CES = R >= 4;
  V f[R], a[R], b[R], ce[CES ? 1 : R];
  unsigned char* const ces = smem + L::CES + w * R * 512 + lane * 16;
  const long long o0 = (long long)ia * py + jv;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool ok = live && any && ia + r < H;
    f[r] = pack_of<T>(ldv<T, VEC>(J.in[0], o0 + r * py, ok, full, jv, W));
    a[r] = pack_of<T>(ldv<T, VEC>(J.in[1], o0 + r * py, ok, full, jv, W));
    b[r] = pack_of<T>(ldv<T, VEC>(J.in[2], o0 + r * py, ok, full, jv, W));
    const V c = pack_of<T>(ldv<T, VEC>(J.ce, o0 + r * py, ok, full, jv, W));
    if (CES)
      st16<T>(ces + r * 512, c);
    else
      ce[r < (CES ? 1 : R) ? r : 0] = c;
  }
  // the injected field of the rows above and below before the first step, and
  // this warp's copies of its neighbours' second fields
  // (a block at the grid's edge reads its own row there: no difference)
  V f_up = first_row ? f[0] : pack_of<T>(ldv<T, VEC>(J.in[0], o0 - py, live && any, full, jv, W));
  V f_dn = last_row ? f[R - 1]
                    : pack_of<T>(ldv<T, VEC>(J.in[0], o0 + R * py, any, full, jv, W));
  V hb, hce;      // TM: Hy of row ia-1; TE: Ey of row ia+R and its dt/eps
  T ha[R], hca[R];  // TM: Hx of column j0-1; TE: Ex of column j0+COLS and its dt/eps
  const bool hb_ok = live && any && (POL == DN_TM ? !first_row : !last_row);
  const long long hb_o = POL == DN_TM ? o0 - py : o0 + R * py;
  hb = pack_of<T>(ldv<T, VEC>(J.in[2], hb_o, hb_ok, full, jv, W));
  if (POL == DN_TE) hce = pack_of<T>(ldv<T, VEC>(J.ce, hb_o, hb_ok, full, jv, W));
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

  // shared-memory addresses of this warp and of the rows and columns it reads
  unsigned char* const my_row = smem + L::row(0, 0, w) + lane * 16;
  constexpr int ROW_PAR = L::row(1, 0, 0) - L::row(0, 0, 0);
  constexpr int ROW_BOT = L::row(0, 1, 0) - L::row(0, 0, 0);
  constexpr int EDGE_R = L::edge(0, 1, 0) - L::edge(0, 0, 0);
  const unsigned char* const up_row =
      smem + (CLUSTER && band_up ? L::inrow(0, 0, strip)
              : first_row        ? L::row(0, 0, w)
                                 : L::row(0, 1, group > 0 ? w - S.strips : w)) + lane * 16;
  const unsigned char* const dn_row =
      smem + (CLUSTER && band_dn ? L::inrow(1, 0, strip)
              : last_row         ? L::row(0, 1, w)
                                 : L::row(0, 0, group + 1 < S.groups ? w + S.strips : w)) +
      lane * 16;
  constexpr int IN_PAR = L::inrow(0, 1, 0) - L::inrow(0, 0, 0);
  const int up_par = CLUSTER && band_up ? IN_PAR : ROW_PAR;
  const int dn_par = CLUSTER && band_dn ? IN_PAR : ROW_PAR;
  // the last lane with a neighbour to the right: lane 31, or the one that holds
  // column W-1, which reads its own column there
  const bool right_lane = last_col ? tail : lane == 31;
  T* const my_left = reinterpret_cast<T*>(smem + L::edge(0, 0, w));
  T* const my_right = reinterpret_cast<T*>(smem + L::edge(0, 1, w));
  const T* const l_edge = reinterpret_cast<const T*>(smem + L::edge(0, 1, first_col ? w : w - 1));
  const T* const r_edge =
      reinterpret_cast<const T*>(smem + (last_col ? L::edge(0, 1, w) : L::edge(0, 0, w + 1)));
  constexpr int EDGE_P = L::EDGE_PAR / (int)sizeof(T);
  const unsigned char* const cc = smem + L::COLC + strip * 512 + lane * 16;
  const unsigned char* const cf = smem + L::COEF + 32 * group * R;
  // mailboxes
  uint64_t *bar_up = nullptr, *bar_dn = nullptr;  // of the rows this warp receives
  uint32_t to_up = 0, to_dn = 0, tob_up = 0, tob_dn = 0;
  const uint64_t *in_up = nullptr, *in_dn = nullptr;
  uint64_t *out_up = nullptr, *out_dn = nullptr;
  const long long slot = (long long)S.strips * ROW_WORDS;
  if constexpr (CLUSTER) {
    bar_up = reinterpret_cast<uint64_t*>(smem + L::bar(0, 0, strip));
    bar_dn = reinterpret_cast<uint64_t*>(smem + L::bar(1, 0, strip));
    const int up = band > 0 ? band - 1 : band, dn_ = band + 1 < nbands ? band + 1 : band;
    to_up = map_cta(smem_u32(smem + L::inrow(1, 0, strip) + lane * 16), up);
    tob_up = map_cta(smem_u32(bar_dn), up);
    to_dn = map_cta(smem_u32(smem + L::inrow(0, 0, strip) + lane * 16), dn_);
    tob_dn = map_cta(smem_u32(bar_up), dn_);
  } else {
    // mail[up/down][band][parity][strip]
    const long long mine = (long long)strip * ROW_WORDS + lane;
    uint64_t* const up_box = mail;
    uint64_t* const dn_box = mail + (long long)nbands * 2 * slot;
    in_up = up_box + (long long)band * 2 * slot + mine;
    in_dn = dn_box + (long long)band * 2 * slot + mine;
    out_up = dn_box + (long long)(band - 1) * 2 * slot + mine;
    out_dn = up_box + (long long)(band + 1) * 2 * slot + mine;
  }
  constexpr int BAR_PAR = MAX_WARPS;  // mbarriers between the two slots

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
  // rows and edge columns of the injected field for the CTA's other warps
  auto publish = [&](int par) {
    st16<T>(my_row + par * ROW_PAR, f[0]);
    st16<T>(my_row + par * ROW_PAR + ROW_BOT, f[R - 1]);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) my_left[par * EDGE_P + r] = f[r].get(0);
    }
    if (right_lane) {
#pragma unroll
      for (int r = 0; r < R; ++r) my_right[par * EDGE_P + r] = f[r].get(VEC - 1);
    }
  };
  // one step of the block's fields (parity of the published edge columns)
  auto coef_e = [&](int r) -> V { return CES ? ld16<T>(ces + r * 512) : ce[CES ? 0 : r]; };
  auto step = [&](int par, int n) {
    const T* const fl = l_edge + par * EDGE_P;
    const T* const fr = r_edge + par * EDGE_P;
    const V bx = ld16<T>(cc), hk = ld16<T>(cc + MAX_WARPS * 512);
    const V gk = ld16<T>(cc + 2 * MAX_WARPS * 512);
    if (POL == DN_TM) {
      hb = fmav<T>(hk, subv<T>(f[0], f_up), mulv<T>(bx, hb));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const V rc = ld16<T>(cf + 32 * r);
        const C by = rc.p[0], nck = rc.p[1];
        T right = __shfl_down_sync(ALL, f[r].get(0), 1);
        right = right_lane ? fr[r] : right;
        ha[r] = fma1(low(nck), f[r].get(0) - fl[r], mul1(low(by), ha[r]));
        a[r] = fmav<T>(nck, fwd_cols<T>(f[r], right), mulv<T>(a[r], by));
        b[r] = fmav<T>(hk, subv<T>(r + 1 < R ? f[r + 1 < R ? r + 1 : r] : f_dn, f[r]),
                       mulv<T>(bx, b[r]));
      }
      if (first_row) hb = b[0];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const C by = ld16<T>(cf + 32 * r).p[0], nyk = ld16<T>(cf + 32 * r + 16).p[0];
        T left = __shfl_up_sync(ALL, a[r].get(VEC - 1), 1);
        left = lane == 0 ? (first_col ? a[r].get(0) : ha[r]) : left;
        const V cz = fmav<T>(gk, subv<T>(b[r], r > 0 ? b[r > 0 ? r - 1 : 0] : hb),
                             mulv<T>(bwd_cols<T>(a[r], left), nyk));
        f[r] = fmav<T>(coef_e(r), cz, mulv<T>(mulv<T>(bx, by), f[r]));
        if (REC && any && ia + r < H)
          stv(J.curl[0] + (long long)n * J.curl_stride, o0 + r * py, vec_of<T>(cz), full, jv, W);
      }
    } else {
      const C byn = ld16<T>(cf + 32 * R).p[0], nykn = ld16<T>(cf + 32 * R + 16).p[0];
      hb = fmav<T>(hce, mulv<T>(subv<T>(f_dn, f[R - 1]), nykn), mulv<T>(hb, byn));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const C by = ld16<T>(cf + 32 * r).p[0], nyk = ld16<T>(cf + 32 * r + 16).p[0];
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
        const V rc = ld16<T>(cf + 32 * r);
        const C by = rc.p[0], nck = rc.p[1];
        T right = __shfl_down_sync(ALL, a[r].get(0), 1);
        right = right_lane ? (last_col ? a[r].get(VEC - 1) : ha[r]) : right;
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
  publish(0);
  if (threadIdx.x == 0) *reinterpret_cast<int2*>(smem + L::FLAG) = make_int2(0, 0);
  __syncthreads();  // also: coefficients and monitor sums in place

  // step n, reading the buffers of parity PAR and filling the others; false
  // after the last step
  auto advance = [&](auto par_c, int n) -> bool {
    constexpr int PAR = decltype(par_c)::value;
    constexpr int NXT = PAR ^ 1;
    const int t = J.t0 + n;
    step(PAR, n);
    if (src_rows) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((src_rows >> r) & 1u) f[r] = fmav<T>(both(wv), src_cols, f[r]);
      if (n + 1 < J.nsteps) wv = __ldg(J.wave + t + 1);
    }
    const bool more = n + 1 < J.nsteps;
    if (more) {
      if (has_ghosts) ghosts();
      if (CLUSTER) {
        if (band_up) post_async<T>(to_up + NXT * IN_PAR, tob_up + NXT * BAR_PAR * 8, f[0]);
        if (band_dn) post_async<T>(to_dn + NXT * IN_PAR, tob_dn + NXT * BAR_PAR * 8, f[R - 1]);
      } else {
        if (band_up) post_words<T>(out_up + NXT * slot, n + 1, f[0]);
        if (band_dn) post_words<T>(out_dn + NXT * slot, n + 1, f[R - 1]);
      }
      publish(NXT);
    }
    if (SMP && smp_mask) {
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
    __syncthreads();
    const int failed = *reinterpret_cast<volatile int*>(smem + L::FLAG + NXT * 4);
    bool bad = false;
    if constexpr (CLUSTER) {
      if (band_up || band_dn) {
        // slot NXT's (n / 2 + 1)-th use
        const uint32_t ph = (uint32_t)(n >> 1) & 1u;
        if (band_up) {
          bad |= !wait_bar(bar_up + NXT * BAR_PAR, ph);
          if (lane == 0) mbar_arrive_expect_tx(bar_up + NXT * BAR_PAR, 512);
        }
        if (band_dn) {
          bad |= !wait_bar(bar_dn + NXT * BAR_PAR, ph);
          if (lane == 0) mbar_arrive_expect_tx(bar_dn + NXT * BAR_PAR, 512);
        }
        __syncwarp();
      }
      f_up = ld16<T>(up_row + NXT * up_par);
      f_dn = ld16<T>(dn_row + NXT * dn_par);
    } else {
      if (!band_up) f_up = ld16<T>(up_row + NXT * ROW_PAR);
      if (!band_dn) f_dn = ld16<T>(dn_row + NXT * ROW_PAR);
      if (band_up && band_dn) {
        bad = !take_words<T, true>(in_up + NXT * slot, in_dn + NXT * slot, n + 1, f_up, f_dn,
                                   status);
      } else if (band_up || band_dn) {
        V v, unused;
        bad = !take_words<T, false>((band_up ? in_up : in_dn) + NXT * slot, nullptr, n + 1, v,
                                    unused, status);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          f_up.p[h] = band_up ? v.p[h] : f_up.p[h];
          f_dn.p[h] = band_up ? f_dn.p[h] : v.p[h];
        }
      }
    }
    if (bad) {  // seen by every warp behind the next barrier
      report_status(status, DN_ETIMEOUT);
      *reinterpret_cast<volatile int*>(smem + L::FLAG + PAR * 4) = 1;
    }
    return failed == 0;
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
  if constexpr (MAIL == MAIL_CLUSTER) {
    if (threadIdx.x == 0) {
      for (int e = 0; e < 4 * MAX_WARPS; ++e) {
        uint64_t* bar = reinterpret_cast<uint64_t*>(r_smem + L::BAR) + e;
        mbar_init(bar, 1);
        mbar_arrive_expect_tx(bar, 512);
      }
      fence_barrier_init();
    }
    cg::this_cluster().sync();  // every mailbox armed before any row is sent
  }
  // a previous launch that recorded an error turns this one into a no-op
  const bool skip = status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
  if (!skip && (int)blockIdx.x < S.bands)
    run_band<T, POL, R, MAIL, REC, SMP>(J, S, blockIdx.x, S.bands, r_smem, mail, status, smps.s,
                                   smps.n);
  if constexpr (MAIL == MAIL_CLUSTER) cg::this_cluster().sync();  // no row still under way
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <typename T, int POL, int R, int MAIL, bool REC, bool SMP>
int launch(const Job<T>& J, const SampleSet<T>& smps, const Split& S, uint64_t* mail, int* status,
           cudaStream_t s) {
  auto kern = k_resident2d<T, POL, R, MAIL, REC, SMP>;
  constexpr int smem = Smem<T, R, MAIL == MAIL_CLUSTER>::BYTES;
  DN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  if (MAIL == MAIL_CLUSTER)
    DN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[1];
  lc.blockDim = dim3(S.strips * S.groups * 32);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  lc.attrs = at;
  lc.numAttrs = 1;
  if (MAIL == MAIL_CLUSTER) {
    int cl = 1;
    while (cl < S.bands) cl *= 2;
    lc.gridDim = dim3(cl);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cl;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    lc.gridDim = dim3(S.bands);
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  DN_CUDA_CHECK(cudaLaunchKernelEx(&lc, kern, J, smps, S, mail, status));
  return DN_OK;
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

