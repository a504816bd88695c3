// Device code shared by the resident forward run and its reverse sweep
// (dn_resident2d.cuh): packed values, mailboxes, a CTA's shared memory, and a
// warp's place in the grid with its exchange of rows and columns.
#pragma once

#include <type_traits>

#include <cooperative_groups.h>

#include "dn_resident2d.cuh"

namespace dn {
namespace res {

namespace cg = cooperative_groups;

constexpr unsigned ALL = STRIP_FULL_MASK;
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
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ double add2(double a, double b) { return __dadd_rn(a, b); }
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
__device__ __forceinline__ Pack<T> addv(const Pack<T>& a, const Pack<T>& b) {
  return {{add2(a.p[0], b.p[0]), add2(a.p[1], b.p[1])}};
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
// `next` = the column after the lane's last), own minus next, and backward
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
__device__ __forceinline__ Pack<T> minus_next(const Pack<T>& v, T next) {
  constexpr int VEC = 16 / (int)sizeof(T);
  Pack<T> r = {};
#pragma unroll
  for (int q = 0; q < VEC; ++q) r.set(q, v.get(q) - (q + 1 < VEC ? v.get(q + 1 < VEC ? q + 1 : q) : next));
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
// bounded wait for a row, or for two at once (TWO: both boxes are read in one round
// trip); false when it gave up or another CTA recorded an error.  SPIN_LIMIT polls, in a
// batch (LISTED) about `polls`, looked at now and then (at every poll it cost 96 label
// grids 0.8 %; a lone 1024 x 1024 run is 0.5 % faster with the constant).
template <typename T, bool TWO, bool LISTED>
__device__ __forceinline__ bool take_words(const uint64_t* a, const uint64_t* b, uint32_t tag,
                                           Pack<T>& va, Pack<T>& vb, unsigned polls,
                                           const int* status) {
  constexpr int N = TWO ? 8 : 4;
  for (unsigned n = 0; LISTED || n < SPIN_LIMIT; ++n) {
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
    if ((n & 4095u) == 4095u &&
        ((LISTED && n >= polls) ||
         (status && *reinterpret_cast<const volatile int*>(status) != 0)))
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
// colc[b_x, dt (1+c_x)/dl, (1+c_x)/dl, j < W-1][strip][COLS]
// coef[row] = (b_y, -dt (1+c_y)/dl, -(1+c_y)/dl, i < H-1), 8 bytes each (FP32: the
//   value in both halves), 32 bytes per row, row = 0 .. 16 R
// edge[parity][left/right][warp][R]        published edge columns
// bar[up/down][parity][strip]              mbarriers of inrow
// flag[2]                a wait ran out, by step parity
// ces[warp][R][COLS]     dt/eps where it is not in registers (R >= 3)
template <typename T, int R, bool CLUSTER>
struct Smem {
  static constexpr int VEC = 16 / (int)sizeof(T);
  static constexpr int COLS = 32 * VEC;
  static constexpr int ROW_BYTES = 512;  // COLS values
  static constexpr int ROWS = 0;
  static constexpr int INROW = ROWS + 4 * MAX_WARPS * ROW_BYTES;
  static constexpr int COLC = INROW + (CLUSTER ? 4 * MAX_WARPS * ROW_BYTES : 0);
  static constexpr int COEF = COLC + 4 * MAX_WARPS * ROW_BYTES;
  static constexpr int EDGE = COEF + (MAX_WARPS * R + 1) * 32;
  static constexpr int EDGE_PAR = 2 * MAX_WARPS * R * (int)sizeof(T);
  static constexpr int BAR = (EDGE + 2 * EDGE_PAR + 7) / 8 * 8;
  static constexpr int FLAG = (BAR + (CLUSTER ? 4 * MAX_WARPS * 8 : 0) + 15) / 16 * 16;
  static constexpr int CES = FLAG + 16;
  static constexpr int BYTES = CES + (R >= 3 ? MAX_WARPS * R * ROW_BYTES : 0);

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

// the 16 bytes at `a` where ok, else v as it was: one predicated load straight into
// v's registers.  (A choice between the value read and another one is made on the
// spot: it waits for the load that was meant to be under way.)
template <typename T>
__device__ __forceinline__ void ld16_where(const T* a, bool ok, Pack<T>& v) {
  uint64_t x = bits(v.p[0]), y = bits(v.p[1]);
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p ld.global.v2.b64 {%0, %1}, [%2];\n\t}"
      : "+l"(x), "+l"(y)
      : "l"(a), "r"((int)ok));
  from_bits(x, v.p[0]);
  from_bits(y, v.p[1]);
}

// bounded wait for a phase of an mbarrier
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity) {
  for (unsigned n = 0; n < PROBE_LIMIT; ++n)
    if (mbar_try_wait_sleep(bar, parity, PROBE_NS)) return true;
  return false;
}

// ---------------------------------------------------------------------------
// a warp's block: its place in the grid, and its exchange with its neighbours
// ---------------------------------------------------------------------------
template <typename T, int R, int MAIL, bool LISTED>
struct Block {
  static constexpr bool CLUSTER = MAIL == MAIL_CLUSTER;
  using L = Smem<T, R, CLUSTER>;
  static constexpr int VEC = L::VEC;
  static constexpr int COLS = L::COLS;
  using V = Pack<T>;
  static constexpr int ROW_PAR = L::row(1, 0, 0) - L::row(0, 0, 0);
  static constexpr int ROW_BOT = L::row(0, 1, 0) - L::row(0, 0, 0);
  static constexpr int IN_PAR = L::inrow(0, 1, 0) - L::inrow(0, 0, 0);
  static constexpr int EDGE_P = L::EDGE_PAR / (int)sizeof(T);
  static constexpr int BAR_PAR = MAX_WARPS;  // mbarriers between the two slots

  unsigned char* smem;
  unsigned polls;  // LISTED: bound of one wait
  int* status;
  int lane, w, strip, group, ia0, ia, j0, jv;
  bool active;  // has a block (a CTA may have more warps than a grid's bands use)
  bool live, any, full;
  bool first_row, last_row, first_col, last_col;
  bool band_up, band_dn;  // rows from and to another CTA
  bool tail;              // the lane that holds column W-1
  // the last lane with a neighbour to the right: lane 31, or the one that holds
  // column W-1, which reads its own column there
  bool right_lane;
  // this warp's rows and columns in shared memory, and those it reads
  unsigned char* my_row;
  const unsigned char *up_row, *dn_row;
  int up_par, dn_par;
  T *my_left, *my_right;
  const T *l_edge, *r_edge;
  const unsigned char *cc, *cf;  // column and row coefficients
  // mailboxes
  uint64_t *bar_up, *bar_dn;
  uint32_t to_up, to_dn, tob_up, tob_dn;
  const uint64_t *in_up, *in_dn;
  uint64_t *out_up, *out_dn;
  long long slot;

  __device__ __forceinline__ Block(int H, int W, const Split& S, int band, unsigned char* smem_,
                                   uint64_t* mail, unsigned polls_, int* status_) {
    smem = smem_;
    polls = polls_;
    status = status_;
    lane = threadIdx.x & 31;
    w = threadIdx.x >> 5;
    strip = w % S.strips;
    group = w / S.strips;
    ia0 = band * S.groups * R;
    ia = ia0 + group * R;
    j0 = strip * COLS;
    jv = j0 + lane * VEC;
    active = group < S.groups;
    live = active && ia < H;
    any = jv < W;
    full = jv + VEC <= W;
    first_row = ia == 0;
    last_row = ia + R >= H;
    first_col = strip == 0;
    last_col = strip + 1 == S.strips;
    band_up = live && !first_row && group == 0;
    band_dn = live && !last_row && group + 1 == S.groups;
    tail = any && jv + VEC >= W;
    right_lane = last_col ? tail : lane == 31;
    my_row = smem + L::row(0, 0, w) + lane * 16;
    up_row = smem +
             (CLUSTER && band_up ? L::inrow(0, 0, strip)
              : first_row        ? L::row(0, 0, w)
                                 : L::row(0, 1, group > 0 ? w - S.strips : w)) +
             lane * 16;
    dn_row = smem +
             (CLUSTER && band_dn ? L::inrow(1, 0, strip)
              : last_row         ? L::row(0, 1, w)
                                 : L::row(0, 0, group + 1 < S.groups ? w + S.strips : w)) +
             lane * 16;
    up_par = CLUSTER && band_up ? IN_PAR : ROW_PAR;
    dn_par = CLUSTER && band_dn ? IN_PAR : ROW_PAR;
    my_left = reinterpret_cast<T*>(smem + L::edge(0, 0, w));
    my_right = reinterpret_cast<T*>(smem + L::edge(0, 1, w));
    l_edge = reinterpret_cast<const T*>(smem + L::edge(0, 1, first_col ? w : w - 1));
    r_edge = reinterpret_cast<const T*>(smem + (last_col ? L::edge(0, 1, w) : L::edge(0, 0, w + 1)));
    cc = smem + L::COLC + strip * 512 + lane * 16;
    cf = smem + L::COEF + 32 * group * R;
    slot = (long long)S.strips * ROW_WORDS;
    if constexpr (CLUSTER) {
      bar_up = reinterpret_cast<uint64_t*>(smem + L::bar(0, 0, strip));
      bar_dn = reinterpret_cast<uint64_t*>(smem + L::bar(1, 0, strip));
      const int up = band > 0 ? band - 1 : band, dn_ = band + 1 < S.bands ? band + 1 : band;
      to_up = map_cta(smem_u32(smem + L::inrow(1, 0, strip) + lane * 16), up);
      tob_up = map_cta(smem_u32(bar_dn), up);
      to_dn = map_cta(smem_u32(smem + L::inrow(0, 0, strip) + lane * 16), dn_);
      tob_dn = map_cta(smem_u32(bar_up), dn_);
    } else {
      // mail[up/down][band][parity][strip]
      const long long mine = (long long)strip * ROW_WORDS + lane;
      uint64_t* const up_box = mail;
      uint64_t* const dn_box = mail + (long long)S.bands * 2 * slot;
      in_up = up_box + (long long)band * 2 * slot + mine;
      in_dn = dn_box + (long long)band * 2 * slot + mine;
      out_up = dn_box + (long long)(band - 1) * 2 * slot + mine;
      out_dn = up_box + (long long)(band + 1) * 2 * slot + mine;
    }
  }

  // coefficients of the band's rows and the strips' columns, and cleared flags
  template <typename P>
  __device__ __forceinline__ void coefficients(const P& J, const Split& S) const {
    using C = typename V::S;
    const double idl = 1.0 / J.dl;
    C* coef = reinterpret_cast<C*>(smem + L::COEF);
    for (int e = threadIdx.x; e < S.groups * R + 1; e += blockDim.x) {
      const int i = ia0 + e;
      const double g = i < J.H ? 1.0 + J.c[0][i] : 1.0;
      coef[4 * e] = both(i < J.H ? static_cast<T>(J.b[0][i]) : T(1));
      coef[4 * e + 1] = both(static_cast<T>(-(J.dt * g * idl)));
      coef[4 * e + 2] = both(static_cast<T>(-(g * idl)));
      coef[4 * e + 3] = both(T(i < J.H - 1 ? 1 : 0));
    }
    T* colc = reinterpret_cast<T*>(smem + L::COLC);
    for (int j = threadIdx.x; j < S.strips * COLS; j += blockDim.x) {
      const double g = j < J.W ? 1.0 + J.c[1][j] : 1.0;
      colc[j] = j < J.W ? static_cast<T>(J.b[1][j]) : T(1);
      colc[MAX_WARPS * COLS + j] = static_cast<T>(J.dt * g * idl);
      colc[2 * MAX_WARPS * COLS + j] = static_cast<T>(g * idl);
      colc[3 * MAX_WARPS * COLS + j] = T(j < J.W - 1 ? 1 : 0);
    }
    if (threadIdx.x == 0) *reinterpret_cast<int2*>(smem + L::FLAG) = make_int2(0, 0);
  }

  // one row of an array, zero outside the grid
  __device__ __forceinline__ V load(const T* a, long long o, bool ok, int W) const {
    return pack_of<T>(ldv<T, VEC>(a, o, ok && live && any, full, jv, W));
  }

  // rows and edge columns of `f` for the CTA's other warps
  __device__ __forceinline__ void publish(int par, const V (&f)[R]) const {
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
  }

  // the block's first and last row to the neighbour bands (after step n)
  __device__ __forceinline__ void post(int nxt, int n, const V (&f)[R]) const {
    if constexpr (CLUSTER) {
      if (band_up) post_async<T>(to_up + nxt * IN_PAR, tob_up + nxt * BAR_PAR * 8, f[0]);
      if (band_dn) post_async<T>(to_dn + nxt * IN_PAR, tob_dn + nxt * BAR_PAR * 8, f[R - 1]);
    } else {
      if (band_up) post_words<T>(out_up + nxt * slot, n + 1, f[0]);
      if (band_dn) post_words<T>(out_dn + nxt * slot, n + 1, f[R - 1]);
    }
  }

  // after the CTA's barrier: the rows above and below after step n (slot and
  // buffer parity nxt); false when some wait of the step before ran out
  __device__ __forceinline__ bool gather(int nxt, int n, V& f_up, V& f_dn) const {
    const int failed = *reinterpret_cast<volatile int*>(smem + L::FLAG + nxt * 4);
    bool bad = false;
    if constexpr (CLUSTER) {
      if (band_up || band_dn) {
        const uint32_t ph = (uint32_t)(n >> 1) & 1u;  // the slot's (n / 2 + 1)-th use
        if (band_up) {
          bad |= !wait_bar(bar_up + nxt * BAR_PAR, ph);
          if (lane == 0) mbar_arrive_expect_tx(bar_up + nxt * BAR_PAR, 512);
        }
        if (band_dn) {
          bad |= !wait_bar(bar_dn + nxt * BAR_PAR, ph);
          if (lane == 0) mbar_arrive_expect_tx(bar_dn + nxt * BAR_PAR, 512);
        }
        __syncwarp();
      }
      f_up = ld16<T>(up_row + nxt * up_par);
      f_dn = ld16<T>(dn_row + nxt * dn_par);
    } else {
      if (!band_up) f_up = ld16<T>(up_row + nxt * ROW_PAR);
      if (!band_dn) f_dn = ld16<T>(dn_row + nxt * ROW_PAR);
      if (band_up && band_dn) {
        bad = !take_words<T, true, LISTED>(in_up + nxt * slot, in_dn + nxt * slot, n + 1, f_up, f_dn,
                                   polls, status);
      } else if (band_up || band_dn) {
        V v, unused;
        bad = !take_words<T, false, LISTED>((band_up ? in_up : in_dn) + nxt * slot, nullptr, n + 1, v,
                                    unused, polls, status);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          f_up.p[h] = band_up ? v.p[h] : f_up.p[h];
          f_dn.p[h] = band_up ? f_dn.p[h] : v.p[h];
        }
      }
    }
    if (bad) {  // seen by every warp behind the next barrier
      report_status(status, DN_ETIMEOUT);
      *reinterpret_cast<volatile int*>(smem + L::FLAG + (nxt ^ 1) * 4) = 1;
    }
    return failed == 0;
  }
};

// a cluster's mailboxes, armed before any row is sent
template <typename L>
__device__ __forceinline__ void arm_mailboxes(unsigned char* smem) {
  if (threadIdx.x == 0) {
    for (int e = 0; e < 4 * MAX_WARPS; ++e) {
      uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::BAR) + e;
      mbar_init(bar, 1);
      mbar_arrive_expect_tx(bar, 512);
    }
    fence_barrier_init();
  }
  cg::this_cluster().sync();
}

// launch of `kern` with one CTA per band: as a cluster, or cooperative
template <typename K, typename... A>
int launch_bands(K kern, const Split& S, int smem, cudaStream_t s, A... args) {
  DN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  if (S.cluster)
    DN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[1];
  lc.blockDim = dim3(S.strips * S.groups * 32);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  lc.attrs = at;
  lc.numAttrs = 1;
  if (S.cluster) {
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
  DN_CUDA_CHECK(cudaLaunchKernelEx(&lc, kern, args...));
  return DN_OK;
}

}  // namespace res
}  // namespace dn
