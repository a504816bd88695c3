// Resident 3-D runs: all steps of a small FP32 grid in one launch, the six field
// components and dt/eps in shared memory from the first step to the last.
//
// Replaces, for grids that fit, the loop of dn_fdtd3d.cu over one launch per step
// (the reference's FDTDSolver3D._run_steps, diffnano/solvers/fdtd3d.py:490-502),
// which below ~100^3 waits for launches and for its pipeline to fill rather than
// for memory.
//
// The (z, y) rows of the grid are cut into one block per CTA (cooperative launch,
// one CTA per SM); a row along x stays whole.  A block holds E of its rows and of a
// one-row frame around them, and H of its rows and of the frame's low sides.  A
// step updates H of all of these from E, then E of the block's own rows from H: the
// H rows of the low frame are the neighbours' own, computed here again with the
// same explicitly rounded operations, so only E travels, once per step.
//   H rows that need no neighbour's E, while E of this step is on its way;
//   take the frame's E rows;  H rows that needed them;
//   E of the own rows, those that others wait for first and sent at once.
// A row travels as 16-byte words (Ex, Ey, Ez, step number) in global memory (two
// sets by the step's parity), written and polled with single 128-bit accesses, so a
// word's values have arrived when its number has.  A CTA writes the words of step
// n + 2 only after its neighbours' words of step n + 1, which they send after they
// took those of step n.
//
// A thread owns four columns for the whole run (their x profiles stay in
// registers) and walks rows; the x neighbours of its four cells come by shuffle.
//
// B200, us per step: 40^3 2.2, 64^3 2.9, 80^3 5.1, 90^3 6.9; one launch per step takes
// 3.4 (40^3) to 11 (90^3).  Small grids wait for the trip of the rows (about 1.3 us)
// and three barriers; from 70^3 on shared memory is the bound (27 16-byte accesses per
// four cells; 59 % of its wavefronts at 90^3 over the whole step, 39 % of the issue
// slots).
#include <algorithm>

#include "dn_host.cuh"
#include "dn_sample_dft.cuh"

namespace dn {
namespace res3 {
namespace {

constexpr int NT = 512;
constexpr unsigned ALL = 0xffffffffu;
constexpr unsigned SPIN_LIMIT = 1u << 22;  // ~ seconds per wait
constexpr int SMEM_MAX = 227 * 1024;
constexpr int MAX_SAMPLES = DN_MAX_MONITORS + 1;  // the monitors and the probe

struct Samples {
  int lo[3], hi[3];
  int comp;
  long long stride;  // per step
  float* buf;
};

struct Job {
  int D, H, W;
  long long py, pz;
  const float* in[6];
  float* out[6];
  const float* ce;
  const double* b[3];
  const double* c[3];
  float dt, idl;
  int src;  // component (E), or DN_NONE
  int src_lo[3], src_hi[3];
  const float* wave;  // of the run's first step
  int n_samples;
  Samples s[MAX_SAMPLES];
  float* curl[3];  // of the run's first step
  long long curl_stride;
  int nsteps;
  int bz, by;        // blocks along z and y
  int nzm, nym;      // rows of the largest block
  uint4* words;      // [parity][i][j][column % 4][column / 4]
  int* status;
};

// ---- shared memory ---------------------------------------------------------------
// E[3][nz + 2][ny + 2][P]  H[3][nz + 1][ny + 1][P]  ce[nz][ny][P]
// rows: (b_y, dt (1+c_y)/dl, (1+c_y)/dl, 1+c_y) of the frame's rows, planes alike
// the row lists, the samples, the abort flag
struct Sizes {
  int P;       // floats per row
  int e, h;    // floats per component
  int tab, lists, total;  // byte offsets, bytes
};
__host__ __device__ inline Sizes sizes_of(int W, int nz, int ny) {
  Sizes z;
  z.P = (W + 3) / 4 * 4;
  z.e = (nz + 2) * (ny + 2) * z.P;
  z.h = (nz + 1) * (ny + 1) * z.P;
  z.tab = (4 + 3 * z.e + 3 * z.h + nz * ny * z.P + 4) * 4;  // 4 floats around: x neighbours
  z.lists = z.tab + (ny + 2 + nz + 2) * 16;
  const int rows = 2 * (nz + 1) * (ny + 1) + 2 * (nz + ny + 2) + nz * ny;
  z.total = z.lists + rows * 4 + MAX_SAMPLES * (int)sizeof(Samples) + 64;
  return z;
}

__device__ __forceinline__ float4 ld4(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ void st4(float* p, const float v[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void un4(const float4 v, float o[4]) {
  o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
}
// the first n of four columns to global memory
__device__ __forceinline__ void put4(float* p, const float v[4], int n) {
  if (n >= 4) {
    st4(p, v);
  } else {
    for (int q = 0; q < 3; ++q)
      if (q < n) p[q] = q == 0 ? v[0] : q == 1 ? v[1] : v[2];
  }
}

// a b - c d, rounded as the launch-by-launch kernel is compiled (whole runs agree
// with it bit for bit)
__device__ __forceinline__ float fms(float a, float b, float c, float d) {
  return __fmaf_rn(a, b, -__fmul_rn(c, d));
}

__device__ __forceinline__ void send_word(uint4* p, float a, float b, float c, uint32_t tag) {
  const uint64_t lo = (uint64_t)__float_as_uint(b) << 32 | __float_as_uint(a);
  const uint64_t hi = (uint64_t)tag << 32 | __float_as_uint(c);
  asm volatile(
      "{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(
          p),
      "l"(lo), "l"(hi)
      : "memory");
}
__device__ __forceinline__ void read_word(const uint4* p, uint64_t& lo, uint64_t& hi) {
  asm volatile(
      "{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
}

template <int AXES, bool REC>
__global__ void __launch_bounds__(NT, 1) k_resident3d(const __grid_constant__ Job J) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (J.status != nullptr && *reinterpret_cast<const volatile int*>(J.status) != 0) return;
  const int tid = threadIdx.x, lane = tid & 31;
  const int D = J.D, H = J.H, W = J.W;
  const int bi = blockIdx.x / J.by, bj = blockIdx.x % J.by;
  const int z0 = (int)((long long)bi * D / J.bz), z1 = (int)((long long)(bi + 1) * D / J.bz);
  const int y0 = (int)((long long)bj * H / J.by), y1 = (int)((long long)(bj + 1) * H / J.by);
  const int nz = z1 - z0, ny = y1 - y0;
  const Sizes Z = sizes_of(W, J.nzm, J.nym);
  const int P = Z.P;
  float* const sE = reinterpret_cast<float*>(smem) + 4;
  float* const sH = sE + 3 * Z.e;
  float* const sC = sH + 3 * Z.h;
  float4* const rowc = reinterpret_cast<float4*>(smem + Z.tab);
  float4* const planec = rowc + J.nym + 2;
  int* const lists = reinterpret_cast<int*>(smem + Z.lists);
  int* const l_free = lists;                              // H rows without a neighbour's E
  int* const l_late = l_free + (J.nzm + 1) * (J.nym + 1);  // the other H rows
  int* const l_send = l_late + (J.nzm + 1) * (J.nym + 1);  // own rows, sent ones first
  int* const l_take = l_send + J.nzm * J.nym;              // rows of the frame
  Samples* const smp =
      reinterpret_cast<Samples*>(((uintptr_t)(l_take + 2 * (J.nzm + J.nym + 2)) + 7) & ~7ull);
  __shared__ int n_free, n_late, n_send, n_own, n_take;
  __shared__ int failed;

  // ---- set-up ------------------------------------------------------------------------
  const bool has_zm = z0 > 0, has_zp = z1 < D, has_ym = y0 > 0, has_yp = y1 < H;
  const float dti = J.dt * J.idl;
  for (int e = tid; e < Z.tab / 4; e += NT) reinterpret_cast<float*>(smem)[e] = 0.0f;
  for (int e = tid; e < ny + 2; e += NT) {
    const int j = y0 - 1 + e;
    const bool ok = j >= 0 && j < H;
    const float b = ok ? (float)J.b[1][j] : 1.0f, g = ok ? (float)(1.0 + J.c[1][j]) : 1.0f;
    rowc[e] = make_float4(b, j < H - 1 ? dti * g : 0.0f, j > 0 ? g * J.idl : 0.0f, g);
  }
  for (int e = tid; e < nz + 2; e += NT) {
    const int i = z0 - 1 + e;
    const bool ok = AXES == DN_AXES_PHYSICAL && i >= 0 && i < D;
    const float b = ok ? (float)J.b[0][i] : 1.0f, g = ok ? (float)(1.0 + J.c[0][i]) : 1.0f;
    planec[e] = make_float4(b, dti * g, g * J.idl, 0.0f);
  }
  // the lists hold (plane << 16 | row), counted from the frame's low corner
  if (tid == 0) {
    int nf = 0, nl = 0, nt = 0;
    for (int a = 0; a <= nz; ++a)
      for (int b = 0; b <= ny; ++b) {
        if ((a == 0 && (!has_zm || b == 0)) || (b == 0 && !has_ym)) continue;
        const bool late = a == 0 || b == 0 || (a == nz && has_zp) || (b == ny && has_yp);
        (late ? l_late[nl++] : l_free[nf++]) = a << 16 | b;
      }
    for (int a = 0; a <= nz + 1; ++a)
      for (int b = 0; b <= ny + 1; ++b) {
        if (a > 0 && a <= nz && b > 0 && b <= ny) continue;
        if ((a == 0 && !has_zm) || (a == nz + 1 && !has_zp) || (b == 0 && !has_ym) ||
            (b == ny + 1 && !has_yp) || (a == 0 && b == 0) || (a == nz + 1 && b == ny + 1))
          continue;
        l_take[nt++] = a << 16 | b;
      }
    n_free = nf;
    n_late = nl;
    n_take = nt;
    failed = 0;
  }
  if (tid == 32) {
    int k = 0;
    for (int pass = 0; pass < 2; ++pass) {
      for (int a = 1; a <= nz; ++a)
        for (int b = 1; b <= ny; ++b) {
          const bool send = (a == 1 && has_zm) || (a == nz && has_zp) || (b == 1 && has_ym) ||
                            (b == ny && has_yp);
          if (send == (pass == 0)) l_send[k++] = a << 16 | b;
        }
      if (pass == 0) n_send = k;
    }
    n_own = k;
  }
  if (tid == 64)
    for (int m = 0; m < MAX_SAMPLES; ++m) smp[m] = J.s[m];
  __syncthreads();

  // ---- this thread's columns ------------------------------------------------------------
  const int nvec = P / 4, groups = NT / nvec;
  const int g = tid / nvec, v = tid - g * nvec, k0 = 4 * v;
  const bool on = g < groups;
  const int kn = W - k0;  // columns inside the grid (may be above 4)
  const bool last_v = v == nvec - 1;
  float bK[4], hK[4], eK[4];  // b_x, dt (1+c_x)/dl, (1+c_x)/dl; 0 beyond the grid
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = k0 + q;
    const bool ok = on && k < W;
    const float gk = ok ? (float)(1.0 + J.c[2][k]) : 0.0f;
    bK[q] = ok ? (float)J.b[2][k] : 0.0f;
    hK[q] = dti * gk;
    eK[q] = gk * J.idl;
  }
  // forward x difference at column q, backward x difference at column q
  auto kf = [&](int q) { return k0 + q < W - 1 ? 1.0f : 0.0f; };
  auto kb = [&](int q) { return k0 + q > 0 && k0 + q < W ? 1.0f : 0.0f; };

  const int eR = (J.nym + 2) * P, hR = (J.nym + 1) * P;  // floats per plane
  auto e_at = [&](int a, int b) { return a * eR + b * P + k0; };
  auto h_at = [&](int a, int b) { return a * hR + b * P + k0; };

  // ---- fields in ------------------------------------------------------------------------
  auto load = [&](const float* base, int i, int j, float o[4]) {
    un4(__ldcg(reinterpret_cast<const float4*>(base + i * J.pz + j * J.py + k0)), o);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q >= kn) o[q] = 0.0f;
  };
  if (on) {
    for (int r = g; r < (nz + 2) * (ny + 2); r += groups) {
      const int a = r / (ny + 2), b = r % (ny + 2), i = z0 - 1 + a, j = y0 - 1 + b;
      if (i < 0 || i >= D || j < 0 || j >= H) continue;
      float o[4];
      for (int c = 0; c < 3; ++c) {
        load(J.in[c], i, j, o);
        st4(sE + c * Z.e + e_at(a, b), o);
      }
      if (a <= nz && b <= ny)
        for (int c = 0; c < 3; ++c) {
          load(J.in[3 + c], i, j, o);
          st4(sH + c * Z.h + h_at(a, b), o);
        }
      if (a > 0 && a <= nz && b > 0 && b <= ny) {
        load(J.ce, i, j, o);
        st4(sC + ((a - 1) * J.nym + b - 1) * P + k0, o);
      }
    }
  }
  __syncthreads();

  // new H of the rows of a list
  auto h_rows = [&](const int* list, int n) {
    for (int r0 = 0; r0 < n; r0 += groups) {
      const bool act = on && r0 + g < n;
      if (!__any_sync(ALL, act)) continue;
      const int ab = act ? list[r0 + g] : list[r0];
      const int a = ab >> 16, b = ab & 0xffff;
      const int e = e_at(a, b), h = h_at(a, b);
      const int en = z0 - 1 + a < D - 1 ? e + eR : e;  // no difference on the last plane
      float ex[4], ey[4], ez[4], exj[4], ezj[4], exi[4], eyi[4], hx[4], hy[4], hz[4];
      un4(ld4(sE + e), ex);
      un4(ld4(sE + Z.e + e), ey);
      un4(ld4(sE + 2 * Z.e + e), ez);
      un4(ld4(sE + e + P), exj);
      un4(ld4(sE + 2 * Z.e + e + P), ezj);
      un4(ld4(sE + en), exi);
      un4(ld4(sE + Z.e + en), eyi);
      un4(ld4(sH + h), hx);
      un4(ld4(sH + Z.h + h), hy);
      un4(ld4(sH + 2 * Z.h + h), hz);
      float eyk = __shfl_down_sync(ALL, ey[0], 1), ezk = __shfl_down_sync(ALL, ez[0], 1);
      if (lane == 31) {
        eyk = sE[Z.e + e + 4];
        ezk = sE[2 * Z.e + e + 4];
      }
      if (last_v) eyk = ezk = 0.0f;
      const float4 rc = rowc[b], pc = planec[a];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float yk = q < 3 ? ey[q < 3 ? q + 1 : 3] : eyk, zk = q < 3 ? ez[q < 3 ? q + 1 : 3] : ezk;
        const float cKf = kf(q) * hK[q];
        const float c_i = AXES == DN_AXES_REFERENCE ? hK[q] : pc.y;
        const float hy_b = AXES == DN_AXES_REFERENCE ? bK[q] : pc.x;
        const float hy_k = AXES == DN_AXES_REFERENCE ? kf(q) * (dti * rc.w) : cKf;
        hx[q] = __fmaf_rn(c_i, __fsub_rn(eyi[q], ey[q]),
                          fms(rc.x, hx[q], rc.y, __fsub_rn(ezj[q], ez[q])));
        hy[q] = __fmaf_rn(hy_k, __fsub_rn(zk, ez[q]),
                          fms(hy_b, hy[q], c_i, __fsub_rn(exi[q], ex[q])));
        hz[q] = __fmaf_rn(rc.y, __fsub_rn(exj[q], ex[q]),
                          fms(bK[q], hz[q], cKf, __fsub_rn(yk, ey[q])));
      }
      if (act) {
        st4(sH + h, hx);
        st4(sH + Z.h + h, hy);
        st4(sH + 2 * Z.h + h, hz);
      }
    }
  };

  // new E of the own rows; `more`: the first n_send to the neighbours too
  auto e_rows = [&](int n, float w, bool more) {
    for (int r0 = 0; r0 < n_own; r0 += groups) {
      const bool act = on && r0 + g < n_own, send = more && r0 + g < n_send;
      if (!__any_sync(ALL, act)) continue;
      const int ab = act ? l_send[r0 + g] : l_send[r0];
      const int a = ab >> 16, b = ab & 0xffff;
      const int i = z0 - 1 + a, j = y0 - 1 + b;
      const int e = e_at(a, b), h = h_at(a, b);
      const int hp = i > 0 ? h - hR : h;  // no difference on the first plane
      float hx[4], hy[4], hz[4], hxj[4], hzj[4], hxi[4], hyi[4], ex[4], ey[4], ez[4], ce[4];
      un4(ld4(sH + h), hx);
      un4(ld4(sH + Z.h + h), hy);
      un4(ld4(sH + 2 * Z.h + h), hz);
      un4(ld4(sH + h - P), hxj);
      un4(ld4(sH + 2 * Z.h + h - P), hzj);
      un4(ld4(sH + hp), hxi);
      un4(ld4(sH + Z.h + hp), hyi);
      un4(ld4(sE + e), ex);
      un4(ld4(sE + Z.e + e), ey);
      un4(ld4(sE + 2 * Z.e + e), ez);
      un4(ld4(sC + ((a - 1) * J.nym + b - 1) * P + k0), ce);
      float hyk = __shfl_up_sync(ALL, hy[3], 1), hzk = __shfl_up_sync(ALL, hz[3], 1);
      if (lane == 0) {
        hyk = sH[Z.h + h - 1];
        hzk = sH[2 * Z.h + h - 1];
      }
      if (v == 0) hyk = hzk = 0.0f;
      const float4 rc = rowc[b], pc = planec[a];
      float crl[3][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float yk = q > 0 ? hy[q > 0 ? q - 1 : 0] : hyk, zk = q > 0 ? hz[q > 0 ? q - 1 : 0] : hzk;
        const float c_i = AXES == DN_AXES_REFERENCE ? eK[q] : pc.z;
        const float cKb = kb(q) * eK[q];
        const float ey_k = AXES == DN_AXES_REFERENCE ? kb(q) * (rc.w * J.idl) : cKb;
        const float bI = AXES == DN_AXES_REFERENCE ? 1.0f : pc.x;
        const float ex_b = AXES == DN_AXES_REFERENCE ? __fmul_rn(rc.x, bK[q]) : __fmul_rn(rc.x, bI);
        const float ey_b = AXES == DN_AXES_REFERENCE ? ex_b : __fmul_rn(bI, bK[q]);
        const float ez_b = __fmul_rn(bK[q], rc.x);
        crl[0][q] = fms(rc.z, __fsub_rn(hz[q], hzj[q]), c_i, __fsub_rn(hy[q], hyi[q]));
        crl[1][q] = fms(c_i, __fsub_rn(hx[q], hxi[q]), ey_k, __fsub_rn(hz[q], zk));
        crl[2][q] = fms(cKb, __fsub_rn(hy[q], yk), rc.z, __fsub_rn(hx[q], hxj[q]));
        ex[q] = __fmaf_rn(ce[q], crl[0][q], __fmul_rn(ex_b, ex[q]));
        ey[q] = __fmaf_rn(ce[q], crl[1][q], __fmul_rn(ey_b, ey[q]));
        ez[q] = __fmaf_rn(ce[q], crl[2][q], __fmul_rn(ez_b, ez[q]));
      }
      if (!act) continue;  // (no shuffle below)
      if (J.src >= 0 && i >= J.src_lo[0] && i < J.src_hi[0] && j >= J.src_lo[1] &&
          j < J.src_hi[1]) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float add = k0 + q >= J.src_lo[2] && k0 + q < J.src_hi[2] ? w : 0.0f;
          ex[q] += J.src == DN_EX ? add : 0.0f;
          ey[q] += J.src == DN_EY ? add : 0.0f;
          ez[q] += J.src == DN_EZ ? add : 0.0f;
        }
      }
      st4(sE + e, ex);
      st4(sE + Z.e + e, ey);
      st4(sE + 2 * Z.e + e, ez);
      if (send) {
        uint4* const to = J.words + ((long long)((n + 1) & 1) * D * H + (long long)i * H + j) * P + v;
#pragma unroll
        for (int q = 0; q < 4; ++q) send_word(to + q * nvec, ex[q], ey[q], ez[q], n + 1);
      }
      if (REC) {
        const long long o = (long long)n * J.curl_stride + i * J.pz + j * J.py + k0;
#pragma unroll
        for (int c = 0; c < 3; ++c) put4(J.curl[c] + o, crl[c], kn);
      }
      for (int m = 0; m < J.n_samples; ++m) {
        const Samples& S = smp[m];
        if (i < S.lo[0] || i >= S.hi[0] || j < S.lo[1] || j >= S.hi[1]) continue;
        float* const to = S.buf + n * S.stride +
                          ((long long)(i - S.lo[0]) * (S.hi[1] - S.lo[1]) + j - S.lo[1]) *
                              (S.hi[2] - S.lo[2]) - S.lo[2] + k0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int c = S.comp;
          const float x = c == DN_EX ? ex[q] : c == DN_EY ? ey[q] : c == DN_EZ ? ez[q]
                          : c == DN_HX ? hx[q] : c == DN_HY ? hy[q] : hz[q];
          if (k0 + q >= S.lo[2] && k0 + q < S.hi[2]) to[q] = x;
        }
      }
    }
  };

  // the frame's E rows of step n (bounded)
  auto take_rows = [&](int n) {
    const uint4* const from = J.words + (long long)(n & 1) * D * H * P + v;
    for (int r = g; on && r < n_take; r += groups) {
      const int ab = l_take[r], a = ab >> 16, b = ab & 0xffff;
      const uint4* const p = from + ((long long)(z0 - 1 + a) * H + y0 - 1 + b) * P;
      uint64_t lo[4], hi[4];
      bool ok = false;
      for (unsigned t = 0; t < SPIN_LIMIT && !ok; ++t) {
        ok = true;
#pragma unroll
        for (int q = 0; q < 4; ++q) read_word(p + q * nvec, lo[q], hi[q]);
#pragma unroll
        for (int q = 0; q < 4; ++q) ok = ok && (uint32_t)(hi[q] >> 32) == (uint32_t)n;
        if (!ok && (t & 1023u) == 1023u && J.status != nullptr &&
            *reinterpret_cast<const volatile int*>(J.status) != 0)
          break;
      }
      if (!ok) {
        report_status(J.status, DN_ETIMEOUT);
        failed = 1;
        return;
      }
      float ex[4], ey[4], ez[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ex[q] = __uint_as_float((uint32_t)lo[q]);
        ey[q] = __uint_as_float((uint32_t)(lo[q] >> 32));
        ez[q] = __uint_as_float((uint32_t)hi[q]);
      }
      const int e = e_at(a, b);
      st4(sE + e, ex);
      st4(sE + Z.e + e, ey);
      st4(sE + 2 * Z.e + e, ez);
    }
  };

  // ---- steps ------------------------------------------------------------------------------
  for (int n = 0; n < J.nsteps; ++n) {
    const float w = J.src >= 0 ? __ldg(J.wave + n) : 0.0f;
    h_rows(l_free, n_free);
    if (n > 0) take_rows(n);
    __syncthreads();
    if (failed) return;
    h_rows(l_late, n_late);
    __syncthreads();
    e_rows(n, w, n + 1 < J.nsteps);
    __syncthreads();
  }

  // ---- fields out ---------------------------------------------------------------------------
  for (int r = g; on && r < n_own; r += groups) {
    const int ab = l_send[r], a = ab >> 16, b = ab & 0xffff;
    const long long o = (z0 - 1 + a) * J.pz + (long long)(y0 - 1 + b) * J.py + k0;
    float x[4];
    for (int c = 0; c < 3; ++c) {
      un4(ld4(sE + c * Z.e + e_at(a, b)), x);
      put4(J.out[c] + o, x, kn);
      un4(ld4(sH + c * Z.h + h_at(a, b)), x);
      put4(J.out[3 + c] + o, x, kn);
    }
  }
}

// ---- host -----------------------------------------------------------------------------------
constexpr long long SAMPLE_BYTES = 64LL << 20;  // most workspace for samples
constexpr int MIN_STEPS = 8;  // shorter runs go launch by launch
constexpr int MIN_PIECE = 4 * MIN_STEPS;  // so do runs whose samples allow fewer steps per launch

struct Plan {
  bool ok;
  int bz, by, nz, ny, smem;
  long long word_bytes;    // both sets of the rows on their way
  long long sample_bytes;  // one step's samples of all monitors
  int piece;               // most steps per launch
};

// Blocks of rows, at most one per SM: among the splits whose largest block fits in
// shared memory, the one with the fewest turns of the threads through its three
// passes over rows, then with the fewest rows to update and to take per step.
Plan make_plan(const dn_grid* g, const dn_source* src, const dn_monitor* mons, int n_mon,
               int nsteps, int nsm = sm_count()) {
  Plan P{};
  if (g->dtype != DN_F32 || nsteps < MIN_STEPS || g->W > 4 * NT || g->D > 0x7fff || g->H > 0x7fff)
    return P;
  if (src && src->component != DN_NONE && src->component > DN_EZ) return P;
  long long best = -1;
  for (int bz = 1; bz <= nsm && bz <= g->D; ++bz)
    for (int by = 1; by * bz <= nsm && by <= g->H; ++by) {
      const int nz = (g->D + bz - 1) / bz, ny = (g->H + by - 1) / by;
      if ((long long)nz * ny > 4096) continue;
      const long long floats = 3LL * (nz + 2) * (ny + 2) + 3LL * (nz + 1) * (ny + 1) + nz * ny;
      if (floats * ((g->W + 3) / 4 * 4) * 4 > SMEM_MAX) continue;
      const Sizes Z = sizes_of(g->W, nz, ny);
      if (Z.total + 1024 > SMEM_MAX) continue;  // (the static variables)
      const int groups = NT / (Z.P / 4), late = 2 * (nz + ny) - 1;
      auto turns = [&](int rows) { return (long long)(rows + groups - 1) / groups; };
      const long long cost =
          (turns(nz * ny) + turns(std::max(0, nz * ny + nz + ny - late)) + turns(late)) * 1024 +
          nz * ny + (nz + 1LL) * (ny + 1) + 2LL * (nz + ny);
      if (best >= 0 && cost >= best) continue;
      best = cost;
      P.bz = bz;
      P.by = by;
      P.nz = nz;
      P.ny = ny;
      P.smem = Z.total;
    }
  if (best < 0) return P;
  P.word_bytes = 2LL * g->D * g->H * ((g->W + 3) / 4 * 4) * 16;
  P.piece = nsteps;
  for (int m = 0; m < n_mon; ++m)
    P.sample_bytes += (to_dev(mons[m].box).cells() * 4 + 15) / 16 * 16;
  if (P.sample_bytes * nsteps > SAMPLE_BYTES) {
    P.piece = (int)(SAMPLE_BYTES / P.sample_bytes);
    if (P.piece < MIN_PIECE) return P;
  }
  P.ok = true;
  return P;
}

long long workspace_of(const Plan& P) {
  return P.ok ? P.word_bytes + P.sample_bytes * P.piece : 0;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int AXES, bool REC>
int launch(const Job& J, int smem, cudaStream_t s) {
  auto kern = k_resident3d<AXES, REC>;
  DN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  lc.gridDim = dim3(J.bz * J.by);
  lc.blockDim = dim3(NT);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  lc.attrs = at;
  lc.numAttrs = 1;
  DN_CUDA_CHECK(cudaLaunchKernelEx(&lc, kern, J));
  return DN_OK;
}

int run(const dn_grid* g, void* const fa[6], void* const fb[6], const void* ce,
        const dn_cpml* cpml, const dn_source* src, const dn_monitor* mons, int32_t n_mon,
        const dn_probe* probe, const dn_curl_record* rec, int32_t t0, int32_t nsteps,
        int32_t* status, cudaStream_t s, int32_t* final_in_b, unsigned char* ws, int64_t ws_bytes,
        bool* done) {
  *done = false;
  StepParams<float> p;
  int rc = build_params<float>(true, g, fa, fb, ce, cpml, src, mons, n_mon, probe, status, &p);
  if (rc != DN_OK) return rc;
  if (t0 < 0 || !final_in_b || !steps_ok(src, mons, n_mon, probe, t0, (int64_t)t0 + nsteps))
    return DN_EINVAL;
  const Plan P = make_plan(g, src, mons, n_mon, nsteps);
  bool ok = P.ok && workspace_of(P) <= ws_bytes && aligned16(ws) && aligned16(ce) &&
            g->pitch_y % 4 == 0 && g->pitch_z % 4 == 0;
  for (int c = 0; c < 6; ++c) ok = ok && aligned16(fa[c]) && aligned16(fb[c]);
  if (rec) {
    for (int c = 0; c < 3; ++c) ok = ok && rec->curl[c] && aligned16(rec->curl[c]);
    ok = ok && rec->step_stride % 4 == 0 && rec->step_stride >= g->pitch_z * (int64_t)g->D &&
         rec->t0 >= 0 && t0 >= rec->t0 && t0 + nsteps <= rec->t0 + rec->nslots;
  }
  if (!ok) return DN_OK;  // (dn_fdtd3d_run takes it or refuses it)
  *done = true;
  Job J{};
  J.D = g->D;
  J.H = g->H;
  J.W = g->W;
  J.py = g->pitch_y;
  J.pz = g->pitch_z;
  J.ce = static_cast<const float*>(ce);
  for (int a = 0; a < 3; ++a) {
    J.b[a] = p.b[a];
    J.c[a] = p.c[a];
    J.src_lo[a] = p.src.box.lo[a];
    J.src_hi[a] = p.src.box.hi[a];
  }
  J.dt = p.dt;
  J.idl = p.inv_dl;
  J.src = p.src.comp;
  J.bz = P.bz;
  J.by = P.by;
  J.nzm = P.nz;
  J.nym = P.ny;
  J.words = reinterpret_cast<uint4*>(ws);
  J.status = status;
  if (rec) J.curl_stride = rec->step_stride;
  const Pieces cut(nsteps, P.piece);
  for (int piece = 0; piece < cut.count; ++piece) {
    const int n = cut.begin(piece), k = cut.begin(piece + 1) - n;
    J.nsteps = k;
    if (J.src >= 0) J.wave = p.src.wave + t0 + n;
    for (int c = 0; c < 6; ++c) {
      void* const to = nsteps % 2 ? fb[c] : fa[c];
      J.in[c] = static_cast<const float*>(n == 0 ? fa[c] : to);
      J.out[c] = static_cast<float*>(to);
    }
    for (int c = 0; c < 3 && rec; ++c)
      J.curl[c] = static_cast<float*>(rec->curl[c]) + (long long)(t0 + n - rec->t0) * J.curl_stride;
    J.n_samples = 0;
    unsigned char* at = ws + P.word_bytes;
    auto add = [&](int comp, const BoxDev& b, float* buf, long long stride) {
      Samples& q = J.s[J.n_samples++];
      for (int a = 0; a < 3; ++a) {
        q.lo[a] = b.lo[a];
        q.hi[a] = b.hi[a];
      }
      q.comp = comp;
      q.buf = buf;
      q.stride = stride;
    };
    for (int m = 0; m < p.n_mon; ++m) {
      const long long stride = (p.mon[m].ncell * 4 + 15) / 16 * 4;
      add(p.mon[m].comp, p.mon[m].box, reinterpret_cast<float*>(at), stride);
      at += stride * 4 * k;
    }
    if (p.probe.comp >= 0) {
      BoxDev b{};
      for (int a = 0; a < 3; ++a) b.lo[a] = p.probe.pos[a], b.hi[a] = p.probe.pos[a] + 1;
      add(p.probe.comp, b, p.probe.out + t0 + n, 1);
    }
    DN_CUDA_CHECK(cudaMemsetAsync(ws, 0, P.word_bytes, s));  // no step's number is 0
    if (g->axes == DN_AXES_REFERENCE)
      rc = rec ? launch<DN_AXES_REFERENCE, true>(J, P.smem, s)
               : launch<DN_AXES_REFERENCE, false>(J, P.smem, s);
    else
      rc = rec ? launch<DN_AXES_PHYSICAL, true>(J, P.smem, s)
               : launch<DN_AXES_PHYSICAL, false>(J, P.smem, s);
    if (rc != DN_OK) return rc;
    for (int m = 0; m < p.n_mon; ++m) {
      const MonDev& M = p.mon[m];
      res::k_sample_dft<float><<<(unsigned)((M.ncell + 31) / 32), res::DFT_WARPS * 32, 0, s>>>(
          J.s[m].buf, J.s[m].stride, k, M.ncell, M.phase + (long long)(t0 + n) * M.nf * 2, M.nf,
          M.acc, status);
    }
    DN_CUDA_CHECK(cudaGetLastError());
  }
  *final_in_b = nsteps % 2;
  return DN_OK;
}

}  // namespace
}  // namespace res3
}  // namespace dn

extern "C" int64_t dn_fdtd3d_workspace_bytes(const dn_grid* g, const dn_source* src,
                                             const dn_monitor* mons, int32_t n_mon,
                                             int32_t nsteps) {
  if (!g || g->D < 1 || g->H < 1 || g->W < 1 || (g->dtype != DN_F32 && g->dtype != DN_F64) ||
      n_mon < 0 || n_mon > DN_MAX_MONITORS || (n_mon > 0 && !mons))
    return -1;
  for (int m = 0; m < n_mon; ++m)
    if (!dn::box_ok(mons[m].box, g->D, g->H, g->W)) return -1;
  return dn::res3::workspace_of(dn::res3::make_plan(g, src, mons, n_mon, nsteps));
}

extern "C" int32_t dn_fdtd3d_resident_plan(const dn_grid* g, const dn_source* src,
                                           const dn_monitor* mons, int32_t n_mon, int32_t nsteps,
                                           int32_t n_sm, dn_resident_plan* out) {
  if (!out || n_sm < 0 || nsteps < 0 ||
      dn_fdtd3d_workspace_bytes(g, src, mons, n_mon, nsteps) < 0)
    return DN_EINVAL;
  *out = dn_resident_plan{};
  const dn::res3::Plan P =
      dn::res3::make_plan(g, src, mons, n_mon, nsteps, n_sm > 0 ? n_sm : dn::sm_count());
  if (!P.ok) return DN_OK;
  out->rows = P.nz * P.ny;
  out->bands = P.bz * P.by;
  return dn::describe_pieces(nsteps, P.piece, out);
}

extern "C" int32_t dn_fdtd3d_run_ws(const dn_grid* g, void* const fa[6], void* const fb[6],
                                    const void* ce, const dn_cpml* cpml, const dn_source* src,
                                    const dn_monitor* mons, int32_t n_mon, const dn_probe* probe,
                                    const dn_curl_record* rec, int32_t t0, int32_t nsteps,
                                    int32_t* status, void* stream, int32_t* final_in_b, void* ws,
                                    int64_t ws_bytes) {
  if (!g) return DN_EINVAL;
  if (g->dtype == DN_F32 && nsteps >= dn::res3::MIN_STEPS && ws) {
    bool done = false;
    const int rc = dn::res3::run(g, fa, fb, ce, cpml, src, mons, n_mon, probe, rec, t0, nsteps,
                                 status, static_cast<cudaStream_t>(stream), final_in_b,
                                 static_cast<unsigned char*>(ws), ws_bytes, &done);
    if (rc != DN_OK || done) return rc;
  }
  return dn_fdtd3d_run(g, fa, fb, ce, cpml, src, mons, n_mon, probe, rec, t0, nsteps, status,
                       stream, final_in_b);
}
