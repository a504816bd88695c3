// Resident runs and reverse sweeps of many TM grids in one launch
// (dn_resident2d.cuh, struct List).
#pragma once

#include "dn_resident2d_adj.cuh"
#include "dn_resident2d_fwd.cuh"

namespace dn {
namespace res {

// the run of one band of a listed grid; its description is built in shared memory
template <typename T, int R, bool ADJ, bool REC>
__global__ void __launch_bounds__(MAX_WARPS * 32, 1)
    k_resident2d_list(const List L, int* status) {
  using LY = Smem<T, R, false>;
  constexpr int VEC = 16 / (int)sizeof(T);
  extern __shared__ __align__(16) unsigned char r_smem[];
  __shared__ Job<T> J;
  __shared__ AdjJob<T> A;
  __shared__ Samples<T> smp;
  if (status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0) return;
  for (int q = L.start[blockIdx.x]; q < L.start[blockIdx.x + 1]; ++q) {
    const ListJob job = L.jobs[q];
    const ListGrid& G = L.grids[job.grid];
    const dn_batch2d_inst& I = L.inst[job.grid];
    const Split S{R, G.strips, G.groups, G.bands, 0};
    __syncthreads();  // the job before is done with shared memory
    if (threadIdx.x == 0) {
      const int T_ = I.n_steps;
      for (int a = 0; a < 2; ++a) {
        smp.lo[a] = I.mon_box.lo[1 + a];
        smp.hi[a] = I.mon_box.hi[1 + a];
      }
      smp.comp = 0;
      smp.vec = smp.lo[1] % VEC == 0 && (smp.hi[1] - smp.lo[1]) % VEC == 0;
      smp.buf = reinterpret_cast<T*>(L.samples + G.sample);
      smp.step_stride = G.stride;
      if constexpr (ADJ) {
        A.H = I.H, A.W = I.W, A.py = I.pitch;
        for (int c = 0; c < 3; ++c) {
          A.in[c] = static_cast<const T*>(I.lam[T_ & 1][c]);
          A.out[c] = static_cast<T*>(I.lam[0][c]);
        }
        A.ce = static_cast<const T*>(I.ce);
        for (int a = 0; a < 2; ++a) A.b[a] = I.b[a], A.c[a] = I.c[a];
        A.dt = I.dt, A.dl = I.dl;
        A.nsteps = T_;
        A.curl_stride = (long long)I.H * I.pitch;
        A.curl = static_cast<const T*>(I.curl) + (T_ - 1) * A.curl_stride;
        A.grad = I.grad;
      } else {
        J.H = I.H, J.W = I.W, J.py = I.pitch;
        for (int c = 0; c < 3; ++c) {
          J.in[c] = static_cast<const T*>(I.f[0][c]);
          J.out[c] = static_cast<T*>(I.f[T_ & 1][c]);
        }
        J.ce = static_cast<const T*>(I.ce);
        for (int a = 0; a < 2; ++a) {
          J.b[a] = I.b[a], J.c[a] = I.c[a];
          J.src_lo[a] = I.src_box.lo[1 + a];
          J.src_hi[a] = I.src_box.hi[1 + a];
        }
        J.dt = I.dt, J.dl = I.dl;
        J.src = I.src_comp != DN_NONE;
        J.wave = static_cast<const T*>(I.wave);
        J.t0 = 0;
        J.nsteps = T_;
        J.curl[0] = static_cast<T*>(I.curl);
        J.curl[1] = nullptr;
        J.curl_stride = (long long)I.H * I.pitch;
      }
    }
    __syncthreads();
    const int n = I.mon_comp != DN_NONE && (!ADJ || I.gmon != nullptr);
    if constexpr (ADJ)
      sweep_band<T, R, MAIL_GLOBAL, true>(A, S, job.band, r_smem, L.mail + G.mail, L.polls,
                                          status, &smp, n);
    else
      run_band<T, DN_TM, R, MAIL_GLOBAL, REC, true, true>(J, S, job.band, r_smem,
                                                          L.mail + G.mail, L.polls, status, &smp,
                                                          n);
  }
}

template <typename T>
int run_resident_list(const List& L, bool adjoint, bool record, int R, int n_cta, int* status,
                      cudaStream_t s) {
  // a split whose bands are the launch's CTAs of 16 warps each
  const Split grid{R, MAX_WARPS, 1, n_cta, 0};
  using std::integral_constant;
  auto go = [&](auto r_c, auto adj_c, auto rec_c) {
    constexpr int RR = decltype(r_c)::value;
    return launch_bands(k_resident2d_list<T, RR, decltype(adj_c)::value, decltype(rec_c)::value>,
                        grid, Smem<T, RR, false>::BYTES, s, L, status);
  };
  constexpr std::true_type yes{};
  constexpr std::false_type no{};
  constexpr integral_constant<int, 1> r1{};
  constexpr integral_constant<int, 2> r2{};
  constexpr integral_constant<int, 4> r4{};
  if (adjoint) return R == 1 ? go(r1, yes, no) : R == 2 ? go(r2, yes, no) : DN_EINVAL;
  if (record)
    return R == 1 ? go(r1, no, yes) : R == 2 ? go(r2, no, yes) : R == 4 ? go(r4, no, yes) : DN_EINVAL;
  return R == 1 ? go(r1, no, no) : R == 2 ? go(r2, no, no) : R == 4 ? go(r4, no, no) : DN_EINVAL;
}

}  // namespace res
}  // namespace dn
