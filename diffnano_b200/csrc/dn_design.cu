// Design-layer kernels: density -> permittivity for the inverse-design loop.
//
//   rho (n_layers, H, W) --Gaussian filter in each layer--> rho_f
//   rho_f --projection--> p in (0, 1) --> eps = lo + (hi - lo) * p
//
// The filter is separable (a pass along x, then one along y) with the taps of
// the reference's smooth_filter (kernel 2r+1 rounded up to odd, sigma = r/2,
// normalised, zero padding).  Projections: the reference's sigmoid
// Heaviside, and the tanh projection
//   p = (tanh(beta eta) + tanh(beta (x - eta))) / (tanh(beta eta) + tanh(beta (1 - eta))).
// The backward pass maps d eps to d rho: the projection's derivative, then the
// same separable filter (its kernel is symmetric and zero padded, so the
// filter is its own transpose).  Erosion / dilation are 3x3 min / max pools
// per layer (cells outside the layer ignored) whose backward pass is a gather:
// every input adds the output gradients of the windows that selected it, in a
// fixed order, so results are deterministic.
#include "dn_common.cuh"
#include "dn_design.h"

namespace dn {
namespace ds {

constexpr int MAX_TAPS = 63;

struct Taps {
  float t[MAX_TAPS];
  int n;
};

__device__ __forceinline__ float project(float x, int kind, float beta, float eta, float den,
                                         float off) {
  if (kind == DN_PROJ_NONE) return x;
  if (kind == DN_PROJ_SIGMOID) return 1.0f / (1.0f + expf(-beta * (x - eta)));
  return (off + tanhf(beta * (x - eta))) / den;
}

__device__ __forceinline__ float project_grad(float x, int kind, float beta, float eta,
                                              float den) {
  if (kind == DN_PROJ_NONE) return 1.0f;
  if (kind == DN_PROJ_SIGMOID) {
    const float s = 1.0f / (1.0f + expf(-beta * (x - eta)));
    return beta * s * (1.0f - s);
  }
  const float t = tanhf(beta * (x - eta));
  return beta * (1.0f - t * t) / den;
}

// Filter of one 32 x 64 tile of a layer, both axes in one kernel: the tile with a
// border of `c` cells (zero outside the layer) goes to shared memory, a pass along
// x leaves 64 columns of all its rows there, a pass along y the tile itself.  A
// thread sums OUT neighbouring cells at a time from a register window over the
// line, one shared-memory read and one tap per OUT products; every sum adds its
// taps in ascending order.
//
// One read of the input and one write of each output (a pass of its own for each
// axis and one for the projection moved 7 arrays instead of 3 and spent most
// instructions on 64-bit index divisions): 40 x 256 x 256, 9 taps, on B200 59 -> 18 us
// forward, 61 -> 23 us backward.
constexpr int TW = 64, TH = 32, NTF = 256, MP = TW + 1;

__host__ __device__ constexpr int tile_pitch(int c) { return TW + 2 * c + 1; }
// (the window reads one cell past the last tap: a column more per row, and a row)
inline size_t tile_bytes(int taps) {
  const int c = taps / 2, rows = TH + 2 * c;
  return ((size_t)rows * tile_pitch(c) + (size_t)(rows + 1) * MP) * sizeof(float);
}

// a[o] = sum over q of t[q] x[(o + q) * STRIDE], o < OUT
template <int OUT, int STRIDE>
__device__ __forceinline__ void line_sums(const Taps& taps, const float* x, float a[OUT]) {
  float v[OUT];
#pragma unroll
  for (int o = 0; o < OUT; ++o) {
    a[o] = 0.0f;
    v[o] = x[o * STRIDE];
  }
  x += OUT * STRIDE;
  int q = 0;
  for (; q + OUT <= taps.n; q += OUT, x += OUT * STRIDE) {
#pragma unroll
    for (int u = 0; u < OUT; ++u) {
      const float t = taps.t[q + u];
#pragma unroll
      for (int o = 0; o < OUT; ++o) a[o] = fmaf(t, v[(u + o) % OUT], a[o]);
      v[u] = x[u * STRIDE];
    }
  }
#pragma unroll
  for (int u = 0; u < OUT - 1; ++u) {
    if (q + u >= taps.n) break;
    const float t = taps.t[q + u];
#pragma unroll
    for (int o = 0; o < OUT; ++o) a[o] = fmaf(t, v[(u + o) % OUT], a[o]);
    v[u] = x[u * STRIDE];
  }
}

template <typename Load, typename Store>
__device__ __forceinline__ void filter_tile(const Taps& taps, int H, int W, int h0, int w0,
                                            const Load& load, const Store& store) {
  extern __shared__ float f_smem[];
  const int c = taps.n / 2, rows = TH + 2 * c, pitch = tile_pitch(c);
  float* const in = f_smem;
  float* const mid = f_smem + rows * pitch;
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  auto get = [&](int h, int w) {
    return h >= 0 && h < H && w >= 0 && w < W ? load(h, w) : 0.0f;
  };
  // the 64 columns of the tile (several rows' loads in flight), then the border's
#pragma unroll 4
  for (int r = warp; r < rows; r += NTF / 32) {
    const float a = get(h0 - c + r, w0 + lane), b = get(h0 - c + r, w0 + lane + 32);
    in[r * pitch + c + lane] = a;
    in[r * pitch + c + lane + 32] = b;
  }
  for (int e = threadIdx.x; e < rows * 2 * c; e += NTF) {
    const int r = e / (2 * c), b = e % (2 * c), k = b < c ? b : b + TW;
    in[r * pitch + k] = get(h0 - c + r, w0 - c + k);
  }
  __syncthreads();
  constexpr int XO = 8;  // columns of a thread; lanes take rows, which the odd pitches spread over the banks
  for (int e = threadIdx.x; e < rows * (TW / XO); e += NTF) {
    const int r = e % rows, k = e / rows * XO;
    float a[XO];
    line_sums<XO, 1>(taps, in + r * pitch + k, a);
#pragma unroll
    for (int o = 0; o < XO; ++o) mid[r * MP + k + o] = a[o];
  }
  __syncthreads();
  constexpr int RY = TH / (NTF / TW);  // rows per thread
  const int tx = threadIdx.x % TW, ry = threadIdx.x / TW * RY;
  float a[RY];
  line_sums<RY, MP>(taps, mid + ry * MP + tx, a);
#pragma unroll
  for (int o = 0; o < RY; ++o) {
    const int h = h0 + ry + o, w = w0 + tx;
    if (h < H && w < W) store(h, w, a[o]);
  }
}

// filtered = filter(rho), eps = lo + span * project(filtered)
__global__ void __launch_bounds__(NTF)
    k_density_fwd(const float* __restrict__ rho, int nl, int H, int W, int kind, float beta,
                  float eta, float den, float off, float lo, float span,
                  float* filtered, float* eps,  // (may be one buffer: eps is what stays)
                  const __grid_constant__ Taps taps) {
  const int nx = (W + TW - 1) / TW;
  const int h0 = blockIdx.x / nx * TH, w0 = blockIdx.x % nx * TW;
  for (int l = blockIdx.y; l < nl; l += gridDim.y) {
    const long long base = (long long)l * H * W;
    filter_tile(
        taps, H, W, h0, w0,
        [&](int h, int w) { return rho[base + (long long)h * W + w]; },
        [&](int h, int w, float v) {
          const long long o = base + (long long)h * W + w;
          filtered[o] = v;
          eps[o] = lo + span * project(v, kind, beta, eta, den, off);
        });
    __syncthreads();
  }
}

// d rho = filter(d eps * span * project'(filtered)) (the x and y passes commute
// with their transposes)
__global__ void __launch_bounds__(NTF)
    k_density_bwd(const float* __restrict__ filtered, const float* __restrict__ deps, int nl,
                  int H, int W, int kind, float beta, float eta, float den, float span,
                  float* __restrict__ drho, const __grid_constant__ Taps taps) {
  const int nx = (W + TW - 1) / TW;
  const int h0 = blockIdx.x / nx * TH, w0 = blockIdx.x % nx * TW;
  for (int l = blockIdx.y; l < nl; l += gridDim.y) {
    const long long base = (long long)l * H * W;
    filter_tile(
        taps, H, W, h0, w0,
        [&](int h, int w) {
          const long long o = base + (long long)h * W + w;
          return deps[o] * span * project_grad(filtered[o], kind, beta, eta, den);
        },
        [&](int h, int w, float v) { drho[base + (long long)h * W + w] = v; });
    __syncthreads();
  }
}

// 3x3 pool per layer; arg = flat index of the selected input (first extremum
// in row-major window order, as max_pool2d keeps the first maximum)
// A thread takes four rows of a column and loads the six rows of three cells they
// see at once, from clamped positions: a clamped cell repeats one of the same
// window without changing which one is its first extremum.  (Loads behind the
// tests of the border came one after another, and a cell's indices through 64-bit
// divisions: 40 x 256 x 256 on B200 49 -> 18 us, backward 37 -> 18 us.)
constexpr int MR = 4;

__global__ void __launch_bounds__(256)
    k_morph3(const float* __restrict__ x, int nl, int H, int W, int dilate, float* __restrict__ y,
             int* __restrict__ arg) {
  const int nx = (W + 31) / 32;
  const int w = blockIdx.x % nx * 32 + (threadIdx.x & 31);
  const int h0 = (blockIdx.x / nx * 8 + threadIdx.x / 32) * MR;
  if (w >= W || h0 >= H) return;
  const int ww[3] = {max(w - 1, 0), w, min(w + 1, W - 1)};
  int row[MR + 2];
#pragma unroll
  for (int r = 0; r < MR + 2; ++r) row[r] = min(max(h0 + r - 1, 0), H - 1) * W;
  for (int l = blockIdx.y; l < nl; l += gridDim.y) {
    const long long base = (long long)l * H * W;
    const float* xl = x + base;
    float v[MR + 2][3];
#pragma unroll
    for (int r = 0; r < MR + 2; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) v[r][k] = __ldg(xl + row[r] + ww[k]);
#pragma unroll
    for (int o = 0; o < MR; ++o) {
      float best = v[o][0];
      int bi = row[o] + ww[0];
#pragma unroll
      for (int e = 1; e < 9; ++e) {
        const float u = v[o + e / 3][e % 3];
        const bool better = dilate ? u > best : u < best;
        best = better ? u : best;
        bi = better ? row[o + e / 3] + ww[e % 3] : bi;
      }
      if (h0 + o < H) {
        const long long i = base + (long long)row[o + 1] + w;
        y[i] = best;
        arg[i] = bi;  // index inside the layer
      }
    }
  }
}

// dx[j] = sum of dy[i] over the windows i around j that selected j
__global__ void __launch_bounds__(256)
    k_morph3_bwd(const float* __restrict__ dy, const int* __restrict__ arg, int nl, int H, int W,
                 float* __restrict__ dx) {
  const int nx = (W + 31) / 32;
  const int w = blockIdx.x % nx * 32 + (threadIdx.x & 31);
  const int h0 = (blockIdx.x / nx * 8 + threadIdx.x / 32) * MR;
  if (w >= W || h0 >= H) return;
  const int ww[3] = {max(w - 1, 0), w, min(w + 1, W - 1)};
  const bool in_w[3] = {w > 0, true, w + 1 < W};
  int row[MR + 2];
  bool in_h[MR + 2];
#pragma unroll
  for (int r = 0; r < MR + 2; ++r) {
    const int h = h0 + r - 1;
    in_h[r] = h >= 0 && h < H;
    row[r] = min(max(h, 0), H - 1) * W;
  }
  for (int l = blockIdx.y; l < nl; l += gridDim.y) {
    const long long base = (long long)l * H * W;
    const float* dl = dy + base;
    const int* al = arg + base;
    float g[MR + 2][3];
    int a[MR + 2][3];
#pragma unroll
    for (int r = 0; r < MR + 2; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        a[r][k] = in_h[r] && in_w[k] ? __ldg(al + row[r] + ww[k]) : -1;
        g[r][k] = __ldg(dl + row[r] + ww[k]);
      }
#pragma unroll
    for (int o = 0; o < MR; ++o) {
      if (h0 + o >= H) break;
      const int j = row[o + 1] + w;
      float sum = 0.0f;
#pragma unroll
      for (int e = 0; e < 9; ++e)
        if (a[o + e / 3][e % 3] == j) sum += g[o + e / 3][e % 3];
      dx[base + j] = sum;
    }
  }
}

// x: the tiles of a layer, row by row (the only grid axis without a 65535 limit);
// y: layers
dim3 tiles(int H, int W, int nl, int th, int tw) {
  const long long n = ((long long)W + tw - 1) / tw * (((long long)H + th - 1) / th);
  return dim3((unsigned)n, nl < 65535 ? nl : 65535);
}

// the reference smooth_filter's 1-D taps for `radius`
int make_taps(float radius, Taps* t) {
  if (!(radius >= 0.0f)) return DN_EINVAL;
  int k = (int)(2.0f * radius + 1.0f);
  if (k % 2 == 0) k += 1;
  if (k > MAX_TAPS) return DN_EUNSUPPORTED;
  const double sigma = radius / 2.0;
  double sum = 0.0, v[MAX_TAPS];
  for (int i = 0; i < k; ++i) {
    const double x = i - k / 2;
    v[i] = exp(-(x * x) / (2.0 * sigma * sigma + 1e-12));
    sum += v[i];
  }
  for (int i = 0; i < k; ++i) t->t[i] = (float)(v[i] / sum);
  t->n = k;
  return DN_OK;
}

int check(const dn_density* d) {
  if (!d || d->n_layers < 1 || d->H < 1 || d->W < 1) return DN_EINVAL;
  if (d->kind != DN_PROJ_SIGMOID && d->kind != DN_PROJ_TANH && d->kind != DN_PROJ_NONE)
    return DN_EINVAL;
  if (!(d->beta > 0.0f) || !(d->eps_hi >= d->eps_lo)) return DN_EINVAL;
  if (d->kind == DN_PROJ_TANH && !(d->eta > 0.0f && d->eta < 1.0f)) return DN_EINVAL;
  return DN_OK;
}

void proj_consts(const dn_density* d, float* den, float* off) {
  *off = tanhf(d->beta * d->eta);
  *den = *off + tanhf(d->beta * (1.0f - d->eta));
}

// A tile reads its neighbours' cells, so an input that shares memory with an output is
// read from a copy in `work`.
int apart(const dn_density* d, const float** in, const float* out, float* work, cudaStream_t s) {
  const size_t bytes = (size_t)d->n_layers * d->H * d->W * sizeof(float);
  const uintptr_t a = reinterpret_cast<uintptr_t>(*in), b = reinterpret_cast<uintptr_t>(out);
  if (a + bytes <= b || b + bytes <= a) return DN_OK;
  DN_CUDA_CHECK(cudaMemcpyAsync(work, *in, bytes, cudaMemcpyDeviceToDevice, s));
  *in = work;
  return DN_OK;
}

// taps, and the shared memory of a tile with their border
template <typename K>
int prepare(const dn_density* d, K kern, Taps* t, size_t* smem) {
  const int rc = make_taps(d->radius, t);
  if (rc != DN_OK) return rc;
  *smem = tile_bytes(t->n);
  if (*smem > 48 * 1024)
    DN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)*smem));
  return DN_OK;
}

}  // namespace ds
}  // namespace dn

using namespace dn::ds;

extern "C" int32_t dn_density_forward(const dn_density* d, const float* rho, float* work,
                                      float* filtered, float* eps, void* stream) {
  int rc = check(d);
  if (rc != DN_OK) return rc;
  if (!rho || !work || !filtered || !eps) return DN_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Taps t;
  size_t smem;
  if ((rc = prepare(d, k_density_fwd, &t, &smem)) != DN_OK) return rc;
  if ((rc = apart(d, &rho, filtered, work, s)) != DN_OK) return rc;
  if ((rc = apart(d, &rho, eps, work, s)) != DN_OK) return rc;
  float den, off;
  proj_consts(d, &den, &off);
  k_density_fwd<<<tiles(d->H, d->W, d->n_layers, TH, TW), NTF, smem, s>>>(
      rho, d->n_layers, d->H, d->W, d->kind, d->beta, d->eta, den, off, d->eps_lo,
      d->eps_hi - d->eps_lo, filtered, eps, t);
  DN_CUDA_CHECK(cudaGetLastError());
  return DN_OK;
}

extern "C" int32_t dn_density_backward(const dn_density* d, const float* filtered,
                                       const float* deps, float* work, float* drho,
                                       void* stream) {
  int rc = check(d);
  if (rc != DN_OK) return rc;
  if (!filtered || !deps || !work || !drho) return DN_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float den, off;
  proj_consts(d, &den, &off);
  Taps t;
  size_t smem;
  if ((rc = prepare(d, k_density_bwd, &t, &smem)) != DN_OK) return rc;
  if ((rc = apart(d, &filtered, drho, work, s)) != DN_OK) return rc;
  if ((rc = apart(d, &deps, drho, work, s)) != DN_OK) return rc;
  k_density_bwd<<<tiles(d->H, d->W, d->n_layers, TH, TW), NTF, smem, s>>>(
      filtered, deps, d->n_layers, d->H, d->W, d->kind, d->beta, d->eta, den,
      d->eps_hi - d->eps_lo, drho, t);
  DN_CUDA_CHECK(cudaGetLastError());
  return DN_OK;
}

extern "C" int32_t dn_morph3(const float* x, int32_t n_layers, int32_t H, int32_t W,
                             int32_t dilate, float* y, int32_t* arg, void* stream) {
  if (!x || !y || !arg || n_layers < 1 || H < 1 || W < 1) return DN_EINVAL;
  if ((long long)H * W > 0x7fffffffLL) return DN_EUNSUPPORTED;
  k_morph3<<<tiles(H, W, n_layers, 8 * MR, 32), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      x, n_layers, H, W, dilate != 0, y, arg);
  DN_CUDA_CHECK(cudaGetLastError());
  return DN_OK;
}

extern "C" int32_t dn_morph3_backward(const float* dy, const int32_t* arg, int32_t n_layers,
                                      int32_t H, int32_t W, float* dx, void* stream) {
  if (!dy || !arg || !dx || n_layers < 1 || H < 1 || W < 1) return DN_EINVAL;
  if ((long long)H * W > 0x7fffffffLL) return DN_EUNSUPPORTED;  // as the forward
  k_morph3_bwd<<<tiles(H, W, n_layers, 8 * MR, 32), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      dy, arg, n_layers, H, W, dx);
  DN_CUDA_CHECK(cudaGetLastError());
  return DN_OK;
}
