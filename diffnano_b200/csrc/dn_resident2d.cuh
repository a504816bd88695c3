// Whole 2-D runs with the grid held on the chip: the step of dn_fdtd2d.cu on
// fields that stay in registers from the first step to the last.
//
// A grid is cut into bands of rows, one CTA each; inside a band a warp owns a
// block of R rows x 32*VEC columns (VEC = 16 bytes / element) whose three
// fields and dt/eps live in its registers.  Per step a warp needs the injected
// field (Ez / Hz) of the one row above, the one row below and the one column
// left and right of its block, and nothing else: the second field of the row
// above (TM: Hy) or below (TE: Ey) its block, and the one of the column left
// (TM: Hx) or right (TE: Ex), it keeps as copies that it updates itself with
// the owner's arithmetic.  Warps of a CTA exchange rows and columns through
// shared memory (two buffers by step parity, one CTA barrier per step); bands
// exchange one row per step and direction through mailboxes of 64-bit words
// (value | step tag), written and polled with single 64-bit accesses, so a row
// arrives with its flag and no barrier spans the CTAs.  Two places for the
// mailboxes: the neighbour CTA's shared memory, when the bands of a grid form
// one thread-block cluster, and global memory (L2), when a cooperative launch
// keeps all of them resident.
//
// A mailbox has two slots (step parity).  A band writes slot n & 1 again at
// step n + 2, for which it needed its neighbour's row of step n + 1, which the
// neighbour's same warp sent after it had read the row of step n: no
// acknowledgement is needed.  Every wait is bounded; a wait that gives up
// records DN_ETIMEOUT, and the CTA leaves behind its next barrier.
//
// What bounds it: no field crosses L2 inside the run, so a step costs the chain
// row received -> block updated -> row sent -> received by the neighbour, and
// the issue slots of the busiest warp.  Measured on B200, FP32 TM, us per step
// (before: the cluster kernel of dn_batch2d.cu, or one launch per step): 100^2
// 0.42 (2.17), 256^2 with a monitor row 0.89 (3.74), 512^2 0.95 (7.0), 1024^2
// with a monitor row 2.2 (10.4).  What was learned on the way: FP64 monitor
// sums inside the march cost every step 0.35 - 0.9 us (all bands wait for the
// band that has them), stored samples 0.02 - 0.15; 255 registers and 8 rows per
// warp (too few warps) 2.4 where 4 rows and 16 warps take 1.8.
#pragma once

#include <cuda_runtime.h>

#include "dn_host.cuh"
#include "dn_strip.cuh"

namespace dn {
namespace res {

enum { MAIL_CLUSTER = 0, MAIL_GLOBAL = 1 };

// Polls of one wait on a global mailbox, a round trip to L2 (0.3 us and more) each.
// All bands of a lone grid start together; in a batch a band that starts early waits
// for a neighbour whose CTA still runs earlier grids, for as long as the whole launch
// may take: POLLS_PER_STEP for each step of the longest list (a step takes up to
// 4 us) come on top.
constexpr unsigned SPIN_LIMIT = 1u << 22;
constexpr unsigned POLLS_PER_STEP = 64;
inline unsigned polls_of(double steps) {
  const double p = SPIN_LIMIT + POLLS_PER_STEP * steps;
  return p < 4e9 ? (unsigned)p : 4000000000u;
}

constexpr int MAX_WARPS = 16;  // warps per CTA: 128 registers each
constexpr int ROW_WORDS = 4 * 32;  // 64-bit mailbox words per strip and row

// One grid's run, as the kernel sees it.  Fields in the order TM (Ez, Hx, Hy)
// / TE (Hz, Ex, Ey).
template <typename T>
struct Job {
  int H, W;
  long long py;
  const T* in[3];
  T* out[3];
  const T* ce;
  const double* b[2];  // rows, columns
  const double* c[2];
  double dt, dl;
  int src;  // source on the injected field?
  int src_lo[2], src_hi[2];
  const T* wave;
  int t0, nsteps;
  T* curl[2];  // REC: TM one array, TE two
  long long curl_stride;
};

// One grid's reverse sweep (TM): adjoint fields (lambda_Ez, lambda_Hx,
// lambda_Hy); reverse step n = 0 .. nsteps-1 reads the curl record at curl - n *
// curl_stride and adds lambda_Ez . curl to grad.
template <typename T>
struct AdjJob {
  int H, W;
  long long py;
  const T* in[3];
  T* out[3];
  const T* ce;
  const double* b[2];
  const double* c[2];
  double dt, dl;
  int nsteps;
  const T* curl;
  long long curl_stride;
  double* grad;
};

// A box whose values of one component are stored after every step (the reverse
// sweep reads them instead: what is added to lambda_Ez after reverse step n):
// buf[n * step_stride + cell], cells row-major inside the box.
template <typename T>
struct Samples {
  int lo[2], hi[2];  // rows, columns
  int comp;          // 0: injected field, 1 / 2: the second / third field
  int vec;           // a lane's columns are inside or outside as a whole, 16-byte aligned
  T* buf;
  long long step_stride;
};
constexpr int MAX_SAMPLES = DN_MAX_MONITORS + 1;  // the monitors and the probe
template <typename T>
struct SampleSet {
  Samples<T> s[MAX_SAMPLES];
  int n;
};

// work split of one grid: bands of groups * R rows, strips * groups warps
struct Split {
  int R;  // rows per warp
  int strips, groups, bands;
  int cluster;  // bands exchange rows through shared memory (else through global memory)
};

// Many grids in one cooperative launch: every CTA takes the (grid, band) pairs of
// its list in order.  Bands of a grid wait for one another, so all lists keep one
// order of the grids: the bands of the first unfinished grid are always next on
// their CTAs.
struct ListGrid {
  int strips, groups, bands;
  long long mail;    // 64-bit words from the start of the mailboxes
  long long sample;  // bytes from the start of the samples
  long long stride;  // elements between two steps' samples
};
struct ListJob {
  int grid, band;
};
struct List {
  const dn_batch2d_inst* inst;
  const ListGrid* grids;
  const ListJob* jobs;
  const int* start;  // per CTA, its first job (and one past the last CTA's last)
  uint64_t* mail;
  unsigned char* samples;
  unsigned polls;  // bound of one wait
};

// forward (adjoint = false) or reverse sweep of TM grids, R rows per warp
template <typename T>
int run_resident_list(const List& L, bool adjoint, bool record, int R, int n_cta, int* status,
                      cudaStream_t s);

// the run itself (dn_resident2d_fwd.cuh), one instantiation per source file
template <typename T>
int run_resident_adjoint(const AdjJob<T>& J, const SampleSet<T>& adds, const Split& S,
                         uint64_t* mail, int* status, cudaStream_t s);
template <typename T, int POL>
int run_resident(const Job<T>& J, const SampleSet<T>& smps, const Split& S, uint64_t* mail,
                 int* status, cudaStream_t s);

}  // namespace res
}  // namespace dn
