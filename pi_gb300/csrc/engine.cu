// pimul engine: Goldilocks NTT big-integer multiply on one GB300 (sm_103a).
//
// Host orchestration + kernels for the plain drop-in multiply
// (include/pimul.h: pimul_mul, pimul_mul_device).  The algorithm follows the
// reference's mul_mag_ntt (crates/bignum/src/ntt.rs:806-865): pack limbs into
// 16-bit coefficients, forward-transform both operands, multiply pointwise,
// inverse-transform, carry-normalise back to limbs.  Results are exact, so
// every product equals the reference's bit for bit.
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <thread>
#include <unordered_map>
#include <atomic>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "gl.cuh"
#include "ntt_kernels.cuh"
#include "../../include/pimul.h"
#include "hostcopy.h"
#include "splitmerge.h"

namespace pimul {

// ------------------------------------------------------------------ errors
static thread_local std::string t_err;

static int fail(int code, const std::string& msg) {
  t_err = msg;
  return code;
}

#define CU(call)                                                                   \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess)                                                         \
      return fail(e_ == cudaErrorMemoryAllocation ? PIMUL_ENOMEM : PIMUL_ECUDA,    \
                  std::string(#call) + ": " + cudaGetErrorString(e_));             \
  } while (0)

// ------------------------------------------------------------------ launch stats
// Launch counters per kernel class, and optional CUDA-event timing of every
// launch on the stream it runs on (pimul_stats_enable).
enum KClass { K_PACK, K_PASS_FWD, K_PASS_INV, K_POINTWISE, K_CARRY, K_SMALL, K_NCLASS };
static const char* k_names[K_NCLASS] = {"pack", "pass_fwd", "pass_inv", "pointwise", "carry", "small"};
static std::atomic<uint64_t> g_launch[K_NCLASS];
static std::atomic<int> g_timing{0};
struct Pending {
  int cls;
  cudaEvent_t a, b;
};
static std::mutex g_tmu;
static std::vector<Pending> g_pending;
static std::vector<cudaEvent_t> g_evpool;
static double g_ms[K_NCLASS];
static uint64_t g_timed[K_NCLASS];

static cudaEvent_t ev_get() {
  cudaEvent_t e = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_tmu);
    if (!g_evpool.empty()) {
      e = g_evpool.back();
      g_evpool.pop_back();
    }
  }
  if (!e) cudaEventCreate(&e);
  return e;
}

struct KTimer {
  int cls;
  cudaStream_t st;
  cudaEvent_t a = nullptr;
  KTimer(int c, cudaStream_t s, bool on = true) : cls(c), st(s) {
    if (!on) return;
    g_launch[c].fetch_add(1, std::memory_order_relaxed);
    if (g_timing.load(std::memory_order_relaxed)) {
      a = ev_get();
      cudaEventRecord(a, st);
    }
  }
  ~KTimer() {
    if (a) {
      cudaEvent_t b = ev_get();
      cudaEventRecord(b, st);
      std::lock_guard<std::mutex> lk(g_tmu);
      g_pending.push_back(Pending{cls, a, b});
    }
  }
};

static void stats_drain() {
  std::vector<Pending> p;
  {
    std::lock_guard<std::mutex> lk(g_tmu);
    p.swap(g_pending);
  }
  for (auto& x : p) {
    cudaEventSynchronize(x.b);
    float ms = 0;
    cudaEventElapsedTime(&ms, x.a, x.b);
    std::lock_guard<std::mutex> lk(g_tmu);
    g_ms[x.cls] += ms;
    g_timed[x.cls] += 1;
    g_evpool.push_back(x.a);
    g_evpool.push_back(x.b);
  }
}

// ------------------------------------------------------------------ host field
namespace hf {
constexpr uint64_t P = gl::P;
static uint64_t mul(uint64_t a, uint64_t b) {
  unsigned __int128 x = (unsigned __int128)a * b;
  uint64_t lo = (uint64_t)x, hi = (uint64_t)(x >> 64);
  uint64_t x2 = hi & 0xFFFFFFFFull, x3 = hi >> 32;
  uint64_t t = lo - x3;
  if (lo < x3) t -= gl::EPS;
  uint64_t u = (x2 << 32) - x2;
  uint64_t r = t + u;
  if (r < u) r += gl::EPS;
  return r >= P ? r - P : r;
}
static uint64_t pow(uint64_t b, uint64_t e) {
  uint64_t a = 1;
  while (e) {
    if (e & 1) a = mul(a, b);
    e >>= 1;
    b = mul(b, b);
  }
  return a;
}
}  // namespace hf

// rho: primitive 2^32-th root of unity with rho^(2^26) = 8.  Powers of the
// generator 7 (crates/bignum/src/ntt.rs:172) give the 2^32-th roots; the
// odd power t is picked so that the 64th root of unity is exactly 2^3.
static uint64_t find_rho() {
  uint64_t w0 = hf::pow(7, (hf::P - 1) >> 32);
  for (uint64_t t = 1; t < 64; t += 2) {
    uint64_t r = hf::pow(w0, t);
    if (hf::pow(r, 1ull << 26) == 8) return r;
  }
  return 0;
}

// ------------------------------------------------------------------ kernels
// Geometry of the HBM passes (ntt_kernels.cuh): CTAs of 128 threads,
//   first and middle passes: 2^R rows x 8 or 16 columns of one block
//   last pass (S = 1):       four warps, each 32 2^B1 contiguous words
// First-pass rows hold at least 8 consecutive coefficients, one carry window.
// Four CTAs per SM leave 128 registers for a thread's radix-32 round (113 to
// 126 used); 96 (five CTAs) spill, 168 (three) run no faster.  The shorter
// rounds do with less: a 2^24-point product of R = 8 passes takes 667 us at
// five CTAs, 684 at four, 672 at seven; R = 6, 7 differ by under 1 % from
// four to nine.
constexpr int pass_min_ctas(int r) { return r == 9 ? 4 : r == 8 ? 5 : 6; }

// One product of a batch (or the only product of a plain call): operands,
// output and its scratch.  Kernels take `const Job* jobs, Job one`: with a
// device array, blockIdx.y selects the product; with jobs == nullptr the
// by-value `one` is used (no descriptor upload for single products).
struct Job {
  const uint64_t* a;
  const uint64_t* b;
  uint64_t* out;
  uint64_t* A;  // N words: a's spectrum (and the product for a square)
  uint64_t* B;  // N words: b's spectrum and the product (unused for a square)
  uint64_t* H;  // high parts of the carry windows
  uint64_t* W;  // their low parts, two limbs each
  uint32_t* state;  // carry states of the window chunks
  uint64_t la, lb;
  const uint64_t* X;  // spectra of a second product added to the pointwise one (a sum of two products), or null
  const uint64_t* Y;
  uint64_t nout;      // output limbs (0: la + lb); with JF_COEFF, output coefficients
  uint32_t flags;     // JF_* roles inside a batch (0: a plain product)
  // A wrapped product runs a cyclic transform of length N shorter than its
  // wrap + N coefficients: coefficient N + i (i < wrap) lands on i.  low
  // holds the exact coefficients 0 .. wrap - 1 (from a short product of the
  // operands' low limbs), so that coefficient i is low[i] and N + i the
  // cyclic value minus low[i].
  const uint64_t* low;
  uint64_t wrap;
  // A segment of a product of a long a by a short b: its transform covers the
  // coefficients c0 .. c0 + N - 1 of a (zero outside a), and its cyclic values
  // from window wlo on are the product's windows w + woff.
  int64_t c0;
  int64_t woff;
  uint32_t wlo;
  uint32_t segments;  // by value: blockIdx.y selects one of these, each segv coefficients on
  uint64_t segv;
};

// Carry windows of 8 coefficients (2 limbs); see the carry normalisation below.
constexpr int WIN_COEFFS = 8;
constexpr int CARRY_THREADS = 256;  // windows per CTA

// Windows of an output of nout limbs (4 nout - 1 coefficients).
__host__ __device__ __forceinline__ uint64_t n_windows_out(uint64_t nout) {
  return (4 * nout - 1 + WIN_COEFFS - 1) / WIN_COEFFS;
}
__host__ __device__ __forceinline__ uint64_t n_windows(uint64_t la, uint64_t lb) { return n_windows_out(la + lb); }
__host__ __device__ __forceinline__ uint64_t n_chunks(uint64_t nwin) {
  return (nwin + CARRY_THREADS - 1) / CARRY_THREADS;
}
// Roles of a product inside a batch.  A spectrum shared by several products
// with the same operand b is computed once, by its owner; the others point B
// at it (JF_B_SHARED) and skip b's passes.  An addend (JF_ADDEND) produces no
// output: the job it is added to reads its spectra as X and Y.  Every product
// is formed in A.
constexpr uint32_t JF_B_SHARED = 1;
constexpr uint32_t JF_ADDEND = 4;
// The product's canonical coefficients 0 .. nout - 1 go to out (no carry):
// the low part of a wrapped product.
constexpr uint32_t JF_COEFF = 8;
// A segment after a product's first one: its windows are carried by that one.
constexpr uint32_t JF_SEGMENT = 16;

// Every kernel of the pipeline starts with these two (see launch_pdl): the next
// kernel on the stream may be scheduled as this one's CTAs leave, and nothing
// is read or written before the kernels in front are done.  What an earlier
// kernel may have written (operands, spectra, windows) is read with plain
// loads through pointers that promise nothing: the read-only path (__ldg, or
// const __restrict__) wants words that stay the same from the kernel's start
// on, which lies before the wait, and a load from it is not tied to the wait.
// The root and twiddle tables, finished before any launch that reads them, keep it.
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Segment s of a segmented product whose first segment is J.
__host__ __device__ __forceinline__ void to_segment(Job& J, uint32_t s, int L) {
  J.A += (uint64_t)s << L;
  J.c0 = (int64_t)(s * J.segv) - 8 * (int64_t)J.wlo;
  J.woff = (int64_t)(s * (J.segv / 8)) - (int64_t)J.wlo;
  if (s) J.flags |= JF_SEGMENT | JF_B_SHARED;
}

__device__ __forceinline__ Job job_of(const Job* jobs, const Job& one, int L) {
  pdl_wait();
  if (jobs) return jobs[blockIdx.y];
  Job J = one;
  if (J.segments) to_segment(J, blockIdx.y, L);
  return J;
}
__host__ __device__ __forceinline__ bool is_square(const Job& J) { return J.a == J.b && J.la == J.lb; }
// b's own passes are skipped for a square and for a borrowed spectrum.
__device__ __forceinline__ bool skips_b(const Job& J) { return is_square(J) || (J.flags & JF_B_SHARED); }
__host__ __device__ __forceinline__ uint64_t job_nout(const Job& J) { return J.nout ? J.nout : J.la + J.lb; }

// Forward pass 0 with the limb -> 16-bit coefficient split fused in
// (crates/bignum/src/ntt.rs:640-665): element (i, j) of the tile is
// coefficient n = i * 2^S + j0 + j, the n-th 16-bit word of the operand;
// words past its end are zero (the reference's zero tail).  Operand
// w0 + blockIdx.z (0: a, 1: b; skips_b drops b).
// twf: the pass's twiddle table (tw_first), or null to compute the twiddles.
template <int R>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas(R)) k_fwd_first(const Job* jobs, Job one, int w0, int L, Roots RT,
                                                                           const uint64_t* __restrict__ twf) {
  using G = ColGeom<R>;
  constexpr int B1 = G::B1, B2 = G::B2, T = G::T;
  const Job J = job_of(jobs, one, L);
  const int which = w0 + (int)blockIdx.z;
  if (which == 1 && skips_b(J)) return;
  const uint16_t* coef = reinterpret_cast<const uint16_t*>(which ? J.b : J.a);
  const int64_t c0 = which ? 0 : J.c0, nc = (int64_t)(4 * (which ? J.lb : J.la));
  uint64_t* __restrict__ data = which ? J.B : J.A;
  extern __shared__ uint64_t sm[];
  const int tid = threadIdx.x;
  const int S = L - R;
  const uint64_t j0 = (uint64_t)blockIdx.x << T;
  {
    const int64_t n0 = c0 + (int64_t)(((uint64_t)(tid >> T) << S) + j0 + (tid & G::TM));
    const uint64_t step = 1ull << (S + B2);
    // inputs ml <= m < mc exist (ml > 0: a first segment starts before a does)
    const uint32_t ml = n0 < 0 ? (uint32_t)((uint64_t)(-n0 + (int64_t)step - 1) >> (S + B2)) : 0;
    const uint32_t mc = n0 < nc ? (uint32_t)((uint64_t)(nc - n0 + (int64_t)step - 1) >> (S + B2)) - ml : 0;
    const uint16_t* cn = coef + n0;
    uint64_t v[1 << B1];
    gl::Lz x[1 << B1];
    bool done = false;
    if constexpr (B1 > 3) {
      // an operand of at most N/8 limbs leaves the upper half of the rows zero
      // (coefficients N/2 and up): those inputs are neither read nor added
      if (nc - c0 <= (int64_t)(1ull << (L - 1))) {
#pragma unroll
        for (int m = 0; m < (1 << (B1 - 1)); m++) x[m] = gl::Lz{m - ml < mc ? (uint32_t)cn[m * step] : 0u, 0u, 0};
        x[0] = gl::lz_bias(x[0]);
        dft_lz<B1, false, true>(x, v);
        done = true;
      }
    }
    if (!done) {
#pragma unroll
      for (int m = 0; m < (1 << B1); m++) x[m] = gl::Lz{m - ml < mc ? (uint32_t)cn[m * step] : 0u, 0u, 0};
      x[0] = gl::lz_bias(x[0]);
      dft_lz<B1, false>(x, v);
    }
#pragma unroll
    for (int k = 0; k < (1 << B1); k++) sm[k * G::KS + tid] = v[k];
  }
  // Without a table, w^(f (j0 + j)) = w^(f j0) w^(f j) for a long transform: the
  // first factors of the tile's 2^R frequencies are staged, the second
  // (f j < 4096) come from the L1-resident near table.
  uint64_t* tw = sm + G::XWORDS;
  const bool staged = !twf && L > LVL_MAX;
  if (staged)
    for (uint32_t f = tid; f < (1u << R); f += PASS_THREADS) tw[f] = root_pow32(RT, L, f * (uint32_t)j0, false);
  __syncthreads();
  const uint64_t* __restrict__ rt = RT.rt + rt_offset(R, false);
#pragma unroll 1
  for (int it = 0; it < G::ITERS2; it++) {
    const uint32_t w = it * PASS_THREADS + tid, j = w & G::TM, k1 = w >> T;
    uint64_t v[1 << B2];
    pass_fwd2<R>(sm + k1 * G::KS + j, 1u << T, rt, k1, v);
    const uint64_t at = ((uint64_t)(k1 << B2) << S) + j0 + j;
    if (twf) {
      // twiddles laid out like the data: one coalesced load each
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) data[at + ((uint64_t)k << S)] = gl::mul(v[k], __ldg(twf + at + ((uint64_t)k << S)));
    } else if (staged) {
      const uint64_t* __restrict__ nt = near_table(RT, L, false);
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) {
        const uint32_t f = k1 + (k << B1);
        data[at + ((uint64_t)k << S)] = gl::mul(v[k], gl::mul(tw[f], __ldg(nt + f * j)));
      }
    } else {
#pragma unroll
      for (int k = 0; k < (1 << B2); k++)
        data[at + ((uint64_t)k << S)] = gl::mul(v[k], root_pow32(RT, L, (k1 + (k << B1)) * (uint32_t)(j0 + j), false));
    }
  }
}

// Middle column pass of stride 2^S; forward pass twiddles w_M^(f*j) after the
// rounds (operand w0 + blockIdx.z), inverse ones before (on the product).
// twm: the pass's twiddle table (tw_mid), or null to compute the twiddles.
template <int R, bool FWD>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas(R)) k_col_mid(const Job* jobs, Job one, int w0, int L, int S,
                                                                         Roots RT, const uint64_t* __restrict__ twm) {
  using G = ColGeom<R>;
  constexpr int B1 = G::B1, B2 = G::B2, T = G::T;
  const Job J = job_of(jobs, one, L);
  const int which = w0 + (int)blockIdx.z;
  if (FWD && which == 1 && skips_b(J)) return;
  if (!FWD && (J.flags & JF_ADDEND)) return;
  extern __shared__ uint64_t sm[];
  const int tid = threadIdx.x;
  const int mlog = R + S;
  const uint64_t j0 = (uint64_t)(blockIdx.x & ((1u << (S - T)) - 1)) << T;
  const uint64_t b0 = (uint64_t)blockIdx.x >> (S - T);
  uint64_t* __restrict__ data = (FWD && which ? J.B : J.A) + (b0 << mlog) + j0;
  // element (m, column) of this thread in the round that has m fixed
  const uint64_t mat = ((uint64_t)(tid >> T) << S) + (tid & G::TM);
  if constexpr (FWD) {
    {
      uint64_t v[1 << B1];
      gl::Lz x[1 << B1];
#pragma unroll
      for (int m = 0; m < (1 << B1); m++) v[m] = data[mat + ((uint64_t)m << (S + B2))];
#pragma unroll
      for (int m = 0; m < (1 << B1); m++) x[m] = gl::lz(v[m]);
      x[0] = gl::lz_bias(x[0]);
      dft_lz<B1, false>(x, v);
#pragma unroll
      for (int k = 0; k < (1 << B1); k++) sm[k * G::KS + tid] = v[k];
    }
    __syncthreads();
    const uint64_t* __restrict__ rt = RT.rt + rt_offset(R, false);
#pragma unroll 1
    for (int it = 0; it < G::ITERS2; it++) {
      const uint32_t w = it * PASS_THREADS + tid, j = w & G::TM, k1 = w >> T;
      uint64_t v[1 << B2];
      pass_fwd2<R>(sm + k1 * G::KS + j, 1u << T, rt, k1, v);
      const uint64_t at = ((uint64_t)(k1 << B2) << S) + j;
      if (twm) {
#pragma unroll
        for (int k = 0; k < (1 << B2); k++)
          data[at + ((uint64_t)k << S)] = gl::mul(v[k], __ldg(twm + j0 + at + ((uint64_t)k << S)));
      } else {
#pragma unroll
        for (int k = 0; k < (1 << B2); k++)
          data[at + ((uint64_t)k << S)] = gl::mul(v[k], root_pow32(RT, mlog, (k1 + (k << B1)) * (uint32_t)(j0 + j), false));
      }
    }
  } else {
#pragma unroll 1
    for (int it = 0; it < G::ITERS2; it++) {
      const uint32_t w = it * PASS_THREADS + tid, j = w & G::TM, k1 = w >> T;
      const uint64_t at = ((uint64_t)(k1 << B2) << S) + j;
      uint64_t v[1 << B2];
      gl::Lz x[1 << B2];
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) v[k] = data[at + ((uint64_t)k << S)];
      if (twm) {
#pragma unroll
        for (int k = 0; k < (1 << B2); k++) x[k] = gl::lz_mul(v[k], __ldg(twm + j0 + at + ((uint64_t)k << S)));
      } else {
#pragma unroll
        for (int k = 0; k < (1 << B2); k++)
          x[k] = gl::lz_mul(v[k], root_pow32(RT, mlog, (k1 + (k << B1)) * (uint32_t)(j0 + j), true));
      }
      x[0] = gl::lz_bias(x[0]);
      dft_lz<B2, true>(x, v);
#pragma unroll
      for (int m = 0; m < (1 << B2); m++) sm[k1 * G::KS + (m << T) + j] = v[m];
    }
    __syncthreads();
    uint64_t v[1 << B1];
    pass_inv2<R>(sm + tid, G::KS, RT.rt + rt_offset(R, true), tid >> T, v);
#pragma unroll
    for (int m = 0; m < (1 << B1); m++) data[mat + ((uint64_t)m << (S + B2))] = v[m];
  }
}

// Last forward pass (stride 1) of operand w0 + blockIdx.z.  Fused with the
// pointwise product and the first inverse pass it ran slower (2^25 points:
// 442 us for both operands' last passes and the inverse's first one, against
// 113 per operand and 150-170 here): four unrolled rounds overflow the
// instruction caches, and two tiles per CTA cost a CTA per SM.  A warp's 32 2^B1
// words hold whole blocks; it leaves its spectrum as rows of 32 words, one
// per (iteration, k2), the order in which the inverse's first round reads it.
template <int R>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas(R)) k_fwd_last(const Job* jobs, Job one, int w0, int L, Roots RT) {
  using G = RowGeom<R>;
  constexpr int B1 = G::B1, B2 = G::B2;
  const Job J = job_of(jobs, one, L);
  const int which = w0 + (int)blockIdx.z;
  if (which == 1 && skips_b(J)) return;
  extern __shared__ uint64_t sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* __restrict__ chunk = (which ? J.B : J.A) + ((uint64_t)blockIdx.x << G::TILE) + warp * G::WWORDS;
  uint64_t* sw = sm + warp * G::XWORDS;
  {
    const uint32_t m0 = lane & ((1u << B2) - 1), blk = lane >> B2;
    uint64_t v[1 << B1];
    gl::Lz x[1 << B1];
#pragma unroll
    for (int m = 0; m < (1 << B1); m++) v[m] = chunk[(blk << R) + (m << B2) + m0];
#pragma unroll
    for (int m = 0; m < (1 << B1); m++) x[m] = gl::lz(v[m]);
    x[0] = gl::lz_bias(x[0]);
    dft_lz<B1, false>(x, v);
    uint64_t* sx = sw + (blk << B1) * G::KS + blk * G::BPAD + m0;
#pragma unroll
    for (int k = 0; k < (1 << B1); k++) sx[k * G::KS] = v[k];
  }
  __syncwarp();
  const uint64_t* __restrict__ rt = RT.rt + rt_offset(R, false);
#pragma unroll 1
  for (int it = 0; it < G::ITERS2; it++) {
    const uint32_t idx = it * 32 + lane, k1 = idx & ((1u << B1) - 1), blk = idx >> B1;
    uint64_t v[1 << B2];
    pass_fwd2<R>(sw + idx * G::KS + blk * G::BPAD, 1, rt, k1, v);
#pragma unroll
    for (int k = 0; k < (1 << B2); k++) chunk[(((it << B2) + k) << 5) + lane] = v[k];
  }
}

// Pointwise product of the two spectra (plus X Y, a second product, for a sum),
// entering the first inverse pass as lazy products; the result overwrites A.
// (The inverse's 1/N, crates/bignum/src/ntt.rs:383-390 and 845-853, comes with
// its last pass's twiddles; a scaling here, though skipped where those have a
// table, cost 0.3 to 1.3 % of a whole product in instruction cache misses.)
// The second iteration's words are fetched into L2 while the first one runs: a
// 2^30-bit product 5420 -> 5377 us, shorter ones as before.
template <int R>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas(R)) k_inv_last(const Job* jobs, Job one, int L, Roots RT) {
  using G = RowGeom<R>;
  constexpr int B1 = G::B1, B2 = G::B2;
  const Job J = job_of(jobs, one, L);
  if (J.flags & JF_ADDEND) return;
  if (!(J.flags & (JF_COEFF | JF_SEGMENT))) {
    // no carry state published yet
    const uint64_t nchunk = n_chunks(n_windows_out(job_nout(J)));
    for (uint64_t t = (uint64_t)blockIdx.x * PASS_THREADS + threadIdx.x; t < nchunk; t += (uint64_t)gridDim.x * PASS_THREADS)
      J.state[t] = 0;
  }
  extern __shared__ uint64_t sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t off = ((uint64_t)blockIdx.x << G::TILE) + warp * G::WWORDS;
  const bool sq = is_square(J);
  uint64_t* __restrict__ chunk = J.A + off;
  const uint64_t* bspec = J.B + off;
  uint64_t* sw = sm + warp * G::XWORDS;
  constexpr uint32_t LINE = 16;  // words of 128 bytes
  for (uint32_t t = G::WWORDS / G::ITERS2 + LINE * lane; t < G::WWORDS; t += LINE * 32) {
    prefetch_l2(chunk + t);
    if (!sq) prefetch_l2(bspec + t);
  }
#pragma unroll 1
  for (int it = 0; it < G::ITERS2; it++) {
    const uint32_t idx = it * 32 + lane, blk = idx >> B1;
    const uint32_t at = (it << (B2 + 5)) + lane;
    uint64_t v[1 << B2], y[1 << B2];
    gl::Lz x[1 << B2];
#pragma unroll
    for (int k = 0; k < (1 << B2); k++) v[k] = chunk[at + (k << 5)];
    if (sq) {
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) y[k] = v[k];
    } else {
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) y[k] = bspec[at + (k << 5)];
    }
    if (J.X) {
      const uint64_t* X = J.X + off;
      const uint64_t* Y = J.Y + off;
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) x[k] = gl::lz(gl::add(gl::mul(v[k], y[k]), gl::mul(X[at + (k << 5)], Y[at + (k << 5)])));
    } else {
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) x[k] = gl::lz_mul(v[k], y[k]);
    }
    x[0] = gl::lz_bias(x[0]);
    dft_lz<B2, true>(x, v);
    uint64_t* sx = sw + idx * G::KS + blk * G::BPAD;
#pragma unroll
    for (int m = 0; m < (1 << B2); m++) sx[m] = v[m];
  }
  __syncwarp();
  const uint32_t m0 = lane & ((1u << B2) - 1), blk = lane >> B2;
  uint64_t v[1 << B1];
  pass_inv2<R>(sw + (blk << B1) * G::KS + blk * G::BPAD + m0, G::KS, RT.rt + rt_offset(R, true), m0, v);
#pragma unroll
  for (int m = 0; m < (1 << B1); m++) chunk[(blk << R) + (m << B2) + m0] = v[m];
}

// ---- carry normalisation (crates/bignum/src/ntt.rs:676-791) --------------
// Coefficients are grouped in windows of 8 (= 2 limbs).  Window w has value
// V_w = sum_t c[8w+t] 2^(16t) = lo_w + hi_w 2^128 (hi_w < 2^49).  The
// product is sum_w (lo_w + hi_(w-1)) 2^(128w); s_w = lo_w + hi_(w-1) may
// carry one bit (g_w) into window w+1, which a run of all-ones windows (p_w)
// propagates.  Carries are resolved by lookahead over (g, p) bit vectors: with
// A = g|p and B = g, the carry into each window of a warp is bit w of
// (A + B + cin) ^ A ^ B.

struct Win2 {
  uint64_t l[2];
  uint64_t hi;
};

// Window value from 8 canonical coefficients (u128 accumulator, as the
// reference's unpack loop, ntt.rs:694-707).
__device__ __forceinline__ Win2 fold8(const uint64_t* c8) {
  Win2 r;
  unsigned __int128 acc = 0;
#pragma unroll
  for (int k = 0; k < 2; k++) {
#pragma unroll
    for (int q = 0; q < 4; q++) acc += (unsigned __int128)c8[4 * k + q] << (16 * q);
    r.l[k] = (uint64_t)acc;
    acc >>= 64;
  }
  r.hi = (uint64_t)acc;
  return r;
}

// 16-coefficient windows of the one-CTA multiply (its own carry chain).
struct Win {
  uint64_t l[4];
  uint64_t hi;
};

__device__ __forceinline__ Win fold16(const uint64_t* c16, int stride) {
  Win r;
  unsigned __int128 acc = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
#pragma unroll
    for (int q = 0; q < 4; q++) acc += (unsigned __int128)c16[(4 * k + q) * stride] << (16 * q);
    r.l[k] = (uint64_t)acc;
    acc >>= 64;
  }
  r.hi = (uint64_t)acc;
  return r;
}

// Words of the carry scratch of a product with nwin windows: high parts, then
// the chunk states (the low parts lie in an array of 2 nwin words of their own).
__host__ __device__ __forceinline__ uint64_t carry_words(uint64_t nwin) { return nwin + (n_chunks(nwin) + 1) / 2; }

// The eight canonical coefficients c of window wl of a 2^L-point transform: the
// window's low limbs go to W and its high part to H (coefficients out for
// JF_COEFF, both windows that fall on it for a wrapped product).
__device__ __forceinline__ void put_window(const Job& J, int L, uint64_t wl, uint64_t* c) {
  if (wl < J.wlo) return;
  const uint64_t nlimbs = job_nout(J), nwin = n_windows_out(nlimbs);
  const uint64_t w = wl + (uint64_t)J.woff;  // window of the whole product
  ulonglong2* W = reinterpret_cast<ulonglong2*>(J.W);
  if (J.flags & JF_COEFF) {
#pragma unroll
    for (int t = 0; t < 8; t++)
      if (8 * w + t < nlimbs) J.out[8 * w + t] = c[t];
    return;
  }
  if (w >= nwin) return;
  if (J.wrap) {
    // coefficient 8w + t: low[8w + t] below wrap; N + 8w + t: the rest of the cyclic value
    uint64_t d[8];
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const uint64_t pos = 8 * w + t;
      const uint64_t lo = pos < J.wrap ? J.low[pos] : c[t];
      d[t] = c[t] - lo;
      c[t] = lo;
    }
    const uint64_t w2 = w + ((1ull << L) >> 3);
    if (w2 < nwin) {
      const Win2 v2 = fold8(d);
      W[w2] = make_ulonglong2(v2.l[0], v2.l[1]);
      J.H[w2] = v2.hi;
    }
  }
  const Win2 v = fold8(c);
  W[w] = make_ulonglong2(v.l[0], v.l[1]);
  J.H[w] = v.hi;
}

// Inverse pass 0 (natural order out) fused with the window fold: each tile
// row holds 2^T consecutive coefficients = 2^(T-3) windows; every window
// writes its low 2 limbs to W and its high part to H.
// twi: the pass's twiddle table (tw_first, inverse, with N^-1), or null to
// compute the twiddles, times ninv = N^-1.
// The rows are handed to the windows through shared memory, one pad word each.
template <int R>
constexpr uint32_t INV_FIRST_XWORDS = ColGeom<R>::XWORDS > ((ColGeom<R>::TM + 2) << R) ? ColGeom<R>::XWORDS
                                                                                      : (ColGeom<R>::TM + 2) << R;
template <int R>
__global__ void __launch_bounds__(PASS_THREADS, pass_min_ctas(R)) k_inv_first_carry(const Job* jobs, Job one, int L, Roots RT,
                                                                                 const uint64_t* __restrict__ twi, uint64_t ninv) {
  using G = ColGeom<R>;
  constexpr int B1 = G::B1, B2 = G::B2, T = G::T;
  const Job J = job_of(jobs, one, L);
  if (J.flags & JF_ADDEND) return;
  const uint64_t* data = J.A;
  extern __shared__ uint64_t sm[];
  const int tid = threadIdx.x;
  const int S = L - R;
  const uint64_t j0 = (uint64_t)blockIdx.x << T;
  uint64_t* tw = sm + INV_FIRST_XWORDS<R>;
  const bool staged = !twi && L > LVL_MAX;
  if (staged) {
    // w^-(f (j0 + j)) = w^-(f j0) w^-(f j), as in k_fwd_first
    for (uint32_t f = tid; f < (1u << R); f += PASS_THREADS) tw[f] = gl::mul(root_pow32(RT, L, f * (uint32_t)j0, true), ninv);
    __syncthreads();
  }
#pragma unroll 1
  for (int it = 0; it < G::ITERS2; it++) {
    const uint32_t w = it * PASS_THREADS + tid, j = w & G::TM, k1 = w >> T;
    const uint64_t at = ((uint64_t)(k1 << B2) << S) + j0 + j;
    uint64_t v[1 << B2];
    gl::Lz x[1 << B2];
#pragma unroll
    for (int k = 0; k < (1 << B2); k++) v[k] = data[at + ((uint64_t)k << S)];
    if (twi) {
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) x[k] = gl::lz_mul(v[k], __ldg(twi + at + ((uint64_t)k << S)));
    } else if (staged) {
      const uint64_t* __restrict__ nt = near_table(RT, L, true);
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) {
        const uint32_t f = k1 + (k << B1);
        x[k] = gl::lz_mul(v[k], gl::mul(tw[f], __ldg(nt + f * j)));
      }
    } else {
#pragma unroll
      for (int k = 0; k < (1 << B2); k++)
        x[k] = gl::lz_mul(v[k], gl::mul(root_pow32(RT, L, (k1 + (k << B1)) * (uint32_t)(j0 + j), true), ninv));
    }
    x[0] = gl::lz_bias(x[0]);
    dft_lz<B2, true>(x, v);
#pragma unroll
    for (int m = 0; m < (1 << B2); m++) sm[k1 * G::KS + (m << T) + j] = v[m];
  }
  __syncthreads();
  constexpr uint32_t RS = G::TM + 2;  // row stride of the coefficients
  {
    uint64_t v[1 << B1];
    pass_inv2<R>(sm + tid, G::KS, RT.rt + rt_offset(R, true), tid >> T, v);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < (1 << B1); m++) sm[((tid >> T) + (m << B2)) * RS + (tid & G::TM)] = gl::canon(v[m]);
  }
  __syncthreads();
  for (uint32_t q = tid; q < (1u << (G::TILE - 3)); q += PASS_THREADS) {
    const uint32_t i = q >> (T - 3), k = q & ((1u << (T - 3)) - 1);
    uint64_t c[8];
    const uint64_t* row = sm + i * RS + 8 * k;
#pragma unroll
    for (int t = 0; t < 8; t++) c[t] = row[t];
    put_window(J, L, ((((uint64_t)i << S) + j0) >> 3) + k, c);
  }
}

// First and last pass of a transform of N = 3 2^k points (192 rows of stride
// 2^S, S = k - 6); w_N = w_(2^k)^a w_3^b with 3 a + 2^k b = 1 mod N.  A product
// that fills at most three quarters of its power of two takes three quarters
// of the work.
__global__ void __launch_bounds__(128, 5) k_fwd_first3(const Job* jobs, Job one, int w0, int S, Roots RT,
                                                       const uint64_t* __restrict__ twf) {
  using G = ThreeGeom;
  const Job J = job_of(jobs, one, 0);
  const int which = w0 + (int)blockIdx.z;
  if (which == 1 && skips_b(J)) return;
  const uint16_t* coef = reinterpret_cast<const uint16_t*>(which ? J.b : J.a);
  const uint64_t nc = 4 * (which ? J.lb : J.la);
  uint64_t* __restrict__ data = which ? J.B : J.A;
  extern __shared__ uint64_t sm[];
  const int tid = threadIdx.x;
  const uint64_t j0 = (uint64_t)blockIdx.x << G::T;
  if (tid < 96) {
    // round 1: rows (tid >> 3) + 12 m
    const uint64_t n0 = ((uint64_t)(tid >> 3) << S) + j0 + (tid & 7), step = 12ull << S;
    uint64_t v[16];
    gl::Lz x[16];
    if (nc <= 96ull << S) {  // the upper half of the rows is zero
#pragma unroll
      for (int m = 0; m < 8; m++) x[m] = gl::Lz{n0 + m * step < nc ? (uint32_t)coef[n0 + m * step] : 0u, 0u, 0};
      x[0] = gl::lz_bias(x[0]);
      dft_lz<4, false, true>(x, v);
    } else {
#pragma unroll
      for (int m = 0; m < 16; m++) x[m] = gl::Lz{n0 + m * step < nc ? (uint32_t)coef[n0 + m * step] : 0u, 0u, 0};
      x[0] = gl::lz_bias(x[0]);
      dft_lz<4, false>(x, v);
    }
#pragma unroll
    for (int k = 0; k < 16; k++) sm[k * G::KS + tid] = v[k];
  }
  __syncthreads();
  const uint64_t* __restrict__ rt = RT.rt + RT_WORDS;
  const uint32_t j = tid & 7, k1 = tid >> 3;
  uint64_t v[12];
  gl::Lz x[12];
  x[0] = gl::lz_bias(gl::lz(sm[k1 * G::KS + j]));
#pragma unroll
  for (int m = 1; m < 12; m++) x[m] = gl::lz_mul(sm[k1 * G::KS + m * 8 + j], __ldg(rt + m * 16 + k1));
  dft12_lz<false>(x, v);
  const uint64_t at = ((uint64_t)(k1 * 12) << S) + j0 + j;
#pragma unroll
  for (int k = 0; k < 12; k++) data[at + ((uint64_t)k << S)] = gl::mul(v[k], __ldg(twf + at + ((uint64_t)k << S)));
}

__global__ void __launch_bounds__(128, 5) k_inv_first3_carry(const Job* jobs, Job one, int S, Roots RT,
                                                             const uint64_t* __restrict__ twi) {
  using G = ThreeGeom;
  const Job J = job_of(jobs, one, 0);
  if (J.flags & JF_ADDEND) return;
  const uint64_t* data = J.A;
  extern __shared__ uint64_t sm[];
  const int tid = threadIdx.x;
  const uint64_t j0 = (uint64_t)blockIdx.x << G::T;
  const uint64_t* __restrict__ rt = RT.rt + RT_WORDS + 192;
  {
    const uint32_t j = tid & 7, k1 = tid >> 3;
    const uint64_t at = ((uint64_t)(k1 * 12) << S) + j0 + j;
    uint64_t v[12];
    gl::Lz x[12];
#pragma unroll
    for (int k = 0; k < 12; k++) v[k] = data[at + ((uint64_t)k << S)];
#pragma unroll
    for (int k = 0; k < 12; k++) x[k] = gl::lz_mul(v[k], __ldg(twi + at + ((uint64_t)k << S)));
    x[0] = gl::lz_bias(x[0]);
    dft12_lz<true>(x, v);
#pragma unroll
    for (int m = 0; m < 12; m++) sm[k1 * G::KS + m * 8 + j] = v[m];
  }
  __syncthreads();
  const uint32_t m0 = tid >> 3;
  uint64_t v[16];
  if (tid < 96) {
    gl::Lz x[16];
    x[0] = gl::lz_bias(gl::lz(sm[tid]));
#pragma unroll
    for (int k = 1; k < 16; k++) x[k] = gl::lz_mul(sm[k * G::KS + tid], __ldg(rt + k * 12 + m0));
    dft_lz<4, true>(x, v);
  }
  __syncthreads();
  if (tid < 96) {
#pragma unroll
    for (int m = 0; m < 16; m++) sm[(m0 + 12 * m) * 9 + (tid & 7)] = gl::canon(v[m]);
  }
  __syncthreads();
  for (uint32_t row = tid; row < G::ROWS; row += 128) {
    uint64_t c[8];
#pragma unroll
    for (int t = 0; t < 8; t++) c[t] = sm[row * 9 + t];
    put_window(J, 0, (((uint64_t)row << S) + j0) >> 3, c);
  }
}

// Window w after its left neighbour's high part: s_w = lo_w + hi_(w-1), and
// its (generate, propagate) bits; the windows past the end do neither.
struct WinSum {
  uint64_t s0, s1;
  bool g, p;
};
__device__ __forceinline__ WinSum win_sum(const Job& J, uint64_t w, uint64_t nwin) {
  WinSum r{0, 0, false, false};
  if (w < nwin) {
    const ulonglong2 l = reinterpret_cast<const ulonglong2*>(J.W)[w];
    const uint64_t hprev = w > 0 ? J.H[w - 1] : 0;
    r.s0 = l.x + hprev;
    const uint64_t c = r.s0 < hprev;
    r.s1 = l.y + c;
    r.g = c && r.s1 == 0;
    r.p = (r.s0 & r.s1) == ~0ull;
  }
  return r;
}

// Carry function of a run of windows as two bits: bit 0 = carry out for carry
// in 0, bit 1 = carry out for carry in 1.
__device__ __forceinline__ uint32_t cf_of_masks(uint32_t A, uint32_t B) {
  const uint64_t s = (uint64_t)A + B;
  return (uint32_t)(s >> 32) | (uint32_t)((s + 1) >> 32) << 1;
}
// Running `first`, then `then`.
__device__ __forceinline__ uint32_t cf_then(uint32_t first, uint32_t then) {
  return ((then >> (first & 1)) & 1) | ((then >> ((first >> 1) & 1)) & 1) << 1;
}

// Carry function of chunk c from its windows, by one warp.
__device__ uint32_t chunk_function(const Job& J, uint64_t c, uint64_t nwin, int lane) {
  uint32_t f = 2;  // identity
  for (int k = 0; k < CARRY_THREADS / 32; k++) {
    const WinSum x = win_sum(J, c * CARRY_THREADS + 32 * k + lane, nwin);
    const uint32_t A = __ballot_sync(0xFFFFFFFFu, x.g || x.p), B = __ballot_sync(0xFFFFFFFFu, x.g);
    f = cf_then(f, cf_of_masks(A, B));
  }
  return f;
}

// Carry normalisation in one pass (chunks of 256 windows over grid.x, grid.y =
// product).  A chunk's carry in almost always shows in the 32 windows to its
// left, which warp 0 sums as well: no chunk waits for another.  Where all 32
// pass a carry on (each all ones), the chunks' states are read instead: every
// chunk publishes its carry function as soon as it has it (4 | function; the
// states were zeroed by k_inv_last), one that passes its carry on replaces it
// once it knows that carry, and the nearest chunk with a fixed carry out
// gives the carry in.  A state that stays away for CARRY_POLLS reads (its CTA
// may not run yet) is not waited for: the warp works the function out from
// that chunk's windows, which are only read here.  Memory-bound: 24 bytes read
// and 16 written per window; against three kernels (sums in place, scan,
// increments) 240 -> 141 us at 2^27 points and two launches less.
constexpr int CARRY_POLLS = 32;
constexpr uint64_t CARRY_CTAS = 8192;  // of a batch (4096 and 16384 within 0.5 %)

__global__ void __launch_bounds__(CARRY_THREADS) k_carry(const Job* jobs, Job one) {
  const Job J = job_of(jobs, one, 0);
  if (J.flags & (JF_ADDEND | JF_COEFF)) return;
  const uint64_t nlimbs = job_nout(J), nwin = n_windows_out(nlimbs), nchunk = n_chunks(nwin);
  __shared__ uint32_t sA[CARRY_THREADS / 32], sB[CARRY_THREADS / 32], s_cin;
  for (uint64_t chunk = blockIdx.x; chunk < nchunk; chunk += gridDim.x) {  // uniform per CTA
    const uint64_t w = chunk * CARRY_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const WinSum x = win_sum(J, w, nwin);
    uint32_t left = 0;  // function of the 32 windows to the left (chunk 0: no carry)
    if (warp == 0 && chunk > 0) {
      const WinSum y = win_sum(J, w - 32, nwin);
      const uint32_t yA = __ballot_sync(0xFFFFFFFFu, y.g || y.p), yB = __ballot_sync(0xFFFFFFFFu, y.g);
      left = cf_of_masks(yA, yB);
    }
    const uint32_t A = __ballot_sync(0xFFFFFFFFu, x.g || x.p);
    const uint32_t B = __ballot_sync(0xFFFFFFFFu, x.g);
    if (lane == 0) {
      sA[warp] = A;
      sB[warp] = B;
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t f = 2;
      for (int k = 0; k < CARRY_THREADS / 32; k++) f = cf_then(f, cf_of_masks(sA[k], sB[k]));
      volatile uint32_t* state = J.state;
      if (lane == 0) state[chunk] = 4 | f;
      uint32_t cin = left & 1;
      // chunks chunk - 1 - lane, 32 at a time; left of chunk 0 the carry is 0
      for (int64_t base = (int64_t)chunk - 1; left == 2; base -= 32) {
        const int64_t c = base - lane;
        uint32_t st = c < 0 ? 4 : state[c];
        for (int poll = 0; poll < CARRY_POLLS && __any_sync(0xFFFFFFFFu, st == 0); poll++) {
          if (st == 0) st = state[c];
          // enough once a known chunk with a fixed carry out comes before the first unknown one
          const uint32_t unknown = __ballot_sync(0xFFFFFFFFu, st == 0);
          const uint32_t fixed = __ballot_sync(0xFFFFFFFFu, st != 0 && (st & 3) != 2);
          if (fixed && (!unknown || __ffs(fixed) < __ffs(unknown))) break;
        }
        // the nearest chunk whose carry out is fixed (identity passes it on)
        bool done = false;
        for (int k = 0; k < 32; k++) {
          uint32_t sk = __shfl_sync(0xFFFFFFFFu, st, k);
          if (sk == 0) sk = 4 | chunk_function(J, (uint64_t)(base - k), nwin, lane);
          if ((sk & 3) != 2) {
            cin = sk & 1;
            done = true;
            break;
          }
        }
        if (done) break;
      }
      if (lane == 0) {
        s_cin = cin;
        // a chunk that passes its carry on now has a fixed one: look-backs stop here
        if (f == 2) state[chunk] = 4 | (cin ? 3 : 0);
      }
    }
    __syncthreads();
    uint32_t cin = s_cin;
    for (int k = 0; k < warp; k++) cin = (cf_of_masks(sA[k], sB[k]) >> cin) & 1;
    const uint32_t carries = (A + B + cin) ^ A ^ B;
    if (w < nwin) {
      const uint64_t inc = (carries >> lane) & 1;
      const uint64_t s0 = x.s0 + inc, s1 = x.s1 + (inc && s0 == 0);
      if (2 * w < nlimbs) J.out[2 * w] = s0;
      if (2 * w + 1 < nlimbs) J.out[2 * w + 1] = s1;
    }
    __syncthreads();  // the next chunk reuses the shared words
  }
}

// ---- whole multiply in one CTA (N <= 2^SMALL_LOG_MAX) --------------------
// Products of up to 64 limbs in all are schoolbook column sums by one warp
// (class 7); longer ones take three transforms of 2^c points (class c = 9 ..
// 12) as two or three rounds of radix 8 or 16 in registers.  A lone product
// holds operands a and b side by side in the halves of
// its threads: one SM is all it has, and a thread's instructions are its time.
// In a batch a group of G threads transforms one operand after the other, two
// CTAs per SM, so that no thread idles through the inverse and other groups
// run while one waits.  Lone products: 10.3 -> 6.2 us at 2^10 bits, 18.0 -> 7.7 at
// 100 x 100 limbs.
constexpr int SMALL_THREADS = 256;
constexpr int SMALL_LOG_MAX = 12;
constexpr int SMALL_TINY = 7;        // class of the one-warp products
constexpr uint64_t TINY_LIMBS = 64;  // la + lb

// Radix (log2) of round q of a 2^c-point transform (0: no such round; 2^8 points come
// in the merged splitting levels only).
__host__ __device__ constexpr int small_b(int c, int q) {
  return c == 8 ? (q < 2 ? 4 : 0) : c == 9 ? 3 : c == 10 ? (q == 0 ? 4 : 3) : c == 11 ? (q < 2 ? 4 : 3) : 4;
}
// Threads per operand: one radix-16 item (8 for class 9) each; per product.
__host__ __device__ constexpr int small_op_threads(int c) { return c == 9 ? 64 : (1 << c) / 16; }
__host__ __device__ constexpr int small_threads(int c, bool split) {
  return c == SMALL_TINY ? 32 : (split ? 2 : 1) * small_op_threads(c);
}
// Class of a product of la + lb limbs.
__host__ __device__ __forceinline__ int small_class(uint64_t la, uint64_t lb) {
  if (la + lb <= TINY_LIMBS) return SMALL_TINY;
  const uint32_t n = (uint32_t)(4 * (la + lb) - 1);
  return n <= 512 ? 9 : n <= 1024 ? 10 : n <= 2048 ? 11 : 12;
}
// Dynamic shared memory words of one product: a padded array per operand held
// at a time, and the windows' high parts (a tiny product: its operands, 64 zero
// limbs on either side of the longer).
__host__ __device__ constexpr uint32_t small_words(int c, bool split) {
  return c == SMALL_TINY ? 256 : split ? 2 * spad(1u << c) : spad(1u << c) + (1u << c) / 16;
}
// Products of one class side by side in a batch CTA, and its shared memory.
__host__ __device__ __forceinline__ uint32_t small_per_cta(int c) { return SMALL_THREADS / small_threads(c, false); }
__host__ __device__ __forceinline__ size_t small_cta_smem(int c) {
  return (size_t)small_per_cta(c) * small_words(c, false) * 8;
}

struct SmallJob {
  const uint64_t* a;
  const uint64_t* b;
  uint64_t* out;
  uint32_t la, lb;
};

// count (<= small_per_cta) consecutive jobs of class c from first.
struct SmallChunk {
  uint32_t first, count;
  int c;
};

// Barrier of a product's T threads (group grp of the CTA).
template <int T>
__device__ __forceinline__ void small_sync(int grp) {
  if constexpr (T == 32)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(T) : "memory");
}

// Forward transform of an operand of nc coefficients by G threads (u) of a
// group of T (all of which pass the barriers; run = false: nothing else).
// After the rounds of radix 2^B1, 2^B2, 2^B3, element (k1, k2, k3) of the
// spectrum has index (k1 2^B2 + k2) 2^B3 + k3; thread u ends up with items it G
// + u of the last round in s.  A round's twiddles w^(k j) enter the next
// round's inputs as lazy products, from the table of 4096th roots.
template <int C, int T>
__device__ __forceinline__ void small_forward(const uint64_t* limbs, uint32_t nc, const Roots& R, uint64_t* sm, int u, int grp,
                                              bool run, uint64_t* s) {
  constexpr int B1 = small_b(C, 0), B2 = small_b(C, 1), B3 = small_b(C, 2);
  constexpr int G = small_op_threads(C);
  constexpr int S1 = C - B1, S2 = S1 - B2;  // log2 sub-problem sizes after rounds 1 and 2
  static_assert(S2 == B3, "the rounds make up the transform");
  if (run) {
    // round 1: coefficients m 2^S1 + j
    const uint16_t* coef = reinterpret_cast<const uint16_t*>(limbs);
#pragma unroll
    for (int it = 0; it < (1 << S1) / G; it++) {
      const uint32_t j = it * G + u;
      uint64_t v[1 << B1];
      gl::Lz x[1 << B1];
#pragma unroll
      for (int m = 0; m < (1 << B1); m++) {
        const uint32_t n = (m << S1) + j;
        x[m] = gl::Lz{n < nc ? (uint32_t)coef[n] : 0u, 0u, 0};
      }
      x[0] = gl::lz_bias(x[0]);
      dft_lz<B1, false>(x, v);
#pragma unroll
      for (int k = 0; k < (1 << B1); k++) sm[spad((k << S1) + j)] = v[k];
    }
  }
  small_sync<T>(grp);
  constexpr int BL = B3 ? B3 : B2;             // last round
  constexpr int ITL = (1 << (C - BL)) / G;     // its items per thread
  if constexpr (B3 > 0) {
    if (run) {
      // round 2: (k1, j2), inputs j = m 2^S2 + j2 with twiddles w_N^(k1 j)
#pragma unroll
      for (int it = 0; it < (1 << (C - B2)) / G; it++) {
        const uint32_t w = it * G + u, j2 = w & ((1u << S2) - 1), k1 = w >> S2;
        const uint32_t base = (k1 << S1) + j2;
        uint64_t v[1 << B2];
        gl::Lz x[1 << B2];
#pragma unroll
        for (int m = 0; m < (1 << B2); m++)
          x[m] = gl::lz_mul(sm[spad(base + (m << S2))], __ldg(R.w12 + ((k1 * (j2 + (m << S2))) << (12 - C))));
        x[0] = gl::lz_bias(x[0]);
        dft_lz<B2, false>(x, v);
#pragma unroll
        for (int k = 0; k < (1 << B2); k++) sm[spad(base + (k << S2))] = v[k];
      }
    }
    small_sync<T>(grp);
  }
  if (run) {
    // last round: (k1, k2) with twiddles w_(2^S1)^(k2 m), or k1 with w_N^(k1 m)
    constexpr int mlog = B3 ? S1 : C;
    constexpr uint32_t kmask = (1u << (B3 ? B2 : B1)) - 1;
#pragma unroll
    for (int it = 0; it < ITL; it++) {
      const uint32_t w = it * G + u, k = w & kmask;
      gl::Lz x[1 << BL];
      x[0] = gl::lz_bias(gl::lz(sm[spad(w << BL)]));
#pragma unroll
      for (int m = 1; m < (1 << BL); m++)
        x[m] = gl::lz_mul(sm[spad((w << BL) + m)], __ldg(R.w12 + ((k * m) << (12 - mlog))));
      dft_lz<BL, false>(x, s + (it << BL));
    }
  }
}

// The inverse's rounds after its first one, on all T threads of the group:
// natural order in sm.
template <int C, int T>
__device__ __forceinline__ void small_inverse(const Roots& R, uint64_t* sm, int t, int grp) {
  constexpr int B1 = small_b(C, 0), B2 = small_b(C, 1), B3 = small_b(C, 2);
  constexpr int S1 = C - B1, S2 = S1 - B2;
  small_sync<T>(grp);
  if constexpr (B3 > 0) {
    for (uint32_t w = t; w < (1u << (C - B2)); w += T) {
      const uint32_t j2 = w & ((1u << S2) - 1), k1 = w >> S2, base = (k1 << S1) + j2;
      uint64_t v[1 << B2];
      gl::Lz x[1 << B2];
      x[0] = gl::lz_bias(gl::lz(sm[spad(base)]));
#pragma unroll
      for (int k = 1; k < (1 << B2); k++)
        x[k] = gl::lz_mul(sm[spad(base + (k << S2))], __ldg(R.w12 + ((4096 - ((k * j2) << (12 - S1))) & 4095)));
      dft_lz<B2, true>(x, v);
#pragma unroll
      for (int m = 0; m < (1 << B2); m++) sm[spad(base + (m << S2))] = v[m];
    }
    small_sync<T>(grp);
  }
  for (uint32_t j = t; j < (1u << S1); j += T) {
    uint64_t v[1 << B1];
    gl::Lz x[1 << B1];
    x[0] = gl::lz_bias(gl::lz(sm[spad(j)]));
#pragma unroll
    for (int k = 1; k < (1 << B1); k++)
      x[k] = gl::lz_mul(sm[spad((k << S1) + j)], __ldg(R.w12 + ((4096 - ((k * j) << (12 - C))) & 4095)));
    dft_lz<B1, true>(x, v);
#pragma unroll
    for (int m = 0; m < (1 << B1); m++) sm[spad((m << S1) + j)] = v[m];
  }
  small_sync<T>(grp);
}

// One product by its T threads (t = thread in the group, grp = group of the
// CTA).  SPLIT: threads 0 .. G - 1 hold operand a, the others b.
template <int C, bool SPLIT>
__device__ __forceinline__ void small_multiply(const SmallJob& job, const Roots& R, uint64_t* smA, int t, int grp, uint32_t* sA,
                                               uint32_t* sBm) {
  constexpr int B1 = small_b(C, 0), B2 = small_b(C, 1), B3 = small_b(C, 2);
  constexpr int G = small_op_threads(C), T = small_threads(C, SPLIT);
  constexpr int BL = B3 ? B3 : B2, ITL = (1 << (C - BL)) / G;
  constexpr uint32_t N = 1u << C;
  uint64_t* smB = smA + spad(N);  // b's array (SPLIT); the windows' high parts
  const uint32_t la = job.la, lb = job.lb;
  const bool square = job.a == job.b && la == lb;
  // times N^-1 = 2^(-C): with 2^96 = -1 and 2^64 = 2^32 - 1 (mod p),
  // 2^(-C) = -2^(96-C) = p - (2^(64-C) - 2^(32-C))
  constexpr uint64_t ninv = gl::P - ((1ull << (64 - C)) - (1ull << (32 - C)));
  uint64_t s[ITL << BL], y[SPLIT ? 1 : ITL << BL];
  const bool isb = SPLIT && t >= G;
  if constexpr (SPLIT) {
    const bool idle = isb && square;
    uint64_t* sm = isb ? smB : smA;
    small_forward<C, T>(isb ? job.b : job.a, 4 * (isb ? lb : la), R, sm, isb ? t - G : t, grp, !idle, s);
    // b's spectrum to the threads that hold a's
    if (isb && !idle) {
#pragma unroll
      for (int it = 0; it < ITL; it++)
#pragma unroll
        for (int k = 0; k < (1 << BL); k++) sm[spad(((it * G + t - G) << BL) + k)] = gl::mul(s[(it << BL) + k], ninv);
    }
    small_sync<T>(grp);
  } else {
    small_forward<C, T>(job.a, 4 * la, R, smA, t, grp, true, s);
    if (square) {
#pragma unroll
      for (int k = 0; k < (ITL << BL); k++) y[k] = s[k];
    } else {
      small_sync<T>(grp);
      small_forward<C, T>(job.b, 4 * lb, R, smA, t, grp, true, y);
    }
    // (a thread overwrites below what it alone has read)
  }
  if (!isb) {
#pragma unroll
    for (int it = 0; it < ITL; it++) {
      const uint32_t base = (it * G + t) << BL;
      uint64_t v[1 << BL];
      gl::Lz x[1 << BL];
#pragma unroll
      for (int k = 0; k < (1 << BL); k++) {
        const int i = (it << BL) + k;
        const uint64_t z = !SPLIT ? gl::mul(y[SPLIT ? 0 : i], ninv) : square ? gl::mul(s[i], ninv) : smB[spad(base + k)];
        x[k] = gl::lz_mul(s[i], z);
      }
      x[0] = gl::lz_bias(x[0]);
      dft_lz<BL, true>(x, v);
#pragma unroll
      for (int m = 0; m < (1 << BL); m++) smA[spad(base + m)] = v[m];
    }
  }
  small_inverse<C, T>(R, smA, t, grp);
  // carry: windows of 16 coefficients, one per thread (N/16 <= T)
  const uint32_t n_out = 4 * la + 4 * lb - 1, nwin = (n_out + 15) / 16, nl = la + lb;
  uint64_t* sH = smB;  // b's spectrum is no longer needed
  Win v{{0, 0, 0, 0}, 0};
  const uint32_t w = t;
  if (w < nwin) {
    uint64_t c[16];
#pragma unroll
    for (int q = 0; q < 16; q++) c[q] = gl::canon(smA[spad(16 * w + q)]);
    v = fold16(c, 1);
    sH[w] = v.hi;  // nwin <= N/16 words
  }
  small_sync<T>(grp);
  const uint64_t hprev = (w > 0 && w < nwin) ? sH[w - 1] : 0;
  uint64_t s0 = v.l[0] + hprev;
  uint64_t c = s0 < hprev;
  uint64_t s1 = v.l[1] + c;  c = c && s1 == 0;
  uint64_t s2 = v.l[2] + c;  c = c && s2 == 0;
  uint64_t s3 = v.l[3] + c;  c = c && s3 == 0;
  const bool gg = w < nwin && c;
  const bool pp = w < nwin && (s0 & s1 & s2 & s3) == ~0ull;
  const uint32_t A = __ballot_sync(0xFFFFFFFFu, gg || pp), Bm = __ballot_sync(0xFFFFFFFFu, gg);
  uint32_t cin = 0;
  if constexpr (T > 32) {
    const int gw0 = grp * (T / 32), gw = gw0 + (t >> 5);
    if ((t & 31) == 0) sA[gw] = A, sBm[gw] = Bm;
    small_sync<T>(grp);
    for (int k = gw0; k < gw; k++) {
      const uint64_t x = (uint64_t)sA[k] + sBm[k] + cin;
      cin = (uint32_t)(x >> 32);
    }
  }
  const uint32_t carries = (A + Bm + cin) ^ A ^ Bm;
  if ((carries >> (t & 31)) & 1) {
    if (++s0 == 0) if (++s1 == 0) if (++s2 == 0) ++s3;
  }
  if (w < nwin) {
    const uint32_t base = 4 * w;
    if (base + 0 < nl) job.out[base + 0] = s0;
    if (base + 1 < nl) job.out[base + 1] = s1;
    if (base + 2 < nl) job.out[base + 2] = s2;
    if (base + 3 < nl) job.out[base + 3] = s3;
  }
}

// (x2 x1 x0) += a * b, 192 bits.
__device__ __forceinline__ void mac192(uint64_t a, uint64_t b, uint64_t& x0, uint64_t& x1, uint64_t& x2) {
  const uint64_t lo = a * b, hi = __umul64hi(a, b);
  asm("add.cc.u64 %0, %0, %3;\n\taddc.cc.u64 %1, %1, %4;\n\taddc.u64 %2, %2, 0;"
      : "+l"(x0), "+l"(x1), "+l"(x2)
      : "l"(lo), "l"(hi));
}

// la + lb <= 64 by one warp: lane w sums the columns 2w and 2w + 1 over the
// shorter operand's limbs (the longer one lies between zeros in shared memory)
// and resolves its window's carry with the warp's ballots.
__device__ void tiny_multiply(const SmallJob& job, uint64_t* sm, int lane) {
  const bool sw = job.lb > job.la;
  const uint64_t* a = sw ? job.b : job.a;  // the longer
  const uint64_t* b = sw ? job.a : job.b;
  const uint32_t la = sw ? job.lb : job.la, lb = sw ? job.la : job.lb, nl = la + lb;
  uint64_t* sa = sm + 64;   // 64 zeros, a, zeros up to 192 words
  uint64_t* sb = sm + 192;  // b: at most 32 words
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const uint32_t i = q * 32 + lane;
    sm[i] = i >= 64 && i - 64 < la ? a[i - 64] : 0;
  }
  if ((uint32_t)lane < lb) sb[lane] = b[lane];
  __syncwarp();
  uint64_t e0 = 0, e1 = 0, e2 = 0, o0 = 0, o1 = 0, o2 = 0;
  const uint64_t* col = sa + 2 * lane;
  for (uint32_t i = 0; i < lb; i++) {
    const uint64_t y = sb[i];
    mac192(col[-(int)i], y, e0, e1, e2);
    mac192(col[1 - (int)i], y, o0, o1, o2);
  }
  // window value e + o 2^64: low 128 bits here, high 128 bits to the next lane
  const uint64_t l1 = e1 + o0;
  uint64_t h0 = e2 + (l1 < o0);
  uint64_t h1 = o2;
  h0 += o1;
  h1 += h0 < o1;
  uint64_t p0 = __shfl_up_sync(0xFFFFFFFFu, h0, 1), p1 = __shfl_up_sync(0xFFFFFFFFu, h1, 1);
  if (lane == 0) p0 = p1 = 0;
  uint64_t s0 = e0 + p0;
  const uint64_t c0 = s0 < p0;
  uint64_t s1 = l1 + c0;
  uint64_t g = s1 < c0;
  s1 += p1;
  g |= s1 < p1;
  const uint32_t A = __ballot_sync(0xFFFFFFFFu, g || (s0 & s1) == ~0ull), B = __ballot_sync(0xFFFFFFFFu, g != 0);
  if ((((A + B) ^ A ^ B) >> lane) & 1)
    if (++s0 == 0) ++s1;
  if (2 * (uint32_t)lane < nl) job.out[2 * lane] = s0;
  if (2 * (uint32_t)lane + 1 < nl) job.out[2 * lane + 1] = s1;
  __syncwarp();
}

template <int C>
__device__ __noinline__ void small_chunk(const SmallJob* jobs, const SmallChunk& ch, const Roots& R, uint64_t* sm,
                                         uint32_t* sA, uint32_t* sBm) {
  constexpr int T = small_threads(C, false);
  const uint32_t grp = threadIdx.x / T;
  if (grp >= ch.count) return;
  const SmallJob job = jobs[ch.first + grp];
  uint64_t* base = sm + (size_t)grp * small_words(C, false);
  if constexpr (C == SMALL_TINY)
    tiny_multiply(job, base, threadIdx.x & 31);
  else
    small_multiply<C, false>(job, R, base, (int)(threadIdx.x % T), (int)grp, sA, sBm);
}

// Chunks of same-class products; the CTAs stride over the chunks (a
// persistent kernel over a size-sorted batch).
// Against the former kernel (one radix-8 butterfly per thread and round, runtime
// geometry): 16384 products of 128 .. 256 limbs 1132 -> 712 us, 4096 of 64 .. 128
// limbs 154 -> 90.  Three CTAs per SM (80 registers) run no faster.
__global__ void __launch_bounds__(SMALL_THREADS, 2) k_small_mul(const SmallJob* jobs, const SmallChunk* chunks, uint32_t nchunks,
                                                               Roots R) {
  pdl_wait();
  extern __shared__ uint64_t sm[];
  __shared__ uint32_t sA[SMALL_THREADS / 32], sBm[SMALL_THREADS / 32];
  for (uint32_t k = blockIdx.x; k < nchunks; k += gridDim.x) {
    const SmallChunk ch = chunks[k];
    switch (ch.c) {
      case SMALL_TINY: small_chunk<SMALL_TINY>(jobs, ch, R, sm, sA, sBm); break;
      case 9: small_chunk<9>(jobs, ch, R, sm, sA, sBm); break;
      case 10: small_chunk<10>(jobs, ch, R, sm, sA, sBm); break;
      case 11: small_chunk<11>(jobs, ch, R, sm, sA, sBm); break;
      default: small_chunk<12>(jobs, ch, R, sm, sA, sBm); break;
    }
    __syncthreads();
  }
}

// One product (the plain call).
template <int C>
__global__ void __launch_bounds__(small_threads(C, true), 1) k_small_one(SmallJob job, Roots R) {
  pdl_wait();
  extern __shared__ uint64_t sm[];
  __shared__ uint32_t sA[SMALL_THREADS / 32], sBm[SMALL_THREADS / 32];
  if constexpr (C == SMALL_TINY)
    tiny_multiply(job, sm, threadIdx.x);
  else
    small_multiply<C, true>(job, R, sm, threadIdx.x, 0, sA, sBm);
}

// ---- whole multiply in one cluster (a lone product of 2^11 .. 2^14 points, few of a batch) --
// One SM takes 10.5 us for a lone product of 2^11 points and 18.7 for 2^12, and
// the pass pipeline 17 us for 2^13 (five launches of mostly idle grids): eight
// CTAs take 8.5 us for up to 2^12 points, sixteen 10.5 for 2^13 and 13.6 for
// 2^14 (eight: 13.3 and 21.5).  Half of them hold each operand: two passes of
// radix 2^R1 (columns) and 2^R2 (rows) of two register rounds each, with the
// transposes between them (and the hand-over of b's spectrum, of the inverse's
// columns and of the coefficients in natural order) as stores into the other
// CTAs' shared memory.  Below 2^11 points one CTA is as fast.
//
// Few products of up to 2^11 points of a batch take four CTAs each: in
// k_small_mul one of 2^11 points is 24 us of instructions, most of them fetched
// for the first time (11 stall cycles per issue), and 8 of 250 x 250 limbs took
// 32.4 us, 28.7 with the kernel before that one, 16 so; 100 of them 33.2 and 20.4,
// 250 33.6 and 30.2, 300 33.7 and 33.5.  The batch's shorter products of 2^9
// points and more go along (32 of 32 to 256 limbs 32.5 and 17.0 us), which saves
// their turn in k_small_mul; without one of 2^11 points that is the faster
// (14.9 against 15.3 us for 32 of 2^9 points, 17.2 and 29.2 for 250).
constexpr int CLUSTER_LOG_MIN = 11, CLUSTER_LOG_MAX = 14;
constexpr size_t CLUSTER_FEW = 256;

template <int L>
struct ClusterGeom {
  static constexpr int LOP = L == 11 ? 1 : L == 12 ? 2 : 3, OP = 1 << LOP;  // CTAs per operand
  static constexpr int R1 = (L + 1) / 2, R2 = L / 2;
  static constexpr int B1 = pass_b1(R1), B2 = pass_b2(R1), D1 = pass_b1(R2), D2 = pass_b2(R2);
  static constexpr int TC = R2 - LOP;                // log2 columns per CTA
  static constexpr int RC = R1 - LOP;                // log2 rows per CTA
  static constexpr uint32_t WORDS = 1u << (L - LOP); // of one operand, per CTA
  static constexpr int NT = WORDS / 8 < 256 ? WORDS / 8 : 256;
  static constexpr uint32_t CS = (1u << TC) + 1;     // row stride of a CTA's columns
  static constexpr uint32_t YS = (1u << R2) + 1;     // stride of its rows
  static constexpr uint32_t XW = CS << R1;           // words: columns, rows (or coefficients), spectrum
  static constexpr uint32_t YW = (YS << RC) > WORDS + WORDS / 16 ? YS << RC : WORDS + WORDS / 16;
  static constexpr uint32_t SMEM = (XW + YW + WORDS) * 8;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() {
  cluster_arrive();
  cluster_wait();
}
// p's counterpart in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint64_t* cluster_ptr(uint64_t* p, uint32_t rank) {
  uint64_t r;
  asm("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
  return reinterpret_cast<uint64_t*>(r);
}

// LIST: a cluster per blockIdx.y and its job from a device list; else one product
// by value (read from either, a lone 2^13-point product took 10.7 us, not 10.5).
template <int L, bool LIST = false>
__global__ void __cluster_dims__(2 * ClusterGeom<L>::OP, 1, 1) __launch_bounds__(ClusterGeom<L>::NT, 1)
    k_cluster_mul(std::conditional_t<LIST, const SmallJob*, SmallJob> from, Roots R) {
  using G = ClusterGeom<L>;
  constexpr int R1 = G::R1, R2 = G::R2, B1 = G::B1, B2 = G::B2, D1 = G::D1, D2 = G::D2, TC = G::TC, RC = G::RC, NT = G::NT;
  constexpr uint32_t N = 1u << L, CM = (1u << TC) - 1;
  cluster_arrive();  // waited on before the first store into another CTA: all of them run by then
  pdl_wait();
  SmallJob job;
  if constexpr (LIST) job = from[blockIdx.y];
  else job = from;
  extern __shared__ uint64_t sm[];
  uint64_t* X = sm;            // this CTA's columns: [row][column], stride CS
  uint64_t* Y = X + G::XW;     // its rows: [row][2^R2 words], stride YS; later its coefficients
  uint64_t* Z = Y + G::YW;     // b's spectrum; later the windows' high parts
  __shared__ uint32_t sA[NT / 32], sB[NT / 32];
  __shared__ uint64_t sF[G::OP];
  const uint32_t rank = blockIdx.x & (G::OP - 1);
  const bool isb = blockIdx.x >= G::OP;
  const uint32_t mine = isb ? G::OP : 0;           // first CTA of this operand
  const uint32_t la = job.la, lb = job.lb;
  const bool square = job.a == job.b && la == lb;
  const int t = threadIdx.x;
  const uint32_t col0 = rank << TC;
  constexpr uint64_t ninv = gl::P - ((1ull << (64 - L)) - (1ull << (32 - L)));  // 2^-L
  if (!(isb && square)) {
    // pass 1, round 1: coefficients row 2^R2 + column, rows (m << B2) + jp
    const uint16_t* coef = reinterpret_cast<const uint16_t*>(isb ? job.b : job.a);
    const uint32_t nc = 4 * (isb ? lb : la);
#pragma unroll 1
    for (uint32_t w = t; w < (1u << (B2 + TC)); w += NT) {
      const uint32_t c = w & CM, jp = w >> TC;
      uint64_t v[1 << B1];
      gl::Lz x[1 << B1];
#pragma unroll
      for (int m = 0; m < (1 << B1); m++) {
        const uint32_t n = (((m << B2) + jp) << R2) + col0 + c;
        x[m] = gl::Lz{n < nc ? (uint32_t)coef[n] : 0u, 0u, 0};
      }
      x[0] = gl::lz_bias(x[0]);
      dft_lz<B1, false>(x, v);
#pragma unroll
      for (int k = 0; k < (1 << B1); k++) X[((k << B2) + jp) * G::CS + c] = v[k];
    }
  }
  __syncthreads();
  cluster_wait();
  if (!(isb && square)) {
    // round 2, pass twiddles, rows to the CTAs that own them
#pragma unroll 1
    for (uint32_t w = t; w < (1u << (B1 + TC)); w += NT) {
      const uint32_t c = w & CM, k1 = w >> TC, J = col0 + c;
      uint64_t v[1 << B2];
      pass_fwd2<R1>(X + (k1 << B2) * G::CS + c, G::CS, R.rt + rt_offset(R1, false), k1, v);
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) {
        const uint32_t row = (k1 << B2) + k, f = k1 + (k << B1);
        const uint64_t y = gl::mul(v[k], __ldg(R.lvl + N + f * J));
        cluster_ptr(Y, mine + (row >> (RC)))[(row & ((1u << (RC)) - 1)) * G::YS + J] = y;
      }
    }
  }
  cluster_barrier();
  // pass 2 on the rows; the last round's outputs stay in registers
  constexpr int IT2 = (1 << (RC + D1)) / NT;  // (row, k1) items per thread
  uint64_t s[IT2 << D2];
  static_assert((IT2 * NT) == (1 << (RC + D1)), "rows divide evenly");
  if (!(isb && square)) {
#pragma unroll 1
    for (uint32_t w = t; w < (1u << (RC + D2)); w += NT) {
      const uint32_t jp = w & ((1u << D2) - 1), row = w >> D2;
      uint64_t* y = Y + row * G::YS + jp;
      uint64_t v[1 << D1];
      gl::Lz x[1 << D1];
#pragma unroll
      for (int m = 0; m < (1 << D1); m++) x[m] = gl::lz(y[m << D2]);
      x[0] = gl::lz_bias(x[0]);
      dft_lz<D1, false>(x, v);
#pragma unroll
      for (int k = 0; k < (1 << D1); k++) y[k << D2] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < IT2; it++) {
      const uint32_t w = it * NT + t, k1 = w & ((1u << D1) - 1), row = w >> D1;
      pass_fwd2<R2>(Y + row * G::YS + (k1 << D2), 1, R.rt + rt_offset(R2, false), k1, s + (it << D2));
    }
    if (isb) {
      uint64_t* z = cluster_ptr(Z, rank);
#pragma unroll
      for (int it = 0; it < IT2; it++)
#pragma unroll
        for (int k = 0; k < (1 << D2); k++) z[((it << D2) + k) * NT + t] = gl::mul(s[(it << D2) + k], ninv);
    }
  }
  cluster_barrier();
  if (!isb) {
    // pointwise product and the inverse of pass 2
#pragma unroll
    for (int it = 0; it < IT2; it++) {
      const uint32_t w = it * NT + t, k1 = w & ((1u << D1) - 1), row = w >> D1;
      uint64_t v[1 << D2];
      gl::Lz x[1 << D2];
#pragma unroll
      for (int k = 0; k < (1 << D2); k++) {
        const uint64_t u = s[(it << D2) + k];
        x[k] = gl::lz_mul(u, square ? gl::mul(u, ninv) : Z[((it << D2) + k) * NT + t]);
      }
      x[0] = gl::lz_bias(x[0]);
      dft_lz<D2, true>(x, v);
#pragma unroll
      for (int m = 0; m < (1 << D2); m++) Y[row * G::YS + (k1 << D2) + m] = v[m];
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t w = t; w < (1u << (RC + D2)); w += NT) {
      const uint32_t jp = w & ((1u << D2) - 1), row = w >> D2;
      uint64_t v[1 << D1];
      pass_inv2<R2>(Y + row * G::YS + jp, 1u << D2, R.rt + rt_offset(R2, true), jp, v);
      // columns to the CTAs that own them
      const uint32_t grow = (rank << (RC)) + row;
#pragma unroll
      for (int m = 0; m < (1 << D1); m++) {
        const uint32_t J = (m << D2) + jp;
        cluster_ptr(X, J >> TC)[grow * G::CS + (J & CM)] = v[m];
      }
    }
  }
  cluster_barrier();
  if (!isb) {
    // inverse of pass 1
#pragma unroll 1
    for (uint32_t w = t; w < (1u << (B1 + TC)); w += NT) {
      const uint32_t c = w & CM, k1 = w >> TC, J = col0 + c;
      uint64_t* xc = X + (k1 << B2) * G::CS + c;
      uint64_t v[1 << B2];
      gl::Lz x[1 << B2];
#pragma unroll
      for (int k = 0; k < (1 << B2); k++) {
        const uint32_t e = (k1 + (k << B1)) * J;
        x[k] = gl::lz_mul(xc[k * G::CS], __ldg(R.lvl + N + ((N - e) & (N - 1))));
      }
      x[0] = gl::lz_bias(x[0]);
      dft_lz<B2, true>(x, v);
#pragma unroll
      for (int m = 0; m < (1 << B2); m++) xc[m * G::CS] = v[m];
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t w = t; w < (1u << (B2 + TC)); w += NT) {
      const uint32_t c = w & CM, jp = w >> TC;
      uint64_t v[1 << B1];
      pass_inv2<R1>(X + jp * G::CS + c, G::CS << B2, R.rt + rt_offset(R1, true), jp, v);
      // coefficients in natural order, a quarter per CTA
#pragma unroll
      for (int m = 0; m < (1 << B1); m++) {
        const uint32_t row = (m << B2) + jp;
        const uint32_t n = (row << R2) + col0 + c;
        const uint32_t i = n & (G::WORDS - 1);
        cluster_ptr(Y, n >> (L - G::LOP))[i + (i >> 4)] = gl::canon(v[m]);
      }
    }
  }
  cluster_barrier();
  // carry: windows of 16 coefficients (4 limbs), one per thread
  const uint32_t nl = la + lb, nwin = (4 * nl - 1 + 15) / 16, w = rank * (G::WORDS / 16) + t;
  const bool have = !isb && t < (int)(G::WORDS / 16) && w < nwin;
  Win v{{0, 0, 0, 0}, 0};
  uint64_t hprev = 0;
  if (have) {
    v = fold16(Y + 17 * t, 1);
    Z[t] = v.hi;
    if (t == 0 && rank > 0) hprev = fold16(cluster_ptr(Y, rank - 1) + 17 * (G::WORDS / 16 - 1), 1).hi;
  }
  __syncthreads();
  if (have && t > 0) hprev = Z[t - 1];
  uint64_t s0 = v.l[0] + hprev;
  uint64_t c = s0 < hprev;
  uint64_t s1 = v.l[1] + c;  c = c && s1 == 0;
  uint64_t s2 = v.l[2] + c;  c = c && s2 == 0;
  uint64_t s3 = v.l[3] + c;  c = c && s3 == 0;
  const bool gg = have && c, pp = have && (s0 & s1 & s2 & s3) == ~0ull;
  const uint32_t A = __ballot_sync(0xFFFFFFFFu, gg || pp), B = __ballot_sync(0xFFFFFFFFu, gg);
  if ((t & 31) == 0) sA[t >> 5] = A, sB[t >> 5] = B;
  __syncthreads();
  constexpr int WARPS = ((int)(G::WORDS / 16) + 31) / 32;
  if (!isb && t == 0) {
    uint32_t f = 2; 
    for (int k = 0; k < WARPS; k++) f = cf_then(f, cf_of_masks(sA[k], sB[k]));
    for (uint32_t q = rank + 1; q < G::OP; q++) cluster_ptr(sF, q)[rank] = f;
  }
  cluster_barrier();
  if (have) {
    uint32_t cin = 0;
    for (uint32_t q = 0; q < rank; q++) cin = ((uint32_t)sF[q] >> cin) & 1;
    for (int k = 0; k < (t >> 5); k++) cin = (cf_of_masks(sA[k], sB[k]) >> cin) & 1;
    const uint32_t carries = (A + B + cin) ^ A ^ B;
    if ((carries >> (t & 31)) & 1) {
      if (++s0 == 0) if (++s1 == 0) if (++s2 == 0) ++s3;
    }
    const uint32_t base = 4 * w;
    if (base + 0 < nl) job.out[base + 0] = s0;
    if (base + 1 < nl) job.out[base + 1] = s1;
    if (base + 2 < nl) job.out[base + 2] = s2;
    if (base + 3 < nl) job.out[base + 3] = s3;
  }
}

// ---- merged binary-splitting levels (one node pair per thread group) ------
// The lowest levels of a Chudnovsky splitting segment hold hundreds of
// thousands of node pairs whose products all fit one CTA's shared memory.
// A group of T = N/16 threads merges one pair (L, R) into
//   P = P_L P_R,  Q = Q_L Q_R,  T = T_L Q_R + P_L T_R
// (magnitudes; crates/pi-core/src/algorithm/chudnovsky.rs:377-413).  The
// spectra of Q_R and P_L serve two products each and T's two products are
// added in the transform domain: six forward and three inverse transforms
// per pair instead of eight and four, no temporaries in HBM and no separate
// addition.  Three padded arrays per group, 256 threads and at most 3 * 2^12
// padded words per CTA, two CTAs per SM.  Bound by the integer pipes; against
// radix-8 rounds by N/8 threads, three arrays at a time: pi to 10^8 digits 204.9 ->
// 200.7 ms.
constexpr int MERGE_THREADS = 256;

struct MergeLevel {
  const uint64_t* in;
  const uint32_t* in_len;
  uint64_t* out;
  uint32_t* out_len;
  uint32_t sp, sq, st, op, oq, ot;
  uint32_t n_in;
  int L;
  int* bad;
};

// Threads of a node pair: one radix-16 item (8 at 2^9 points) each, a warp or more.
__host__ __device__ constexpr int merge_group_threads(int L) { return L == 8 ? 32 : small_op_threads(L); }
__host__ __device__ __forceinline__ size_t merge_cta_smem(int L) {
  return (size_t)(MERGE_THREADS / merge_group_threads(L)) * 3 * spad(1u << L) * 8;
}

// Carry normalisation of a group's inverse-transformed array (exact
// convolution values, below 2^45) into nl limbs at out, one 16-coefficient
// window per thread: nl <= N/4 + 1, and a limb past the T windows takes the last
// one's high part and carry.  Returns the trimmed length to every thread of the
// group.  Same window arithmetic as the one-CTA multiply above.
template <int C, int T>
__device__ __forceinline__ uint32_t merge_carry(uint64_t* sm, uint32_t nl, uint64_t* out, int t, int grp, uint32_t* sA,
                                                uint32_t* sBm, uint32_t* sTop) {
  const uint32_t nwin = nl ? (4 * nl + 14) / 16 : 0, w = t;
  Win v{{0, 0, 0, 0}, 0};
  if (w < nwin && w < (1u << C) / 16) {
    uint64_t c[16];
#pragma unroll
    for (int q = 0; q < 16; q++) c[q] = gl::canon(sm[spad(16 * w + q)]);
    v = fold16(c, 1);
  }
  small_sync<T>(grp);
  sm[w] = v.hi;
  small_sync<T>(grp);
  const uint64_t hprev = w > 0 ? sm[w - 1] : 0;
  uint64_t s0 = v.l[0] + hprev;
  uint64_t c = s0 < hprev;
  uint64_t s1 = v.l[1] + c;  c = c && s1 == 0;
  uint64_t s2 = v.l[2] + c;  c = c && s2 == 0;
  uint64_t s3 = v.l[3] + c;  c = c && s3 == 0;
  const bool gg = w < nwin && c;
  const bool pp = w < nwin && (s0 & s1 & s2 & s3) == ~0ull;
  const uint32_t A = __ballot_sync(0xFFFFFFFFu, gg || pp), Bm = __ballot_sync(0xFFFFFFFFu, gg);
  const int gw0 = grp * (T / 32), gw = gw0 + (t >> 5);
  uint32_t cin = 0;
  if constexpr (T > 32) {
    if ((t & 31) == 0) sA[gw] = A, sBm[gw] = Bm;
    small_sync<T>(grp);
    for (int k = gw0; k < gw; k++) {
      const uint64_t x = (uint64_t)sA[k] + sBm[k] + cin;
      cin = (uint32_t)(x >> 32);
    }
  }
  const bool in = (((A + Bm + cin) ^ A ^ Bm) >> (t & 31)) & 1;
  if (in) {
    if (++s0 == 0) if (++s1 == 0) if (++s2 == 0) ++s3;
  }
  uint32_t top = 0;
  if (w < nwin) {
    const uint64_t s[4] = {s0, s1, s2, s3};
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (4 * w + q < nl) {
        out[4 * w + q] = s[q];
        if (s[q]) top = 4 * w + q + 1;
      }
    if (w == T - 1 && nwin > T) {
      const uint64_t last = v.hi + (gg || (pp && in));
      out[4 * T] = last;
      if (last) top = 4 * T + 1;
    }
  }
  top = __reduce_max_sync(0xFFFFFFFFu, top);
  if constexpr (T > 32) {
    if ((t & 31) == 0) sTop[gw] = top;
    small_sync<T>(grp);
    for (int k = gw0; k < gw0 + T / 32; k++) top = max(top, sTop[k]);
  }
  small_sync<T>(grp);
  return top;
}

// One node pair by a group of T threads.  Every pair of the level runs transforms
// of 2^L points (a pair that needs fewer gets a longer transform, which changes
// nothing).  The six operands go through one forward transform in a loop (six
// copies of it would not fit the instruction caches), a thread's part of the
// spectrum in registers: Q_R's and P_L's, times N^-1, stay in keep for the
// products that share them, T_L Q_R waits in acc (both read by the thread that
// wrote them).
template <int L>
__device__ __forceinline__ void merge_pair(const MergeLevel& M, const Roots& R, uint32_t item, uint64_t* work, uint64_t* acc,
                                           uint64_t* keep, int t, int grp, uint32_t* sA, uint32_t* sBm, uint32_t* sTop) {
  constexpr int T = merge_group_threads(L), G = small_op_threads(L);
  constexpr int BL = small_b(L, 2) ? small_b(L, 2) : small_b(L, 1), ITL = (1 << (L - BL)) / G;
  constexpr uint32_t N = 1u << L;
  const size_t in_stride = (size_t)M.sp + M.sq + M.st, out_stride = (size_t)M.op + M.oq + M.ot;
  const uint32_t* len = M.in_len + 6 * (size_t)item;  // P, Q, T of the left node, then the right one
  const uint64_t* node = M.in + 2 * (size_t)item * in_stride;
  const uint32_t pl = len[0], ql = len[1], tl = len[2], pr = len[3], qr = len[4], tr = len[5];
  const uint32_t n_p = pl + pr, n_q = ql + qr, n_t = max(tl + qr, pl + tr) + 1;
  // output coefficients of the longest product: 4 len - 1 <= 2^L
  const uint32_t need = max(max(n_p, n_q), max(tl + qr, pl + tr));
  if (!(4ull * need <= N + 1ull && n_p <= M.op && n_q <= M.oq && n_t <= M.ot)) {
    if (t == 0) atomicExch(M.bad, 1);
    return;
  }
  // N^-1 = 2^-L = p - (2^(64-L) - 2^(32-L))  (2^96 = -1, 2^64 = 2^32 - 1)
  constexpr uint64_t ninv = gl::P - ((1ull << (64 - L)) - (1ull << (32 - L)));
  const bool run = T == G || t < G;
#pragma unroll 1
  for (int step = 0; step < 6; step++) {
    // Q_R, T_L, Q_L, P_L, T_R, P_R
    const int right = (0x31 >> step) & 1, kind = (0x0219 >> (2 * step)) & 3;
    const uint64_t* x = node + (right ? in_stride : 0) + (kind > 0 ? M.sp : 0) + (kind > 1 ? M.sq : 0);
    uint64_t s[ITL << BL];
    small_forward<L, T>(x, 4 * len[3 * right + kind], R, work, t, grp, run, s);
    if (step == 0 || step == 3) {
      if (run) {
#pragma unroll
        for (int it = 0; it < ITL; it++)
#pragma unroll
          for (int k = 0; k < (1 << BL); k++) keep[spad(((it * G + t) << BL) + k)] = gl::mul(s[(it << BL) + k], ninv);
      }
      small_sync<T>(grp);
      continue;
    }
    if (step == 1) {
      if (run) {
#pragma unroll
        for (int it = 0; it < ITL; it++)
#pragma unroll
          for (int k = 0; k < (1 << BL); k++) {
            const uint32_t i = spad(((it * G + t) << BL) + k);
            acc[i] = gl::mul(s[(it << BL) + k], keep[i]);
          }
      }
      small_sync<T>(grp);
      continue;
    }
    if (run) {
#pragma unroll
      for (int it = 0; it < ITL; it++) {
        const uint32_t base = (it * G + t) << BL;
        uint64_t v[1 << BL];
        gl::Lz y[1 << BL];
#pragma unroll
        for (int k = 0; k < (1 << BL); k++) v[k] = gl::mul(s[(it << BL) + k], keep[spad(base + k)]);
        if (step == 4) {
#pragma unroll
          for (int k = 0; k < (1 << BL); k++) v[k] = gl::add(v[k], acc[spad(base + k)]);
        }
#pragma unroll
        for (int k = 0; k < (1 << BL); k++) y[k] = gl::lz(v[k]);
        y[0] = gl::lz_bias(y[0]);
        dft_lz<BL, true>(y, v);
#pragma unroll
        for (int m = 0; m < (1 << BL); m++) work[spad(base + m)] = v[m];
      }
    }
    small_inverse<L, T>(R, work, t, grp);
    const uint32_t off = step == 2 ? M.op : step == 4 ? M.op + M.oq : 0;
    const uint32_t n = merge_carry<L, T>(work, step == 2 ? n_q : step == 4 ? n_t : n_p, M.out + item * out_stride + off, t, grp,
                                         sA, sBm, sTop);
    if (t == 0) M.out_len[3 * (size_t)item + (step == 2 ? 1 : step == 4 ? 2 : 0)] = n;
  }
}

// Persistent over the level's items (pairs, then the odd last node), each by
// one of the MERGE_THREADS / T groups of a CTA.  8 <= L <= 12.
template <int L>
__global__ void __launch_bounds__(MERGE_THREADS, 2) k_split_merge(MergeLevel M, Roots R) {
  extern __shared__ uint64_t sm[];
  __shared__ uint32_t sA[MERGE_THREADS / 32], sBm[MERGE_THREADS / 32], sTop[MERGE_THREADS / 32];
  constexpr int T = merge_group_threads(L);
  constexpr uint32_t gpc = MERGE_THREADS / T, words = spad(1u << L);
  const uint32_t grp = threadIdx.x / T;
  const int t = (int)(threadIdx.x % T);
  const uint32_t np = M.n_in / 2, items = np + (M.n_in & 1);
  uint64_t* work = sm + (size_t)grp * 3 * words;
  for (uint32_t item = blockIdx.x * gpc + grp; item < items; item += gridDim.x * gpc) {
    if (item < np) {
      merge_pair<L>(M, R, item, work, work + words, work + 2 * words, t, (int)grp, sA, sBm, sTop);
      continue;
    }
    // the odd last node is copied
    const uint32_t i = M.n_in - 1;
    const uint64_t* p = M.in + (size_t)i * ((size_t)M.sp + M.sq + M.st);
    uint64_t* z = M.out + (size_t)item * ((size_t)M.op + M.oq + M.ot);
    const uint32_t pn = M.in_len[3 * i], qn = M.in_len[3 * i + 1], tn = M.in_len[3 * i + 2];
    for (uint32_t k = t; k < pn; k += T) z[k] = p[k];
    for (uint32_t k = t; k < qn; k += T) z[M.op + k] = p[M.sp + k];
    for (uint32_t k = t; k < tn; k += T) z[M.op + M.oq + k] = p[M.sp + M.sq + k];
    if (t == 0) {
      M.out_len[3 * item] = pn;
      M.out_len[3 * item + 1] = qn;
      M.out_len[3 * item + 2] = tn;
    }
  }
}

// ------------------------------------------------------------------ host side
static int log2_ceil(uint64_t x) { return x <= 1 ? 0 : 64 - __builtin_clzll(x - 1); }

// Host copies of the root tables: lo, hi, w12, level tables (in this order).
constexpr size_t ROOT_WORDS = 2 * 65536 + 4096 + (2u << LVL_MAX) + (size_t)NEAR_LEVELS * 2 * 4096 + RT_WORDS + RT3_WORDS;

static void build_roots(uint64_t* t) {
  uint64_t rho = find_rho();
  uint64_t* lo = t;
  uint64_t* hi = lo + 65536;
  uint64_t* w12 = hi + 65536;
  uint64_t* lvl = w12 + 4096;
  uint64_t x = 1;
  for (int i = 0; i < 65536; i++) { lo[i] = x; x = hf::mul(x, rho); }
  uint64_t step = x;  // rho^(2^16)
  x = 1;
  for (int i = 0; i < 65536; i++) { hi[i] = x; x = hf::mul(x, step); }
  uint64_t w4096 = hf::pow(rho, 1ull << 20);
  x = 1;
  for (int i = 0; i < 4096; i++) { w12[i] = x; x = hf::mul(x, w4096); }
  // level k (1 <= k <= LVL_MAX): w_(2^k)^x at lvl[2^k + x]; level k is every
  // other entry of level k+1, starting from the longest
  const uint32_t top = 1u << LVL_MAX;
  uint64_t wm = hf::pow(rho, 1ull << (32 - LVL_MAX));
  x = 1;
  for (uint32_t i = 0; i < top; i++) { lvl[top + i] = x; x = hf::mul(x, wm); }
  for (int k = LVL_MAX - 1; k >= 1; k--)
    for (uint32_t i = 0; i < (1u << k); i++) lvl[(1u << k) + i] = lvl[(2u << k) + 2 * i];
  lvl[0] = lvl[1] = 1;
  // near tables: w_(2^L)^(+-x) = rho^(+-x 2^(32-L)) for x < 4096
  uint64_t* nt = lvl + (2u << LVL_MAX);
  for (int L = LVL_MAX + 1; L <= 32; L++)
    for (int dir = 0; dir < 2; dir++)
      for (uint32_t xx = 0; xx < 4096; xx++) {
        const uint32_t e0 = (uint32_t)((uint64_t)xx << (32 - L));
        const uint32_t e = dir ? 0u - e0 : e0;
        nt[((size_t)(L - LVL_MAX - 1) * 2 + dir) * 4096 + xx] = hf::mul(lo[e & 0xFFFFu], hi[e >> 16]);
      }
  // round twiddles of the passes
  uint64_t* rt = nt + (size_t)NEAR_LEVELS * 2 * 4096;
  for (int r = 5; r <= 9; r++) {
    const uint64_t* w = lvl + (1u << r);
    const uint32_t n1 = 1u << pass_b1(r), n2 = 1u << pass_b2(r), n = 1u << r;
    for (uint32_t k = 0; k < n1; k++)
      for (uint32_t m = 0; m < n2; m++) {
        rt[rt_offset(r, false) + m * n1 + k] = w[k * m];
        rt[rt_offset(r, true) + k * n2 + m] = w[(n - k * m) & (n - 1)];
      }
  }
  uint64_t* rt3 = rt + RT_WORDS;
  for (uint32_t k = 0; k < 16; k++)
    for (uint32_t m = 0; m < 12; m++) {
      rt3[m * 16 + k] = hf::pow(2, k * m);
      rt3[192 + k * 12 + m] = hf::pow(2, 192 - k * m);
    }
}

static Roots roots_at(const uint64_t* d) {
  const uint64_t* nt = d + 2 * 65536 + 4096 + (2u << LVL_MAX);
  return Roots{d, d + 65536, d + 2 * 65536, d + 2 * 65536 + 4096, nt, nt + (size_t)NEAR_LEVELS * 2 * 4096};
}

struct DeviceState {
  int device = -1;
  bool ready = false;
  int lone_log = SMALL_LOG_MAX;  // longest transform (log2) of a lone product in one cluster
  uint64_t* d_roots = nullptr;
  Roots roots{};
  cudaMemPool_t pool = nullptr;
};

static std::mutex g_mu;
static DeviceState g_dev;
static thread_local cudaStream_t t_stream = nullptr;
static thread_local int t_stream_dev = -1;

// Opt the short products', cluster and merge kernels into their dynamic shared
// memory (the pass kernels stay below 48 KB) and the sixteen-CTA clusters into
// their size.
static cudaError_t set_smem_attrs() {
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_small_mul, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_cta_smem(SMALL_LOG_MAX));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cluster_mul<11, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, ClusterGeom<11>::SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cluster_mul<12>, cudaFuncAttributeMaxDynamicSharedMemorySize, ClusterGeom<12>::SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cluster_mul<13>, cudaFuncAttributeMaxDynamicSharedMemorySize, ClusterGeom<13>::SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cluster_mul<13>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cluster_mul<14>, cudaFuncAttributeMaxDynamicSharedMemorySize, ClusterGeom<14>::SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_cluster_mul<14>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_split_merge<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)merge_cta_smem(8));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_split_merge<9>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)merge_cta_smem(9));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_split_merge<10>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)merge_cta_smem(10));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_split_merge<11>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)merge_cta_smem(11));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_split_merge<12>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)merge_cta_smem(12));
  return e;
}

// Longest transform (log2) that a lone product runs within a cluster here.  From
// 2^13 points on that takes sixteen CTAs, more than every GPU or partition of one
// need be able to place at once; where they cannot be (or PIMUL_WIDE_CLUSTERS=0
// says so) those lengths take the passes.
template <int L>
static bool wide_cluster_fits() {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(2 * ClusterGeom<L>::OP);
  c.blockDim = dim3(ClusterGeom<L>::NT);
  c.dynamicSmemBytes = ClusterGeom<L>::SMEM;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 2 * ClusterGeom<L>::OP;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k_cluster_mul<L>, &c) == cudaSuccess) return n > 0;
  cudaGetLastError();
  return false;
}
static int lone_log_here() {
  const char* e = getenv("PIMUL_WIDE_CLUSTERS");
  if (e && atoi(e) == 0) return SMALL_LOG_MAX;
  return !wide_cluster_fits<13>() ? SMALL_LOG_MAX : wide_cluster_fits<14>() ? CLUSTER_LOG_MAX : 13;
}

static int ensure_init(int device) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_dev.ready) {
    if (device >= 0 && device != g_dev.device)
      return fail(PIMUL_EINVAL, "pimul already initialised on another device");
    return PIMUL_OK;
  }
  if (device < 0) device = 0;
  CU(cudaSetDevice(device));
  std::vector<uint64_t> tables(ROOT_WORDS);
  build_roots(tables.data());
  CU(cudaMalloc(&g_dev.d_roots, ROOT_WORDS * 8));
  CU(cudaMemcpy(g_dev.d_roots, tables.data(), ROOT_WORDS * 8, cudaMemcpyHostToDevice));
  g_dev.roots = roots_at(g_dev.d_roots);
  CU(cudaDeviceGetDefaultMemPool(&g_dev.pool, device));
  uint64_t thr = UINT64_MAX;  // keep freed blocks cached in the pool
  CU(cudaMemPoolSetAttribute(g_dev.pool, cudaMemPoolAttrReleaseThreshold, &thr));
  CU(set_smem_attrs());
  g_dev.lone_log = lone_log_here();
  g_dev.device = device;
  g_dev.ready = true;
  return PIMUL_OK;
}

static int get_stream(cudaStream_t* s) {
  int rc = ensure_init(-1);
  if (rc) return rc;
  if (!t_stream || t_stream_dev != g_dev.device) {
    CU(cudaSetDevice(g_dev.device));
    CU(cudaStreamCreateWithFlags(&t_stream, cudaStreamNonBlocking));
    t_stream_dev = g_dev.device;
  }
  CU(cudaSetDevice(g_dev.device));
  *s = t_stream;
  return PIMUL_OK;
}

// ------------------------------------------------------------- host copies
// cudaMemcpy from or to PAGEABLE host memory (the limb arrays of a host
// driver) runs through the driver's bounce buffer at a few GB/s.  From 1 MiB
// up such copies are staged instead: host threads copy 32 MiB chunks into
// one of two pinned buffers while the copy engine drains (or fills) the
// other.  Pinned or registered host memory is copied directly.
constexpr size_t STAGE_MIN = (size_t)1 << 20;
constexpr size_t STAGE_CHUNK = (size_t)32 << 20;

// memcpy on all host cores: a fixed set of workers, one copy at a time.
class CopyPool {
 public:
  void copy(void* dst, const void* src, size_t bytes) {
    std::call_once(once_, [this] { start(); });
    if (bytes < ((size_t)4 << 20) || workers_ == 0) {
      memcpy(dst, src, bytes);
      return;
    }
    std::lock_guard<std::mutex> run(run_mu_);
    {
      std::lock_guard<std::mutex> lk(mu_);
      dst_ = static_cast<char*>(dst);
      src_ = static_cast<const char*>(src);
      bytes_ = bytes;
      pending_ = workers_;
      gen_++;
    }
    cv_.notify_all();
    part(0);
    std::unique_lock<std::mutex> lk(mu_);
    done_.wait(lk, [this] { return pending_ == 0; });
  }

 private:
  void start() {
    unsigned hw = std::thread::hardware_concurrency();
    workers_ = (int)std::min(hw ? hw : 1u, 16u) - 1;
    for (int i = 0; i < workers_; i++) std::thread([this, i] { run(i + 1); }).detach();
  }
  void part(int id) {
    const size_t n = (size_t)workers_ + 1;
    const size_t per = ((bytes_ + n - 1) / n + 63) & ~(size_t)63;
    const size_t lo = std::min(bytes_, per * id), hi = std::min(bytes_, lo + per);
    if (hi > lo) memcpy(dst_ + lo, src_ + lo, hi - lo);
  }
  void run(int id) {
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return gen_ != seen; });
        seen = gen_;
      }
      part(id);
      std::lock_guard<std::mutex> lk(mu_);
      if (--pending_ == 0) done_.notify_one();
    }
  }
  std::once_flag once_;
  std::mutex run_mu_, mu_;
  std::condition_variable cv_, done_;
  int workers_ = 0, pending_ = 0;
  uint64_t gen_ = 0;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t bytes_ = 0;
};
static CopyPool& copy_pool() {
  static CopyPool* p = new CopyPool;  // workers are detached: never destroyed
  return *p;
}

struct StageBuf {
  void* h[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};  // last copy-engine use of h[j]
  int device = -1;
};
static std::mutex g_stage_mu;
static std::vector<StageBuf*> g_stage_free, g_stage_all;

static StageBuf* stage_acquire() {
  int dev = 0;
  cudaGetDevice(&dev);
  {
    // a free buffer whose last copies are done, else (up to four buffers
    // per device) a new one, else any free one: the caller would wait for
    // a busy buffer's copies, i.e. for the work queued before them
    std::lock_guard<std::mutex> lk(g_stage_mu);
    int any = -1, mine = 0;
    for (StageBuf* x : g_stage_all) mine += x->device == dev;
    for (size_t i = 0; i < g_stage_free.size(); i++) {
      StageBuf* x = g_stage_free[i];
      if (x->device != dev) continue;
      if (any < 0) any = (int)i;
      if (cudaEventQuery(x->ev[0]) == cudaSuccess && cudaEventQuery(x->ev[1]) == cudaSuccess) {
        g_stage_free.erase(g_stage_free.begin() + i);
        return x;
      }
    }
    cudaGetLastError();  // cudaEventQuery's cudaErrorNotReady
    if (any >= 0 && mine >= 4) {
      StageBuf* x = g_stage_free[any];
      g_stage_free.erase(g_stage_free.begin() + any);
      return x;
    }
  }
  StageBuf* b = new StageBuf;
  b->device = dev;
  for (int j = 0; j < 2; j++) {
    if (cudaHostAlloc(&b->h[j], STAGE_CHUNK, cudaHostAllocPortable) != cudaSuccess ||
        cudaEventCreateWithFlags(&b->ev[j], cudaEventDisableTiming) != cudaSuccess) {
      cudaGetLastError();
      for (int k = 0; k < 2; k++) {
        if (b->h[k]) cudaFreeHost(b->h[k]);
        if (b->ev[k]) cudaEventDestroy(b->ev[k]);
      }
      delete b;
      return nullptr;
    }
  }
  std::lock_guard<std::mutex> lk(g_stage_mu);
  g_stage_all.push_back(b);
  return b;
}
static void stage_release(StageBuf* b) {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  g_stage_free.push_back(b);
}

// Uploads below STAGE_MIN from pageable memory go through a ring of small
// pinned slots: a plain cudaMemcpyAsync from pageable memory synchronises
// its stream first, so every batch call (its descriptor image) would wait
// for the work already queued instead of preparing the next launch.
constexpr int RING_SLOTS = 16;
struct SmallRing {
  std::mutex mu;
  void* h[RING_SLOTS] = {};
  cudaEvent_t ev[RING_SLOTS] = {};  // the last copy from each slot
  int next = 0;
  int device = -1;
  bool ok = false;
};
static SmallRing& small_ring() {
  static SmallRing* r = new SmallRing;  // pinned slots live until exit
  return *r;
}

static bool is_pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// A small pageable upload through the ring; false when the ring cannot be
// set up (the caller then copies directly).
// A second piece src2 goes to dst + off2 in the same copy.
static bool ring_upload(void* dst, const void* src, size_t bytes, cudaStream_t st, cudaError_t* err,
                        const void* src2 = nullptr, size_t off2 = 0, size_t bytes2 = 0) {
  SmallRing& r = small_ring();
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(r.mu);
  if (r.device != dev) {
    if (r.device >= 0) return false;  // set up on another device
    for (int k = 0; k < RING_SLOTS; k++)
      if (cudaHostAlloc(&r.h[k], STAGE_MIN, cudaHostAllocPortable) != cudaSuccess ||
          cudaEventCreateWithFlags(&r.ev[k], cudaEventDisableTiming) != cudaSuccess) {
        cudaGetLastError();
        r.device = dev;
        r.ok = false;
        return false;
      }
    r.device = dev;
    r.ok = true;
  }
  if (!r.ok) return false;
  const int k = r.next;
  r.next = (k + 1) % RING_SLOTS;
  cudaError_t e = cudaEventSynchronize(r.ev[k]);  // the copy RING_SLOTS uploads ago is done
  if (e == cudaSuccess) {
    memcpy(r.h[k], src, bytes);
    if (bytes2) memcpy(static_cast<char*>(r.h[k]) + off2, src2, bytes2);
    e = cudaMemcpyAsync(dst, r.h[k], bytes2 ? off2 + bytes2 : bytes, cudaMemcpyHostToDevice, st);
  }
  if (e == cudaSuccess) e = cudaEventRecord(r.ev[k], st);
  *err = e;
  return true;
}

int host_to_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (!bytes) return PIMUL_OK;
  const bool pageable = is_pageable(src);
  if (pageable && bytes < STAGE_MIN) {
    cudaError_t e = cudaSuccess;
    if (ring_upload(dst, src, bytes, st, &e)) {
      if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("small upload: ") + cudaGetErrorString(e));
      return PIMUL_OK;
    }
  }
  StageBuf* b = bytes >= STAGE_MIN && pageable ? stage_acquire() : nullptr;
  if (!b) {
    CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
    return PIMUL_OK;
  }
  cudaError_t e = cudaSuccess;
  int j = 0;
  for (size_t off = 0; off < bytes && e == cudaSuccess; off += STAGE_CHUNK, j ^= 1) {
    const size_t n = std::min(STAGE_CHUNK, bytes - off);
    e = cudaEventSynchronize(b->ev[j]);  // the copy engine is done with h[j]
    if (e != cudaSuccess) break;
    copy_pool().copy(b->h[j], static_cast<const char*>(src) + off, n);
    e = cudaMemcpyAsync(static_cast<char*>(dst) + off, b->h[j], n, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaEventRecord(b->ev[j], st);
  }
  stage_release(b);
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("staged upload: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}

int device_to_host(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  if (!bytes) return PIMUL_OK;
  const bool pageable = is_pageable(dst);
  StageBuf* b = bytes >= STAGE_MIN && pageable ? stage_acquire() : nullptr;
  if (!b) {
    // The GPU writes pageable memory through the host's page tables, and takes
    // a fault per page of a fresh array (150 us for 520 KB, 13 without): touch
    // the pages while the work in front of the copy runs.
    if (pageable)
      for (size_t i = 0; i < bytes; i += 4096) {
        volatile char* p = static_cast<char*>(dst) + i;
        *p = *p;
      }
    CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    return PIMUL_OK;
  }
  const size_t nch = (bytes + STAGE_CHUNK - 1) / STAGE_CHUNK;
  auto issue = [&](size_t i) {
    const size_t off = i * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - off);
    const int j = (int)(i & 1);
    cudaError_t e = cudaEventSynchronize(b->ev[j]);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(b->h[j], static_cast<const char*>(src) + off, n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaEventRecord(b->ev[j], st);
    return e;
  };
  cudaError_t e = issue(0);
  for (size_t i = 0; i < nch && e == cudaSuccess; i++) {
    // chunk i + 1 lands in the other buffer while chunk i is copied out
    if (i + 1 < nch) e = issue(i + 1);
    if (e == cudaSuccess) e = cudaEventSynchronize(b->ev[i & 1]);
    if (e != cudaSuccess) break;
    const size_t off = i * STAGE_CHUNK, n = std::min(STAGE_CHUNK, bytes - off);
    copy_pool().copy(static_cast<char*>(dst) + off, b->h[i & 1], n);
  }
  stage_release(b);
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("staged download: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}

int set_error(int code, const char* msg) { return fail(code, msg); }

void release_host_staging() {
  std::lock_guard<std::mutex> lk(g_stage_mu);
  for (StageBuf* b : g_stage_all) {
    for (int j = 0; j < 2; j++) {
      cudaEventSynchronize(b->ev[j]);
      cudaEventDestroy(b->ev[j]);
      cudaFreeHost(b->h[j]);
    }
    delete b;
  }
  g_stage_all.clear();
  g_stage_free.clear();
  SmallRing& r = small_ring();
  std::lock_guard<std::mutex> rl(r.mu);
  for (int k = 0; k < RING_SLOTS; k++) {
    if (r.ev[k]) {
      cudaEventSynchronize(r.ev[k]);
      cudaEventDestroy(r.ev[k]);
    }
    if (r.h[k]) cudaFreeHost(r.h[k]);
    r.ev[k] = nullptr;
    r.h[k] = nullptr;
  }
  r.device = -1;
  r.ok = false;
  r.next = 0;
}

// L bits split into np HBM passes of radix 2^r[0] .. 2^r[np - 1].
struct Plan {
  int L;
  int np;
  int r[5];  // (r[0] unused for a length of 3 2^k points)
};

// Transform lengths: 2^L as L, 3 2^k as THREE + k (3 2^13 .. 3 2^15 and 3 2^17 ..
// 3 2^24 points have passes).
constexpr int THREE = 64;
constexpr int N_LENGTHS = THREE + 33;
// Points of 2^L that must be there for a batch to run them at 3 2^(L-2) beside
// others of 2^L: six to nine launches more against a quarter of the work (2^20
// .. 2^23: 4096 uneven products within 0.3 %, 512 short ones 616 us at 2^20, 593
// from 2^22 on; 2^24: 7.17 against 6.99 ms).
constexpr uint64_t THREE_SPLIT = 1ull << 22;
static bool is_three(int L) { return L >= THREE; }
// Whether 3 2^(L-2) points hold n coefficients and have passes.
static bool three_holds(uint64_t n, int L) {
  const int k = L - 2;
  return k >= 13 && k != 16 && k <= 24 && n <= 3ull << k;
}
static uint64_t length_words(int L) { return is_three(L) ? 3ull << (L - THREE) : 1ull << L; }

// Pass-count override per L chosen by the autotuner (0 = default).
static std::atomic<int> g_tuned_np[33];
// Persistent grid of the short products' kernel in a batch: CTAs per SM (autotuned).
static std::atomic<int> g_small_ctas_per_sm{4};

static int default_np(int L) {
  int np = (L + 8) / 9;
  return np < 2 ? 2 : np;
}

static bool plan_valid(const Plan& p) { return p.np != 0; }

// The splits.  Three passes: measured per length, the short radices first (a
// lone 2^20-point product takes 49.6 us as 6 + 6 + 8, 52.9 as 7 + 7 + 6; 2^21
// points 84.8 as 7 + 6 + 8, 87.7 as 7 + 7 + 7, 88.4 as 6 + 6 + 9; 2^25 points
// 1285 as 8 + 8 + 9, 1301 as 9 + 8 + 8).  Two passes: even, the longer first (16
// products of 2^15 points: 40.0 us as 8 + 7, 43.5 as 7 + 8, 45.3 as 6 + 9).  Four
// and five: even, the longer last.  np passes must leave radices of 2^6 .. 2^9 and
// one of at least 2^7; an invalid plan (np 0) for anything else.  (make_plan's
// three passes for few transforms of 2^17 or 2^18 points are not among these.)
static Plan make_plan_np(int L, int np) {
  Plan p{L, 0, {0, 0, 0, 0, 0}};
  if (np < 2 || np > 5 || L < 6 * np + 1 || L > 9 * np) return p;
  p.np = np;
  static const int three[9][3] = {{6, 6, 7}, {6, 6, 8}, {7, 6, 8}, {6, 8, 8}, {7, 8, 8}, {8, 8, 8}, {8, 8, 9}, {8, 9, 9}, {9, 9, 9}};
  for (int i = 0; i < np; i++) {
    const int from = np == 2 ? i : np - 1 - i;
    p.r[i] = np == 3 ? three[L - 19][i] : L / np + (from < L % np ? 1 : 0);
  }
  return p;
}

// The plan for transforms of 2^L points, `points` of them in all: few of 2^17 or
// 2^18 points run three short passes, whose threads hold 8 elements, where two
// leave a warp or less per SM sub-partition with 32 elements a thread.  2^18
// points: a lone product 31.0 us against 45.0, four 59.6 against 65.7, eight 90.8
// against 82.3; 2^17 points: a lone one 26.7 against 35.9, two 39.1 against 45.3, four
// 48.5 against 46.9.  A tuned count is for more than those: two passes are all it can
// say at these lengths.
static Plan make_plan(int L, uint64_t points = ~0ull) {
  if (is_three(L)) {
    // 192 rows, then 2^S points in one pass or two, the shorter first
    const int S = L - THREE - 6;
    if (S <= 9) return Plan{L, 2, {0, S, 0, 0, 0}};
    const int r1 = S <= 14 ? 6 : S / 2;
    return Plan{L, 3, {0, r1, S - r1, 0, 0}};
  }
  if (L == 17 && points <= 1ull << 18) return Plan{L, 3, {6, 6, 5, 0, 0}};
  if (L == 18 && points <= 1ull << 20) return Plan{L, 3, {6, 6, 6, 0, 0}};
  int np = (L >= 0 && L <= 32) ? g_tuned_np[L].load(std::memory_order_relaxed) : 0;
  if (np) {
    Plan p = make_plan_np(L, np);
    if (plan_valid(p)) return p;
  }
  return make_plan_np(L, default_np(L));
}

struct Sizes {
  uint64_t n_out, N, nwin, nchunk;
  int L;
};

static Sizes sizes_for(uint64_t la, uint64_t lb) {
  Sizes z;
  z.n_out = 4 * la + 4 * lb - 1;
  z.L = log2_ceil(z.n_out);
  z.N = 1ull << z.L;
  z.nwin = n_windows(la, lb);
  z.nchunk = n_chunks(z.nwin);
  return z;
}

// Products of a long operand by a short one are cut into segments (overlap-save):
// a transform of N points over N - 8 wlo new coefficients of the long operand
// and the 8 wlo >= 4 lb - 1 before them gives N - 8 wlo exact coefficients of the
// product (the first 8 wlo values have wrapped around), and all segments share
// the short operand's spectrum: 2 S + 1 transforms of a length near the short
// operand's instead of 3 of a length above the sum.  The cost of a transform
// is taken as N (30 passes + 5.5 log2 N), from the kernels' times per point
// (2 passes, 2^18 points: 8.0 us forward and 10.7 us inverse per 2^20 points; 3
// passes, 2^24 points: 11.7 and 13.5).  Cut only where that saves a tenth.
struct SegPlan {
  int L = 0;          // transform length of a segment (0: not cut)
  uint32_t S = 0;     // segments
  uint64_t wlo = 0;   // windows of the overlap
  uint64_t segv = 0;  // new coefficients per segment
};
constexpr uint32_t SEG_MAX = 8192;

static double transform_cost(int L) {
  static const std::vector<double> table = [] {
    std::vector<double> t(33);
    for (int l = 0; l <= 32; l++) t[l] = (double)(1ull << l) * (30.0 * default_np(l) + 5.5 * l);
    return t;
  }();
  return table[L];
}

static SegPlan plan_segments(uint64_t la, uint64_t lb) {
  SegPlan best;
  if (la < lb) std::swap(la, lb);
  const Sizes z = sizes_for(la, lb);
  if (z.L <= SMALL_LOG_MAX + 1 || z.L > 32 || la < 2 * lb) return best;
  double cost = 0.9 * 3 * transform_cost(z.L) * (three_holds(z.n_out, z.L) ? 0.8 : 1.0);
  const uint64_t wlo = (4 * lb - 1 + WIN_COEFFS - 1) / WIN_COEFFS;
  for (int L = SMALL_LOG_MAX + 1; L < z.L; L++) {
    const uint64_t N = 1ull << L;
    if (2 * WIN_COEFFS * wlo > N) continue;
    const uint64_t v = N - WIN_COEFFS * wlo, S = (z.n_out + v - 1) / v;
    if (S > SEG_MAX) continue;
    const double c = (double)(2 * S + 1) * transform_cost(L);
    if (c < cost) {
      cost = c;
      best.L = L, best.S = (uint32_t)S, best.wlo = wlo, best.segv = v;
    }
  }
  return best;
}

// Scratch bytes of one large product, each piece rounded to 256 bytes: A, B
// (whose words hold the windows' low parts once the spectra are multiplied;
// a square allots just those), and the carry scratch.
static uint64_t round256(uint64_t x) { return (x + 255) & ~255ull; }
__host__ __device__ __forceinline__ uint64_t round_up_u64(uint64_t x, uint64_t m) { return (x + m - 1) / m * m; }
static uint64_t scratch_bytes(uint64_t la, uint64_t lb, bool square) {
  Sizes z = sizes_for(la, lb);
  const SegPlan sg = square ? SegPlan{} : plan_segments(la, lb);
  if (sg.L) return ((uint64_t)(sg.S + 1) << sg.L) * 8 + round256(z.nwin * 16) + round256(carry_words(z.nwin) * 8);
  return round256(z.N * 8) + round256(square ? z.nwin * 16 : z.N * 8) + round256(carry_words(z.nwin) * 8);
}
// Device memory that a pipeline product of a batch takes at most, descriptors
// included, whatever it is batched with: whole, or cut, which it is not where
// another product of the batch has the same b.  (One that lends its spectrum
// holds the windows' low parts, at most N/4 words, apart, and the one that
// borrows it has N words less.)
static uint64_t batch_bytes(uint64_t la, uint64_t lb) {
  const Sizes z = sizes_for(la, lb);
  const SegPlan sg = plan_segments(la, lb);
  const uint64_t carry = round256(carry_words(z.nwin) * 8);
  const uint64_t cut = sg.L ? ((uint64_t)(sg.S + 1) << sg.L) * 8 + round256(z.nwin * 16) + sg.S * sizeof(Job) : 0;
  return std::max(2 * round256(z.N * 8) + sizeof(Job), cut) + carry;
}
static void carve_carry(Job& J, uint64_t* base, uint64_t nwin) {
  J.H = base;
  J.state = reinterpret_cast<uint32_t*>(base + nwin);
}
static void carve_scratch(Job& J, uint8_t* base, bool square) {
  Sizes z = sizes_for(J.la, J.lb);
  J.A = reinterpret_cast<uint64_t*>(base);
  if (J.segments) {
    const uint64_t N = J.segv + WIN_COEFFS * (uint64_t)J.wlo;
    J.B = J.A + J.segments * N;
    base += (J.segments + 1) * N * 8;
    J.W = reinterpret_cast<uint64_t*>(base);
    carve_carry(J, reinterpret_cast<uint64_t*>(base + round256(z.nwin * 16)), z.nwin);
    return;
  }
  base += round256(z.N * 8);
  J.W = reinterpret_cast<uint64_t*>(base);
  J.B = square ? nullptr : J.W;
  base += round256(square ? z.nwin * 16 : z.N * 8);
  carve_carry(J, reinterpret_cast<uint64_t*>(base), z.nwin);
}

// Launch helpers (template dispatch on the pass radix; a last pass may be 2^5).
#define PIMUL_DISPATCH_ROW(r, ...)                      \
  if ((r) == 5) { constexpr int RR = 5; __VA_ARGS__; } else PIMUL_DISPATCH_R(r, __VA_ARGS__)
#define PIMUL_DISPATCH_R(r, ...)                        \
  switch (r) {                                          \
    case 6: { constexpr int RR = 6; __VA_ARGS__; } break; \
    case 7: { constexpr int RR = 7; __VA_ARGS__; } break; \
    case 8: { constexpr int RR = 8; __VA_ARGS__; } break; \
    default: { constexpr int RR = 9; __VA_ARGS__; } break; \
  }

// Programmatic dependent launch: the pipeline's kernels may be scheduled while
// the one before them on the stream drains, and wait for its completion and
// memory (pdl_wait) before they read or write anything of it.  The gaps and
// ramps between six to nine short kernels were a third of a mid-size product:
// 2^16 bits 25.2 -> 17.3 us, 2^24 bits 117 -> 99 us, 2^30 bits 5.47 -> 5.45 ms.
template <class... P, class... A>
static void launch_pdl(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, (P)args...);
}

template <int C>
static void launch_small_c(const SmallJob& job, const Roots& R, cudaStream_t st) {
  launch_pdl(k_small_one<C>, dim3(1), small_threads(C, true), small_words(C, true) * 8, st, job, R);
}
// One product within a cluster.
template <int L>
static void launch_cluster_c(const SmallJob& job, const Roots& R, cudaStream_t st) {
  launch_pdl(k_cluster_mul<L>, dim3(2 * ClusterGeom<L>::OP), ClusterGeom<L>::NT, ClusterGeom<L>::SMEM, st, job, R);
}
// n products of a batch, up to 2^11 points, a cluster each.
static void launch_clusters(const SmallJob* d_jobs, unsigned n, const Roots& R, cudaStream_t st) {
  using G = ClusterGeom<11>;
  launch_pdl(k_cluster_mul<11, true>, dim3(2 * G::OP, n), G::NT, G::SMEM, st, d_jobs, R);
}
static void launch_cluster(int L, const SmallJob& job, const Roots& R, cudaStream_t st) {
  if (L <= 12) launch_cluster_c<12>(job, R, st);
  else if (L == 13) launch_cluster_c<13>(job, R, st);
  else launch_cluster_c<14>(job, R, st);
}
// One product within a CTA.
static void launch_small(const SmallJob& job, const Roots& R, cudaStream_t st) {
  switch (small_class(job.la, job.lb)) {
    case SMALL_TINY: launch_small_c<SMALL_TINY>(job, R, st); break;
    case 9: launch_small_c<9>(job, R, st); break;
    default: launch_small_c<10>(job, R, st); break;  // longer ones: launch_cluster
  }
}


struct Launcher {
  cudaStream_t st;
  bool stats;  // count and (optionally) time launches
  const Roots& R;
  cudaEvent_t b_ready = nullptr;  // operand b's upload (plain host-buffer call): waited on before its first pass
  bool tables = true;             // read pass twiddles from the cached tables (false: compute them)
};

// ---------------------------------------------------------------- twiddle tables
// Pass twiddles can be read from tables laid out like the data they
// multiply, one coalesced load per element, instead of being computed from
// the root tables (a product of two table entries per element in the first
// passes, a scattered lookup in a 2^(R+S)-entry level table in the middle
// ones).  With f_R the digit-reversed row frequency (pass_freq<R>):
//   first pass of length N = 2^L, radix 2^R, S = L - R:
//     forward  tw[i 2^S + J] = w_N^(f_R(i) J)
//     inverse  tw[i 2^S + J] = w_N^-(f_R(i) J) N^-1   (the inverse's 1/N for free)
//   middle pass of radix 2^R and stride 2^S, M = 2^(R+S):
//     tw[r 2^S + j] = w_M^(+-f_R(r) j)
// Tables are built once per shape, on first use, and kept until
// pimul_shutdown (the reference keeps its twiddles in a cache too,
// crates/bignum/src/ntt.rs:571-611), up to a byte cap; first passes longer
// than 2^TW_LOG_MAX compute their twiddles.
constexpr int TW_LOG_MAX = 28;

template <int R>
__global__ void k_tw_first(uint64_t* tw, int L, int inv, uint64_t scale, Roots RT) {
  const int S = L - R;
  const uint64_t n = 1ull << L, smask = (1ull << S) - 1;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(e >> S), J = (uint32_t)(e & smask);
    uint64_t t = root_pow32(RT, L, pass_freq<R>(i) * J, inv != 0);
    if (inv) t = gl::mul(t, scale);
    tw[e] = gl::canon(t);
  }
}

// The 192-row first pass of N = 3 2^k points: tw[i 2^S + J] = w_N^(+-f J) with f = i
// / 12 + 16 (i mod 12) (inverse: times `scale`), w_N^x = w_(2^k)^(x / 3) w_3^(2^k x).
__global__ void k_tw_first3(uint64_t* tw, int k, int inv, uint64_t scale, Roots RT) {
  const int S = k - 6;
  const uint64_t n = 3ull << k, smask = (1ull << S) - 1;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)(e >> S), J = (uint32_t)(e & smask);
    const uint32_t x = (i / 12 + 16 * (i % 12)) * J;  // < 192 2^18
    uint64_t t = root_pow32(RT, k, x * 0xAAAAAAABu, inv != 0);  // 3^-1 mod 2^32
    uint32_t c = x % 3 * ((k & 1) ? 2 : 1) % 3;                // 2^k = 2^-k mod 3
    if (inv) c = (3 - c) % 3;
    if (c == 1) t = gl::mul(t, gl::EPS);                       // w_3 = 2^64
    if (c == 2) t = gl::mul(t, gl::P - (1ull << 32));          // 2^128 = -2^32
    if (inv) t = gl::mul(t, scale);
    tw[e] = gl::canon(t);
  }
}

template <int R>
__global__ void k_tw_mid(uint64_t* tw, int S, int inv, Roots RT) {
  const int M = R + S;
  const uint64_t n = 1ull << M, smask = (1ull << S) - 1;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t r = (uint32_t)(e >> S), j = (uint32_t)(e & smask);
    tw[e] = gl::canon(root_pow32(RT, M, pass_freq<R>(r) * j, inv != 0));
  }
}

struct TwCache {
  std::mutex mu;
  std::unordered_map<uint64_t, uint64_t*> tables;
  uint64_t bytes = 0;
  uint64_t cap = 8ull << 30;
  cudaStream_t st = nullptr;
};
static TwCache& tw_cache() {
  static TwCache* c = new TwCache;  // never destroyed: usable during static destruction
  return *c;
}

// The table of one pass (kind 0: first pass, R + S = L; kind 1: middle pass;
// kind 2: 192-row first pass),
// built on first use.  Null (compute the twiddles) when the shape is above
// TW_LOG_MAX or the cap, while `caller` is capturing a graph (a table is
// never built inside a capture), or when allocating it fails.
static const uint64_t* tw_table(int kind, int R, int S, bool inv, cudaStream_t caller) {
  if (kind == 0 && R + S > TW_LOG_MAX) return nullptr;
  const uint64_t key = ((uint64_t)kind << 24) | ((uint64_t)R << 16) | ((uint64_t)S << 8) | (inv ? 1u : 0u);
  TwCache& c = tw_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  auto it = c.tables.find(key);
  if (it != c.tables.end()) return it->second;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (caller && (cudaStreamIsCapturing(caller, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)) return nullptr;
  const uint64_t words = kind == 2 ? 192ull << S : 1ull << (R + S);
  if (c.bytes + 8 * words > c.cap) return nullptr;
  if (!c.st && cudaStreamCreateWithFlags(&c.st, cudaStreamNonBlocking) != cudaSuccess) {
    cudaGetLastError();
    c.st = nullptr;
    return nullptr;
  }
  uint64_t* d = nullptr;
  if (cudaMalloc(&d, 8 * words) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  const unsigned blocks = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(words / 256, 152 * 16));
  const Roots& RT = g_dev.roots;
  if (kind == 0) {
    const uint64_t ninv = hf::pow(hf::pow(2, 191), (uint64_t)(R + S));  // 2^-L (2^192 = 1)
    PIMUL_DISPATCH_R(R, (k_tw_first<RR><<<blocks, 256, 0, c.st>>>(d, R + S, inv ? 1 : 0, ninv, RT)));
  } else if (kind == 2) {
    const uint64_t ninv = hf::mul(hf::pow(hf::pow(2, 191), (uint64_t)(S + 6)), hf::pow(3, hf::P - 2));  // 1 / (3 2^k)
    k_tw_first3<<<blocks, 256, 0, c.st>>>(d, S + 6, inv ? 1 : 0, ninv, RT);
  } else {
    PIMUL_DISPATCH_R(R, (k_tw_mid<RR><<<blocks, 256, 0, c.st>>>(d, S, inv ? 1 : 0, RT)));
  }
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(c.st) != cudaSuccess) {
    cudaFree(d);
    return nullptr;
  }
  c.tables[key] = d;
  c.bytes += 8 * words;
  return d;
}

// log2 stride of the first pass's rows.
static int first_stride(const Plan& pl) { return is_three(pl.L) ? pl.L - THREE - 6 : pl.L - pl.r[0]; }
// Pointers of every pass table of a plan (null entries: compute).
struct PassTables {
  const uint64_t* first_fwd = nullptr;
  const uint64_t* first_inv = nullptr;  // carries N^-1
  const uint64_t* mid_fwd[5] = {};
  const uint64_t* mid_inv[5] = {};
};
static PassTables pass_tables(const Plan& pl, cudaStream_t caller) {
  PassTables t;
  int S = first_stride(pl);
  const int kind = is_three(pl.L) ? 2 : 0, r0 = is_three(pl.L) ? 0 : pl.r[0];
  t.first_fwd = tw_table(kind, r0, S, false, caller);
  t.first_inv = tw_table(kind, r0, S, true, caller);
  for (int p = 1; p < pl.np - 1; p++) {
    S -= pl.r[p];
    t.mid_fwd[p] = tw_table(1, pl.r[p], S, false, caller);
    t.mid_inv[p] = tw_table(1, pl.r[p], S, true, caller);
  }
  return t;
}

// The length that `count` products of at most n coefficients take, L the power
// of two at or above n: 3 2^(L-2) points where they hold n, have passes, and
// have their twiddle tables (which a 192-row pass cannot do without: none above
// the cache's cap, none built inside a capture).  At 70 % of a power of two:
// 2.56 -> 2.05 ms (2^26), 158 -> 128.5 us (2^22), 83.1 -> 69.4 (2^21), 21.2 ->
// 18.8 (2^15).  One or two of 2^17 points are left in their three short passes
// (make_plan: 27.9 us against 29.8 for 3 2^15 in two passes).
static int product_length(uint64_t n, int L, uint64_t count, cudaStream_t caller) {
  if (!three_holds(n, L) || (L == 17 && count <= 2)) return L;
  const PassTables t = pass_tables(make_plan(THREE + L - 2), caller);
  return t.first_fwd && t.first_inv ? THREE + L - 2 : L;
}

static void tw_release_all() {
  TwCache& c = tw_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  for (auto& kv : c.tables) cudaFree(kv.second);
  c.tables.clear();
  c.bytes = 0;
  if (c.st) cudaStreamDestroy(c.st);
  c.st = nullptr;
}

// All launches of the large-product pipeline for `nj` products sharing the
// transform length L (see THREE): the products come from the device array `jobs`
// (blockIdx.y) or, for nj == 1 and jobs == nullptr, from `one`.
// nc: how many of them, from the first, have carries to run (the others are
// addends and further segments); max_chunk: largest carry-chunk count among
// those.
static void run_large(const Launcher& X, const Job* jobs, const Job& one, uint32_t nj, int L, uint32_t nc, uint64_t max_chunk) {
  const uint64_t N = length_words(L);
  const Plan pl = make_plan(L, nj * N);
  const bool three = is_three(L);
  const PassTables tw = X.tables ? pass_tables(pl, X.st) : PassTables{};
  // 2^-L (2^192 = 1), unless the inverse first pass's table has it (a length of 3 2^k points has its tables)
  const uint64_t ninv = tw.first_inv ? 0 : hf::pow(hf::pow(2, 191), L);
  const int rl = pl.r[pl.np - 1];
  const bool one_operand = !jobs && is_square(one);
  // both operands in one launch per pass (unless b is still on its way up):
  // half the launches and partial waves, 98.5 -> 87.8 us for a lone 2^21-point
  // product, 5.46 -> 5.43 ms at 2^27, where the arrays are far larger than L2
  const bool merged = !X.b_ready && !one_operand;
  const unsigned nz = merged ? 2 : 1;
  auto grid = [&](int tile, unsigned z) { return dim3((unsigned)(N >> tile), nj, z); };
  const int S0 = first_stride(pl);
  for (int which = 0; which < (merged || one_operand ? 1 : 2); which++) {
    if (which == 1 && X.b_ready) cudaStreamWaitEvent(X.st, X.b_ready, 0);
    {
      KTimer kt(K_PACK, X.st, X.stats);
      if (three)
        launch_pdl(k_fwd_first3, dim3(1u << (S0 - ThreeGeom::T), nj, nz), 128, ThreeGeom::XWORDS * 8, X.st, jobs, one, which, S0,
                   X.R, tw.first_fwd);
      else
        PIMUL_DISPATCH_R(pl.r[0], {
          launch_pdl(k_fwd_first<RR>, grid(ColGeom<RR>::TILE, nz), PASS_THREADS, (ColGeom<RR>::XWORDS + (1u << RR)) * 8, X.st,
                     jobs, one, which, L, X.R, tw.first_fwd);
        });
    }
    int S = S0;
    for (int p = 1; p < pl.np - 1; p++) {
      S -= pl.r[p];
      KTimer kt(K_PASS_FWD, X.st, X.stats);
      PIMUL_DISPATCH_R(pl.r[p], {
        launch_pdl(k_col_mid<RR, true>, grid(ColGeom<RR>::TILE, nz), PASS_THREADS, ColGeom<RR>::XWORDS * 8, X.st, jobs, one,
                   which, L, S, X.R, tw.mid_fwd[p]);
      });
    }
    KTimer kt(K_PASS_FWD, X.st, X.stats);
    PIMUL_DISPATCH_ROW(rl, {
      launch_pdl(k_fwd_last<RR>, grid(RowGeom<RR>::TILE, nz), PASS_THREADS, 4 * RowGeom<RR>::XWORDS * 8, X.st, jobs, one, which,
                 L, X.R);
    });
  }
  {
    KTimer kt(K_POINTWISE, X.st, X.stats);
    PIMUL_DISPATCH_ROW(rl, {
      launch_pdl(k_inv_last<RR>, grid(RowGeom<RR>::TILE, 1), PASS_THREADS, 4 * RowGeom<RR>::XWORDS * 8, X.st, jobs, one, L,
                 X.R);
    });
  }
  int S = rl;
  for (int p = pl.np - 2; p >= 1; S += pl.r[p--]) {
    KTimer kt(K_PASS_INV, X.st, X.stats);
    PIMUL_DISPATCH_R(pl.r[p], {
      launch_pdl(k_col_mid<RR, false>, grid(ColGeom<RR>::TILE, 1), PASS_THREADS, ColGeom<RR>::XWORDS * 8, X.st, jobs, one, 0, L,
                 S, X.R, tw.mid_inv[p]);
    });
  }
  {
    KTimer kt(K_PASS_INV, X.st, X.stats);
    if (three)
      launch_pdl(k_inv_first3_carry, dim3(1u << (S0 - ThreeGeom::T), nj), 128, ThreeGeom::CWORDS * 8, X.st, jobs, one, S0, X.R,
                 tw.first_inv);
    else
      PIMUL_DISPATCH_R(pl.r[0], {
        launch_pdl(k_inv_first_carry<RR>, grid(ColGeom<RR>::TILE, 1), PASS_THREADS, (INV_FIRST_XWORDS<RR> + (1u << RR)) * 8,
                   X.st, jobs, one, L, X.R, tw.first_inv, ninv);
      });
  }
  {
    KTimer kt(K_CARRY, X.st, X.stats);
    // a CTA per chunk of a lone product; in a batch of uneven lengths the CTAs
    // of a product stride over its chunks (a CTA per chunk of the longest left
    // nearly all of them without work: 630 of 7200 us in 4096 uneven products,
    // 290 so)
    const uint64_t per = std::min<uint64_t>(max_chunk, nc == 1 ? max_chunk : (CARRY_CTAS + nc - 1) / nc);
    launch_pdl(k_carry, dim3((unsigned)per, nc), CARRY_THREADS, 0, X.st, jobs, one);
  }
}

// Device multiply: d_out[0 .. la+lb) = a * b, scratch from the memory pool.
static int mul_device(const uint64_t* d_a, uint64_t la, const uint64_t* d_b, uint64_t lb, uint64_t* d_out,
                      cudaStream_t st, cudaEvent_t b_ready = nullptr, uint8_t* scratch = nullptr) {
  if (la == 0 || lb == 0) return PIMUL_OK;
  const Sizes z = sizes_for(la, lb);
  if (z.L > 32) return fail(PIMUL_EINVAL, "transform length above 2^32");
  const Roots& R = g_dev.roots;
  const bool square = d_a == d_b && la == lb;
  if (z.L <= g_dev.lone_log) {
    if (b_ready) cudaStreamWaitEvent(st, b_ready, 0);
    SmallJob job{d_a, d_b, d_out, (uint32_t)la, (uint32_t)lb};
    {
      KTimer kt(K_SMALL, st, true);
      if (z.L < CLUSTER_LOG_MIN) launch_small(job, R, st);
      else launch_cluster(z.L, job, R, st);
    }
    CU(cudaGetLastError());
    return PIMUL_OK;
  }
  uint8_t* base = scratch;
  cudaError_t e = base ? cudaSuccess : cudaMallocAsync((void**)&base, scratch_bytes(la, lb, square), g_dev.pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("scratch allocation: ") + cudaGetErrorString(e));
  }
  Job J{};
  J.a = d_a, J.la = la, J.b = d_b, J.lb = lb, J.out = d_out;
  const SegPlan sg = square ? SegPlan{} : plan_segments(la, lb);
  if (sg.L) {
    if (la < lb) {  // the long operand is cut; it must be there before the first pass
      std::swap(J.a, J.b);
      std::swap(J.la, J.lb);
      if (b_ready) cudaStreamWaitEvent(st, b_ready, 0);
      b_ready = nullptr;
    }
    J.segments = sg.S, J.segv = sg.segv, J.wlo = (uint32_t)sg.wlo;
  }
  carve_scratch(J, base, square);
  Launcher X{st, true, R, b_ready};
  run_large(X, nullptr, J, std::max(1u, sg.S), sg.L ? sg.L : product_length(z.n_out, z.L, 1, st), 1, z.nchunk);
  cudaError_t le = cudaGetLastError();
  if (!scratch) cudaFreeAsync(base, st);
  if (le != cudaSuccess) return fail(PIMUL_ECUDA, std::string("kernel launch: ") + cudaGetErrorString(le));
  return PIMUL_OK;
}

// ------------------------------------------------------------------ batches
// A batch of independent products (and sums of two products) on device
// buffers.  Products are grouped by transform length: those of up to 2^12
// points run whole in shared memory, several of one class side by side in the
// CTAs of a persistent kernel over a list sorted by class (few of up to 2^11
// points in a cluster each); longer ones run the pass pipeline once per length
// with one grid row (blockIdx.y) per descriptor.  Within a group of one length, products whose
// operand b is the same array share b's spectrum (computed once), and a sum
// a1 b1 + a2 b2 runs as two descriptors whose spectra are added before one
// inverse transform and one carry pass.

// One unit of a batch: a b, or a b + a2 b2 (la2 > 0; large lengths only).
struct Unit {
  const uint64_t* a;
  uint64_t la;
  const uint64_t* b;
  uint64_t lb;
  const uint64_t* a2;
  uint64_t la2;
  const uint64_t* b2;
  uint64_t lb2;
  uint64_t* out;
  uint64_t nout;
  int forceL = 0;                 // transform length (log2) when not the one nout implies
  bool coeff = false;             // JF_COEFF: nout canonical coefficients to out, no carry
  const uint64_t* low = nullptr;  // a wrapped product's low coefficients (Job::low)
  uint64_t wrap = 0;              // and their count (Job::wrap)
};

struct BatchLayout {
  std::vector<uint32_t> small;  // unit indices, size-sorted descending
  struct Desc {
    uint32_t unit;
    bool second;             // the a2 b2 half of a sum (an addend)
    uint32_t segment = 0;    // segment of a cut product
    uint32_t flags;          // JF_*
    int64_t owner = -1;      // descriptor whose B this one borrows
    int64_t addend = -1;     // descriptor whose A holds this one's X
    bool lent = false;       // others borrow its B
    uint64_t off_a = 0, off_b = 0, off_w = 0, off_h = 0;
  };
  std::vector<Desc> desc;  // large descriptors in launch order
  struct Bucket {
    int L;
    size_t d0, nd;    // descriptors
    size_t nc;        // of which the first nc have carries to run
    uint64_t max_chunk;
  };
  std::vector<Bucket> large;
  uint64_t arena_bytes = 0;
  std::vector<SegPlan> seg;  // per unit: how a product of a long by a short operand is cut
  size_t clusters = 0;             // of the small jobs the first ones that run in a cluster each
  std::vector<SmallChunk> chunks;  // the others in same-length chunks
  size_t small_smem = 0;           // dynamic shared memory of their CTAs
};

// Scratch bound of one group of same-length descriptors in a batch.  Only
// the descriptors of one group share spectra, so a group should hold every
// product of a splitting level's pairs: at the top of a 10^9-digit tree one
// pair's products take 32 GiB at 2^29 points.  PIMUL_BATCH_ARENA_GIB sets it.
static const uint64_t BATCH_ARENA_CAP = [] {
  const char* e = getenv("PIMUL_BATCH_ARENA_GIB");
  const long long g = e ? atoll(e) : 96;
  return (uint64_t)(g > 0 ? g : 96) << 30;
}();

static int unit_log_n(const Unit& u) {
  if (u.la == 0 || u.lb == 0) return -1;
  if (u.forceL) return u.forceL;
  return log2_ceil(4 * u.nout - 1);
}

// Open-addressing map from (pointer, number) to a number, for at most n keys: a
// batch's shared operands (with std::unordered_map the layout of 2500 products took
// 770 us, longer than their kernels).
class PairMap {
 public:
  explicit PairMap(size_t n) {
    size_t c = 16;
    while (c < 2 * n) c *= 2;
    slots_.resize(c);
  }
  // The number of (p, k), `fresh` where there is none yet.
  uint64_t& at(const void* p, uint64_t k, uint64_t fresh) {
    const uint64_t h = ((uint64_t)(uintptr_t)p + k * 0x9E3779B97F4A7C15ull) * 0xD6E8FEB86659FD93ull;
    for (size_t i = (h >> 32) & (slots_.size() - 1);; i = (i + 1) & (slots_.size() - 1)) {
      Slot& s = slots_[i];
      if (!s.used) s = Slot{p, k, fresh, true};
      if (s.p == p && s.k == k) return s.v;
    }
  }

 private:
  struct Slot {
    const void* p = nullptr;
    uint64_t k = 0, v = 0;
    bool used = false;
  };
  std::vector<Slot> slots_;
};

// share: let products with the same operand b borrow one spectrum (a batch
// plan lays out a shape without pointers and never shares).
static int layout_batch(const Unit* units, size_t n, BatchLayout& B, bool share, cudaStream_t st) {
  std::vector<int> Ls(n);
  for (size_t i = 0; i < n; i++) {
    Ls[i] = unit_log_n(units[i]);
    if (Ls[i] > 32) return fail(PIMUL_EINVAL, "transform length above 2^32 in batch");
  }
  // uneven products are cut into segments, unless others share their b (a
  // shared spectrum saves more)
  if (std::any_of(Ls.begin(), Ls.end(), [](int L) { return L > SMALL_LOG_MAX; })) {
    B.seg.assign(n, SegPlan{});
    PairMap uses(share ? 2 * n : 0), most(share ? 2 * n : 0);  // most: coefficients, by b and power of two
    if (share)
      for (size_t i = 0; i < n; i++)
        if (Ls[i] > SMALL_LOG_MAX) {
          uses.at(units[i].b, 0, 0)++;
          if (units[i].la2) uses.at(units[i].b2, 0, 0)++;
        }
    for (size_t i = 0; i < n; i++) {
      const Unit& u = units[i];
      if (Ls[i] <= SMALL_LOG_MAX || u.la2 || u.coeff || u.forceL || (share && uses.at(u.b, 0, 0) > 1)) continue;
      B.seg[i] = plan_segments(u.la, u.lb);
      if (B.seg[i].L) Ls[i] = B.seg[i].L;
    }
    // three quarters of a power of two where that holds the product, and every
    // other one of that power of two that shares its b (else the spectrum
    // would be computed twice)
    auto three_ok = [&](size_t i) { return Ls[i] > SMALL_LOG_MAX + 1 && !units[i].coeff && !units[i].forceL && !B.seg[i].L; };
    if (share)
      for (size_t i = 0; i < n; i++) {
        const Unit& u = units[i];
        if (Ls[i] <= SMALL_LOG_MAX || B.seg[i].L) continue;
        const uint64_t need = three_ok(i) ? 4 * u.nout - 1 : ~0ull;
        for (const uint64_t* b : {u.b, u.la2 ? u.b2 : nullptr})
          if (b) {
            uint64_t& m = most.at(b, (uint64_t)Ls[i], 0);
            m = std::max(m, need);
          }
      }
    uint64_t all[33] = {}, fit[33] = {};  // transforms of 2^L, and those that could be shorter
    std::vector<bool> shorter(n, false);
    for (size_t i = 0; i < n; i++) {
      const Unit& u = units[i];
      const int L = Ls[i];
      if (L <= SMALL_LOG_MAX) continue;
      const uint64_t w = u.la2 ? 2 : B.seg[i].L ? B.seg[i].S : 1;
      all[L] += w;
      if (!three_ok(i)) continue;
      uint64_t need = 4 * u.nout - 1;
      if (share) {
        need = std::max(need, most.at(u.b, (uint64_t)L, 0));
        if (u.la2) need = std::max(need, most.at(u.b2, (uint64_t)L, 0));
      }
      shorter[i] = three_holds(need, L);
      if (shorter[i]) fit[L] += w;
    }
    for (int L = SMALL_LOG_MAX + 1; L <= 32; L++)
      if (fit[L] && (fit[L] == all[L] || fit[L] << L >= THREE_SPLIT)) fit[L] = (uint64_t)product_length(1, L, fit[L], st);
      else fit[L] = (uint64_t)L;
    for (size_t i = 0; i < n; i++)
      if (shorter[i]) Ls[i] = (int)fit[Ls[i]];
  }
  std::vector<std::vector<uint32_t>> byL(N_LENGTHS);
  size_t count[SMALL_LOG_MAX + 1] = {}, at[SMALL_LOG_MAX + 1] = {};  // of a class of short products: number, place
  size_t n_large = 0;
  for (size_t i = 0; i < n; i++) {
    if (Ls[i] < 0) continue;
    if (Ls[i] <= SMALL_LOG_MAX) {
      if (units[i].la2) return fail(PIMUL_EINVAL, "a sum of products below 2^13 in the pass pipeline");
      Ls[i] = small_class(units[i].la, units[i].lb);
      count[Ls[i]]++;
    } else {
      byL[Ls[i]].push_back((uint32_t)i);
      n_large += units[i].la2 ? 2 : B.seg[i].L ? B.seg[i].S : 1;
    }
  }
  B.desc.reserve(n_large);
  // longest transforms first
  size_t total = 0, longer = 0;
  for (int c = 9; c <= SMALL_LOG_MAX; c++) longer += count[c];
  if (count[11] && !count[12] && longer <= CLUSTER_FEW) B.clusters = longer;
  for (int c = SMALL_LOG_MAX; c >= SMALL_TINY; c--) {
    if (!count[c]) continue;
    at[c] = total;
    if (total >= B.clusters) {
      const uint32_t per = small_per_cta(c);
      for (size_t k = 0; k < count[c]; k += per)
        B.chunks.push_back(SmallChunk{(uint32_t)(total + k), (uint32_t)std::min<size_t>(per, count[c] - k), c});
      B.small_smem = std::max(B.small_smem, small_cta_smem(c));
    }
    total += count[c];
  }
  B.small.resize(total);
  if (total)
    for (size_t i = 0; i < n; i++)
      if (Ls[i] >= 0 && Ls[i] <= SMALL_LOG_MAX) B.small[at[Ls[i]]++] = (uint32_t)i;
  // Groups of one length: at most 65535 descriptors (grid.y) whose scratch
  // fits BATCH_ARENA_CAP; groups run one after another on the stream, so
  // they all reuse the same arena.
  uint64_t arena = 0;
  for (int q = 2 * 32; q > 2 * SMALL_LOG_MAX; q--) {
    const int L = q % 2 ? THREE + (q + 1) / 2 - 2 : q / 2;  // 2^32, 3 2^30, 2^31, ...
    if (byL[L].empty()) continue;
    const uint64_t N = length_words(L);
    size_t s = 0;
    while (s < byL[L].size()) {
      BatchLayout::Bucket bk{L, B.desc.size(), 0, 0, 0};
      // the group's units: descriptor count and a scratch bound (no sharing)
      uint64_t bound = 0;
      size_t e = s;
      for (; e < byL[L].size(); e++) {
        const Unit& u = units[byL[L][e]];
        const SegPlan& sg = B.seg[byL[L][e]];
        const size_t nd = u.la2 ? 2 : sg.L ? sg.S : 1;
        const uint64_t nwin = n_windows_out(u.nout);
        const uint64_t need = round256(N * 8) * (sg.L ? nd + 1 : 2 * nd) + round256(nwin * 16) + round256(carry_words(nwin) * 8);
        if (e > s && (bk.nd + nd > 65535 || bound + need > BATCH_ARENA_CAP)) break;
        bk.nd += nd;
        bound += need;
      }
      // descriptors, those with carries first; the first of several with the
      // same b owns its spectrum, a product's first segment that of the others
      PairMap owner_of(share ? bk.nd : 0);  // by array and length
      auto lend = [&](const uint64_t* b, uint64_t lb, size_t di) {
        const size_t o = owner_of.at(b, lb, di);
        if (o == di) return;
        B.desc[di].flags |= JF_B_SHARED;
        B.desc[di].owner = (int64_t)o;
        B.desc[o].lent = true;
      };
      bk.nc = e - s;
      for (size_t k = s; k < e; k++) {
        const Unit& u = units[byL[L][k]];
        BatchLayout::Desc d1;
        d1.unit = byL[L][k];
        d1.second = false;
        d1.flags = 0;
        d1.lent = B.seg[d1.unit].S > 1;
        const bool sq1 = u.a == u.b && u.la == u.lb;
        B.desc.push_back(d1);
        if (share && !sq1 && !B.seg[d1.unit].L) lend(u.b, u.lb, B.desc.size() - 1);
      }
      for (size_t k = s; k < e; k++) {
        const uint32_t ui = byL[L][k];
        const Unit& u = units[ui];
        const size_t i1 = bk.d0 + (k - s);
        if (u.la2) {
          BatchLayout::Desc d2;
          d2.unit = ui;
          d2.second = true;
          d2.flags = JF_ADDEND;
          B.desc[i1].addend = (int64_t)B.desc.size();
          B.desc.push_back(d2);
          if (share) lend(u.b2, u.lb2, B.desc.size() - 1);
        }
        for (uint32_t g = 1; g < B.seg[ui].S; g++) {
          BatchLayout::Desc d2;
          d2.unit = ui;
          d2.second = false;
          d2.segment = g;
          d2.flags = JF_SEGMENT | JF_B_SHARED;
          d2.owner = (int64_t)i1;
          B.desc.push_back(d2);
        }
      }
      // scratch offsets
      uint64_t off = 0;
      for (size_t di = bk.d0; di < bk.d0 + bk.nd; di++) {
        BatchLayout::Desc& d = B.desc[di];
        const Unit& u = units[d.unit];
        const bool sq = !d.second && u.a == u.b && u.la == u.lb;
        d.off_a = off;
        off += round256(N * 8);
        if (!sq && !(d.flags & JF_B_SHARED)) {
          d.off_b = off;
          off += round256(N * 8);
        }
        if (!d.second && !d.segment) {
          const uint64_t nwin = n_windows_out(u.nout);
          // the windows' low parts go to B where the product has one to itself
          d.off_w = d.off_b;
          if (sq || (d.flags & JF_B_SHARED) || d.lent) {
            d.off_w = off;
            off += round256(nwin * 16);
          }
          d.off_h = off;
          off += round256(carry_words(nwin) * 8);
          bk.max_chunk = std::max<uint64_t>(bk.max_chunk, n_chunks(nwin));
        }
      }
      arena = std::max(arena, off);
      B.large.push_back(bk);
      s = e;
    }
  }
  B.arena_bytes = arena;
  return PIMUL_OK;
}

// Host images of the device descriptors, in launch order: small jobs first,
// then each large bucket.
// Bytes of the small jobs' descriptors and chunks at the head of the image.
static size_t small_desc_bytes(const BatchLayout& B) {
  return round256(B.small.size() * sizeof(SmallJob)) + round256(B.chunks.size() * sizeof(SmallChunk));
}

static void fill_descriptors(const Unit* units, const BatchLayout& B, uint8_t* arena, SmallJob* sd, Job* ld) {
  size_t k = 0;
  for (uint32_t i : B.small)
    sd[k++] = SmallJob{units[i].a, units[i].b, units[i].out, (uint32_t)units[i].la, (uint32_t)units[i].lb};
  SmallChunk* sc = reinterpret_cast<SmallChunk*>(reinterpret_cast<uint8_t*>(sd) + round256(B.small.size() * sizeof(SmallJob)));
  for (size_t c = 0; c < B.chunks.size(); c++) sc[c] = B.chunks[c];
  for (size_t di = 0; di < B.desc.size(); di++) {
    const BatchLayout::Desc& d = B.desc[di];
    const Unit& u = units[d.unit];
    Job J{};
    if (d.second) {
      J.a = u.a2, J.la = u.la2, J.b = u.b2, J.lb = u.lb2;
      J.out = nullptr;
      J.nout = u.la2 + u.lb2;
    } else {
      J.a = u.a, J.la = u.la, J.b = u.b, J.lb = u.lb;
      J.out = u.out;
      J.nout = u.nout;
      J.low = u.low;
      J.wrap = u.wrap;
    }
    const SegPlan& sg = B.seg[d.unit];
    if (sg.L) {
      if (u.la < u.lb) {  // the long operand is the one that is cut
        std::swap(J.a, J.b);
        std::swap(J.la, J.lb);
      }
      J.segv = sg.segv, J.wlo = (uint32_t)sg.wlo;
      to_segment(J, d.segment, 0);  // (A comes from the arena below)
    }
    J.flags = d.flags | (!d.second && u.coeff ? JF_COEFF : 0);
    const bool sq = !d.second && u.a == u.b && u.la == u.lb;
    J.A = reinterpret_cast<uint64_t*>(arena + d.off_a);
    if (d.flags & JF_B_SHARED)
      J.B = reinterpret_cast<uint64_t*>(arena + B.desc[d.owner].off_b);
    else
      J.B = sq ? nullptr : reinterpret_cast<uint64_t*>(arena + d.off_b);
    if (!d.second) {
      const BatchLayout::Desc& first = d.segment ? B.desc[d.owner] : d;  // a segment writes its product's windows
      J.W = reinterpret_cast<uint64_t*>(arena + first.off_w);
      carve_carry(J, reinterpret_cast<uint64_t*>(arena + first.off_h), n_windows_out(u.nout));
    }
    if (d.addend >= 0) {
      const BatchLayout::Desc& x = B.desc[d.addend];
      J.X = reinterpret_cast<const uint64_t*>(arena + x.off_a);
      J.Y = reinterpret_cast<const uint64_t*>(arena + (x.flags & JF_B_SHARED ? B.desc[x.owner].off_b : x.off_b));
    }
    ld[di] = J;
  }
}

static void launch_batch(const Launcher& X, const BatchLayout& B, const SmallJob* d_small, const Job* d_large) {
  if (B.clusters) {
    KTimer kt(K_SMALL, X.st, X.stats);
    launch_clusters(d_small, (unsigned)B.clusters, X.R, X.st);
  }
  if (!B.chunks.empty()) {
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g_dev.device);
    uint64_t grid = (uint64_t)sms * (uint64_t)g_small_ctas_per_sm.load();
    if (grid > B.chunks.size()) grid = B.chunks.size();
    const SmallChunk* d_chunks = reinterpret_cast<const SmallChunk*>(reinterpret_cast<const uint8_t*>(d_small) +
                                                                     round256(B.small.size() * sizeof(SmallJob)));
    KTimer kt(K_SMALL, X.st, X.stats);
    launch_pdl(k_small_mul, dim3((unsigned)grid), SMALL_THREADS, B.small_smem, X.st, d_small, d_chunks,
               (uint32_t)B.chunks.size(), X.R);
  }
  for (const auto& bk : B.large)
    run_large(X, d_large + bk.d0, Job{}, (uint32_t)bk.nd, bk.L, (uint32_t)bk.nc, bk.max_chunk);
}

// The calling thread's buffer for a batch's host descriptor image, kept and
// grown: a fresh image per call (tens of MB at the lowest levels of a
// conversion) cost its page faults every time.  host_to_device has staged
// the image before it returns, so the next call may overwrite it.
static uint8_t* host_image(size_t bytes) {
  thread_local std::unique_ptr<uint8_t[]> buf;
  thread_local size_t cap = 0;
  if (bytes > cap) {
    cap = std::max(bytes, cap + cap / 2);
    buf.reset(new uint8_t[cap]);
  }
  return buf.get();
}

static int run_units(const Unit* units, size_t n, cudaStream_t st, bool share) {
  BatchLayout B;
  int rc = layout_batch(units, n, B, share, st);
  if (rc) return rc;
  const size_t ns = B.small.size(), nl = B.desc.size();
  if (ns + nl == 0) return PIMUL_OK;
  const size_t desc_bytes = small_desc_bytes(B) + nl * sizeof(Job);
  uint8_t* dev = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&dev, round256(B.arena_bytes) + desc_bytes, g_dev.pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("batch scratch allocation: ") + cudaGetErrorString(e));
  }
  uint8_t* arena = dev;
  uint8_t* desc = dev + round256(B.arena_bytes);
  uint8_t* host = host_image(desc_bytes);  // every used byte is written below
  SmallJob* hs = reinterpret_cast<SmallJob*>(host);
  Job* hl = reinterpret_cast<Job*>(host + small_desc_bytes(B));
  fill_descriptors(units, B, arena, hs, hl);
  // descriptors of a large batch go up through the staged copy
  if (host_to_device(desc, host, desc_bytes, st)) e = cudaErrorUnknown;
  if (e == cudaSuccess) {
    Launcher X{st, true, g_dev.roots};
    launch_batch(X, B, reinterpret_cast<SmallJob*>(desc), reinterpret_cast<Job*>(desc + small_desc_bytes(B)));
    e = cudaGetLastError();
  }
  // the host image must outlive the copy (pageable source: staged before return)
  cudaFreeAsync(dev, st);
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("batch launch: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}

static Unit unit_of(const pimul_job& j) {
  return Unit{j.a, j.la, j.b, j.lb, nullptr, 0, nullptr, 0, j.out, j.la + j.lb};
}

static int mul_batch(const pimul_job* jobs, size_t n, cudaStream_t st) {
  std::vector<Unit> u(n);
  for (size_t i = 0; i < n; i++) u[i] = unit_of(jobs[i]);
  return run_units(u.data(), n, st, true);
}

// A batch plan: the layout, arena and descriptors of a fixed batch shape,
// with every launch captured once into a CUDA graph.  Running it writes the
// new operand pointers into a pinned staging image, and one graph launch
// copies the descriptors in and runs all kernels.
struct BatchPlan {
  std::vector<uint64_t> la, lb;
  BatchLayout B;
  uint8_t* dev = nullptr;      // arena + descriptors
  uint8_t* staging = nullptr;  // pinned host image of the descriptors
  size_t desc_bytes = 0, ns = 0, nl = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t done = nullptr;
  bool launched = false;
};

static int plan_create(const size_t* la, const size_t* lb, size_t n, BatchPlan** out) {
  int rc = ensure_init(-1);
  if (rc) return rc;
  CU(cudaSetDevice(g_dev.device));
  auto* P = new BatchPlan();
  P->la.assign(la, la + n);
  P->lb.assign(lb, lb + n);
  // shape-only jobs (distinct dummy pointers: no job is a square)
  std::vector<Unit> shape(n);
  for (size_t i = 0; i < n; i++)
    shape[i] = unit_of(pimul_job{nullptr, la[i], (const uint64_t*)(uintptr_t)(8 + 16 * i), lb[i], nullptr});
  rc = layout_batch(shape.data(), n, P->B, false, nullptr);
  if (rc) { delete P; return rc; }
  P->ns = P->B.small.size();
  P->nl = P->B.desc.size();
  P->desc_bytes = small_desc_bytes(P->B) + P->nl * sizeof(Job);
  cudaError_t e = cudaMalloc((void**)&P->dev, round256(P->B.arena_bytes) + P->desc_bytes + 256);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&P->staging, P->desc_bytes + 256);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&P->done, cudaEventDisableTiming);
  cudaStream_t cs = nullptr;
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (e == cudaSuccess) {
    // twiddle tables are never built inside a capture: build them first
    for (const auto& bk : P->B.large) pass_tables(make_plan(bk.L, bk.nd * length_words(bk.L)), nullptr);
    uint8_t* desc = P->dev + round256(P->B.arena_bytes);
    e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      cudaMemcpyAsync(desc, P->staging, P->desc_bytes, cudaMemcpyHostToDevice, cs);
      Launcher X{cs, false, g_dev.roots};
      launch_batch(X, P->B, reinterpret_cast<SmallJob*>(desc), reinterpret_cast<Job*>(desc + small_desc_bytes(P->B)));
      e = cudaStreamEndCapture(cs, &P->graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&P->exec, P->graph, 0);
  }
  if (cs) cudaStreamDestroy(cs);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (P->exec) cudaGraphExecDestroy(P->exec);
    if (P->graph) cudaGraphDestroy(P->graph);
    if (P->dev) cudaFree(P->dev);
    if (P->staging) cudaFreeHost(P->staging);
    if (P->done) cudaEventDestroy(P->done);
    delete P;
    return fail(e == cudaErrorMemoryAllocation ? PIMUL_ENOMEM : PIMUL_ECUDA,
                std::string("batch plan: ") + cudaGetErrorString(e));
  }
  *out = P;
  return PIMUL_OK;
}

static int plan_run(BatchPlan* P, const pimul_job* jobs, size_t n, cudaStream_t st) {
  if (n != P->la.size()) return fail(PIMUL_EINVAL, "batch size differs from the plan");
  for (size_t i = 0; i < n; i++)
    if (jobs[i].la != P->la[i] || jobs[i].lb != P->lb[i]) return fail(PIMUL_EINVAL, "job sizes differ from the plan");
  // the previous run's descriptor copy must have read the staging image
  if (P->launched) CU(cudaEventSynchronize(P->done));
  SmallJob* hs = reinterpret_cast<SmallJob*>(P->staging);
  Job* hl = reinterpret_cast<Job*>(P->staging + small_desc_bytes(P->B));
  std::vector<Unit> u(n);
  for (size_t i = 0; i < n; i++) u[i] = unit_of(jobs[i]);
  fill_descriptors(u.data(), P->B, P->dev, hs, hl);
  CU(cudaGraphLaunch(P->exec, st));
  CU(cudaEventRecord(P->done, st));
  P->launched = true;
  return PIMUL_OK;
}

static void plan_destroy(BatchPlan* P) {
  if (!P) return;
  if (P->launched) cudaEventSynchronize(P->done);
  if (P->exec) cudaGraphExecDestroy(P->exec);
  if (P->graph) cudaGraphDestroy(P->graph);
  if (P->dev) cudaFree(P->dev);
  if (P->staging) cudaFreeHost(P->staging);
  if (P->done) cudaEventDestroy(P->done);
  delete P;
}

// ------------------------------------------------------------------ autotuner
// Times the candidate pass counts for each length in [Lmin, Lmax] on a
// batch of `reps` synthetic products (device-resident), keeps the fastest,
// and tunes the short products' persistent grid on a batch of small
// products.  The choice only changes the schedule; products are identical.
static int autotune(int Lmin, int Lmax, int reps, char* report, size_t cap) {
  int rc = ensure_init(-1);
  if (rc) return rc;
  cudaStream_t st;
  rc = get_stream(&st);
  if (rc) return rc;
  std::string rep = "{";
  cudaEvent_t e0, e1;
  CU(cudaEventCreate(&e0));
  CU(cudaEventCreate(&e1));
  auto time_batch = [&](std::vector<pimul_job>& js, float* ms_out) -> int {
    for (int w = 0; w < 2; w++) {
      int r2 = mul_batch(js.data(), js.size(), st);
      if (r2) return r2;
    }
    cudaEventRecord(e0, st);
    for (int w = 0; w < 3; w++) {
      int r2 = mul_batch(js.data(), js.size(), st);
      if (r2) return r2;
    }
    cudaEventRecord(e1, st);
    CU(cudaEventSynchronize(e1));
    CU(cudaEventElapsedTime(ms_out, e0, e1));
    return PIMUL_OK;
  };
  // operands: one buffer of random-ish limbs, reused by every synthetic job
  // large lengths read 2 * max_limbs input words and write reps * 2 * max_limbs;
  // the small-kernel batch reads 1024 words and writes 4096 * 1024
  const uint64_t max_limbs = Lmax >= 3 ? (1ull << (Lmax - 3)) : 1;
  const uint64_t in_words = std::max<uint64_t>(2 * max_limbs, 1024);
  const uint64_t out_words = std::max<uint64_t>((uint64_t)reps * 2 * max_limbs, 4096ull * 1024);
  uint64_t* d_in = nullptr;
  uint64_t* d_out = nullptr;
  CU(cudaMallocAsync((void**)&d_in, in_words * 8, g_dev.pool, st));
  CU(cudaMallocAsync((void**)&d_out, out_words * 8, g_dev.pool, st));
  CU(cudaMemsetAsync(d_in, 0xA5, in_words * 8, st));
  bool first = true;
  for (int L = std::max(Lmin, SMALL_LOG_MAX + 1); L <= Lmax && L <= 32; L++) {
    uint64_t limbs = (1ull << (L - 3)) - 1;  // la = lb: 4(la+lb) - 1 < 2^L
    std::vector<pimul_job> js(reps);
    for (int k = 0; k < reps; k++)
      js[k] = pimul_job{d_in, limbs, d_in + limbs, limbs, d_out + (uint64_t)k * 2 * limbs};
    int best_np = 0;
    float best = 1e30f;
    for (int np = 2; np <= 5; np++) {
      if (!plan_valid(make_plan_np(L, np))) continue;
      g_tuned_np[L].store(np);
      float ms = 0;
      rc = time_batch(js, &ms);
      if (rc) break;
      if (ms < best) { best = ms; best_np = np; }
    }
    if (rc) break;
    g_tuned_np[L].store(best_np);
    char buf[96];
    snprintf(buf, sizeof buf, "%s\"np_%d\": %d", first ? "" : ", ", L, best_np);
    rep += buf;
    first = false;
  }
  if (!rc && Lmin <= SMALL_LOG_MAX) {
    // small kernel: CTAs per SM for a batch of 4096 products of 16..512 limbs
    std::vector<pimul_job> js(4096);
    for (int k = 0; k < 4096; k++) {
      uint64_t l = 16 + (k * 37) % 497;
      js[k] = pimul_job{d_in, l, d_in + l, l, d_out + (uint64_t)k * 1024};
    }
    int best_c = 4;
    float best = 1e30f;
    for (int c : {1, 2, 3, 4, 6, 8}) {
      g_small_ctas_per_sm.store(c);
      float ms = 0;
      rc = time_batch(js, &ms);
      if (rc) break;
      if (ms < best) { best = ms; best_c = c; }
    }
    g_small_ctas_per_sm.store(best_c);
    char buf[96];
    snprintf(buf, sizeof buf, "%s\"small_ctas_per_sm\": %d", first ? "" : ", ", best_c);
    rep += buf;
  }
  rep += "}";
  cudaFreeAsync(d_in, st);
  cudaFreeAsync(d_out, st);
  cudaStreamSynchronize(st);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (report && cap) {
    strncpy(report, rep.c_str(), cap - 1);
    report[cap - 1] = 0;
  }
  return rc;
}

// ------------------------------------------------------------------ service
// Served form: device-resident integers (handles) and an asynchronous
// multiply service.  submit() queues a request and returns its result handle
// at once; the handle can feed later requests before it is computed
// (dependencies are CUDA events, never a host round trip).  A service thread
// admits queued requests while their memory fits the HBM budget, launches
// each admitted group as one batch on one of several streams (continuous
// batching: new requests join as earlier ones complete and release memory,
// and groups on different streams overlap on the device), and records every
// request's latency from submit to completion.
struct SvcHandle {
  uint64_t* d = nullptr;
  uint64_t limbs = 0;        // stored length (a product stores la + lb limbs)
  cudaEvent_t ready = nullptr;  // recorded after the producing batch (or upload)
  bool pending = false;      // produced by a request not yet launched
  int64_t producer = -1;     // ticket of the producing request
  bool freed = false;
  uint64_t bytes = 0;
  int readers = 0;           // queued or running requests that read this handle
  bool borrowed = false;     // the caller's device memory (pimul_adopt): never freed here
  bool release = false;      // pimul_release: free once its producer and readers are done
};

struct SvcRequest {
  uint64_t ticket;
  int op;  // 0 multiply, 1 square, 2 add, 3 subtract (PIMUL_OP_*)
  int L = 0;  // transform length (log2) of a product, from the input lengths at submit
  uint64_t a, b, out;  // handle ids
  double t_submit;
  double t_done = 0;
  uint64_t scratch = 0;
  int state = 0;  // 0 queued, 1 launched, 2 done, 3 cancelled
};

struct SvcBatch {
  cudaEvent_t done;
  std::vector<uint64_t> tickets;
  uint64_t scratch = 0;
  int stream = 0;
};

struct Service {
  std::mutex mu;
  std::condition_variable cv;       // wakes the service thread
  std::condition_variable done_cv;  // wakes waiters
  std::thread th;
  bool running = false, stop = false;
  uint64_t budget = 120ull << 30;
  uint64_t in_use = 0;  // handle bytes + scratch of launched requests
  uint64_t next_handle = 1, next_ticket = 1;
  std::unordered_map<uint64_t, SvcHandle> handles;
  std::unordered_map<uint64_t, SvcRequest> requests;
  std::deque<uint64_t> queue;
  std::vector<SvcBatch> inflight;
  std::vector<cudaStream_t> streams;
  std::vector<int> stream_busy;
  std::vector<double> latencies;  // seconds, completed requests
  uint64_t completed = 0, batches = 0;
  int max_batch = 4096;
  int big_log_n = 24;  // requests with transforms of 2^big_log_n and longer run alone on stream 0
  bool dirty = true;   // something admission depends on changed since the last admission pass
  // Handles' memory (uploads and results) comes from a pool of its own:
  // after a long run of plain products allocating and freeing scratch on
  // another stream, allocations from the shared pool on the service's
  // stream took about 0.1-0.2 ms each, and a thread submitting a tree of
  // 2000 requests spent half a second in them.
  cudaMemPool_t pool = nullptr;
};
// Heap-allocated and never destroyed: its thread is joined by an atexit
// handler (registered after the CUDA runtime's, so it runs first).
static Service& svc_obj() {
  static Service* s = new Service();
  return *s;
}
#define g_svc (svc_obj())

static void svc_atexit() {
  std::unique_lock<std::mutex> lk(g_svc.mu);
  if (!g_svc.running) return;
  g_svc.stop = true;
  g_svc.cv.notify_all();
  lk.unlock();
  if (g_svc.th.joinable()) g_svc.th.join();
  lk.lock();
  g_svc.running = false;
}

static double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

static void svc_loop();

static int svc_start() {
  int rc = ensure_init(-1);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(g_svc.mu);
  if (g_svc.running) return PIMUL_OK;
  CU(cudaSetDevice(g_dev.device));
  if (g_svc.streams.empty()) {
    // stream 0: highest priority, reserved for large requests (one per
    // group) so they run at near-solo speed; streams 1-4 carry batched
    // groups of smaller requests
    int lo = 0, hi = 0;
    CU(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    for (int i = 0; i < 5; i++) {
      cudaStream_t s;
      CU(cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, i == 0 ? hi : lo));
      g_svc.streams.push_back(s);
      g_svc.stream_busy.push_back(0);
    }
  }
  if (!g_svc.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = g_dev.device;
    CU(cudaMemPoolCreate(&g_svc.pool, &props));
    uint64_t thr = UINT64_MAX;  // keep freed handle memory for later requests
    CU(cudaMemPoolSetAttribute(g_svc.pool, cudaMemPoolAttrReleaseThreshold, &thr));
  }
  g_svc.stop = false;
  g_svc.running = true;
  g_svc.th = std::thread(svc_loop);
  static bool registered = (std::atexit(svc_atexit), true);
  (void)registered;
  return PIMUL_OK;
}

// Free a handle whose producer has been launched and whose readers are done
// (the free is ordered after the producer's batch on stream 0).
static void svc_free_now(uint64_t id) {
  auto it = g_svc.handles.find(id);
  if (it == g_svc.handles.end()) return;
  SvcHandle& h = it->second;
  if (h.ready) {
    cudaStreamWaitEvent(g_svc.streams[0], h.ready, 0);
    cudaEventDestroy(h.ready);
  }
  if (!h.borrowed && h.d) cudaFreeAsync(h.d, g_svc.streams[0]);
  g_svc.in_use -= h.bytes;
  g_svc.handles.erase(it);
}

// Released handles that have become free.
static void svc_free_released() {
  std::vector<uint64_t> done;
  for (auto& kv : g_svc.handles)
    if (kv.second.release && !kv.second.pending && kv.second.readers <= 0) done.push_back(kv.first);
  for (uint64_t id : done) svc_free_now(id);
}


int svc_addsub(const pimul_addsub_job* jobs, size_t n, cudaStream_t st);  // unchecked, asynchronous (below)

// Group kind of a request: 0 a product below the big length, 1 a big
// product (alone on stream 0), 2 an addition or subtraction.
static int svc_kind(const SvcRequest& r) {
  if (r.op >= 2) return 2;
  return r.L >= g_svc.big_log_n ? 1 : 0;
}

static bool svc_ready(const SvcRequest& r) {
  return !g_svc.handles[r.a].pending && !g_svc.handles[r.b].pending;
}

// One group: the kind of the first ready request in the queue whose stream
// is free (stream 0 for a big product, a free batch stream otherwise), then
// every ready request of that kind among the first SVC_SCAN queued (in
// order), within the budget.  A request whose input is not launched yet
// waits without holding back the ready ones behind it (continuous batching
// of whatever is ready).  Returns whether a group was launched.
constexpr size_t SVC_SCAN = 1 << 14;

static bool svc_admit(std::unique_lock<std::mutex>& lk) {
  if (g_svc.queue.empty()) return false;
  // the free streams first: with none, nothing can be admitted and the
  // queue is not scanned (the submitting threads share this mutex)
  int batch_si = -1;
  for (size_t i = 1; i < g_svc.streams.size(); i++)
    if (!g_svc.stream_busy[i]) { batch_si = (int)i; break; }
  const bool big_free = !g_svc.stream_busy[0];
  if (batch_si < 0 && !big_free) return false;
  int kind = -1;
  size_t scanned = 0;
  for (auto it = g_svc.queue.begin(); it != g_svc.queue.end() && scanned < SVC_SCAN; ++it, ++scanned) {
    const SvcRequest& r = g_svc.requests[*it];
    if (!svc_ready(r)) continue;
    const int k = svc_kind(r);
    if (k == 1 ? big_free : batch_si >= 0) {
      kind = k;
      break;
    }
  }
  if (kind < 0) return false;
  const int si = kind == 1 ? 0 : batch_si;
  std::vector<uint64_t> take;
  uint64_t add = 0;
  scanned = 0;
  for (auto it = g_svc.queue.begin();
       it != g_svc.queue.end() && scanned < SVC_SCAN && (int)take.size() < g_svc.max_batch; scanned++) {
    SvcRequest& r = g_svc.requests[*it];
    if (!svc_ready(r) || svc_kind(r) != kind) {
      ++it;
      continue;
    }
    if (g_svc.in_use + add + r.scratch > g_svc.budget && !(take.empty() && g_svc.inflight.empty())) break;
    take.push_back(*it);
    add += r.scratch;
    it = g_svc.queue.erase(it);
    if (kind == 1) break;  // a big request forms its own group
  }
  if (take.empty()) return false;
  cudaStream_t st = g_svc.streams[si];
  const bool linear = g_svc.requests[take.front()].op >= 2;
  std::vector<pimul_job> jobs;
  std::vector<pimul_addsub_job> asj;
  jobs.reserve(take.size());
  for (uint64_t t : take) {
    SvcRequest& r = g_svc.requests[t];
    SvcHandle& A = g_svc.handles[r.a];
    SvcHandle& B = g_svc.handles[r.b];
    SvcHandle& O = g_svc.handles[r.out];
    if (A.ready) cudaStreamWaitEvent(st, A.ready, 0);
    if (r.op != 1 && B.ready) cudaStreamWaitEvent(st, B.ready, 0);
    if (O.ready) cudaStreamWaitEvent(st, O.ready, 0);  // result buffer allocated
    if (linear) {
      // out = a + b (max + 1 limbs) or a - b (a's limbs; a >= b): no carry
      // or borrow can leave the output, so nothing is checked
      asj.push_back(pimul_addsub_job{A.d, A.limbs, B.d, B.limbs, O.d, O.limbs, r.op == 3 ? PIMUL_SUB_MOD : 0});
    } else {
      const uint64_t* pa = A.d;
      const uint64_t* pb = r.op == 1 ? A.d : B.d;
      uint64_t lb = r.op == 1 ? A.limbs : B.limbs;
      jobs.push_back(pimul_job{pa, A.limbs, pb, lb, O.d});
    }
    r.state = 1;
  }
  SvcBatch bt;
  bt.stream = si;
  bt.scratch = add;
  bt.tickets = take;
  g_svc.in_use += add;
  lk.unlock();
  int rc = linear ? svc_addsub(asj.data(), asj.size(), st) : mul_batch(jobs.data(), jobs.size(), st);
  cudaEventCreateWithFlags(&bt.done, cudaEventDisableTiming);
  cudaEventRecord(bt.done, st);
  lk.lock();
  for (uint64_t t : take) {
    SvcRequest& r = g_svc.requests[t];
    SvcHandle& O = g_svc.handles[r.out];
    cudaEvent_t e;
    cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    cudaEventRecord(e, st);
    if (O.ready) cudaEventDestroy(O.ready);
    O.ready = e;
    O.pending = false;
    if (rc) r.state = 3;
  }
  g_svc.stream_busy[si] = 1;
  g_svc.inflight.push_back(std::move(bt));
  g_svc.batches++;
  return true;
}

static bool svc_reap(std::unique_lock<std::mutex>& lk) {
  bool any = false;
  for (size_t i = 0; i < g_svc.inflight.size();) {
    SvcBatch& bt = g_svc.inflight[i];
    if (cudaEventQuery(bt.done) == cudaSuccess) {
      double t = now_s();
      for (uint64_t tk : bt.tickets) {
        SvcRequest& r = g_svc.requests[tk];
        if (r.state != 3) r.state = 2;
        r.t_done = t;
        auto ia = g_svc.handles.find(r.a);
        if (ia != g_svc.handles.end()) ia->second.readers--;
        if (r.b != r.a) {
          auto ib = g_svc.handles.find(r.b);
          if (ib != g_svc.handles.end()) ib->second.readers--;
        }
        g_svc.latencies.push_back(t - r.t_submit);
        g_svc.completed++;
      }
      g_svc.in_use -= bt.scratch;
      g_svc.stream_busy[bt.stream] = 0;
      svc_free_released();
      cudaEventDestroy(bt.done);
      g_svc.inflight.erase(g_svc.inflight.begin() + i);
      g_svc.done_cv.notify_all();
      any = true;
    } else {
      i++;
    }
  }
  return any;
}

static void svc_loop() {
  cudaSetDevice(g_dev.device);
  std::unique_lock<std::mutex> lk(g_svc.mu);
  while (!g_svc.stop) {
    if (svc_reap(lk)) g_svc.dirty = true;  // streams and budget freed
    // admission only after a change (a submission, a completion, a release,
    // a new budget or policy), and again after every group it launched
    if (g_svc.dirty) g_svc.dirty = svc_admit(lk);
    if (g_svc.inflight.empty() && g_svc.queue.empty()) {
      g_svc.cv.wait_for(lk, std::chrono::milliseconds(50));
    } else {
      // bounded poll: completions are checked every 20 us while work is in flight
      g_svc.cv.wait_for(lk, std::chrono::microseconds(20));
    }
  }
}

static uint64_t svc_new_handle(uint64_t limbs, uint64_t* d, bool pending, uint64_t bytes) {
  uint64_t id = g_svc.next_handle++;
  SvcHandle h;
  h.d = d;
  h.limbs = limbs;
  h.pending = pending;
  h.bytes = bytes;
  g_svc.handles[id] = h;
  return id;
}

void noalloc_forget();  // defined with the no-alloc entry point below
}  // namespace pimul

// ====================================================================== C ABI
using namespace pimul;

extern "C" {

const char* pimul_version(void) { return "pimul 0.2 (sm_103a)"; }

const char* pimul_last_error(void) { return t_err.c_str(); }

int pimul_init(int device) { return ensure_init(device); }

int pimul_shutdown(void) {
  pimul::noalloc_forget();
  {
    std::unique_lock<std::mutex> sl(g_svc.mu);
    if (g_svc.running) {
      g_svc.stop = true;
      g_svc.cv.notify_all();
      sl.unlock();
      if (g_svc.th.joinable()) g_svc.th.join();
      sl.lock();
      g_svc.running = false;
    }
  }
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_dev.ready) return PIMUL_OK;
  cudaSetDevice(g_dev.device);
  cudaDeviceSynchronize();
  release_host_staging();
  tw_release_all();
  cudaFree(g_dev.d_roots);
  if (g_dev.pool) cudaMemPoolTrimTo(g_dev.pool, 0);
  if (g_svc.pool) cudaMemPoolTrimTo(g_svc.pool, 0);  // handles still held keep their memory
  g_dev = DeviceState{};
  return PIMUL_OK;
}

int pimul_plan(size_t la, size_t lb, uint64_t* n_transform, int* passes) {
  if (!n_transform || !passes) return fail(PIMUL_EINVAL, "null output pointer");
  if (la == 0 || lb == 0) { *n_transform = 0; *passes = 0; return PIMUL_OK; }
  int L = log2_ceil(4 * (uint64_t)la + 4 * (uint64_t)lb - 1);
  if (L > 32) return fail(PIMUL_EINVAL, "transform length above 2^32");
  *n_transform = 1ull << L;
  *passes = L <= SMALL_LOG_MAX ? 0 : make_plan(L).np;
  return PIMUL_OK;
}

int pimul_stats_enable(int on) {
  g_timing.store(on ? 1 : 0);
  return PIMUL_OK;
}

int pimul_stats_reset(void) {
  stats_drain();
  std::lock_guard<std::mutex> lk(g_tmu);
  for (int i = 0; i < K_NCLASS; i++) {
    g_launch[i].store(0);
    g_ms[i] = 0;
    g_timed[i] = 0;
  }
  return PIMUL_OK;
}

int pimul_stats_get(int kclass, const char** name, uint64_t* launches, uint64_t* timed, double* ms) {
  if (kclass < 0 || kclass >= K_NCLASS) return fail(PIMUL_EINVAL, "kernel class out of range");
  stats_drain();
  std::lock_guard<std::mutex> lk(g_tmu);
  if (name) *name = k_names[kclass];
  if (launches) *launches = g_launch[kclass].load();
  if (timed) *timed = g_timed[kclass];
  if (ms) *ms = g_ms[kclass];
  return PIMUL_OK;
}

int pimul_sync(void) {
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  CU(cudaStreamSynchronize(st));
  return PIMUL_OK;
}

int pimul_mul_batch(const pimul_job* jobs, size_t n, void* stream) {
  if (n && !jobs) return fail(PIMUL_EINVAL, "null job list");
  for (size_t i = 0; i < n; i++)
    if (jobs[i].la && jobs[i].lb && (!jobs[i].a || !jobs[i].b || !jobs[i].out))
      return fail(PIMUL_EINVAL, "null device pointer in batch");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  return mul_batch(jobs, n, st);
}

int pimul_batch_plan_create(const size_t* la, const size_t* lb, size_t n, pimul_batch_plan** plan) {
  if (!plan || (n && (!la || !lb))) return fail(PIMUL_EINVAL, "null argument");
  BatchPlan* P = nullptr;
  int rc = plan_create(la, lb, n, &P);
  if (rc) return rc;
  *plan = reinterpret_cast<pimul_batch_plan*>(P);
  return PIMUL_OK;
}

int pimul_batch_plan_run(pimul_batch_plan* plan, const pimul_job* jobs, size_t n, void* stream) {
  if (!plan || (n && !jobs)) return fail(PIMUL_EINVAL, "null argument");
  for (size_t i = 0; i < n; i++)
    if (jobs[i].la && jobs[i].lb && (!jobs[i].a || !jobs[i].b || !jobs[i].out))
      return fail(PIMUL_EINVAL, "null device pointer in batch");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  return plan_run(reinterpret_cast<BatchPlan*>(plan), jobs, n, st);
}

int pimul_batch_plan_destroy(pimul_batch_plan* plan) {
  plan_destroy(reinterpret_cast<BatchPlan*>(plan));
  return PIMUL_OK;
}

int pimul_autotune(int log_n_min, int log_n_max, int reps, char* report, size_t report_cap) {
  if (log_n_min < 1 || log_n_max > 28 || log_n_min > log_n_max || reps < 1)
    return fail(PIMUL_EINVAL, "autotune range must lie in [1, 28] and reps >= 1");
  return autotune(log_n_min, log_n_max, reps, report, report_cap);
}

int pimul_tuning_set(int log_n, int passes, int small_ctas_per_sm) {
  if (log_n >= 0 && log_n <= 32) {
    if (passes && !plan_valid(make_plan_np(log_n, passes))) return fail(PIMUL_EINVAL, "no kernels for that split");
    g_tuned_np[log_n].store(passes);
  }
  if (small_ctas_per_sm > 0) g_small_ctas_per_sm.store(small_ctas_per_sm);
  return PIMUL_OK;
}

int pimul_twiddle_cache(uint64_t max_bytes, uint64_t* held) {
  TwCache& c = tw_cache();
  std::lock_guard<std::mutex> lk(c.mu);
  c.cap = max_bytes;
  if (held) *held = c.bytes;
  return PIMUL_OK;
}

int pimul_set_budget(uint64_t bytes) {
  std::lock_guard<std::mutex> lk(g_svc.mu);
  g_svc.budget = bytes;
  g_svc.dirty = true;
  return PIMUL_OK;
}

int pimul_upload(const uint64_t* host, size_t n, uint64_t* handle) {
  if (!handle || (n && !host)) return fail(PIMUL_EINVAL, "null argument");
  int rc = svc_start();
  if (rc) return rc;
  uint64_t bytes = round256(std::max<uint64_t>(n, 1) * 8);
  {
    std::lock_guard<std::mutex> lk(g_svc.mu);
    if (g_svc.in_use + bytes > g_svc.budget) return fail(PIMUL_ENOMEM, "upload exceeds the HBM budget");
    g_svc.in_use += bytes;
  }
  cudaStream_t st;
  rc = get_stream(&st);
  if (rc) return rc;
  uint64_t* d = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&d, bytes, g_svc.pool, st);
  if (e == cudaSuccess && n && host_to_device(d, host, n * 8, st)) e = cudaErrorUnknown;
  cudaEvent_t ev = nullptr;
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventRecord(ev, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // the host buffer may be reused on return
  std::lock_guard<std::mutex> lk(g_svc.mu);
  if (e != cudaSuccess) {
    g_svc.in_use -= bytes;
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("upload: ") + cudaGetErrorString(e));
  }
  uint64_t id = svc_new_handle(n, d, false, bytes);
  g_svc.handles[id].ready = ev;
  *handle = id;
  return PIMUL_OK;
}

int pimul_submit(int op, uint64_t a, uint64_t b, uint64_t* out_handle, uint64_t* ticket) {
  if (!out_handle || !ticket || op < PIMUL_OP_MUL || op > PIMUL_OP_SUB) return fail(PIMUL_EINVAL, "bad argument");
  int rc = svc_start();
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(g_svc.mu);
  auto ia = g_svc.handles.find(a);
  auto ib = g_svc.handles.find(op == PIMUL_OP_SQR ? a : b);
  if (ia == g_svc.handles.end() || ib == g_svc.handles.end() || ia->second.freed || ib->second.freed)
    return fail(PIMUL_ENOTFOUND, "unknown or freed handle");
  uint64_t la = ia->second.limbs, lb = ib->second.limbs;
  const bool linear = op == PIMUL_OP_ADD || op == PIMUL_OP_SUB;
  // a sum keeps every carry in max + 1 limbs; a difference (a >= b) fits in max
  uint64_t outl = op == PIMUL_OP_ADD ? std::max(la, lb) + 1 : op == PIMUL_OP_SUB ? std::max(la, lb) : la + lb;
  uint64_t obytes = round256(std::max<uint64_t>(outl, 1) * 8);
  const int L = !linear && la && lb ? sizes_for(la, lb).L : 0;
  if (L > 32) return fail(PIMUL_EINVAL, "transform length above 2^32");
  uint64_t scratch = L > SMALL_LOG_MAX ? batch_bytes(la, lb) : 0;
  if (obytes + scratch > g_svc.budget) return fail(PIMUL_ENOMEM, "request larger than the HBM budget");
  uint64_t* d = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync((void**)&d, obytes, g_svc.pool, g_svc.streams[0]);
  // every limb of a result is written, but a zero operand launches nothing
  if (e == cudaSuccess && !linear && (!la || !lb)) e = cudaMemsetAsync(d, 0, obytes, g_svc.streams[0]);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("result allocation: ") + cudaGetErrorString(e));
  }
  // the result buffer must exist before any batch stream writes it
  cudaEvent_t alloc_ev;
  cudaEventCreateWithFlags(&alloc_ev, cudaEventDisableTiming);
  cudaEventRecord(alloc_ev, g_svc.streams[0]);
  g_svc.in_use += obytes;
  uint64_t oid = svc_new_handle(outl, d, true, obytes);
  g_svc.handles[oid].ready = alloc_ev;
  uint64_t t = g_svc.next_ticket++;
  SvcRequest r;
  r.ticket = t;
  r.op = op;
  r.L = L;
  r.a = a;
  r.b = op == PIMUL_OP_SQR ? a : b;
  r.out = oid;
  r.t_submit = now_s();
  r.scratch = scratch;
  g_svc.handles[oid].producer = (int64_t)t;
  ia->second.readers++;
  if (r.b != r.a) g_svc.handles[r.b].readers++;
  g_svc.requests[t] = r;
  g_svc.queue.push_back(t);
  g_svc.dirty = true;
  *out_handle = oid;
  *ticket = t;
  g_svc.cv.notify_one();
  return PIMUL_OK;
}

int pimul_wait(uint64_t ticket, int64_t timeout_us) {
  std::unique_lock<std::mutex> lk(g_svc.mu);
  auto it = g_svc.requests.find(ticket);
  if (it == g_svc.requests.end()) return fail(PIMUL_ENOTFOUND, "unknown ticket");
  SvcRequest* rp = &it->second;  // element pointers survive rehashing
  auto pred = [&] { return rp->state >= 2; };
  if (timeout_us < 0) {
    g_svc.done_cv.wait(lk, pred);
  } else if (!g_svc.done_cv.wait_for(lk, std::chrono::microseconds(timeout_us), pred)) {
    return fail(PIMUL_ETIMEDOUT, "request not finished within the timeout");
  }
  return rp->state == 3 ? fail(PIMUL_ECUDA, "request failed") : PIMUL_OK;
}

int pimul_handle_size(uint64_t handle, size_t* limbs) {
  std::lock_guard<std::mutex> lk(g_svc.mu);
  auto it = g_svc.handles.find(handle);
  if (it == g_svc.handles.end() || it->second.freed || !limbs) return fail(PIMUL_ENOTFOUND, "unknown handle");
  *limbs = it->second.limbs;
  return PIMUL_OK;
}

int pimul_download(uint64_t handle, uint64_t* host, size_t cap, size_t* len) {
  if (!len) return fail(PIMUL_EINVAL, "null len");
  uint64_t* d;
  uint64_t n;
  cudaEvent_t ready;
  int64_t producer;
  {
    std::lock_guard<std::mutex> lk(g_svc.mu);
    auto it = g_svc.handles.find(handle);
    if (it == g_svc.handles.end() || it->second.freed) return fail(PIMUL_ENOTFOUND, "unknown handle");
    d = it->second.d;
    n = it->second.limbs;
    producer = it->second.producer;
  }
  if (producer >= 0) {
    int rc = pimul_wait((uint64_t)producer, -1);
    if (rc) return rc;
  }
  {
    std::lock_guard<std::mutex> lk(g_svc.mu);
    ready = g_svc.handles[handle].ready;
  }
  if (cap < n) return fail(PIMUL_EINVAL, "capacity below the stored length");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (ready) CU(cudaStreamWaitEvent(st, ready, 0));
  rc = device_to_host(host, d, n * 8, st);
  if (rc) return rc;
  size_t m = n;
  while (m && host[m - 1] == 0) m--;
  *len = m;
  return PIMUL_OK;
}

int pimul_free(uint64_t handle) {
  std::unique_lock<std::mutex> lk(g_svc.mu);
  auto it = g_svc.handles.find(handle);
  if (it == g_svc.handles.end() || it->second.freed) return fail(PIMUL_ENOTFOUND, "unknown or already freed handle");
  int64_t producer = it->second.producer;
  lk.unlock();
  if (producer >= 0) pimul_wait((uint64_t)producer, -1);
  lk.lock();
  // requests that read the handle must finish first
  g_svc.done_cv.wait(lk, [&] {
    auto f = g_svc.handles.find(handle);
    return f == g_svc.handles.end() || f->second.readers <= 0;
  });
  auto f = g_svc.handles.find(handle);
  if (f == g_svc.handles.end()) return fail(PIMUL_ENOTFOUND, "handle freed concurrently");
  svc_free_now(handle);
  g_svc.dirty = true;
  return PIMUL_OK;
}

int pimul_release(uint64_t handle) {
  std::lock_guard<std::mutex> lk(g_svc.mu);
  auto it = g_svc.handles.find(handle);
  if (it == g_svc.handles.end() || it->second.freed || it->second.release)
    return fail(PIMUL_ENOTFOUND, "unknown, freed or released handle");
  it->second.release = true;
  if (!it->second.pending && it->second.readers <= 0) {
    svc_free_now(handle);
    g_svc.dirty = true;
  }
  return PIMUL_OK;
}

int pimul_adopt(const uint64_t* d, size_t n, uint64_t* handle) {
  if (!handle || (n && !d)) return fail(PIMUL_EINVAL, "null argument");
  int rc = svc_start();
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(g_svc.mu);
  uint64_t id = svc_new_handle(n, const_cast<uint64_t*>(d), false, 0);
  g_svc.handles[id].borrowed = true;
  *handle = id;
  return PIMUL_OK;
}

int pimul_handle_device(uint64_t handle, const uint64_t** d, size_t* limbs) {
  if (!d || !limbs) return fail(PIMUL_EINVAL, "null argument");
  int64_t producer;
  {
    std::lock_guard<std::mutex> lk(g_svc.mu);
    auto it = g_svc.handles.find(handle);
    if (it == g_svc.handles.end() || it->second.freed) return fail(PIMUL_ENOTFOUND, "unknown handle");
    producer = it->second.producer;
  }
  if (producer >= 0) {
    int rc = pimul_wait((uint64_t)producer, -1);
    if (rc) return rc;
  }
  std::lock_guard<std::mutex> lk(g_svc.mu);
  auto it = g_svc.handles.find(handle);
  if (it == g_svc.handles.end()) return fail(PIMUL_ENOTFOUND, "handle freed concurrently");
  *d = it->second.d;
  *limbs = it->second.limbs;
  return PIMUL_OK;
}

int pimul_service_stats(double* p50_ms, double* p99_ms, uint64_t* completed, uint64_t* batches, uint64_t* in_use) {
  std::lock_guard<std::mutex> lk(g_svc.mu);
  std::vector<double> v = g_svc.latencies;
  std::sort(v.begin(), v.end());
  auto pct = [&](double q) { return v.empty() ? 0.0 : 1e3 * v[std::min(v.size() - 1, (size_t)(q * (v.size() - 1) + 0.5))]; };
  if (p50_ms) *p50_ms = pct(0.50);
  if (p99_ms) *p99_ms = pct(0.99);
  if (completed) *completed = g_svc.completed;
  if (batches) *batches = g_svc.batches;
  if (in_use) *in_use = g_svc.in_use;
  return PIMUL_OK;
}

int pimul_service_config(int big_log_n, int max_batch) {
  std::lock_guard<std::mutex> lk(g_svc.mu);
  if (big_log_n > 0) g_svc.big_log_n = big_log_n;
  if (max_batch > 0) g_svc.max_batch = max_batch;
  g_svc.dirty = true;
  return PIMUL_OK;
}

int pimul_service_reset_stats(void) {
  std::lock_guard<std::mutex> lk(g_svc.mu);
  g_svc.latencies.clear();
  g_svc.completed = 0;
  g_svc.batches = 0;
  return PIMUL_OK;
}

// ------------------------------------------------- batched add / subtract
// out = x + y or x - y (x >= y) for many limb arrays at once, the additions
// and subtractions of a binary-splitting level done where its products
// live.  Windows of 4 limbs add with carry-in 0 and report (generate,
// propagate) and chunks of 256 windows their carry function; a chunk's carry in
// comes from the nearest chunk on its left that has a fixed carry out, or from a
// scan where there are many chunks; windows that receive a carry ripple it (+1 /
// -1) through their limbs.  An array of one chunk is finished by the first
// kernel.  A carry or borrow out of the top limb is reported (it means x < y for
// a subtraction).
constexpr int AS_THREADS = 256;
constexpr int AS_W = 4;

struct AsJob {
  const uint64_t* x;
  const uint64_t* y;
  uint64_t* out;
  uint64_t nx, ny, nout;
  uint8_t* aux;  // per-warp masks, per-chunk (g, p) and carry-in bytes
  uint32_t sub;
  uint32_t check;  // report a carry or borrow out of the top limb
};

__host__ __device__ __forceinline__ uint64_t as_nwin(uint64_t nout) { return (nout + AS_W - 1) / AS_W; }
__host__ __device__ __forceinline__ uint64_t as_nchunk(uint64_t nout) {
  return (as_nwin(nout) + AS_THREADS - 1) / AS_THREADS;
}
__host__ __device__ __forceinline__ uint64_t as_aux_bytes(uint64_t nout) {
  uint64_t nc = as_nchunk(nout);
  return round_up_u64(nc * (AS_THREADS / 32) * 8 + 2 * nc + 16, 16);
}

// Carries of a warp's 32 windows for the carry in of its chunk: bit i is
// window i's carry in.
__device__ __forceinline__ uint32_t as_carries(const uint32_t* A, const uint32_t* B, int stride, int warp, uint32_t cin) {
  for (int k = 0; k < warp; k++) cin = (uint32_t)(((uint64_t)A[k * stride] + B[k * stride] + cin) >> 32);
  const uint32_t a = A[warp * stride], b = B[warp * stride];
  return (a + b + cin) ^ a ^ b;
}
// The top window's carry out (generated, or propagated from its carry in).
__device__ __forceinline__ bool as_out(uint32_t A, uint32_t B, uint32_t carries, int lane) {
  return ((B | (A & carries)) >> lane) & 1;
}

// An array of one chunk is finished here: its carries are known in the CTA.
__global__ void __launch_bounds__(AS_THREADS) k_as_local(const AsJob* jobs, int* overflow) {
  const AsJob J = jobs[blockIdx.y];
  const uint64_t nwin = as_nwin(J.nout), nchunk = as_nchunk(J.nout);
  if (blockIdx.x >= nchunk) return;
  uint32_t* masks = reinterpret_cast<uint32_t*>(J.aux);
  uint8_t* chunk_gp = J.aux + nchunk * (AS_THREADS / 32) * 8;
  __shared__ uint32_t sA[AS_THREADS / 32], sB[AS_THREADS / 32];
  const uint64_t w = (uint64_t)blockIdx.x * AS_THREADS + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool one = nchunk == 1;
  bool g = false, p = false;
  uint64_t z[AS_W];
  if (w < nwin) {
    uint64_t c = 0;
    bool all = true;
#pragma unroll
    for (int t = 0; t < AS_W; t++) {
      const uint64_t i = AS_W * w + t;
      if (i >= J.nout) break;
      const uint64_t xi = i < J.nx ? J.x[i] : 0, yi = i < J.ny ? J.y[i] : 0;
      if (J.sub) {
        const uint64_t d = xi - yi;
        const uint64_t b1 = xi < yi, b2 = d < c;
        z[t] = d - c;
        c = b1 | b2;
        all = all && z[t] == 0;
      } else {
        const uint64_t s0 = xi + yi;
        const uint64_t c1 = s0 < xi;
        z[t] = s0 + c;
        c = c1 | (z[t] < s0);
        all = all && z[t] == ~0ull;
      }
      if (!one) J.out[i] = z[t];
    }
    g = c != 0;
    p = all;
  }
  const uint32_t A = __ballot_sync(0xFFFFFFFFu, g || p);
  const uint32_t Bm = __ballot_sync(0xFFFFFFFFu, g);
  if (lane == 0) {
    if (!one) {
      const uint64_t wi = (uint64_t)blockIdx.x * (AS_THREADS / 32) + warp;
      masks[2 * wi] = A;
      masks[2 * wi + 1] = Bm;
    }
    sA[warp] = A;
    sB[warp] = Bm;
  }
  __syncthreads();
  if (one) {
    const uint32_t carries = as_carries(sA, sB, 1, warp, 0);
    if (J.check && w + 1 == nwin && as_out(A, Bm, carries, lane)) atomicExch(overflow, 1);
    if (w < nwin) {
      bool c = (carries >> lane) & 1;
#pragma unroll
      for (int t = 0; t < AS_W; t++) {
        const uint64_t i = AS_W * w + t;
        if (i >= J.nout) break;
        if (c) {
          c = z[t] == (J.sub ? 0 : ~0ull);
          z[t] += J.sub ? ~0ull : 1;
        }
        J.out[i] = z[t];
      }
    }
    return;
  }
  if (threadIdx.x == 0) {
    uint32_t cg = 0, cp = 1;  // chunk carry out for carry in 0 / 1
    for (int k = 0; k < AS_THREADS / 32; k++) {
      uint64_t sg = (uint64_t)sA[k] + sB[k] + cg;
      uint64_t sp = (uint64_t)sA[k] + sB[k] + cp;
      cg = (uint32_t)(sg >> 32);
      cp = (uint32_t)(sp >> 32);
    }
    chunk_gp[blockIdx.x] = (uint8_t)(cg | (cp << 1));
  }
}

// Arrays of up to AS_LOOK chunks look left for a chunk's carry in (as_carry_in);
// longer ones, whose look-back over an all-propagating array would cost more,
// have it scanned.  The scan takes 14 us whatever the length; a look-back is one
// byte in general and at most AS_LOOK / 512 steps of about 1 us (pi to 10^5, 10^6,
// 10^8 digits 7.64 -> 7.34, 11.97 -> 11.67, 205.3 -> 203.1 ms, one-chunk arrays in one
// kernel included).
constexpr uint64_t AS_LOOK = 2048;

// Carry into a chunk: that out of the nearest chunk on its left whose carry out
// does not depend on its carry in (all lanes of the warp call).
__device__ uint32_t as_carry_in(const uint8_t* chunk_gp, uint64_t chunk, int lane) {
  if (chunk == 0) return 0;
  const uint32_t f = chunk_gp[chunk - 1];
  if (f != 2) return f & 1;
  for (int64_t base = (int64_t)((chunk - 1) & ~511ull); base >= 0; base -= 512) {
    uint32_t near = 2;  // of this lane's 16 chunks
#pragma unroll
    for (int t = 0; t < 16; t++) {
      const uint64_t c = (uint64_t)base + 16 * lane + t;
      const uint32_t v = c < chunk ? chunk_gp[c] : 2;
      if (v != 2) near = v;
    }
    const uint32_t fixed = __ballot_sync(0xFFFFFFFFu, near != 2);
    if (fixed) return __shfl_sync(0xFFFFFFFFu, near, 31 - __clz((int)fixed)) & 1;
  }
  return 0;
}

// One CTA per job: carry into every chunk (segments of chunks per thread,
// chained by thread 0).
__global__ void __launch_bounds__(1024) k_as_scan(const AsJob* jobs) {
  const AsJob J = jobs[blockIdx.x];
  const uint64_t nchunk = as_nchunk(J.nout);
  if (nchunk <= AS_LOOK) return;
  const uint8_t* chunk_gp = J.aux + nchunk * (AS_THREADS / 32) * 8;
  uint8_t* chunk_cin = J.aux + nchunk * (AS_THREADS / 32) * 8 + nchunk;
  __shared__ uint8_t seg_g[1024], seg_p[1024], seg_cin[1024];
  const uint64_t per = (nchunk + 1023) / 1024;
  const uint64_t lo = threadIdx.x * per, hi = lo + per < nchunk ? lo + per : nchunk;
  uint8_t cg = 0, cp = 1;
  for (uint64_t k = lo; k < hi; k++) {
    uint8_t gp = chunk_gp[k];
    uint8_t o0 = gp & 1, o1 = (gp >> 1) & 1;
    cg = cg ? o1 : o0;
    cp = cp ? o1 : o0;
  }
  seg_g[threadIdx.x] = cg;
  seg_p[threadIdx.x] = cp;
  __syncthreads();
  if (threadIdx.x == 0) {
    // only the first ceil(nchunk / per) segments hold chunks
    const int used = (int)((nchunk + per - 1) / per);
    uint8_t cin = 0;
    for (int k = 0; k < used; k++) {
      seg_cin[k] = cin;
      cin = cin ? seg_p[k] : seg_g[k];
    }
  }
  __syncthreads();
  uint8_t cin = seg_cin[threadIdx.x];
  for (uint64_t k = lo; k < hi; k++) {
    chunk_cin[k] = cin;
    uint8_t gp = chunk_gp[k];
    cin = cin ? ((gp >> 1) & 1) : (gp & 1);
  }
}

// Windows that receive a carry ripple it; the top window's carry out
// (generated, or propagated from its carry in) sets *overflow.
__global__ void __launch_bounds__(AS_THREADS) k_as_apply(const AsJob* jobs, int* overflow) {
  const AsJob J = jobs[blockIdx.y];
  const uint64_t nwin = as_nwin(J.nout), nchunk = as_nchunk(J.nout);
  if (blockIdx.x >= nchunk || nchunk == 1) return;
  const uint32_t* masks = reinterpret_cast<const uint32_t*>(J.aux) + 2 * (uint64_t)blockIdx.x * (AS_THREADS / 32);
  const uint8_t* chunk_gp = J.aux + nchunk * (AS_THREADS / 32) * 8;
  const uint64_t w = (uint64_t)blockIdx.x * AS_THREADS + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t cin = nchunk > AS_LOOK ? chunk_gp[nchunk + blockIdx.x] : as_carry_in(chunk_gp, blockIdx.x, lane);
  const uint32_t carries = as_carries(masks, masks + 1, 2, warp, cin);
  if (J.check && w + 1 == nwin && as_out(masks[2 * warp], masks[2 * warp + 1], carries, lane)) atomicExch(overflow, 1);
  if (w < nwin && ((carries >> lane) & 1)) {
    for (int t = 0; t < AS_W; t++) {
      const uint64_t i = AS_W * w + t;
      if (i >= J.nout) break;
      if (J.sub) {
        if (J.out[i]-- != 0) break;
      } else {
        if (++J.out[i] != 0) break;
      }
    }
  }
}

// Highest nonzero limb + 1 of each array (0 for zero): *len must be zero
// on entry; CTAs scan 2^12-limb chunks and keep the maximum.
__global__ void __launch_bounds__(256) k_top_limb(const uint64_t* const* arrs, const uint64_t* n, uint64_t* len) {
  const uint32_t j = blockIdx.y;
  const uint64_t lo = (uint64_t)blockIdx.x << 12;
  if (lo >= n[j]) return;
  const uint64_t hi = lo + 4096 < n[j] ? lo + 4096 : n[j];
  const uint64_t* a = arrs[j];
  uint64_t best = 0;
  for (uint64_t i = lo + threadIdx.x; i < hi; i += 256)
    if (a[i]) best = i + 1;
  for (int o = 16; o > 0; o >>= 1) {
    uint64_t other = __shfl_down_sync(0xFFFFFFFFu, best, o);
    best = other > best ? other : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax((unsigned long long*)&len[j], (unsigned long long)best);
}

static void as_launch(const AsJob* jobs, size_t n, uint64_t max_chunk, cudaStream_t st, int* d_overflow) {
  for (size_t j0 = 0; j0 < n; j0 += 65535) {
    const unsigned nj = (unsigned)std::min<size_t>(65535, n - j0);
    const dim3 grid((unsigned)max_chunk, nj);
    k_as_local<<<grid, AS_THREADS, 0, st>>>(jobs + j0, d_overflow);
    if (max_chunk > AS_LOOK) k_as_scan<<<nj, 1024, 0, st>>>(jobs + j0);
    if (max_chunk > 1) k_as_apply<<<grid, AS_THREADS, 0, st>>>(jobs + j0, d_overflow);
  }
}

// Batched add/subtract on `st` (asynchronous); *d_overflow (device int,
// zeroed by the caller) is set when a carry or borrow leaves a top limb.
static int addsub_launch(const pimul_addsub_job* jobs, size_t n, cudaStream_t st, int* d_overflow, bool unchecked) {
  if (n == 0) return PIMUL_OK;
  uint64_t aux_total = 0, max_chunk = 0;
  for (size_t i = 0; i < n; i++) {
    aux_total += as_aux_bytes(jobs[i].nout);
    max_chunk = std::max<uint64_t>(max_chunk, as_nchunk(jobs[i].nout));
  }
  const uint64_t desc = round_up_u64(n * sizeof(AsJob), 256);
  uint8_t* dev = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&dev, desc + aux_total, g_dev.pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("add/subtract scratch: ") + cudaGetErrorString(e));
  }
  AsJob* h = reinterpret_cast<AsJob*>(host_image(n * sizeof(AsJob)));
  uint64_t off = desc;
  for (size_t i = 0; i < n; i++) {
    h[i] = AsJob{jobs[i].x, jobs[i].y, jobs[i].out, jobs[i].nx, jobs[i].ny, jobs[i].nout, dev + off,
                 (uint32_t)(jobs[i].sub != 0), (uint32_t)(!unchecked && jobs[i].sub != PIMUL_SUB_MOD)};
    off += as_aux_bytes(jobs[i].nout);
  }
  if (host_to_device(dev, h, n * sizeof(AsJob), st)) e = cudaErrorUnknown;
  if (e == cudaSuccess) {
    as_launch(reinterpret_cast<const AsJob*>(dev), n, max_chunk, st, d_overflow);
    e = cudaGetLastError();
  }
  // the host image is pageable: the copy has been staged before return
  cudaFreeAsync(dev, st);
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("add/subtract launch: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}

int pimul_addsub_batch(const pimul_addsub_job* jobs, size_t n, void* stream) {
  if (n && !jobs) return fail(PIMUL_EINVAL, "null job list");
  for (size_t i = 0; i < n; i++) {
    const pimul_addsub_job& j = jobs[i];
    if (j.nout && !j.out) return fail(PIMUL_EINVAL, "null output");
    if ((j.nx && !j.x) || (j.ny && !j.y)) return fail(PIMUL_EINVAL, "null operand");
    if (j.nout < std::max(j.nx, j.ny)) return fail(PIMUL_EINVAL, "output shorter than an operand");
  }
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  int* d_flag = nullptr;
  CU(cudaMallocAsync((void**)&d_flag, sizeof(int), g_dev.pool, st));
  CU(cudaMemsetAsync(d_flag, 0, sizeof(int), st));
  bool all_mod = true;
  for (size_t i = 0; i < n && all_mod; i++) all_mod = jobs[i].sub == PIMUL_SUB_MOD;
  rc = addsub_launch(jobs, n, st, d_flag, false);
  if (all_mod) {  // nothing to check: stay asynchronous
    cudaFreeAsync(d_flag, st);
    return rc;
  }
  int h_flag = 0;
  if (!rc) {
    cudaError_t e = cudaMemcpyAsync(&h_flag, d_flag, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = fail(PIMUL_ECUDA, std::string("add/subtract: ") + cudaGetErrorString(e));
  }
  cudaFreeAsync(d_flag, st);
  if (!rc && h_flag) rc = fail(PIMUL_EINVAL, "carry or borrow out of the top limb (x < y in a subtraction?)");
  return rc;
}

// Wrapped products (PIMUL_BATCH_WRAP): a unit of 2^20 points or more whose
// coefficients fill at most 5/8 of its transform, with every operand within
// half of it, runs as a cyclic product of half the length; the coefficients
// that wrap around (wrap of them, at most a quarter of the half length) are
// separated again with the exact low coefficients of the product, from a
// short product of the operands' low limbs computed first (coefficients
// out, no carry).  plan_wraps marks the eligible units (forceL, wrap) and
// returns their short products, whose output buffers (and the units' low
// pointers) the caller assigns from one allocation of `words` words.
struct WrapPlan {
  std::vector<Unit> low;      // the short products, in the order of the wrapped units
  std::vector<size_t> which;  // the wrapped units
  uint64_t words = 0;
};

static WrapPlan plan_wraps(std::vector<Unit>& units) {
  WrapPlan W;
  for (size_t i = 0; i < units.size(); i++) {
    Unit& u = units[i];
    if (u.coeff || u.forceL || !u.la || !u.lb) continue;
    const int L = log2_ceil(4 * u.nout - 1);
    if (L < 20 || L > 32) continue;
    const uint64_t Nw = 1ull << (L - 1);
    const uint64_t n1 = 4 * (u.la + u.lb), n2 = u.la2 ? 4 * (u.la2 + u.lb2) : 0;
    const uint64_t ncoef = std::max(n1, n2) - 1;
    if (ncoef <= Nw || ncoef - Nw > Nw / 4) continue;
    if (4 * u.la > Nw || 4 * u.lb > Nw || 4 * u.la2 > Nw || 4 * u.lb2 > Nw) continue;
    const uint64_t m = ncoef - Nw, ml = (m + 3) / 4;  // wrapped coefficients; limbs holding them
    Unit lo{};
    lo.a = u.a, lo.la = std::min(u.la, ml), lo.b = u.b, lo.lb = std::min(u.lb, ml);
    if (u.la2) lo.a2 = u.a2, lo.la2 = std::min(u.la2, ml), lo.b2 = u.b2, lo.lb2 = std::min(u.lb2, ml);
    const uint64_t nl = std::max(4 * (lo.la + lo.lb), lo.la2 ? 4 * (lo.la2 + lo.lb2) : 0) - 1;
    lo.forceL = std::max(SMALL_LOG_MAX + 1, log2_ceil(nl));
    lo.coeff = true;
    lo.nout = m;
    W.low.push_back(lo);
    W.which.push_back(i);
    u.forceL = L - 1;
    u.wrap = m;
    W.words += round_up_u64(m, 32);
  }
  return W;
}

static int sum_batch_impl(const pimul_sum_job* jobs, size_t n, cudaStream_t st, bool allow_wrap);

int pimul_sum_batch(const pimul_sum_job* jobs, size_t n, void* stream) {
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  return sum_batch_impl(jobs, n, st, false);
}

int pimul_sum_batch_ex(const pimul_sum_job* jobs, size_t n, void* stream, unsigned flags) {
  if (flags & ~PIMUL_BATCH_WRAP) return fail(PIMUL_EINVAL, "unknown batch flags");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  return sum_batch_impl(jobs, n, st, (flags & PIMUL_BATCH_WRAP) != 0);
}

static int sum_batch_impl(const pimul_sum_job* jobs, size_t n, cudaStream_t st, bool allow_wrap) {
  int rc = PIMUL_OK;
  if (n && !jobs) return fail(PIMUL_EINVAL, "null job list");
  // fused sums go to the pass pipeline; a sum of short products (or with a
  // square) is two products into scratch and one batched addition
  std::vector<Unit> units;
  units.reserve(n);
  std::vector<size_t> fb;  // jobs computed as two products + an addition
  std::vector<std::pair<uint64_t*, uint64_t>> zero;  // output limbs above the result
  uint64_t tmp_words = 0;
  for (size_t i = 0; i < n; i++) {
    const pimul_sum_job& j = jobs[i];
    const bool p1 = j.la1 && j.lb1, p2 = j.la2 && j.lb2;
    if ((p1 && (!j.a1 || !j.b1)) || (p2 && (!j.a2 || !j.b2))) return fail(PIMUL_EINVAL, "null operand");
    const uint64_t n1 = p1 ? j.la1 + j.lb1 : 0, n2 = p2 ? j.la2 + j.lb2 : 0;
    const uint64_t need = std::max(n1, n2) + (p1 && p2 ? 1 : 0);
    if (j.nout < need) return fail(PIMUL_EINVAL, "nout below max(la1 + lb1, la2 + lb2) + 1");
    if (j.nout && !j.out) return fail(PIMUL_EINVAL, "null output");
    if (j.nout > need) zero.emplace_back(j.out + need, j.nout - need);
    if (!p1 && !p2) continue;
    if (p1 != p2) {
      units.push_back(p1 ? Unit{j.a1, j.la1, j.b1, j.lb1, nullptr, 0, nullptr, 0, j.out, n1}
                         : Unit{j.a2, j.la2, j.b2, j.lb2, nullptr, 0, nullptr, 0, j.out, n2});
      continue;
    }
    const bool sq = (j.a1 == j.b1 && j.la1 == j.lb1) || (j.a2 == j.b2 && j.la2 == j.lb2);
    const int L = log2_ceil(4 * need - 1);
    if (L > 32) return fail(PIMUL_EINVAL, "transform length above 2^32 in batch");
    // fused only when both products already need that transform length (a
    // shorter second product would run at twice its own length)
    const bool same = log2_ceil(4 * n1 - 1) == L && log2_ceil(4 * n2 - 1) == L;
    if (sq || L <= SMALL_LOG_MAX || !same) {
      fb.push_back(i);
      tmp_words += n1 + n2;
      continue;
    }
    units.push_back(Unit{j.a1, j.la1, j.b1, j.lb1, j.a2, j.la2, j.b2, j.lb2, j.out, need});
  }
  uint8_t* tmp = nullptr;
  std::vector<pimul_addsub_job> aj;
  if (!fb.empty()) {
    CU(cudaMallocAsync((void**)&tmp, tmp_words * 8 + 256, g_dev.pool, st));
    uint64_t* t = reinterpret_cast<uint64_t*>(tmp + 256);  // first 256 bytes: the overflow flag
    for (size_t i : fb) {
      const pimul_sum_job& j = jobs[i];
      const uint64_t n1 = j.la1 + j.lb1, n2 = j.la2 + j.lb2;
      units.push_back(Unit{j.a1, j.la1, j.b1, j.lb1, nullptr, 0, nullptr, 0, t, n1});
      units.push_back(Unit{j.a2, j.la2, j.b2, j.lb2, nullptr, 0, nullptr, 0, t + n1, n2});
      aj.push_back(pimul_addsub_job{t, n1, t + n1, n2, j.out, std::max(n1, n2) + 1, 0});
      t += n1 + n2;
    }
  }
  for (const auto& z : zero) {
    cudaError_t e = cudaMemsetAsync(z.first, 0, z.second * 8, st);
    if (e != cudaSuccess && !rc) rc = fail(PIMUL_ECUDA, std::string("sum batch: ") + cudaGetErrorString(e));
  }
  // wrapped units: their low coefficients first, into one buffer
  uint64_t* lowbuf = nullptr;
  if (!rc && allow_wrap) {
    WrapPlan W = plan_wraps(units);
    if (!W.low.empty()) {
      cudaError_t e = cudaMallocAsync((void**)&lowbuf, W.words * 8, g_dev.pool, st);
      if (e != cudaSuccess) {
        cudaGetLastError();
        rc = fail(PIMUL_ENOMEM, std::string("wrapped products: ") + cudaGetErrorString(e));
      } else {
        uint64_t off = 0;
        for (size_t k = 0; k < W.low.size(); k++) {
          W.low[k].out = lowbuf + off;
          units[W.which[k]].low = lowbuf + off;
          off += round_up_u64(W.low[k].nout, 32);
        }
        rc = run_units(W.low.data(), W.low.size(), st, true);
      }
    }
  }
  if (!rc) rc = run_units(units.data(), units.size(), st, true);
  if (lowbuf) cudaFreeAsync(lowbuf, st);
  if (!rc && !aj.empty()) {
    cudaError_t e = cudaMemsetAsync(tmp, 0, sizeof(int), st);
    if (e == cudaSuccess) rc = addsub_launch(aj.data(), aj.size(), st, reinterpret_cast<int*>(tmp), false);
    else rc = fail(PIMUL_ECUDA, std::string("sum batch: ") + cudaGetErrorString(e));
  }
  if (tmp) cudaFreeAsync(tmp, st);
  return rc;
}

int pimul_top_limbs(const uint64_t* const* arrays, const size_t* lens, size_t n, size_t* out_lens, void* stream) {
  if (n == 0) return PIMUL_OK;
  if (!arrays || !lens || !out_lens) return fail(PIMUL_EINVAL, "null argument");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  uint64_t max_chunk = 0;
  for (size_t i = 0; i < n; i++) max_chunk = std::max<uint64_t>(max_chunk, (lens[i] + 4095) / 4096);
  if (max_chunk == 0) {
    for (size_t i = 0; i < n; i++) out_lens[i] = 0;
    return PIMUL_OK;
  }
  const uint64_t bytes = round_up_u64(n * 8, 256);
  uint8_t* dev = nullptr;
  CU(cudaMallocAsync((void**)&dev, 3 * bytes, g_dev.pool, st));
  std::vector<uint64_t> hn(lens, lens + n);
  if (!rc) rc = host_to_device(dev, arrays, n * 8, st);
  if (!rc) rc = host_to_device(dev + bytes, hn.data(), n * 8, st);
  if (rc) {
    cudaFreeAsync(dev, st);
    return rc;
  }
  CU(cudaMemsetAsync(dev + 2 * bytes, 0, n * 8, st));
  for (size_t j0 = 0; j0 < n; j0 += 65535) {
    const unsigned nj = (unsigned)std::min<size_t>(65535, n - j0);
    k_top_limb<<<dim3((unsigned)max_chunk, nj), 256, 0, st>>>(
        reinterpret_cast<const uint64_t* const*>(dev) + j0, reinterpret_cast<const uint64_t*>(dev + bytes) + j0,
        reinterpret_cast<uint64_t*>(dev + 2 * bytes) + j0);
  }
  CU(cudaGetLastError());
  std::vector<uint64_t> res(n);
  rc = device_to_host(res.data(), dev + 2 * bytes, n * 8, st);
  cudaFreeAsync(dev, st);
  if (rc) return rc;
  for (size_t i = 0; i < n; i++) out_lens[i] = (size_t)res[i];
  return PIMUL_OK;
}

// pimul_mul's contract through the served form: upload, submit, wait,
// download, free.  A drop-in multiply backend for host drivers that want
// every product to pass through the service.
int pimul_mul_served(const uint64_t* a, size_t la, const uint64_t* b, size_t lb, uint64_t* out, size_t out_cap,
                     size_t* out_len) {
  if (!out_len) return fail(PIMUL_EINVAL, "null out_len");
  *out_len = 0;
  if (la == 0 || lb == 0) return PIMUL_OK;
  if (!a || !b || !out) return fail(PIMUL_EINVAL, "null pointer");
  if (out_cap < la + lb) return fail(PIMUL_EINVAL, "out_cap < la + lb");
  const bool sq = a == b && la == lb;
  uint64_t ha = 0, hb = 0, hc = 0, ticket = 0;
  bool has_a = false, has_b = false, has_c = false;
  int rc = pimul_upload(a, la, &ha);
  has_a = rc == PIMUL_OK;
  if (!rc && !sq) {
    rc = pimul_upload(b, lb, &hb);
    has_b = rc == PIMUL_OK;
  }
  if (!rc) {
    rc = pimul_submit(sq ? PIMUL_OP_SQR : PIMUL_OP_MUL, ha, sq ? ha : hb, &hc, &ticket);
    has_c = rc == PIMUL_OK;
  }
  if (!rc) rc = pimul_wait(ticket, -1);
  if (!rc) rc = pimul_download(hc, out, out_cap, out_len);
  if (has_c) pimul_free(hc);
  if (has_b) pimul_free(hb);
  if (has_a) pimul_free(ha);
  return rc;
}

int pimul_mul_device(const uint64_t* d_a, size_t la, const uint64_t* d_b, size_t lb, uint64_t* d_out,
                     void* stream) {
  if (la && lb && (!d_a || !d_b || !d_out)) return fail(PIMUL_EINVAL, "null device pointer");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  if (stream) st = (cudaStream_t)stream;
  return mul_device(d_a, la, d_b, lb, d_out, st);
}

// pimul_mul for operands of up to 1 MiB in all, in pageable memory: both go up
// in one copy from a pinned slot into one allocation that also holds the
// product and the scratch.  The longer way overlaps b's upload with a's
// transform, which costs four stream operations and a launch per operand and
// pass: 130 us against 99 at 33001 x 32003 limbs.
constexpr int SMALL_DECLINED = -1;  // no pinned slot
static int mul_host_small(const uint64_t* a, size_t la, const uint64_t* b, size_t lb, bool square, uint64_t* out,
                          cudaStream_t st) {
  const size_t off_b = round256(la * 8), off_out = off_b + (square ? 0 : round256(lb * 8));
  const size_t off_s = off_out + round256((la + lb) * 8);
  const size_t scratch = sizes_for(la, lb).L > g_dev.lone_log ? scratch_bytes(la, lb, square) : 0;
  uint8_t* d = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&d, off_s + scratch, g_dev.pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("operand allocation: ") + cudaGetErrorString(e));
  }
  if (!ring_upload(d, a, la * 8, st, &e, square ? nullptr : b, off_b, square ? 0 : lb * 8)) {
    cudaFreeAsync(d, st);
    return SMALL_DECLINED;
  }
  int rc = e == cudaSuccess ? PIMUL_OK : fail(PIMUL_ECUDA, std::string("upload: ") + cudaGetErrorString(e));
  uint64_t* da = reinterpret_cast<uint64_t*>(d);
  uint64_t* dout = reinterpret_cast<uint64_t*>(d + off_out);
  if (!rc) rc = mul_device(da, la, square ? da : reinterpret_cast<uint64_t*>(d + off_b), lb, dout, st, nullptr, d + off_s);
  if (!rc) rc = device_to_host(out, dout, (la + lb) * 8, st);
  cudaFreeAsync(d, st);
  if (rc) cudaStreamSynchronize(st);
  return rc;
}

int pimul_mul(const uint64_t* a, size_t la, const uint64_t* b, size_t lb, uint64_t* out, size_t out_cap,
              size_t* out_len) {
  if (!out_len) return fail(PIMUL_EINVAL, "null out_len");
  *out_len = 0;
  if (la == 0 || lb == 0) return PIMUL_OK;  // empty means zero (ntt.rs:807-809)
  if (!a || !b || !out) return fail(PIMUL_EINVAL, "null pointer");
  if (out_cap < la + lb) return fail(PIMUL_EINVAL, "out_cap < la + lb");
  if (log2_ceil(4 * (uint64_t)la + 4 * (uint64_t)lb - 1) > 32)
    return fail(PIMUL_EINVAL, "transform length above 2^32");
  cudaStream_t st;
  int rc = get_stream(&st);
  if (rc) return rc;
  const bool square = a == b && la == lb;
  if (8 * (la + lb) + 256 <= STAGE_MIN && is_pageable(a) && (square || is_pageable(b))) {
    const int small = mul_host_small(a, la, b, lb, square, out, st);
    if (small != SMALL_DECLINED) {
      if (small) return small;
      size_t n = la + lb;
      while (n && out[n - 1] == 0) n--;
      *out_len = n;
      return PIMUL_OK;
    }
  }
  uint64_t *da = nullptr, *db = nullptr, *dout = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&da, la * 8, g_dev.pool, st);
  if (e == cudaSuccess && !square) e = cudaMallocAsync((void**)&db, lb * 8, g_dev.pool, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&dout, (la + lb) * 8, g_dev.pool, st);
  if (e != cudaSuccess) {
    if (da) cudaFreeAsync(da, st);
    if (db) cudaFreeAsync(db, st);
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("operand allocation: ") + cudaGetErrorString(e));
  }
  // a is uploaded first; b follows on a helper stream while a's forward
  // transform runs, and b's first pass waits for it
  rc = host_to_device(da, a, la * 8, st);
  thread_local cudaStream_t t_copy = nullptr;
  thread_local cudaEvent_t t_ev[2] = {nullptr, nullptr};
  thread_local int t_copy_dev = -1;
  cudaEvent_t b_ready = nullptr;
  if (!square) {
    if (!t_copy || t_copy_dev != g_dev.device) {
      CU(cudaStreamCreateWithFlags(&t_copy, cudaStreamNonBlocking));
      CU(cudaEventCreateWithFlags(&t_ev[0], cudaEventDisableTiming));
      CU(cudaEventCreateWithFlags(&t_ev[1], cudaEventDisableTiming));
      t_copy_dev = g_dev.device;
    }
    CU(cudaEventRecord(t_ev[0], st));  // after db's allocation and a's upload
    CU(cudaStreamWaitEvent(t_copy, t_ev[0], 0));
    if (!rc) rc = host_to_device(db, b, lb * 8, t_copy);
    CU(cudaEventRecord(t_ev[1], t_copy));
    b_ready = t_ev[1];
  }
  if (!rc) rc = mul_device(da, la, square ? da : db, lb, dout, st, b_ready);
  if (rc && b_ready) cudaStreamWaitEvent(st, b_ready, 0);  // db is freed below
  if (rc == PIMUL_OK) rc = device_to_host(out, dout, (la + lb) * 8, st);
  cudaFreeAsync(da, st);
  if (db) cudaFreeAsync(db, st);
  cudaFreeAsync(dout, st);
  cudaError_t se = cudaStreamSynchronize(st);
  if (rc) return rc;
  if (se != cudaSuccess) return fail(PIMUL_ECUDA, std::string("multiply: ") + cudaGetErrorString(se));
  size_t n = la + lb;
  while (n && out[n - 1] == 0) n--;  // trimmed, as the reference's unpack (ntt.rs:713-716)
  *out_len = n;
  return PIMUL_OK;
}

}  // extern "C"

// ====================================================================
// Multiply entry point that allocates nothing (pimul_mul_device_noalloc)
// ====================================================================
// Some callers cannot allocate device memory at the moment they multiply:
// a host that has handed the whole GPU to another allocator (a framework's
// caching allocator, a fixed arena reserved at start-up), a latency-bound
// loop where cudaMalloc's implicit device synchronisation is not allowed,
// or an embedding runtime whose rule is "allocate at init, never in the
// steady state".  For them this variant takes its scratch from a
// file-scope device array instead of the stream-ordered pool.
//
// Limits and sharing rules:
//  * scratch holds two transform arrays of at most 2^20 words plus the carry
//    windows and chunk states: la + lb <= 262144 limbs (transform length
//    N <= 2^20); larger products are rejected with PIMUL_EINVAL.  The
//    scratch (17 MiB) and this path's own root tables (18 MiB) stay
//    resident on every GPU that loads this library, until the process exits.
//  * every call uses the same array, and the array keeps the previous call's
//    contents; the kernels overwrite every scratch word before reading it,
//    so nothing needs clearing.  Calls whose work overlaps on the GPU
//    (different streams, or different host threads without ordering) race
//    on the array and corrupt each other's results: serialise them.
//  * the first call on each device does a one-time set-up with that device
//    current: it resolves the arrays' device addresses with
//    cudaGetSymbolAddress and copies the root tables in with a synchronous
//    cudaMemcpyToSymbol.  Make that first call before any stream capture.
//    pimul_shutdown forgets the set-up, so a call after a cudaDeviceReset
//    (made after pimul_shutdown) resolves the addresses and copies the
//    tables again.
namespace pimul {
// The service's additions and subtractions: no carry or borrow can leave
// their outputs (sums get max + 1 limbs, differences are of a >= b), so the
// batch is launched unchecked and stays asynchronous.
int svc_addsub(const pimul_addsub_job* jobs, size_t n, cudaStream_t st) {
  return ::addsub_launch(jobs, n, st, nullptr, true);
}

// ---- strided batches: n operations of one shape at fixed strides --------
// (a level of the decimal conversion holds up to 5 * 10^5 nodes of one
// shape).  The descriptors are written by a kernel instead of the host, so
// queueing such a batch costs a few launches whatever n is.

// Descriptors and chunks of n products (a + i sa) * b -> out + i so, all of
// one class (transform length up to 2^SMALL_LOG_MAX), per products per chunk.
__global__ void k_fill_small(SmallJob* jobs, SmallChunk* chunks, SmallJob base, uint64_t sa, uint64_t so, uint32_t n,
                             uint32_t per, int c) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  jobs[i] = SmallJob{base.a + (uint64_t)i * sa, base.b, base.out + (uint64_t)i * so, base.la, base.lb};
  if (i < ((uint64_t)n + per - 1) / per) chunks[i] = SmallChunk{i * per, per < n - i * per ? per : n - i * per, c};
}

int mul_batch_strided(const uint64_t* a, uint64_t sa, size_t la, const uint64_t* b, size_t lb, uint64_t* out,
                      uint64_t so, size_t n, cudaStream_t st) {
  if (!n) return PIMUL_OK;
  const int L = la && lb ? log2_ceil(4 * (uint64_t)(la + lb) - 1) : -1;
  if (L < 0 || L > SMALL_LOG_MAX || n > 0xFFFFFFFFull) {
    // the pass pipeline, or an empty product: the general batch
    std::vector<pimul_job> jobs(n);
    for (size_t i = 0; i < n; i++) jobs[i] = pimul_job{a + i * sa, la, b, lb, out + i * so};
    return pimul_mul_batch(jobs.data(), n, st);
  }
  cudaStream_t own;
  int rc = get_stream(&own);  // initialises the engine on first use
  if (rc) return rc;
  const int c = small_class(la, lb);
  const uint32_t per = small_per_cta(c);
  const size_t nch = (n + per - 1) / per;
  const size_t jb = round256(n * sizeof(SmallJob));
  uint8_t* dev = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&dev, jb + nch * sizeof(SmallChunk), g_dev.pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("strided batch descriptors: ") + cudaGetErrorString(e));
  }
  SmallJob* dj = reinterpret_cast<SmallJob*>(dev);
  SmallChunk* dc = reinterpret_cast<SmallChunk*>(dev + jb);
  k_fill_small<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dj, dc, SmallJob{a, b, out, (uint32_t)la, (uint32_t)lb},
                                                           sa, so, (uint32_t)n, per, c);
  if (c == 11 && n <= CLUSTER_FEW) {
    launch_clusters(dj, (unsigned)n, g_dev.roots, st);
  } else {
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g_dev.device);
    const uint64_t grid = std::min<uint64_t>((uint64_t)sms * (uint64_t)g_small_ctas_per_sm.load(), nch);
    launch_pdl(k_small_mul, dim3((unsigned)grid), SMALL_THREADS, small_cta_smem(c), st, dj, dc, (uint32_t)nch, g_dev.roots);
  }
  e = cudaGetLastError();
  cudaFreeAsync(dev, st);
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("strided batch launch: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}

__global__ void k_fill_as(AsJob* jobs, AsJob base, uint64_t sx, uint64_t sy, uint64_t so, uint64_t saux, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  AsJob j = base;
  j.x += (uint64_t)i * sx;
  j.y += (uint64_t)i * sy;
  j.out += (uint64_t)i * so;
  j.aux += (uint64_t)i * saux;
  jobs[i] = j;
}

int addsub_strided(const uint64_t* x, uint64_t sx, size_t nx, const uint64_t* y, uint64_t sy, size_t ny, uint64_t* out,
                   uint64_t so, size_t nout, int sub, size_t n, cudaStream_t st) {
  if (!n || !nout) return PIMUL_OK;
  if (nout < std::max(nx, ny)) return fail(PIMUL_EINVAL, "output shorter than an operand");
  if (n > 0xFFFFFFFFull) {
    std::vector<pimul_addsub_job> jobs(n);
    for (size_t i = 0; i < n; i++) jobs[i] = pimul_addsub_job{x + i * sx, nx, y + i * sy, ny, out + i * so, nout, sub};
    return svc_addsub(jobs.data(), n, st);
  }
  const uint64_t saux = as_aux_bytes(nout), nchunk = as_nchunk(nout);
  const uint64_t desc = round_up_u64(n * sizeof(AsJob), 256);
  uint8_t* dev = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&dev, desc + n * saux, g_dev.pool, st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(PIMUL_ENOMEM, std::string("strided add/subtract scratch: ") + cudaGetErrorString(e));
  }
  AsJob* dj = reinterpret_cast<AsJob*>(dev);
  k_fill_as<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
      dj, AsJob{x, y, out, nx, ny, nout, dev + desc, (uint32_t)(sub != 0), 0u}, sx, sy, so, saux, (uint32_t)n);
  as_launch(dj, n, nchunk, st, nullptr);
  e = cudaGetLastError();
  cudaFreeAsync(dev, st);
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("strided add/subtract launch: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}
}  // namespace pimul

namespace pimul {
constexpr int NOALLOC_LOG_MAX = 20;
constexpr uint64_t NOALLOC_N_MAX = 1ull << NOALLOC_LOG_MAX;
constexpr uint64_t NOALLOC_WIN_MAX = NOALLOC_N_MAX / WIN_COEFFS;
constexpr uint64_t NOALLOC_CARRY_WORDS = NOALLOC_WIN_MAX + (NOALLOC_WIN_MAX / CARRY_THREADS + 2) / 2;

static __device__ __align__(256) uint64_t g_noalloc_scratch[2 * NOALLOC_N_MAX + NOALLOC_CARRY_WORDS];
static __device__ __align__(256) uint64_t g_noalloc_roots[ROOT_WORDS];

struct NoAllocDev {
  bool ready = false;
  int lone_log = SMALL_LOG_MAX;  // as DeviceState::lone_log
  uint64_t* scratch = nullptr;  // device address of g_noalloc_scratch on this device
  Roots roots{};
};
static std::mutex g_na_mu;
static NoAllocDev g_na[64];
static uint64_t g_na_host_roots[ROOT_WORDS];  // staging, no heap use

// Forget every device's set-up (pimul_shutdown): the next no-alloc call on a
// device resolves the symbol addresses and copies the root tables again, as
// it must after a cudaDeviceReset.
void noalloc_forget() {
  std::lock_guard<std::mutex> lk(g_na_mu);
  for (NoAllocDev& d : g_na) d = NoAllocDev{};
}

static int noalloc_setup(NoAllocDev** out) {
  int dev = 0;
  CU(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(PIMUL_EINVAL, "device index out of range");
  std::lock_guard<std::mutex> lk(g_na_mu);
  NoAllocDev& d = g_na[dev];
  if (!d.ready) {
    build_roots(g_na_host_roots);
    uint64_t* scratch = nullptr;
    uint64_t* roots = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&scratch, g_noalloc_scratch);
    if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
    e = cudaGetSymbolAddress((void**)&roots, g_noalloc_roots);
    if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("cudaGetSymbolAddress(roots): ") + cudaGetErrorString(e));
    CU(cudaMemcpyToSymbol(g_noalloc_roots, g_na_host_roots, sizeof(g_na_host_roots)));
    CU(set_smem_attrs());
    d.lone_log = lone_log_here();
    d.scratch = scratch;
    d.roots = roots_at(roots);
    d.ready = true;
  }
  *out = &d;
  return PIMUL_OK;
}

static int mul_device_noalloc(const uint64_t* d_a, uint64_t la, const uint64_t* d_b, uint64_t lb, uint64_t* d_out,
                              cudaStream_t st) {
  NoAllocDev* nd = nullptr;
  int rc = noalloc_setup(&nd);
  if (rc) return rc;
  const Sizes z = sizes_for(la, lb);
  const Roots& R = nd->roots;
  if (z.L <= nd->lone_log) {  // whole product in shared memory: no scratch
    SmallJob job{d_a, d_b, d_out, (uint32_t)la, (uint32_t)lb};
    if (z.L < CLUSTER_LOG_MIN) launch_small(job, R, st);
    else launch_cluster(z.L, job, R, st);
    CU(cudaGetLastError());
    return PIMUL_OK;
  }
  const bool square = d_a == d_b && la == lb;
  Job J{};
  J.a = d_a, J.la = la, J.b = d_b, J.lb = lb, J.out = d_out;
  J.A = nd->scratch;
  J.W = nd->scratch + NOALLOC_N_MAX;
  J.B = square ? nullptr : J.W;
  carve_carry(J, nd->scratch + 2 * NOALLOC_N_MAX, z.nwin);
  Launcher X{st, false, R};  // no statistics hook: its event timing would create CUDA events
  X.tables = false;          // nor the twiddle tables, which are allocated on first use
  run_large(X, nullptr, J, 1, z.L, 1, z.nchunk);
  CU(cudaGetLastError());
  return PIMUL_OK;
}
}  // namespace pimul

extern "C" int pimul_mul_device_noalloc(const uint64_t* d_a, size_t la, const uint64_t* d_b, size_t lb,
                                        uint64_t* d_out, void* stream) {
  if (la == 0 || lb == 0) return PIMUL_OK;
  if (!d_a || !d_b || !d_out) return fail(PIMUL_EINVAL, "null device pointer");
  // each operand is checked before the sum is formed, so that no size_t
  // wrap-around can let an oversized pair through
  if (la > NOALLOC_N_MAX / 4 || lb > NOALLOC_N_MAX / 4 - la)
    return fail(PIMUL_EINVAL, "product too large for the no-alloc scratch: la + lb must be <= 262144 limbs "
                              "(transform length <= 2^20)");
  return mul_device_noalloc(d_a, la, d_b, lb, d_out, (cudaStream_t)stream);
}

// ---------------------------------------- merged splitting levels (internal)
namespace pimerge {

int prepare() { return pimul::ensure_init(-1); }

int merge_level(const Level& lv, int* d_bad, cudaStream_t stream) {
  using namespace pimul;
  if (lv.L < MIN_LOG || lv.L > MAX_LOG || !d_bad || lv.op < lv.sp || lv.oq < lv.sq || lv.ot < lv.st)
    return PIMUL_EINVAL;
  if (lv.n_in < 2) return PIMUL_OK;
  int rc = ensure_init(-1);
  if (rc) return rc;
  const MergeLevel M{lv.in, lv.in_len, lv.out, lv.out_len, lv.sp, lv.sq, lv.st, lv.op, lv.oq, lv.ot,
                     lv.n_in, lv.L, d_bad};
  const uint32_t gpc = MERGE_THREADS / merge_group_threads(lv.L);
  const uint32_t items = lv.n_in / 2 + (lv.n_in & 1);
  const uint32_t nchunks = (items + gpc - 1) / gpc;
  int sms = 152;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g_dev.device);
  const uint32_t grid = std::min<uint32_t>(nchunks, (uint32_t)sms * 2);
  const size_t smem = merge_cta_smem(lv.L);
  switch (lv.L) {
    case 8: k_split_merge<8><<<grid, MERGE_THREADS, smem, stream>>>(M, g_dev.roots); break;
    case 9: k_split_merge<9><<<grid, MERGE_THREADS, smem, stream>>>(M, g_dev.roots); break;
    case 10: k_split_merge<10><<<grid, MERGE_THREADS, smem, stream>>>(M, g_dev.roots); break;
    case 11: k_split_merge<11><<<grid, MERGE_THREADS, smem, stream>>>(M, g_dev.roots); break;
    default: k_split_merge<12><<<grid, MERGE_THREADS, smem, stream>>>(M, g_dev.roots); break;
  }
  g_launch[K_SMALL].fetch_add(1, std::memory_order_relaxed);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(PIMUL_ECUDA, std::string("merged splitting level: ") + cudaGetErrorString(e));
  return PIMUL_OK;
}

}  // namespace pimerge
