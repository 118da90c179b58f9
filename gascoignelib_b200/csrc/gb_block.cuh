// Block-system kernels (ncomp = B > 1 components per node, Stokes-type
// systems), the pressure filter, the Vanka smoother and the block ILU.
// Included by gb_context.cuh after gb_kernels.cuh.
#pragma once
#include "gb_ilu_plan.cuh"
#include "gb_kernels.cuh"
#include <type_traits>

namespace gb {

// Block SpMV over SELL-32 block rows: one thread per node; block entry j of
// lane l holds its B*B values component-major inside the slice, value q at
// val[(sptr[s] + 32 j) * B*B + 32 q + l] (coalesced per q). Per block the row
// sums are formed first and then added (FMatrixBlock::cadd,
// LinAlg/fmatrixblock.h:110-122; SparseBlockMatrix::vmult,
// LinAlg/sparseblockmatrix.xx:378-392). Modes as k_spmv; kJacobi applies the
// node's inverse diagonal block (FMatrixBlock::vmult order).
template<int MODE, int B, class TV, class TX, class TO, bool PAT>
__global__ void __launch_bounds__(kSpmvThreads)
k_bspmv(SellView<TV> A, const TX* __restrict__ x, TO* __restrict__ y,
        const TO* __restrict__ b, const TV* __restrict__ dinv,
        const uint8_t* __restrict__ dirmask, double alpha_,
        const int* __restrict__ yidx, int64_t ystride, TX* __restrict__ xcopy)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TV, TO>::type;
  constexpr int B2 = B * B;
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.n)
    return;
  const int row = A.perm ? __ldg(A.perm + slot) : slot;
  const int s = slot >> 5, lane = slot & 31;
  const int beg = A.sptr[s];
  const int w = (A.sptr[s + 1] - beg) >> 5;
  const TV* vp = A.val + int64_t(beg) * B2 + lane;
  const int* cp = PAT ? (A.ptab + int(A.pid[row]) * A.W) : (A.col + beg + lane);
  constexpr bool NEG = (MODE == kResid || MODE == kResidDir || MODE == kJacobi);
  TA acc[B];
#pragma unroll
  for (int r = 0; r < B; ++r)
    acc[r] = NEG ? static_cast<TA>(b[int64_t(row) * B + r]) : TA(0);
#pragma unroll 4
  for (int j = 0; j < w; ++j) {
    const int c = PAT ? row + ldg(cp + j) : ldg(cp + j * kSlice);
    TA xv[B], m[B2];
#pragma unroll
    for (int k = 0; k < B; ++k)
      xv[k] = static_cast<TA>(ldg(x + int64_t(c) * B + k));
#pragma unroll
    for (int q = 0; q < B2; ++q)
      m[q] = static_cast<TA>(ldg(vp + int64_t(j) * kSlice * B2 + q * kSlice));
#pragma unroll
    for (int r = 0; r < B; ++r) {
      TA sum = TA(0);
#pragma unroll
      for (int k = 0; k < B; ++k)
        sum = fma(m[r * B + k], xv[k], sum);
      acc[r] = NEG ? acc[r] - sum : acc[r] + sum;
    }
  }
  const TA alpha = static_cast<TA>(alpha_);
  const int64_t o = int64_t(row) * B;
  if (yidx) { // device-indexed output, as k_spmv
    const int64_t jj = *yidx;
#pragma unroll
    for (int r = 0; r < B; ++r)
      xcopy[jj * ystride + o + r] = x[o + r];
    y += (jj + 1) * ystride;
  }
  if (MODE == kJacobi) {
#pragma unroll
    for (int r = 0; r < B; ++r) {
      TA h = TA(0);
#pragma unroll
      for (int k = 0; k < B; ++k)
        h = fma(static_cast<TA>(dinv[o * B + r * B + k]), acc[k], h);
      y[o + r] = static_cast<TO>(static_cast<TA>(x[o + r]) + alpha * h);
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < B; ++r) {
    if (MODE == kAx)
      y[o + r] = static_cast<TO>(alpha * acc[r]);
    else if (MODE == kAddAx)
      y[o + r] = static_cast<TO>(static_cast<TA>(y[o + r]) + alpha * acc[r]);
    else if (MODE == kResid)
      y[o + r] = static_cast<TO>(acc[r]);
    else
      y[o + r] = dirmask[o + r] ? TO(0) : static_cast<TO>(acc[r]);
  }
}

// Component r of a block row: its part of every block's product, in the order
// of k_bspmv (a row's sums over the block, then added), so the same bits.
template<int B, bool NEG, bool PAT, class TV, class TX, class TA>
__device__ __forceinline__ TA
bspmv_component(const SellView<TV>& A, const TX* __restrict__ x, int s, int lane, int row, int r,
                TA acc)
{
  constexpr int B2 = B * B;
  const int beg = A.sptr[s];
  const int w = (A.sptr[s + 1] - beg) >> 5;
  const TV* vp = A.val + int64_t(beg) * B2 + r * B * kSlice + lane;
  const int* cp = PAT ? (A.ptab + int(A.pid[row]) * A.W) : (A.col + beg + lane);
  constexpr int U = 4; // blocks in flight
  for (int j0 = 0; j0 < w; j0 += U) {
    TA xv[U][B], m[U][B];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int j = j0 + q;
      const int c = j >= w ? row : PAT ? row + ldg(cp + j) : ldg(cp + j * kSlice);
#pragma unroll
      for (int k = 0; k < B; ++k) {
        xv[q][k] = j < w ? static_cast<TA>(ldg(x + int64_t(c) * B + k)) : TA(0);
        m[q][k] = j < w ? static_cast<TA>(ldg(vp + (int64_t(j) * B2 + k) * kSlice)) : TA(0);
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      TA sum = TA(0);
#pragma unroll
      for (int k = 0; k < B; ++k)
        sum = fma(m[q][k], xv[q][k], sum);
      acc = NEG ? acc - sum : acc + sum; // past the end: a sum of 0
    }
  }
  return acc;
}

// k_bspmv with a thread per row and component (warp = slice and component): a
// thread has B of a block's B^2 values to load, and there are B times as many
// threads. For small levels (block_split), whose one thread per row leaves most
// of the GPU idle and is a chain of 27 x B^2 loads. Measured with events around
// the launch: residual of 17^3 rows, B = 4, FP64 30 -> 15 us; of the seven levels
// below 513^2 rows, B = 3, FP32 about 14 -> 11.8 us each. On the 513^2 level
// itself the x loads, B times as many, cost more than they gain (the solve 13.9 ->
// 14.3 ms).
// The lines of block_split: products with a thread per row and with this, us in
// FP64 and in FP32.
//   9 blocks a row,  B = 2: 40,401 rows 10.1 10.3, 9.5 8.8; 57,600 10.5 11.3, 8.7 9.3
//                    B = 3: 75,625 14.3 14.0, 12.1 11.9; 96,100 14.5 15.7, 12.2 12.2
//                    B = 4: 25,600 16.0 15.5, 14.6 12.2; 40,401 16.3 18.2, 13.0 12.5
//   27 blocks a row, B = 2: 68,921 14.7 14.8, 12.9 12.0; 97,336 16.5 22.3, 12.9 14.0
//                    B = 3: 97,336 57.7 37.8, 41.4 20.9
//                    B = 4: 97,336 78.4 68.6, 65.5 41.9; 117,649 was not split
inline bool
block_split(int64_t rows, int blocks_per_row, int B)
{
  if (blocks_per_row > 16)
    return rows <= (B == 2 ? 70000 : 100000);
  return rows <= (B == 2 ? 48000 : B == 3 ? 80000 : 32768);
}
template<int MODE, int B, class TV, class TX, class TO, bool PAT>
__global__ void __launch_bounds__(kSpmvThreads, 2)
k_bspmv_split(SellView<TV> A, const TX* __restrict__ x, TO* __restrict__ y,
              const TO* __restrict__ b, const uint8_t* __restrict__ dirmask, double alpha_,
              const int* __restrict__ yidx, int64_t ystride, TX* __restrict__ xcopy)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TV, TO>::type;
  constexpr bool NEG = MODE == kResid || MODE == kResidDir;
  const int wid = (blockIdx.x * kSpmvThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int s = wid / B, r = wid % B, slot = s * kSlice + lane;
  if (slot >= A.n)
    return;
  const int row = A.perm ? __ldg(A.perm + slot) : slot;
  const int64_t o = int64_t(row) * B + r;
  const TA acc = bspmv_component<B, NEG, PAT, TV, TX, TA>(
    A, x, s, lane, row, r, NEG ? static_cast<TA>(b[o]) : TA(0));
  const TA alpha = static_cast<TA>(alpha_);
  if (yidx) {
    const int64_t jj = *yidx;
    xcopy[jj * ystride + o] = x[o];
    y += (jj + 1) * ystride;
  }
  if (MODE == kAx)
    y[o] = static_cast<TO>(alpha * acc);
  else if (MODE == kAddAx)
    y[o] = static_cast<TO>(static_cast<TA>(y[o]) + alpha * acc);
  else if (MODE == kResid)
    y[o] = static_cast<TO>(acc);
  else
    y[o] = dirmask[o] ? TO(0) : static_cast<TO>(acc);
}

// y = b - A x on block rows with the pressure filter's plain mean of
// component pc of y (StdSolver::MatrixResidual with SubtractMeanAlgebraic):
// the last block writes sum / denom to *mean; consumers subtract it on read.
template<int B, class TV, class T, bool PAT>
__global__ void __launch_bounds__(kSpmvThreads)
k_bspmv_resid_mean(SellView<TV> A, const T* __restrict__ x, T* __restrict__ y,
                   const T* __restrict__ b, int pc, double denom, double* partials,
                   unsigned* ticket, double* mean)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TV, T>::type;
  constexpr int B2 = B * B;
  __shared__ double sh[32];
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (slot < A.n) {
    const int row = A.perm ? __ldg(A.perm + slot) : slot;
    const int s = slot >> 5, lane = slot & 31;
    const int beg = A.sptr[s];
    const int w = (A.sptr[s + 1] - beg) >> 5;
    const TV* vp = A.val + int64_t(beg) * B2 + lane;
    const int* cp = PAT ? (A.ptab + int(A.pid[row]) * A.W) : (A.col + beg + lane);
    TA acc[B];
#pragma unroll
    for (int r = 0; r < B; ++r)
      acc[r] = static_cast<TA>(b[int64_t(row) * B + r]);
#pragma unroll 4
    for (int j = 0; j < w; ++j) {
      const int c = PAT ? row + ldg(cp + j) : ldg(cp + j * kSlice);
      TA xv[B], m[B2];
#pragma unroll
      for (int k = 0; k < B; ++k)
        xv[k] = static_cast<TA>(ldg(x + int64_t(c) * B + k));
#pragma unroll
      for (int q = 0; q < B2; ++q)
        m[q] = static_cast<TA>(ldg(vp + int64_t(j) * kSlice * B2 + q * kSlice));
#pragma unroll
      for (int r = 0; r < B; ++r) {
        TA sum = TA(0);
#pragma unroll
        for (int k = 0; k < B; ++k)
          sum = fma(m[r * B + k], xv[k], sum);
        acc[r] = acc[r] - sum;
      }
    }
#pragma unroll
    for (int r = 0; r < B; ++r) {
      const T o = static_cast<T>(acc[r]);
      y[int64_t(row) * B + r] = o;
      if (r == pc)
        v = static_cast<double>(o);
    }
  }
  v = block_sum(v, sh);
  red_finish(partials, ticket, v, RedOut{ mean, nullptr, nullptr, 0, denom }, sh);
}

// The same with a thread per row and component (k_bspmv_split's rule).
template<int B, class TV, class T, bool PAT>
__global__ void __launch_bounds__(kSpmvThreads, 2)
k_bspmv_resid_mean_split(SellView<TV> A, const T* __restrict__ x, T* __restrict__ y,
                         const T* __restrict__ b, int pc, double denom, double* partials,
                         unsigned* ticket, double* mean)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TV, T>::type;
  __shared__ double sh[32];
  const int wid = (blockIdx.x * kSpmvThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int s = wid / B, r = wid % B, slot = s * kSlice + lane;
  double v = 0.0;
  if (slot < A.n) {
    const int row = A.perm ? __ldg(A.perm + slot) : slot;
    const int64_t o = int64_t(row) * B + r;
    const T res = static_cast<T>(bspmv_component<B, true, PAT, TV, T, TA>(
      A, x, s, lane, row, r, static_cast<TA>(b[o])));
    y[o] = res;
    if (r == pc)
      v = static_cast<double>(res);
  }
  v = block_sum(v, sh);
  red_finish(partials, ticket, v, RedOut{ mean, nullptr, nullptr, 0, denom }, sh);
}

// Plain or weighted mean of component pc (no subtraction): *mean =
// (sum_j x(j, pc) [* w_j]) / denom.
template<class T>
__global__ void __launch_bounds__(kRedThreads)
k_comp_mean(int n, int B, int pc, const T* __restrict__ x, const double* __restrict__ w,
            double denom, double* partials, unsigned* ticket, double* mean)
{
  GB_PDL_ENTRY();
  __shared__ double sh[32];
  double v = 0.0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const double xv = static_cast<double>(x[int64_t(j) * B + pc]);
    v = w ? fma(xv, w[j], v) : v + xv;
  }
  v = block_sum(v, sh);
  red_finish(partials, ticket, v, RedOut{ mean, nullptr, nullptr, 0, denom }, sh);
}

// u = (u_zero ? 0 : u) + omega * (D^-1 h) per node: SparseBlockMatrix::Jacobi
// (LinAlg/sparseblockmatrix.xx:47-56) followed by Add(x, omega, h).
// Pressure filter around it (pc >= 0): h's component pc is read minus *hmean
// (its algebraic mean, when hmean is set), and the weighted mean of the new
// u's component pc is reduced into *umean (sum of u(j, pc) w_j / domain) when
// w is set.
struct PfArgs
{
  int pc;              // filtered component, -1: none
  const double* hmean; // subtract from h(., pc) on read, or null
  const double* w;     // weights for the mean of the result, or null
  double domain;
  double* partials;
  unsigned* ticket;
  double* umean;
};

template<int B, class TV, class T>
__global__ void __launch_bounds__(256)
k_block_jacobi_apply(int n, const TV* __restrict__ dinv, const T* __restrict__ h,
                     T* __restrict__ u, double omega, int u_zero, PfArgs pf)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TV, T>::type;
  __shared__ double sh[32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double wv = 0.0;
  if (i < n) {
    const int64_t o = int64_t(i) * B;
    const double hm = pf.hmean ? *pf.hmean : 0.0;
    TA t[B];
#pragma unroll
    for (int k = 0; k < B; ++k)
      t[k] = (pf.hmean && k == pf.pc)
               ? static_cast<TA>(static_cast<double>(h[o + k]) - hm)
               : static_cast<TA>(h[o + k]);
#pragma unroll
    for (int r = 0; r < B; ++r) {
      TA v = TA(0);
#pragma unroll
      for (int k = 0; k < B; ++k)
        v = fma(static_cast<TA>(dinv[o * B + r * B + k]), t[k], v);
      const TA base = u_zero ? TA(0) : static_cast<TA>(u[o + r]);
      const T un = static_cast<T>(base + static_cast<TA>(omega) * v);
      u[o + r] = un;
      if (pf.w && r == pf.pc)
        wv = static_cast<double>(un) * pf.w[i];
    }
  }
  if (pf.w) {
    wv = block_sum(wv, sh);
    red_finish(pf.partials, pf.ticket, wv, RedOut{ pf.umean, nullptr, nullptr, 0, pf.domain },
               sh);
  }
}

// Block transfers: the scalar tables applied to each of the B components. A thread
// takes C components of a node: one (the B threads of a node read B consecutive
// values, eight entries in flight), or all B. The sum runs over the entries in order
// from acc (0, or the target for an in-place add: the weights are powers of two, so
// each fused add rounds like the reference's y += w x), so both give the same bits.
// Component pc is read minus smean.
// One component per thread hides the entries' latency on small levels, and reads
// every entry B times: up to kDofThreadRows nodes. Thread per node and per component,
// us with events around the launch, B = 3 in 2D, FP64:
//   prolongation to   66,049 nodes 10.3 8.6; 263,169 10.6 17.8; 1,050,625 20.8 46.3
//   restriction to    66,049 nodes 14.7 12.6; 263,169 16.7 26.4
//   the Vanka averages of a cycle on two levels (4 on the finer, 1 on the coarser),
//                     66,049 nodes 62 61; 263,169 88 104; 1,050,625 194 294
// B = 4 in 3D: prolongation to 117,649 nodes 12.7 14.1, averages 82 86.
constexpr int64_t kDofThreadRows = 70000;

template<class T, int B, int C>
__device__ __forceinline__ void
transfer_row_b(const int* __restrict__ tsp, const uint32_t* __restrict__ tent,
               const T* __restrict__ src, int i, int c0, T (&acc)[C], int pc = -1,
               double smean = 0.0)
{
  const int beg = __ldg(tsp + (i >> 5));
  const int w = (__ldg(tsp + (i >> 5) + 1) - beg) >> 5;
  const uint32_t* ep = tent + beg + (i & 31);
  if constexpr (C > 1) {
    for (int j = 0; j < w; ++j) {
      const uint32_t e = __ldg(ep + j * kSlice);
      const T wgt = wcode<T>(e);
      const T* sp = src + int64_t(e & kIdxMask) * B;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const T sv = c == pc ? static_cast<T>(static_cast<double>(__ldg(sp + c)) - smean)
                             : __ldg(sp + c);
        acc[c] = fma(wgt, sv, acc[c]);
      }
    }
  } else {
    for (int j0 = 0; j0 < w; j0 += 8) {
      const uint32_t* pe[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        pe[q] = ep + min(j0 + q, w - 1) * kSlice;
      uint32_t e[8];
      ld8(e, pe);
      const T* ps[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        ps[q] = src + int64_t(e[q] & kIdxMask) * B + c0;
      T f[8];
      ld8(f, ps);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (j0 + q < w) {
          const T sv = c0 == pc ? static_cast<T>(static_cast<double>(f[q]) - smean) : f[q];
          acc[0] = fma(wcode<T>(e[q]), sv, acc[0]);
        }
    }
  }
}

// fine's component pc is read minus *smean when smean is set (the filtered
// residual of MatrixResidual, restricted).
template<class T, int B, int C>
__global__ void __launch_bounds__(256)
k_restrict_b(int nc, const int* __restrict__ tsp, const uint32_t* __restrict__ tent,
             const T* __restrict__ fine, T* __restrict__ coarse,
             const uint8_t* __restrict__ cdir, int pc, const double* __restrict__ smean)
{
  GB_PDL_ENTRY();
  constexpr int S = B / C; // threads of a node
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int i = static_cast<int>(t / S), c0 = static_cast<int>(t % S);
  if (i >= nc)
    return;
  T acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c)
    acc[c] = T(0);
  transfer_row_b<T, B, C>(tsp, tent, fine, i, c0, acc, smean ? pc : -1, smean ? *smean : 0.0);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int64_t d = int64_t(i) * B + c0 + c;
    coarse[d] = (cdir && cdir[d]) ? T(0) : acc[c];
  }
}

template<int MODE, class T, int B, int C>
__global__ void __launch_bounds__(256)
k_prolong_b(int nf, const int* __restrict__ tsp, const uint32_t* __restrict__ tent,
            const T* __restrict__ coarse, T* __restrict__ fine,
            const uint8_t* __restrict__ fdir, double mgomega)
{
  GB_PDL_ENTRY();
  constexpr int S = B / C;
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int i = static_cast<int>(t / S), c0 = static_cast<int>(t % S);
  if (i >= nf)
    return;
  const int64_t d0 = int64_t(i) * B + c0;
  T acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c)
    acc[c] = MODE == 0 ? fine[d0 + c] : T(0);
  transfer_row_b<T, B, C>(tsp, tent, coarse, i, c0, acc);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int64_t d = d0 + c;
    if (MODE == 0) {
      fine[d] = acc[c];
    } else {
      const T a = (fdir && fdir[d]) ? T(0) : acc[c];
      fine[d] = fine[d] + static_cast<T>(mgomega) * a;
    }
  }
}

// ------------------------------------------------------ pressure filter
//
// PressureFilter::IntegrateVector / SubtractMeanAlgebraic's sum
// (Discretization/Q1/pressurefilter.cc:56-100): sum over nodes of
// x(j, c) * w_j (w null: plain sum), deterministic FP64 reduction.
template<class T>
__global__ void __launch_bounds__(kRedThreads)
k_comp_sum(int n, int B, int c, const T* __restrict__ x, const double* __restrict__ w,
           double* partials, unsigned* ticket, RedOut ro)
{
  GB_PDL_ENTRY();
  __shared__ double sh[32];
  double v = 0.0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const double xv = static_cast<double>(x[int64_t(j) * B + c]);
    v = w ? fma(xv, w[j], v) : v + xv;
  }
  v = block_sum(v, sh);
  red_finish(partials, ticket, v, ro, sh);
}

// x(., c) += -(sum / denom): CompAdd(comp, -mean / domainsize) or
// CompAdd(comp, -sum / (n - nhanging)).
template<class T>
__global__ void
k_comp_sub(int n, int B, int c, T* __restrict__ x, const double* __restrict__ sum,
           double denom)
{
  GB_PDL_ENTRY();
  const double sub = sum[0] / denom;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    x[int64_t(j) * B + c] = static_cast<T>(static_cast<double>(x[int64_t(j) * B + c]) - sub);
}

// ------------------------------------------------------------------ Vanka
//
// VankaSmoother::solve (LinAlg/vankasmoother.cc:192-237) in two kernels: the
// local solves (one per patch, writing the patch solutions), then a gather per
// node that sums the solutions of the patches containing it in ascending
// patch order (the reference's order on one thread), scales by 1/count and
// adds omega times it to u (StdSolver::smooth's Add).
//
// The local solves apply each patch's inverse (formed once per assembly from
// its LU factors): one warp per patch, lane i computing rows i, i+32, ..;
// the inverse is stored transposed per patch ([patch][j][i]) so that for each
// column j the warp's loads are contiguous; the patch's right-hand side
// (component pc read minus *hmean when set) is staged in shared memory.
constexpr int kVankaMaxM = 128;
constexpr int kVankaWarps = 4;

// Per assembly, the patches' local matrices and their inverses on the device
// (VankaSmoother::copy_entries_sparseblockmatrix, LinAlg/vankasmoother.cc:
// 65-113, then the LU solves of VankaSmoother::solve, :192-237, applied to the
// unit vectors). One CTA per patch, the M x M matrix in shared memory:
//  - gather: entry (B r + cr, B q + cc) from the level's FP64 SELL values at
//    map[p][r][q] + 32 (cr B + cc) (a host-built offset per node pair of the
//    patch, -1 where the matrix holds no block), zero elsewhere;
//  - LU with partial pivoting in the order of the partial-pivot LU the
//    reference calls (pivot = the first row of largest |a_ik|, rows swapped,
//    column scaled by the pivot when it is nonzero, rank-1 update of the
//    trailing block), each product and difference rounded separately;
//  - column j of the inverse (thread j): forward substitution with the unit
//    lower factor on P e_j, backward with the upper, the same operation order;
//    stored transposed ([patch][j][i]), FP64 and FP32.
// The result equals the host factorisation of the same arithmetic bit for bit.
constexpr int kVankaFactorThreads = 128;

static __global__ void __launch_bounds__(kVankaFactorThreads)
k_vanka_factor(int npatch, int npp, int B, int M, const int* __restrict__ map,
               const double* __restrict__ val, double* __restrict__ inv64,
               float* __restrict__ inv32)
{
  GB_PDL_ENTRY();
  extern __shared__ double sm_vf[];
  const int ld = M + 1;
  double* A = sm_vf;                                   // [M][M + 1]
  int* pv = reinterpret_cast<int*>(A + M * ld);        // [M]
  __shared__ int s_piv;
  const int p = blockIdx.x;
  if (p >= npatch)
    return; // whole CTA
  const int t = threadIdx.x, nt = blockDim.x;
  for (int e = t; e < M * M; e += nt) {
    const int i = e / M, jc = e - i * M;
    const int r = i / B, cr = i - r * B, q = jc / B, cc = jc - q * B;
    const int base = __ldg(map + (int64_t(p) * npp + r) * npp + q);
    A[i * ld + jc] = base < 0 ? 0.0 : __ldg(val + int64_t(base) + int64_t(kSlice) * (cr * B + cc));
  }
  for (int i = t; i < M; i += nt)
    pv[i] = i;
  __syncthreads();
  for (int k = 0; k < M; ++k) {
    if (t == 0) {
      int piv = k;
      double best = fabs(A[k * ld + k]);
      for (int i = k + 1; i < M; ++i) {
        const double v = fabs(A[i * ld + k]);
        if (v > best) {
          best = v;
          piv = i;
        }
      }
      s_piv = piv;
      if (piv != k) {
        const int tmp = pv[k];
        pv[k] = pv[piv];
        pv[piv] = tmp;
      }
    }
    __syncthreads();
    const int piv = s_piv;
    if (piv != k)
      for (int j = t; j < M; j += nt) {
        const double tmp = A[k * ld + j];
        A[k * ld + j] = A[piv * ld + j];
        A[piv * ld + j] = tmp;
      }
    __syncthreads();
    const double akk = A[k * ld + k];
    if (akk != 0.0)
      for (int i = k + 1 + t; i < M; i += nt)
        A[i * ld + k] = __ddiv_rn(A[i * ld + k], akk);
    __syncthreads();
    const int rem = M - k - 1;
    for (int e = t; e < rem * rem; e += nt) {
      const int i = k + 1 + e / rem, j = k + 1 + e % rem;
      A[i * ld + j] = __dsub_rn(A[i * ld + j], __dmul_rn(A[i * ld + k], A[k * ld + j]));
    }
    __syncthreads();
  }
  for (int j = t; j < M; j += nt) {
    double* x = inv64 + (int64_t(p) * M + j) * M; // the column, built in place
    for (int i = 0; i < M; ++i)
      x[i] = pv[i] == j ? 1.0 : 0.0;
    for (int i = 1; i < M; ++i) {
      double sacc = x[i];
      for (int q = 0; q < i; ++q)
        sacc = __dsub_rn(sacc, __dmul_rn(A[i * ld + q], x[q]));
      x[i] = sacc;
    }
    for (int i = M - 1; i >= 0; --i) {
      double sacc = x[i];
      for (int q = i + 1; q < M; ++q)
        sacc = __dsub_rn(sacc, __dmul_rn(A[i * ld + q], x[q]));
      x[i] = __ddiv_rn(sacc, A[i * ld + i]);
    }
    float* y = inv32 + (int64_t(p) * M + j) * M;
    for (int i = 0; i < M; ++i)
      y[i] = static_cast<float>(x[i]);
  }
}

// Patches of more than 32 unknowns (3D: 108): one CTA of kVankaWide warps per
// patch, warp q taking the columns j = q, q + kVankaWide, ..; a row's partial
// sums are added in the warps' order. With a warp per patch the 512 patches of
// a 17^3 Stokes level were 3.5 warps per SM with 12 loads each in flight: 27 us
// against 7.4 us for their 48 MB at the copy rate; 10.7 us in this form.
constexpr int kVankaWide = 8;

// Taken up to so many patches; with more of them a warp per patch fills the SMs and
// the two block barriers of a patch are what is left to see. Warp and CTA, us with
// events around the launch, patches of 27 nodes:
//   54 unknowns, FP64: 1,000 10.7 10.6; 1,728 10.8 12.9; 13,824 62 111
//                FP32: 1,000 10.6 8.6; 1,728 10.6 10.7; 13,824 37 62
//   81 unknowns, FP64: 1,728 33.7 24.9; 2,744 41.4 45.7; 13,824 122 171
//                FP32: 1,728 13.8 12.8; 2,744 18.8 17.0; 4,096 27.8 33.3
//  108 unknowns, FP64: 4,096 81.7 74.3; 5,832 99.6 100.9; 13,824 214 222
//                FP32: 2,744 37.2 36.5; 4,096 44.7 47.4; 13,824 120 134
template<class T>
constexpr int
vanka_wide_patches(int R)
{
  return R == 2 ? 1000 : R == 3 ? 2000 : sizeof(T) == 8 ? 5000 : 3000;
}
template<int R, class TL, class T>
__global__ void __launch_bounds__(32 * kVankaWide)
k_vanka_inv_wide(int npatch, int M, int B, const int* __restrict__ pn,
                 const TL* __restrict__ inv, const T* __restrict__ h, int pc,
                 const double* __restrict__ hmean, T* __restrict__ hout)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TL, T>::type;
  __shared__ TA H[kVankaMaxM];
  __shared__ TA part[kVankaWide][R * 32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x;
  const int64_t np = npatch;
  const double hm = hmean ? *hmean : 0.0;
  for (int i = threadIdx.x; i < M; i += 32 * kVankaWide) {
    const int r = i / B, c = i - r * B;
    const int node = __ldg(pn + r * np + p);
    const T hv = __ldg(h + int64_t(node) * B + c);
    H[i] = (hmean && c == pc) ? static_cast<TA>(static_cast<double>(hv) - hm)
                              : static_cast<TA>(hv);
  }
  __syncthreads();
  const TL* ip = inv + int64_t(p) * M * M + lane;
  TA acc[R];
#pragma unroll
  for (int k = 0; k < R; ++k)
    acc[k] = TA(0);
#pragma unroll 7
  for (int j = wid; j < M; j += kVankaWide) {
    const TA hj = H[j];
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (lane + 32 * k < M)
        acc[k] = fma(static_cast<TA>(__ldg(ip + j * M + 32 * k)), hj, acc[k]);
  }
#pragma unroll
  for (int k = 0; k < R; ++k)
    part[wid][k * 32 + lane] = acc[k];
  __syncthreads();
  for (int i = threadIdx.x; i < M; i += 32 * kVankaWide) {
    TA v = part[0][i];
#pragma unroll
    for (int q = 1; q < kVankaWide; ++q)
      v += part[q][i];
    hout[int64_t(p) * M + i] = static_cast<T>(v);
  }
}

template<int R, class TL, class T>
__global__ void __launch_bounds__(32 * kVankaWarps)
k_vanka_inv(int npatch, int M, int B, const int* __restrict__ pn,
            const TL* __restrict__ inv, const T* __restrict__ h, int pc,
            const double* __restrict__ hmean, T* __restrict__ hout)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<TL, T>::type;
  __shared__ TA sH[kVankaWarps][kVankaMaxM];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x * kVankaWarps + wid;
  if (p >= npatch)
    return; // whole warp
  const int64_t np = npatch;
  TA* H = sH[wid];
  const double hm = hmean ? *hmean : 0.0;
  for (int i = lane; i < M; i += 32) {
    const int r = i / B, c = i - r * B;
    const int node = __ldg(pn + r * np + p);
    const T hv = __ldg(h + int64_t(node) * B + c);
    H[i] = (hmean && c == pc) ? static_cast<TA>(static_cast<double>(hv) - hm)
                              : static_cast<TA>(hv);
  }
  __syncwarp();
  const TL* ip = inv + int64_t(p) * M * M + lane;
  TA acc[R];
#pragma unroll
  for (int k = 0; k < R; ++k)
    acc[k] = TA(0);
#pragma unroll 3
  for (int j = 0; j < M; ++j) {
    const TA hj = H[j];
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (lane + 32 * k < M)
        acc[k] = fma(static_cast<TA>(__ldg(ip + j * M + 32 * k)), hj, acc[k]);
  }
#pragma unroll
  for (int k = 0; k < R; ++k)
    if (lane + 32 * k < M)
      hout[int64_t(p) * M + lane + 32 * k] = static_cast<T>(acc[k]);
}

// The same for a patch size known at compile time (M <= 32: one row per lane):
// every load of the warp's 27 (or 9) inverse columns is issued up front.
template<int M, class TL, class T>
__global__ void __launch_bounds__(32 * kVankaWarps)
k_vanka_inv_ct(int npatch, int B, const int* __restrict__ pn, const TL* __restrict__ inv,
               const T* __restrict__ h, int pc, const double* __restrict__ hmean,
               T* __restrict__ hout)
{
  GB_PDL_ENTRY();
  static_assert(M <= 32, "one row per lane");
  using TA = typename Acc<TL, T>::type;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x * kVankaWarps + wid;
  if (p >= npatch)
    return; // whole warp
  const int64_t np = npatch;
  const bool act = lane < M;
  // this lane's row of the inverse (column j at ip[j * M]) and its residual entry
  const TL* ip = inv + int64_t(p) * M * M + (act ? lane : 0);
  TL a[M];
#pragma unroll
  for (int j = 0; j < M; ++j)
    a[j] = __ldg(ip + j * M);
  TA hv = TA(0);
  if (act) {
    const int r = lane / B, c = lane - r * B;
    const int node = __ldg(pn + r * np + p);
    const T x = __ldg(h + int64_t(node) * B + c);
    hv = (hmean && c == pc) ? static_cast<TA>(static_cast<double>(x) - *hmean)
                            : static_cast<TA>(x);
  }
  TA acc = TA(0);
#pragma unroll
  for (int j = 0; j < M; ++j)
    acc = fma(static_cast<TA>(a[j]), __shfl_sync(0xffffffffu, hv, j), acc);
  if (act)
    hout[int64_t(p) * M + lane] = static_cast<T>(acc);
}

// u(i, c) = (u_zero ? 0 : u(i, c)) + omega * ((sum over the node's patches of
// their solution at (i, c)) * (1 / count)), C components of a node per thread
// (kDofThreadRows, the block transfers' rule; the same bits). ent packs (patch,
// local node): patch * 32 + r (npp <= 27). Solution (patch p, local dof q) at
// hout[p * M + q].
template<int B, int C, class T>
__global__ void __launch_bounds__(256)
k_vanka_gather(int n, const int* __restrict__ nptr, const int* __restrict__ ent,
               const T* __restrict__ hout, int M, T* __restrict__ u, double omega,
               int u_zero, PfArgs pf)
{
  GB_PDL_ENTRY();
  using TA = typename Acc<T, T>::type;
  constexpr int S = B / C;         // threads of a node
  constexpr int F = C == 1 ? 4 : 1; // patches' values in flight
  __shared__ double sh[32];
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int i = static_cast<int>(t / S), c0 = static_cast<int>(t % S);
  double wv = 0.0;
  if (i < n) {
    const int k0 = __ldg(nptr + i), k1 = __ldg(nptr + i + 1);
    TA acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c)
      acc[c] = TA(0);
    for (int k = k0; k < k1; k += F) {
      int e[F];
#pragma unroll
      for (int q = 0; q < F; ++q)
        e[q] = k + q < k1 ? __ldg(ent + k + q) : -1;
      TA v[F][C];
#pragma unroll
      for (int q = 0; q < F; ++q)
#pragma unroll
        for (int c = 0; c < C; ++c)
          v[q][c] =
            e[q] >= 0
              ? static_cast<TA>(hout[int64_t(e[q] >> 5) * M + (e[q] & 31) * B + c0 + c])
              : TA(0);
#pragma unroll
      for (int q = 0; q < F; ++q)
        if (e[q] >= 0)
#pragma unroll
          for (int c = 0; c < C; ++c)
            acc[c] += v[q][c];
    }
    const TA sc = TA(1) / static_cast<TA>(k1 - k0);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int64_t d = int64_t(i) * B + c0 + c;
      const TA base = u_zero ? TA(0) : static_cast<TA>(u[d]);
      const T un = static_cast<T>(base + static_cast<TA>(omega) * (acc[c] * sc));
      u[d] = un;
      if (pf.w && c0 + c == pf.pc)
        wv = static_cast<double>(un) * pf.w[i];
    }
  }
  if (pf.w) {
    wv = block_sum(wv, sh);
    red_finish(pf.partials, pf.ticket, wv, RedOut{ pf.umean, nullptr, nullptr, 0, pf.domain },
               sh);
  }
}

} // namespace gb

namespace gb {

// ------------------------------------------------------------ hanging nodes
//
// HNStructureQ12d/Q13d/Q22d/Q23d (Discretization/Q1/hnstructureq12d.cc,
// hnstructureq13d.cc, Discretization/Q2/hnstructureq22d.cc,
// hnstructureq23d.cc) act in phases (edges, faces, in the discretisation's
// order); within a phase no hanging node is a parent of another. Products and
// sums are rounded separately (no fused multiply-add) and associated as
// CompVector::equ_node/add_node write them, so the FP64 results are the
// reference's bit for bit.
__device__ __forceinline__ double hn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double hn_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float hn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float hn_add(float a, float b) { return __fadd_rn(a, b); }

// u(h) = sum over groups (left to right inside a group, groups added in
// turn); parents slot-major: par[s * nh + k], weights w[s].
template<class T>
__global__ void
k_hn_average(int nh, int B, const int* __restrict__ node, const int* __restrict__ par,
             int nslots, int gsize, const double* __restrict__ w, T* __restrict__ u)
{
  GB_PDL_ENTRY();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nh)
    return;
  for (int c = 0; c < B; ++c) {
    T acc = T(0);
    for (int g = 0; g < nslots; g += gsize) {
      T sg = hn_mul(static_cast<T>(w[g]), u[int64_t(par[g * nh + k]) * B + c]);
      for (int s = g + 1; s < g + gsize; ++s)
        sg = hn_add(sg, hn_mul(static_cast<T>(w[s]), u[int64_t(par[s * nh + k]) * B + c]));
      acc = g == 0 ? sg : hn_add(acc, sg);
    }
    u[int64_t(node[k]) * B + c] = acc;
  }
}

// parents += w * u(h) in ascending hanging-node order (one thread per parent:
// its contributions in the reference's sequence)
template<class T>
__global__ void
k_hn_distribute(int np, int B, const int* __restrict__ pnode, const int* __restrict__ ptr,
                const int* __restrict__ hnode, const double* __restrict__ wt,
                T* __restrict__ u)
{
  GB_PDL_ENTRY();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= np)
    return;
  const int64_t p = pnode[k];
  for (int c = 0; c < B; ++c) {
    T acc = u[p * B + c];
    for (int e = ptr[k]; e < ptr[k + 1]; ++e)
      acc = hn_add(acc, hn_mul(static_cast<T>(wt[e]), u[int64_t(hnode[e]) * B + c]));
    u[p * B + c] = acc;
  }
}

template<class T>
__global__ void
k_hn_zero(int nh, int B, const int* __restrict__ node, T* __restrict__ u)
{
  GB_PDL_ENTRY();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nh)
    return;
  for (int c = 0; c < B; ++c)
    u[int64_t(node[k]) * B + c] = T(0);
}

// --------------------------------------------------------- block ILU

template<class T>
__device__ __forceinline__ T ilu_mul(T a, T b);
template<>
__device__ __forceinline__ double ilu_mul(double a, double b) { return __dmul_rn(a, b); }
template<>
__device__ __forceinline__ float ilu_mul(float a, float b) { return __fmul_rn(a, b); }
template<class T>
__device__ __forceinline__ T ilu_sub(T a, T b);
template<>
__device__ __forceinline__ double ilu_sub(double a, double b) { return __dsub_rn(a, b); }
template<>
__device__ __forceinline__ float ilu_sub(float a, float b) { return __fsub_rn(a, b); }
template<class T>
__device__ __forceinline__ T ilu_add(T a, T b);
template<>
__device__ __forceinline__ double ilu_add(double a, double b) { return __dadd_rn(a, b); }
template<>
__device__ __forceinline__ float ilu_add(float a, float b) { return __fadd_rn(a, b); }

// SparseBlockIlu::compute_ilu (LinAlg/sparseblockilu.xx:246-275) on the
// device, one dependency level per launch, one thread per row: a row waits
// only for the rows of its lower part (earlier levels), exactly as in the
// forward substitution. Each row runs the host factorisation's steps in its
// order: for every lower entry k ascending, a(i,k) times the inverted
// diagonal block of row k, then a(i,j) -= a(i,k) a(k,j) over row k's upper
// entries (the target found by a search of row i), and finally the
// Gauss-Jordan inverse of the diagonal block; products and sums rounded
// separately, as on the host: the factors are the host's bit for bit.
template<int B>
__global__ void __launch_bounds__(128)
k_ilu_factor(int nr, const int* __restrict__ rows, const int* __restrict__ ptr,
             const int* __restrict__ col, const int* __restrict__ diag,
             double* __restrict__ v)
{
  GB_PDL_ENTRY();
  constexpr int B2 = B * B;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nr)
    return;
  const int i = rows[t];
  const int pb = ptr[i], pe = ptr[i + 1], pd = diag[i];
  double tmp[B2];
  for (int pk = pb; pk < pd; ++pk) {
    const int k = col[pk];
    double* a = v + int64_t(pk) * B2;
    const double* dk = v + int64_t(diag[k]) * B2;
#pragma unroll
    for (int q = 0; q < B2; ++q)
      tmp[q] = a[q];
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
      for (int cc = 0; cc < B; ++cc) {
        double acc = 0.0;
#pragma unroll
        for (int u = 0; u < B; ++u)
          acc = rn_add(acc, rn_mul(tmp[r * B + u], dk[u * B + cc]));
        a[r * B + cc] = acc;
      }
    const int ke = ptr[k + 1];
    for (int pj = diag[k] + 1; pj < ke; ++pj) {
      const int j = col[pj];
      for (int ph = pb; ph < pe; ++ph) {
        if (col[ph] != j)
          continue;
        double* h = v + int64_t(ph) * B2;
        const double* cj = v + int64_t(pj) * B2;
#pragma unroll
        for (int r = 0; r < B; ++r)
#pragma unroll
          for (int cc = 0; cc < B; ++cc)
#pragma unroll
            for (int u = 0; u < B; ++u)
              h[r * B + cc] = rn_sub(h[r * B + cc], rn_mul(a[r * B + u], cj[u * B + cc]));
        break;
      }
    }
  }
  gauss_jordan<B>(v + int64_t(pd) * B2);
}

// The ILU's values in its row-sorted layout from the level's SELL values:
// entry e, component q at val[map[e] + 32 q].
static __global__ void
k_ilu_gather(int64_t nnz, int B2, const int* __restrict__ map,
             const double* __restrict__ val, double* __restrict__ v)
{
  GB_PDL_ENTRY();
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < nnz;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = map[e];
    for (int q = 0; q < B2; ++q)
      v[e * B2 + q] = __ldg(val + base + int64_t(kSlice) * q);
  }
}

static __global__ void
k_to_float(int64_t n, const double* __restrict__ a, float* __restrict__ b)
{
  GB_PDL_ENTRY();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x)
    b[i] = static_cast<float>(a[i]);
}

// FP64 rows one entry at a time: groups of 4 FP64 entries measured slower
// (C2 ILU solve 240 against 168 ms with a launch per level), FP32 groups of 8
// faster (123.9 against 133.7 ms)
#ifndef GB_ILU_GROUP_F64
#define GB_ILU_GROUP_F64 1
#endif

// One row of a substitution. Forward, with the unit lower factor
// (SparseBlockIlu::forward, LinAlg/sparseblockilu.xx:202-214): y_i -= L_ik y_k
// over the row's lower blocks in stored (ascending column) order, block
// entries as FMatrixBlock::subtract (LinAlg/fmatrixblock.h:136-145).
// Backward (SparseBlockIlu::backward, LinAlg/sparseblockilu.xx:217-231):
// y_i -= U_ik y_k over the upper blocks in descending order, then
// y_i = D_i^-1 y_i with the inverted diagonal block (FMatrixBlock::vmult,
// LinAlg/fmatrixblock.h:194-217). The entries are taken G at a time: their
// columns, then their y blocks and values are loaded together before the
// subtractions run in the reference's order, so a row waits for about two
// memory round trips per G entries instead of one per entry. The rows of one
// dependency level depend only on rows of earlier levels, so running the
// levels in order gives the sequential sweep bit for bit. (Levels too large for
// k_ilu_cluster.)
template<int B, class T, bool UP>
__device__ __forceinline__ void
ilu_row(int i, const int* __restrict__ ptr, const int* __restrict__ col,
        const int* __restrict__ diag, const T* __restrict__ val, T* __restrict__ y)
{
  constexpr int B2 = B * B;
  // the G value blocks of a group take at most 32 registers; FP64 rows take
  // GB_ILU_GROUP_F64 entries at a time at most
  constexpr int G0 = 32 / (B2 * int(sizeof(T) / 4));
  constexpr int GM = sizeof(T) == 8 ? GB_ILU_GROUP_F64 : 8;
  constexpr int G = G0 < 1 ? 1 : (G0 > GM ? GM : G0);
  T yi[B];
#pragma unroll
  for (int r = 0; r < B; ++r)
    yi[r] = y[int64_t(i) * B + r];
  const int d = __ldg(diag + i);
  const int first = UP ? __ldg(ptr + i + 1) - 1 : __ldg(ptr + i);
  const int cnt = UP ? first - d : d - first;
  for (int q0 = 0; q0 < cnt; q0 += G) {
    int pos[G];
    int64_t k[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
      pos[g] = UP ? first - (q0 + g) : first + (q0 + g);
      k[g] = q0 + g < cnt ? __ldg(col + pos[g]) : i; // past the end: a harmless load of y_i
    }
    T yk[G][B], m[G][B2];
#pragma unroll
    for (int g = 0; g < G; ++g) {
#pragma unroll
      for (int c = 0; c < B; ++c)
        yk[g][c] = y[k[g] * B + c];
#pragma unroll
      for (int q = 0; q < B2; ++q)
        m[g][q] = q0 + g < cnt ? __ldg(val + int64_t(pos[g]) * B2 + q) : T(0);
    }
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (q0 + g < cnt) {
#pragma unroll
        for (int r = 0; r < B; ++r)
#pragma unroll
          for (int c = 0; c < B; ++c)
            yi[r] = ilu_sub(yi[r], ilu_mul(m[g][r * B + c], yk[g][c]));
      }
  }
  if (!UP) {
#pragma unroll
    for (int r = 0; r < B; ++r)
      y[int64_t(i) * B + r] = yi[r];
    return;
  }
  const T* D = val + int64_t(d) * B2;
#pragma unroll
  for (int r = 0; r < B; ++r) {
    T acc = ilu_mul(__ldg(D + r * B), yi[0]);
#pragma unroll
    for (int c = 1; c < B; ++c)
      acc = ilu_add(acc, ilu_mul(__ldg(D + r * B + c), yi[c]));
    y[int64_t(i) * B + r] = acc;
  }
}

// One wide dependency level of a substitution, one thread per row.
template<int B, class T, bool UP>
__global__ void
k_ilu_level(int nr, const int* __restrict__ rows, const int* __restrict__ ptr,
            const int* __restrict__ col, const int* __restrict__ diag,
            const T* __restrict__ val, T* __restrict__ y)
{
  GB_PDL_ENTRY();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nr)
    return;
  ilu_row<B, T, UP>(__ldg(rows + t), ptr, col, diag, val, y);
}

__device__ __forceinline__ void
prefetch_l1(const void* p)
{
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// The consecutive narrow levels lv0..lv1-1 of a substitution in one CTA: the
// levels run in order with a block barrier between them, which makes the rows
// one level wrote visible to the threads of the next (y is read by coherent
// loads). Per level a thread takes rows t, t + 1024, ... of the level. Before
// the barrier it fetches the first row of its next level, that row's entry
// range and the cache lines of the row's columns and values into L1, so that
// after the barrier only the loads of y wait on the previous level. The rows
// run the same arithmetic in the same order as k_ilu_level's.
template<int B, class T, bool UP>
__global__ void __launch_bounds__(kIluCtaThreads, 1)
k_ilu_levels(int lv0, int lv1, const int* __restrict__ lptr, const int* __restrict__ rows,
             const int* __restrict__ ptr, const int* __restrict__ col,
             const int* __restrict__ diag, const T* __restrict__ val, T* __restrict__ y)
{
  GB_PDL_ENTRY();
  int o0 = __ldg(lptr + lv0), o1 = __ldg(lptr + lv0 + 1);
  for (int lv = lv0; lv < lv1; ++lv) {
    for (int t = o0 + threadIdx.x; t < o1; t += kIluCtaThreads)
      ilu_row<B, T, UP>(__ldg(rows + t), ptr, col, diag, val, y);
    int o2 = o1;
    if (lv + 1 < lv1) {
      o2 = __ldg(lptr + lv + 2);
      const int t = o1 + threadIdx.x;
      if (t < o2) {
        const int i = __ldg(rows + t);
        const int pb = __ldg(ptr + i), pe = __ldg(ptr + i + 1) - 1;
        prefetch_l1(col + pb);
        prefetch_l1(col + pe);
        prefetch_l1(val + int64_t(pb) * B * B);
        prefetch_l1(val + (int64_t(pb + pe) / 2) * B * B);
        prefetch_l1(val + (int64_t(pe) + 1) * B * B - 1);
      }
    }
    __syncthreads();
    o0 = o1;
    o1 = o2;
  }
}

// ------------------------------------- both substitutions in one cluster
//
// A packed copy of the factors for k_ilu_cluster, one per direction (0 forward,
// 1 backward). CTA r of the cluster owns the rows [r chunk, (r + 1) chunk). Its
// rows are put in groups of 32 (one per lane) of one dependency level each, the
// groups in level order: group g's lane l works on row[32 g + l] (-1: none).
// base[g] >> 1 is the group's first entry, bit 0 whether some entry is in
// another CTA's rows. A row's entries are in the substitution's order at the
// end of the group's width, a multiple of ilu_half(B); before them it has entries
// of value 0 and a column that is always there (place chunk * B of the own
// CTA, which holds zeros). A column is coded owner << 24 | place of its first
// component; its block follows component-major.
// Where a CTA's rows use few rows of other CTAs (a row goes to at most kIluPush
// others), the CTA keeps copies of those behind its own (places chunk + 1 + k
// for the k-th of its list ghost[gofs[r]..], ascending), which their owners
// write (push: coded places, -1 none, kIluPush per slot); no column then is in
// another CTA.
template<class T>
struct IluPack
{
  int chunk;
  const int *gptr, *row, *base, *col, *push, *gofs;
  const T* val;
  const T* dinv; // backward only: the inverted diagonal blocks
};

constexpr int kIluPush = 2;

// The "not yet computed" mark of a word of y: all bits set, a NaN. It is told
// by the upper 32 bits, and a computed value with such bits is stored as
// another NaN.
template<class T>
struct IluWord;
template<>
struct IluWord<float>
{
  using U = uint32_t;
  static constexpr U kMark = 0xffffffffu, kNaN = 0x7fffffffu;
  static __device__ __forceinline__ U bits(float v) { return __float_as_uint(v); }
  static __device__ __forceinline__ float value(U u) { return __uint_as_float(u); }
  static __device__ __forceinline__ uint32_t upper(U u) { return u; }
  template<bool FAR>
  static __device__ __forceinline__ U load(uint32_t a)
  {
    U v;
    if (FAR)
      asm volatile("ld.relaxed.cluster.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    else
      asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(uint32_t a, U v)
  {
    asm volatile("st.relaxed.cluster.shared::cta.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
  static __device__ __forceinline__ void send(uint32_t a, U v)
  {
    asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
  }
};
template<>
struct IluWord<double>
{
  using U = unsigned long long;
  static constexpr U kMark = 0xffffffffffffffffull, kNaN = 0x7fffffffffffffffull;
  static __device__ __forceinline__ U bits(double v) { return __double_as_longlong(v); }
  static __device__ __forceinline__ double value(U u) { return __longlong_as_double(u); }
  static __device__ __forceinline__ uint32_t upper(U u) { return uint32_t(u >> 32); }
  template<bool FAR>
  static __device__ __forceinline__ U load(uint32_t a)
  {
    U v;
    if (FAR)
      asm volatile("ld.relaxed.cluster.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    else
      asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
  }
  static __device__ __forceinline__ void store(uint32_t a, U v)
  {
    asm volatile("st.relaxed.cluster.shared::cta.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
  }
  static __device__ __forceinline__ void send(uint32_t a, U v)
  {
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
  }
};

// entries consumed together: their blocks and y in registers
__host__ __device__ constexpr int
ilu_half(int B)
{
  return B == 1 ? 8 : B == 2 ? 4 : 2;
}

// The packed layout from the row-sorted factors, one warp per group; col is
// null when only the values changed.
template<class T, bool UP>
__global__ void
k_ilu_pack(int ngroups, int B, int chunk, const int* __restrict__ row,
           const int* __restrict__ base, const int* __restrict__ ptr,
           const int* __restrict__ fcol, const int* __restrict__ diag,
           const double* __restrict__ v, const int* __restrict__ gptr,
           const int* __restrict__ gofs, const int* __restrict__ ghost,
           int* __restrict__ col, T* __restrict__ val, T* __restrict__ dinv)
{
  GB_PDL_ENTRY();
  const int lane = threadIdx.x & 31, B2 = B * B;
  const int g = static_cast<int>((blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5);
  if (g >= ngroups)
    return;
  int rank = 0;
  while (g >= gptr[rank + 1])
    ++rank;
  const int i = row[int64_t(g) * kSlice + lane];
  const int e0 = base[g] >> 1, w = (base[g + 1] >> 1) - e0;
  const int d = i < 0 ? 0 : diag[i];
  const int first = i < 0 ? 0 : (UP ? ptr[i + 1] - 1 : ptr[i]);
  const int cnt = i < 0 ? 0 : (UP ? first - d : d - first);
  const int pad = w - cnt;
  for (int e = 0; e < w; ++e) {
    const int64_t at = int64_t(e0) + e;
    const int p = UP ? first - (e - pad) : first + (e - pad);
    if (col) {
      const int k = e < pad ? 0 : fcol[p];
      int code = (rank << kIluOwnerShift) | (chunk * B);
      if (e >= pad) {
        code = ((k / chunk) << kIluOwnerShift) | ((k % chunk) * B);
        if (k / chunk != rank && gofs[rank] < gofs[rank + 1]) {
          int lo = gofs[rank], hi = gofs[rank + 1] - 1; // k is in the list
          while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (ghost[mid] < k)
              lo = mid + 1;
            else
              hi = mid;
          }
          code = (rank << kIluOwnerShift) | ((chunk + 1 + lo - gofs[rank]) * B);
        }
      }
      col[at * kSlice + lane] = code;
    }
    for (int q = 0; q < B2; ++q)
      val[(at * B2 + q) * kSlice + lane] =
        e < pad ? T(0) : static_cast<T>(v[int64_t(p) * B2 + q]);
  }
  if (UP)
    for (int q = 0; q < B2; ++q)
      dinv[(int64_t(g) * B2 + q) * kSlice + lane] =
        i < 0 ? T(0) : static_cast<T>(v[int64_t(d) * B2 + q]);
}

template<class T>
__host__ __device__ constexpr int
ilu_threads()
{
  return sizeof(T) == 4 ? 768 : 512;
}

// One direction of k_ilu_cluster: this CTA's groups, warp by warp in level
// order. in: the rows' right-hand side; out: the result in global memory. All
// that does not depend on other rows (columns, values, addresses) is done
// before a group waits; from the moment its last dependency is stored to its
// own store there is one poll, one read of 8 entries and their multiply-adds.
template<int B, class T, bool UP>
__device__ __forceinline__ void
ilu_cluster_run(const IluPack<T>& A, uint32_t y, int rank, const T* in, T* out, T* u, T omega,
                bool u_zero, volatile int* give_up, const volatile int* err,
                unsigned long long wait_ns)
{
  using W = IluWord<T>;
  using U = typename W::U;
  constexpr int B2 = B * B, H = ilu_half(B);
  // halves loaded together
  constexpr int N = B == 1 ? 2 : 1;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int g1 = A.gptr[rank + 1];
  int g = A.gptr[rank] + int(threadIdx.x >> 5);
  if (g >= g1)
    return;
  // after a round of polls: whether the warp gives up, which it does when one
  // wait has taken wait_ns, with another warp of the CTA, or with a wait of an
  // earlier launch that nothing has reported yet; it then waits no more
  unsigned spins = 0;
  unsigned long long t0 = 0;
  bool ended = __any_sync(kAll, *give_up);
  auto expired = [&]() -> bool {
    if (ended || (++spins & 1023u) != 0)
      return ended;
    const unsigned long long t = global_ns();
    t0 = t0 ? t0 : t;
    ended = __any_sync(kAll, *give_up || *err || t - t0 > wait_ns);
    if (ended)
      *give_up = 1;
    return ended;
  };
  int ni = __ldg(A.row + int64_t(g) * kSlice + lane);
  int n0 = __ldg(A.base + g), n1 = __ldg(A.base + g + 1);
  for (; g < g1; g += nw) {
    const int i = ni, b0 = n0 >> 1, b1 = n1 >> 1;
    const bool far = n0 & 1;
    if (g + nw < g1) { // the next group's head, while this one waits
      ni = __ldg(A.row + int64_t(g + nw) * kSlice + lane);
      n0 = __ldg(A.base + g + nw);
      n1 = __ldg(A.base + g + nw + 1);
    }
    T acc[B], D[UP ? B2 : 1];
#pragma unroll
    for (int r = 0; r < B; ++r)
      acc[r] = i < 0 ? T(0)
                     : (UP ? __ldcg(in + int64_t(i) * B + r) : in[int64_t(i) * B + r]);
    if (UP) {
#pragma unroll
      for (int q = 0; q < B2; ++q)
        D[q] = __ldg(A.dinv + (int64_t(g) * B2 + q) * kSlice + lane);
    }
    int push[kIluPush];
#pragma unroll
    for (int k = 0; k < kIluPush; ++k)
      push[k] = A.push ? __ldg(A.push + (int64_t(g) * kIluPush + k) * kSlice + lane) : -1;
    T ui[UP ? B : 1];
    if (UP && u && !u_zero && i >= 0) {
#pragma unroll
      for (int r = 0; r < B; ++r)
        ui[r] = u[int64_t(i) * B + r];
    }
    const uint32_t own = y + uint32_t((i - rank * A.chunk) * B) * uint32_t(sizeof(T));
    for (int b = b0; b < b1; b += N * H) {
      uint32_t at[N * H];
      T m[N * H][B2];
      const int* cp = A.col + int64_t(b) * kSlice + lane;
      const T* vp = A.val + int64_t(b) * B2 * kSlice + lane;
#pragma unroll
      for (int e = 0; e < N * H; ++e)
        if (e < H || b + H < b1) {
          at[e] = uint32_t(__ldg(cp + e * kSlice));
#pragma unroll
          for (int p = 0; p < B2; ++p)
            m[e][p] = __ldg(vp + (e * B2 + p) * kSlice);
        }
#pragma unroll
      for (int e = 0; e < N * H; ++e)
        if (e < H || b + H < b1) {
          const uint32_t c = at[e];
          at[e] = y + (c & uint32_t(kIluPlaceMask)) * uint32_t(sizeof(T));
          if (far)
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                         : "=r"(at[e]) : "r"(at[e]), "r"(c >> kIluOwnerShift));
        }
      auto consume = [&](auto is_far, auto half) {
        constexpr bool kFar = decltype(is_far)::value;
        constexpr int h = decltype(half)::value * H;
        spins = 0; // a wait of its own
        t0 = 0;
        // what a row waits for longest is mostly its last entry: that one is
        // polled alone (a load and a vote), then all are read
        while (__any_sync(kAll, W::upper(W::template load<kFar>(at[h + H - 1])) ==
                                  0xffffffffu) &&
               !expired())
          ;
        U v[H][B];
        uint32_t top;
        do {
#pragma unroll
          for (int e = 0; e < H; ++e)
#pragma unroll
            for (int q = 0; q < B; ++q)
              v[e][q] = W::template load<kFar>(at[h + e] + q * uint32_t(sizeof(T)));
          uint32_t t[2] = { 0, 0 }; // two chains
#pragma unroll
          for (int e = 0; e < H; ++e)
#pragma unroll
            for (int q = 0; q < B; ++q)
              t[(e * B + q) & 1] = max(t[(e * B + q) & 1], W::upper(v[e][q]));
          top = max(t[0], t[1]);
        } while (__any_sync(kAll, top == 0xffffffffu) && !expired());
#pragma unroll
        for (int e = 0; e < H; ++e)
#pragma unroll
          for (int r = 0; r < B; ++r)
#pragma unroll
            for (int q = 0; q < B; ++q) // before the row's first entry: 0 * 0
              acc[r] = ilu_sub(acc[r], ilu_mul(m[h + e][r * B + q], W::value(v[e][q])));
      };
      using First = std::integral_constant<int, 0>;
      using Second = std::integral_constant<int, N - 1>;
      if (far)
        consume(std::true_type{}, First{});
      else
        consume(std::false_type{}, First{});
      if (N == 2 && b + H < b1) {
        if (far)
          consume(std::true_type{}, Second{});
        else
          consume(std::false_type{}, Second{});
      }
    }
    if (UP) {
      T z[B];
#pragma unroll
      for (int r = 0; r < B; ++r) {
        z[r] = ilu_mul(D[r * B], acc[0]);
#pragma unroll
        for (int q = 1; q < B; ++q)
          z[r] = ilu_add(z[r], ilu_mul(D[r * B + q], acc[q]));
      }
#pragma unroll
      for (int r = 0; r < B; ++r)
        acc[r] = z[r];
    }
    if (i >= 0) {
#pragma unroll
      for (int r = 0; r < B; ++r) {
        const U w = W::bits(acc[r]);
        W::store(own + r * uint32_t(sizeof(T)), W::upper(w) == 0xffffffffu ? W::kNaN : w);
      }
#pragma unroll
      for (int k = 0; k < kIluPush; ++k)
        if (push[k] >= 0) {
          uint32_t a;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                       : "=r"(a)
                       : "r"(y + uint32_t(push[k] & kIluPlaceMask) * uint32_t(sizeof(T))),
                         "r"(push[k] >> kIluOwnerShift));
#pragma unroll
          for (int r = 0; r < B; ++r) {
            const U w = W::bits(acc[r]);
            W::send(a + r * uint32_t(sizeof(T)), W::upper(w) == 0xffffffffu ? W::kNaN : w);
          }
        }
#pragma unroll
      for (int r = 0; r < B; ++r) {
        const int64_t k = int64_t(i) * B + r;
        out[k] = acc[r];
        if (UP && u) {
          const T s = ilu_mul(omega, acc[r]);
          u[k] = u_zero ? s : ilu_add(ui[r], s);
        }
      }
    }
    __syncwarp();
  }
}

// h = (L U)^-1 rhs by both substitutions in one launch of one thread-block
// cluster, then u = (u_zero ? 0 : u) + omega h (u may be null). What bounds it
// is the chain of dependency levels (449 per direction on a 65^3 lexicographic
// mesh), not the bytes: so y lives in the CTAs' shared memory, where a row sees
// a dependency about 0.1 us after it was written (its own CTA's memory, or the
// owner's over the cluster network), and rows wait for the values themselves,
// with no barrier or launch between levels. A group's matrix entries are loaded
// before it waits, so the other warps' loads run meanwhile. Each row runs
// ilu_row's arithmetic in its order: the same bits. Measured on the 65^3 Q1
// level (FP64, both substitutions): 0.57 ms against about 3.4 ms with the level
// launches; a mixed solve of that mesh (6 steps) 112.9 -> 16.7 ms. About 0.42
// us per level within one CTA. Reading other CTAs' memory in place of the copies
// made it 0.65 ms (a group with one such column polls over the network). More
// warps hide the matrix loads: 128 / 256 / 384 / 512 threads 1.81 / 0.98 / 0.74
// / 0.65 ms in FP64, and in FP32, whose rows need 80 registers, 512 / 768
// threads 18.8 / 16.7 ms for the solve. Rows of an average level per CTA
// (kIluRowsPerLevel): 64 / 32 / 16 measured 213 / 183 / 180 us on the 33^3
// level. Levels whose y exceeds the cluster's shared memory (about 440,000 rows
// in FP64, twice that in FP32), and chains whose packed factors would be mostly
// padding, keep the level launches (gb_ilu_plan.cuh). Every wait ends: a row
// waits only for rows of earlier levels, a warp takes its groups in level
// order, and the CTAs of a cluster run at the same time; bounded all the same, by
// wait_ns for each wait. A warp that gives up goes through its remaining groups
// without waiting, so every row is stored and every thread reaches the barriers.
template<int B, class T>
__global__ void __launch_bounds__(ilu_threads<T>(), 1)
k_ilu_cluster(IluPack<T> lo, IluPack<T> up, int n, const T* rhs, T* h, T* u, double omega,
              int u_zero, int* err, unsigned long long wait_ns, unsigned phantoms)
{
  extern __shared__ __align__(16) unsigned char ilu_smem[];
  __shared__ int give_up;
  using W = IluWord<T>;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const uint32_t y = static_cast<uint32_t>(__cvta_generic_to_shared(ilu_smem));
  const int mine = min(lo.chunk, n - int(rank) * lo.chunk) * B, copies = (lo.chunk + 1) * B;
  auto mark = [&](const IluPack<T>& A) {
    for (int k = threadIdx.x; k < mine; k += blockDim.x)
      W::store(y + uint32_t(k) * uint32_t(sizeof(T)), W::kMark);
    const int nc = (A.gofs[rank + 1] - A.gofs[rank]) * B;
    for (int k = threadIdx.x; k < nc; k += blockDim.x)
      W::store(y + uint32_t(copies + k) * uint32_t(sizeof(T)), W::kMark);
  };
  if (threadIdx.x == 0)
    give_up = 0;
  // what the entries before a row's first one read; with phantoms (a test) it
  // never comes
  if (threadIdx.x < B)
    W::store(y + uint32_t(lo.chunk * B + threadIdx.x) * uint32_t(sizeof(T)),
             phantoms ? W::kMark : 0);
  GB_PDL_ENTRY();
  mark(lo);
  cluster_barrier();
  ilu_cluster_run<B, T, false>(lo, y, int(rank), rhs, h, nullptr, T(0), false, &give_up, err,
                               wait_ns);
  cluster_barrier();
  mark(up);
  cluster_barrier();
  ilu_cluster_run<B, T, true>(up, y, int(rank), h, h, u, static_cast<T>(omega), u_zero != 0,
                              &give_up, err, wait_ns);
  cluster_barrier(); // no CTA leaves while another reads its part of y
  if (threadIdx.x == 0 && give_up)
    atomicCAS(err, 0, kWaitIlu);
}

// u = (u_zero ? 0 : u) + omega h (StdSolver::Add after the ILU solve, unfused)
template<class T>
__global__ void
k_ilu_axpy(int64_t n, T* __restrict__ u, double omega, const T* __restrict__ h, int u_zero)
{
  GB_PDL_ENTRY();
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n)
    return;
  const T w = ilu_mul(static_cast<T>(omega), h[i]);
  u[i] = u_zero ? w : ilu_add(u[i], w);
}

} // namespace gb
