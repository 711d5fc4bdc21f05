// gain_grad.cu -- loss and gradient of gain calibration on packed triangles.
//
// For per-input complex gains g (shared by all channels), observed and model
// visibilities R_obs, R_mod and real weights W (all packed lower triangles,
// Hermitian, one per channel):
//   M_ij = g_i R_mod,ij conj(g_j),   E_ij = R_obs,ij - M_ij
//   L    = sum_f sum_{i,j} W_ij |E_ij|^2          (full matrices: off-diagonal
//                                                 entries of the triangle count twice)
//   grad_k = dL/dRe(g_k) + i dL/dIm(g_k) = 2 dL/dconj(g_k)
//          = -4 sum_f sum_j W_kj E_kj conj(R_mod,kj) g_j
// For a stored element (i, j < i), c = W E_ij conj(R_mod,ij) feeds row i
// through c g_j and row j through conj(c) g_i (the Hermitian mirror).
//
// Memory bound (20 bytes per stored element, read once).  One block per tile
// of 64 rows x 128 columns of one channel's triangle.  Warp w owns rows w,
// w + 8, ... of the tile and lane l its columns l, l + 32, l + 64, l + 96, so
// each load of a warp covers 32 consecutive packed elements (a lane that
// owned neighbouring columns asked for every sector twice) and a row segment's
// sum is one warp reduction per 128 elements, with no block barrier per row.
// Column sums stay in registers until
// one shared-memory combine per tile.  Within a tile the partial sums are FP32
// (a row's four terms per lane, then the warp's; a column's eight per warp,
// then the warps'); across tiles they are added to FP64 accumulators with
// atomics, and the loss is accumulated in FP64.
// 2048 inputs x 32 channels (1.34 GB): 244 -> 207 us in short runs, 278 -> 234
// us at the power limit; with no occupancy bound (91 registers, two blocks per
// SM) 261 us.
#include <cstdint>
#include <type_traits>

#include "herk_fp8.cuh"

namespace ftdx {
namespace {

constexpr int kGT = 64;          // rows per tile
constexpr int kGCols = 4;        // columns per lane
constexpr int kGW = 32 * kGCols; // columns per tile
constexpr int kGWarps = 8;       // rows of a tile are dealt to 8 warps

struct GainTerms {
  float rre, rim;   // row i's contribution c g_j
  float cre, cim;   // column j's contribution conj(c) g_i (zero on the diagonal)
  double l;         // W |E|^2 (times 2 off the diagonal)
};

__device__ __forceinline__ GainTerms gain_terms(float2 o, float2 m0, float wt, float2 a, float2 b,
                                                bool diag) {
  // M = g_i R_mod conj(g_j), E = R_obs - M, c = W E conj(R_mod)
  const float tr = a.x * m0.x - a.y * m0.y, tim = a.x * m0.y + a.y * m0.x;
  const float mr = tr * b.x + tim * b.y, mi = tim * b.x - tr * b.y;
  const float er = o.x - mr, ei = o.y - mi;
  const float cr = wt * (er * m0.x + ei * m0.y), ci = wt * (ei * m0.x - er * m0.y);
  GainTerms t;
  t.rre = cr * b.x - ci * b.y;
  t.rim = cr * b.y + ci * b.x;
  t.cre = diag ? 0.f : cr * a.x + ci * a.y;
  t.cim = diag ? 0.f : cr * a.y - ci * a.x;
  t.l = (diag ? 1.0 : 2.0) * double(wt) * (double(er) * er + double(ei) * ei);
  return t;
}

__global__ void __launch_bounds__(256, 4) gain_grad_kernel(const float2* __restrict__ robs,
                                                        const float2* __restrict__ rmod,
                                                        const float* __restrict__ w,
                                                        const float2* __restrict__ g, int n,
                                                        int tiles_per_chan,
                                                        double* __restrict__ grad,  // [n][2]
                                                        double* __restrict__ loss) {
  const int ch = blockIdx.y;
  // tile (ti, tj) from the linear index: row tiles 2p and 2p + 1 have p + 1
  // column tiles each, and p(p + 1) tiles lie before row tile 2p
  const int r = blockIdx.x;
  if (r >= tiles_per_chan) return;
  int p = int((sqrtf(4.f * float(r) + 1.f) - 1.f) * 0.5f);
  while (p > 0 && p * (p + 1) > r) --p;
  while ((p + 1) * (p + 2) <= r) ++p;
  const int rest = r - p * (p + 1);
  const int ti = 2 * p + (rest > p ? 1 : 0), tj = rest > p ? rest - (p + 1) : rest;
  const int i0 = ti * kGT, j0 = tj * kGW;
  const int64_t P = int64_t(n) * (n + 1) / 2;
  const float2* ro = robs + int64_t(ch) * P;
  const float2* rm = rmod + int64_t(ch) * P;
  const float* wc = w + int64_t(ch) * P;

  __shared__ float2 gi[kGT];
  __shared__ float row_re[kGT], row_im[kGT];
  __shared__ float col_re[kGWarps][kGW], col_im[kGWarps][kGW];
  __shared__ double lsum[kGWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < kGT) gi[tid] = (i0 + tid < n) ? g[i0 + tid] : make_float2(0.f, 0.f);
  // this lane's columns and their gains
  float2 gj[kGCols];
#pragma unroll
  for (int c = 0; c < kGCols; ++c) {
    const int j = j0 + lane + 32 * c;
    gj[c] = j < n ? __ldg(g + j) : make_float2(0.f, 0.f);
  }
  __syncthreads();

  float cre[kGCols] = {}, cim[kGCols] = {};
  double lacc = 0.0;
  // one row segment of the tile; kWhole: all of it lies below the diagonal and
  // inside n, so no element needs a bounds check or the diagonal's rule
  auto row_segment = [&](int row, auto whole) {
    constexpr bool kWhole = decltype(whole)::value;
    const int i = i0 + row;
    const int64_t e0 = int64_t(i) * (i + 1) / 2 + j0 + lane;
    float2 o[kGCols], m[kGCols];
    float wt[kGCols];
#pragma unroll
    for (int c = 0; c < kGCols; ++c) {
      const bool ok = kWhole || (i < n && j0 + lane + 32 * c <= i);
      o[c] = ok ? __ldcs(ro + e0 + 32 * c) : make_float2(0.f, 0.f);
      m[c] = ok ? __ldcs(rm + e0 + 32 * c) : make_float2(0.f, 0.f);
      wt[c] = ok ? __ldcs(wc + e0 + 32 * c) : 0.f;
    }
    const float2 a = gi[row];
    float rre[kGCols] = {}, rim[kGCols] = {};
#pragma unroll
    for (int c = 0; c < kGCols; ++c) {
      const int j = j0 + lane + 32 * c;
      if (!kWhole && (i >= n || j > i)) continue;
      const GainTerms t = gain_terms(o[c], m[c], wt[c], a, gj[c], !kWhole && i == j);
      rre[c] = t.rre;
      rim[c] = t.rim;
      cre[c] += t.cre;
      cim[c] += t.cim;
      lacc += t.l;
    }
    float sre = (rre[0] + rre[1]) + (rre[2] + rre[3]);
    float sim = (rim[0] + rim[1]) + (rim[2] + rim[3]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      sre += __shfl_xor_sync(0xffffffffu, sre, off);
      sim += __shfl_xor_sync(0xffffffffu, sim, off);
    }
    if (lane == 0) {
      row_re[row] = sre;
      row_im[row] = sim;
    }
  };
  if (j0 + kGW <= i0 && i0 + kGT <= n) {
#pragma unroll 1
    for (int row = warp; row < kGT; row += kGWarps) row_segment(row, std::true_type{});
  } else {
#pragma unroll 1
    for (int row = warp; row < kGT; row += kGWarps) row_segment(row, std::false_type{});
  }
#pragma unroll
  for (int c = 0; c < kGCols; ++c) {
    col_re[warp][lane + 32 * c] = cre[c];
    col_im[warp][lane + 32 * c] = cim[c];
  }
  for (int off = 16; off > 0; off >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, off);
  if (lane == 0) lsum[warp] = lacc;
  __syncthreads();
  if (tid < kGT) {
    const int i = i0 + tid;
    if (i < n) {
      atomicAdd(grad + 2 * i, -4.0 * double(row_re[tid]));
      atomicAdd(grad + 2 * i + 1, -4.0 * double(row_im[tid]));
    }
  } else if (tid < kGT + kGW) {
    const int c = tid - kGT;
    const int jj = j0 + c;
    if (jj < n) {
      float sre = 0.f, sim = 0.f;
#pragma unroll
      for (int q = 0; q < kGWarps; ++q) {
        sre += col_re[q][c];
        sim += col_im[q][c];
      }
      atomicAdd(grad + 2 * jj, -4.0 * double(sre));
      atomicAdd(grad + 2 * jj + 1, -4.0 * double(sim));
    }
  } else if (tid == kGT + kGW) {
    double sacc = 0.0;
    for (int q = 0; q < kGWarps; ++q) sacc += lsum[q];
    atomicAdd(loss, sacc);
  }
}

// The accumulators of both outputs, in one launch.
__global__ void __launch_bounds__(256) zero_outputs_kernel(double* __restrict__ grad, int len,
                                                           double* __restrict__ loss) {
  const int x = blockIdx.x * 256 + threadIdx.x;
  if (x < len) grad[x] = 0.0;
  if (x == len) *loss = 0.0;
}

}  // namespace

cudaError_t launch_gain_grad(const float2* robs, const float2* rmod, const float* w,
                             const float2* g, int n, int nchan, double* grad, double* loss,
                             cudaStream_t s) {
  zero_outputs_kernel<<<unsigned((2 * n + 256) / 256), 256, 0, s>>>(grad, 2 * n, loss);
  // row tiles 2p and 2p + 1 reach p + 1 column tiles each
  const int nt = (n + kGT - 1) / kGT, np = nt / 2;
  const int per = np * (np + 1) + (nt & 1 ? np + 1 : 0);
  gain_grad_kernel<<<dim3(unsigned(per), unsigned(nchan)), 256, 0, s>>>(robs, rmod, w, g, n, per,
                                                                       grad, loss);
  return cudaGetLastError();
}

}  // namespace ftdx
