// precision.cu -- promotion of float complex voltages to the FP8 operand
// planes with a per-channel scale, plain or split into hi + lo parts.
//
//   amax pass   : per channel, the largest |Re| or |Im| (atomicMax on the
//                 bit patterns of non-negative floats, which order like ints)
//   scale       : s_c = 448 / amax_c (448 = largest finite E4M3); the
//                 correlator multiplies channel c's result by 1 / s_c^2
//   quantise    : hi = E4M3(s_c x) (round to nearest even, saturating) into
//                 columns [0, Kp) of the planes; in split mode also
//                 lo = E4M3(s_c x - hi) into columns [Kp, 2 Kp).  With the
//                 correlator's K segments (hi,hi) + (hi,lo) + (lo,hi) this
//                 carries about 7 significant bits per sample instead of 4.
//
// In the plain mode large channels take one cooperative persistent kernel
// (scale_quantize_kernel) when the device can hold its grid: each
// block takes the same share of every channel, finds the amax of its share
// of channel c while it quantises its share of channel c - 1, which it read
// one channel earlier and which is still in L2, so HBM sees the input once.
// Small channels (launch_float_to_planes says which), the split mode, and a
// grid that cannot be co-resident, use two kernels (amax, quantise) that read
// it twice.
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <mutex>

#include "herk_fp8.cuh"
#include "sm100.cuh"

namespace ftdx {
namespace {

// Per channel c (blockIdx.y): the largest |Re| or |Im|.  Each thread reads
// two samples (16 bytes) per load, four loads in flight; `vec` (uniform)
// says the channel starts 16-byte aligned and per_chan is even.
__global__ void __launch_bounds__(256) amax_kernel(const float2* __restrict__ a, int64_t per_chan,
                                                   uint32_t* __restrict__ amax_bits, int vec) {
  dev::griddep_launch();
  const int c = blockIdx.y;
  const float2* p = a + int64_t(c) * per_chan;
  float m = 0.f;
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  const int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (vec) {
    const float4* p4 = reinterpret_cast<const float4*>(p);
    const int64_t n4 = per_chan >> 1;
    int64_t i = t0;
    for (; i + 3 * stride < n4; i += 4 * stride) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(p4 + i + u * stride);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        m = fmaxf(m, fmaxf(fmaxf(fabsf(v[u].x), fabsf(v[u].y)), fmaxf(fabsf(v[u].z), fabsf(v[u].w))));
    }
    for (; i < n4; i += stride) {
      const float4 v = __ldg(p4 + i);
      m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
  } else {
    for (int64_t i = t0; i < per_chan; i += stride) {
      const float2 v = __ldg(p + i);
      m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
    }
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float wm[8];
  if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < int(blockDim.x >> 5); ++w) m = fmaxf(m, wm[w]);
    if (!(m == m)) m = 0.f;  // NaN input: treat as empty
    atomicMax(amax_bits + c, __float_as_uint(m));
  }
}

// A channel's scale from its largest component; the correlator multiplies its
// result by 1 / scale^2.
__device__ __forceinline__ float channel_scale(float amax) {
  return (amax > 0.f && amax < 3.0e38f) ? 448.f / amax : 1.f;
}

__device__ __forceinline__ uint32_t e4m3x2(float a, float b) {
  return uint32_t(__nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ float e4m3_to_float(uint32_t byte) {
  const __half_raw hr = __nv_cvt_fp8_to_halfraw(__nv_fp8_storage_t(byte), __NV_E4M3);
  return __half2float(__half(hr));
}

// L2 policy that makes lines the first to be evicted (for data read for
// the last time).
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ float4 ldg_last_use(const float4* p, uint64_t pol) {
  float4 v;
  asm volatile("ld.global.nc.L1::evict_first.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p), "l"(pol));
  return v;
}

// Half a warp takes a span of 128 samples of one row, in two layouts: loaded,
// lane h (0..15) holds the samples 32 q + 2 h and 32 q + 2 h + 1 (q < 4), so that
// each 16-byte load of the half warp covers 256 consecutive bytes; stored, the
// samples 8 h .. 8 h + 7, 8 bytes of every plane.  (Lanes that loaded their own
// 8 samples asked for 32 sectors with every load, four times over: 203 against
// 178 us for 16 channels of 4096 x 1024 in the cooperative kernel.)  src = the row + the span's first sample t0; samples at or past K
// read as 0.  pol != 0: an L2 policy for the 16-byte loads (the samples' last
// use).
__device__ __forceinline__ void load_span(const float2* __restrict__ src, int t0, int K, bool vec,
                                          float (&xr)[8], float (&xi)[8], uint64_t pol = 0) {
  const int h = int(threadIdx.x) & 15;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int t = 32 * q + 2 * h;
    if (vec && t0 + t < K) {  // K is even
      const float4* p4 = reinterpret_cast<const float4*>(src + t);
      const float4 v = pol ? ldg_last_use(p4, pol) : __ldg(p4);
      xr[2 * q] = v.x, xi[2 * q] = v.y, xr[2 * q + 1] = v.z, xi[2 * q + 1] = v.w;
    } else {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float2 v = t0 + t + b < K ? __ldg(src + t + b) : make_float2(0.f, 0.f);
        xr[2 * q + b] = v.x, xi[2 * q + b] = v.y;
      }
    }
  }
}

// The bytes of a span from the loaded to the stored layout: w[q] holds this
// lane's pair q as Re, Re, Im, Im; re and im receive the 8 bytes of the samples
// 8 h .. 8 h + 7.  buf: 64 words of shared memory of the half warp.
__device__ __forceinline__ void span_bytes(const uint32_t (&w)[4], uint32_t* buf, uint2& re,
                                           uint2& im) {
  const int h = int(threadIdx.x) & 15;
  const uint32_t half = 0xFFFFu << (int(threadIdx.x) & 16);
#pragma unroll
  for (int q = 0; q < 4; ++q) buf[16 * q + h] = w[q];
  __syncwarp(half);
  const uint4 v = *reinterpret_cast<const uint4*>(buf + 4 * h);
  __syncwarp(half);  // read before the next span is written
  re = make_uint2(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410));
  im = make_uint2(__byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));
}

// E4M3 of a span's scaled samples, in the loaded layout (span_bytes).
__device__ __forceinline__ void span_e4m3(const float (&xr)[8], const float (&xi)[8],
                                          uint32_t (&w)[4]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    w[q] = e4m3x2(xr[2 * q], xr[2 * q + 1]) | (e4m3x2(xi[2 * q], xi[2 * q + 1]) << 16);
}

// A half warp quantises 128 samples of one row (load_span; Kp is a multiple of
// 128); the thread with a channel's first samples stores its out_scale.  vec
// (uniform): K even and the input 16-byte aligned.
__global__ void __launch_bounds__(256) quantize_kernel(const float2* __restrict__ a,
                                                       uint8_t* __restrict__ z, int64_t rows,
                                                       int K, int Kp, int zpitch, int n,
                                                       const uint32_t* amax_bits,
                                                       float* __restrict__ out_scale, int split,
                                                       int rows_per_block, int vec) {
  __shared__ __align__(16) uint32_t bytes[16][64];
  dev::griddep_wait();  // the channels' amax
  dev::griddep_launch();
  const int chunks = Kp >> 3;
  const int64_t r0 = int64_t(blockIdx.x) * rows_per_block;
  const int64_t nrows64 = rows - r0 < rows_per_block ? rows - r0 : rows_per_block;
  const int nloc = int(nrows64) * chunks;  // a multiple of 16: half warps stay together
  const int64_t plane = rows * int64_t(zpitch);
  uint32_t* buf = bytes[threadIdx.x >> 4];
  // the block's rows belong to at most a few channels: 32-bit channel index
  const int c0 = int(r0 / n), rin0 = int(r0 - int64_t(c0) * n);
  int cs = -1;  // the channel s belongs to
  float s = 1.f;
  for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
    const int rl = l / chunks;
    const int t0 = (l - rl * chunks) << 3;  // this lane's samples in the stored layout
    const int64_t r = r0 + rl;
    const int c = c0 + (rin0 + rl) / n;
    if (c != cs) {
      s = channel_scale(__uint_as_float(amax_bits[c]));
      cs = c;
    }
    if (t0 == 0 && r == int64_t(c) * n) out_scale[c] = 1.f / (s * s);
    const int ts = t0 & ~127;
    float xr[8], xi[8];
    load_span(a + r * K + ts, ts, K, vec, xr, xi);
#pragma unroll
    for (int b = 0; b < 8; ++b) xr[b] *= s, xi[b] *= s;
    uint32_t w[4];
    uint2 re, im;
    span_e4m3(xr, xi, w);
    span_bytes(w, buf, re, im);
    uint8_t* dst = z + r * zpitch + t0;
    *reinterpret_cast<uint2*>(dst) = re;
    *reinterpret_cast<uint2*>(dst + plane) = im;
    if (split) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          xr[2 * q + b] -= e4m3_to_float((w[q] >> (8 * b)) & 0xFFu);
          xi[2 * q + b] -= e4m3_to_float((w[q] >> (16 + 8 * b)) & 0xFFu);
        }
      }
      span_e4m3(xr, xi, w);
      span_bytes(w, buf, re, im);
      *reinterpret_cast<uint2*>(dst + Kp) = re;
      *reinterpret_cast<uint2*>(dst + plane + Kp) = im;
    }
  }
}

// (row, unit column) of unit u0 + threadIdx.x of a channel of `chunks` units
// per row, advanced by blockDim.x units per next() without a division.
struct UnitWalk {
  int row, col, drow, dcol, chunks;
  __device__ __forceinline__ UnitWalk(int64_t u0, int chunks_) : chunks(chunks_) {
    const int u = int(u0) + int(threadIdx.x);
    row = u / chunks;
    col = u - row * chunks;
    drow = int(blockDim.x) / chunks;
    dcol = int(blockDim.x) - drow * chunks;
  }
  __device__ __forceinline__ void next() {
    row += drow;
    col += dcol;
    if (col >= chunks) col -= chunks, ++row;
  }
  // first sample of the unit's span (load_span)
  __device__ __forceinline__ int t0() const { return (col & ~15) << 3; }
  // offsets of the span's first sample in a channel's input ([n][K]), and of
  // the unit's in the planes (pitch zpitch)
  __device__ __forceinline__ int64_t offset(int K) const { return int64_t(row) * K + t0(); }
  __device__ __forceinline__ int64_t zoffset(int zpitch) const {
    return int64_t(row) * zpitch + (col << 3);
  }
};

// Number of units of the block range starting at u0 (per_blk units, cut at
// the channel's end; 0 past it).
__device__ __forceinline__ int u1_len(int64_t u0, int64_t per_blk, int64_t units) {
  const int64_t u1 = u0 + per_blk < units ? u0 + per_blk : units;
  return u1 > u0 ? int(u1 - u0) : 0;
}

// Thread 0 of a block of scale_quantize_kernel: wait until every block has
// counted its amax of channel cq into its arrival word (acquire; bounded by
// FTDX_WAIT_NS, after which the status word gets kStatusTimeoutOther and the
// block's later waits are skipped), then the channel's scale (block 0 also
// stores its out_scale).
__device__ __forceinline__ float wait_channel_scale(int cq, float* __restrict__ out_scale,
                                                    uint32_t* amax_bits, uint32_t* arrive_word,
                                                    uint32_t* status, bool& aborted) {
  if (!aborted && !dev::flag_wait_limit(arrive_word, gridDim.x, FTDX_WAIT_NS)) {
    atomicOr(status, dev::kStatusTimeoutOther);
    aborted = true;
  }
  uint32_t mb;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(mb) : "l"(amax_bits + cq) : "memory");
  const float mx = __uint_as_float(mb);
  const float sc = channel_scale(mx);
  if (blockIdx.x == 0) out_scale[cq] = 1.f / (sc * sc);
  return sc;
}

// Quantise one unit's span (load_span) with scale sc into the planes, this
// lane's 8 samples at dst (plane 1 at + plane, plane 2 = -plane 0 at + 2 plane
// when neg), with quantize_kernel's arithmetic; streaming stores (the planes
// are not read again by this kernel).
__device__ __forceinline__ void quantise_unit(float (&xr)[8], float (&xi)[8], float sc,
                                              uint32_t* buf, uint8_t* __restrict__ dst,
                                              int64_t plane, int neg) {
#pragma unroll
  for (int b = 0; b < 8; ++b) xr[b] *= sc, xi[b] *= sc;
  uint32_t w[4];
  uint2 re, im;
  span_e4m3(xr, xi, w);
  span_bytes(w, buf, re, im);
  constexpr uint32_t kS = 0x80808080u;
  __stcs(reinterpret_cast<uint2*>(dst), re);
  __stcs(reinterpret_cast<uint2*>(dst + plane), im);
  if (neg) __stcs(reinterpret_cast<uint2*>(dst + 2 * plane), make_uint2(re.x ^ kS, re.y ^ kS));
}

// Channel amax, scale and quantisation in one cooperative launch (every
// block resident: the blocks wait on one another).  A channel is n rows x
// Kp / 8 units of 8 samples; block b owns the same contiguous unit range of
// every channel, and thread t the units L[k] = t + k blockDim.x of it
// (k < cnt).  With p = ceil(cnt / 2), step c (0 .. batch) is:
//   1. amax over L[0 .. p) of channel c, two units per round trip;
//   2. thread 0 waits for channel c - 1's amax (wait_channel_scale);
//   3. amax over L[p .. cnt) of channel c, each beside the quantisation of
//      L[k] of channel c - 1 (k = 0 ..), both loads in flight together;
//   4. the block's amax of channel c into amax_bits[c] (atomicMax on the
//      bits, as amax_kernel), and the block counted into channel c's
//      arrival word (release; one 128-byte line per channel, so the blocks
//      polling channel c - 1 do not contend with these atomics);
//   5. the rest of channel c - 1's units quantised, two per round trip.
// Two block barriers per step (after 2 and inside 4); the shared scale and
// warp maxima alternate between two slots by step parity, so a step needs
// no closing barrier.  A unit is re-read about one channel of reads (n K
// samples) after its first read, so the re-read hits L2 while a channel is
// well below the L2's size.  neg: also write plane 2 = plane 0 with every
// sign flipped.  Per-element arithmetic is that of the two-kernel path,
// so both give the same bits.
__global__ void __launch_bounds__(256, 4) scale_quantize_kernel(
    const float2* __restrict__ a, uint8_t* __restrict__ z, int K, int Kp, int zpitch, int n,
    int batch, int neg, float* __restrict__ out_scale, uint32_t* amax_bits, uint32_t* arrive,
    uint32_t* status, int vec) {
  dev::griddep_launch();
  const int chunks = Kp >> 3;
  const int64_t units = int64_t(n) * chunks;
  // whole spans of 16 units per block, so that half warps stay together
  const int64_t per_blk = ((units + gridDim.x - 1) / gridDim.x + 15) / 16 * 16;
  const int64_t u0 = int64_t(blockIdx.x) * per_blk;
  const int len = u1_len(u0, per_blk, units);
  const int t = int(threadIdx.x), bd = int(blockDim.x);
  const int cnt = t < len ? (len - t + bd - 1) / bd : 0;  // this thread's units
  const int p = (cnt + 1) / 2;
  const int64_t plane = int64_t(n) * batch * zpitch;
  const int64_t chan_in = int64_t(n) * K, chan_z = int64_t(n) * zpitch;
  const uint64_t pol = l2_evict_first_policy();  // channel c - 1's samples: read for the last time
  __shared__ float wm[2][8];
  __shared__ float s_scale[2];
  __shared__ __align__(16) uint32_t bytes[16][64];
  uint32_t* buf = bytes[threadIdx.x >> 4];
  bool aborted = false;  // thread 0's
  for (int c = 0; c <= batch; ++c) {
    const bool amax_step = c < batch, quant_step = c >= 1;
    const int par = c & 1;
    const float2* cur = a + int64_t(amax_step ? c : 0) * chan_in;        // channel c (amax)
    const float2* prev = a + int64_t(quant_step ? c - 1 : 0) * chan_in;  // channel c - 1
    uint8_t* zprev = z + int64_t(quant_step ? c - 1 : 0) * chan_z;
    float m = 0.f;
    float xr[8], xi[8], yr[8], yi[8];
    UnitWalk wa(u0, chunks), wb(u0, chunks);
    auto amax_of = [&](const float (&r)[8], const float (&im)[8]) {
#pragma unroll
      for (int b = 0; b < 8; ++b) m = fmaxf(m, fmaxf(fabsf(r[b]), fabsf(im[b])));
    };
    int ka = 0, kb = 0;  // next L index of the amax / quantisation walks
    float sc = 1.f;
    if (amax_step) {  // 1
      const int kend = quant_step ? p : cnt;  // the first step has nothing to wait for
      for (; ka + 1 < kend; ka += 2) {
        UnitWalk w2 = wa;
        w2.next();
        load_span(cur + wa.offset(K), wa.t0(), K, vec, xr, xi);
        load_span(cur + w2.offset(K), w2.t0(), K, vec, yr, yi);
        amax_of(xr, xi);
        amax_of(yr, yi);
        w2.next();
        wa = w2;
      }
      if (ka < kend) {
        load_span(cur + wa.offset(K), wa.t0(), K, vec, xr, xi);
        amax_of(xr, xi);
        wa.next();
        ++ka;
      }
    }
    if (quant_step) {
      if (t == 0)  // 2
        s_scale[par] = wait_channel_scale(c - 1, out_scale, amax_bits,
                                          arrive + int64_t(c - 1) * 32, status, aborted);
      __syncthreads();
      sc = s_scale[par];
      if (amax_step) {  // 3
        for (; ka < cnt; ++ka, ++kb) {
          load_span(cur + wa.offset(K), wa.t0(), K, vec, xr, xi);
          load_span(prev + wb.offset(K), wb.t0(), K, vec, yr, yi, pol);
          amax_of(xr, xi);
          quantise_unit(yr, yi, sc, buf, zprev + wb.zoffset(zpitch), plane, neg);
          wa.next();
          wb.next();
        }
      }
    }
    if (amax_step) {  // 4
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((t & 31) == 0) wm[par][t >> 5] = m;
      __syncthreads();
      if (t == 0) {
        for (int x = 1; x < (bd >> 5); ++x) m = fmaxf(m, wm[par][x]);
        if (!(m == m)) m = 0.f;
        atomicMax(amax_bits + c, __float_as_uint(m));
        __threadfence();
        atomicAdd(arrive + int64_t(c) * 32, 1u);
      }
    }
    if (quant_step) {  // 5
      for (; kb + 1 < cnt; kb += 2) {
        UnitWalk w2 = wb;
        w2.next();
        load_span(prev + wb.offset(K), wb.t0(), K, vec, xr, xi, pol);
        load_span(prev + w2.offset(K), w2.t0(), K, vec, yr, yi, pol);
        quantise_unit(xr, xi, sc, buf, zprev + wb.zoffset(zpitch), plane, neg);
        quantise_unit(yr, yi, sc, buf, zprev + w2.zoffset(zpitch), plane, neg);
        w2.next();
        wb = w2;
      }
      if (kb < cnt) {
        load_span(prev + wb.offset(K), wb.t0(), K, vec, xr, xi, pol);
        quantise_unit(xr, xi, sc, buf, zprev + wb.zoffset(zpitch), plane, neg);
      }
    }
  }
}

// Blocks of scale_quantize_kernel per SM that can be resident (0: unknown).
int scale_quantize_blocks_per_sm() {
  static std::once_flag once;
  static int nb = 0;
  std::call_once(once, [] {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, scale_quantize_kernel, 256, 0) !=
        cudaSuccess) {
      nb = 0;
      cudaGetLastError();
    }
  });
  return nb;
}

}  // namespace

cudaError_t launch_channel_amax(const void* a, int64_t per_chan, int batch, uint32_t* amax_bits,
                                int sm_count, cudaStream_t s) {
  // about 8 blocks of 256 threads per SM over all channels, each thread with
  // at least 4 x 16-byte loads
  int bx = int((per_chan + 256 * 8 - 1) / (256 * 8));
  const int cap = (sm_count * 8 + batch - 1) / batch;
  if (bx > cap) bx = cap;
  if (bx < 1) bx = 1;
  const int vec = (per_chan % 2 == 0) && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  // one grid row per channel, as many launches as that takes (blocks that step
  // through the channels lose 7%: 83 against 77 us for 16 channels of 33.6 MB)
  constexpr int kMostRows = 65535;
  for (int c = 0; c < batch; c += kMostRows)
    amax_kernel<<<dim3(unsigned(bx), unsigned(std::min(batch - c, kMostRows))), 256, 0, s>>>(
        static_cast<const float2*>(a) + int64_t(c) * per_chan, per_chan, amax_bits + c, vec);
  return cudaGetLastError();
}

cudaError_t launch_float_to_planes(const void* a, uint8_t* z, int64_t rows, int K, int Kp,
                                   int zpitch, int n, int batch, int split, int neg,
                                   float* out_scale, uint32_t* amax_bits,
                                   uint32_t* arrive, uint32_t* status, int sm_count,
                                   cudaStream_t s) {
  // the arrival words (32 per channel) directly followed by amax_bits: one
  // memset zeroes both
  const bool adjacent = amax_bits == arrive + int64_t(batch) * 32;
  cudaError_t e = adjacent ? cudaMemsetAsync(arrive, 0, sizeof(uint32_t) * size_t(batch) * 33, s)
                           : cudaMemsetAsync(amax_bits, 0, sizeof(uint32_t) * size_t(batch), s);
  if (e != cudaSuccess) return e;
  const int vec = (K % 2 == 0) && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
  const int64_t units = int64_t(n) * (Kp >> 3);
  // The cooperative kernel takes a step per channel, each with a wait for the
  // whole grid, and saves the second read from HBM: it needs a channel that is
  // long against the wait, or a single one.  Promotion in us, cooperative / two
  // kernels: one channel of 1.2 MB 10.3 / 10.9, of 8.4 MB 12.4 / 12.7, of 33.6 MB
  // 18.5 / 21.0; 16 of 1.2 MB 49 / 16, of 4.2 MB 56 / 35; 4 of 8.4 MB 22 / 19, 16 of
  // them 67 / 66; 8 of 16.8 MB 57 / 68, of 22.9 MB 70 / 88; 16 of 33.6 MB 181 / 223.
  // So the two meet between 9 and 12 MB; the line at 24 MB is where they met before
  // either loaded whole spans (8 of 16.8 MB 76 / 71 then), and calls of 12 to 24
  // MB a channel run up to 16% above what the other choice gives.  The split mode
  // (hi and lo columns) was slower on it at any size: 1.02 against 0.91 ms at
  // 4096 x 64 x 1024.
  const bool large = batch == 1 || int64_t(n) * K * int64_t(sizeof(float2)) >= 24000000;
  const int per_sm = split || !large ? 0 : scale_quantize_blocks_per_sm();
  if (per_sm > 0 && adjacent && (reinterpret_cast<uintptr_t>(arrive) & 127) == 0 &&
      units < (int64_t(1) << 30)) {
    // at least 256 units (one per thread) per block, at most every resident block
    int64_t grid = (units + 255) / 256;
    if (grid > int64_t(per_sm) * sm_count) grid = int64_t(per_sm) * sm_count;
    if (grid < 1) grid = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, scale_quantize_kernel, static_cast<const float2*>(a), z, K, Kp,
                           zpitch, n, batch, neg, out_scale, amax_bits, arrive, status,
                           vec);
    if (e == cudaSuccess) return e;
    cudaGetLastError();  // not launchable as one cooperative grid: the two-kernel path
  }
  const int64_t per_chan = int64_t(n) * K;
  e = launch_channel_amax(a, per_chan, batch, amax_bits, sm_count, s);
  if (e != cudaSuccess) return e;
  const int rpb = promotion_rows_per_block(rows, Kp >> 3);
  const int64_t blocks = (rows + rpb - 1) / rpb;
  // An early start saves about 2 us: whole calls without / with it, 2 channels of
  // 1024 x 1024 26.6 / 24.4 us, 8 of them (the line, 8 M samples) 51.3 / 49.4, 16
  // 100.3 / 98.0, hi + lo 160.9 / 158.2; past the line the gain is below what runs
  // differ by (hi + lo, 16 channels of 4096 x 1024: 1451 / 1549, 32: 3023 / 3019).
  const bool early = rows * K <= (int64_t(8) << 20);
  e = launch_after(early, quantize_kernel, dim3(unsigned(blocks)), dim3(256), 0, s, static_cast<const float2*>(a), z, rows, K, Kp, zpitch, n, amax_bits, out_scale,
                   split, rpb, vec);
  if (e == cudaSuccess && neg) e = launch_negate_plane(z, rows * zpitch, sm_count, s);
  return e;
}

}  // namespace ftdx
