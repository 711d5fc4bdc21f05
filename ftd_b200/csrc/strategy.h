// strategy.h -- the launch strategy of a correlator call, the rules that pick it
// where the user has set none, the device memory that split-K needs, and the
// block size of the promotion passes.  Host code without CUDA headers.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ftdx {

constexpr int kTile = 128;    // antennas per operand tile (M = N = 128)
constexpr int kStageK = 128;  // samples per pipeline stage (= bytes per plane row)

constexpr int kStoreFp6 = 4;
constexpr int kStoreS8 = 8;   // with store mode 2: signed 8-bit operands, kind::i8 MMAs
constexpr int kStoreFused = 16;  // alone (mode 0 + 16): QC promotion fused into the single-CTA kernel
// Launch strategy of the correlator kernel; chosen by the autotuner.
struct Strategy {
  // 0: direct stores, 1: shared-memory staging + bulk copies,
  // 2: CTA-pair kernel (256 x 128 tiles on two SMs, direct stores);
  // 3: CTA-pair kernel with bulk-copy stores for interior tiles;
  // + kStoreFp6: operands as packed FP6 E3M2 planes (QC input, exact);
  // + kStoreS8 (pair only): signed 8-bit planes, integer MMAs (QC input, exact)
  // kStoreFused (alone): single CTA, direct stores, the QC bytes converted to
  // E4M3 inside the correlator (uniform INT4 calls; others run as 0)
  int store_mode = 0;
  int grid = 0;        // persistent CTAs (0: one per SM); -1: one CTA per tile (not persistent)
  int splits = 1;      // split-K: K is cut into this many ranges, partials summed afterwards
  bool operator==(const Strategy& o) const {
    return store_mode == o.store_mode && grid == o.grid && splits == o.splits;
  }
};

// Rows per block of a promotion pass over `rows` rows of `chunks` per-thread
// pieces: at most the eight blocks of 256 threads that each of 148 SMs holds at
// once, at most 32 pieces per thread (rows stay together, and fewer blocks
// start) and at least one.  Promotion in us:
//   one size of 8192 pieces / this: 32 channels of 128 x 256 (eight blocks
//   before) 16.9 / 6.6, 16 of 1024 x 1024 FP16 samples (256) 33.8 / 22.9;
//   rows rounded down, a few blocks more than fit at once / this: 16 of 3000 x
//   2048 (1200 blocks) 65.2 / 61.4, 40 of 700 x 2000 FP16 samples 68.5 / 60.8.
constexpr int kPromotionBlocks = 8 * 148;
inline int promotion_rows_per_block(int64_t rows, int chunks) {
  const int64_t most = 8192 / chunks, least = (256 + chunks - 1) / chunks;
  int64_t r = (rows + kPromotionBlocks - 1) / kPromotionBlocks;
  if (r < least) r = least;
  if (r > most) r = most;
  return r < 1 ? 1 : int(r);
}

// Split-K: the most ranges, and the most bytes of partial triangles that the
// rule below takes.
constexpr int kMostSplits = 32;
constexpr size_t kMostSplitBytes = 256000000;
inline size_t split_bytes(int N, int batch, int splits) {
  return size_t(splits) * size_t(batch) * size_t(int64_t(N) * (N + 1) / 2) * 8;
}

// Strategy of a call on a handle whose user has set none: the single-CTA
// kernel, with the promotion fused in or not and K split or not, whichever a
// small model of the device time puts first.  Its terms, in us, fitted to 54
// shapes of 1 to 2112 tiles and 2 to 512 k-blocks on 148 SMs (the pick is
// within 13% of the best split and kernel tried at each, most within 3%):
//   a tile of b k-blocks takes max(0.58 b, 2.2) + 0.6 -- the MMAs or the
//     stores, then the pipeline's fill; 0.95 b with the conversion fused in;
//   the separate promotion 2 for its launch + the planes' bytes at 5.5 TB/s;
//   split-K 3 for its reduction + the partial triangles at 3 TB/s.
// 256 inputs x 65536 samples x 4 channels (12 tiles): 333 us unsplit with the
// promotion apart, 56 us as 12 ranges with it fused in; 128 x 256 x 32: 12.6
// apart, 8.0 fused in; 1024 x 1024 x 16 (576 tiles): 41.1 apart, 43.5 fused in.
// The choice depends on sizes and on `fused` alone, so that a call prepared
// for capture (ftdx_init_herk) finds its plan.
// It also decides for FP16 and FP32 input and for hi + lo, whose promotion costs
// more and whose k-blocks take three products: it then splits too little, never
// where unsplit is faster.  Rule / best split / unsplit, us, promotion apart:
// FP16 128 x 2048 x 4 14.5 / 12.5 / 18.6, 256 x 16384 x 4 37.4 / 37.2 / 95.3; FP8 of
// floats 512 x 8192 x 1 28.9 / 28.9 / 55.6; hi + lo 300 x 1024 x 1 30.9 / 20.6 / 30.9,
// 256 x 4096 x 2 29.8 / 27.0 / 78.0, 512 x 8192 x 1 44.5 / 41.1 / 142.3.  Of 36 such
// shapes 28 are within 8% of the best; the others have at most six tiles, and the
// worst (hi + lo, one tile of 8 k-blocks) takes 28.8 us where 17.2 could be had.
inline Strategy auto_strategy(int sm_count, int N, int K, int batch, bool fused_ok,
                              bool split_ok) {
  const int64_t nb = (N + kTile - 1) / kTile, tiles = nb * (nb + 1) / 2 * batch;
  const int64_t kb = (int64_t(K) + kStageK - 1) / kStageK;
  const double planes = 3.0 * N * double(batch) * double(kb * kStageK);
  const double partial = double(split_bytes(N, batch, 1));
  Strategy best;
  // past eight tiles per SM the last round costs little and partials much
  const int64_t most = split_ok && tiles <= 8 * sm_count ? std::min<int64_t>(kMostSplits, kb) : 1;
  double best_us = 0;
  for (int sp = 1; sp <= int(most) && (sp == 1 || sp * partial <= kMostSplitBytes); ++sp) {
    const double b = double((kb + sp - 1) / sp);
    const double rounds = double((tiles * sp + sm_count - 1) / sm_count);
    const double sum = sp > 1 ? 3.0 + 0.1 * sp + sp * partial / 3e6 : 0.0;
    const double apart = 2.0 + planes / 5.5e6 + rounds * (std::max(0.58 * b, 2.2) + 0.6) + sum;
    const double in_one = rounds * (std::max(0.95 * b, 2.2) + 0.6) + sum;
    const bool f = fused_ok && in_one < apart;
    const double us = f ? in_one : apart;
    if (sp == 1 || us < best_us) {
      best = Strategy{f ? kStoreFused : 0, 0, sp};
      best_us = us;
    }
  }
  return best;
}

// NVFP4 without a strategy of the user's: the CTA pair where the operand bytes
// it saves per k-block outweigh its coarser tiles -- more than four blocks of 256
// inputs, four rounds of its tiles, four k-blocks (of 128 samples), and 40
// products of k-blocks per pair (hi + lo has three per k-block).  Single CTA /
// pair, us, 74 pairs, Gaussian voltages:
//   plain   2048 x 1024 x 8 (9 rounds of 8): 169 / 158; 4096 x 1024 x 2: 129 / 113;
//           1500 x 700 x 14 (9 of 6): 144 / 137; 1700 x 700 x 6 (5 of 6): 77 / 80;
//           2048 x 512 x 5 (5 of 4): 60 / 66; 4096 x 512 x 1 (4 of 4): 43 / 45;
//           2048 x 300 x 14 (16 of 3): 144 / 151;
//   hi + lo 2048 x 512 x 4 (4 of 4): 89 / 83; 1100 x 1024 x 19: 286 / 265;
//   up to 1024 inputs, both: 1024 x 512 x 16: 74 / 80 and 115 / 125; 512 x 1024
//           x 65: 204 / 206 and 311 / 327; 300 x 1024 x 97: 164 / 177 and 245 / 272.
// Of 374 shapes of 300 to 4096 inputs, both modes, none that takes the pair is
// more than 4% behind the single CTA.
inline Strategy fp4_strategy(int pairs, int N, int kblocks, int batch, bool split) {
  const int64_t nj = (N + 255) / 256, tiles = nj * (nj + 1) * 8 / 7 * batch;  // ~ of 256 x 112
  const int64_t work = tiles * kblocks * (split ? 3 : 1);
  const bool pair = pairs >= 1 && nj > 4 && tiles >= 4 * pairs && kblocks >= 4 && work >= 40 * pairs;
  return Strategy{pair ? 2 : 0, 0};
}

// The most bytes of partial triangles that auto_strategy takes for any shape up
// to (N, K, batch).  A smaller shape can take more than a larger one: on 148 SMs
// 512 inputs x 8192 samples take three ranges for 4 channels (12.6 MB) and seven
// for 2 (14.7 MB).
inline size_t most_split_bytes(int N, int K, int batch) {
  const int64_t kb = (int64_t(K) + kStageK - 1) / kStageK;
  const int sp = int(std::min<int64_t>(kMostSplits, kb));
  return sp > 1 ? std::min(kMostSplitBytes, split_bytes(N, batch, sp)) : 0;
}

// The rule's choice where have(splits) says whether the partial triangles and
// the tile plan of that many ranges are there or can be had; else unsplit.
template <typename Have>
Strategy untuned_choice(int sm_count, int N, int K, int batch, bool fused_ok, bool split_ok,
                        Have have) {
  const Strategy s = auto_strategy(sm_count, N, K, batch, fused_ok, split_ok);
  if (s.splits <= 1 || have(s.splits)) return s;
  return auto_strategy(sm_count, N, K, batch, fused_ok, false);
}

// Device memory of the partial triangles, grown on demand.  A buffer that a
// caller's graph was captured with is not freed when a larger one replaces it,
// since every replay of that graph writes to it: it stays until release().
struct Partials {
  uint8_t* ptr = nullptr;
  size_t cap = 0;
  bool captured = false;       // a caller's capture holds ptr
  std::vector<uint8_t*> held;  // replaced buffers that captures hold
  size_t refused = 0;          // the least size that there was no memory for (0: none)

  // alloc(bytes) returns nullptr on failure; drop(p) waits for p's users and
  // frees it.  False: not enough memory, and what was there is there again.
  template <typename Alloc, typename Drop>
  bool grow(size_t bytes, Alloc alloc, Drop drop) {
    if (bytes <= cap) return true;
    const bool ok = replace(bytes, alloc, drop);
    if (!ok)
      refused = refused ? std::min(refused, bytes) : bytes;
    else if (refused && bytes >= refused)
      refused = 0;
    return ok;
  }

  // A size that was refused before is not asked for again until release() or
  // until `refused` is cleared: each try would cost a failing allocation.
  bool hopeless(size_t bytes) const { return bytes > cap && refused && bytes >= refused; }

  template <typename Alloc, typename Drop>
  bool replace(size_t bytes, Alloc alloc, Drop drop) {
    uint8_t* p = nullptr;
    if (captured) {
      // half as large again, so that all that is held stays below twice the
      // last buffer, whatever the order of calls and captures
      size_t n = std::max(bytes, cap + cap / 2);
      p = alloc(n);
      if (!p && n > bytes) p = alloc(n = bytes);
      if (!p) return false;
      held.push_back(ptr);
      bytes = n;
    } else {
      if (ptr) drop(ptr);
      ptr = nullptr;
      p = alloc(bytes);
      if (!p) {
        if (cap) ptr = alloc(cap);
        if (!ptr) cap = 0;
        return false;
      }
    }
    ptr = p;
    cap = bytes;
    captured = false;
    return true;
  }

  template <typename Free>
  void release(Free free) {
    if (ptr) free(ptr);
    for (uint8_t* p : held) free(p);
    *this = Partials{};
  }
};

}  // namespace ftdx
