// Token tiles and K slices of the weight-stationary matmul (host arithmetic only).
#pragma once
#include <cstdint>

namespace b200 {

constexpr int kWsMaxNB = 192;                  // batch columns of a token tile (UMMA N), multiple of 16
constexpr int kWsSpanBytes = 128 * 128 + 128 * 16;   // packed words and scales of 256 k of a row tile

struct WsSplit {
  int nb;       // rows of x per token tile, a multiple of 16
  int ksplit;   // K slices = CTAs per cluster
  int tried;    // combinations looked at
};

// A model of the time in nanoseconds, fitted to measurements at N = 4096, 12288 and 22016,
// K = 4096 and 11008 and batches of 16, 64 and 128, and at 129..2048 tokens.  A 256-k span takes a CTA 0.53-0.65 us (up
// to 128 columns) or 0.9-0.95 us; with many CTAs at work, what they fetch from L2 at about 14 TB/s if that is more.
// Draining a tile is cheap with one slice (stores to y, behind the next tile's MMAs) and costs the exchange of the
// partial tiles with several, which the next tile hides only as far as its own MMAs last; a larger cluster starts
// later, unless (one token tile, four or eight CTAs) the clusters at work leave room for as many again: the set-up of a
// launch then runs beside the launch before it; in part for more than four clusters of eight.  Where one round of up to 128 rows fills the
// GPU, the next launch's clusters start later still: without that, 16 x 4096 x 2080 took four slices, 6.9 us where two take 5.3, 64 x 8192 x 2080
// two, 9.5 / 8.4.  Above 128 rows clusters have to be ahead by 1.5 %: 777 x 12288 x 7168 took two slices for less, 136 / 114.  Chosen / best of the slices
// with these two, over 1470 shapes of up to 128 rows 1.011 -> 1.008 on average and over 720 above 1.006 -> 1.0055, on a GPU that holds 74, 33 and 15 clusters at once
// (a number that differs from GPU to GPU: 36 and 16 were seen too).  Measured first: M = 64, K = 4096, 1 / 2 / 4 / 8 slices: N = 4096 11.0 / 8.7 / 9.0 / 10.8 us, N = 12288 12.9 / 14.3 / 15.6 / 23.2,
// N = 22016 22.1 / 20.5 / 24.0 / 40.3; N = 4096 and K = 11008: 26.4 / 16.4 / 13.5 / 14.6.  M = 300, N = 12288, K = 4096 in 2 / 3 / 4
// token tiles: 31.7 / 29.5 / 34.8.  Few row tiles, M = 64, K = 2048, N = 512: 6.7 / 6.3 / 5.1 / 4.9, N = 1024: 6.7 / 6.3 / 5.2 / 5.8,
// N = 2048: 6.8 / 6.5 / 5.1 / 7.3; N = 1024, K = 8192: 20.0 / 13.0 / 8.4 / 7.6.
// M rows of x, row_tiles tiles of 128 weight rows, units spans of 256 k; forced: the largest power of two of slices up to
// it (0 = by the model); clusters[i]: clusters of 2^i CTAs that run at once.  Every width of a token tile is looked at
// once, so at most 12 x 4 combinations whatever M is.
inline WsSplit choose_ws_split(int64_t M, int64_t row_tiles, int units, int forced, const int (&clusters)[4]) {
  constexpr int64_t kStart[4] = {0, 500, 1000, 3500}, kCrowd[4] = {0, 500, 2400, 0};
  WsSplit best = {0, 1, 0};
  int64_t best_cost = 0;
  const int64_t mt0 = (M + kWsMaxNB - 1) / kWsMaxNB;
  // (up to 128 rows the weights stream once: one token tile)
  const int64_t mt_max = M <= 128 ? 1 : mt0 + mt0 / 2 + 3;
  for (int nb = M < kWsMaxNB ? (int)((M + 15) / 16) * 16 : kWsMaxNB; nb >= 16; nb -= 16) {
    const int64_t mt = (M + nb - 1) / nb;
    if (mt > mt_max) break;
    if (((M + mt - 1) / mt + 15) / 16 * 16 != nb) continue;      // as many token tiles of fewer columns do it
    const int64_t tiles = row_tiles * mt;
    for (int i = 0, c = 1; i < 4 && c <= units; ++i, c *= 2) {
      if (forced > 0 && !(c <= forced && (c * 2 > forced || c * 2 > units || c == 8))) continue;
      const int64_t rounds = (tiles + clusters[i] - 1) / clusters[i];
      const int64_t busy = tiles * c / rounds;                                   // CTAs at work, on average
      const int64_t l2 = busy * (nb * 512 + kWsSpanBytes) / 14000;
      const int64_t span = nb <= 128 ? 520 + nb : 760 + nb;
      const int64_t tile = (int64_t)((units + c - 1) / c) * (span > l2 ? span : l2);   // a tile's MMAs
      const int64_t drain = c == 1 ? 300 + 12 * nb : 800 + 50 * nb;              // ... and what the next tile must hide
      const bool room = M <= 128 && c >= 4 && 2 * tiles <= clusters[i] + (c == 8 ? 2 : 0);
      const int64_t tail = c == 1 ? drain : room ? 900 + 38 * nb : 600 + 35 * nb;   // the last tile's drain
      int64_t start = room ? (c == 8 && tiles > 4 ? 1600 - 8 * nb : 0) : kStart[i];
      if (M <= 128 && rounds == 1 && !room && 2 * tiles > clusters[i]) {
        const int64_t crowd = kCrowd[i] * (2 * tiles - clusters[i]) / clusters[i];          // of the next launch's clusters, those without a place
        start = c == 4 ? (crowd > start ? crowd : start) : start + crowd;
      }
      int64_t cost = start + tile + (rounds - 1) * (tile > drain ? tile : drain) + tail;
      if (M > 128 && c > 1) cost += cost * 15 / 1000;
      ++best.tried;
      if (best_cost == 0 || cost < best_cost) { best_cost = cost; best.ksplit = c; best.nb = nb; }
    }
  }
  return best;
}

// Whether the prefill kernel's 256 x 256 tiles suit a prompt better.  One wave of them takes a long K as long as three rounds of
// wide token tiles here, so where these leave more of their last round empty than its wave leaves of the SMs, it is
// ahead: this kernel / the prefill kernel in us, M x N x K 2048 x 4096 x 8192 104.0 / 103.8, 2048 x 4096 x 11008 142 / 134,
// 4096 x 2048 x 8192 114 / 111, 4096 x 2048 x 11008 154 / 140, 8192 x 1024 x 8192 126 / 113; with equal shares or a shorter K it is
// not: 1024 x 8192 x 8192 104 / 105, 2048 x 4096 x 4096 53 / 56, 4096 x 2048 x 4096 54 / 57.
inline bool prefill_kernel_is_ahead(int64_t M, int64_t N, int64_t K, const WsSplit& split, int64_t row_tiles, int sms) {
  if (K < 8192 || split.nb < 160 || split.ksplit != 1) return false;
  const int64_t wave = ((M + 255) / 256) * ((N + 255) / 256);
  const int64_t tiles = row_tiles * ((M + split.nb - 1) / split.nb);
  const int64_t rounds = (tiles + sms - 1) / sms;
  return wave <= sms && rounds >= 3 && 100 * wave * rounds > 100 * tiles + 3 * rounds * sms;
}

}  // namespace b200
