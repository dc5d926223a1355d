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
// to 128 columns) or 0.9-0.95 us; with many CTAs at work, what they fetch from L2 at about 14 TB/s (13 in clusters) if that is more.
// Draining a tile is cheap with one slice (stores to y, behind the next tile's MMAs) and costs the exchange of the
// partial tiles with several, which the next tile hides only as far as its own MMAs last.  A larger cluster starts
// later: up to 128 rows by as much as the clusters of the last round leave too little room for the first ones of the next launch, whose
// set-up runs beside them where there is room (in part for more than four clusters of eight).  One figure for every
// launch without room made 16 x 4096 x 2080 take four slices, 6.8 us where two take 5.2, and 96 x 8192 x 2560 two, 9.8 / 8.8; above 128 rows
// 777 x 12288 x 7168 took two, 135 / 111.  Chosen / best of the slices over 2200 shapes on a GPU that holds 74, 33 and 15 clusters
// at once, up to 128 rows 1.012 -> 1.0045 on average and at most 1.31 -> 1.15, above 1.006 -> 1.004.  (That number differs from GPU to GPU: 36 and 16
// were seen too.)  Measured first: M = 64, K = 4096, 1 / 2 / 4 / 8 slices: N = 4096 11.0 / 8.7 / 9.0 / 10.8 us, N = 12288 12.9 / 14.3 / 15.6 / 23.2,
// N = 22016 22.1 / 20.5 / 24.0 / 40.3; N = 4096 and K = 11008: 26.4 / 16.4 / 13.5 / 14.6.  M = 300, N = 12288, K = 4096 in 2 / 3 / 4
// token tiles: 31.7 / 29.5 / 34.8.  Few row tiles, M = 64, K = 2048, N = 512: 6.7 / 6.3 / 5.1 / 4.9, N = 1024: 6.7 / 6.3 / 5.2 / 5.8,
// N = 2048: 6.8 / 6.5 / 5.1 / 7.3; N = 1024, K = 8192: 20.0 / 13.0 / 8.4 / 7.6.
// M rows of x, row_tiles tiles of 128 weight rows, units spans of 256 k; forced: the largest power of two of slices up to
// it (0 = by the model); clusters[i]: clusters of 2^i CTAs that run at once.  Every width of a token tile is looked at
// once, so at most 12 x 4 combinations whatever M is.
inline WsSplit choose_ws_split(int64_t M, int64_t row_tiles, int units, int forced, const int (&clusters)[4]) {
  constexpr int64_t kStart[4] = {0, 500, 0, 3000}, kCrowdedStart[4] = {0, 2000, 2400, 1300};     // up to 128 rows; more where there is no room at all
  constexpr int64_t kManyRowsStart[4] = {0, 0, 600, 1900};
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
      const int64_t l2 = busy * (nb * 512 + kWsSpanBytes) / (c == 1 ? 14000 : 13000);
      const int64_t span = nb <= 128 ? 520 + nb : 760 + nb;
      const int64_t tile = (int64_t)((units + c - 1) / c) * (span > l2 ? span : l2);   // a tile's MMAs
      const int64_t drain = c == 1 ? 300 + 12 * nb : 800 + 50 * nb;              // ... and what the next tile must hide
      // clusters of the next launch's first round that find no place beside this one's last
      const int64_t all = clusters[i], excess = tiles - (rounds - 1) * all + (tiles < all ? tiles : all) - all - (c == 8 ? 2 : 0);
      const int64_t crowd = excess > 0 ? excess : 0;
      const bool room = M <= 128 && c >= 4 && rounds == 1 && crowd == 0;
      const int64_t tail = c == 1 ? drain : room ? 900 + 38 * nb : (M <= 128 ? 300 + 38 * nb : 400 + 35 * nb);   // the last tile's drain
      const int64_t start = M > 128 ? kManyRowsStart[i] : room ? (c == 8 && tiles > 4 ? 1600 - 8 * nb : 0)
                                                               : kStart[i] + kCrowdedStart[i] * crowd / all;
      const int64_t cost = start + tile + (rounds - 1) * (tile > drain ? tile : drain) + tail;
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
