// Which tiles the products of a token block take on persistent CTAs (umma_kernel, seq_gemm_umma.cuh); host code only.
#pragma once

namespace kllm {
namespace seq {
namespace umma {

constexpr int kSms = 148;
enum TileForm {
  kNarrow,  // 128 weight rows x 128 tokens, a CTA
  kWide,    // 128 x 256, a CTA
  kPair     // 256 x 256, two CTAs
};
struct TileWaves {  // times that the chip takes tiles of each form until all are done
  int narrow, wide, pair;
};
// N: weight rows, or gated features (a CTA's 128 rows are 64 gate rows and their 64 up rows)
inline TileWaves tile_waves(bool gated, int T, int N) {
  const int features = gated ? (N + 63) / 64 : (N + 127) / 128, tokens = (T + 255) / 256;
  return TileWaves{(features * ((T + 127) / 128) + kSms - 1) / kSms, (features * tokens + kSms - 1) / kSms,
                   ((features + 1) / 2 * tokens + kSms / 2 - 1) / (kSms / 2)};
}
// Measured with every form at 40 shapes from 900 to 6001 tokens and 4 to 6 lengths of K, bf16 and TF32 (a block of K is 128 bytes of a
// row, 64 bf16 values).  us, wide / pair / narrow:
//   plain, 32 blocks   one wide wave 21.2 / 23.2 / 29.3 (2048 x 2048); two 33.3 / 33.9 / 39.3 (2048 x 3072), 35.3 / 34.4 / 49.9 (x 4352);
//                      three 50.3 / 45.7 / 72.1 (x 6144); five 75.7 / 69.1 / 102.6 (6001 x 3456)
//   plain, 16 blocks   one 15.3 / 17.3 / 19.4; two 23.1 / 23.2 / 25.3; three 31.1 / 30.0 / 41.6
//   plain, 8 blocks    one 14.5 / 16.2 / 16.3; two 18.5 / 20.4 / 18.8; three 23.3 / 24.0 / 27.2; five 33.7 / 33.9 / 37.2
//   a pair too many    an odd number of feature tiles can cost pairs a wave more: 900 x 4736 21.5 / 33.4 / 29.5 (32 blocks), 33.2 / 53.8 /
//                      49.8 (64), 2048 x 4736 35.5 / 45.7 / 50.1
//   all narrow tiles at once    520 x 3072: - / 18.6 / 16.5 (32 blocks), - / 32.9 / 30.2 (64)
//   gated, 8 to 32     the way out of a tile bounds it, and a pair's CTAs wait for one another: one 33.7 / 35.6 / 38.9 (2048 x 1024, 32 blocks),
//                      eleven 232 / 244 / 266 (6001 x 4096); two and three 54.3 / 50.9 / 51.0 (2048 x 1536), 79.1 / 75.4 / 88.1 (x 3328);
//                      16 blocks 47.8 / 45.4 / 40.5 (x 1536), 103.9 / 108.7 / 99.5 (6001 x 1728)
//   gated, 64 blocks   one 48.0 / 48.9 / 64.3; two 71.8 / 68.7 / 86.1; five 147 / 142 / 215
inline TileForm tile_form(bool gated, int T, int N, int kblocks) {
  const TileWaves w = tile_waves(gated, T, N);
  // a narrow tile takes this many hundredths of a wide one's time
  const int narrow = gated ? (kblocks <= 16 ? 55 : kblocks < 48 ? 70 : 80) : (kblocks < 16 ? 70 : 80);
  if (100 * w.wide > narrow * w.narrow) return kNarrow;
  if (w.wide == 1 || w.pair > w.wide) return kWide;
  if (gated) return kblocks >= 64 || w.wide <= 3 ? kPair : kWide;
  return kblocks >= (w.wide == 2 ? 32 : 16) ? kPair : kWide;
}

}  // namespace umma
}  // namespace seq
}  // namespace kllm
