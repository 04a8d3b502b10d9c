// How a launch of attn_decode.cuh is split over CTAs and warps.  Plain C++, so that the rules can be compiled and checked on the
// host.
#pragma once
#include <cstdint>

namespace b200 {

constexpr int kDecodeMaxCluster = 16;
constexpr int kDecodePortableCluster = 8;

// CTAs per unit and warps per CTA.  One eight-warp CTA (192 KB of ring: one per SM) streams 86 GB/s, so 76 of them saturate
// the HBM; a unit is therefore split by the largest power of two that keeps the launch within one CTA per SM -- every CTA
// resident, no second wave, no merge that is not needed -- with at least two 16-key tiles for every warp.  Measured
// (head_dim 128, us; the choice in brackets):  128 units x 512 keys: [1 CTA, 8 warps: 7.0], 2 x 4 warps 8.0;  64 x 8192:
// [2 x 8: 41.9], 4 x 4: 42.4, 1 x 8: 51.8;  40 x 12195: [2 x 8: 40.9], 4 x 4: 42.3;  10 x 2729: [8 x 8: 7.1], 16 x 4: 7.7.
// Clusters above the portable size of 8 need a whole GPC each, and more than four of them queue (8 x 16384: [8 x 8: 18.3],
// 16 x 8: 24.7;  2 x 16384: 8 x 8: 17.5, [16 x 8: 11.7]).
// More units than SMs: one four-warp CTA per unit, two per SM.
//
// A unit's keys are merged in the order that this split gives, so the last bits of its result depend on how many units the
// launch has.  An order that is a function of the unit alone -- the keys in up to 128 leaves, merged pairwise in a tree, of
// which a warp takes as many as the launch asks for -- was built: the same bits for every split, but a warp has to keep the
// partial results that wait for their partner (in local memory: shared memory is full of the ring), and every doubling of its
// leaves costs 4 to 6 % (64 units x 8192 keys, 1 / 2 / 4 / 8 leaves per warp: 41.7 / 43.8 / 46.2 / 48.4 us; with 16 query rows
// 43.3 ... 56.8; 512 units x 4096 keys, 1 ... 32 leaves: 150 ... 197).  One split for every number of units costs 1.3 to 5 times.
struct DecodeSplit {
  int ctas;
  bool wide;   // eight warps per CTA (head_dim 128; four at 256), else half of that
};
inline DecodeSplit decode_split(int64_t units, int n_tiles, int sms) {
  if (units > sms) return {1, false};
  const int most = units <= 4 ? kDecodeMaxCluster : kDecodePortableCluster;
  int c = 1;
  while (2 * c <= most && 2 * c * units <= sms && n_tiles >= 32 * c) c *= 2;
  return {c, n_tiles > 8 * c};
}

// `placeable` is how many clusters of that size the device holds at once: none where no GPC has as many free SMs (a partitioned
// device), and fewer than units means a second wave.
inline int decode_cluster_that_fits(int ctas, int64_t units, int placeable) {
  return ctas > kDecodePortableCluster && placeable < units ? kDecodePortableCluster : ctas;
}

}  // namespace b200
