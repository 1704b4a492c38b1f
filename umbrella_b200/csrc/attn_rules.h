// Which of two attention kernels a call's sizes ask for.  Plain functions of sizes, so that they can be held against the measured times of both.
#pragma once

namespace umb {

inline long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

// Attention of many query rows under a causal or tree mask (attn.cu): tiles of 64 flattened rows (of a key/value head's group) instead of slabs of 16, whose
// rounds each fetch all keys again.
//
// Heads of 128: from 128 tiles on, where a fit of both kernels' times says so with 5 % to spare.  A slab's round of the SMs takes
// 5.1 us and 6.7 ns a key; a tile 22 ns a key, of which two share an SM at half the speed, so that what counts is one round of tiles (up to one an SM) or pairs of rounds (from
// then on in steps of two an SM: 152 to 296 tiles take as long as 296).  us, slabs / tiles, 32 heads over 8, causal: 256 rows 18 / 15, behind 7000 205 / 173; 300
// rows (152 tiles) 28 / 17, behind 1500 76 / 83 and 7000 253 / 320; 520 rows (264) 51 / 29, behind 7000 410 / 332; 600 rows (304) 60 / 33, behind 7000
// 459 / 546.  Trees also read their mask a word at a time, tile by tile: 800 nodes behind 500 163 / 170.  Of 979 measured calls the rule takes
// tiles for 530, which are between 0.99 and 2.6 times as fast as slabs, 1.27 times in the mean.
//
// Heads of 64: a slab's round costs half as much and a tile's key nearly the same, so only causal prompts without much behind them gain, from four heads to a
// key/value head on: 300 rows 17 / 12, behind 150 19 / 16, behind 450 24 / 24, behind 7000 (384 rows) 175 / 265; up to 256 keys the slabs run on four
// warps and are as fast (180 rows, 64 heads over 8: 8.9 / 9.6).
//
// Dense masks are read a byte at a time, by one thread per row of a tile: 300 rows behind 2000 235 / 387.
constexpr int kMaskCausal = 2, kMaskTree = 0;               // UMB_MASK_*
inline bool row_tiles_pay(int mask_mode, int rows, int keys, int heads, int kv_heads, int head_dim, int sms) {
    const long long flat = (long long)rows * (heads / kv_heads), tiles = ceil_div(flat, 64) * kv_heads, slabs = ceil_div(flat, 16) * kv_heads;
    if (mask_mode != kMaskCausal && mask_mode != kMaskTree) return false;
    if (head_dim == 64) return mask_mode == kMaskCausal && heads >= 4 * kv_heads && tiles > sms && keys > 256 && 2ll * keys <= 3ll * rows;
    if (head_dim != 128 || tiles < 128) return false;
    const double slab_rounds = (double)ceil_div(slabs, sms), tile_rounds = tiles <= sms ? 1. : 2. * ceil_div(tiles, 2ll * sms);
    const double seen = mask_mode == kMaskCausal ? keys - 0.5 * rows : keys;                   // keys of a row, in the mean
    const double by_slabs = slab_rounds * (5.1 + 0.0067 * seen) - 1.6;
    const double by_tiles = mask_mode == kMaskCausal ? 14.7 + tile_rounds * (0.022 * seen - 0.5)
                                                     : 24.6 + tile_rounds * (0.0214 * seen + 24e-6 * rows * rows - 6.8);
    return by_slabs > 1.05 * by_tiles;
}

// A decode step's grouped attention, unsplit (seq/seq_cached_attn.cu): blocks of six warps instead of four.  A round of six warps takes 192 keys instead of 128, but two
// such blocks fit on an SM instead of three: what counts is waves of blocks times rounds, a wave's first and last round as one more, with 5 % to spare.  us, four warps /
// six, 16 heads over 4 of 128, keys 200, 300, 1200: 64 sequences (256 blocks) 14 / 15, 19 / 16, 48 / 41; 100 (400 blocks, one wave / two) 16 / 28,
// 21 / 26, 57 / 78; 128 (two / two) 27 / 28, 38 / 30, 98 / 78; 256 (three / four) 46 / 58, 59 / 59, 150 / 151.
inline bool six_warps_pay(long long blocks, int keys, int sms) {
    const long long waves4 = ceil_div(blocks, 3ll * sms), waves6 = ceil_div(blocks, 2ll * sms), rounds4 = ceil_div(keys, 128), rounds6 = ceil_div(keys, 192);
    return blocks >= sms && 21 * waves6 * (rounds6 + 1) < 20 * waves4 * (rounds4 + 1);
}

}  // namespace umb
