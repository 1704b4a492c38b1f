// Which of two attention kernels a call's sizes ask for.  Plain functions of sizes, so that they can be held against the measured times of both.
#pragma once

namespace umb {

inline long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

// A decode step's grouped attention, unsplit (seq/seq_cached_attn.cu): blocks of six warps instead of four.  A round of six warps takes 192 keys instead of 128, but two
// such blocks fit on an SM instead of three: what counts is waves of blocks times rounds, a wave's first and last round as one more, with 5 % to spare.  us, four warps /
// six, 16 heads over 4 of 128, keys 200, 300, 1200: 64 sequences (256 blocks) 14 / 15, 19 / 16, 48 / 41; 100 (400 blocks, one wave / two) 16 / 28,
// 21 / 26, 57 / 78; 128 (two / two) 27 / 28, 38 / 30, 98 / 78; 256 (three / four) 46 / 58, 59 / 59, 150 / 151.
inline bool six_warps_pay(long long blocks, int keys, int sms) {
    const long long waves4 = ceil_div(blocks, 3ll * sms), waves6 = ceil_div(blocks, 2ll * sms), rounds4 = ceil_div(keys, 128), rounds6 = ceil_div(keys, 192);
    return blocks >= sms && 21 * waves6 * (rounds6 + 1) < 20 * waves4 * (rounds4 + 1);
}

}  // namespace umb
