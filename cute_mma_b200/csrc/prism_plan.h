// Launch plans that follow from sizes alone: tile widths of the forward and dB.  Host code without CUDA, so that the rules can
// be called where there is no GPU.
#pragma once

namespace prism {

// Widest n-tile of a group: the largest multiple of 32 up to 256 that divides group_size, or 16; 0 where there is none.  A
// narrow tile reloads A and repeats the rotation and the gate for every tile of the group.
// Measured against the powers of two used before, 2000 x 3000 -> 6144 with groups of 192 (64 -> 192 wide): forward 218 ->
// 92 us, dB 323 -> 134 us; 1000 x 1000 -> 1440 with groups of 96 (32 -> 96): 31 -> 17 and 40 -> 16 us.  Widths that are
// multiples of 16 only are left at 16.
inline int default_bn(int gs) {
  for (int c = 256; c >= 32; c -= 32)
    if (gs % c == 0) return c;
  return gs % 16 == 0 ? 16 : 0;
}

// Widest power of two up to 256 that divides group_size (a multiple of 16).
inline int pow2_bn(int gs) {
  int bn = 256;
  while (gs % bn != 0) bn /= 2;
  return bn;
}

inline long long fwd_tiles(int M, int N, int bn) { return (long long)((M + 255) / 256) * (N / bn); }

// Estimated time (us) of the general forward with tiles of bn columns: waves of CTA pairs x (64-wide chunks of K x the time of
// one + epilogue).  A chunk takes 0.41 us at 64 columns, 0.44 at 128, 0.48 at 192 and 0.57 at 256; the epilogue 0.007 us a
// column by TMA stores (multiples of 64), 0.0145 by plain ones, and 0.010 and 0.034 with a bias, which only the former
// stages in shared memory (waves of 74 tiles of 256 rows, 2 to 32 chunks).
inline double fwd_tile_us(int M, int N, int K, int bn, bool bias, int pairs) {
  const double w = bn / 256.0;
  const double epilogue = bn % 64 == 0 ? (bias ? 0.010 : 0.007) * bn : (bias ? 0.034 : 0.0145) * bn;
  return (double)((fwd_tiles(M, N, bn) + pairs - 1) / pairs) * ((K + 63) / 64 * (0.40 + 0.17 * w * w) + epilogue);
}

// n-tile of the general forward.  A narrow tile repeats its group's rotation and gate, but on a CTA pair that would be idle,
// and its epilogue is shorter.
// Groups whose widest tile is a power of two: that tile, halved (down to 64) as long as the narrower tiles still run in one
// wave.  Measured, 256 against 64 wide: 1024 x 256 -> 1024 8.9 / 7.1 us, 1024 x 768 -> 768 12.8 / 10.7; 200 x 4096 -> 1024
// 32.6 / 30.4; 32 wide is no faster (8.8, 15.7, 30.3), and two waves lose (128 x 4096 -> 14336: 36.7 / 104.9).
// Other groups (96, 160, 192, 224, ...): of the widest tile, the widest power of two and the multiples of 64 between, the
// one with the least estimated time, the wider of two within 3 %.  The widest alone lost to the powers of two in short calls,
// the more so with a bias: 207 x 496 -> 448 with groups of 224, 224 / 32 wide 11.8 / 8.5 us, with a bias 15.2 / 9.0; 300 x 1024 -> 768 with
// groups of 192, 96 / 64 wide 13.7 / 12.2 us with a bias.  Over 600 drawn shapes with and without a bias the rule takes 0.4 %
// longer than the best width in the mean; the widest tile halved to fit took 5.8 %, powers of two 26 %.
inline int fwd_default_bn(int M, int N, int K, int gs, bool bias, int sms) {
  const int pairs = sms / 2 > 0 ? sms / 2 : 1;
  const int widest = default_bn(gs), pow2 = pow2_bn(gs);
  int best = widest;
  if (widest == pow2) {
    while (best >= 128 && fwd_tiles(M, N, best / 2) <= pairs) best /= 2;
    return best;
  }
  double best_us = fwd_tile_us(M, N, K, widest, bias, pairs);
  for (int c = widest - 32; c >= 16; c -= 16) {
    if (gs % c != 0 || (c % 64 != 0 && c != pow2)) continue;
    const double us = fwd_tile_us(M, N, K, c, bias, pairs);
    if (us < 0.97 * best_us) { best = c; best_us = us; }
  }
  return best;
}

// Whether the general forward widens rotations of 8 itself or gets a widened copy of R from a launch before it (about 2 us,
// and its host time): itself where a CTA pair has few chunks of 64 features to go through.  Measured, copy against
// itself: 4 chunks 10.3 -> 9.1 us, 12 chunks 12.7 -> 11.9, 16 chunks 14.5 -> 13.9; 132 chunks (plain mode) 80 -> 78-81;
// 448 chunks 269 -> 318, 448 of a deeper layer 228 -> 303.
inline bool fwd_widens(int M, int N, int K, int bn, int sms) {
  const long long tiles = fwd_tiles(M, N, bn), pairs = sms / 2 > 0 ? sms / 2 : 1;
  return (tiles + pairs - 1) / pairs * ((K + 63) / 64) <= 32;
}

// Launch plan of the dB kernel: tile width, and how the token range of the tiles is split.
struct DbPlan {
  int bn;           // outputs per tile
  int splits;       // token-range splits of every tile (1: none)
  int tail_rows;    // n-tile rows of a mostly empty last wave that go to a second launch (0: none) ...
  int tail_splits;  // ... with their token range split this often
};

inline int db_tokblocks(int M) { return M > 128 ? (M - 1) / 128 + 1 : 1; }

// Estimated time (us) of one launch over `rows` n-tile rows: waves of CTA pairs x (token blocks x the time of one + a pair's
// start and epilogue).  A block of 128 tokens takes 0.97 us up to 128 outputs a tile, 1.15 at 192, 1.30 at 256; start and
// epilogue 4.4 us at 16 outputs, 5.8 at 256 (74 to 444 tiles, 1 to 64 blocks; rotations of 8 to 32 and both 16-bit types
// alike, rotations of 64 up to 11 % longer).  A split launch has its sum after it, with the fp32 partial sums written and read
// once: 10 TB/s while they stay in L2, 6.4 from memory.
inline double db_launch_us(int M, int K, int rows, int bn, int splits, int pairs) {
  const int tokblocks = db_tokblocks(M);
  const int per = (tokblocks + splits - 1) / splits;
  splits = (tokblocks + per - 1) / per;   // splits that would own no token block are dropped
  const long long tiles = (long long)((K + 255) / 256) * rows * splits;
  const double block = 0.97 + (bn > 128 ? 0.0026 * (bn - 128) : 0.0);
  double us = (double)((tiles + pairs - 1) / pairs) * (per * block + 4.3 + 0.006 * bn) + 1.0;
  if (splits > 1) {
    const double bytes = 8.0 * splits * rows * bn * K;
    us += 2.0 + 0.1 * splits + bytes / (bytes < 64e6 ? 10e6 : 6.4e6);
  }
  return us;
}

// The last wave's n-tile rows and their splits, where that wave is at most half full and another launch can fill it.
inline bool db_tail(int M, int N, int K, int bn, int pairs, int* tail_rows, int* tail_splits) {
  const int x_pairs = (K + 255) / 256, rows = N / bn, tokblocks = db_tokblocks(M);
  const int tiles = x_pairs * rows, tail = tiles % pairs;
  if (tiles <= pairs || tail == 0 || 2 * tail > pairs) return false;
  const int yb = (tail + x_pairs - 1) / x_pairs;
  int sb = pairs / (yb * x_pairs);
  if (sb > 16) sb = 16;
  if (sb > tokblocks) sb = tokblocks;
  if (sb < 2 || yb >= rows) return false;
  *tail_rows = yb;
  *tail_splits = sb;
  return true;
}

// Whether an unsplit 16-bit tile of bn outputs and `blocks` token blocks leaves by the instances that store by TMA: their
// epilogue is shorter, by 1.3 us at 256 outputs and nothing to speak of at 32.  `bf16_silu`: the bf16 silu instances with
// reconn_sz 16 and above, whose TMA form takes 1.5 to 4 % longer a block.  Measured, plain / TMA, one wave: 1 block of 256
// outputs 12.1 / 10.4 us; bf16 silu 64 blocks of 256 88.0 / 88.5, of 64 67.1 / 69.2; sigmoid 86.5 / 85.2 and 63.9 / 63.3; fp16
// silu 0.984 and 0.988 of the plain time.
inline bool db_tma_out(int bn, int blocks, bool bf16_silu) {
  return bf16_silu ? 1600ll * blocks <= (long long)bn * bn : bn >= 32;
}

// cfg = {bn, splits} or null, 0 = default; splits > 0 splits the token range of every tile, splits < 0 never splits.
// Default: the plan with the least estimated time of no splits, 2 to 16 splits of every tile, and splits of the rows of a mostly
// empty last wave only, each with the widest tile and with the widest power of two that divides the group.
// Over 500 timed shapes (16 to 512 outputs a group, both widths, up to 12 plans each) the rule is 0.2 % above the best plan in
// the mean.  Two rules before it: splits until the tiles fill the GPU twice, powers of two (59 % above); the widest tile and one
// time for a block of any width, tails not compared with splits of everything (3 %, up to 29 %: 10031 x 1728 -> 2816, groups of
// 64, 473 us split against 413 with a split tail).
inline void db_plan(int M, int N, int K, int gs, int sms, const int* cfg, DbPlan* pl) {
  const int pairs = sms / 2 > 0 ? sms / 2 : 1, tokblocks = db_tokblocks(M);
  const int user_bn = cfg ? cfg[0] : 0, user = cfg ? cfg[1] : 0;
  const int widths[2] = {user_bn > 0 ? user_bn : default_bn(gs), user_bn > 0 ? user_bn : pow2_bn(gs)};
  pl->bn = widths[0]; pl->splits = 1; pl->tail_rows = 0; pl->tail_splits = 1;
  if (user > 0) pl->splits = user;
  double best = 0;
  for (int i = 0; i < (widths[1] != widths[0] ? 2 : 1); ++i) {
    const int bn = widths[i], rows = N / bn;
    auto consider = [&](double us, int splits, int tail_rows, int tail_splits) {
      if (best > 0 && us >= best) return;
      best = us;
      pl->bn = bn; pl->splits = splits; pl->tail_rows = tail_rows; pl->tail_splits = tail_splits;
    };
    if (user != 0) {
      consider(db_launch_us(M, K, rows, bn, user > 0 ? user : 1, pairs), user > 0 ? user : 1, 0, 1);
      continue;
    }
    for (int s = 1; s <= 16 && s <= tokblocks; ++s) consider(db_launch_us(M, K, rows, bn, s, pairs), s, 0, 1);
    int yb, sb;
    if (db_tail(M, N, K, bn, pairs, &yb, &sb))
      consider(db_launch_us(M, K, rows - yb, bn, 1, pairs) + db_launch_us(M, K, yb, bn, sb, pairs), 1, yb, sb);
  }
}

// Groups per part of the dA+dR kernel when the tiles alone (`pairs` CTA pairs of `slots`) leave at least half of the SM pairs idle
// and the groups are split over blockIdx.y (see DadrExtra); G: one part.  A group takes a pair 1.0 us and 0.2 us per 64
// outputs in plain mode (1.2 us for 64 outputs, 2.4 for 512, 4.0 for 1024); gates add 0.4 us, an internal bias 1.5, rotations of 32
// and 64 0.5 and 1.8, which the workspace's size does not know of and the rule leaves out.  A split costs the fp32 sums of dA, written and
// read once (about 5 TB/s); they are added in the launch that adds dR's.  Split for a gain of 0.5 us or more.
// Over 300 timed shapes of few tiles (all modes) 0.7 % above the best split in the mean and none slower than unsplit; with
// 0.6 us per 64 outputs and 5 us against a split, as before, 13 %, up to 2.9 times.
inline int dadr_groups_per_part(int M, int K, int G, int gs, int pairs, int slots) {
  if (G < 2 || 2 * pairs > slots) return G;
  const double step = 1.0 + 0.2 * ((gs + 63) / 64);
  double best_us = G * step - 0.5;
  int best = G;
  for (int parts = 2; parts <= G && pairs * parts <= slots; ++parts) {
    const int per = (G + parts - 1) / parts;
    const double us = per * step + (double)parts * M * K * 8.0 / 5e6;
    if (us < best_us) { best_us = us; best = per; }
  }
  return best;
}

}  // namespace prism
