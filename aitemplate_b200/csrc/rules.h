// The rules by which a call is sent to one form of a kernel or another where the choice changes its time only, never
// its result. Plain functions of sizes, so that they can be checked without a GPU. Times: B200, fp16 unless stated.
#pragma once

#include <algorithm>

namespace b200ait {

// Attention, heads above 64 channels: one CTA per SM with four K / V stages instead of two CTAs with two each. Taken
// where a second CTA would find nothing to do. One query row against 4096 keys of 96 channels, two CTAs' form -> lone:
// 16 heads 49 -> 46 us, 64 heads 55 -> 48, 148 heads 57 -> 49; with 160 heads two CTAs on some SMs are ahead (92 -> 68).
inline bool attn_lone(long long items, int sms) { return items <= sms; }

// Attention: how the work items (128 query rows of one head of one sequence) reach the CTAs. Two CTAs per SM either walk
// fixed shares of the items, which pays the set-up of a CTA once, or every item gets a CTA of its own, which pays it per
// item (2 x 16 heads x 2048 rows of 64, all items alike: 57.6 us in fixed shares, 59.2) and lets the hardware hand the
// items out as SMs fall free.
struct AttnItems {
  long long items;  // all of them, with the empty tiles past the end of shorter sequences
  int q_blocks;     // tiles of a head in the longest sequence
  int kv_blocks;    // key blocks (of 64) of the longest sequence
  bool causal;
  bool lengths;           // the sequences' lengths are known to the device alone (lengths_kv / lengths_q)
  long long mean, bound;  // rows of a sequence on average, and of the longest one as the caller states it; equal if not packed
  int d;                  // channels of a head (of q and k or of v, whichever are more)
};

// The longest fixed share of a causal problem whose sequences are all alike, in key blocks: CTA c walks items c, c + slots,
// c + 2 slots, .., and its length depends on how slots falls on the tiles of a head.
inline long long attn_longest_share(const AttnItems& a, int slots) {
  long long longest = 0;
  const long long starts = std::min<long long>(std::min(a.q_blocks, slots), a.items);  // CTAs further on start on the same tiles, with no more items
  for (long long c = 0; c < starts; ++c) {
    long long share = 0;
    for (long long i = c; i < a.items; i += slots) share += std::min<long long>(a.kv_blocks, 2 * (a.q_blocks - i % a.q_blocks));
    longest = std::max(longest, share);
  }
  return longest;
}

inline bool attn_item_per_cta(const AttnItems& a, int sms) {
  const int slots = 2 * sms;
  if (a.items <= slots) return false;  // (one and the same)
  // Lengths the host cannot see may be short, and then the set-up is most of the time (8 x 16 heads x 4096 rows of 64 with
  // 128 keys each: 45 us in fixed shares, 79).
  if (a.lengths) return false;
  if (a.mean >= a.bound) {  // every sequence is as long as the bound
    // Equal items gain nothing (heads of 16, 32, 48, 64, 80 and 128 channels, 297 .. 591 items of 4096 rows: 0 .. 2 %
    // slower). The exception are narrow heads whose rows are not whole 32-byte sectors: the time of their fixed shares
    // varies with where the operands lie (512 items of 4096 rows of 40: 113 .. 134 us, handed out 111 .. 117), and with a
    // second round of items that is not nearly empty a CTA per item is 4 % faster on average from 3072 rows on (14 % at
    // best; 432 items of 6144 rows 8 % slower), level at 2048.
    if (!a.causal)
      return a.d < 48 && a.d % 16 != 0 && a.kv_blocks >= 48 && 4 * a.items >= 5ll * slots && a.items < 2ll * slots;
    // Causal: a tile's length grows with its position, and fixed shares are as uneven as the stride falls on the heads.
    // Handed out, the shares end about 0.6 of the longest item after their mean. Measured over 24 problems of 1024 .. 6144
    // rows and two head widths: above 1.15 times that a CTA per item is 2 .. 27 % faster (16 heads x 2560 rows: 53.7 ->
    // 41.1 us), below it 6 % faster .. 5 % slower (32 heads x 2048 rows: 47.1 -> 49.1). Shorter sequences do not pay for
    // the set-up of their items, however uneven the shares (768 heads x 200 rows: 39.5 us in fixed shares, 42.3; 384 x 256:
    // 23.4 and 24.5; 256 x 512: 38.9 and 39.5).
    if (a.kv_blocks < 16) return false;
    long long blocks = 0;
    for (int t = 0; t < a.q_blocks; ++t) blocks += std::min(a.kv_blocks, 2 * (t + 1));
    const double mean_share = static_cast<double>(blocks) * (a.items / a.q_blocks) / slots;
    const double handed_out = mean_share + 0.6 * std::min(a.kv_blocks, 2 * a.q_blocks);
    return attn_longest_share(a, slots) > 1.15 * handed_out;
  }
  // Packed sequences of different lengths (or a bound above all of them, which the host cannot tell apart). An empty tile
  // costs a CTA launch: at most half of the tiles may be empty (64 sequences of 128 rows, 12 heads x 64, bound 4096: 99 us
  // in fixed shares, 134; 8 x 2048 rows with a bound of 16384: 150 and 156). Short items do not pay for their set-up: over
  // evenly and randomly spread lengths of 16 heads, causal, a mean below 2048 rows runs from 29 % faster to 14 % slower,
  // above it from 49 % faster to 2 % slower (8 sequences of 512 .. 4096 rows, 16 heads x 128: 292 -> 277 us). Without a
  // mask, over 13 sizes of five head widths and five spreads, a mean from 2048 rows on runs from 26 % faster to 6 % slower (8
  // sequences of 512 .. 4096 rows, 16 heads x 128 in any order: 485 -> 421 us) but for nearly equal lengths, which lose up to 10 %
  // below 2560 rows (8 x 2048 with a bound of 2560, 24 heads x 96).
  if (2 * a.mean < a.bound) return false;
  return a.mean >= 2048 && (a.causal || a.mean >= 2560 || 2 * a.bound >= 3 * a.mean);
}

// GEMM, one to four rows of X against 256 to 1023 channels: one row of W after the other on the CUDA cores, or the tensor
// cores. The CUDA cores do M multiplications per weight and a conversion that bfloat16
// pays twice; the tile kernels' time goes by whole key blocks of 64 channels and jumps where W leaves the L2 cache.
// `whole`: the rows of the output are whole 16-byte units. Others cost the tile kernels 1.5 to 2 times as much, and the
// CUDA cores nothing (4 x 80001 x 640: 31 us, tiles 46).
// CUDA cores -> tiles, us. M = 4, fp16: 8192 x 320: 5.0 -> 6.3, 16384 x 320: 7.9 -> 6.6, 50256 x 384: 17.8 -> 10.7, 128256 x
// 256: 29.6 -> 15.8, 50256 x 512: 17.9 -> 19.7, 128256 x 512: 39.4 -> 36.6 .. 39.0, 24576 x 640: 12.3 -> 13.6, 50256 x 576: 20.9 -> 18.1, 50256 x 776: 21.2 ->
// 24.9. M = 4, bf16: 20480 x 320: 9.7 -> 10.1, 30520 x 320: 12.9 -> 10.7, 50256 x 576: 24.7 -> 17.9, 50256 x 512: 19.2 ->
// 19.5, 50256 x 768: 24.1 -> 22.3, 50256 x 832: 24.6 -> 24.5. M = 2, fp16: 50256 x 256: 9.3 -> 10.7, 80000 x 256: 13.7 -> 12.1. M = 1 always gains.
inline bool gemm_rowdot_short(long long m, long long n, long long k, bool whole, bool bf16) {
  if (k < 256 || k >= 1024 || n < 64) return false;
  if (m == 1 || !whole) return true;
  if (m == 2) return bf16 || k > 384 || n <= 56000;
  if (k <= 448) return n <= (bf16 ? 28000 : 10000);
  if (k <= 512) return n <= 80000;
  return k > (bf16 ? 768 : 704) || n <= 28000;
}

// GEMM, an output that TMA cannot describe: the staging boxes written row by row, or every thread its own row. Row by row
// fills the sectors of an output of some width, but pays for 64 columns whatever the width. Every thread its own row -> row
// by row, 32768 x N x 320 fp16, 64-wide tiles, ratio of the times: N = 3: 1.51, 17: 1.35, 33: 1.08, 41: 0.98, 47: 0.85; 3000 x
// N x 768: 17: 1.23, 41: 1.06, 43: 1.01, 47: 0.96; with one residual, which goes through the boxes too, 17: 1.46 and 1.30, 43:
// 1.06 and 1.07, 47: 0.97 and 1.03, 49: 0.93 and 0.99. Wider tiles give such an output half of their warps: N = 7: 1.25 ..
// 1.6, 31: 1.0 .. 1.4, 33: 0.63 .. 1.08.
inline bool gemm_rows_output(int n, int tile_n, bool one_residual) {
  return n > (tile_n > 64 ? 32 : one_residual ? 47 : 42);
}

// GEMM: the time of a launch of the tile kernels (128 x 64, 128 x 128, 128 x 256 tiles, and 256 x 256 on CTA pairs: width 512)
// and of the weight-streaming kernel, in us. Both were fitted to a sweep of 650 problems (M = 64 .. 3000, N and K = 256 .. 8192,
// N whole and not whole 16-byte rows, three epilogues, every tile and every weight-streaming kernel forced, fp16, one launch
// behind the other), with 5 % root mean square. Launches have become shorter since (launch_early): over 160 other problems of these
// ranges the estimates lie 15 % off (root mean square; -30 % and +35 % at worst), mostly too long, all widths alike. The launch
// they pick takes 1.017 times the best one's time on average, 1.49 at worst (625 x 368 x 320), and 18 of the 160 more than
// 1.05. (The rules before, a width by whole waves at 512 cycles per k-block, K split over CTAs and the weight-streaming
// kernel up to a number of tiles, took 1.055 and, with N not a multiple of 8, 1.14 times in the first sweep.)
struct GemmProblem {
  long long batch, m, n, k;
  int epilogue;      // 0: bias [+ relu], 1: a residual operand, 2: another activation
  int swap_epilogue; // as the weight-streaming kernel sees it: 0: bias [+ relu], 1: an added residual, 2: anything else
  long long pitch;   // of the operands' rows, in elements (the worse aligned one's)
  bool generic;      // an epilogue read from the parameters (row-major B, several destinations)
  bool pairs = true; // CTA pairs can take it (they do not write the permuted batches of bmm_*_permute)
};
constexpr int kGemmPairWidth = 512;
// What TMA takes for a 128-byte row of an operand box that does not start on a 128-byte boundary, in us: 2.85 cycles if it starts
// on a 16-byte one only, 1.97 on 32, 1.7 on 64 (1.3 if aligned, which the costs below contain). 2048 x 2048 x 2040 takes 44,
// 31, 24 and 19 us with 64-, 128-, 256-wide tiles and pairs, x 2048 23, 18, 16 and 16.
inline double gemm_copy_row_us(long long pitch) {
  return pitch % 64 == 0 ? 0.0 : pitch % 32 == 0 ? 0.00086 : pitch % 16 == 0 ? 0.00100 : 0.00146;
}
// The same for batched problems, most of which are a few k-blocks deep and give every CTA many tiles: the step from one tile to the next,
// not the launch, decides. Fitted to 1600 problems of 2 .. 1024 products (M 32 .. 1024, N 64 .. 1024, K 32 .. 1024, both storage
// orders of B, fp16 and bf16, every width forced), 7 .. 16 % root mean square by row of the table; the widths they pick take 1.012
// times the best one's time on average, 1.41 at worst. The estimate of single products, which was used here before, took 1.06 and 2.3
// times, and 47 of the 1600 were slower by more than 2 % than by the rule of whole waves ahead of it (now 11, the worst by 7 %):
// 78 x [160 x 80 x 72] row-major B 11.8 us, 5.6 now (128 wide); 285 x [374 x 136 x 88] 22.4, 17.9 (256); 445 x [295 x 392 x 40] 50.9, 39.8.
inline double gemm_batched_tile_us(const GemmProblem& g, int width, int sms) {
  // launch and one epilogue; a k-block; a step's own cost and its share that goes by how full the tiles are; how much of the shorter one
  // of step and main loop is not hidden by the longer; a chunk of 32 columns that the edge of N cuts, which the threads of
  // 64-wide tiles store element by element
  struct Cost {
    double once, k_block, step, filled, exposed, cut;
  };
  static constexpr Cost whole[4] = {{2.90, 0.151, 0.10, 1.04, 0.96, 2.07},
                                    {2.80, 0.149, 0.37, 0.56, 1.00, 0.0},
                                    {3.31, 0.250, 0.38, 1.71, 1.00, 0.0},
                                    {3.93, 0.219, 0.67, 1.42, 1.00, 0.0}};
  static constexpr Cost ragged[4] = {{7.11, 0.220, 4.54, 0.56, 0.06, 0.0},
                                     {7.64, 0.122, 4.93, 0.0, 0.20, 0.0},
                                     {11.74, 0.348, 9.53, 0.0, 0.16, 0.0},
                                     {11.90, 0.324, 8.94, 0.59, 0.39, 0.0}};
  static constexpr Cost row_major[4] = {{3.10, 0.196, 0.55, 0.48, 0.91, 2.75},
                                        {4.04, 0.300, 1.32, 0.35, 0.36, 0.0},
                                        {5.35, 0.468, 2.30, 1.31, 0.38, 0.0},
                                        {5.69, 0.337, 2.42, 0.73, 0.39, 0.0}};
  const bool pair = width == kGemmPairWidth;
  const Cost& c = (g.generic ? row_major : g.n % 8 == 0 ? whole : ragged)[width == 64 ? 0 : width == 128 ? 1 : pair ? 3 : 2];
  const long long bm = pair ? 256 : 128, bn = pair ? 256 : width, walkers = pair ? sms / 2 : sms;
  const long long tiles_m = (g.m + bm - 1) / bm, tiles_n = (g.n + bn - 1) / bn, tiles = tiles_m * tiles_n * g.batch;
  const double ctas = static_cast<double>(std::min(tiles, walkers) * (pair ? 2 : 1));
  const int rows = pair ? 256 : 128 + width;
  const double loop = static_cast<double>((g.k + 63) / 64) * std::max({c.k_block, 128.0 * rows * ctas / 22.1e6, rows * gemm_copy_row_us(g.pitch)});
  const double cut = g.n % 8 == 0 && g.n % 32 != 0 ? c.cut : 0.0;
  const double filled = static_cast<double>(g.m) * static_cast<double>(g.n) / static_cast<double>(tiles_m * bm * tiles_n * bn);
  const double step = c.step + c.filled * filled + cut / static_cast<double>(tiles_n);
  return c.once + cut + loop +
         static_cast<double>((tiles + walkers - 1) / walkers - 1) * (std::max(loop, step) + c.exposed * std::min(loop, step));
}
inline double gemm_tile_us(const GemmProblem& g, int width, int sms) {
  if (g.batch > 1) return gemm_batched_tile_us(g, width, sms);
  // launch, k-block, and a tile's epilogue by GemmProblem::epilogue; then what an epilogue costs beyond that where the tiles
  // of a CTA follow on each other's heels
  struct Cost {
    double launch, k_block, epilogue[3], next;
  };
  // A k-block of 64-wide tiles is bound by the issue of its copies, of 128-wide ones by shared memory (operands come in and are
  // read by the MMA at 128 bytes a cycle), above that by the MMA. All CTAs together draw at most 22 TB/s of operands from L2.
  static constexpr Cost whole[4] = {{2.28, 0.130, {1.63, 2.05, 1.89}, 0.14},
                                    {2.56, 0.176, {1.27, 2.42, 1.91}, 0.19},
                                    {2.67, 0.327, {2.02, 4.10, 2.89}, 0.98},
                                    {2.18, 0.305, {3.31, 3.95, 4.01}, -0.68}};
  static constexpr Cost ragged[4] = {{3.01, 0.128, {3.22, 4.96, 3.50}, 0.62},
                                     {3.73, 0.175, {4.52, 7.20, 5.09}, 1.40},
                                     {4.82, 0.315, {8.24, 13.43, 9.46}, 2.73},
                                     {5.47, 0.301, {8.21, 13.43, 9.30}, 2.40}};
  const int at = width == 64 ? 0 : width == 128 ? 1 : width == 256 ? 2 : 3;
  const Cost& c = (g.n % 8 == 0 ? whole : ragged)[at];
  const bool pair = width == kGemmPairWidth;
  const long long bm = pair ? 256 : 128, bn = pair ? 256 : width, walkers = pair ? sms / 2 : sms;
  const long long tiles = ((g.m + bm - 1) / bm) * ((g.n + bn - 1) / bn) * g.batch;
  const long long waves = (tiles + walkers - 1) / walkers;
  const double ctas = static_cast<double>(std::min(tiles, walkers) * (pair ? 2 : 1));
  const int rows = pair ? 256 : 128 + width;  // that a CTA fetches per k-block
  const double k_block = std::max({c.k_block, 128.0 * rows * ctas / 22.1e6, rows * gemm_copy_row_us(g.pitch)});
  const double loop = static_cast<double>((g.k + 63) / 64) * k_block;
  constexpr double kGeneric[4] = {0.0, 1.2, 1.5, 1.0};
  const double epilogue = c.epilogue[g.epilogue] + (g.generic ? kGeneric[at] : 0.0) + (width == 64 && g.n % 8 != 0 ? 2.1 : 0.0);
  // 64-wide tiles are stored by the threads, element by element where the edge of N cuts a chunk of 32 columns (625 x 368 x 320:
  // 5.6 us, 3.8 with 128-wide tiles, which were passed over as long as this was charged by sectors, N % 16)
  const double cut = width == 64 && g.n % 8 == 0 && g.n % 32 != 0 ? (g.n % 16 == 0 ? 1.1 : 2.1) : 0.0;
  return c.launch + loop + epilogue + cut +
         static_cast<double>(waves - 1) * std::max(loop, epilogue + c.next + cut / static_cast<double>((g.n + 63) / 64));
}
// mx rows of X per group, K split r ways over a cluster, `resident` clusters on the GPU at once
inline double gemm_swap_us(const GemmProblem& g, int mx, int r, int resident) {
  const long long units = ((g.m + mx - 1) / mx) * ((g.n + 127) / 128);
  const long long waves = (units + resident - 1) / resident;
  const double ctas = static_cast<double>(std::min<long long>(units, resident) * r);
  const long long k_blocks = ((g.k + 63) / 64 + r - 1) / r;
  const double stream = static_cast<double>(k_blocks) * std::max({0.0754 + 0.0012 * mx, (16384.0 + mx * 128.0) * ctas / 26.6e6,
                                                                  (128 + mx) * gemm_copy_row_us(g.pitch)});
  // the exchange of partial sums, then the rows a rank finishes; output rows that are not whole 16-byte units go out by element
  const double row = 0.0105 + (g.swap_epilogue == 1 ? 0.0121 : g.swap_epilogue == 2 ? 0.0229 : 0.0) + (g.n % 8 == 0 ? 0.0 : 0.26);
  const double tail = 0.0268 * mx * (r - 1) / r + row * mx / r;
  return 3.79 + stream + tail + static_cast<double>(waves - 1) * (std::max(stream, tail) + 0.8);
}
// The weight-streaming kernel in more rows than 2048: only where its units are one wave. The estimate does not hold for several waves
// of large groups (8192 x 640 x 8192: 111 us, 74 by the estimate, tiles 91), in one wave it does (4096 x 128 x 8192: 12.7 us, tiles
// 19.3, tiles with K in two parts 18.8; 2049 x 128 x 8192: 8.7, 17.2 and 15.6, 4096 x 128 x 2048: 6.2, 6.8 and 11.7).
inline bool gemm_swap_in_range(long long m, long long units, int resident) { return m <= 2048 || units <= resident; }
inline int gemm_best_width(const GemmProblem& g, int sms) {
  int best = 64;
  for (int width : {128, 256, kGemmPairWidth}) {
    if (width == kGemmPairWidth && (!g.pairs || (g.batch == 1 && (g.n < 256 || (g.generic && g.k < 512))))) break;
    if (gemm_tile_us(g, width, sms) < gemm_tile_us(g, best, sms)) best = width;
  }
  return best;
}

// GEMM, unbatched, aligned operands, neither a tile width nor a number of splits asked for: one to four rows of X against long rows of
// W (which fit in shared memory, 160 KB) go to the CUDA cores,
inline bool gemm_rowdot_long(long long m, long long n, long long k) {
  return m <= 4 && n >= 64 && k >= 1024 && (m <= 2 ? m : 4) * k <= 80 * 1024;
}
// and K is shared out through scratch memory only where no weight-streaming kernel could have taken the problem. Where one could, it or
// whole tiles are ahead of K in parts: over M = 5 .. 8192, N = 128 .. 640 and K = 2048 .. 8192 the best of three widths and five
// numbers of parts took 1.08 to 2.7 times as long as the launch chosen here.
inline bool gemm_may_split(long long m, long long n, long long k) {
  return !(m >= 5 && n >= 128) && !gemm_rowdot_long(m, n, k);
}

// May a tile kernel's CTAs become resident before the kernel ahead of it has ended (launch_early)? It saves 0.4 .. 0.8 us (3 .. 25 %
// of launches under 15 us), but CTAs then take the SMs in the order in which these fall free, so that neighbouring tiles no
// longer lie on neighbouring SMs: where the CTAs walk several tiles each that costs more than it saves (4096^3 bf16 99 -> 103
// us, 8192^3 857 -> 876, bmm 855 x [430 x 88 x 96] 30.0 -> 31.2 and 204 x [221 x 168 x 120], 2.8 tiles a CTA, 13.6 -> 14.1;
// 352 x [76 x 88 x 128], 2.4 a CTA, 7.9 -> 7.3 and 8192 x 1280 x 320, 2.2, 13.2 -> 12.7), and where tiles are stored straight to
// rows that share sectors it already does with one (700 x 5003 x 1024 + add 23.2 -> 25.5; 384 x 769 x 768 11.3 -> 10.8).
inline bool gemm_starts_early(int units, int walkers, bool staged, int sms) {
  return staged ? 2ll * units <= 5ll * walkers : 2ll * units <= sms;  // (unstaged: at most half of the SMs get a tile)
}
// The same for kernels of which an SM holds many blocks (rows, copies, permutes, element-wise), in a graph. They take the SMs in the order in which these
// fall free as well, several blocks to an SM: a grid that would put a block or a few on every SM piles up on the first ones and
// the others stay idle. Behind one another, us, early -> plain: softmax of 3521 x 896 (441 blocks of 256 threads) 5.65 -> 3.84, layernorm of
// 2575 x 832 (322) 5.20 -> 3.90, concatenate 2 x [172 x 112 x 56] 4.62 -> 3.38, 11 x [112 x 758] transposed (264) 2.92 -> 2.38. Fewer
// blocks than half the SMs have room anywhere (softmax of 365 x 1024: 2.46 -> 2.09 early), and so has a grid that fills the
// SMs (13863 x 512: 5.54 -> 5.12; copies from half of the threads on, 1074 blocks: 8.8 -> 8.1). `light`: rows of one 16-byte
// vector per lane at most, which gain up to four blocks an SM (1455 x 48: 1.90 -> 1.79, 634 x 40: 1.79 -> 1.40). Over 720 calls of
// seven kinds: early always 0.92 of the plain launch's time and 105 calls slower, by this rule 0.91 and 2, by 4 and 6 %.
// Outside of a graph a plain launch is dearer, its times come in steps of 2.05 us (4.11, 6.16), and everything starts early: softmax of
// 1055 x 768 2.7 us, plain 4.1, 64 x [384 x 64] transposed 2.2 and 4.1, layernorm of 2575 x 832 5.6 and 6.2 (but softmax of 3521 x 896 6.5 and
// 6.2); encoder layers of 5 x 211 and 7 x 150 rows, each run waited for, 82 and 80 us, 87 both with this rule.
inline bool blocks_start_early(long long blocks, int threads, int sms, int filled_threads, bool light = false) {
  return 2 * blocks <= sms || blocks * threads >= static_cast<long long>(filled_threads) * sms || (light && blocks <= 4ll * sms);
}

}  // namespace b200ait
