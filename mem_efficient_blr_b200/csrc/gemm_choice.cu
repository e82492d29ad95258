// Choice among the GEMM kernels and their tile widths by a model of their time (see gemm_choice.h).
#include "gemm_choice.h"

#include <algorithm>

#include "tmap.h"
#include "umma_pair.h"
#include "umma_wq.h"

namespace blr {

// Cycles (at 1.965 GHz) of one launch, fitted to 18 400 timed ones of 1387 GEMMs (1 to 16 groups, 48 to 11008 rows each, K = 48 to 2048, 17 to
// 4096 tokens, back to back with operands in L2 where they fit; 8 to 10 % off in the root mean square).  A step is 64 k of a tile: four MMAs at
// the tensor core's rate (46 cycles each up to 92 columns, then half a cycle per column), or its operands at the bytes per cycle that one
// SM can fetch, or at its share of what L2 delivers to all.  The tiles of a CTA overlap, the steps of the next with the stores of the last.
// The kernel and width with the least cycles take 1.5 % more than the best of all measured ones on average over the GEMMs that the model was fitted
// to, 4 % more at the ninth decile (a rule on waves and lengths that was tuned while every MMA cost the same, see elect_one, 10 and 31 %); over the last
// GEMMs of 260 other calls, every choice measured within its call, 1.3 and 4.7 %, 22 % at worst (Monarch 0.6 % up to 128 tokens and 3.5 above, BLAST
// 1.1, low rank 0.5).
// Not in the model: that a GEMM behind another one finds only some of the SMs free.  Monarch 4096 -> 11008, rank 1536, 128 tokens would take its 88
// CTAs of 128 rows instead of 116 of 96 then (18.9 against 20.1 us of the call), but a charge on the CTAs beyond the free SMs is no rule: in proportion to
// them it gains nothing (136 chains of two GEMMs 1.34 -> 1.25 % over the best, 192 others 1.31 -> 1.28), as a step it loses (1.34 -> 1.95, 1.31 -> 2.15).
// Nor that the element-wise stores of an interleaved output cost several times a tile's others (Monarch with more outputs a block than 2 rank, up to 20 % at
// the wrong width).
struct GemmCost {
  double launch, launch_col, launch_full;  // per launch; per column of the tile; on top where every SM has a tile
  double store, store_col, extra_col;      // per tile; per column; on top where the epilogue adds
  double bytes_sm, bytes_all;              // per cycle: into one SM; into each of them when all load
  double step;
};
static const GemmCost kDirect = {2898., 0., 1573., 1109., 10.85, 20., 84., 71.4, 104.};
static const GemmCost kDirectRagged = {2805., 0., 1905., 960., 18.6, 25.5, 77.7, 54.3, 73.};  // rows of 16-byte pieces only
static const GemmCost kSingle = {3543., 10.95, 416., 2027., 0.6, 12.9, 69.6, 54.7, 0.};
static const GemmCost kPair = {4242., 9.9, 1392., 1882., 1.85, 12.1, 68.2, 52., 25.6};
static const GemmCost kInt8 = {2979., 0., 1804., 1231., 18.2, 20., 53.8, 48.7, 231.};
static const GemmCost kInt4 = {2866., 0., 1510., 1493., 19.2, 20., 45.5, 38., 176.};

static long long gemm_tiles(const GemmParams& p, int rows, int bn) { return (long long)p.G * ((p.M + bn - 1) / bn) * ((p.N + rows - 1) / rows); }

static double gemm_cycles(const GemmCost& c, const GemmParams& p, int cg, int bn, int sms) {
  const long long tiles = gemm_tiles(p, 128 * cg, bn);
  const int slots = sms / cg;
  const long long waves = (tiles + slots - 1) / slots;
  const double active = tiles < slots ? (double)tiles / slots : 1., cols = waves > 1 ? (double)p.M / ((p.M + bn - 1) / bn) : bn;
  const double bytes = 128. * (umma_a_tile_rows(p) + (double)bn / cg);
  double step = 4. * (cols < 92. ? 46. : cols / 2.);
  if (bytes / c.bytes_sm > step) step = bytes / c.bytes_sm;
  if (bytes * active / c.bytes_all > step) step = bytes * active / c.bytes_all;
  const double main = (p.K + 63) / 64 * (step + c.step), out = c.store + (c.store_col + (p.bias || p.residual || p.act_out ? c.extra_col : 0.)) * cols;
  return c.launch + c.launch_col * bn + c.launch_full * active + main + out + (waves - 1) * (main > out ? main : out);
}

static GemmChoice gemm_look(const GemmParams& p, int sms, bool stores, double* cycles) {
  GemmChoice best = {0, 64};
  double& least = *cycles;
  least = -1.;
  auto look = [&](const GemmCost& c, int kernel, int bn) {
    // (pairs a little ahead of their fit: it sees too little of what they save where a long contraction shares few operands, such as 4 x (512 x
    // 2504) at 2500 tokens, 47 us on single CTAs and 36 on pairs)
    const double t = gemm_cycles(c, p, kernel == 2 ? 2 : 1, bn, sms) * (kernel == 2 ? .96 : 1.);
    if (least < 0. || t < least) least = t, best = {kernel, bn};
  };
  const bool quant = p.w_bits == 8 || p.w_bits == 4;
  const int unit = p.kmajor && !quant ? 32 : 64;
  const GemmCost& direct = p.w_bits == 8 ? kInt8 : p.w_bits == 4 ? kInt4 : p.M % 16 == 0 ? kDirect : kDirectRagged;
  for (int bn = unit; bn <= 256 && bn < p.M + unit; bn += unit) look(direct, 0, bn);
  if (!stores) return best;
  // Where the model is not asked: single CTAs with TMA stores for one wave of tiles of 256 rows, or for long contractions, where they win
  // little (over the 692 GEMMs of more than 128 tokens this line costs 0.2 % on average); pairs for one wave of 128 x 128 tiles, which a narrower tile of
  // single CTAs spreads over more SMs, and where K x waves is short, the more so with few groups and a ragged last tile of rows (0.3 %).
  const bool extra = p.bias || p.residual || p.act_out;
  const long long waves1 = (gemm_tiles(p, 128, 256) + sms - 1) / sms, waves2 = (gemm_tiles(p, 256, 256) + sms / 2 - 1) / (sms / 2);
  if (waves1 >= 2 && p.K <= (extra ? 1000 : 600))
    for (int bn = 64; bn <= 256 && bn < p.M + 64; bn += 64) look(kSingle, 1, p.kmajor && bn >= p.M ? (p.M + 31) / 32 * 32 : bn);
  if (gemm_tiles(p, 128, 128) > sms && p.K * waves2 > (p.G >= 8 ? 704 : p.M % 256 == 0 ? 2048 : 3000))
    for (int bn = p.kmajor ? 64 : 128; bn <= 256 && bn < p.M + 64; bn += p.kmajor ? 64 : 128) look(kPair, 2, bn);
  return best;
}

// The weights as the rows (umma_wq.cu), the tokens cut into c shares: its cycles by a model of the same form, fitted to 4449 sets of one GEMM's calls (linears of
// the networks and others, 17 to 1500 tokens, every share count timed within its call).  A step is 64 k of 128 rows by the share, at the slowest of its
// MMAs, shared memory and what L2 delivers.  Taken where it is 2 % ahead: calls 2.7 % faster on average for each of their GEMMs, 0.6 % more than the best choice;
// slower by more than 3 % in 51 sets, most of them Monarch's last GEMMs with 16 blocks, whose neighbours gain as much (us, tokens as rows | weights as
// rows: 4096 -> 11008, R = 1024, 17 / 128 / 200 tokens 14.5 / 17.2 / 21.9 | 12.4 / 16.4 / 19.3; Monarch 4096 -> 11008, rank 1536, 128 tokens 21.7 | 19.3; low
// rank 11008 -> 4096, R = 1024, 17 / 128 tokens 15.7 / 17.8 | 13.4 / 16.1).  Up to the tokens of one CTA: beyond, each row's weights are staged again, and what the model sees
// in single calls (1 to 3 %) is lost in a network, where a launch's neighbours share the SMs: denoising steps of 768 / 1024 / 1536 tokens, 28 blocks, 1890 /
// 1993 / 2407 | 2001 / 2206 / 2696.
// Not where long rows of a single block, or rows of 16-byte pieces off 32 bytes, cost the 128-row boxes more than the narrow tiles (us, tokens as rows | weights as
// rows): contraction-contiguous rows of one block, 3072 -> 768, 60 / 218 tokens 10.9 / 11.4 | 11.7 / 12.5, 4096 -> 4096, 384 tokens 16.1 | 18.8 (but 4096 -> 11008, 20 tokens
// 19.5 | 17.5), or of slices off 32 bytes, low rank 10672 -> 5024, R = 800, 24 tokens 24.1 | 30.7; few tokens on long output-contiguous rows off 32 bytes, 3344 -> 7048, 49 / 180
// tokens 13.8 / 20.6 | 17.0 / 18.5; many results in rows off 32 bytes, 1224 -> 11000, 340 tokens 17.1 | 23.4 (11008: 12.8 | 13.0).
static int rows_look(const GemmParams& p, int sms, double others) {
  if (p.N > kWqMaxTokens) return 0;
  if (p.kmajor ? p.K > 1536 && (p.w_odd || (p.G == 1 && p.M < 8192)) : p.w_odd && p.K > 2048 && p.N <= 64) return 0;
  if (p.G == 1 && p.M > 4096 && p.K >= 512 && p.N > 256 && p.os_n % 16 != 0) return 0;
  int best = 0;
  double least = .98 * others;
  for (int c = 1; c <= 6 && c <= (p.N + 15) / 16; ++c) {
    int tn, tt;
    umma_wq_share(p.N, c, &tn, &tt);
    const double share = (double)tn * tt, bytes = 128. * (share + 128.);
    const long long tiles = (long long)p.G * ((p.M + 127) / 128) * ((p.N + tn * tt - 1) / (tn * tt)), waves = (tiles + sms - 1) / sms;
    const double active = tiles < sms ? (double)tiles / sms : 1.;
    double step = share > 92. ? 2. * share : 95. > 2. * share ? 95. : 2. * share;
    if (bytes / 77. > step) step = bytes / 77.;
    if (bytes * active / 65.5 > step) step = bytes * active / 65.5;
    const double main = (p.K + 63) / 64 * (step + 5.), out = 1260. + 14.7 * share;
    const double t = 2750. + 660. * active + main + out + (waves - 1) * (main + out + 2800.);
    if (t < least) least = t, best = c;
  }
  return best;
}

// (A look costs the host 0.3 to 0.6 us, which shows in calls that it cannot enqueue ahead of the GPU: the last few shapes of a
// thread keep their answer.)
GemmChoice gemm_choice(const GemmParams& p, int* row_shares) {
  struct Kept {
    int v[6];  // G, M, K, N, SMs (0: empty), the rest
    GemmChoice choice;
    int rows;
  };
  static thread_local Kept kept[64];
  const int sms = sm_count();
  const bool stores = umma_pair_takes(p), by_rows = umma_wq_takes(p);
  const int rest = p.w_bits * 64 + (p.os_n % 16 != 0 ? 32 : 0) + (p.w_odd ? 16 : 0) + (by_rows ? 8 : 0) + (p.kmajor ? 4 : 0) +
                   (p.bias || p.residual || p.act_out ? 2 : 0) + (stores ? 1 : 0);
  const int v[6] = {p.G, p.M, p.K, p.N, sms, rest};
  unsigned h = 0;
  for (int x : v) h = (h ^ (unsigned)x) * 0x9E3779B1u;
  Kept& k = kept[h >> 26];
  if (!std::equal(v, v + 6, k.v)) {
    double cycles;
    k.choice = gemm_look(p, sms, stores, &cycles);
    k.rows = by_rows ? rows_look(p, sms, cycles) : 0;
    std::copy(v, v + 6, k.v);
  }
  if (row_shares != nullptr) *row_shares = k.rows;
  return k.choice;
}

}  // namespace blr
