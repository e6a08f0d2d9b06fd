// Which kernel a call runs on, as far as sizes decide it: plain C++ without CUDA, so that the rules can be checked
// on any machine.  Costs are SM cycles at 1.92 GHz.
#pragma once

#ifdef __CUDACC__
#define TCEC_HOST_DEVICE __host__ __device__
#else
#define TCEC_HOST_DEVICE
#endif

namespace tcec_host {

inline long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

// Whether the wide tiles of the panel GEMM go to CTA pairs, which bring a third fewer bytes through L2 per product (a half fewer
// of B).  Long calls run at the board's power limit, where those bytes cost clock: with its pairs kept together along K (below)
// 16384^3 takes 19.3 ms on pairs and 20.0 on single SMs, 8192^3 2.41 and 2.53, tf32 4.20 and 4.34, 8192^3 without correction 0.91 and
// 1.0.  Not where the 256 rows of a pair tile are half empty and the call is long: what is lost is one part in the number of
// 128-row blocks.
constexpr double kLongCall = 2.5e11;  // flop
inline bool pairs_pay(int m, int n, int k, int batch, bool ec) {
  const long long blocks = ceil_div(m, 128);
  return !ec || 2.0 * m * static_cast<double>(n) * k * batch <= kLongCall || blocks % 2 == 0 || blocks >= 19;
}

// Pair tiles are taken in groups of kPairGroupM tile rows, column by column.  A launch is paced (tcec_gemm_panels_pair.cuh) if it
// has several rounds of tiles, over which they get out of step, and the panels that one wave of tiles reads do not stay in L2 (126
// MB) all the while.  Unpaced and paced, ms: 16384^3 (290 MB) 21.5, 19.3; 12000 x 4000 x 12000 (212 MB) 2.79, 2.70; 8192^3 (145 MB) 2.46,
// 2.44; without correction 16384^3 (145 MB) 7.9, 7.3, but 8192^3 (72 MB) 0.912, 0.925.  Two
// rounds do not earn the clearing of the word between split and GEMM (tf32 534 x 8189 x 1828, 105 MB: 147.6, 148.7 us).
constexpr int kPairGroupM = 8;
inline bool pace_pays(int tiles_m, int tiles_n, int batch, int nkb, int images, int pairs) {
  if (static_cast<long long>(tiles_m) * tiles_n * batch < 4 * pairs) return false;
  const long long rows = tiles_m < kPairGroupM ? tiles_m : kPairGroupM, wave = ceil_div(pairs, rows), cols = tiles_n < wave ? tiles_n : wave;
  return static_cast<double>(rows + cols) * 256 * 64 * images * nkb >= 100e6;
}

// Whether the tiles of a pair launch are drawn from a counter: calls with correction above the size up to which pairs were always
// taken.  Longer ones ran on single SMs, which draw theirs, and have to do as well as those beside another stream's kernel.
inline bool draws_pay(int m, int n, int k, int batch, bool ec, long long tiles, int pairs) {
  return ec && tiles > pairs && 2.0 * m * static_cast<double>(n) * k * batch > kLongCall;
}

// The panel GEMM of a call: `width` of the narrow tiles if they would finish the call sooner than 256-wide ones, else 0,
// and what the call is expected to take without its split.
struct PanelChoice {
  double cycles;
  int width;
};

// Cycles per K block of a tile, fitted to what was measured: wide tiles pay their MMAs and, per promotion, about 1700 cycles in
// which the main products wait (2048^3 on CTA pairs, a promotion every 2 blocks: 69 us; 4096^3, every 4: 83 us a tile); narrow
// ones take the larger of their MMAs and their copies at 42 bytes per cycle and SM (2048^3 in 128-wide tiles: 62 us), and at
// least what their epilogue takes.  Both sides at the sizes where the choice turns: 1000 x 777 x 1111 36 us wide, 25 with 64;
// 1500^3 41 and 34 (128); 2048^3 69 and 63 (128); 1000 x 4096 x 4096 107 and 108; 4096^3 stays wide.
// `promo`: K blocks per promotion, 0 = one at the end; `tile_n`: width of the one-SM kernel's tiles; `pair`: the wide
// tiles would be 256 x 256 on CTA pairs.
inline PanelChoice panel_choice(int m, int n, int batch, int nkb, int promo, bool ec, int tile_n, int sms, bool pair) {
  const long long tiles_m = ceil_div(m, 128);
  const int rows = m < 128 ? (m + 7) & ~7 : 128;
  const long long wide_tiles = pair ? ceil_div(m, 256) * ceil_div(n, 256) * batch : tiles_m * ceil_div(n, tile_n) * batch;
  const int wide_slots = pair ? (sms / 2 > 1 ? sms / 2 : 1) : sms;
  const double rounds = static_cast<double>(ceil_div(wide_tiles, wide_slots));
  PanelChoice c{0.0, 0};
  // Beyond two rounds of wide tiles the last, partly empty one weighs little (256 x 512^3: 308 us wide, 324 with 128).
  if (wide_tiles <= 2 * wide_slots) {
    const double wide_block = (ec ? 768.0 : 300.0) + 1700.0 / (promo ? promo : nkb);
    c.cycles = rounds * (nkb * wide_block + 10000.0);
    const double mma[3] = {240.0, 288.0, 446.0};
    double expected = c.cycles;
    for (int i = 0; i < 3; ++i) {
      const int bn = 32 << i;
      if (i > 0 && n <= bn / 2) break;
      const long long tiles = tiles_m * ceil_div(n, bn) * batch;
      const double copy = (rows + bn) * 64.0 * (ec ? 2 : 1) / 42.0, products = ec ? mma[i] : mma[i] / 3.0;
      const double tile = nkb * (products > copy ? products : copy);
      const double in_a_row = static_cast<double>(ceil_div(tiles, sms)), cost = in_a_row * (tile > 6000.0 ? tile : 6000.0) + 4000.0;
      if (cost < c.cycles) {
        c.cycles = cost;
        c.width = bn;
        // tiles in a row wait for one another's epilogues (2 x 2048 x 2048 x 256, four rounds: 28 us with its split), and a K
        // block takes 290 cycles at least (74 x 36 x 136 x 1412 without correction, three rounds: 48 us)
        double all = tile > nkb * 290.0 ? tile : nkb * 290.0;
        if (in_a_row > 1 && all < 10000.0) all = 10000.0;
        expected = in_a_row * (all > 6000.0 ? all : 6000.0) + 4000.0;
      }
    }
    c.cycles = expected;
  }
  // What wide tiles take in a row: on pairs a round adds 9400 cycles to its K blocks, on one SM 14000, and 28000 where a tile is
  // mostly padding (55 x 120 x 3536 x 16 is six rounds and 77 us, 2 x 128 x 20000 x 2048 two and 229).
  if (c.width == 0 && !pair) c.cycles = rounds * (nkb * (ec ? 1130.0 : 480.0) + (m > 128 ? 14000.0 : 28000.0));
  else if (c.width == 0 && wide_tiles > 2 * wide_slots) c.cycles = rounds * (nkb * (ec ? 1150.0 : 255.0) + 9400.0);
  return c;
}

// How many CTAs share the K of a 128 x 128 tile (1: undivided, and then other widths are open): as many as have room at a time.  The
// B200s seen run 74 clusters of two, 33 of four and 15 of eight; GPUs differ in which SMs of their GPCs are there, so the rule has these
// numbers and does not ask the device: a call has the same bits on every GPU.  (A GPU with room for 16 clusters of eight gives up
// what 15 tiles, 128 x 1920 x 4096, gain from it: 14.8 us in four parts, 12.0 in eight.)  Only one that runs no such cluster at all,
// runs[i] = 0, does without.  Undivided against 2, 4, 8 parts, us, GEMM alone on packed operands:
//   64 x 4096 x 4096 (32 tiles) 27.3, 24.0, 15.8    300 x 500 x 4100 (12, with split) 33.9, 28.9, 22.5, 18.8
//   33 x 206 x 11446 (2) 67.6, 48.0, 28.4, 18.8    110 x 1161 x 3881 (10) 26.2, 22.3, 15.7, 13.3    813 x 1122 x 3183 (63) 24.0, 21.1
//   344 x 402 x 2524 no correction (12) 15.8, 15.5, 11.7, 10.8    128 x 512 x 8192 tf32 (4, with split) 51, 47, 31, 24
// The exchange costs about 3 us, which few K blocks do not earn: in two parts 77 x 6331 x 1115 11.9, 12.9 and 54 x 122 x 1626 13.1, 14.0;
// in four and eight it is even at K = 800 to 1000 (12 x 1276 x 789 8.1, 8.7, 8.5; 20 x 80 x 1203 10.3, 8.9, 8.3).  Calls below K = 1200
// stay undivided and keep the bits of the other kernels.  So do batches and matrices of one tile, which have another kernel to
// go to where no workspace can be allocated (a first call that is captured): its bits would differ.
// `forced`: -1 = by this rule, else that many wherever they have room.
constexpr int kClusterRoom[3] = {74, 33, 15};  // clusters of 2, 4, 8 CTAs
inline int divide_k(int m, int n, int k, int batch, int nkb, bool ec, const int (&runs)[3], int forced) {
  const long long tiles = ceil_div(m, 128) * ceil_div(n, 128);
  if (batch > 1 || tiles == 1) return 1;
  for (int i = 2; i >= 0; --i) {
    const int parts = 2 << i;
    if (tiles > kClusterRoom[i] || runs[i] < 1 || nkb < parts) continue;
    if (forced == parts || (forced == -1 && k >= 1200 && (parts > 2 || nkb >= (ec ? 64 : 96)))) return parts;
  }
  return 1;
}

// The split in front of the panel GEMM: a launch, and reading FP32 and writing the images at 2970 bytes per cycle.
inline double split_cycles(int m, int n, int k, int batch, bool ec) {
  return 7700.0 + (static_cast<double>(m) + n) * k * batch * (ec ? 8.0 : 6.0) / 2970.0;
}

// How C leaves the FP32-tile kernel: by tensor stores (row-major, beta = 0), by plain ones, or through pointer tables, which add
// the launch that writes the tensor maps and the launches that then do nothing (16 x 256 x 256 x 128: 14 us strided, 22 by
// tables).  Plain stores keep a tile for 18000 cycles at least (1024 x 160^3 by tables 155 us, 4096 x 132^3 503).
enum class FusedStores { kTensor, kPlain, kTables };

// The FP32-tile kernel (fp16 policies): rounds of 256 x 256 tiles on CTA pairs, each loading and converting its own
// operands.
inline double fused_cycles(int m, int n, int nkb, int batch, bool ec, int sms, FusedStores stores) {
  const long long tiles = ceil_div(m, 256) * ceil_div(n, 256) * batch;
  double tile = 3425.0 + nkb * (ec ? 1634.0 : 1043.0);
  if (stores != FusedStores::kTensor && tile < 18000.0) tile = 18000.0;
  return 12300.0 + (stores == FusedStores::kTables ? 15400.0 : 0.0) +
         static_cast<double>(ceil_div(tiles, sms / 2 > 1 ? sms / 2 : 1)) * tile;
}

// Whether a batch (fp16 policy, n > 128, operands that TMA can address) is expected to take less time on the FP32-tile kernel
// than split and multiplied from panels.  Conversion is repeated in every tile of a matrix and K runs serially in tiles
// of 256 x 256, so large matrices and few of them are better off with panels; the split moves all operands through DRAM once
// more, so many matrices of one or a few tiles are better off without.  On 321 shapes (2 to 1400 matrices of 16 to 8192, K
// from 16 to 6000) the fit is within 12 % (this kernel) and 17 % (panels) rms, and the rule takes the slower side by more
// than 5 % on 19 of them, against 85 with a bound on K alone.  Panels against this kernel, us:
//   64 x 400 x 400 x 1000 171, 128    32 x 1024^3 281, 220    8 x 1024 x 1024 x 2048 137, 123    128 x 256^3 46, 25
//   2 x 8192 x 8192 x 2048 1500, 1808    2 x 1024^3 22, 37    16 x 256 x 256 x 2048 40, 73    2 x 256 x 256 x 512 10, 23
inline bool fused_pays(int m, int n, int k, int batch, int nkb, int promo, bool ec, int sms, bool pair,
                       FusedStores stores) {
  // about equal: this kernel, which needs no workspace
  return fused_cycles(m, n, nkb, batch, ec, sms, stores) <
         1.03 * (split_cycles(m, n, k, batch, ec) + panel_choice(m, n, batch, nkb, promo, ec, 256, sms, pair).cycles);
}

// Whether matrices of at most one 128 x 128 tile go to the direct kernel.  It needs one launch instead of two and moves nothing
// twice, but one CTA walks the K of its tile (0.8 us per 32 of K; tf32 1.4), where panels in narrow tiles give a matrix four
// CTAs and every K block little more than 0.15 us.  Few matrices (weighed by their rows, of which the panels' split has as
// much to do) of long K are therefore multiplied from panels.  One call after another, us, direct against panels:
//   one 128 x 128 x K, K = 96: 11, 15   192: 13, 15   256: 15, 15   512: 22, 13   1024: 35, 16 (tf32 96: 12, 13   128: 14, 13)
//   32 of them, K = 256: 14, 14   512: 22, 17   64 of them, K = 1024: 35, 39   2048: 71, 65   100, K = 4096: 136, 197
//   100 x 32 x 32 x 1024: 31, 23   200: 31, 42
// tf32 panels are twice the bytes: 64 x 128 x 128 x 1024 54, 61; 48 of them 52, 46
inline bool direct_pays(int m, int n, int nkb, int batch, bool tf32, int sms) {
  const double matrices = batch * (0.35 + 0.65 * (static_cast<double>(m) + n) / 256.0) * (tf32 ? 1.2 : 1.0), slots = sms / 2;
  return nkb * (slots - matrices) <= 6.0 * slots;
}

// ---------------------------------------------------------------- results that lie over operands
// Where the matrices of a call lie: `outer` runs of `inner` consecutive floats, `ld` apart, and matrix i `stride` floats behind
// matrix 0.
struct Extent {
  const void* base;
  long long ld, stride;
  int inner, outer;
};

// Whether one matrix at `c` and one at `x` may share an element: not if their spans are apart, nor if they are column ranges
// of rows of one length (blocks of one larger matrix).
TCEC_HOST_DEVICE inline bool matrices_may_overlap(unsigned long long c, long long ldc, int c_inner, int c_outer,
                                                  unsigned long long x, long long ldx, int x_inner, int x_outer) {
  const unsigned long long c_span = 4ull * ((c_outer - 1) * ldc + c_inner), x_span = 4ull * ((x_outer - 1) * ldx + x_inner);
  if (c >= x + x_span || x >= c + c_span) return false;
  if (ldc == ldx && ldc > 0) {
    const long long row = 4 * ldc;
    long long d = static_cast<long long>(c - x) % row;  // columns of C begin d bytes behind those of X
    if (d < 0) d += row;
    if (d >= 4ll * x_inner && d + 4ll * c_inner <= row) return false;
  }
  return true;
}

// Which matrices of a batch a result may share elements with: those of the same index, those of another one.
struct Overlap {
  bool own, across;
};
inline Overlap batch_overlap(const Extent& c, const Extent& x, int batch) {
  typedef __int128 wide;  // strides are the caller's and may be anything
  const wide c0 = reinterpret_cast<unsigned long long>(c.base), x0 = reinterpret_cast<unsigned long long>(x.base);
  const wide c_span = 4 * (static_cast<wide>(c.outer - 1) * c.ld + c.inner), x_span = 4 * (static_cast<wide>(x.outer - 1) * x.ld + x.inner);
  const wide cs = 4 * static_cast<wide>(c.stride), xs = 4 * static_cast<wide>(x.stride), last = batch - 1;
  const wide c_lo = c0 + (cs < 0 ? last * cs : 0), c_hi = c0 + c_span + (cs > 0 ? last * cs : 0);
  const wide x_lo = x0 + (xs < 0 ? last * xs : 0), x_hi = x0 + x_span + (xs > 0 ? last * xs : 0);
  if (c_lo >= x_hi || x_lo >= c_hi) return {false, false};
  if (c.ld == x.ld && (batch == 1 || (c.stride % c.ld == 0 && x.stride % x.ld == 0))) {
    // column ranges of the rows of one larger matrix
    const wide row = 4 * static_cast<wide>(c.ld);
    wide d = (c0 - x0) % row;
    if (d < 0) d += row;
    if (d >= 4 * static_cast<wide>(x.inner) && d + 4 * static_cast<wide>(c.inner) <= row) return {false, false};
  }
  if (batch == 1) return {true, false};
  if (cs != xs) return {true, true};
  // C_j and X_i, j = i + t: spans meet where -c_span < (c0 - x0) + t * stride < x_span
  Overlap o{c0 - x0 > -c_span && c0 - x0 < x_span, false};
  const wide step = cs < 0 ? -cs : cs;
  if (step == 0) return {o.own, o.own};
  auto down = [](wide a, wide b) { return a >= 0 ? a / b : -((-a + b - 1) / b); };  // floor, b > 0
  wide first = down(-c_span - (c0 - x0), step) + 1, past = -down(-(x_span - (c0 - x0)), step);  // first <= t < past
  if (first < -last) first = -last;
  if (past > last + 1) past = last + 1;
  o.across = past - first > 1 || (past - first == 1 && first != 0);
  return o;
}

}  // namespace tcec_host
