// Shift-reuse implicit-GEMM convolution (device body): any filter of a few
// taps, stride 1 or 2, on the tcgen05 tensor cores straight from the NCHW
// input.
//
//   D[pos][k] = sum over 16-channel blocks cb, taps (r, s) of
//               X16[pos + shift(r, s)][16 channels] . W16[k][16 channels at the tap]
//
// Positions number the outputs of all images on a grid of GX columns and GY
// rows an image, GX and GY a little larger than OW and OH, flat with columns
// fastest.  With the stride split off into planes (plane (a, b) holds input
// rows y = gy * U + a - P and columns x = gx * V + b - Q; stride 1 has one
// plane), tap (r, s) reads plane (r % U, s % V) at position
//   pos + (r / U) * GX + s / V,
// the same shift for every position of a tile.  GX is the smallest width for
// which a shift past the right edge lands on a column of the next row that is
// zero padding where padding is due (GY likewise for rows of the next image),
// so one zero column and one zero row separate neighbours: (W + 1)(H + 1) /
// (W H) of the outputs' positions for 3x3 / stride 1 / pad 1.  Positions past
// OW or OH compute values nobody stores.
//
// So a position tile's input is staged in shared memory ONCE per 16-channel
// block -- its 128 positions plus the shifts' halo -- and every tap reads it
// through a descriptor that starts shift * 16 bytes later: the K-major
// no-swizzle operand is stored as [8-channel half][position][16 bytes], whose
// 8-row groups follow each other without a gap (SBO = 128), so any row may
// start a tile.  Against one staged operand per tap that is 9 * 128 = 1152
// rows down to 128 + 2 GX + 2 per 16 channels of a 3x3 layer (190 at 28x28),
// few enough that the block's own warps bring them in from NCHW and no pre-pass
// over the input is needed.
//
// Those producers read the input as quads of pixels: a channel's plane is
// contiguous, so four consecutive pixels of eight channels are eight 8-byte
// loads whatever the row breaks; each pixel's eight channels then go to its
// position's 16-byte row.  (One pixel and channel per 2-byte load, four times
// the load instructions, left the kernel waiting on them: 1.5 k cycles to
// issue a stage of a 28x28 layer against 1.15 k cycles of its MMAs.)
//
// What bounds it: the tensor cores for C >= 128 (each 16-channel block of a
// stage is R * S MMAs back to back on one staged input), the weight stream
// from L2 beside them -- every CTA reads all its weights once per tile,
// taps * 32 bytes per output channel and 16 channels.  CG = 2 (a cluster of
// two CTAs, M = 256 positions) halves that stream per SM: each CTA holds half
// of the weights' rows and the pair's MMA reads both halves.
//
// Measured (B200): N128 C256 28x28 K256 94 us for the conv alone with L2
// flushed = 1253 TFLOP/s direct (the Winograd two-stage kernels it replaces
// there: 61 + 79 + 54 us).  Whole drop-in calls against the kernels replaced: N64
// C256 14x14 K256 27 us (54), N32 C512 7x7 K512 29 (62), N32 C128 56x56 K128
// stride 2 31 (74, gathering implicit GEMM), N32 C64 56x56 K256 1x1 25 (53).
//
// The weight operand (shift_weight_kernel) is laid out as the stages read it:
// per unit block of output channels and CTA of the unit, 16-channel block by
// 16-channel block, tap by tap, each piece the K-major core-matrix
// interleave (row k, channel c at (k >> 3) * 256 + (c >> 3) * 128 + (k & 7)
// * 16 + (c & 7) * 2).  A stage is then one run (36 KB for a 3x3
// filter at 128 rows a CTA; as at least two stages fit, at most half of SMEM_STAGES)
// and one bulk copy (one per tap issued no faster than a stage per 1.8 k
// cycles; splitting the run over lanes gained nothing).
//
// The reference computes only 3x3 / stride 1 / pad 1 and round-trips V and M
// through HBM (src/preprocessing.cuh:273-424, src/matrixmul.cuh:139-556,
// src/conv2d.cpp:17-250).
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include "tc_sm100.cuh"
#include "wino_common.cuh"
#include "wino_param.h"
#include "wino_batch.h"

namespace wino {
namespace sc {

constexpr int TM = 128;                   // positions per CTA and unit
constexpr int MAXTAP = 64;
constexpr int MAXSTAGE = 8;
constexpr int SMEM_STAGES = 225 * 1024;   // dynamic shared memory of the stages
constexpr int SMEM_BYTES = SMEM_STAGES + 128;
constexpr int NSM = 148;                  // SMs of a B200 (the rules below count units against them)
constexpr int NWARP_Z = 2;
// Warp roles: EW epilogue warps, then MMA issue, weight copies and two warps
// for padding rows, then input producers in two groups of PW warps that take
// alternate stages (or, strided, alternate channel halves of every stage).
// Epilogue and producers are a few hundred instructions a turn which one warp
// issues every ten cycles or so, so their number sets the pace: 28 warps of 72
// registers.  Conv alone back to back, 16 warps -> 28: 1x1 N128 C64 56x56 K256
// 94 -> 66 us, N32 C512 28x28 K128 23 -> 16, 3x3 N32 C64 56x56 K64 21.5 -> 20.2.
constexpr int EW = 8, PW = 8;
constexpr int W_MMA = EW, W_LOAD = EW + 1, W_Z0 = EW + 2, W_P0 = EW + 4;
constexpr int NPROD = PW * 32;            // producers of a group
constexpr int NTHREAD = (W_P0 + 2 * PW) * 32;
constexpr uint32_t SLEEP_NS = 32;
constexpr int BYUNIT = 2;                 // stages a unit up to which producer groups alternate by unit
// Producer items (a quad of pixels and eight channels, four where the input is
// not aligned) a group may own per stage, and operand rows.
constexpr int MAXITEMS = 512, MAXROWS = 1024;

struct Shared {
  uint64_t full[MAXSTAGE], empty[MAXSTAGE];
  uint64_t accfull[2], accempty[2];
  uint64_t mmadone;
  uint32_t tmem_base;
  int abort_flag;
  int aoff[MAXTAP];                       // tap -> operand row offset in the stage
};

// The problem as the kernel sees it.  GX, GY, NB, log2 cps, nstage and qmax
// are worked out on the host and travel packed in the kernel argument's
// transform_pin (no workspace pointer is needed there), the rest follows
// from them in a few operations: the divisions of the rules below cost a
// CTA 6 k cycles before its first load.
struct Plan {
  int N, C, H, W, K, R, S, U, V, P, Q, OH, OW;
  int GX, GY;          // position grid of an image
  int nu, nv;          // planes: nu * nv
  int rows;            // operand rows of a stage per 8 channels, all planes
  int taps, CB, NKS, Kp;
  int lcps, cps, nst;  // 16-channel blocks per stage (a power of two), stages per unit
  int NB, nKU;         // output channels per unit, units per position tile
  int units;
  int stageA, stageB, nstage;
  int pitch;           // bytes from stage to stage
  int qmax, qpi;       // quads of pixels a tile's rows may touch, quads per image
  long long npos;
  // Few input channels (a network's stem): the filter's columns become
  // channels, virtual channel c * S + s being input channel c at column offset
  // s, so that C * S channels and R taps fill K-steps which C channels and R * S
  // taps would leave mostly empty (3 of 16 for an RGB stem).  C, S, V, Q and W
  // above are then the virtual problem's (C * S, 1, 1, 0, OW) and these the real ones.
  bool fold;
  int fC, fS, fV, fQ, fW;
};

// Whether a problem folds: two K-steps hold its virtual channels.
__host__ __device__ __forceinline__ bool folds(int c, int s) { return c <= 8 && s > 1 && s <= 16 && c * s <= 32; }

// Smallest grid extent for `o` outputs with filter extent f, stride st, pad
// pd over an input extent e: a shift past the end must find zero padding on
// both sides (positions GX + j of a row are positions j of the next).
__host__ __device__ __forceinline__ int grid_extent(int o, int f, int st, int pd, int e) {
  const int dmax = (f - 1) / st, np = st < f ? st : f;
  for (int g = o; g < o + dmax; ++g) {
    bool ok = true;
    for (int b = 0; b < np; ++b) {
      const int wrap = o + (f - 1 - b) / st - g;
      for (int j = 0; j < wrap; ++j)
        ok = ok && j < g && j * st + b - pd < 0 && (g + j) * st + b - pd >= e;
    }
    if (ok) return g;
  }
  return o + dmax;
}

__host__ __device__ __forceinline__ int div_stride(int x, int st) { return st == 1 ? x : st == 2 ? x >> 1 : x / st; }

// Operand rows of plane (a, b): the tile's positions and its largest shift.
__host__ __device__ __forceinline__ int plane_rows(const Plan& g, int a, int b) {
  return TM + div_stride(g.R - 1 - a, g.U) * g.GX + div_stride(g.S - 1 - b, g.V);
}

// Cycles of one MMA of N output channels (issue_mmas): its arithmetic, or its
// shared-memory reads; a pair's CTAs read half of B each.
__host__ __device__ __forceinline__ int mma_cycles(int cg, int n) {
  const int reads = 64 + n / (4 * cg), math = n >> 1;
  return reads > math ? reads : math;
}

// What a kernel knows of its problems at compile time.
enum Host : int { OWN, TABLE };       // kernels the schedule runs in: one convolution's, a table's
enum Kind : int { ANY, PLAIN, FOLDED, CONV33 };   // CONV33: 3x3 / stride 1 / pad 1

template <int KIND = ANY>
__host__ __device__ __forceinline__ void plan_dims(Plan& g, const KernelParam& p) {
  g.N = p.n; g.C = p.c; g.H = p.h; g.W = p.w; g.K = p.k;
  if (KIND == CONV33) {
    g.R = g.S = 3;
    g.U = g.V = g.P = g.Q = 1;
    g.OH = g.H; g.OW = g.W;
  } else {
    g.R = p.r; g.S = p.s;
    g.U = p.u; g.V = p.v; g.P = p.p; g.Q = p.q; g.OH = p.Oh; g.OW = p.Ow;
  }
  g.fold = KIND == FOLDED || (KIND == ANY && folds(g.C, g.S));
  if (g.fold) {
    g.fC = g.C; g.fS = g.S; g.fV = g.V; g.fQ = g.Q; g.fW = g.W;
    g.C *= g.S;
    g.S = g.V = 1;
    g.Q = 0;
    g.W = g.OW;
  }
  g.nu = g.U < g.R ? g.U : g.R;
  g.nv = g.V < g.S ? g.V : g.S;
  g.taps = g.R * g.S;
  g.CB = (g.C + 15) >> 4;
  g.NKS = g.taps * g.CB;
  g.Kp = (g.K + 15) & ~15;
  g.qpi = (g.H * g.W + 3) >> 2;
}

// What follows from GX, GY, NB, lcps.
__host__ __device__ __forceinline__ void plan_finish(Plan& g, int cg) {
  g.rows = 0;
  for (int a = 0; a < g.nu; ++a)
    for (int b = 0; b < g.nv; ++b) g.rows += plane_rows(g, a, b);
  // positions up to the last image's last output
  g.npos = ((long long)(g.N - 1) * g.GY + g.OH - 1) * g.GX + g.OW;
  g.nKU = (g.Kp + g.NB - 1) / g.NB;
  g.units = (int)((g.npos + TM * cg - 1) >> (cg == 2 ? 8 : 7)) * g.nKU;
  g.cps = 1 << g.lcps;
  g.nst = (g.CB + g.cps - 1) >> g.lcps;
  const int rows_b = cg == 2 ? ((g.Kp < g.NB ? (g.Kp + 31) & ~31 : g.NB) >> 1) : (g.Kp < g.NB ? g.Kp : g.NB);
  // one more row: where producers drop pixels of a quad that are not the tile's
  g.stageA = (g.cps * g.rows * 32 + 16 + 127) & ~127;
  g.stageB = g.cps * g.taps * rows_b * 32;
  g.pitch = g.stageA + g.stageB;
}

// Items of a producer group and stage.
__host__ __device__ __forceinline__ int stage_items(const Plan& g, bool aligned) {
  const int eights = g.cps * g.qmax * (g.U > 1 || g.V > 1 ? 1 : 2);
  return aligned ? eights : 2 * eights;
}

// Plan of a problem for CG CTAs a unit (host; the rules).
__host__ inline Plan make_plan(const KernelParam& p, int cg, Host host = OWN) {
  Plan g;
  plan_dims(g, p);
  g.GX = grid_extent(g.OW, g.S, g.V, g.Q, g.W);
  g.GY = grid_extent(g.OH, g.R, g.U, g.P, g.H);
  // even rows of outputs on an even grid: pairs of neighbouring outputs then
  // sit on lanes 2i, 2i + 1 and share 4-byte stores
  if ((g.OW & 1) == 0) g.GX = (g.GX + 1) & ~1;
  g.npos = ((long long)(g.N - 1) * g.GY + g.OH - 1) * g.GX + g.OW;
  // Output channels per unit: a wave's time is its MMA time, so the fewest
  // waves x cycles; wide units win ties (less of the input staged twice).
  g.NB = 256;
  if (cg == 1) {
    long long best_t = -1;
    for (int nb = 128; nb >= 32; nb >>= 1) {
      const long long tiles = (g.npos + TM - 1) / TM, un = tiles * ((g.Kp + nb - 1) / nb);
      const long long t = ((un + NSM - 1) / NSM) * mma_cycles(1, g.Kp < nb ? g.Kp : nb);
      if (best_t < 0 || t < best_t) { best_t = t; g.NB = nb; }
    }
  }
  // Quads a tile's rows touch: stride 1, at most the positions' own pixels
  // (padding only lessens them); else whole grid rows.
  int longest = 0;
  for (int a = 0; a < g.nu; ++a)
    for (int b = 0; b < g.nv; ++b) longest = plane_rows(g, a, b) > longest ? plane_rows(g, a, b) : longest;
  const long long lines = (longest + 2 * g.GX - 2) / g.GX;
  // (strided, an image may end in rows that no output reads -- 2x2 / 2 without
  // padding over odd H -- which a tile that runs into the next image steps over)
  const int unread = g.H > g.GY * g.U - g.P ? g.H - (g.GY * g.U - g.P) : 0;
  const long long px = g.U == 1 && g.V == 1 ? longest : (lines * g.U + (lines / g.GY + 1) * unread) * g.W;
  // (images end in a partial quad when H * W is not a multiple of 4)
  const long long imgs = lines / g.GY + 2;
  // (a grid without padding, 1x1: tiles are whole quads)
  const bool odd = (g.H * g.W) % 4 != 0;
  const long long q = g.taps == 1 && g.GX == g.W && g.GY == g.H && !odd && g.U == 1 && g.V == 1
                          ? px / 4 : px / 4 + 2 + (odd ? imgs : 0);
  g.qmax = (int)(q < 4096 ? q : 4096);
  // Several 16-channel blocks a stage where a block has few taps, and two of a
  // 3x3 filter's where four stages still fit (at most 64 output channels a
  // CTA): the producers' and the MMA thread's work per stage then covers twice
  // the MMAs.
  int cps = g.fold ? 2 : g.taps >= 3 ? 2 : 4;
  while (cps > 1 && (cps >> 1) >= g.CB) cps >>= 1;
  for (;; cps >>= 1) {
    g.lcps = cps == 4 ? 2 : cps == 2 ? 1 : 0;
    plan_finish(g, cg);
    // (a folded problem's unit is one stage; else an item a producer, two of the
    // smaller unaligned ones: N32 C512 7x7 K512 28.0 -> 25.1 us)
    if (cps == 1 || g.fold || (stage_items(g, !odd) <= (odd && host == OWN ? 512 : 256) &&
                               (g.taps >= 6 ? 4 : 3) * (g.stageA + g.stageB) <= SMEM_STAGES))
      break;
  }
  const int fit = SMEM_STAGES / (g.stageA + g.stageB);
  g.nstage = fit < MAXSTAGE ? fit : MAXSTAGE;
  return g;
}

// Whether every channel's quads of pixels are 8-byte words.
__host__ __device__ __forceinline__ bool input_aligned(int hw, const void* x) {
  return (hw & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 7) == 0;
}

// Whether the 8-byte words around unaligned quads may reach outside the input:
// it starts or ends inside such a word.
__host__ inline bool input_edges(const KernelParam& p) {
  const unsigned long long total = 2ull * p.n * p.c * p.h * p.w;
  return ((reinterpret_cast<uintptr_t>(p.pin) | total) & 7) != 0;
}

// Bytes from the first pixel of an item of `ch` channels to the end of the last
// word it loads (saturated: more than any input).
__host__ __device__ __forceinline__ uint32_t item_span(uint32_t plane, int ch) {
  const unsigned long long b = (unsigned long long)(ch - 1) * plane + 16;
  return b < 0xffffffffull ? (uint32_t)b : 0xffffffffu;
}

// Whether an unaligned item's words, the first pixel `o` bytes into an input of
// `total` bytes that starts `head` bytes past a word, may be such ones.
__host__ __device__ __forceinline__ bool item_at_edge(uint32_t o, uint32_t head, uint32_t total, uint32_t span) {
  return total - o < span || (head != 0 && o < 8);
}

__host__ inline unsigned long long pack_plan(const Plan& g) {
  return (unsigned long long)g.GX | (unsigned long long)g.GY << 16 | (unsigned long long)(g.NB / 16) << 32 |
         (unsigned long long)g.lcps << 40 | (unsigned long long)g.nstage << 44 | (unsigned long long)g.qmax << 48;
}

template <int KIND = ANY>
__device__ __forceinline__ Plan unpack_plan(const KernelParam& p, int cg) {
  Plan g;
  plan_dims<KIND>(g, p);
  const unsigned long long w = reinterpret_cast<unsigned long long>(p.transform_pin);
  g.GX = (int)(w & 0xffff);
  g.GY = (int)(w >> 16 & 0xffff);
  g.NB = (int)(w >> 32 & 0xff) * 16;
  g.lcps = (int)(w >> 40 & 15);
  g.nstage = (int)(w >> 44 & 15);
  g.qmax = (int)(w >> 48);
  plan_finish(g, cg);
  return g;
}

// One convolution of a launch as one CTA sees it: its plan and tensors, this
// CTA's first unit and number of units.
struct Conv {
  Plan g;
  const unsigned short* x;
  __half* y;
  const uint8_t* wop;      // weight operand
  int u0, cnt;
};

// A launch over one convolution (its argument carries the packed plan).  EDGES:
// its input starts or ends inside an 8-byte word (input_edges), whose pixels the
// producers then load one by one; kernels of their own, as the few more
// registers cost the others 5 % (N32 C512 7x7 K512 29.3 -> 30.7 us).
template <int KIND, bool EDGES = false>
struct OneConv {
  static constexpr int kind = KIND;
  static constexpr bool edges = EDGES;
  static constexpr bool table = false;
  const KernelParam& p;
  __device__ __forceinline__ int layers() const { return 1; }
  __device__ __forceinline__ bool strided() const { return KIND == PLAIN && (p.u > 1 || p.v > 1); }
  __device__ __forceinline__ bool get(int, int cg, int u, int step, Conv& c) const {
    c.g = unpack_plan<KIND>(p, cg);
    c.x = static_cast<const unsigned short*>(p.pin);
    c.y = static_cast<__half*>(p.pout);
    c.wop = static_cast<const uint8_t*>(p.transform_filter);
    c.u0 = u;
    c.cnt = u < c.g.units ? (c.g.units - 1 - u) / step + 1 : 0;
    return c.cnt > 0;
  }
};

// ... and over a table of them, units numbered through (wino_batch.h): the
// ring of stages runs on across layers, so its pitch is the largest stage's.
struct ConvTable {
  static constexpr int kind = CONV33;
  // An item a producer: with two for some layers too, the producers' variants
  // spilled into an L1 cache that the stages leave little of (N32 C512 7x7
  // K512 with its operand 69 -> 37 us, the set's eight layers N32 186 -> 130).
  static constexpr bool table = true, edges = false;
  const ShiftTable& t;                    // the kernel's argument (constant bank)
  __device__ __forceinline__ int layers() const { return t.nlayers; }
  __device__ __forceinline__ bool strided() const { return false; }
  __device__ __forceinline__ bool get(int l, int cg, int u, int step, Conv& c) const {
    const ShiftLayer& d = t.layer[l];
    // first unit of the layer that is u modulo step
    const int begin = d.unit_begin, skip = (u - begin % step + step) % step;
    c.u0 = skip;
    c.cnt = skip < d.units ? (d.units - 1 - skip) / step + 1 : 0;
    if (c.cnt == 0) return false;
    c.g = unpack_plan<CONV33>(d.p, cg);
    c.g.pitch = t.pitch;
    c.g.nstage = t.nstage;
    c.x = static_cast<const unsigned short*>(d.p.pin);
    c.y = static_cast<__half*>(d.p.pout);
    c.wop = static_cast<const uint8_t*>(d.p.transform_filter);
    return true;
  }
};

// Position in the ring of stages; a waiter for empty stages starts in phase
// 1 (the first pass over the ring is free), one for full stages in phase 0.
struct RingPos {
  int st;
  uint32_t phase;
  __device__ __forceinline__ void next(int nstage, int by = 1) {
    for (st += by; st >= nstage; st -= nstage) phase ^= 1;
  }
};

// Rows of the weight operand one CTA of a unit holds (the unit's output
// channels k0 .., padded to the MMA's granularity).
__host__ __device__ __forceinline__ int unit_n(const Plan& g, int cg, int k0) {
  const int n = g.Kp - k0 < g.NB ? g.Kp - k0 : g.NB;
  return cg == 2 ? (n + 31) & ~31 : n;
}

// Bytes of the weight operand.
__host__ __device__ __forceinline__ size_t weight_bytes(const Plan& g, int cg) {
  const int last = (g.nKU - 1) * g.NB;
  return (size_t)(last + unit_n(g, cg, last)) * g.NKS * 32;
}

// n / d for 0 <= n < 2^31: m = ceil(2^32 / d) overestimates the quotient by
// at most one.
struct Div {
  unsigned m;
  int d;
};
__device__ __forceinline__ Div make_div(int d) { return Div{0xffffffffu / (unsigned)d + 1u, d}; }
__device__ __forceinline__ int quot(int n, const Div& v) {
  if (v.d == 1) return n;
  const int q = (int)__umulhi((unsigned)n, v.m);
  return q * v.d > n ? q - 1 : q;
}

// Unit u: position tile and output-channel block (k-blocks of one position
// tile on neighbouring CTAs, so its input comes from L2 the second time).
__device__ __forceinline__ void unit_of(const Plan& g, int u, int& pt, int& k0) {
  pt = g.nKU == 1 ? u : (int)((unsigned)u / (unsigned)g.nKU);
  k0 = (u - pt * g.nKU) * g.NB;
}

// t / d for 0 <= t < 2^20, with rd = 1.0f / d: (t + 1/2) / d is at least
// 1 / (2 d) away from a whole number, more than the product's rounding error.
__device__ __forceinline__ int small_div(int t, float rd) { return __float2int_rz(((float)t + 0.5f) * rd); }

// Grid coordinates of a tile's first position, and of the position o later.
struct Base {
  int n, gy, gx;
};
struct Grid {
  Div gx, gy;
  float rgx, rgy;
};
__device__ __forceinline__ Grid make_grid(const Plan& g) {
  return Grid{make_div(g.GX), make_div(g.GY), 1.0f / (float)g.GX, 1.0f / (float)g.GY};
}
__device__ __forceinline__ Base tile_base(const Grid& gr, int pos0) {
  Base b;
  const int line = quot(pos0, gr.gx);
  b.gx = pos0 - line * gr.gx.d;
  b.n = quot(line, gr.gy);
  b.gy = line - b.n * gr.gy.d;
  return b;
}
__device__ __forceinline__ Base advance(const Grid& gr, const Base& b, int o) {
  Base r;
  const int t = b.gx + o, dl = small_div(t, gr.rgx);
  r.gx = t - dl * gr.gx.d;
  const int l = b.gy + dl, dn = small_div(l, gr.rgy);
  r.gy = l - dn * gr.gy.d;
  r.n = b.n + dn;
  return r;
}

// All of the block's threads (both CTAs' with CG = 2), each role from its own
// place: barriers initialised and TMEM allocated before anyone relies on them.
template <int CG>
__device__ __forceinline__ void setup_sync() {
  tc_fence_before();
  __syncwarp();
  if (CG == 2) cluster_sync();
  else asm volatile("bar.sync 0;" ::: "memory");
  tc_fence_after();
}

// Every lane polls (no broadcast behind the poll); the outcome is the warp's.
template <bool kCluster = false>
__device__ __forceinline__ bool wait_all_lanes(uint64_t* bar, uint32_t parity, volatile int* abort, uint32_t* err,
                                               uint32_t code) {
  return __all_sync(0xffffffffu, mbar_wait_impl<kCluster>(bar, parity, abort, err, code)) != 0;
}

// Whether producer groups alternate by unit (a run of nst stages; two rounds of
// the ring are apart as long as that is not all of it).
__device__ __forceinline__ bool runs_by_unit(const Plan& g) { return g.nst <= BYUNIT && g.nst < g.nstage; }

// One stage's loads of a producer thread, and where they go.
template <int NI, int NW, int CH>
struct Slot {
  uint2 w[NI][CH][NW];
  uint2 row[NI];                          // 16-byte rows of the stage its pixels go to, 16 bits each, store order
  uint32_t shifts;                        // unaligned quads: first pixel's place in its 8-byte word, 4 bits an item
};

// Input producers with NI items a thread and stage, one stage of loads ahead
// of the stores.  An item is (8-channel group of the
// stage, quad of the tile's pixel range), quads fastest, so a warp's loads
// are 256-byte runs of a channel's plane.  ALIGNED: a quad is one 8-byte
// word of every channel (input 8-byte aligned, H * W a multiple of 4);
// otherwise the two words around it and a shift.
// The two groups take alternate stages, or with few stages a unit alternate
// units (each then works out every other unit's addresses only): a group's
// stages are `run` in a row, then `run` skipped, from layer to layer too
// (`turn`: the group whose turn the layer's first run is; done: stages of the
// layers before).  A group must not skip a whole round of the ring: the empty
// barrier's parity it then waits for could be two rounds old.
// Strided, a stage's pixels are many and each group takes one channel half of
// every stage.
// EDGES: items whose words may reach outside the input load pixel by pixel.
template <int CG, int NI, bool ALIGNED, bool STRIDED, bool EDGES>
__device__ __forceinline__ bool produce(const Conv& cv, uint8_t* smem, Shared& sh, int tid, int group, int done, int turn,
                                        int ustep, int tile_pos, int tile_stride, bool& set, uint32_t* err) {
  const Plan& g = cv.g;
  const int u0 = cv.u0, cnt = cv.cnt;
  constexpr int NW = ALIGNED ? 1 : 2;     // 8-byte words per channel
  // channels of an item: two words a channel are many registers
  constexpr int CH = ALIGNED ? 8 : 4;
  volatile int* abort_flag = &sh.abort_flag;
  const unsigned short* X = cv.x;
  const int HW = g.H * g.W, ngrp = 2 * g.cps;
  const uint32_t trash = (uint32_t)(ngrp * g.rows);
  const Grid gr = make_grid(g);
  const float rw = 1.0f / (float)g.W, rqpi = 1.0f / (float)g.qpi;
  const int ushift = STRIDED ? g.U - 1 : 0, vshift = STRIDED ? g.V - 1 : 0;      // strides 1 and 2
  // Pixel order of this lane's stores: pixel k ^ rot k-th, so that the eight
  // lanes of a 16-byte store phase, whose quads are 64 bytes apart, meet in
  // pairs on a bank rather than in fours (all four orders would part them, at
  // 16 selects an item; a producer warp's instructions are what this role
  // waits for).
  const int rot = (tid >> 1) & 1;
  const uint32_t sel0 = rot ? 0x7632u : 0x5410u, sel1 = rot ? 0x5410u : 0x7632u;
  int iq[NI], ich[NI];                    // quad (-1: none) and first channel of the stage
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int idx = tid + i * NPROD, grp = idx / g.qmax;   // channel group of the stage (strided: of its half)
    iq[i] = grp < (STRIDED ? g.cps : ngrp) * (8 / CH) ? idx - grp * g.qmax : -1;
    ich[i] = STRIDED ? (grp * CH >> 3) * 16 + group * 8 + (grp * CH & 7) : grp * CH;
  }
  // planes by (row parity, column parity): first operand row, rows (0: none)
  constexpr int NPL = STRIDED ? 4 : 1;
  int pbase[NPL], prow[NPL];
  {
    int r = 0;
#pragma unroll
    for (int pl = 0; pl < NPL; ++pl) {
      const int a = pl >> vshift, b = pl & vshift;
      const bool there = a <= ushift && a < g.nu && b < g.nv;
      pbase[pl] = r;
      prow[pl] = STRIDED ? (there ? plane_rows(g, a, b) : 0) : g.rows;
      r += prow[pl];
    }
  }
  uint32_t off[NI];                       // byte offset of the quad in the input, channel 0
  int npx[NI];                            // its pixels inside the image (0: no pixel of the tile's)
  uint2 row_l[NI];
  // load and store cursors: stage of the layer (unit lu, stage lj), ring slot
  const bool by_unit = runs_by_unit(g);
  const int stages = cnt * g.nst;
  const int run = STRIDED ? stages : by_unit ? g.nst : 1;
  const int first = STRIDED ? 0 : (group ^ turn) * run;
  int lu = 0, lj = first;
  while (lj >= g.nst) { lj -= g.nst; ++lu; }
  int s_left = run, l_left = run;         // stages left of the run
  RingPos pos;
  pos.st = (done + first) % g.nstage;
  pos.phase = 1u ^ (uint32_t)(((done + first) / g.nstage) & 1);
  int entered = -1;
  const bool whole = (g.C & 15) == 0;     // no channel of a block is missing
  const char* XB = reinterpret_cast<const char*>(X);
  Slot<NI, NW, CH> slot;
  auto enter = [&]() {
    int pt, k0;
    unit_of(g, u0 + lu * ustep, pt, k0);
    const Base b0 = tile_base(gr, pt * tile_stride + tile_pos);
    // (a pair's second tile may start past the last image: its loads, of which
    // no row is stored, stay inside)
    const uint32_t img = (uint32_t)(min(b0.n, g.N - 1) * g.C) * (uint32_t)HW * 2u;
    // the range starts with the first position's pixel (stride 1) or the
    // first pixel row of its grid row
    const int y0 = (b0.gy << ushift) - g.P;
    int lo = y0 * g.W;
    if (!STRIDED) lo += min(max(b0.gx - g.Q, 0), g.W);
    lo = min(max(lo, 0), HW);
    const int q0 = lo >> 2, yb = max(y0, 0);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      off[i] = img;                       // (a quad without pixels loads what is there)
      npx[i] = 0;
      row_l[i].x = row_l[i].y = trash | trash << 16;
      if (iq[i] < 0) continue;
      int q = q0 + iq[i], dn = 0;
      if (q >= g.qpi) {
        q -= g.qpi;
        dn = small_div(q, rqpi);
        q -= dn * g.qpi;
        ++dn;
      }
      if (b0.n + dn >= g.N) continue;
      const int i0 = q * 4;
      // pixel row and column, from the row the range starts in (rel >= -3)
      const int rel = dn == 0 ? i0 - yb * g.W : i0;
      const int dy = rel < 0 ? -1 : small_div(rel, rw);
      int y = (dn == 0 ? yb : 0) + dy, x = rel - dy * g.W;
      while (x < 0) { x += g.W; --y; }    // images narrower than the overhang
      bool any = false;
      uint32_t d[4];
      if (!STRIDED) {
        // rows of consecutive pixels are consecutive but for the padding
        // between image rows (at stride 1 the grid has room for every pixel:
        // GX >= W + Q, GY >= H + P)
        const int r0 = (dn * g.GY + y + g.P - b0.gy) * g.GX + x + g.Q - b0.gx;
        const int first_row = (ich[i] >> 3) * g.rows;
#pragma unroll
        for (int px = 0; px < 4; ++px) {
          int r = r0 + px;
          if (g.W >= 4) {
            if (px >= g.W - x) r += g.GX - g.W;
          } else {
            r += (x + px) / g.W * (g.GX - g.W);
          }
          const bool in = (unsigned)r < (unsigned)g.rows && (ALIGNED || i0 + px < HW);
          d[px] = in ? (uint32_t)(first_row + r) : trash;
          any = any || in;
        }
      } else {
#pragma unroll
        for (int px = 0; px < 4; ++px) {
          d[px] = trash;
          const int yy = y + g.P, xx = x + g.Q;
          const int gy = yy >> ushift, gx = xx >> vshift;
          const int pl = ((yy & ushift) << vshift) | (xx & vshift);
          int pb = pbase[0], pr = prow[0];
#pragma unroll
          for (int z = 1; z < NPL; ++z)
            if (pl == z) { pb = pbase[z]; pr = prow[z]; }
          const int r = (dn * g.GY + gy - b0.gy) * g.GX + gx - b0.gx;
          if (i0 + px < HW && gx < g.GX && gy < g.GY && r >= 0 && r < pr) {
            d[px] = (uint32_t)((ich[i] >> 3) * g.rows + pb + r);
            any = true;
          }
          if (++x == g.W) { x = 0; ++y; }
        }
      }
      // stored in the order px ^ rot
      row_l[i] = make_uint2(__byte_perm(d[0], d[1], rot ? 0x1054 : 0x5410), __byte_perm(d[2], d[3], rot ? 0x1054 : 0x5410));
      if (any) {
        npx[i] = min(4, HW - i0);
        off[i] = img + (uint32_t)(dn * g.C * HW + i0) * 2u;
      }
    }
  };
  auto issue = [&](Slot<NI, NW, CH>& s) {
    const int c0 = lj << (g.lcps + 4);
    const uint32_t plane = (uint32_t)HW * 2u;
    uint32_t shifts = 0;
    if (ALIGNED && whole) {
      // Channels past C are those of a block no MMA reads.
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int c = c0 + ich[i];
        uint32_t o = off[i] + (c < g.C ? (uint32_t)c * plane : 0u);
        s.row[i] = row_l[i];
#pragma unroll
        for (int e = 0; e < CH; ++e, o += plane) s.w[i][e][0] = __ldg(reinterpret_cast<const uint2*>(XB + o));
      }
    } else {
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int c = c0 + ich[i], nc = npx[i] > 0 ? g.C - c : 0;   // channels to load
        uint32_t o = off[i] + (nc > 0 ? (uint32_t)c * plane : 0u);
        s.row[i] = row_l[i];
        if (!ALIGNED) shifts |= ((uint32_t)(reinterpret_cast<uintptr_t>(XB + o) >> 1) & 3u) << (4 * i);
        if constexpr (EDGES) {
          const uint32_t head = (uint32_t)reinterpret_cast<uintptr_t>(XB) & 7u;
          if (nc > 0 && item_at_edge(o, head, (uint32_t)(g.N * g.C) * plane, item_span(plane, CH))) {
#pragma unroll
            for (int e = 0; e < CH; ++e, o += plane) {
              unsigned long long px = 0;
#pragma unroll
              for (int k = 0; k < 4; ++k)
                if (e < nc && k < npx[i])
                  px |= (unsigned long long)__ldg(reinterpret_cast<const unsigned short*>(XB + o) + k) << (16 * k);
              // where the two words around them would hold them
              const uint32_t by = ((head + o) & 6u) * 8u;
              const unsigned long long w0 = px << by, w1 = by ? px >> (64 - by) : 0;
              s.w[i][e][0] = make_uint2((uint32_t)w0, (uint32_t)(w0 >> 32));
              s.w[i][e][NW - 1] = make_uint2((uint32_t)w1, (uint32_t)(w1 >> 32));
            }
            continue;
          }
        }
#pragma unroll
        for (int e = 0; e < CH; ++e, o += plane) {
          const bool on = e < nc;
          if (ALIGNED) {
            s.w[i][e][0] = on ? __ldg(reinterpret_cast<const uint2*>(XB + o)) : make_uint2(0, 0);
          } else {
            const uintptr_t ad = reinterpret_cast<uintptr_t>(XB + o);
            const uint2* wp = reinterpret_cast<const uint2*>(ad & ~uintptr_t(7));
            s.w[i][e][0] = on ? __ldg(wp) : make_uint2(0, 0);
            // the next word only where it holds a pixel of the quad
            s.w[i][e][NW - 1] = on && ((int)(ad >> 1) & 3) + npx[i] > 4 ? __ldg(wp + 1) : make_uint2(0, 0);
          }
        }
      }
    }
    s.shifts = shifts;
  };
  auto consume = [&](const Slot<NI, NW, CH>& s) -> bool {
    if (!wait_all_lanes(&sh.empty[pos.st], pos.phase, abort_flag, err, ERR_WAIT_EMPTY)) return false;
    uint8_t* dst = smem + pos.st * g.pitch;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      uint32_t lo[CH], hi[CH];            // pixels 0, 1 and 2, 3 of the channels
#pragma unroll
      for (int e = 0; e < CH; ++e) {
        uint32_t a = s.w[i][e][0].x, b = s.w[i][e][0].y;
        if (!ALIGNED) {
          const uint32_t sh16 = ((s.shifts >> (4 * i)) + (uint32_t)(e * HW)) & 3u;
          uint32_t t0 = a, t1 = b, t2 = s.w[i][e][NW - 1].x;
          if (sh16 & 2u) { t0 = b; t1 = s.w[i][e][NW - 1].x; t2 = s.w[i][e][NW - 1].y; }
          a = sh16 & 1u ? __byte_perm(t0, t1, 0x5432) : t0;
          b = sh16 & 1u ? __byte_perm(t1, t2, 0x5432) : t1;
        }
        lo[e] = a;
        hi[e] = b;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t rw2 = k < 2 ? s.row[i].x : s.row[i].y, r = k & 1 ? rw2 >> 16 : rw2 & 0xffffu;
        const uint32_t sel = k & 1 ? sel1 : sel0;
        const uint32_t* v = k < 2 ? lo : hi;
        const uint32_t a = __byte_perm(v[0], v[1], sel), b = __byte_perm(v[2], v[3], sel);
        if (CH == 8)
          *reinterpret_cast<uint4*>(dst + r * 16) =
              make_uint4(a, b, __byte_perm(v[CH - 4], v[CH - 3], sel), __byte_perm(v[CH - 2], v[CH - 1], sel));
        else
          *reinterpret_cast<uint2*>(dst + r * 16 + (ich[i] & 4) * 2) = make_uint2(a, b);
      }
    }
    fence_proxy_async_shared();
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(&sh.full[pos.st]);
    int by = 1;
    if (--s_left == 0) { s_left = run; by += run; }
    pos.next(g.nstage, by);
    return true;
  };
  // Turn t stores the loads of the turn before and issues new ones.  One loop
  // body: unrolled, the unit entry above was compiled in several times and its
  // first pass through the instruction cache held the first stage up by 10 us.
  const int total = STRIDED ? stages : ((by_unit ? cnt : stages) - (group ^ turn) + 1) / 2 * run;
  bool ok = true;
  for (int t = 0; ok && t <= total; ++t) {
    // the first loads go out before the block's setup is complete
    if (t == 1 && !set) {
      setup_sync<CG>();
      set = true;
    }
    const bool more = t < total;
    if (more && lu != entered) {
      enter();
      entered = lu;
    }
    if (t > 0) ok = consume(slot);
    if (more && ok) issue(slot);
    int by = 1;
    if (--l_left == 0) { l_left = run; by += run; }
    for (lj += by; lj >= g.nst; lj -= g.nst) ++lu;
  }
  return ok;
}

// Producers of a folded problem (Plan): thread = operand row, a position's
// C * S values gathered with 2-byte loads (lanes on neighbouring output
// columns) into up to four 16-byte words.  N32 224x224 RGB 7x7 / 2
// K64 takes 61 us, waiting on these gathers (CUDA-core direct kernel: 590 us;
// its bytes take 9).  A unit is one stage and the groups
// take alternate units.  FC, FS: channels and columns known at compile time
// (0: as the plan says).
template <int CG, int FC, int FS>
__device__ __forceinline__ bool produce_fold(const Conv& cv, uint8_t* smem, Shared& sh, int tid, int group, int ustep,
                                             int tile_pos, int tile_stride, uint32_t* err) {
  const Plan& g = cv.g;
  volatile int* abort_flag = &sh.abort_flag;
  const int C = FC ? FC : g.fC, S = FC ? FS : g.fS, HW = g.H * g.fW, ngrp = 2 * g.cps;
  const Grid gr = make_grid(g);
  const int plane0 = plane_rows(g, 0, 0);
  RingPos pos{group % g.nstage, 1u ^ (uint32_t)((group / g.nstage) & 1)};
  for (int i = group; i < cv.cnt; i += 2, pos.next(g.nstage, 2)) {
    int pt, k0;
    unit_of(g, cv.u0 + i * ustep, pt, k0);
    const Base b0 = tile_base(gr, pt * tile_stride + tile_pos);
    if (!wait_all_lanes(&sh.empty[pos.st], pos.phase, abort_flag, err, ERR_WAIT_EMPTY)) return false;
    uint8_t* dst = smem + pos.st * g.pitch;
#pragma unroll 1
    for (int r = tid; r < g.rows; r += NPROD) {
      const int a = r >= plane0 ? 1 : 0;
      const Base c = advance(gr, b0, r - (a ? plane0 : 0));
      const int y = c.gy * g.U + a - g.P, x0 = c.gx * g.fV - g.fQ;
      // columns s of the filter that lie in the image
      const int lo = max(0, -x0), hi = min(S, g.fW - x0);
      uint32_t in = c.n < g.N && (unsigned)y < (unsigned)g.H && c.gx < g.OW && hi > lo
                        ? ((1u << hi) - 1u) & ~((1u << lo) - 1u) : 0u;
      const unsigned short* src = cv.x + ((long long)(c.n * C) * HW + (long long)y * g.fW + x0);
      if (FC) {
        uint32_t v[32];
#pragma unroll
        for (int ch = 0; ch < FC; ++ch)
#pragma unroll
          for (int s = 0; s < FS; ++s) {
            uint32_t e = 0;
            if (in >> s & 1u) e = __ldg(src + ch * HW + s);
            v[ch * FS + s] = e;
          }
#pragma unroll
        for (int e = FC * FS; e < 32; ++e) v[e] = 0;
#pragma unroll
        for (int grp = 0; grp < 4; ++grp)
          if (grp < ngrp)
            *reinterpret_cast<uint4*>(dst + (grp * g.rows + r) * 16) =
                make_uint4(v[8 * grp] | v[8 * grp + 1] << 16, v[8 * grp + 2] | v[8 * grp + 3] << 16,
                           v[8 * grp + 4] | v[8 * grp + 5] << 16, v[8 * grp + 6] | v[8 * grp + 7] << 16);
      } else {
        int ch = 0, s = 0;
        for (int grp = 0; grp < ngrp; ++grp) {
          uint32_t v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            v[e] = ch < C && (in >> s & 1u) ? (uint32_t)__ldg(src + ch * HW + s) : 0u;
            if (++s == S) { s = 0; ++ch; }
          }
          *reinterpret_cast<uint4*>(dst + (grp * g.rows + r) * 16) =
              make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
        }
      }
    }
    fence_proxy_async_shared();
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(&sh.full[pos.st]);
  }
  return true;
}

// Padding rows of the operand (two warps): the zero columns and rows of a
// tile's positions, written to every stage (a slot's last tile had them
// elsewhere).
__device__ __forceinline__ bool pad_rows(const Conv& cv, uint8_t* smem, Shared& sh, int tid, int ustep, int tile_pos,
                                         int tile_stride, RingPos& pos, uint32_t* err) {
  const Plan& g = cv.g;
  constexpr int NT = NWARP_Z * 32;
  volatile int* abort_flag = &sh.abort_flag;
  const Grid gr = make_grid(g);
  const int ngrp = 2 * g.cps;
  for (int i = 0; i < cv.cnt; ++i) {
    int pt, k0;
    unit_of(g, cv.u0 + i * ustep, pt, k0);
    const Base b0 = tile_base(gr, pt * tile_stride + tile_pos);
    uint32_t zero = 0;                    // bit z: row tid + z * NT is padding
    int pbase = 0;
    for (int a = 0; a < g.nu; ++a)
      for (int b = 0; b < g.nv; ++b) {
        const int pr = plane_rows(g, a, b);
        for (int z = 0, r = tid - pbase; r < pr; ++z, r += NT) {
          if (r < 0) continue;
          const Base c = advance(gr, b0, r);
          const int y = c.gy * g.U + a - g.P, x = c.gx * g.V + b - g.Q;
          if (!(c.n < g.N && (unsigned)y < (unsigned)g.H && (unsigned)x < (unsigned)g.W)) zero |= 1u << z;
        }
        pbase += pr;
      }
    for (int j = 0; j < g.nst; ++j) {
      if (!wait_all_lanes(&sh.empty[pos.st], pos.phase, abort_flag, err, ERR_WAIT_EMPTY)) return false;
      uint8_t* dst = smem + pos.st * g.pitch + tid * 16;
      for (uint32_t m = zero; m != 0; m &= m - 1)
        for (int grp = 0; grp < ngrp; ++grp)
          *reinterpret_cast<uint4*>(dst + (grp * g.rows + (__ffs(m) - 1) * NT) * 16) = make_uint4(0, 0, 0, 0);
      fence_proxy_async_shared();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&sh.full[pos.st]);
      pos.next(g.nstage);
    }
  }
  return true;
}

// Operand row at which tap (r, s) starts reading a stage: its plane's first
// row plus its shift.
__device__ __forceinline__ int tap_row(const Plan& g, int r, int s) {
  const int dr = div_stride(r, g.U), ds = div_stride(s, g.V), a = r - dr * g.U, b = s - ds * g.V;
  int base = 0;
  for (int x = 0; x <= a; ++x)
    for (int z = 0; z < (x < a ? g.nv : b); ++z) base += plane_rows(g, x, z);
  return base + dr * g.GX + ds;
}

// MMA issue: per stage and 16-channel block one MMA a tap, all on the same
// staged input.  The whole warp runs the loop and one elected lane issues, so
// descriptors stay in uniform registers (from one lane's branch a stage of
// nine took 960 cycles to issue against 800).  An MMA here costs its
// shared-memory reads: 64 cycles for the 128 rows of A, which a shift takes
// off the 128-byte lines, plus a cycle per 4 rows of B (N = 64: 80 cycles a
// CTA; a pair's N = 256 is at its arithmetic 128).  The pipe takes an MMA ahead at most, so what the thread
// does between stages shows: the next stage's barrier is polled in the middle
// of a stage, and only if it was not ready then is it waited for.  TAPS > 0:
// that many taps, their shifts kept in registers.
template <int CG, int TAPS>
__device__ __forceinline__ bool issue_mmas(const Conv& cv, Shared& sh, uint32_t sbase, uint32_t tmem, int ustep,
                                           bool leader, RingPos& pos, int& unit, bool& ready, uint32_t* err) {
  const Plan& g = cv.g;
  constexpr uint16_t BOTH = 3;
  constexpr int NOFF = TAPS > 0 ? TAPS : 1;
  volatile int* abort_flag = &sh.abort_flag;
  const uint32_t stage16 = (uint32_t)g.pitch >> 4, a16 = (uint32_t)g.stageA >> 4;
  const uint64_t adesc0 = smem_desc(sbase, (uint32_t)g.rows * 16, 128), bdesc0 = smem_desc(sbase, 128, 256) + a16;
  const uint32_t qstep = (uint32_t)g.rows * 2;
  uint32_t off[NOFF];
#pragma unroll
  for (int t = 0; t < NOFF; ++t) off[t] = (uint32_t)__shfl_sync(0xffffffffu, sh.aoff[t], 0);
  int st = pos.st;
  uint32_t phase = pos.phase, s16 = (uint32_t)st * stage16;
  bool ok = true;
  for (int i = 0; ok && i < cv.cnt; ++i, ++unit) {
    int pt, k0;
    unit_of(g, cv.u0 + i * ustep, pt, k0);
    const int nn = unit_n(g, CG, k0);
    const uint32_t idesc = instr_desc(CG * 128, (uint32_t)nn, 0, 0, 0, 0);
    const uint32_t bstep = (uint32_t)((nn / CG) * 32) >> 4;
    const int ab = unit & 1;
    if (unit >= 2) {
      ok = wait_all_lanes<CG == 2>(&sh.accempty[ab], ((unit >> 1) - 1) & 1, abort_flag, err, ERR_WAIT_DRAIN);
      if (!ok) break;
    }
    tc_fence_after();
    const uint32_t d = tmem + ab * 256;
    auto mma = [&](uint64_t ad, uint64_t bd, uint32_t acc) {
      if (leader) {
        if (CG == 2) mma_f16_pair(d, ad, bd, idesc, acc);
        else mma_f16(d, ad, bd, idesc, acc);
      }
    };
    for (int j = 0; j < g.nst; ++j) {
      if (!ready) {
        ok = wait_all_lanes<CG == 2>(&sh.full[st], phase, abort_flag, err, ERR_WAIT_FULL);
        if (!ok) break;
      }
      tc_fence_after();
      const int nk = min(g.cps, g.CB - j * g.cps);
      const int nst_ = st + 1 == g.nstage ? 0 : st + 1;
      const uint32_t nphase = nst_ == 0 ? phase ^ 1 : phase;
      auto poll = [&]() {
        ready = __all_sync(0xffffffffu, mbar_test_wait<CG == 2>(&sh.full[nst_], nphase)) != 0;
      };
      uint64_t aq = adesc0 + s16, bd = bdesc0 + s16;
      for (int q = 0; q < nk; ++q, aq += qstep) {
        if (TAPS > 0) {
#pragma unroll
          for (int t = 0; t < TAPS; ++t, bd += bstep) {
            mma(aq + off[t], bd, t > 0 || j > 0 || q > 0 ? 1u : 0u);
            if (t == TAPS / 2 && q + 1 == nk) poll();
          }
        } else {
          if (q + 1 == nk) poll();
#pragma unroll 4
          for (int t = 0; t < g.taps; ++t, bd += bstep)
            mma(aq + (uint32_t)sh.aoff[t], bd, t > 0 || j > 0 || q > 0 ? 1u : 0u);
        }
      }
      if (leader) {
        if (CG == 2) mma_commit_pair(&sh.empty[st], BOTH);
        else mma_commit(&sh.empty[st]);
      }
      st = nst_;
      phase = nphase;
      s16 = st == 0 ? 0 : s16 + stage16;
    }
    if (ok && leader) {
      if (CG == 2) mma_commit_pair(&sh.accfull[ab], BOTH);
      else mma_commit(&sh.accfull[ab]);
    }
  }
  pos.st = st;
  pos.phase = phase;
  return ok;
}

// Whether outputs (and residuals) are stored in pairs.
__host__ __device__ __forceinline__ bool store_pairs(int ow, const void* y, const void* residual) {
  return (ow & 1) == 0 && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(residual)) & 3) == 0;
}

// Epilogue operands of the fused form: y = relu?(conv + bias[k] + residual).
struct Epi {
  const float* bias;
  const __half* residual;  // y's layout
  int relu;
};

// Stores NC accumulator columns (output channels) of a position per lane:
// column c < lim of this lane goes to byte offset o + c * step of Y (32-bit
// offsets: an output of 4 GB or more is not this kernel's).  With `pair` the
// lanes 2i and 2i + 1 hold neighbouring outputs of one row, live together:
// two columns are rounded into one word, the pair swaps words, and each lane
// stores one column of both -- a conversion, a shuffle, a byte permute, an
// add and a 4-byte store for two columns (40 -> 25 cycles a column of a 128 x
// 256 unit against float shuffles and 64-bit addresses).
// Epilogue: + bias (rounded to fp16), + residual in fp32, ReLU last; a kernel
// for even rows of 4-byte aligned outputs and one for others.  The residuals
// `rv` of the columns come from load_cols, ahead of the accumulators: a load
// between stores waits for them, as they may alias (N8 C32 51x51 K528 197 us,
// so 67).  All 32 lanes call.
enum EpiKind : int { NOEPI, EPI_PAIR, EPI_ODD };
template <int NC>
__device__ __forceinline__ void load_cols(const Epi& epi, uint32_t o, uint32_t step, int lim, bool live, bool pair,
                                          __half2* rv) {
  const char* R = reinterpret_cast<const char*>(epi.residual);
  if (!R) return;
  if (pair) {
    const bool odd = (threadIdx.x & 1) != 0;
    uint32_t ra = o - (odd ? 2u : 0u) + (odd ? step : 0u);
#pragma unroll
    for (int j = 0; j < NC / 2; ++j, ra += 2 * step)
      rv[j] = live && 2 * j + odd < lim ? *reinterpret_cast<const __half2*>(R + ra) : __half2{};
  } else {
    uint32_t ra = o;
#pragma unroll
    for (int j = 0; j < NC / 2; ++j, ra += 2 * step)
      rv[j] = __halves2half2(live && 2 * j < lim ? *reinterpret_cast<const __half*>(R + ra) : __half{},
                             live && 2 * j + 1 < lim ? *reinterpret_cast<const __half*>(R + ra + step) : __half{});
  }
}
template <int NC, int EPI>
__device__ __forceinline__ void store_cols(const Epi& epi, const float* bias, char* Y, uint32_t o, uint32_t step,
                                           const float* v, const __half2* rv, int lim, bool live, bool pair) {
  auto finish = [&](__half2 h, __half2 r) {
    float2 f = __half22float2(h);
    if (epi.residual) {
      const float2 g = __half22float2(r);
      f.x += g.x;
      f.y += g.y;
    }
    if (epi.relu) {
      f.x = fmaxf(f.x, 0.f);
      f.y = fmaxf(f.y, 0.f);
    }
    return __floats2half2_rn(f.x, f.y);
  };
  auto rounded = [&](int j) {
    float a = v[2 * j], b = v[2 * j + 1];
    if (EPI && bias) {
      // (bias of channels past K is not read: lim)
      a += 2 * j < lim ? __ldg(bias + 2 * j) : 0.f;
      b += 2 * j + 1 < lim ? __ldg(bias + 2 * j + 1) : 0.f;
    }
    return __floats2half2_rn(a, b);
  };
  if (pair) {
    const bool odd = (threadIdx.x & 1) != 0;
    const uint32_t sel = odd ? 0x3276u : 0x5410u;
    // the pair's even position, this lane's column of the first two
    uint32_t at = o - (odd ? 2u : 0u) + (odd ? step : 0u);
    const int mine = odd ? 1 : 0;
#pragma unroll
    for (int j = 0; j < NC / 2; ++j, at += 2 * step) {
      const __half2 h = rounded(j);
      const uint32_t own = *reinterpret_cast<const uint32_t*>(&h);
      const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
      const uint32_t w = __byte_perm(own, other, sel);
      __half2 out = *reinterpret_cast<const __half2*>(&w);
      if (EPI) out = finish(out, rv[j]);
      if (live && 2 * j + mine < lim) *reinterpret_cast<__half2*>(Y + at) = out;
    }
  } else if (live) {
    uint32_t at = o;
#pragma unroll
    for (int j = 0; j < NC / 2; ++j, at += 2 * step) {
      __half2 h = rounded(j);
      if (EPI) h = finish(h, rv[j]);
      if (2 * j < lim) *reinterpret_cast<__half*>(Y + at) = __low2half(h);
      if (2 * j + 1 < lim) *reinterpret_cast<__half*>(Y + at + step) = __high2half(h);
    }
  }
}

}  // namespace sc

// KCRS weights -> the weight operand of a problem's plan, one 16-byte word
// per thread.
template <int CG>
__device__ __forceinline__ void shift_weight_body(const KernelParam& p, uint8_t* wop) {
  using namespace sc;
  grid_dep_launch();
  const Plan g = unpack_plan(p, CG);
  const unsigned wi = blockIdx.x * blockDim.x + threadIdx.x;
  if (wi >= (unsigned)(weight_bytes(g, CG) >> 4)) return;
  // (row of the operand, 16-channel block, tap, half), halves fastest, so
  // neighbouring threads read one output channel's weights
  const int hh = (int)(wi & 1);
  const unsigned r2 = wi >> 1;
  const int row = (int)(r2 / (unsigned)g.NKS), ks = (int)(r2 - (unsigned)row * (unsigned)g.NKS);
  const int cb = (int)((unsigned)ks / (unsigned)g.taps), tap = ks - cb * g.taps;
  // NB is a power of two
  const int k0 = row & ~(g.NB - 1), rk = row - k0;
  const int rows = unit_n(g, CG, k0) / CG, rank = CG == 2 && rk >= rows ? 1 : 0, rr = rk - rank * rows;
  const unsigned short* w = static_cast<const unsigned short*>(p.pweight);
  uint32_t v[4];
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const int c = cb * 16 + hh * 8 + e;
    auto at = [&](int ch) {
      if (row >= g.K || ch >= g.C) return 0u;
      if (!g.fold) return (uint32_t)w[((size_t)row * g.C + ch) * g.taps + tap];
      const int rc = ch / g.fS;           // virtual channel -> input channel, filter column
      return (uint32_t)w[(((size_t)row * g.fC + rc) * g.R + tap) * g.fS + ch - rc * g.fS];
    };
    v[e >> 1] = at(c) | at(c + 1) << 16;
  }
  uint8_t* dst = wop + ((size_t)(k0 + rank * rows) * g.NKS + (size_t)ks * rows) * 32 + (rr >> 3) * 256 + hh * 128 +
                 (rr & 7) * 16;
  *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
}

// The weight operand from a fused U cache (u_offset's layout): the 3x3 filter
// back from U = G g G^T, one thread an output channel's eight input channels.
// With G's rows e0, (e0 + e1 + e2) / 2, (e0 - e1 + e2) / 2, e2 a vector's
// inverse is (u0, u1 - u2, u3): the corner taps are U's own fp16 values, the
// others sums of two or four, formed in fp32 and rounded to the fp16 grid the
// filter came from (more than half of them land on it exactly; 2.2e-4 of the
// filter in the 2-norm, against the 2.9e-4 to which U itself was rounded).
template <int CG>
__device__ __forceinline__ void shift_weight_from_u(const KernelParam& p, const __half* u, uint8_t* wop, unsigned item) {
  using namespace sc;
  grid_dep_launch();
  const Plan g = unpack_plan<CONV33>(p, CG);
  // rows fastest: neighbouring threads read and write neighbouring 16-byte rows
  const int last = (g.nKU - 1) * g.NB, nrow = last + unit_n(g, CG, last);
  const int grp = (int)(item / (unsigned)nrow), row = (int)(item - (unsigned)grp * (unsigned)nrow), c = grp * 8;
  if (c >= g.C) return;
  // NB is a power of two
  const int k0 = row & ~(g.NB - 1), rk = row - k0;
  const int rows = unit_n(g, CG, k0) / CG, rank = CG == 2 && rk >= rows ? 1 : 0, rr = rk - rank * rows;
  uint8_t* dst = wop + ((size_t)(k0 + rank * rows) * g.NKS + (size_t)(c >> 4) * 9 * rows) * 32 + (rr >> 3) * 256 +
                 ((c >> 3) & 1) * 128 + (rr & 7) * 16;
  uint4 uw[16];
#pragma unroll
  for (int t = 0; t < 16; ++t)
    uw[t] = row < g.K ? __ldg(reinterpret_cast<const uint4*>(u + u_offset(t, row, c, g.K, g.C))) : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        auto at = [&](int a, int b) {
          const uint4& w = uw[4 * a + b];
          const uint32_t x = e == 0 ? w.x : e == 1 ? w.y : e == 2 ? w.z : w.w;
          return __half22float2(*reinterpret_cast<const __half2*>(&x));
        };
        auto col = [&](int a) {
          if (s != 1) return at(a, s == 0 ? 0 : 3);
          const float2 m = at(a, 1), n = at(a, 2);
          return make_float2(m.x - n.x, m.y - n.y);
        };
        float2 v;
        if (r != 1) {
          v = col(r == 0 ? 0 : 3);
        } else {
          const float2 m = col(1), n = col(2);
          v = make_float2(m.x - n.x, m.y - n.y);
        }
        const __half2 h = __floats2half2_rn(v.x, v.y);
        o[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
      *reinterpret_cast<uint4*>(dst + (size_t)(r * 3 + s) * rows * 32) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// The kernel body.  CG = 2: clusters of two CTAs (__cluster_dims__(2, 1, 1)),
// a unit is 256 positions, rank 0 issues the pair's MMAs.  Every role walks
// the source's layers and its own units of each.
template <int CG, int EPI, class Src>
__device__ __forceinline__ void shift_conv_body(const Src& src, const sc::Epi& epi, uint32_t* err) {
  using namespace sc;
  extern __shared__ __align__(128) uint8_t shift_smem[];
  __shared__ Shared sh;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(shift_smem) + 127) & ~uintptr_t(127));
  // a warp-uniform warp index, so that what the MMA warp derives stays in
  // uniform registers
  const int warp = __shfl_sync(0xffffffffu, (int)warp_id(), 0), lane = lane_id();
  const int rank = CG == 2 ? (int)cluster_ctarank() : 0;
  const int u0 = CG == 2 ? (int)cluster_id_x() : (int)blockIdx.x;
  const int ustep = CG == 2 ? (int)cluster_count_x() : (int)gridDim.x;
  constexpr int TS = TM * CG;             // positions of a unit
  const int tp = rank * TM;               // this CTA's first of them

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAXSTAGE; ++s) {
      // producers, padding, weights (and at a pair's rank 0 the peer's whole stage)
      mbar_init(&sh.full[s], (src.strided() ? 2 : 1) * PW + NWARP_Z + 1 + (CG == 2 && rank == 0 ? 1 : 0));
      mbar_init(&sh.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sh.accfull[a], 1);
      mbar_init(&sh.accempty[a], CG * EW);
    }
    mbar_init(&sh.mmadone, 1);
    sh.abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == W_MMA) {
    if (CG == 2) { tmem_alloc_pair(&sh.tmem_base, 512); tmem_relinquish_pair(); }
    else { tmem_alloc(&sh.tmem_base, 512); tmem_relinquish(); }
  }
  volatile int* abort_flag = &sh.abort_flag;
  const uint32_t sbase = smem_u32(smem);
  const int nl = src.layers();
  bool ok = true;

  if (warp >= W_MMA && warp < W_P0) {
    setup_sync<CG>();
    if (warp == W_LOAD) {
      // the stages' weights, one bulk copy each: this CTA's rows of the unit's
      // output channels
      if (lane == 0) {
        RingPos pos{0, 1};
        int issued = 0, nstage = 1;
        // the operand is the kernel before's (programmatic launch); setup and
        // the first input loads overlap with it
        grid_dep_wait();
        // what a batch launches next works on other layers
        grid_dep_launch();
        for (int l = 0; ok && l < nl; ++l) {
          Conv cv;
          if (!src.get(l, CG, u0, ustep, cv)) continue;
          const Plan& g = cv.g;
          nstage = g.nstage;
          for (int i = 0; ok && i < cv.cnt; ++i) {
            int pt, k0;
            unit_of(g, cv.u0 + i * ustep, pt, k0);
            const uint32_t piece = (uint32_t)(unit_n(g, CG, k0) / CG) * 32;      // one tap of 16 channels
            const uint32_t block = piece * (uint32_t)g.taps;
            const uint8_t* from = cv.wop + (size_t)k0 * g.NKS * 32 + (size_t)rank * piece * g.NKS;
            for (int cb = 0; cb < g.CB; cb += g.cps) {
              ok = mbar_wait(&sh.empty[pos.st], pos.phase, abort_flag, err, ERR_WAIT_EMPTY);
              if (!ok) break;
              const uint32_t bytes = block * (uint32_t)min(g.cps, g.CB - cb);
              mbar_arrive_expect_tx(&sh.full[pos.st], bytes);
              bulk_g2s(smem + pos.st * g.pitch + g.stageA, from, bytes, &sh.full[pos.st]);
              from += bytes;
              ++issued;
              pos.next(nstage);
            }
          }
        }
        // copies still in flight land before the CTA leaves (an abort may have
        // kept the MMA side from waiting for them)
        if (*abort_flag)
          for (int b = issued > nstage ? issued - nstage : 0; b < issued; ++b)
            mbar_wait(&sh.full[b % nstage], (b / nstage) & 1, nullptr, err, ERR_WAIT_FULL);
      }
    } else if (warp >= W_Z0) {
      RingPos pos{0, 1};
      for (int l = 0; ok && l < nl; ++l) {
        Conv cv;
        if (src.get(l, CG, u0, ustep, cv))
          ok = pad_rows(cv, smem, sh, threadIdx.x - W_Z0 * 32, ustep, tp, TS, pos, err);
      }
    } else {
      const uint32_t tmem = __shfl_sync(0xffffffffu, sh.tmem_base, 0);
      RingPos pos{0, 0};
      if (CG == 2 && rank == 1) {
        // tell rank 0 that this CTA's half of each stage is complete
        const uint32_t lead = mapa_shared(smem_u32(&sh.full[0]), 0);
        for (int l = 0; ok && l < nl; ++l) {
          Conv cv;
          if (!src.get(l, CG, u0, ustep, cv)) continue;
          for (int left = cv.cnt * cv.g.nst; ok && left > 0; --left) {
            ok = wait_all_lanes(&sh.full[pos.st], pos.phase, abort_flag, err, ERR_WAIT_FULL);
            if (ok && lane == 0) mbar_arrive_remote(lead + pos.st * 8);
            pos.next(cv.g.nstage);
          }
        }
      } else {
        const bool leader = elect_one();
        int unit = 0;
        bool ready = false;
        for (int l = 0; ok && l < nl; ++l) {
          Conv cv;
          if (!src.get(l, CG, u0, ustep, cv)) continue;
          __syncwarp();
          for (int t = lane; t < cv.g.taps; t += 32) sh.aoff[t] = tap_row(cv.g, t / cv.g.S, t % cv.g.S);
          __syncwarp();
          if (Src::kind == CONV33 || (Src::kind != FOLDED && cv.g.taps == 9)) ok = issue_mmas<CG, 9>(cv, sh, sbase, tmem, ustep, leader, pos, unit, ready, err);
          else if (Src::kind != FOLDED && cv.g.taps == 1) ok = issue_mmas<CG, 1>(cv, sh, sbase, tmem, ustep, leader, pos, unit, ready, err);
          else ok = issue_mmas<CG, 0>(cv, sh, sbase, tmem, ustep, leader, pos, unit, ready, err);
        }
        // every MMA issued (also on an abort) has finished before TMEM is freed
        if (leader) {
          if (CG == 2) mma_commit_pair(&sh.mmadone, 1);
          else mma_commit(&sh.mmadone);
          mbar_wait(&sh.mmadone, 0, nullptr, err, ERR_WAIT_ACCUM);
        }
      }
    }
    __syncwarp();
  } else if (warp < EW) {
    setup_sync<CG>();
    const uint32_t tmem = sh.tmem_base;
    // epilogue: TMEM lane 32 * quarter + lane = position of this CTA's tile;
    // a quarter's warps take alternate 32-column chunks
    const int quarter = warp & 3, part = warp >> 2;
    constexpr int PARTS = EW / 4;
    const uint32_t lead_accempty = mapa_shared(smem_u32(&sh.accempty[0]), 0);
    int unit = 0;
    for (int l = 0; ok && l < nl; ++l) {
      Conv cv;
      if (!src.get(l, CG, u0, ustep, cv)) continue;
      const Plan& g = cv.g;
      __half* Y = cv.y;
      const int OHOW = g.OH * g.OW;
      const uint32_t step = (uint32_t)OHOW * 2u;
      const Grid gr = make_grid(g);
      // even output rows sit on an even grid: neighbouring outputs on lanes
      // 2i, 2i + 1 share 4-byte stores
      const bool pair = EPI == NOEPI ? store_pairs(g.OW, Y, nullptr) : EPI == EPI_PAIR;
      for (int i = 0; i < cv.cnt; ++i, ++unit) {
        int pt, k0;
        unit_of(g, cv.u0 + i * ustep, pt, k0);
        const int nrows = min(g.NB, g.Kp - k0);
        const int kval = min(nrows, g.K - k0);             // output channels that exist
        const int ab = unit & 1;
        const Base c = advance(gr, tile_base(gr, pt * TS + tp), quarter * 32 + lane);
        const bool live = c.n < g.N && c.gy < g.OH && c.gx < g.OW;
        const uint32_t at = live ? ((uint32_t)(c.n * g.K + k0) * (uint32_t)OHOW + (uint32_t)(c.gy * g.OW + c.gx)) * 2u : 0u;
        __half2 rv[EPI ? 16 : 1];
        auto res = [&](int cc) {
          if (EPI) load_cols<32>(epi, at + (uint32_t)cc * step, step, kval - cc, live, pair, rv);
        };
        res(part * 32);
        ok = mbar_wait_warp(&sh.accfull[ab], (unit >> 1) & 1, abort_flag, err, ERR_WAIT_ACCUM, SLEEP_NS);
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + ab * 256;
        auto ld = [&](int cc, float* v) {
          tmem_ld16(taddr + cc, v);
          if (cc + 16 < nrows) tmem_ld16(taddr + cc + 16, v + 16);
        };
        auto stc = [&](int cc, const float* v) {
          store_cols<32, EPI>(epi, EPI && epi.bias ? epi.bias + k0 + cc : nullptr, reinterpret_cast<char*>(Y),
                              at + (uint32_t)cc * step, step, v, rv, kval - cc, live, pair);
        };
#pragma unroll 1
        for (int cc = part * 32; cc < nrows; cc += 32 * PARTS) {
          float va[32];
          ld(cc, va);
          tmem_ld_wait();
          stc(cc, va);
          if (cc + 32 * PARTS < nrows) res(cc + 32 * PARTS);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CG == 2) mbar_arrive_peer(lead_accempty + ab * 8);
          else mbar_arrive(&sh.accempty[ab]);
        }
      }
    }
  } else {
    const int group = (warp - W_P0) / PW, tid = threadIdx.x - (W_P0 + group * PW) * 32;
    int done = 0, turn = 0;               // stages of the layers before, whose turn the next run is
    bool set = false;                     // setup_sync passed
    for (int l = 0; ok && l < nl; ++l) {
      Conv cv;
      if (!src.get(l, CG, u0, ustep, cv)) continue;
      const Plan& g = cv.g;
      if constexpr (Src::kind == FOLDED) {
        setup_sync<CG>();
        set = true;
        if (g.fC == 3 && g.fS == 7) ok = produce_fold<CG, 3, 7>(cv, smem, sh, tid, group, ustep, tp, TS, err);
        else ok = produce_fold<CG, 0, 0>(cv, smem, sh, tid, group, ustep, tp, TS, err);
      } else {
        const bool aligned = !Src::edges && input_aligned(g.H * g.W, cv.x);
        const bool one = stage_items(g, aligned) <= NPROD;
        constexpr int MORE = MAXITEMS / NPROD;   // items a producer may own
#define SC_PRODUCE(ni, al, strd) \
  ok = produce<CG, ni, al, strd, Src::edges && !al>(cv, smem, sh, tid, group, done, turn, ustep, tp, TS, set, err)
        if constexpr (Src::kind == PLAIN) {
          if (src.strided()) {
            if (aligned && one) SC_PRODUCE(1, true, true);
            else if (aligned) SC_PRODUCE(MORE, true, true);
            else if (one) SC_PRODUCE(1, false, true);
            else SC_PRODUCE(MORE, false, true);
            continue;
          }
        }
        if (Src::table) {
          if (aligned) SC_PRODUCE(1, true, false);
          else SC_PRODUCE(1, false, false);
        } else if (aligned && one) SC_PRODUCE(1, true, false);
        else if (aligned) SC_PRODUCE(MORE, true, false);
        else if (one) SC_PRODUCE(1, false, false);
        else SC_PRODUCE(MORE, false, false);
#undef SC_PRODUCE
      }
      done += cv.cnt * g.nst;
      turn ^= (runs_by_unit(g) ? cv.cnt : cv.cnt * g.nst) & 1;
    }
    if (!set) setup_sync<CG>();           // no stage for this group
  }
  tc_fence_before();
  __syncthreads();
  // the peer may still read this CTA's shared memory or arrive on its
  // barriers until both CTAs get here
  if (CG == 2) cluster_sync();
  if (warp == W_MMA) {
    tc_fence_after();
    if (CG == 2) tmem_dealloc_pair(sh.tmem_base, 512);
    else tmem_dealloc(sh.tmem_base, 512);
  }
}

}  // namespace wino
