// rh_tile.cu — the tiles a mesh's levels take when their user chose none: a
// uniform level's here, those of coarse-fine levels at the end.
//
// A CTA marches its pencil layer by layer, so a level's step takes the CTAs'
// waves times a pencil's march: a 64^3 level cut into 8x8-octs x 32-layer
// pencils is 16 CTAs on 148 SMs, each marching 34 layers (FP64 240 us), while
// 256 pencils of 8x4 octs x 4 layers take 43 us; a 256^3 level fills the chip with either
// and wants the tile with the least halo.  choose_tile() evaluates that time
// for the compiled tiles below and the depths that cut the level's layers
// evenly, from three rates per tile measured on a B200 (HLLC, moncen; boxes of
// 16^3 to 256^3 cells, even and uneven; launch gap included): with one CTA on
// an SM or two, a pencil of L layers takes start + L * layer[0 or 1] us.  On
// those boxes its choice is the fastest of these tiles and depths.  The slope
// type and solver of a run are not known when its mesh is set: types 0 and 1
// and the other solvers change all rates alike, slope_type 3 (1.8 times the
// time; one CTA of FP32-bulk 7x7 on an SM) does not, and its runs are up to 15 %
// from their fastest tile (256^3 FP32-bulk 1.45 ms, 15x7 1.26; FP64 2.51, 7x11
// 2.40).  On 25 boxes no choice was slower than 8x8 octs x 32 layers for slope
// types 0, 1 or 3.
#include <algorithm>
#include <new>
#include <vector>

#include "rh_internal.h"

namespace rh {
namespace {

struct TileRate {
  int prec, txo, tyo, minb;
  double start, layer[2];
};
const TileRate kRates[] = {
    {RH_PREC_FP64, 6, 4, 2, 14.5, {4.96, 6.22}},       {RH_PREC_FP64, 8, 4, 2, 14.4, {5.62, 6.95}},
    {RH_PREC_FP64, 8, 8, 1, 15.2, {7.19, 7.19}},       {RH_PREC_FP64, 7, 11, 1, 14.7, {7.04, 7.04}},
    {RH_PREC_FP64, 15, 5, 1, 15.1, {6.74, 6.74}},      {RH_PREC_FP32_BULK, 6, 4, 2, 13.8, {2.45, 3.29}},
    {RH_PREC_FP32_BULK, 8, 4, 2, 13.8, {2.92, 3.78}},  {RH_PREC_FP32_BULK, 7, 7, 2, 14.4, {3.12, 4.93}},
    {RH_PREC_FP32_BULK, 8, 8, 1, 15.1, {3.67, 3.67}},  {RH_PREC_FP32_BULK, 15, 7, 1, 16.0, {5.18, 5.18}},
};
constexpr double kLaunch = 2.0;  // us of start that later waves of a launch do not pay
constexpr int kMaxDepth = 48;    // layers; longer pencils only lost to the wave count

double step_us(const TileRate& r, long long pencils, int lz, int sm_count) {
  if (pencils <= sm_count) return r.start + r.layer[0] * lz;
  const long long slots = (long long)sm_count * r.minb, full = pencils / slots, rest = pencils % slots;
  double t = kLaunch + full * (r.start - kLaunch + r.layer[1] * lz);
  if (rest > 0) t += r.start - kLaunch + r.layer[rest <= sm_count ? 0 : 1] * lz;
  return t;
}

}  // namespace

TileCfg choose_tile(int precision, int nxo, int nyo, int nzo, int sm_count) {
  TileCfg best;
  double tbest = 1e300;
  for (const TileRate& r : kRates) {
    if (r.prec != precision) continue;
    const long long cols = (long long)((nxo + r.txo - 1) / r.txo) * ((nyo + r.tyo - 1) / r.tyo);
    for (int cuts = 1; cuts <= nzo; ++cuts) {
      const int lz = (nzo + cuts - 1) / cuts;
      if (lz > kMaxDepth) continue;
      const double t = step_us(r, cols * ((nzo + lz - 1) / lz), lz, sm_count);
      if (t < tbest) {
        tbest = t;
        best = TileCfg{r.txo, r.tyo, r.minb, lz};
      }
    }
  }
  return best;
}

namespace {

// Layers of the TX x TY tiles that hold an oct of level l: what its pencils
// march through.  Counted in a bitmap over (tile, layer), hashed where the
// level's box is larger than 16 bits an oct (a few per cent of the layers may share
// a bit then, as many with either tile).
template <int TX, int TY> long long occupied_layers(const Context& c, int l) {
  const long long nx = (long long)c.box_nx[0] << (l - 1), ny = (long long)c.box_nx[1] << (l - 1),
                  nz = (long long)c.box_nx[2] << (l - 1);
  const long long ntx = (nx + TX - 1) / TX, nty = (ny + TY - 1) / TY;
  if (c.levels[l].complete_box) return ntx * nty * nz;
  int bits = 12;
  while (bits < 30 && (1ll << bits) < 16ll * c.noct[l]) ++bits;
  const bool dense = (double)ntx * nty * nz <= (double)(1ll << bits);
  std::vector<uint64_t> seen((size_t)1 << (bits - 6), 0);
  long long n = 0;
  const rh_oct* o = c.grid.data() + (c.head[l] - 1);
  for (int i = 0; i < c.noct[l]; ++i) {
    const long long x = o[i].ckey[0], y = o[i].ckey[1], z = o[i].ckey[2];
    if (x < 0 || y < 0 || z < 0 || x >= nx || y >= ny || z >= nz) continue;  // refused by the table builder
    uint64_t k = (uint64_t)((y / TY * ntx + x / TX) * nz + z);
    if (!dense) k = k * 0x9E3779B97F4A7C15ull >> (64 - bits);
    const uint64_t bit = 1ull << (k & 63);
    n += !(seen[k >> 6] & bit);
    seen[k >> 6] |= bit;
  }
  return n;
}

}  // namespace

// Tile of the coarse-fine kernels (levels, boxes and oct records of the mesh
// set).  FP64: 7x11, whose layer costs least per oct column, unless the mesh
// fills so few of its columns that the layers of 8x4 tiles, two CTAs an SM, cost
// less.  The cost ratio follows the measured one: gradient-refined blasts 0.94 to
// 1.01 by layers, 0.86 to 0.98 measured (levels 6-9: 508 against 549 us a coarse
// step), a sheet 0.89 and 0.92, scattered clusters of 27 to 343 octs 1.14 to 1.36
// and 1.17 to 1.29 (levels 6-8: 394 against 311 us; a third fewer ghost octs too).
TileCfg choose_amr_tile(const Context& c) {
  if (c.precision == RH_PREC_FP32_BULK) return TileCfg{7, 7, 2, 32};
  double wide = 0, narrow = 0;
  try {
    for (int l = c.levelmin; l <= c.levelmax; ++l) {
      if (c.noct[l] == 0) continue;
      wide += 7.04 * occupied_layers<7, 11>(c, l);
      narrow += 0.5 * 6.95 * occupied_layers<8, 4>(c, l);
    }
  } catch (const std::bad_alloc&) {  // no room to count in (128 MB at most)
    return TileCfg{7, 11, 1, 32};
  }
  return wide > 1.04 * narrow ? TileCfg{8, 4, 2, 32} : TileCfg{7, 11, 1, 32};
}

}  // namespace rh
