// sepx_unet_plan.h -- launch plans of the U-Net's 3x3x3 kernels: which layers a
// kernel takes, its shared and tensor memory, its work items.  Host code without
// CUDA, so that the plans can be checked on a CPU; the kernels
// (sepx_unet_zwfwd.inc, sepx_unet_kstream.inc, sepx_unet_wgring.inc) take them
// as they are.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define SEPX_HD __host__ __device__
#else
#define SEPX_HD
#endif

namespace sepx {

constexpr int kTM = 128;   // GEMM rows per CTA (tensor-memory lanes)
constexpr int kKC = 64;    // K per pipeline stage (8 K groups of 8)
constexpr int kMaxN = 128;

// input halo of a 16 x 8 tile (y, x)
constexpr int kHaloX = 10, kHaloY = 18, kHaloZ = 3;
constexpr int kHaloGS = 8704;   // bytes per channel group (8640 rounded up to 128)
constexpr int kTileY = 16, kTileX = 8;
constexpr int kMaxPairs = 8;   // channel-group pairs of one halo (up to 128 channels)
// shared memory a CTA may have
constexpr size_t kHaloMaxSmem = 227 * 1024;

// the device's figures that the persistent grids are sized from
struct UnetDev {
  int num_sms = 0;
  size_t smem_per_sm = 0, smem_reserved = 0;
};

// channel groups held per halo buffer: cin/8 rounded up to even (an odd
// count gets one all-zero group, the channel box lying wholly outside x)
SEPX_HD constexpr int halo_groups(int cin) { return ((cin / 8) + 1) & ~1; }

SEPX_HD constexpr size_t halo_smem_bytes(int cin, uint32_t wbytes, int nbuf) {
  return (size_t)wbytes + (size_t)nbuf * (size_t)halo_groups(cin) * kHaloGS + 256 + 128;
}

// The halo-staged and the z-walk convolution take 3x3x3 layers whose planes hold
// at least one 16 x 8 tile and whose weights (wbytes: the packed ones, and zeros
// for an odd count's added group) and one halo buffer fit in shared memory.
inline bool halo_applies(int H, int W, int cin, int np, uint32_t *wbytes) {
  const int ngc = cin / 8;
  *wbytes = (uint32_t)((27 * ngc + (ngc & 1)) * (np / 8) * 128);
  return H >= kTileY && W >= kTileX && halo_groups(cin) / 2 <= kMaxPairs &&
         halo_smem_bytes(cin, *wbytes, 1) <= kHaloMaxSmem;
}

// ---- z-walk convolution (sepx_unet_zwfwd.inc) ----
constexpr int kZfThreads = 320;
constexpr int kZfRow = 32;                       // bytes of a voxel's 16 channels
constexpr int kZfPlane = kHaloX * kHaloY * kZfRow;   // 5760 B
constexpr int kZfSlot = 2 * kZfPlane;            // 11520 B, a multiple of the swizzle's 256
constexpr int kZfMinSlots = 4, kZfMaxSlots = 8;
constexpr int kZfMaxZ = 16;                      // output planes of a window
SEPX_HD constexpr size_t zf_wbytes(int cin, int np) {
  return (size_t)27 * halo_groups(cin) * np * 16;
}
SEPX_HD constexpr size_t zf_smem_bytes(int cin, int np, int nslot) {
  return (zf_wbytes(cin, np) + 255) / 256 * 256 + (size_t)nslot * kZfSlot + kMaxN * 4 +
         (2 * kZfMaxSlots + kZfMaxZ + kMaxPairs) * 8 + 16 + 256;
}

struct ZwalkPlan {
  int per_sm, nslot;                  // CTAs of an SM, ring slots
  int ty, tx, zc, nzc, nitems;        // tiles, planes of a window, windows of a column
  int late_from, late;                // CTAs from late_from on start their MMAs `late` cycles later
  int grid;
  size_t smem;
};

// The z-walk convolution (sepx_unet_zwfwd.inc): every layer the halo-staged
// kernel takes whose three column blocks fit one MMA (3 x np <= 256) and whose
// weights leave room for a ring of four slots (it measured 3.3 to 5.3 times as
// fast on those).  False where it does not apply: np 96 to 128 with cin up
// to 24, np 96 or 112 with cin 32, and np 80 with cin 40 (226 KB of weights and
// halo fit, 249 KB of weights and ring do not) stay on the halo-staged kernel.
inline bool zwalk_plan(const UnetDev &dev, int nb, int D, int H, int W, int cin, int np, bool pool, ZwalkPlan &a) {
  if (3 * np > 256) return false;
  if (pool && (D % 2 || H % 2 || W % 2)) return false;
  auto fit = [&](int nslot) {
    const size_t sm = zf_smem_bytes(cin, np, nslot);
    if (sm > kHaloMaxSmem) return 0;
    return (int)(dev.smem_per_sm / (((sm + 127) / 128) * 128 + dev.smem_reserved));
  };
  // two CTAs per SM (each with half the tensor memory) where two rings fit,
  // so that one's start-up and last planes overlap the other's MMAs
  const int per_sm = a.per_sm = std::min(fit(kZfMinSlots), 2);
  if (per_sm < 1) return false;
  a.nslot = kZfMinSlots;
  while (a.nslot < kZfMaxSlots && fit(a.nslot + 1) >= per_sm) a.nslot++;
  a.ty = (H + kTileY - 1) / kTileY;
  a.tx = (W + kTileX - 1) / kTileX;
  const long long cols = (long long)nb * a.ty * a.tx;
  if (cols * D >= (1LL << 31)) return false;
  // planes per window: the accumulators fill this CTA's share of the 512
  // tensor-memory columns at most; among those the count with the least MMA
  // time on the busiest CTA (an MMA of N columns takes max(32 + N / 4, N / 2)
  // cycles; the two planes outside the window feed one column block, the two
  // inside its ends two)
  const long long slots = (long long)dev.num_sms * per_sm;
  const int zmax = std::min(std::min(kZfMaxZ, D), (512 / per_sm) / np);
  auto mma_cycles = [&](int zc) {   // a tap's MMAs over a window
    double c = 0;
    for (int p = 0; p < zc + 2; p++) {
      const int blk = std::min(p, zc - 1) - std::max(p - 2, 0) + 1;
      c += std::max(32.0 + 0.25 * np * blk, 0.5 * np * blk);
    }
    return c;
  };
  double best = 1e300;
  a.zc = 1;
  const int zstep = pool ? 2 : 1;   // (pooled: windows of whole plane pairs)
  for (int zc = zstep; zc <= zmax; zc += zstep) {
    const long long items = cols * ((D + zc - 1) / zc);
    const long long per = (items + slots - 1) / slots;
    const double cost = (double)per * mma_cycles(zc);
    if (cost < best) {
      best = cost;
      a.zc = zc;
    }
  }
  a.nzc = (D + a.zc - 1) / a.zc;
  a.zc = (D + a.nzc - 1) / a.nzc;   // the same windows, evenly filled
  if (pool) {
    a.zc += a.zc & 1;
    a.nzc = (D + a.zc - 1) / a.zc;
  }
  a.nitems = (int)(cols * a.nzc);
  a.late_from = dev.num_sms;
  a.late = (int)(0.75 * 9 * (halo_groups(cin) / 2) * mma_cycles(a.zc));
  a.grid = (int)std::min<long long>(a.nitems, slots);
  a.smem = zf_smem_bytes(cin, np, a.nslot);
  return true;
}

// ---- convolution with streamed weights (sepx_unet_kstream.inc) ----
constexpr int kKsThreads = 448;
constexpr int kKsLoaders = 8;
constexpr int kKsMaxRing = 6, kKsMaxW = 4, kKsMaxGroups = 32 * kKsLoaders;
// bytes of a plane's channel group: 18 x 10 voxels, padded to an odd number of
// 16-byte units (lanes copy a voxel's groups side by side: no bank conflicts)
constexpr int kKsGS = (kHaloX * kHaloY + 1) * 16;

SEPX_HD constexpr size_t ks_smem_bytes(int cin, int np, int nring, int nw) {
  return (size_t)nw * np * cin * 2 + (((size_t)nring * (cin / 8) * kKsGS + 127) / 128) * 128 + kMaxN * 4 +
         (2 * kKsMaxRing + 2 * kKsMaxW + 5) * 8 + 16 + 128;
}

// The convolution with streamed weights (sepx_unet_kstream.inc): 3x3x3 layers
// whose weights do not fit in shared memory or whose planes are smaller than a
// tile, where channels come in pairs of groups (a K16 step stays in one tap),
// the planes a K range reads fit in shared memory, staging them moves at most
// 0.4 of what the gather kernel copies for the range and the tile's real
// voxels, and a range's MMAs take at least 1400 cycles (an item's fixed costs).
// Measured (gather -> this, us a call; share staged, cycles): 112 -> 48 on 32^3
// voxels 91 -> 30 (0.20, 4224), 64 -> 64 on 40 x 12 x 40 26.4 -> 17.5 (0.26,
// 2592), 32 -> 48 on 116 x 12 x 122 83 -> 61 (0.22, 2376), 48 -> 16 on 68 x 12 x
// 40 27.9 -> 22.5 (0.26, 1584); at the lines 112 -> 48 on 2 x 30 x 9 x 51 53.5 ->
// 53.3 (0.36), 48 -> 64 on 30 x 9 x 40 18.4 -> 18.4 (1152); short of them 16 ->
// 16 on 2 x 14 x 9 x 100 11.6 -> 20.9 (0.33, 576), 16 -> 32 on 50 x 9 x 100 15.9
// -> 26.6 (1080), 64 -> 64 on 16^3, the kernels, 10.5 -> 11.2 (0.47).
// The K range of a layer is split into `splits` of kper chunks of 64.  Returns the
// planes of one output plane that any range reads, 0 where it does not apply.
inline int kstream_span(int nb, int D, int H, int W, int cin, int np, int splits, int kper) {
  if (cin % 16 || cin / 8 > kKsMaxGroups) return 0;
  const long long cols = (long long)nb * ((H + kTileY - 1) / kTileY) * ((W + kTileX - 1) / kTileX);
  if (cols * D * splits >= (1LL << 31)) return 0;
  int span = 1;
  const int per9 = 9 * (cin / 16);
  for (int s = 0; s < splits; s++) {
    const int k0 = s * kper * (kKC / 16), k1 = std::min(k0 + kper * (kKC / 16), 3 * per9);
    span = std::max(span, (k1 - 1) / per9 - k0 / per9 + 1);
  }
  const double staged = (double)cols * D * span * (kHaloX * kHaloY) * cin, gathered = (double)nb * D * H * W * kper * kKC;
  const int steps = std::min(kper * (kKC / 16), 3 * per9);
  return 2.5 * staged > gathered || steps * std::max(32.0 + 0.25 * np, 0.5 * np) < 1400 ? 0 : span;
}

struct KstreamPlan {
  int per_sm, nring, nw;              // CTAs of an SM, plane and weight slots
  int ty, tx, zc, nzc, nitems;
  int grid;
  size_t smem;
};

// span: of kstream_span; false where the planes do not fit
inline bool kstream_plan(const UnetDev &dev, int nb, int D, int H, int W, int cin, int np, int splits, int span,
                         KstreamPlan &a) {
  a.ty = (H + kTileY - 1) / kTileY;
  a.tx = (W + kTileX - 1) / kTileX;
  const long long cols = (long long)nb * a.ty * a.tx;
  auto fit = [&](int nring, int nw) {
    const size_t sm = ks_smem_bytes(cin, np, nring, nw);
    if (sm > kHaloMaxSmem) return 0;
    return std::min((int)(dev.smem_per_sm / ((sm + 127) / 128 * 128 + dev.smem_reserved)), 2);
  };
  // two CTAs per SM where the planes and two weight slots leave room for them
  const int want = std::max(fit(span, 2), 1);
  a.nw = kKsMaxW;
  while (a.nw > 2 && fit(span, a.nw) < want) a.nw--;
  const int per_sm = a.per_sm = fit(span, a.nw);
  if (!per_sm) return false;
  a.nring = span;
  while (a.nring < kKsMaxRing && fit(a.nring + 1, a.nw) >= per_sm) a.nring++;
  // output planes of an item: all ranges of a split layer are items already;
  // else the count with the fewest planes on the busiest CTA (an item's first
  // planes cost about half an output plane's MMAs)
  const long long slots = (long long)dev.num_sms * per_sm;
  a.zc = 1;
  if (splits == 1) {
    double best = 1e300;
    for (int zc = 1; zc <= D; zc++) {
      const long long items = cols * ((D + zc - 1) / zc);
      const double c = (double)((items + slots - 1) / slots) * (zc + 0.5);
      if (c < best) {
        best = c;
        a.zc = zc;
      }
    }
  }
  a.nzc = (D + a.zc - 1) / a.zc;
  a.zc = (D + a.nzc - 1) / a.nzc;   // the same runs, evenly filled
  a.nitems = (int)(cols * a.nzc * splits);
  a.grid = (int)std::min<long long>(a.nitems, slots);
  a.smem = ks_smem_bytes(cin, np, a.nring, a.nw);
  return true;
}

// ---- ring form of the tap-stacked weight gradient (sepx_unet_wgring.inc) ----
constexpr int kRgEpi = 8;                               // epilogue warps
constexpr int kRgThreads = 32 * (kRgEpi + 2);
constexpr int kRgMaxRing = 12, kRgMaxA = 4;
constexpr int kRgBlk = kHaloY * 8 * 32;                 // one plane of 16 channels, 4608 B

// rows of block b of A: 4 x 16, 4 x 32, or 2 x 64 and 1 x 64
SEPX_HD constexpr int rg_mrows(int pw, int b) { return pw == 16 || b == 1 ? 64 : 128; }
SEPX_HD constexpr uint32_t rg_aslot(int pw) { return 16u * 10u * (uint32_t)pw * 2u; }
SEPX_HD constexpr size_t rg_smem_bytes(int ncb, int pw, int na, int nring) {
  return (size_t)na * rg_aslot(pw) + (size_t)nring * ncb * kRgBlk + 128 * 9 * 4 +
         (2 * kRgMaxRing + 2 * kRgMaxA + 2) * 8 + 16 + 1024;
}

struct RingPlan {
  int ncb, ngo, pw;     // blocks of 16 channels of x, groups of 8 of dy, channels of a dy box
  int nsy, nmb, nmbt;   // sy values and blocks of rows of a job, blocks of rows of the layer
  bool stacked;         // one MMA over (dz, c), or one per dz
  int n, ncols;         // its N; tensor-memory columns of a CTA
  int na, nring;        // dy and plane slots
  int njob, ty, tx, zc, nzc, nitems, groups;
  int seg;              // tiles an accumulator takes between two read-outs
  size_t smem;
};

inline bool ring_applies(int cin, int cout) { return cin <= 112 && cout <= 64; }

// (of a layer that ring_applies says yes to; false where its items are too many)
inline bool ring_plan(const UnetDev &dev, int nb, int D, int H, int W, int cin, int cout, RingPlan &a) {
  const int ngi = cin / 8, ngo = (cout + 7) / 8;
  a.ngo = ngo;
  a.ncb = (ngi + 1) / 2;
  a.pw = cout <= 16 ? 16 : (cout <= 32 ? 32 : 64);
  a.nmbt = a.pw == 64 ? 2 : 1;
  a.stacked = 48 * a.ncb <= 256;
  a.n = a.stacked ? 48 * a.ncb : 16 * a.ncb;
  const int ncn = a.stacked ? a.n : 3 * a.n;
  // as much of a tile's work per CTA as the tensor memory holds: fewer CTAs
  // read the same planes
  a.nsy = a.nmbt * 3 * ncn <= 512 ? 3 : 1;
  a.nmb = a.nmbt * a.nsy * ncn <= 512 ? a.nmbt : 1;
  if (a.nmb * a.nsy * ncn > 512) return false;
  // One CTA per SM with the longest ring that fits (four planes at least).  Two
  // with shorter rings take 41 instead of 47 us for 16 -> 16 channels on 4 x
  // 64^3 voxels alone, but 1155 instead of 1137 in the training step, where a
  // data gradient's CTAs then find no room beside them and twice as many
  // partials are added.
  auto fits = [&](int na, int nring) { return rg_smem_bytes(a.ncb, a.pw, na, nring) <= kHaloMaxSmem; };
  a.na = fits(kRgMaxA, 8) ? kRgMaxA : (fits(3, 6) ? 3 : 2);
  a.nring = kRgMaxRing;
  while (a.nring > 4 && !fits(a.na, a.nring)) a.nring--;
  if (!fits(a.na, a.nring)) return false;
  a.ty = (H + 15) / 16;
  a.tx = (W + 2 + 7) / 8;
  const int njob = a.njob = (3 / a.nsy) * (a.nmbt / a.nmb);
  const int slots = std::max(1, dev.num_sms / njob);
  const long long cols = (long long)nb * a.ty * a.tx;
  if (cols * D >= (1LL << 31)) return false;
  // The tensor cores truncate as they add: a chain of n MMAs (8 a tile) into
  // one accumulator loses about 1.5e-8 n of a sum, in one direction.  So the
  // accumulators are read out, and added in FP32 to the CTA's partial sums,
  // once they have taken the tiles of a chain that `acc` accumulators per SM
  // would leave each, `least` at least (the loads go on meanwhile).  The
  // numbers are those of the forms that ran these layers before (one to four
  // CTAs an SM; the gather kernel's splits), whose errors are the bound.
  // Relative L2 error of one read-out -> of these (and time, us): 8 -> 16
  // channels on 4 x 64^3 voxels 7.2e-6 -> 1.4e-6 (47 -> 53), 32 -> 48 2.2e-5 ->
  // 3.8e-6 (152 -> 167), 112 -> 48 on 2 x 64^3 2.1e-5 -> 7.1e-6 (207 -> 216), 80 ->
  // 32 on 4 x 32^3 2.4e-6 -> 7.1e-7 (33 -> 40), 32 -> 32 there 8.2e-7 -> 5.6e-7
  // (23 -> 25); a training step on 4 x 64^3 1017 -> 1036.
  double acc;
  int least;
  if (njob == 1) {
    acc = a.pw == 16 && a.ncb == 1 ? (cin == 8 ? 4.0 : 2.0) : 1.0;
    least = a.pw == 16 && a.ncb == 1 ? 2 : 4;
  } else if (cout <= 40) {
    acc = a.pw == 64 ? 1.43 : 0.72;
    least = 2;
  } else {
    acc = 10.0 / ((27 * cin + 127) / 128);
    least = 8;
  }
  const int most = (int)std::max((double)least, 1.1 * (double)(cols * D) / (dev.num_sms * acc));   // tiles of a chain
  // planes per window: the run with the least work on the busiest CTA, in tiles
  // (a window loads two planes more than it has tiles: half a tile each; a
  // read-out takes as long as about five)
  double best = 1e300;
  for (int zc = 1; zc <= D; zc++) {
    const int nzc = (D + zc - 1) / zc;
    if (zc > 1 && (D + nzc - 1) / nzc != zc) continue;   // windows as even as the count allows
    const long long per = (cols * nzc + slots - 1) / slots;
    const int run = (int)(per * zc), nout = (run + most - 1) / most;
    const double cost = (double)per * (zc + 1.0) + 5.0 * (nout - 1);
    if (cost <= best) {
      best = cost;
      a.zc = zc;
      a.nzc = nzc;
      a.seg = (run + nout - 1) / nout;
    }
  }
  a.nitems = (int)(cols * a.nzc);
  a.groups = std::min(a.nitems, slots);
  a.ncols = a.nmb * a.nsy * ncn;
  a.smem = rg_smem_bytes(a.ncb, a.pw, a.na, a.nring);
  return true;
}

}  // namespace sepx
