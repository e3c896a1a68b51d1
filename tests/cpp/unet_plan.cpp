// The launch plans of csrc/sepx_unet_plan.h behind C functions, for
// tests/test_unet_plans_cpu.py.
#include "sepx_unet_plan.h"

using namespace sepx;

static UnetDev dev_of(int sms) {   // a GB300's figures but for the number of SMs
  UnetDev d;
  d.num_sms = sms;
  d.smem_per_sm = 228 * 1024;
  d.smem_reserved = 1024;
  return d;
}

extern "C" {
int plan_halo(int H, int W, int cin, int np) {
  uint32_t w;
  return halo_applies(H, W, cin, np, &w);
}
int plan_zwalk(int sms, int nb, int D, int H, int W, int cin, int np, int pool, long long *o) {
  ZwalkPlan p;
  if (!zwalk_plan(dev_of(sms), nb, D, H, W, cin, np, pool != 0, p)) return 0;
  const long long v[] = {p.per_sm, p.nslot, p.ty, p.tx, p.zc, p.nzc, p.nitems, p.grid, (long long)p.smem};
  std::copy(v, v + 9, o);
  return 1;
}
int plan_kstream(int sms, int nb, int D, int H, int W, int cin, int np, int splits, int kper, long long *o) {
  const int span = kstream_span(nb, D, H, W, cin, np, splits, kper);
  KstreamPlan p;
  if (!span || !kstream_plan(dev_of(sms), nb, D, H, W, cin, np, splits, span, p)) return 0;
  const long long v[] = {p.per_sm, p.nring, p.ty, p.tx, p.zc, p.nzc, p.nitems, p.grid, (long long)p.smem, p.nw, span};
  std::copy(v, v + 11, o);
  return 1;
}
int plan_ring(int sms, int nb, int D, int H, int W, int cin, int cout, long long *o) {
  RingPlan p;
  if (!ring_applies(cin, cout) || !ring_plan(dev_of(sms), nb, D, H, W, cin, cout, p)) return 0;
  const long long v[] = {p.ncb, p.ngo, p.pw, p.nsy, p.nmb, p.nmbt, p.stacked, p.n, p.ncols, p.na, p.nring,
                         p.njob, p.ty, p.tx, p.zc, p.nzc, p.nitems, p.groups, p.seg, (long long)p.smem};
  std::copy(v, v + 20, o);
  return 1;
}
}
