// Plans of the direct convolution over many geometries, on the CPU: what the kernel takes for granted must hold in each.
// Prints one line per violation and the number of plans looked at.
#include <cstdio>

#include "conv_halo.cuh"

using namespace elb;

static int bad = 0, plans = 0, refused = 0;

static void check(int kind, int n, int ic, int oc, int h, int w, int k, int stride, int pad, int max_acc) {
  const int oh = (h + 2 * pad - k) / stride + 1, ow = (w + 2 * pad - k) / stride + 1;
  if (oh < 1 || ow < 1) return;
  HaloPlan hp;
  std::string err;
  if (!halo_plan(hp, kind, n, ic, oc, h, w, oh, ow, k, k, stride, pad, pad, 148, err, max_acc)) { ++refused; return; }
  ++plans;
  const HaloParams &p = hp.p;
  const bool f32 = kind == HALO_F32;
  auto need = [&](bool ok, const char *what) {
    if (ok) return;
    ++bad;
    std::printf("%s: %s n %d %d -> %d %dx%d k %d s %d p %d acc %d (BN %d pair %d split %d fine %d)\n", what, f32 ? "f32" : "i8", n, ic, oc,
                h, w, k, stride, pad, max_acc, p.BN, p.pair, p.split, p.fine);
  };
  need(hp.smem_bytes <= 232448, "shared memory");
  need(p.BN >= 16 && p.BN <= 256 && p.BN % 16 == 0 && p.BN * p.n_tiles >= oc && p.BN * (p.n_tiles - 1) < (oc + 15) / 16 * 16, "channel tiles");
  need(static_cast<long long>(n) * p.period + 64 <= 0x7FFFFFFFll, "32-bit rows");
  need(p.groups >= 1 && p.split >= 1 && p.split <= p.groups && !(p.pair && p.split > 1), "split");
  need(!p.pair || (p.BN % 32 == 0 && stride == 1), "pair");
  need(!p.stack || (f32 && p.BN <= 128), "stack");
  need(p.sep == (f32 && p.BN <= 128), "lo accumulators");
  need((p.bufs == 4 ? 128 : 256) * p.bufs <= 512 && (p.bufs != 4 || (!f32 && p.BN <= 128)), "accumulators");
  need(p.b_stages >= 1 && p.a_stages >= 1 && p.a_bytes % 128 == 0 && p.b_stage_bytes % 16 == 0, "rings");
  const int groups = (p.groups + p.split - 1) / p.split;
  if (p.fine) need(f32 && p.BN <= 128 && k == 3 && stride == 1 && p.chunk_groups >= 1 && p.chunk_groups <= groups, "parts");
  if (f32 && max_acc) {
    const int each = p.fine ? p.ksteps / (p.BN <= 64 ? 2 : 1) * p.chunk_groups : p.ksteps * (p.sep ? 1 : 3) * groups;
    need(each <= max_acc, "additions per accumulator");
  }
}

int main() {
  const int channels[] = {3, 16, 40, 64, 96, 144, 208, 256, 512, 1024}, edges[] = {7, 14, 27, 56, 112};
  const int form[][3] = {{1, 1, 0}, {1, 2, 0}, {1, 1, 1}, {3, 1, 1}, {3, 1, 0}, {3, 2, 1}, {5, 1, 2}, {5, 2, 2}, {7, 2, 3}, {7, 1, 3}, {9, 1, 4}, {11, 2, 5}};
  for (int kind : {HALO_I8, HALO_F32})
    for (int n : {1, 3, 64})
      for (int ic : channels)
        for (int oc : channels)
          for (int h : edges)
            for (const auto &f : form) {
              check(kind, n, ic, oc, h, h + n % 2, f[0], f[1], f[2], 0);
              if (kind == HALO_F32 && f[0] == 3 && f[1] == 1 && f[2] == 1)
                for (int acc : {8, 9, 18, 39, 54, 111, 370}) check(kind, n, ic, oc, h, h + n % 2, 3, 1, 1, acc);
            }
  // rows of all images in 32 bits: refused above
  const int before = refused;
  check(HALO_I8, 1 << 24, 16, 16, 128, 1, 3, 1, 1, 0);
  check(HALO_I8, 1 << 24, 16, 16, 126, 1, 3, 1, 1, 0);
  if (refused != before + 1) { ++bad; std::printf("%d of two tall batches refused\n", refused - before); }
  std::printf("%d plans, %d refused, %d violations\n", plans, refused, bad);
  return bad != 0;
}
