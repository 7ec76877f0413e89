// Which matrix products run on the direct kernel, and their launch.
#include <algorithm>
#include <cmath>

#include "direct.cuh"

namespace plb {

namespace {

struct Extent {
  int m, n, k;
};
template <class S> Extent extentOf() { return {S::BM, S::BN, S::kStep}; }
Extent blockOf(DirectKind kind) {
  switch (kind) {
    case kDirectFew: return extentOf<DirectFew>();
    case kDirectSmall: return extentOf<DirectSmall>();
    case kDirectMid: return extentOf<DirectMid>();
    default: return extentOf<DirectWide>();
  }
}

// Whether all rows of both operands start at multiples of a whole load.
bool wholeLoads(const IgemmProblem &p, int type) {
  uint64_t at = reinterpret_cast<uintptr_t>(p.act) | reinterpret_cast<uintptr_t>(p.wgt) | p.act_strides[0] | p.wgt_strides[0];
  if (p.groups > 1) at |= p.act_group_stride | p.wgt_strides[1];
  return at % (type == PLB_QUARTER ? 8 : 16) == 0;
}

// Microseconds of a product on the direct kernel, launched after others of its kind:
// start + waves * (wave + round * K steps per team), fitted to 360 products of up to
// 0.6 GFLOP (16 to 8192 each way, up to 256 groups) of every type and layout; median error
// 6 %.  A block of two teams has an SM to itself, two of one team share one.
struct DirectTime {
  DirectKind kind;
  unsigned teams;
  float start[4], wave[4], round[4];  // half in whole loads, half, float, quarter
};
constexpr DirectTime kDirectTimes[] = {
    {kDirectFew, 2, {0.95f, 1.3f, 0.9f, 2.0f}, {1.15f, 0.8f, 0.2f, 0.3f}, {0.75f, 1.85f, 2.6f, 1.7f}},
    {kDirectSmall, 1, {1.6f, 1.4f, 0.65f, 2.0f}, {0.9f, 1.7f, 1.65f, 0.6f}, {0.45f, 1.15f, 1.4f, 1.25f}},
    {kDirectSmall, 2, {0.95f, 1.0f, 0.7f, 2.0f}, {1.3f, 1.4f, 1.2f, 0.6f}, {0.68f, 1.5f, 1.75f, 1.35f}},
    {kDirectMid, 2, {0.8f, 1.2f, 1.4f, 0.9f}, {1.35f, 1.35f, 0.45f, 1.3f}, {0.95f, 1.9f, 2.75f, 1.85f}},
    {kDirectWide, 1, {1.5f, 0.05f, 0.7f, 1.4f}, {1.25f, 4.0f, 2.2f, 1.9f}, {0.5f, 0.97f, 1.55f, 0.95f}},
    {kDirectWide, 2, {1.0f, 0.9f, 0.25f, 1.45f}, {1.3f, 2.1f, 1.4f, 1.1f}, {0.74f, 1.35f, 2.25f, 1.4f}},
};

// The shape of the least time, and that time.
const DirectTime &directShape(int sm_count, const IgemmProblem &p, int type, float *best) {
  const bool whole = wholeLoads(p, type);
  const int cls = type == PLB_FLOAT ? 2 : type == PLB_QUARTER ? 3 : whole ? 0 : 1;
  const DirectTime *found = nullptr;
  for (const DirectTime &t : kDirectTimes) {
    if (!directHas(t.kind, type, whole)) continue;
    const Extent e = blockOf(t.kind);
    const double blocks = double((p.out_w + e.m - 1) / e.m) * ((p.n_total + e.n - 1) / e.n) * std::max(1, p.groups);
    const int at_once = sm_count * (t.teams == 1 ? 2 : 1), steps = (p.k_per_tap + e.k - 1) / e.k;
    const float us = t.start[cls] + float(std::ceil(blocks / at_once)) * (t.wave[cls] + t.round[cls] * float((steps + t.teams - 1) / t.teams));
    if (found == nullptr || us < *best) {
      found = &t;
      *best = us;
    }
  }
  return *found;
}

// The same for the implicit-GEMM kernel and what goes before and after it; the tile is
// chosen as planIgemm does.
float igemmTime(int sm_count, const IgemmProblem &p, int type, bool copied) {
  const long sms = sm_count, groups = std::max(1, p.groups), m_tiles = (long(p.out_w) + 127) / 128;
  long waves = 0, cost = -1;
  float step = 0.f;
  for (int bn : {256, 128, 64}) {
    const long w = (m_tiles * ((p.n_total + bn - 1) / bn) * groups + sms - 1) / sms, c = w * (bn == 256 ? 155 : bn == 128 ? 95 : 75);
    if (cost < 0 || c < cost) {
      cost = c;
      waves = w;
      step = bn == 256 ? 0.35f : bn == 128 ? 0.2f : 0.12f;
    }
  }
  const long k_bytes = type == PLB_FLOAT ? 6L * p.k_per_tap : type == PLB_QUARTER ? p.k_per_tap : 2L * p.k_per_tap;
  long steps = (k_bytes + 127) / 128;
  float us = 3.3f;
  const long tiles = m_tiles * ((p.n_total + 63) / 64) * groups;
  if (tiles * 2 <= sms && steps >= 20) {  // the K range is split
    steps = std::max<long>(4, steps / (sms / tiles));
    us += 2.8f;
  }
  us += float(waves * steps) * step;
  if ((size_t(p.n_total) * (p.out_f32 ? 4 : 2)) % 16 != 0) us += 0.8f * float(waves);  // rows stored one by one
  if (copied) us += 2.3f + 0.4e-6f * float(groups) * float(k_bytes) * (float(p.out_w) + float(p.n_total));
  if (type == PLB_QUARTER && (p.a_mn || p.b_mn)) us += 1.1f;
  return us;
}

}  // namespace

// Products of which the direct kernel's estimate is a sixth below the other's.  Among the 360
// products this took 230 to 0.64 of their time on average (16 x 512 x 512 4.4 -> 2.9 us,
// 132 x 98 x 181 7.4 -> 3.7, as float 48 x 112 x 288 in 47 groups 11.1 -> 7.0); of those it
// leaves, a few would gain up to 10 %.
bool directSuits(int sm_count, const IgemmProblem &p, int type, bool copied, bool slower_too) {
  if (p.plan_flags != 0 || (type != PLB_HALF && type != PLB_FLOAT && type != PLB_QUARTER)) return false;
  // (pitches that no tensor map holds, negative ones among them, are the general route's to refuse)
  const uint64_t pitch_limit = uint64_t(1) << 40;
  if (std::max({p.act_strides[0], p.act_strides[1], p.wgt_strides[0], p.wgt_strides[1]}) >= pitch_limit) return false;
  if (2.0 * std::max(1, p.groups) * p.out_w * double(p.n_total) * p.k_per_tap > 1e9) return false;
  if (slower_too) return true;
  float us = 0.f;
  const DirectTime &t = directShape(sm_count, p, type, &us);
  // (long reductions of ragged floats in the smallest blocks: 225 x 1442 x 59 17.1 us, on the general
  // route 10.1; with this, 83 of 101 sampled ones that were slower here leave)
  if (t.kind == kDirectFew && type == PLB_FLOAT && !wholeLoads(p, type)) us *= 1.4f;
  return us < 0.86f * igemmTime(sm_count, p, type, copied);
}

int launchDirect(plb_context *ctx, const IgemmProblem &p, int type) {
  float us = 0.f;
  const DirectTime &t = directShape(ctx->sm_count, p, type, &us);
  DirectVariant v{t.kind, p.a_mn, p.b_mn, wholeLoads(p, type), 0, t.teams};
  const Extent block = blockOf(v.kind);
  DirectArgs g{};
  g.a = static_cast<const uint8_t *>(p.act);
  g.b = static_cast<const uint8_t *>(p.wgt);
  g.a_pitch = (long long)p.act_strides[0];
  g.b_pitch = (long long)p.wgt_strides[0];
  g.groups = std::max(1, p.groups);
  g.a_group = g.groups > 1 ? (long long)p.act_group_stride : 0;
  g.b_group = g.groups > 1 ? (long long)p.wgt_strides[1] : 0;
  g.m = p.out_w;
  g.n = p.n_total;
  g.k = p.k_per_tap;
  g.n_tiles = (g.n + block.n - 1) / block.n;
  g.fd_groups = make_fastdiv(uint32_t(g.groups));
  g.fd_n = make_fastdiv(uint32_t(g.n_tiles));
  g.fmt_a = p.fmt_a;
  g.fmt_b = p.fmt_b;
  g.out = p.out;
  g.ldc = p.ldc;
  g.out_group = g.groups > 1 ? p.out_group_stride : 0;
  g.addend = p.beta != 0.f ? p.addend : nullptr;
  g.addend_ld = p.ld_addend;
  g.addend_group = g.groups > 1 ? p.addend_group_stride : 0;
  g.alpha = p.alpha;
  g.beta = p.beta;
  g.out_f32 = p.out_f32 ? 1 : 0;
  g.out_vec = g.n % 4 == 0 && g.ldc % 4 == 0 && g.out_group % 4 == 0 &&
              reinterpret_cast<uintptr_t>(p.out) % (p.out_f32 ? 16 : 8) == 0;
  const unsigned long long blocks = (unsigned long long)((g.m + block.m - 1) / block.m) * g.n_tiles * g.groups;
  if (blocks > 0x3fffffffull) return fail(PLB_ERR_UNSUPPORTED, "too many output tiles for one launch");
  v.blocks = unsigned(blocks);
  switch (type) {
    case PLB_FLOAT: return launchDirectFloat(ctx, v, g);
    case PLB_QUARTER: return launchDirectQuarter(ctx, v, g);
    default: return launchDirectHalf(ctx, v, g);
  }
}

}  // namespace plb
