// Splitting the streamed dimension of the attention kernels when their grids are too small for the GPU.
//
// One CTA normally owns an output tile and walks every block that contributes to it: a few heads on a long causal sequence, or
// grouped queries on one key / value head, then leave most SMs idle behind the longest CTA (10007 tokens, 4 query heads on 1
// kv head: the dK/dV grid is 79 CTAs of up to 316 blocks for 148 SMs, where an even share would be 85 blocks).  With a split
// a tile of `units` blocks is walked by ceil(units / len) CTAs, each writes its fp32 partial result to scratch memory, and
// one more kernel adds the partials in a fixed order (so results stay reproducible) and rounds once.  This step alone, both
// sides in one run: backward of that case 847 -> 480 us, its forward 169 -> 136.  Together with the CTA order, the dQ
// kernel's halves and the one launch of both gradient grids, again in one run: that case 738 -> 361 and 159 -> 128; 1531 tokens, 8
// heads on 2: backward 120 -> 58, forward 32 -> 28; 300 queries on 8000 keys, 2 heads: forward 118 -> 31, backward 120 -> 46.
#pragma once
#include <limits.h>
#include <stdint.h>

namespace ody {

// How many blocks tile `t` of a grid walks: `mul` per visible block of the streamed dimension, which has `n` blocks.
// kind 0: all of them; 1: causal, blocks t .. n-1 (a KV tile and the query blocks that see it); 2: causal, the KV blocks that
// query tile t sees, t * step + 1 of them at most (step: query blocks per CTA; a second query tile's one block more goes
// with the last part).
struct SplitUnits {
  int kind, n, mul, step;
  __host__ __device__ int operator()(int t) const {
    const int vis = kind == 0 ? n : kind == 1 ? (n > t ? n - t : 0) : (n < t * step + 1 ? n : t * step + 1);
    return vis * mul;
  }
};

// len: blocks per CTA; max_parts: parts of the longest tile; no split: {INT_MAX, 1}.  Part z of a tile takes its blocks
// [z * len, (z + 1) * len), so that apart from each tile's last part all CTAs of a split tile are equally long: started
// longest tile first, the short ones fill the end.
struct SplitPlan {
  int len = INT_MAX, max_parts = 1;
  __host__ __device__ int parts(int units) const { return units <= len ? 1 : (units + len - 1) / len; }
  __host__ __device__ int begin(int z) const { return z == 0 ? 0 : z * len; }
  __host__ __device__ int end(int z, int units) const { return units - begin(z) <= len ? units : begin(z) + len; }
};

constexpr int SPLIT_SMS = 148;
constexpr int SPLIT_MAX_PARTS = 32;
constexpr int64_t SPLIT_MAX_BYTES = (int64_t)256 << 20;    // scratch a split may ask for

// Estimated time (us) of a grid of `tiles` x `heads` CTAs split into parts of at most `len` blocks: work and the longest CTA,
// or whole waves when all CTAs are alike; a split pays for one more launch and for its partials' way to memory and back.
// work, top: blocks of all tiles of a head, of the longest tile; unit_us: one block, cta_us: set-up and epilogue of a CTA,
// part_bytes: one CTA's partial.
inline double split_cost_us(bool uniform, int64_t work, int top, int len, int tiles, int heads, double unit_us, double cta_us,
                            int64_t part_bytes) {
  const int c = (top + len - 1) / len;
  const double longest = (double)len * unit_us + cta_us;
  double ctas, t;
  if (uniform) {
    ctas = (double)tiles * heads * c;
    t = (double)(((int64_t)ctas + SPLIT_SMS - 1) / SPLIT_SMS) * longest;
  } else {
    ctas = c == 1 ? (double)tiles * heads : ((double)work / len + 0.5 * tiles) * heads;
    const double even = ((double)work * heads * unit_us + ctas * cta_us) / SPLIT_SMS;
    // longest first, the short ones fill the end: close to an even share, plus a little for the last CTAs
    t = even + (ctas > SPLIT_SMS ? 0.15 * longest : 0.0);
    if (t < longest) t = longest;
  }
  // 4 us for the launch of the sum: measured when a kernel started only after the one before had ended
  return c == 1 ? t : t + 4.0 + ctas * part_bytes * 2.0 / 5.0e6;
}

// The plan with the smallest estimate; a split has to promise a tenth.  Grids of many waves are not looked at: they have
// nothing to gain.
inline SplitPlan split_plan(const SplitUnits& u, int tiles, int heads, double unit_us, double cta_us, int64_t part_bytes) {
  SplitPlan best;
  if ((int64_t)tiles * heads > 6 * SPLIT_SMS) return best;
  int64_t work = 0;
  int top = 0;
  for (int t = 0; t < tiles; ++t) {
    const int n = u(t);
    work += n;
    top = n > top ? n : top;
  }
  if (top < 2) return best;
  const bool uniform = u.kind == 0;
  double best_us = 0.9 * split_cost_us(uniform, work, top, top, tiles, heads, unit_us, cta_us, part_bytes);
  for (int c = 2; c <= SPLIT_MAX_PARTS && c <= top; c = c < 8 ? c + 1 : c + c / 4) {
    SplitPlan p;
    p.len = (top + c - 1) / c;
    p.max_parts = p.parts(top);
    const double us = split_cost_us(uniform, work, top, p.len, tiles, heads, unit_us, cta_us, part_bytes);
    if (us < best_us && (int64_t)tiles * heads * p.max_parts * part_bytes <= SPLIT_MAX_BYTES) { best_us = us; best = p; }
  }
  return best;
}

}  // namespace ody
