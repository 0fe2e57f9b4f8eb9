// Shared pieces of the attention kernels: position maps, tile visibility, dropout hash.
#pragma once
#include "common/bounds.cuh"
#include "common/sm100.cuh"

namespace ra {
namespace attn {

// Global token position of local index i. A shard is one contiguous run (half >= length) or two
// runs of `half` tokens each (zig-zag layout); `half` is a multiple of the 128-row tile.
struct PosMap {
  int off0;
  int off1;
  int half;
  __device__ __forceinline__ int operator()(int i) const {
    return i < half ? off0 + i : off1 + (i - half);
  }
};

struct MaskParams {
  int Sq, Sk;
  int cbs;  // causal block size, 0 = not causal
  PosMap qmap, kmap;
  const int* seg_q;     // (B, Sq) segment ids of the local queries, or null
  const int* seg_k;     // (B, Sk) segment ids of this KV block, or null
  const int* seg_q_mm;  // (B, ceil(Sq/128), 2) per-tile {min, max} segment id, or null
  const int* seg_k_mm;  // (B, ceil(Sk/128), 2)
  const float* bias;    // (B, Hb, Sk) additive key bias in natural-log units, or null
  long long bias_stride_b, bias_stride_h;
  unsigned int seed_lo, seed_hi;
  unsigned int drop_threshold;  // 0 = dropout off; logit dropped iff hash < threshold
  // Optional boolean mask as a bitmap (bit set = attend), rows padded to whole 128-column tiles. The forward
  // reads it by query row (word w of row q: keys 32w..32w+31 of this KV block), the backward by kv row (word w
  // of row k: queries 32w..32w+31); strides in 32-bit words, row stride a multiple of 4.
  const uint32_t* keep;
  long long keep_sb, keep_sh, keep_sr;
  // kind of the bitmap's 128 x 128 tiles [b][h][q tile][k tile]: 0 no bit set, 1 all set, 2 some; or null
  const uint8_t* keep_tiles;
  long long keep_tiles_sb, keep_tiles_sh;
};

// Kind of a tile of the bitmap (2 where it is not known, or there is none).
__device__ __forceinline__ int bitmap_tile(const MaskParams& m, int b, int h, int qi0, int k0) {
  if (!m.keep_tiles) return 2;
  return m.keep_tiles[b * m.keep_tiles_sb + h * m.keep_tiles_sh + static_cast<long long>(qi0 >> 7) * ((m.Sk + 127) >> 7) + (k0 >> 7)];
}

// False when every entry of the (128 q x 128 k) tile is masked by the causal rule or because the
// segment-id ranges of the two tiles are disjoint, or by the bitmap. qi0/k0 are local start indices.
__device__ __forceinline__ bool tile_visible(const MaskParams& m, int b, int h, int qi0, int k0) {
  if (qi0 >= m.Sq || k0 >= m.Sk) return false;
  if (m.keep_tiles && bitmap_tile(m, b, h, qi0, k0) == 0) return false;
  if (m.cbs == 1) {  // plain causal: no divisions on the hot path
    if (m.qmap(min(qi0 + 127, m.Sq - 1)) < m.kmap(k0)) return false;
  } else if (m.cbs) {
    const int q_hi = m.qmap(min(qi0 + 127, m.Sq - 1));
    const int k_lo = m.kmap(k0);
    if (q_hi / m.cbs < k_lo / m.cbs) return false;
  }
  if (m.seg_q_mm) {
    const int nqt = (m.Sq + 127) >> 7, nkt = (m.Sk + 127) >> 7;
    const int* qm = m.seg_q_mm + (static_cast<long long>(b) * nqt + (qi0 >> 7)) * 2;
    const int* km = m.seg_k_mm + (static_cast<long long>(b) * nkt + (k0 >> 7)) * 2;
    if (qm[1] < km[0] || km[1] < qm[0]) return false;
  }
  return true;
}

// ---- per-CTA visibility bitmask ---------------------------------------------------------------------
// With segment ids every evaluation of tile_visible costs a global-memory round trip. A CTA that walked
// its tiles one by one spent ~100 us on that walk alone (256 tiles); instead all threads of the CTA
// evaluate the predicate once, 32 tiles per warp step, into a bitmask in shared memory, and the roles
// walk the set bits.
constexpr int VIS_WORDS = 256;  // capacity: 8192 tiles (1M rows); longer launches fall back to the direct walk

// bit t of `words` = pred(t) for t < n (n <= 32 * VIS_WORDS). Call with every thread of the CTA, converged,
// `nthreads` a multiple of 32; a __syncthreads() must follow before the mask is read.
template <typename F>
__device__ __forceinline__ void fill_visibility(uint32_t* words, int n, int tid, int nthreads, F pred) {
  const int n_pad = (n + 31) & ~31;
  for (int t = tid; t < n_pad; t += nthreads) {  // a warp's 32 values of t share one word: uniform trip count
    const bool v = t < n && pred(t);
    const uint32_t bits = __ballot_sync(0xffffffffu, v);
    if ((tid & 31) == 0) words[t >> 5] = bits;
  }
}

// Smallest set bit at or after t, or n.
__device__ __forceinline__ int vis_next(const uint32_t* words, int t, int n) {
  while (t < n) {
    const uint32_t w = words[t >> 5] >> (t & 31);
    if (w) return t + __ffs(static_cast<int>(w)) - 1;  // bits at or beyond n are never set
    t = (t | 31) + 1;
  }
  return n;
}

// Walks the tiles that are set in a mask, or in one or both of two masks VIS_WORDS apart, in registers: a word is loaded once for its 32
// tiles. vis_next for every tile took some 300 cycles where the tensor core's operands keep shared memory busy, twice a
// tile in the warp that issues the products.
template <int MASKS>
struct VisWalk {
  const uint32_t* words;
  uint32_t a, b;  // what is left of the words of tiles at .. at + 31
  int at, n;
  __device__ __forceinline__ VisWalk(const uint32_t* w, int n_) : words(w), a(n_ > 0 ? w[0] : 0u), b(MASKS == 2 && n_ > 0 ? w[VIS_WORDS] : 0u), at(0), n(n_) {}
  // next tile, or n; in which of the masks it is set
  __device__ __forceinline__ int next(bool& in_a, bool& in_b) {
    while ((a | b) == 0u) {
      at += 32;
      if (at >= n) return n;
      a = words[at >> 5];
      if (MASKS == 2) b = words[VIS_WORDS + (at >> 5)];
    }
    const uint32_t both = a | b, bit = both & (~both + 1u);
    in_a = (a & bit) != 0u;
    in_b = (b & bit) != 0u;
    a &= ~bit;
    b &= ~bit;
    return at + __ffs(static_cast<int>(bit)) - 1;
  }
};

// What may hide single entries of a visible tile; 0: nothing does. With segment ids the common case inside packed documents
// much longer than a tile is that both tiles lie in one and the same segment (per-tile min == max, equal on both sides).
// bits: the bitmap has a hole in this tile, or there is dropout.
enum TileMask : int { kMaskEdge = 1 /* causal rule or end of the keys */, kMaskSeg = 2, kMaskBits = 4 /* bitmap, dropout */ };
__device__ __forceinline__ int tile_mask(const MaskParams& m, int b, bool bits, int qi0, int k0) {
  int kind = bits ? kMaskBits : 0;
  if (k0 + 128 > m.Sk) kind |= kMaskEdge;
  if (m.seg_q) {
    bool one = false;
    if (m.seg_q_mm) {
      const int nqt = (m.Sq + 127) >> 7, nkt = (m.Sk + 127) >> 7;
      const int* qm = m.seg_q_mm + (static_cast<long long>(b) * nqt + (qi0 >> 7)) * 2;
      const int* km = m.seg_k_mm + (static_cast<long long>(b) * nkt + (k0 >> 7)) * 2;
      const int q_lo = qm[0], k_lo = km[0];
      one = q_lo == qm[1] && k_lo == km[1] && q_lo == k_lo;
    }
    if (!one) kind |= kMaskSeg;
  }
  if (m.cbs == 1) {
    if (m.qmap(qi0) < m.kmap(min(k0 + 127, m.Sk - 1))) kind |= kMaskEdge;
  } else if (m.cbs) {
    const int q_lo = m.qmap(qi0);
    const int k_hi = m.kmap(min(k0 + 127, m.Sk - 1));
    if (q_lo / m.cbs < k_hi / m.cbs) kind |= kMaskEdge;
  }
  return kind;
}

// keep[c] bit i &= (seg[32 c + i] == my_seg) for N words, by warp votes: the lanes of a warp have few different ids (rows of a
// tile are neighbours in the sequence), and one vote per word answers for all lanes with the same one. Converged warps.
template <int N>
__device__ __forceinline__ void keep_segment(uint32_t* keep, const int* seg, int my_seg, int lane) {
  int col[N];
#pragma unroll
  for (int c = 0; c < N; ++c) col[c] = seg[32 * c + lane];
  uint32_t todo = 0xffffffffu;
  while (todo) {
    const int id = __shfl_sync(0xffffffffu, my_seg, __ffs(static_cast<int>(todo)) - 1);
    const bool mine = id == my_seg;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const uint32_t same = __ballot_sync(0xffffffffu, col[c] == id);
      if (mine) keep[c] &= same;
    }
    todo &= ~__ballot_sync(0xffffffffu, mine);
  }
}

// Number of leading columns of the k tile that the causal rule and the sequence end leave
// visible to a query at global position qpos: column c is masked iff c >= limit.
__device__ __forceinline__ int causal_col_limit(const MaskParams& m, int qpos, int k0) {
  int limit = m.Sk - k0;
  if (m.cbs) {
    const int kbase = m.kmap(k0);
    const long long lim =
        (m.cbs == 1 ? static_cast<long long>(qpos) + 1 : (static_cast<long long>(qpos / m.cbs) + 1) * m.cbs) - kbase;
    limit = static_cast<int>(lim < limit ? (lim < 0 ? 0 : lim) : limit);
  }
  return limit;
}

__device__ __forceinline__ unsigned int mix32(unsigned int x) {
  x ^= x >> 16;
  x *= 0x7FEB352Du;
  x ^= x >> 15;
  x *= 0x846CA68Bu;
  x ^= x >> 16;
  return x;
}
// Counter-based dropout hash of (seed, b*H+h, q position, k position).
__device__ __forceinline__ unsigned int dropout_hash(unsigned int seed_lo, unsigned int seed_hi,
                                                     unsigned int bh, unsigned int qpos,
                                                     unsigned int kpos) {
  unsigned int x = qpos * 0x9E3779B1u + kpos * 0x85EBCA77u + bh * 0xC2B2AE3Du + seed_lo;
  x = mix32(x);
  x = mix32((x ^ seed_hi) + kpos);
  return x;
}

// Order of the CTAs of a launch. A (batch, head) has n tiles of work; under a causal rule they differ in length and the grid's
// last wave is as long as the longest tile that starts in it. So the heads are walked in `groups` of as good as equal size, the longest
// tiles of a group's heads first: unit idx -> tile rank (0 = longest) and (batch, head).
struct TileOrder {
  int n, base, larger;  // tiles of a head; heads of a group, the first `larger` groups have one more
  TileOrder() = default;
  TileOrder(int n_, int bh, int groups) : n(n_), base(bh / groups), larger(bh % groups) {}
  __device__ __forceinline__ void operator()(int idx, int& rank, int& bh_idx) const {
    int size = base + 1, first = 0;
    if (idx >= larger * n * size) {
      idx -= larger * n * size;
      first = larger * size;
      size = base;
    }
    const int g = idx / (n * size), r = idx - g * n * size;
    rank = r / size;
    bh_idx = first + g * size + r - rank * size;
  }
};

// Into how many groups. A group of `need` heads keeps every SM busy for as long as its longest tile takes (tile lengths 1 .. n:
// n (n + 1) / 2 units a head against n on each of `sms`), so that the tail of the launch is the shortest tiles; heads whose operands take
// no more than 24 MB together lose nothing by sharing the L2 and are walked together anyway; and above 64 MB, about half of the L2, the
// tiles of a head no longer find its operands there. The groups are of equal size: with groups of `need` heads and a rest, 16 heads as
// 3 + 3 + 3 + 3 + 3 + 1, the long tiles of the last head run alone at the end. us on B200, causal, D 128, a build that walks the heads one
// after the other / groups of `need` and a rest / this:
//   backward 16 x 16384 3294 / 3434 / 3187, 16 x 8192 869 / 914 / 761, 8 x 8192 476 / 443 / 385, 32 x 4096 492 / 452 / 440, 16 x 2048 98 / 68 / 68
//   forward 4 x 32768 1036 / 1134 / 979, 8 x 16384 618 / 541 / 490, 16 x 8192 366 / 272 / 264, 32 x 4096 238 / 158 / 161, 32 x 2048 95 / 54 / 54
inline int head_groups(int n, int bh, long long head_bytes, int sms) {
  const long long bytes = head_bytes > 0 ? head_bytes : 1;
  const long long fit = (64ll << 20) / bytes, roomy = (24ll << 20) / bytes;
  long long need = (2ll * sms + n) / (n + 1);
  if (need < roomy) need = roomy;
  if (need > fit) need = fit;
  if (need > bh) need = bh;
  if (need < 1) need = 1;
  const long long most = bh / need, least = fit > 0 ? (bh + fit - 1) / fit : bh;
  return static_cast<int>(most > least ? most : least);
}

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

}  // namespace attn
}  // namespace ra
