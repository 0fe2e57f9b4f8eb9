// Flash-attention forward for sm_100a with carry-in, the per-device compute of one ring step.
//
// One CTA owns 256 query rows (two 128-row tiles) of one (batch, head) and walks the visible
// 128-row KV tiles:
//   warps 0-3   producer group (registers trimmed): warp 0 TMA (Q once, K through a 2-stage ring), warp 2 TMA (V through
//               another), warp 1 tcgen05.mma issuer: S_w = Q_w K^T (SS), O_w += P_w V (P in TMEM)
//   warps 4-7   softmax group for tile 0, warps 8-11 for tile 1 (registers raised): tcgen05.ld S,
//               mask, online softmax with lazy rescale of O in TMEM, P written back over S as bf16
// TMEM: S0 | S1 | O0 | O1 (4 x 128 columns). While one group runs its softmax the tensor core
// works on the other tile, so MMA and exp overlap without a third party.
//
// HALVES: one CTA owns 128 query rows and its two softmax groups take every second visible KV tile each, with accumulators
// of their own (O0, O1) that meet in the epilogue. The pipeline is the same (two tiles of scores in flight), a CTA's chain is half
// as long and there are twice as many CTAs, at the price of loading K and V once per 128 rows. For launches with few
// query tiles; see fwd_shape(). Such a launch may also be split over the keys (`splits`): then every CTA takes its share of
// the visible tiles, partial results go to fp32 buffers and attn_merge_kernel puts them together.
//
// The epilogue normalises O, optionally merges it with the carry (o_prev, lse_prev) of earlier
// ring steps and writes fp32 (intermediate step) or bf16 (last step) plus the log-sum-exp.
// Leading CTAs of the grid can be given a copy job: they pull the next ring step's KV block from
// a peer GPU's memory into a local slab with plain 16-byte loads while the other CTAs compute.
#include "attn_common.cuh"
#include "common/host_util.h"

RA_BOUNDS_TRANSLATION_UNIT()

namespace ra {
namespace attn {

constexpr int FWD_THREADS = 384;
constexpr int KV_STAGES = 2;
// Register re-balancing: the CTA owns 384 x 168 registers (launch bounds); setmaxnreg.inc blocks
// until registers are free, so the per-group budgets must fit in that allocation.
constexpr int FWD_REGS_PRODUCER = 88;   // warps 0-3
constexpr int FWD_REGS_SOFTMAX = 208;   // warps 4-11
static_assert(128 * FWD_REGS_PRODUCER + 256 * FWD_REGS_SOFTMAX <= FWD_THREADS * 168,
              "setmaxnreg budgets exceed the registers the CTA was launched with");

struct FwdParams {
  int B, H;
  TileOrder order;  // of the 256-row query pairs (HALVES: 128-row tiles)
  int splits;       // HALVES: CTAs per query tile, neighbours in the grid; `out` and `lse_out` of split s are s * split_o, s * split_l further
  long long split_o, split_l;
  MaskParams mask;
  float scale_log2;  // log2(e) / sqrt(D)
  void* out;
  int out_fp32;
  long long o_stride_b, o_stride_s, o_stride_h;  // elements
  float* lse_out;         // (B, H, Sq)
  const float* o_prev;    // (B, Sq, H, D) fp32 contiguous, or null
  const float* lse_prev;  // (B, H, Sq), or null
  const uint4* copy_src;
  uint4* copy_dst;
  long long copy_n16;
  int copy_ctas;
  int* status;
  // EXT: width of the values that is stored (the tile's columns past it are zero), per-head attention sink (one more entry
  // exp(sink) in the denominator, without a value), per-head output gate sigmoid(gate[row, h])
  int dv;
  const float* sink;            // (H), or null
  const __nv_bfloat16* gate;    // (B * Sq, gate_ld), or null
  long long gate_ld;
  // EXT: a query sees keys at distances 0 .. window - 1 (0: no limit); kv_share query heads read one key/value head (0 or 1:
  // each its own); keys and values lie in a ring of k_rows rows (a multiple of 128): key 0 in row k_row0 (0 rows: no ring)
  int window, kv_share, k_row0, k_rows;
};

// Window rules for a 128 x 128 tile: some entry lies inside the window; every entry does.
__device__ __forceinline__ bool tile_in_window(const MaskParams& m, int window, int qi0, int k0) {
  return !window || m.qmap(qi0) - m.kmap(min(k0 + 127, m.Sk - 1)) < window;
}
__device__ __forceinline__ bool tile_window_plain(const MaskParams& m, int window, int qi0, int k0) {
  return !window || m.qmap(min(qi0 + 127, m.Sq - 1)) - m.kmap(k0) < window;
}

// NS: 64-wide slabs of the query/key width, DV: value width of the tile. The second K stage is given up where it does not
// fit beside two tiles of wide queries; V keeps two.
template <int NS, int DV>
struct FwdSmem {
  static constexpr int SLAB_BYTES = 128 * 64 * 2;  // one 64-wide d slab of a 128-row tile
  static constexpr int Q_TILE_BYTES = NS * SLAB_BYTES;
  static constexpr int K_TILE_BYTES = NS * SLAB_BYTES;
  static constexpr int V_TILE_BYTES = 128 * DV * 2;
  static constexpr int K_STAGES = (2 + KV_STAGES) * Q_TILE_BYTES + KV_STAGES * V_TILE_BYTES <= 200 * 1024 ? KV_STAGES : 1;
  static constexpr int Q_OFF = 0;
  static constexpr int K_OFF = Q_OFF + 2 * Q_TILE_BYTES;
  static constexpr int V_OFF = K_OFF + K_STAGES * K_TILE_BYTES;
  static constexpr int AUX_OFF = V_OFF + KV_STAGES * V_TILE_BYTES;  // seg/bias staging
  static constexpr int AUX_BYTES = 2 /*wg*/ * 2 /*buf*/ * 128 * 4 * 2 /*seg+bias*/;
  static constexpr int BAR_OFF = AUX_OFF + AUX_BYTES;
  static constexpr int VIS_OFF = BAR_OFF + 256;  // [2 q tiles][VIS_WORDS] visibility of the kv tiles
  static constexpr int BIAS_OFF = VIS_OFF + 2 * VIS_WORDS * 4;  // [2][VIS_WORDS] kv tiles whose bias is not all 0, not all -inf
  static constexpr int TOTAL = BIAS_OFF + 2 * VIS_WORDS * 4 + 1024;
};

// NQ: slabs of the query/key part that every head has of its own; NR: slabs of a second part (maps tma_q2, tma_k2) whose
// keys all heads share; DV: value width. EXT adds the options of an inference layer (see FwdParams); without it NR = 0 and
// the head dim is 64 NQ = DV.
template <int NQ, int NR, int DV, bool EXT, bool HALVES>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                const __grid_constant__ CUtensorMap tma_v, const __grid_constant__ CUtensorMap tma_q2,
                const __grid_constant__ CUtensorMap tma_k2, const FwdParams p) {
  constexpr int NSLAB = NQ + NR, VSLAB = DV / 64;
  using SM = FwdSmem<NSLAB, DV>;
  constexpr int K_STAGES = SM::K_STAGES;

  // A failure recorded earlier on this stream (for example a ring barrier that timed out) turns
  // every later attention kernel into a no-op, so nothing touches the memory of a lost peer.
  if (p.status && *reinterpret_cast<const volatile int*>(p.status) != 0) return;

  // ------------------------------------------------------------ copy CTAs (ring KV pull)
  if (static_cast<int>(blockIdx.x) < p.copy_ctas) {
    const long long stride = static_cast<long long>(p.copy_ctas) * FWD_THREADS;
    long long i = static_cast<long long>(blockIdx.x) * FWD_THREADS + threadIdx.x;
    // 16 loads of 16 bytes in flight per thread: the pull is bound by bytes in flight over the NVLink round
    // trip; finishing early hands the SM to a compute CTA sooner
    for (; i + 15 * stride < p.copy_n16; i += 16 * stride) {
      uint4 r[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) r[u] = p.copy_src[i + u * stride];
#pragma unroll
      for (int u = 0; u < 16; ++u) p.copy_dst[i + u * stride] = r[u];
    }
    for (; i < p.copy_n16; i += stride) p.copy_dst[i] = p.copy_src[i];
    return;
  }

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem + SM::Q_OFF;
  uint8_t* sK = smem + SM::K_OFF;
  uint8_t* sV = smem + SM::V_OFF;
  int* sSeg = reinterpret_cast<int*>(smem + SM::AUX_OFF);              // [wg][buf][128]
  float* sBias = reinterpret_cast<float*>(smem + SM::AUX_OFF) + 512;   // [wg][buf][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFF);
  uint64_t* q_full = bars;             // 1
  uint64_t* k_full = bars + 1;         // KV_STAGES
  uint64_t* k_empty = bars + 3;
  uint64_t* v_full = bars + 5;
  uint64_t* v_empty = bars + 7;
  uint64_t* s_full = bars + 9;         // 2 (per q tile)
  uint64_t* p_full = bars + 11;        // 2
  uint64_t* o_done = bars + 13;        // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const WaitCtx wc{abort_flag, p.status};
  const MaskParams& mk = p.mask;

  // block -> (q pair, head, batch): heavy (late) q tiles first, a few heads at a time
  int bh, qp, split = 0;
  {
    int unit = static_cast<int>(blockIdx.x) - p.copy_ctas;
    if (HALVES) {
      split = unit % p.splits;
      unit /= p.splits;
    }
    p.order(unit, qp, bh);
    qp = p.order.n - 1 - qp;
  }
  const int h = bh % p.H;
  const int b = bh / p.H;
  const int h_kv = EXT && p.kv_share > 1 ? h / p.kv_share : h;
  constexpr int NT = HALVES ? 1 : 2;  // q tiles
  const int q0 = qp * (NT * 128);
  const int nk = (mk.Sk + 127) / 128;
  // row of a key tile (tiles never straddle the end of the ring)
  auto kv_row = [&](int k0) -> int {
    if (!EXT || !p.k_rows) return k0;
    const int r = p.k_row0 + k0;
    return r >= p.k_rows ? r - p.k_rows : r;
  };
  auto visible = [&](int w, int j) -> bool {
    return tile_visible(mk, b, h, q0 + w * 128, j * 128) && (!EXT || tile_in_window(mk, p.window, q0 + w * 128, j * 128));
  };

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < KV_STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int w = 0; w < 2; ++w) {
      mbar_init(&s_full[w], 1);
      mbar_init(&p_full[w], 4);
      mbar_init(&o_done[w], 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tma_q);
    tma_prefetch_desc(&tma_k);
    tma_prefetch_desc(&tma_v);
    if (NR) {
      tma_prefetch_desc(&tma_q2);
      tma_prefetch_desc(&tma_k2);
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  // which kv tiles each of the two q tiles sees
  uint32_t* sVis = reinterpret_cast<uint32_t*>(smem + SM::VIS_OFF);
  const bool use_vis = nk <= 32 * VIS_WORDS;
  // A key bias is mostly a padding mask: tiles whose bias is 0 throughout need no addition, tiles where it is -inf throughout
  // (in the log2 domain, so the type's lowest value too) are not visited. One warp looks at a tile.
  uint32_t* sAdd = reinterpret_cast<uint32_t*>(smem + SM::BIAS_OFF);
  uint32_t* sLive = sAdd + VIS_WORDS;
  if (use_vis && mk.bias) {
    for (int t = threadIdx.x; t < VIS_WORDS; t += FWD_THREADS) sAdd[t] = sLive[t] = 0u;
    __syncthreads();
    const float* bias = mk.bias + b * mk.bias_stride_b + h * mk.bias_stride_h;
    for (int j = warp; j < nk; j += FWD_THREADS / 32) {
      bool add = false, live = false;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int kc = j * 128 + c * 32 + lane;
        const float v = kc < mk.Sk ? bias[kc] * kLog2e : -INFINITY;
        live |= v != -INFINITY;
        add |= kc < mk.Sk && v != 0.f;
      }
      add = __any_sync(0xffffffffu, add);
      live = __any_sync(0xffffffffu, live);
      if (lane == 0) {
        if (add) atomicOr(&sAdd[j >> 5], 1u << (j & 31));
        if (live) atomicOr(&sLive[j >> 5], 1u << (j & 31));
      }
    }
    __syncthreads();
  }
  if (use_vis) {
#pragma unroll
    for (int w = 0; w < NT; ++w)
      fill_visibility(sVis + w * VIS_WORDS, nk, static_cast<int>(threadIdx.x), FWD_THREADS,
                      [&](int j) { return visible(w, j) && (!mk.bias || ((sLive[j >> 5] >> (j & 31)) & 1u)); });
  }
  if (HALVES && p.splits > 1) {  // keep this split's share of the visible tiles (the launcher sees to use_vis)
    __syncthreads();
    if (threadIdx.x == 0) {
      const int words = (nk + 31) >> 5;
      int total = 0;
      for (int i = 0; i < words; ++i) total += __popc(sVis[i]);
      const int lo = static_cast<int>(static_cast<long long>(total) * split / p.splits);
      const int hi = static_cast<int>(static_cast<long long>(total) * (split + 1) / p.splits);
      int seen = 0;
      for (int i = 0; i < words; ++i) {
        uint32_t left = sVis[i], mine = 0;
        const int n = __popc(left);
        if (seen >= lo && seen + n <= hi) {
          mine = left;
        } else {
          for (int at = seen; left; ++at, left &= left - 1)
            if (at >= lo && at < hi) mine |= left & (~left + 1);
        }
        seen += n;
        sVis[i] = mine;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS[2] = {tmem_base, tmem_base + 128};
  const uint32_t tO[2] = {tmem_base + 256, tmem_base + 384};

  // next kv tile of a walk that any of this CTA's query tiles (`next_any`) or query tile w (`next_of`) sees, or nk
  auto next_any = [&](VisWalk<NT>& wk, bool& s0, bool& s1) -> int {
    if (use_vis) return wk.next(s0, s1);
    for (; wk.at < nk; ++wk.at) {
      s0 = visible(0, wk.at);
      s1 = NT == 2 && visible(1, wk.at);
      if (s0 || s1) return wk.at++;
    }
    return nk;
  };
  auto next_of = [&](VisWalk<1>& wk, int w) -> int {
    bool s0, s1;
    if (use_vis) return wk.next(s0, s1);
    for (; wk.at < nk; ++wk.at)
      if (visible(w, wk.at)) return wk.at++;
    return nk;
  };

  if (warp < 4) setmaxnreg_dec<FWD_REGS_PRODUCER>();
  if (warp == 0 || warp == 2) {
    // ================================================================ TMA producers: Q and K (warp 0), V (warp 2)
    // Scores are issued up to two tiles ahead of the product with V, so a stage of K comes free earlier than the stage of V that a common walk
    // would have to fill first.
    if (lane == 0) {
      if (warp == 0) {
        mbar_arrive_expect_tx(q_full, NT * SM::Q_TILE_BYTES);
#pragma unroll
        for (int w = 0; w < NT; ++w)
#pragma unroll
          for (int s = 0; s < NSLAB; ++s)
            tma_load_4d(sQ + w * SM::Q_TILE_BYTES + s * SM::SLAB_BYTES, s < NQ ? &tma_q : &tma_q2, q_full,
                        (s < NQ ? s : s - NQ) * 64, h, q0 + w * 128, b);
      }
      int it = 0;
      VisWalk<NT> walk(sVis, use_vis ? nk : 0);
      bool s0, s1;
      for (int j = next_any(walk, s0, s1); j < nk; j = next_any(walk, s0, s1)) {
        const int row = kv_row(j * 128);
        if (warp == 0) {
          const int st = it % K_STAGES;
          if (!mbar_wait_relaxed(&k_empty[st], ((it / K_STAGES) & 1) ^ 1u, wc, kTimeoutSmemEmpty)) break;
          mbar_arrive_expect_tx(&k_full[st], SM::K_TILE_BYTES);
#pragma unroll
          for (int s = 0; s < NSLAB; ++s)
            tma_load_4d(sK + st * SM::K_TILE_BYTES + s * SM::SLAB_BYTES, s < NQ ? &tma_k : &tma_k2, &k_full[st],
                        (s < NQ ? s : s - NQ) * 64, s < NQ ? h_kv : 0, row, b);
        } else {
          const int st = it & 1;
          if (!mbar_wait_relaxed(&v_empty[st], ((it >> 1) & 1) ^ 1u, wc, kTimeoutSmemEmpty)) break;
          mbar_arrive_expect_tx(&v_full[st], SM::V_TILE_BYTES);
#pragma unroll
          for (int s = 0; s < VSLAB; ++s)
            tma_load_4d(sV + st * SM::V_TILE_BYTES + s * SM::SLAB_BYTES, &tma_v, &v_full[st], s * 64, h_kv, row, b);
        }
        ++it;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================================================ MMA issuer (warp-uniform flow)
    // One warp for both groups: it keeps them half a period apart, so that one group's exponentials run beside the other's products. (With
    // a warp for each they fall into step, fight for the same unit and then wait for the same one: 4790 cycles a pair of tiles instead of 3890.)
    // Nothing but the wait for a group's probabilities may stand between its products: a look at a barrier that has long completed takes
    // some 200 cycles beside a busy tensor core, so the stages of K and V are waited for ahead of it.
    {
      const bool leader = elect_one();
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_o = make_idesc_bf16(128, DV, 0, 1);
      const uint64_t q_desc[2] = {make_smem_desc(smem_u32(sQ), 16, 1024),
                                  make_smem_desc(smem_u32(sQ + SM::Q_TILE_BYTES), 16, 1024)};
      const uint64_t k_desc[2] = {make_smem_desc(smem_u32(sK), 16, 1024),
                                  make_smem_desc(smem_u32(sK + (K_STAGES - 1) * SM::K_TILE_BYTES), 16, 1024)};
      const uint64_t v_desc[2] = {make_smem_desc(smem_u32(sV), SM::SLAB_BYTES, 1024),
                                  make_smem_desc(smem_u32(sV + SM::V_TILE_BYTES), SM::SLAB_BYTES, 1024)};
      auto issue_s = [&](int w, int st) {
#pragma unroll
        for (int kk = 0; kk < NSLAB * 4; ++kk) {
          const uint32_t off = (kk >> 2) * SM::SLAB_BYTES + (kk & 3) * 32;
          if (leader)
            umma_ss(tS[w], desc_advance(q_desc[HALVES ? 0 : w], off), desc_advance(k_desc[st], off), idesc_s,
                    kk != 0 ? 1u : 0u);
        }
        if (leader) umma_commit(&s_full[w]);
      };
      auto issue_pv = [&](int w, int st, bool acc) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          // A = P_w in TMEM: 16 bf16 of K per step = 8 columns. B = V, MN-major: 16 kv rows = 2 KiB.
          if (leader)
            umma_ts(tO[w], tS[w] + kk * 8, desc_advance(v_desc[st], kk * 2048), idesc_o,
                    (acc || kk != 0) ? 1u : 0u);
        }
        if (leader) umma_commit(&o_done[w]);
      };
      VisWalk<NT> walk(sVis, use_vis ? nk : 0);
      bool ok = mbar_wait(q_full, 0, wc, kTimeoutSmemFull);
      bool n0, n1;
      if constexpr (HALVES) {
        // tile `it` of the walk belongs to group it & 1; its scores are issued two tiles ahead, behind the product of
        // the probabilities they overwrite
        int n_s = 0;  // tiles whose scores are issued
        bool more = ok && next_any(walk, n0, n1) < nk;
        for (int i = 0; i < 2 && more; ++i) {
          more = mbar_wait(&k_full[n_s % K_STAGES], (n_s / K_STAGES) & 1, wc, kTimeoutSmemFull);
          if (!(ok = more)) break;
          tc_fence_after();
          issue_s(n_s & 1, n_s % K_STAGES);
          if (leader) umma_commit(&k_empty[n_s % K_STAGES]);
          ++n_s;
          more = next_any(walk, n0, n1) < nk;
        }
        for (int it = 0; ok && it < n_s; ++it) {
          const int w = it & 1, st = it & 1;
          const uint32_t ph = (it >> 1) & 1;
          if (!mbar_wait(&v_full[st], ph, wc, kTimeoutSmemFull)) break;
          if (more && !mbar_wait(&k_full[n_s % K_STAGES], (n_s / K_STAGES) & 1, wc, kTimeoutSmemFull)) break;
          if (!mbar_wait(&p_full[w], ph, wc, kTimeoutTmemFull)) break;
          tc_fence_after();
          issue_pv(w, st, it > 1);
          if (leader) umma_commit(&v_empty[st]);
          if (more) {
            issue_s(n_s & 1, n_s % K_STAGES);
            if (leader) umma_commit(&k_empty[n_s % K_STAGES]);
            ++n_s;
            more = next_any(walk, n0, n1) < nk;
          }
        }
      } else {
        bool v0 = false, v1 = false;
        int it = 0;
        int cnt[2] = {0, 0};
        bool have = ok && next_any(walk, v0, v1) < nk;
        if (have) {
          ok = mbar_wait(&k_full[0], 0, wc, kTimeoutSmemFull);
          if (ok) {
            tc_fence_after();
            if (v0) issue_s(0, 0);
            if (v1) issue_s(1, 0);
            if (leader) umma_commit(&k_empty[0]);
          }
        }
        while (ok && have) {
          n0 = n1 = false;
          const bool more = next_any(walk, n0, n1) < nk;
          const int st = it & 1;
          const uint32_t ph = (it >> 1) & 1;
          const int stn = (it + 1) % K_STAGES;  // K stage of the next tile
          const uint32_t phn = ((it + 1) / K_STAGES) & 1;
          if (!mbar_wait(&v_full[st], ph, wc, kTimeoutSmemFull)) break;
          // (a single stage of K is filled behind the scores of this tile: waited for where it is needed)
          if (K_STAGES > 1 && more && !mbar_wait(&k_full[stn], phn, wc, kTimeoutSmemFull)) break;
          if (v0) {
            if (!mbar_wait(&p_full[0], cnt[0] & 1, wc, kTimeoutTmemFull)) break;
            tc_fence_after();
            issue_pv(0, st, cnt[0] != 0);
            ++cnt[0];
          }
          if (more && n0) {
            if (K_STAGES == 1 && !mbar_wait(&k_full[stn], phn, wc, kTimeoutSmemFull)) break;
            issue_s(0, stn);
          }
          if (v1) {
            if (!mbar_wait(&p_full[1], cnt[1] & 1, wc, kTimeoutTmemFull)) break;
            tc_fence_after();
            issue_pv(1, st, cnt[1] != 0);
            ++cnt[1];
          }
          if (leader) umma_commit(&v_empty[st]);
          if (more) {
            if (K_STAGES == 1 && !mbar_wait(&k_full[stn], phn, wc, kTimeoutSmemFull)) break;
            if (n1) issue_s(1, stn);
            if (leader) umma_commit(&k_empty[stn]);
          }
          have = more;
          v0 = n0;
          v1 = n1;
          ++it;
        }
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ================================================================ softmax groups
    setmaxnreg_inc<FWD_REGS_SOFTMAX>();
    const int w = (warp - 4) >> 2;  // q tile handled by this group (HALVES: parity of its tiles in the walk)
    const int wv = HALVES ? 0 : w;  // visibility mask it walks
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int wg_tid = quad * 32 + lane;
    const int qi0 = q0 + wv * 128;
    const int qi = qi0 + row;
    const bool row_valid = qi < mk.Sq;
    const int qpos = mk.qmap(row_valid ? qi : mk.Sq - 1);
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const int my_seg = (mk.seg_q && row_valid) ? mk.seg_q[static_cast<long long>(b) * mk.Sq + qi] : 0;
    const unsigned int bh_u = static_cast<unsigned int>(b * p.H + h);

    float m_ref = -INFINITY;  // running reference max (scaled log2 domain)
    float l = 0.f;
    int cnt = 0;
    bool alive = true;
    bool settled = false;  // every row of the warp has a reference, and none has outgrown its own for kWatch tiles
    int watch = 0;         // how many of those are to come
    constexpr int kWatch = 64;
    constexpr float kGrown = 255.f;  // no summand of a smaller sum reaches the 2^8 above which the accumulator is rescaled

    // Kinds of this query tile's bitmap tiles; without them every tile's bits are looked at, if there are any. A pointer for the whole
    // walk: asked for per tile out of the launch's parameters they cost every launch, those without a bitmap too (2 x 32 heads x 512, not
    // causal, 19.2 -> 18.5 us; the backward's 16 x 2048 118.6 -> 116.3).
    const uint8_t* tile_kinds = mk.keep_tiles && !mk.drop_threshold
                                    ? mk.keep_tiles + b * mk.keep_tiles_sb + h * mk.keep_tiles_sh + static_cast<long long>(qi0 >> 7) * nk
                                    : nullptr;
    const bool bits = mk.drop_threshold || mk.keep;
    // every role walks the same visibility mask, so skips stay consistent
    VisWalk<1> walk(sVis + wv * VIS_WORDS, use_vis ? nk : 0);
    auto next_mine = [&]() {
      int j = next_of(walk, wv);
      if (HALVES && (w == 1 || cnt > 0) && j < nk) j = next_of(walk, wv);  // the other group takes the one between
      return j;
    };
    for (int j = next_mine(); j < nk && alive; j = next_mine()) {
      const int k0 = j * 128;
      const int kind = tile_mask(mk, b, tile_kinds ? tile_kinds[j] != 1 : bits, qi0, k0) | (EXT && !tile_window_plain(mk, p.window, qi0, k0) ? kMaskEdge : 0);
      const bool biased = mk.bias && (!use_vis || ((sAdd[j >> 5] >> (j & 31)) & 1u));
      const int buf = cnt & 1;
      if ((kind & kMaskSeg) || biased) {
        const int kc = k0 + wg_tid;
        if (kind & kMaskSeg)
          sSeg[(w * 2 + buf) * 128 + wg_tid] =
              kc < mk.Sk ? mk.seg_k[static_cast<long long>(b) * mk.Sk + kc] : -1;
        if (biased)
          sBias[(w * 2 + buf) * 128 + wg_tid] =
              kc < mk.Sk ? mk.bias[b * mk.bias_stride_b + h * mk.bias_stride_h + kc] * kLog2e : 0.f;
        named_bar_sync(1 + w, 128);
      }
      // A wait that gives up must end the loop for the whole warp (the TMEM loads and stores are
      // warp-collective). The lanes agree on that in the vote behind the exponentials, which exists
      // anyway; until then every lane carries on (a lane that gave up merely loads a stale tile).
      const bool s_ok = mbar_wait(&s_full[w], cnt & 1, wc, kTimeoutTmemFull);
      tc_fence_after();
      uint32_t pk[64];
      float sum;
      // The scores of a tile are scaled by the reference of the tiles before it, without a look at their maximum, as long as no row's
      // sum can hold a summand that asks for another reference (also as long as some row of the warp has seen no key, the maximum comes first):
      // the 64 three-way maxima ahead of the first exponential took 490 of a tile's 3900 cycles. Otherwise the tile is taken again from
      // TMEM, with the maximum, and the next kWatch tiles that stay below it are too: a second pass costs a tile, the maximum 2 (D 128) to
      // 7 % (D 64) of one. References, and so results, are those of a walk that always looks. us, always / never twice in kWatch tiles / as often
      // as it comes, 32 heads x 4096, causal, D 128, logits as in training 162 / 156 / 158; a bias that rises by 0.5 a key 240 / 256 / 338.
      for (;;) {
        uint32_t sr[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld_x32(tS[w] + lane_base + c * 32, sr + c * 32);
        tmem_ld_wait();

        float sc = p.scale_log2;  // multiplier still to be applied to sr[] inside the exp
        // Masked tiles differ from plain ones only in this block: what hides an entry is gathered into four words of bits per
        // row first (segment ids by warp votes), a bias is added by a loop of its own, and only words with a hole are walked
        // column by column. One loop over 128 columns that tested bits, ids and bias for each took 8.9 us a tile (D = 64) where a plain
        // tile takes 1.2: far more instructions than the caches hold, refetched every time.
        if (kind != 0 || biased) {
          uint32_t keep[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
          if (kind & kMaskEdge) {
            const int limit = causal_col_limit(mk, qpos, k0);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int n = limit - 32 * c;
              keep[c] = n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : ((1u << n) - 1u));
            }
            if (EXT && p.window) {
              const int first = qpos - p.window + 1 - mk.kmap(k0);  // columns before it are too far away
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const int n = first - 32 * c;
                keep[c] &= n >= 32 ? 0u : (n <= 0 ? 0xffffffffu : ~((1u << n) - 1u));
              }
            }
          }
          if (kind & kMaskBits) {
            if (mk.keep) {
              uint4 kb = make_uint4(0u, 0u, 0u, 0u);
              if (RA_IN_BOUNDS((k0 >> 5), 4, mk.keep_sr, kTagAttnMaskBits))
                kb = *reinterpret_cast<const uint4*>(
                  mk.keep + b * mk.keep_sb + h * mk.keep_sh + static_cast<long long>(row_valid ? qi : mk.Sq - 1) * mk.keep_sr +
                  (k0 >> 5));
              keep[0] &= kb.x;
              keep[1] &= kb.y;
              keep[2] &= kb.z;
              keep[3] &= kb.w;
            }
            if (mk.drop_threshold) {
              const unsigned int kpos0 = static_cast<unsigned int>(mk.kmap(k0));
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                uint32_t drop = 0;
#pragma unroll 1
                for (int i = 0; i < 32; ++i)
                  drop |= static_cast<uint32_t>(dropout_hash(mk.seed_lo, mk.seed_hi, bh_u, static_cast<unsigned int>(qpos),
                                                             kpos0 + c * 32 + i) < mk.drop_threshold)
                          << i;
                keep[c] &= ~drop;
              }
            }
          }
          if (kind & kMaskSeg) keep_segment<4>(keep, sSeg + (w * 2 + buf) * 128, my_seg, lane);
          if (biased) {
            const float4* bias4 = reinterpret_cast<const float4*>(sBias + (w * 2 + buf) * 128);
#pragma unroll
            for (int g = 0; g < 32; ++g) {
              const float4 bs = bias4[g];
              sr[4 * g] = __float_as_uint(fmaf(__uint_as_float(sr[4 * g]), sc, bs.x));
              sr[4 * g + 1] = __float_as_uint(fmaf(__uint_as_float(sr[4 * g + 1]), sc, bs.y));
              sr[4 * g + 2] = __float_as_uint(fmaf(__uint_as_float(sr[4 * g + 2]), sc, bs.z));
              sr[4 * g + 3] = __float_as_uint(fmaf(__uint_as_float(sr[4 * g + 3]), sc, bs.w));
            }
            sc = 1.0f;
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (__all_sync(0xffffffffu, keep[c] == 0xffffffffu)) continue;
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (!((keep[c] >> i) & 1u)) sr[32 * c + i] = 0xff800000u;  // -inf
          }
        }
        if (!settled) {  // online softmax with lazy rescale of the accumulator
          float mc[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) mc[c] = fmaxf(__uint_as_float(sr[32 * c]), __uint_as_float(sr[32 * c + 1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              mc[c] = max3(mc[c], __uint_as_float(sr[32 * c + i]), __uint_as_float(sr[32 * c + i + 1]));
          }
          const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mc[0], mc[1]), fmaxf(mc[2], mc[3])) * sc);
          // also true when m_ref is -inf and m_new is finite
          const bool need = cnt != 0 && m_new > m_ref + 8.0f;
          if (cnt == 0) {
            m_ref = m_new;
          } else if (__any_sync(0xffffffffu, need)) {
            if (!__all_sync(0xffffffffu, mbar_wait(&o_done[w], (cnt - 1) & 1, wc, kTimeoutTmemFull))) {
              alive = false;
              break;
            }
            tc_fence_after();
            if (__any_sync(0xffffffffu, need && m_ref != -INFINITY)) watch = kWatch + 1;
            const float alpha = (m_new == -INFINITY) ? 1.0f : exp2_approx(m_ref - m_new);
#pragma unroll 1
            for (int c = 0; c < DV / 32; ++c) {
              uint32_t o[32];
              tmem_ld_x32(tO[w] + lane_base + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_x32(tO[w] + lane_base + c * 32, o);
            }
            tmem_st_wait();
            l *= alpha;
            m_ref = m_new;
          }
        }
        const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
        const uint64_t neg_m2 = f2_pack(-m_use, -m_use);
        const uint64_t sc2 = f2_pack(sc, sc);
        uint64_t sum2 = f2_pack(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          float x0, x1;
          f2_unpack(f2_fma(f2_pack_u(sr[2 * i], sr[2 * i + 1]), sc2, neg_m2), x0, x1);
          const float p0 = exp2_approx(x0), p1 = exp2_approx(x1);
          sum2 = f2_add(sum2, f2_pack(p0, p1));
          pk[i] = pack_bf16x2(p0, p1);
        }
        float sum_hi;
        f2_unpack(sum2, sum, sum_hi);
        sum += sum_hi;
        const bool grown = !(sum <= kGrown);  // (NaN too)
        if (!__any_sync(0xffffffffu, (settled && grown) || !s_ok)) break;
        if (__any_sync(0xffffffffu, !s_ok)) {
          alive = false;
          break;
        }
        settled = false;
        watch = kWatch + 1;
      }
      if (!alive) break;
      if (!settled) {
        const bool quiet = __all_sync(0xffffffffu, sum <= kGrown && m_ref != -INFINITY);
        watch = quiet ? max(watch - 1, 0) : (watch > 0 ? kWatch : 0);
        settled = quiet && watch == 0;
      }
      l += sum;
      tmem_st_x32(tS[w] + lane_base, pk);
      tmem_st_x32(tS[w] + lane_base + 32, pk + 32);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive_warp(&p_full[w]);
      ++cnt;
    }

    // ---- epilogue: normalise, merge with carry, store
    if (alive && cnt > 0) alive = mbar_wait(&o_done[w], (cnt - 1) & 1, wc, kTimeoutTmemFull);
    tc_fence_after();
    // HALVES: this group finishes half of the columns of all rows. It hands the other half and its (reference, sum) to the
    // other group through shared memory that held K and V: both groups have seen their last product complete, so no
    // load and no MMA touches it any more. 16-byte pieces, XOR-swizzled by the row.
    constexpr int HALF = DV / 2;               // columns
    constexpr int PIECES = HALF / 4;
    float own_mul = 1.f, other_mul = 0.f;      // factors of the two accumulators
    float* const other_row = reinterpret_cast<float*>(sK) + ((1 - w) * 128 + row) * HALF;  // what the other group left for us
    // The carry's log-sum-exp. lse_out may be the same tensor (a ring accumulates in place), and with HALVES both groups need the value
    // that one of them overwrites: so it is read here, ahead of the barriers below, and the store comes behind them.
    const long long lse_idx = (static_cast<long long>(b) * p.H + h) * mk.Sq + qi;
    const float lse_carry = p.o_prev && row_valid ? p.lse_prev[lse_idx] : -INFINITY;
    if (HALVES) {
      float2* stat = reinterpret_cast<float2*>(sSeg);  // [group][128]: masks are done with
      named_bar_sync(3, 256);
      float* dst = reinterpret_cast<float*>(sK) + (w * 128 + row) * HALF;
#pragma unroll 1
      for (int c = 0; c < HALF / 32; ++c) {
        uint32_t o[32];
        if (cnt > 0) {
          tmem_ld_x32(tO[w] + lane_base + (1 - w) * HALF + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<uint4*>(dst + (((c * 8 + i) ^ (row & (PIECES - 1))) << 2)) =
              make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
      }
      stat[w * 128 + row] = make_float2(cnt > 0 ? m_ref : -INFINITY, l);
      named_bar_sync(3, 256);
      const float2 other = stat[(1 - w) * 128 + row];
      const float m_own = cnt > 0 ? m_ref : -INFINITY;
      const float m_all = fmaxf(m_own, other.x);
      const float mu = m_all == -INFINITY ? 0.f : m_all;
      own_mul = exp2_approx(m_own - mu);
      other_mul = exp2_approx(other.x - mu);
      l = l * own_mul + other.y * other_mul;
      m_ref = m_all;
    }
    float inv_l = 0.f;
    float lse = -INFINITY;
    if ((HALVES || cnt > 0) && l > 0.f) {
      inv_l = 1.0f / l;
      lse = (m_ref + log2f(l)) * kLn2;
    } else if (HALVES && p.splits > 1 && l != l) {
      lse = l;  // tells attn_merge_kernel that the row is no number, not that this split sees none of its keys
    }
    float w_prev = 0.f, w_this = 1.f;
    if (p.o_prev && row_valid) {
      const float mxl = fmaxf(lse_carry, lse);
      if (mxl == -INFINITY) {
        w_prev = 0.f;
        w_this = 0.f;
      } else {
        const float ep = __expf(lse_carry - mxl), et = __expf(lse - mxl);
        const float tot = ep + et;
        w_prev = ep / tot;
        w_this = et / tot;
        lse = mxl + __logf(tot);
      }
    }
    if ((!EXT || p.lse_out) && row_valid && (!HALVES || w == 0) &&
        RA_IN_BOUNDS(lse_idx, 1, static_cast<long long>(p.B) * p.H * mk.Sq, kTagAttnFwdLse))
      p.lse_out[(HALVES ? split * p.split_l : 0) + lse_idx] = lse;
    float mul = inv_l * w_this;
    if (EXT && row_valid) {
      if (p.sink) mul /= 1.f + expf(p.sink[h] - lse);
      if (p.gate)
        mul /= 1.f + expf(-__bfloat162float(p.gate[(static_cast<long long>(b) * mk.Sq + qi) * p.gate_ld + h]));
    }
    const float* oprev_row =
        p.o_prev ? p.o_prev + ((static_cast<long long>(b) * mk.Sq + qi) * p.H + h) * DV : nullptr;
    const long long o_off = b * p.o_stride_b + static_cast<long long>(qi) * p.o_stride_s + h * p.o_stride_h +
                            (HALVES ? split * p.split_o : 0);
#pragma unroll 1
    for (int c = HALVES ? w * (HALF / 32) : 0; c < (HALVES ? (w + 1) * (HALF / 32) : DV / 32); ++c) {
      uint32_t o[32];
      if (cnt > 0) {
        tmem_ld_x32(tO[w] + lane_base + c * 32, o);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0u;
      }
      if (row_valid && RA_IN_BOUNDS(qi, 1, mk.Sq, kTagAttnFwdOut) && RA_IN_BOUNDS(c * 32, 32, DV, kTagAttnFwdOut)) {
        float f[32];
        if (HALVES) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(
                other_row + ((((c - w * (HALF / 32)) * 8 + i) ^ (row & (PIECES - 1))) << 2));
            f[4 * i] = (__uint_as_float(o[4 * i]) * own_mul + x.x * other_mul) * mul;
            f[4 * i + 1] = (__uint_as_float(o[4 * i + 1]) * own_mul + x.y * other_mul) * mul;
            f[4 * i + 2] = (__uint_as_float(o[4 * i + 2]) * own_mul + x.z * other_mul) * mul;
            f[4 * i + 3] = (__uint_as_float(o[4 * i + 3]) * own_mul + x.w * other_mul) * mul;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(o[i]) * mul;
        }
        if (oprev_row) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 pv = *reinterpret_cast<const float4*>(oprev_row + c * 32 + 4 * i);
            f[4 * i] += pv.x * w_prev;
            f[4 * i + 1] += pv.y * w_prev;
            f[4 * i + 2] += pv.z * w_prev;
            f[4 * i + 3] += pv.w * w_prev;
          }
        }
        if (p.out_fp32) {
          float* dst = reinterpret_cast<float*>(p.out) + o_off + c * 32;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(dst + 4 * i) =
                make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
        } else {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.out) + o_off + c * 32;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (EXT && c * 32 + i * 8 >= p.dv) continue;
            uint4 v;
            v.x = pack_bf16x2(f[8 * i], f[8 * i + 1]);
            v.y = pack_bf16x2(f[8 * i + 2], f[8 * i + 3]);
            v.z = pack_bf16x2(f[8 * i + 4], f[8 * i + 5]);
            v.w = pack_bf16x2(f[8 * i + 6], f[8 * i + 7]);
            *reinterpret_cast<uint4*>(dst + 8 * i) = v;
          }
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) bounded_drain_pause();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Puts the partial results of a launch split over the keys together: o (splits, B, Sq, H, D) and lse (splits, B, H, Sq) fp32 ->
// out (bf16 or fp32 view) and lse_out (B, H, Sq). A warp per row. Every split's row is read and multiplied, by a weight of 0 where the
// split sees no key (lse = -inf) or its keys weigh nothing beside the others': NaN and infinities then come out as they do of a launch that is
// not split, where a probability of 0 meets them in the product with V. lse is NaN where a split's sum is.
template <int D>
__global__ void __launch_bounds__(256) attn_merge_kernel(const float* __restrict__ o, const float* __restrict__ lse, int splits,
                                                         int B, int H, int Sq, void* out, int out_fp32, long long o_sb,
                                                         long long o_ss, long long o_sh, float* __restrict__ lse_out) {
  constexpr int PER = D / 32;
  const long long rows = static_cast<long long>(B) * Sq * H;
  const long long row = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int h = static_cast<int>(row % H), q = static_cast<int>(row / H % Sq), b = static_cast<int>(row / H / Sq);
  const long long at = (static_cast<long long>(b) * H + h) * Sq + q;
  float mx = -INFINITY;
  for (int s = 0; s < splits; ++s) mx = fmaxf(mx, lse[s * rows + at]);  // (of the numbers among them)
  float acc[PER], sum = 0.f;
#pragma unroll
  for (int e = 0; e < PER; ++e) acc[e] = 0.f;
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float l = lse[s * rows + at];
    const float w = l == -INFINITY ? 0.f : expf(l - mx);
    const float* src = o + (s * rows + row) * D + lane * PER;
    sum += w;
#pragma unroll
    for (int e = 0; e < PER; e += 2) {
      const float2 v = *reinterpret_cast<const float2*>(src + e);
      acc[e] += w * v.x;
      acc[e + 1] += w * v.y;
    }
  }
  const float inv = sum == 0.f ? 0.f : 1.f / sum;
  if (lane == 0 && RA_IN_BOUNDS(at, 1, rows, kTagAttnFwdLse)) lse_out[at] = sum > 0.f ? mx + logf(sum) : -INFINITY;
  const long long off = b * o_sb + static_cast<long long>(q) * o_ss + h * o_sh + lane * PER;
#pragma unroll
  for (int e = 0; e < PER; e += 2) {
    if (out_fp32) {
      *reinterpret_cast<float2*>(static_cast<float*>(out) + off + e) = make_float2(acc[e] * inv, acc[e + 1] * inv);
    } else {
      *reinterpret_cast<uint32_t*>(static_cast<__nv_bfloat16*>(out) + off + e) = pack_bf16x2(acc[e] * inv, acc[e + 1] * inv);
    }
  }
}

// How a launch is cut up: two query tiles a CTA ("pairs"), one (HALVES), or one and its keys over several CTAs. The estimate is the time of
// the launch in hundredths of a step of pairs (two 128 x 128 tiles; 1.8 us at D 128, 1.6 at D 64): a CTA takes its steps and a
// fixed cost (start-up, first loads, epilogue), and the CTAs, longest first, go to whichever SM is free: the SMs are busy for the average load at
// least, and the k-th CTA of an SM is no shorter than the longest that starts behind k - 1 full rounds. Segment ids and bitmaps are not
// looked at: the causal rule alone gives the lengths.
// The constants are fitted to 110 launches of both head dims timed in every form on B200 (256 to 32768 query rows, 2 to 32 heads, causal or not, up to
// 65536 keys): the choice takes 0.2 % longer than the fastest form on average, 6 % at worst (three of them more than 3 %). A step of HALVES
// loads K and V for one query tile only and takes as long as one of pairs all the same; its CTAs end later (the two groups' results
// are put together). us, pairs / HALVES / keys over 2 / over 4 CTAs, D 128, * the choice:
//   32 heads x 512, not causal 17.2 / 13.6* / 35.0 / -       32 x 4096, not causal 277* / 283 / - / -     32 x 4096, causal 153* / 182 / - / -
//   4 x 4096, causal 68.5 / 41.4* / 48.1 / 68.0              16 x 2048, not causal 40.7* / 49.9 / 92 / 126 16 x 500 on 16384 keys 245 / 136 / 85* / 99
//   32 x 1000 on 16384 keys 249* / 275 / 327 / 343           32 x 128 on 4096 keys 62 / 41 / 32 / 25*     2 x 12318, causal 187 / 106* / 120 / 149
// With constants of an earlier kernel (a step of HALVES 15 % longer, its CTA 1.4 steps shorter) the last of them went to keys over two CTAs, and the
// choice took 0.7 % longer than the fastest on average, 14 % at worst.
struct FwdShape {
  bool halves;
  int splits;
};
inline FwdShape fwd_shape(int B, int H, int Sq, int Sk, int D, int cbs, long long q_off, long long k_off, bool one_run, bool may_split) {
  const int step = D == 128 ? 99 : 102, cta = D == 128 ? 630 : 635, cta_pair = D == 128 ? 565 : 590;  // of HALVES, HALVES, pairs
  constexpr int step_pair = 100, merge = 425;  // merge: partial results out and in again, one more launch
  const int nk = (Sk + 127) / 128, nq = (Sq + 127) / 128, sms = sm_count();
  const long long bh = static_cast<long long>(B) * H;
  FwdShape best{false, 1};
  if (nq > 1024 || bh * nq > 64ll * sms) return best;  // plenty of work per SM: two query tiles share the loads of K and V
  auto tiles = [&](int i) -> long long {  // visible kv tiles of query tile i; no fewer than of the tile before
    const long long v = cbs && one_run ? (q_off + i * 128ll + 127 - k_off) / 128 + 1 : nk;
    return v < 0 ? 0 : (v > nk ? nk : v);
  };
  // `each` CTAs of each of n lengths, cost(0) the longest
  auto makespan = [&](int n, long long each, auto cost) -> long long {
    long long sum = 0;
    for (int i = 0; i < n; ++i) sum += cost(i);
    long long t = sum * each / sms;
    for (long long k = 1, at = 0; at < n * each; ++k, at += sms) {
      const long long c = k * cost(static_cast<int>(at / each));
      if (c > t) t = c;
    }
    return t;
  };
  long long t_best = makespan((nq + 1) / 2, bh, [&](int i) {
    const int later = 2 * ((nq + 1) / 2 - 1 - i) + 1;  // second tile of the i-th pair from the end
    return tiles(later < nq ? later : nq - 1) * step_pair + cta_pair;
  });
  long long all = 0;
  for (int i = 0; i < nq; ++i) all += tiles(i);
  for (int s = 1; s <= (may_split ? 32 : 1) && s <= nk; ++s) {
    const long long extra = s > 1 ? merge : 0;
    // more CTAs only add to the average load: no larger s is worth a look
    if (((all * step / 2 + static_cast<long long>(s) * nq * cta) * bh / sms + extra) * 100 >= t_best * 97) break;
    const long long t = extra + makespan(nq, bh * s, [&](int i) { return (tiles(nq - 1 - i) + 2 * s - 1) / (2 * s) * step + cta; });
    if (t * 100 < t_best * 97) {
      t_best = t;
      best = FwdShape{true, s};
    }
  }
  return best;
}

}  // namespace attn
}  // namespace ra

namespace {
// (B, S, H, D) bf16 view with element strides -> 4-D map (d, h, s, b), box 64 x 1 x 128 x 1.
int make_bshd_map(CUtensorMap* m, const void* base, int B, int S, int H, int D, long long sb,
                  long long ss, long long sh) {
  uint64_t dims[4] = {static_cast<uint64_t>(D), static_cast<uint64_t>(H), static_cast<uint64_t>(S),
                      static_cast<uint64_t>(B)};
  uint64_t str[3] = {static_cast<uint64_t>(sh) * 2, static_cast<uint64_t>(ss) * 2,
                     static_cast<uint64_t>(sb) * 2};
  uint32_t box[4] = {64, 1, 128, 1};
  return ra::make_tmap_bf16_sw128(m, base, 4, dims, str, box);
}

template <int NQ, int NR, int DV, bool EXT = (NR > 0), bool HALVES = false>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tq2,
               const CUtensorMap& tk2, const ra::attn::FwdParams& p, long long grid, cudaStream_t s) {
  using namespace ra::attn;
  auto kern = attn_fwd_kernel<NQ, NR, DV, EXT, HALVES>;
  constexpr int smem = FwdSmem<NQ + NR, DV>::TOTAL;
  static_assert(smem <= 227 * 1024, "tile buffers do not fit in shared memory");
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    ra::set_error("attn_fwd: smem attribute");
    return ra::kHostLaunchFail;
  }
  kern<<<static_cast<unsigned>(grid), FWD_THREADS, smem, s>>>(tq, tk, tv, tq2, tk2, p);
  return ra::check_launch("attn_fwd_kernel");
}
}  // namespace

struct RaAttnFwdArgs {
  const void* q; const void* k; const void* v;
  long long q_sb, q_ss, q_sh;   // element strides of (B, Sq, H, D) views; D contiguous
  long long k_sb, k_ss, k_sh;
  long long v_sb, v_ss, v_sh;
  void* out; long long o_sb, o_ss, o_sh; int out_fp32;
  float* lse_out;
  const float* o_prev; const float* lse_prev;
  int B, H, Sq, Sk, D;
  float softmax_scale;          // 1/sqrt(D)
  int causal_block_size;
  int q_off0, q_off1, q_half;
  int k_off0, k_off1, k_half;
  const int* seg_q; const int* seg_k; const int* seg_q_mm; const int* seg_k_mm;
  const float* bias; long long bias_sb, bias_sh;
  unsigned long long seed; unsigned int drop_threshold;
  const unsigned int* keep; long long keep_sb, keep_sh, keep_sr;  // boolean mask bitmap by query row, or null
  const unsigned char* keep_tiles; long long keep_tiles_sb, keep_tiles_sh;  // kinds of its tiles, or null
  const void* copy_src; void* copy_dst; long long copy_bytes; int copy_ctas;
  int* status;
  void* stream;
  // splits > 1 (as ra_attn_fwd_splits says, or any number up to 32): the keys are split over that many CTAs per query tile; ws
  // holds splits * B * Sq * H * (D + 1) floats. Without o_prev and a copy job.
  int splits;
  float* ws;
};

namespace {
ra::attn::FwdShape shape_of(const RaAttnFwdArgs* a, bool may_split) {
  const bool one_run = a->q_half >= a->Sq && a->k_half >= a->Sk;
  return ra::attn::fwd_shape(a->B, a->H, a->Sq, a->Sk, a->D, a->causal_block_size, a->q_off0, a->k_off0, one_run, may_split);
}
}  // namespace

// Over how many CTAs per query tile ra_attn_fwd would like to split the keys of this launch (1: not at all).
extern "C" int ra_attn_fwd_splits(const RaAttnFwdArgs* a) {
  if (a->B <= 0 || a->H <= 0 || a->Sq <= 0 || a->Sk <= 0) return 1;
  if (a->o_prev || a->copy_src || (a->Sk + 127) / 128 > 32 * ra::attn::VIS_WORDS) return 1;
  return shape_of(a, true).splits;
}

extern "C" int ra_attn_fwd(const RaAttnFwdArgs* a) {
  using namespace ra;
  using namespace ra::attn;
  if (a->D != 128 && a->D != 64) {
    set_error("ra_attn_fwd: head_dim must be 64 or 128");
    return kHostBadArg;
  }
  if (a->B <= 0 || a->H <= 0 || a->Sq <= 0 || a->Sk <= 0 || (a->q_half < a->Sq && a->q_half % 128) ||
      (a->k_half < a->Sk && a->k_half % 128) || (a->copy_bytes % 16)) {
    set_error("ra_attn_fwd: bad shape");
    return kHostBadArg;
  }
  const int splits = a->splits > 1 ? a->splits : 1;
  if (splits > 1 && (splits > 32 || !a->ws || (reinterpret_cast<uintptr_t>(a->ws) & 15) || a->o_prev || a->copy_src ||
                     !a->lse_out || (a->Sk + 127) / 128 > 32 * VIS_WORDS)) {
    set_error("ra_attn_fwd: a launch split over the keys takes a workspace, at most 32 splits, no carry and no copy job");
    return kHostBadArg;
  }
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_map(&tq, a->q, a->B, a->Sq, a->H, a->D, a->q_sb, a->q_ss, a->q_sh))) return rc;
  if ((rc = make_bshd_map(&tk, a->k, a->B, a->Sk, a->H, a->D, a->k_sb, a->k_ss, a->k_sh))) return rc;
  if ((rc = make_bshd_map(&tv, a->v, a->B, a->Sk, a->H, a->D, a->v_sb, a->v_ss, a->v_sh))) return rc;
  FwdParams p;
  p.B = a->B;
  p.H = a->H;
  p.mask.Sq = a->Sq;
  p.mask.Sk = a->Sk;
  p.mask.cbs = a->causal_block_size;
  p.mask.qmap = PosMap{a->q_off0, a->q_off1, a->q_half};
  p.mask.kmap = PosMap{a->k_off0, a->k_off1, a->k_half};
  p.mask.seg_q = a->seg_q;
  p.mask.seg_k = a->seg_k;
  p.mask.seg_q_mm = a->seg_q_mm;
  p.mask.seg_k_mm = a->seg_k_mm;
  p.mask.bias = a->bias;
  p.mask.bias_stride_b = a->bias_sb;
  p.mask.bias_stride_h = a->bias_sh;
  p.mask.seed_lo = static_cast<unsigned int>(a->seed & 0xffffffffull);
  p.mask.seed_hi = static_cast<unsigned int>(a->seed >> 32);
  p.mask.drop_threshold = a->drop_threshold;
  p.mask.keep = a->keep;
  p.mask.keep_sb = a->keep_sb;
  p.mask.keep_sh = a->keep_sh;
  p.mask.keep_sr = a->keep_sr;
  p.mask.keep_tiles = a->keep_tiles;
  p.mask.keep_tiles_sb = a->keep_tiles_sb;
  p.mask.keep_tiles_sh = a->keep_tiles_sh;
  if (a->keep && ((a->keep_sr % 4) || (a->keep_sb % 4) || (a->keep_sh % 4) || (reinterpret_cast<uintptr_t>(a->keep) & 15))) {
    set_error("ra_attn_fwd: mask bitmap rows must be 16-byte aligned");
    return kHostBadArg;
  }
  p.scale_log2 = a->softmax_scale * kLog2e;
  p.out = a->out;
  p.out_fp32 = a->out_fp32;
  p.o_stride_b = a->o_sb;
  p.o_stride_s = a->o_ss;
  p.o_stride_h = a->o_sh;
  p.lse_out = a->lse_out;
  p.o_prev = a->o_prev;
  p.lse_prev = a->lse_prev;
  p.copy_src = reinterpret_cast<const uint4*>(a->copy_src);
  p.copy_dst = reinterpret_cast<uint4*>(a->copy_dst);
  p.copy_n16 = a->copy_bytes / 16;
  p.copy_ctas = (a->copy_src && a->copy_bytes > 0) ? a->copy_ctas : 0;
  p.status = a->status;
  p.dv = a->D;
  p.sink = nullptr;
  p.gate = nullptr;
  p.gate_ld = 0;
  p.window = p.kv_share = p.k_row0 = p.k_rows = 0;
  const bool halves = splits > 1 || shape_of(a, false).halves;
  const int n_q = halves ? (a->Sq + 127) / 128 : (a->Sq + 255) / 256;
  p.order = TileOrder{n_q, a->B * a->H,
                      a->causal_block_size ? head_groups(n_q, a->B * a->H, 4ll * a->Sk * a->D, sm_count()) : a->B * a->H};
  p.splits = splits;
  p.split_l = static_cast<long long>(a->B) * a->H * a->Sq;
  p.split_o = p.split_l * a->D;
  if (splits > 1) {
    p.out = a->ws;
    p.out_fp32 = 1;
    p.o_stride_h = a->D;
    p.o_stride_s = static_cast<long long>(a->H) * a->D;
    p.o_stride_b = p.o_stride_s * a->Sq;
    p.lse_out = a->ws + splits * p.split_o;
  }
  const long long grid = static_cast<long long>(n_q) * a->H * a->B * splits + p.copy_ctas;
  cudaStream_t s = static_cast<cudaStream_t>(a->stream);
  if (halves)
    rc = a->D == 128 ? launch_fwd<2, 0, 128, false, true>(tq, tk, tv, tq, tk, p, grid, s)
                     : launch_fwd<1, 0, 64, false, true>(tq, tk, tv, tq, tk, p, grid, s);
  else
    rc = a->D == 128 ? launch_fwd<2, 0, 128>(tq, tk, tv, tq, tk, p, grid, s)
                     : launch_fwd<1, 0, 64>(tq, tk, tv, tq, tk, p, grid, s);
  if (rc || splits == 1) return rc;
  const unsigned blocks = static_cast<unsigned>((p.split_l + 7) / 8);
  auto merge = a->D == 128 ? attn_merge_kernel<128> : attn_merge_kernel<64>;
  merge<<<blocks, 256, 0, s>>>(static_cast<const float*>(p.out), p.lse_out, splits, a->B, a->H, a->Sq, a->out, a->out_fp32, a->o_sb,
                               a->o_ss, a->o_sh, a->lse_out);
  return check_launch("attn_merge_kernel");
}

// Causal attention with two-part queries and keys: score = (q1 . k1 + q2 . k2) * scale, where k2 is shared by all heads.
// q (B, Sq, H, d1 + d2) with q1 first, k1 (B, Sk, H, d1), k2 (B, Sk, d2), v (B, Sk, H, dv), out (B, Sq, H, dv); bf16, element
// strides, innermost contiguous; query i sits at position q_pos0 + i, key j at j. d1 <= 128, d2 <= 64, dv <= 128, all
// multiples of 8. `sink` (H) fp32 and `gate` (B * Sq, gate_ld) bf16 are optional (see FwdParams).
struct RaAttnTwoPartArgs {
  const void* q; long long q_sb, q_ss, q_sh;
  const void* k1; long long k1_sb, k1_ss, k1_sh;
  const void* k2; long long k2_sb, k2_ss;
  const void* v; long long v_sb, v_ss, v_sh;
  void* out; long long o_sb, o_ss, o_sh;
  const float* sink;
  const void* gate; long long gate_ld;
  int B, H, Sq, Sk, d1, d2, dv;
  float scale;
  int q_pos0;
  int* status;
  void* stream;
};

extern "C" int ra_attn_two_part(const RaAttnTwoPartArgs* a) {
  using namespace ra;
  using namespace ra::attn;
  const long long odd = (a->q_sb | a->q_ss | a->q_sh | a->k1_sb | a->k1_ss | a->k1_sh | a->k2_sb | a->k2_ss | a->v_sb |
                         a->v_ss | a->v_sh | a->o_sb | a->o_ss | a->o_sh) & 7;
  if (a->B < 1 || a->H < 1 || a->Sq < 1 || a->Sk < 1 || a->q_pos0 < 0 || a->d1 < 8 || a->d1 > 128 || a->d1 % 8 ||
      a->d2 < 8 || a->d2 > 64 || a->d2 % 8 || a->dv < 8 || a->dv > 128 || a->dv % 8 || odd ||
      ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k1) | reinterpret_cast<uintptr_t>(a->k2) |
        reinterpret_cast<uintptr_t>(a->v) | reinterpret_cast<uintptr_t>(a->out)) & 15)) {
    set_error("ra_attn_two_part: bad shape or alignment");
    return kHostBadArg;
  }
  CUtensorMap tq, tk, tv, tq2, tk2;
  int rc;
  const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(a->q);
  if ((rc = make_bshd_map(&tq, q, a->B, a->Sq, a->H, a->d1, a->q_sb, a->q_ss, a->q_sh))) return rc;
  if ((rc = make_bshd_map(&tq2, q + a->d1, a->B, a->Sq, a->H, a->d2, a->q_sb, a->q_ss, a->q_sh))) return rc;
  if ((rc = make_bshd_map(&tk, a->k1, a->B, a->Sk, a->H, a->d1, a->k1_sb, a->k1_ss, a->k1_sh))) return rc;
  if ((rc = make_bshd_map(&tk2, a->k2, a->B, a->Sk, 1, a->d2, a->k2_sb, a->k2_ss, a->k2_ss))) return rc;
  if ((rc = make_bshd_map(&tv, a->v, a->B, a->Sk, a->H, a->dv, a->v_sb, a->v_ss, a->v_sh))) return rc;
  FwdParams p = {};
  p.B = a->B;
  p.H = a->H;
  p.mask.Sq = a->Sq;
  p.mask.Sk = a->Sk;
  p.mask.cbs = 1;
  p.mask.qmap = PosMap{a->q_pos0, 0, 1 << 30};
  p.mask.kmap = PosMap{0, 0, 1 << 30};
  p.scale_log2 = a->scale * kLog2e;
  p.out = a->out;
  p.o_stride_b = a->o_sb;
  p.o_stride_s = a->o_ss;
  p.o_stride_h = a->o_sh;
  p.status = a->status;
  p.dv = a->dv;
  p.sink = a->sink;
  p.gate = static_cast<const __nv_bfloat16*>(a->gate);
  p.gate_ld = a->gate_ld;
  const int n_qp = (a->Sq + 255) / 256;
  p.order = TileOrder{n_qp, a->B * a->H, a->B * a->H};
  const long long grid = static_cast<long long>(n_qp) * a->H * a->B;
  cudaStream_t s = static_cast<cudaStream_t>(a->stream);
  if (a->d1 > 64)
    return a->dv > 64 ? launch_fwd<2, 1, 128>(tq, tk, tv, tq2, tk2, p, grid, s)
                      : launch_fwd<2, 1, 64>(tq, tk, tv, tq2, tk2, p, grid, s);
  return a->dv > 64 ? launch_fwd<1, 1, 128>(tq, tk, tv, tq2, tk2, p, grid, s)
                    : launch_fwd<1, 1, 64>(tq, tk, tv, tq2, tk2, p, grid, s);
}

// Causal attention over the last `window` keys with grouped heads, a sink per head and keys and values in a ring: query i sits
// at position q_pos0 + i and sees the keys at distances 0 .. window - 1; position j lies in row j % k_rows, k_rows a multiple
// of 128. Head h reads key/value head h / (H / G). q (B, Sq, H, dk), k (B, k_rows, G, dk), v (B, k_rows, G, dv), out (B, Sq,
// H, dv): bf16, element strides, innermost contiguous; dk and dv multiples of 8 up to 128. `sink` (H) fp32.
struct RaAttnWindowArgs {
  const void* q; long long q_sb, q_ss, q_sh;
  const void* k; long long k_sb, k_ss, k_sh;
  const void* v; long long v_sb, v_ss, v_sh;
  void* out; long long o_sb, o_ss, o_sh;
  const float* sink;
  int B, H, G, Sq, dk, dv, window, k_rows;
  float scale;
  long long q_pos0;
  int* status;
  void* stream;
};

extern "C" int ra_attn_window(const RaAttnWindowArgs* a) {
  using namespace ra;
  using namespace ra::attn;
  const long long odd = (a->q_sb | a->q_ss | a->q_sh | a->k_sb | a->k_ss | a->k_sh | a->v_sb | a->v_ss | a->v_sh | a->o_sb |
                         a->o_ss | a->o_sh) & 7;
  if (a->B < 1 || a->G < 1 || a->H < 1 || a->H % a->G || a->Sq < 1 || a->q_pos0 < 0 || a->window < 1 || a->dk < 8 ||
      a->dk > 128 || a->dk % 8 || a->dv < 8 || a->dv > 128 || a->dv % 8 || a->k_rows < 128 || a->k_rows % 128 || odd ||
      ((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) | reinterpret_cast<uintptr_t>(a->v) |
        reinterpret_cast<uintptr_t>(a->out)) & 15)) {
    set_error("ra_attn_window: bad shape or alignment");
    return kHostBadArg;
  }
  // the first tile with a visible key; everything below counts keys from there
  const long long lo = a->q_pos0 - a->window + 1, base = lo > 0 ? lo / 128 * 128 : 0;
  const long long n_keys = a->q_pos0 + a->Sq - base;
  if (n_keys > a->k_rows || n_keys > (1 << 30)) {
    set_error("ra_attn_window: the ring does not hold the window of this step");
    return kHostBadArg;
  }
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_bshd_map(&tq, a->q, a->B, a->Sq, a->H, a->dk, a->q_sb, a->q_ss, a->q_sh))) return rc;
  if ((rc = make_bshd_map(&tk, a->k, a->B, a->k_rows, a->G, a->dk, a->k_sb, a->k_ss, a->k_sh))) return rc;
  if ((rc = make_bshd_map(&tv, a->v, a->B, a->k_rows, a->G, a->dv, a->v_sb, a->v_ss, a->v_sh))) return rc;
  FwdParams p = {};
  p.B = a->B;
  p.H = a->H;
  p.mask.Sq = a->Sq;
  p.mask.Sk = static_cast<int>(n_keys);
  p.mask.cbs = 1;
  p.mask.qmap = PosMap{static_cast<int>(a->q_pos0 - base), 0, 1 << 30};
  p.mask.kmap = PosMap{0, 0, 1 << 30};
  p.scale_log2 = a->scale * kLog2e;
  p.out = a->out;
  p.o_stride_b = a->o_sb;
  p.o_stride_s = a->o_ss;
  p.o_stride_h = a->o_sh;
  p.status = a->status;
  p.dv = a->dv;
  p.sink = a->sink;
  p.window = a->window;
  p.kv_share = a->H / a->G;
  p.k_row0 = static_cast<int>(base % a->k_rows);
  p.k_rows = a->k_rows;
  const int n_qp = (a->Sq + 255) / 256;
  p.order = TileOrder{n_qp, a->B * a->H, a->B * a->H};
  const long long grid = static_cast<long long>(n_qp) * a->H * a->B;
  cudaStream_t s = static_cast<cudaStream_t>(a->stream);
  if (a->dk > 64)
    return a->dv > 64 ? launch_fwd<2, 0, 128, true>(tq, tk, tv, tq, tk, p, grid, s)
                      : launch_fwd<2, 0, 64, true>(tq, tk, tv, tq, tk, p, grid, s);
  return a->dv > 64 ? launch_fwd<1, 0, 128, true>(tq, tk, tv, tq, tk, p, grid, s)
                    : launch_fwd<1, 0, 64, true>(tq, tk, tv, tq, tk, p, grid, s);
}
