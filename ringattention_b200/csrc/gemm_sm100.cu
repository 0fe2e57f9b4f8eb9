// Persistent warp-specialised bf16 GEMM for sm_100a: C[M,N] = A[M,K] * B[N,K]^T (+ C).
//
//   warp 0      TMA producer: 128x64 A tile + BNx64 B tile per stage, mbarrier ring of 192 KiB
//   warp 1      tcgen05.mma issuer (one thread), two 128xBN fp32 accumulators in TMEM
//   warps 2..5  epilogue: tcgen05.ld -> bf16/fp32 -> global, overlapped with the next tile's MMAs
//
// or the same on pairs of CTAs with tiles of 256 rows (gemm_pair.cuh); choose_form() says which.
//
// Each operand is either K-major (contiguous along the reduction dim) or MN-major (contiguous
// along M resp. N); both are loaded with 128-byte-swizzled TMA boxes and described to the tensor
// core by shared-memory descriptors, so the forward (x W^T), dgrad (dy W) and wgrad (dy^T x)
// products of a linear layer all run through this one kernel without any transposes in memory.
#include "gemm_kernel.cuh"
#include "gemm_pair.cuh"

RA_BOUNDS_TRANSLATION_UNIT()

namespace ra {
namespace gemm {

// The form of a product of M rows, n columns (of the accumulator) and num_kb k-blocks: tiles of 128 rows on one CTA or of 256 on a pair, 64, 128
// or 256 columns wide; the one with the shortest estimated time. Wide tiles and pairs move the fewest bytes per column, which decides once
// every SM has several of them; below that a launch takes as long as one SM's tiles, and narrower ones spread over more SMs and have a
// shorter epilogue; a pair costs a launch about 1 us and works for nothing on the second half of its rows where M ends in the first.
// Nanoseconds per k-block, per 32 columns of epilogue (plain, with an addend, SwiGLU) and per tile and launch were fitted together to 295 products
// with 128 to 8192 rows timed on B200 in every form, K-major and MN-major; a single one of them need not be the cost of what it is named for
// (an epilogue that hides behind the products of the next tile leaves the fit little to go by), and shapes far outside have to be timed, not
// worked out. 687 products with 9 to 8192 rows, weights out of memory: the choice takes 0.6 % longer than the fastest of the five on average,
// 16 % at worst (32 of them more than 5 %). With 128 rows or fewer, where a pair's second CTA has no row,
// the 36 products that get pairs all the same take 6 % less on average than the best one-CTA form (-3 to 22 %).
// us, one CTA 256 / 128 / 64 columns, pair 256 / 128, * the choice:
//   8192 x 8192 x 8192 775 / 952 / 1638, 729* / 893         4096 x 4096 x 4096, bf16 addend 125 / 143 / 252, 99* / 113
//   22016 x 4096 x 4096, fp32 sums 550 / 679 / 1190, 510* / 618     2048 x 4096 x 4096 51 / 80 / 126, 48* / 60
//   512 x 4096 x 11008 72 / 49 / 83, 59 / 44*               300 x 11008 x 2048 15.9* / 21.3 / 34.7, 25.4 / 25.7
//   9 x 4096 x 4096 28.5 / 20.2 / 24.1, 24.4 / 18.8*
//   512 x 1536 x 512 7.9 / 6.3 / 5.9*, 8.8 / 7.4            1024 x 2816 x 1024, fp32 sums 15.5 / 15.7 / 16.9, 13.7* / 14.5
struct Form {
  int pair, width;
  int kb, epi[3], tile, fixed;
};
constexpr Form kForms[] = {
    {0, 256, 318, {224, 658, 882}, 3567, 0},
    {0, 128, 264, {374, 559, 423}, 1419, 1719},
    {0, 64, 242, {918, 824, 1}, 733, 1458},
    {1, 256, 306, {396, 429, 236}, 2366, 966},
    {1, 128, 201, {555, 469, 26}, 1716, 2215},
};
inline const Form& choose_form(int M, int n, int num_kb, bool addend, bool swiglu) {
  const Form* best = nullptr;
  long long best_ns = 0;
  for (const Form& f : kForms) {
    const int rows = f.pair ? 2 * BM : BM, units = f.pair ? sm_count() / 2 : sm_count();
    const long long tiles = static_cast<long long>((M + rows - 1) / rows) * ((n + f.width - 1) / f.width);
    const long long waves = (tiles + units - 1) / units;
    const long long main = static_cast<long long>(num_kb) * f.kb, epi = f.width / 32 * f.epi[swiglu ? 2 : (addend ? 1 : 0)];
    const long long ns = f.fixed + waves * ((main > epi ? main : epi) + f.tile) + epi;
    if (!best || ns < best_ns) {
      best = &f;
      best_ns = ns;
    }
  }
  return *best;
}

// The operands' bases and leading dimensions in elements; launch_bn makes their tensor maps, whose boxes depend on the tile's width.
struct Operands {
  const void *a, *b;
  long long lda, ldb;
};

template <int A_MN, int B_MN, int BN_>
int launch_bn(const Operands& o, const Params& p, cudaStream_t stream) {
  CUtensorMap ta;
  TmaSet set;
  int rc;
  uint64_t dims[2], str[1];
  uint32_t box[2];
  if (A_MN) { dims[0] = p.M; dims[1] = p.K; box[0] = 64; box[1] = BK; }
  else      { dims[0] = p.K; dims[1] = p.M; box[0] = BK; box[1] = BM; }
  str[0] = static_cast<uint64_t>(o.lda) * 2;
  if ((rc = make_tmap_bf16_sw128(&ta, o.a, 2, dims, str, box)) != 0) return rc;
  if (B_MN) { dims[0] = p.N; dims[1] = p.K; box[0] = 64; box[1] = BK; }
  else      { dims[0] = p.K; dims[1] = p.N; box[0] = BK; box[1] = p.swiglu_F ? BN_ / 2 : BN_; }
  str[0] = static_cast<uint64_t>(o.ldb) * 2;
  if ((rc = make_tmap_bf16_sw128(&set.m[p.swiglu_F ? 1 : 0], o.b, 2, dims, str, box)) != 0) return rc;
  if (p.swiglu_F) set.m[0] = set.m[1];
  auto kern = gemm_bf16_kernel<A_MN, B_MN, false, BN_>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<BN_>::SMEM_BYTES) != cudaSuccess) {
    set_error("gemm: cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed");
    return kHostLaunchFail;
  }
  const int tiles_n = p.swiglu_F ? (p.swiglu_F + BN_ / 2 - 1) / (BN_ / 2) : (p.N + BN_ - 1) / BN_;
  const int tiles = ((p.M + BM - 1) / BM) * tiles_n;
  const int grid = tiles < sm_count() ? tiles : sm_count();
  GatherParams g = {};
  kern<<<grid, THREADS, Tile<BN_>::SMEM_BYTES, stream>>>(ta, set, p, g);
  return check_launch("gemm_bf16_kernel");
}

template <int A_MN, int B_MN, int BN_>
int launch_pair(const Operands& o, const Params& p, cudaStream_t stream) {
  using T = PairTile<BN_>;
  CUtensorMap ta, tb;
  int rc;
  uint64_t dims[2], str[1];
  uint32_t box[2];
  if (A_MN) { dims[0] = p.M; dims[1] = p.K; box[0] = 64; box[1] = BK; }
  else      { dims[0] = p.K; dims[1] = p.M; box[0] = BK; box[1] = BM; }
  str[0] = static_cast<uint64_t>(o.lda) * 2;
  if ((rc = make_tmap_bf16_sw128(&ta, o.a, 2, dims, str, box)) != 0) return rc;
  if (B_MN) { dims[0] = p.N; dims[1] = p.K; box[0] = 64; box[1] = BK; }
  else      { dims[0] = p.K; dims[1] = p.N; box[0] = BK; box[1] = BN_ / 2; }
  str[0] = static_cast<uint64_t>(o.ldb) * 2;
  if ((rc = make_tmap_bf16_sw128(&tb, o.b, 2, dims, str, box)) != 0) return rc;
  auto kern = gemm_pair_kernel<A_MN, B_MN, BN_>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM_BYTES) != cudaSuccess) {
    set_error("gemm: cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed");
    return kHostLaunchFail;
  }
  const int tiles_n = p.swiglu_F ? (p.swiglu_F + BN_ / 2 - 1) / (BN_ / 2) : (p.N + BN_ - 1) / BN_;
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * tiles_n, pairs = sm_count() / 2;
  kern<<<2 * (tiles < pairs ? tiles : pairs), PAIR_THREADS, T::SMEM_BYTES, stream>>>(ta, tb, p);
  return check_launch("gemm_pair_kernel");
}

template <int A_MN, int B_MN>
int launch(const Operands& o, const Params& p, cudaStream_t stream) {
  const Form& f = choose_form(p.M, p.N, (p.K + BK - 1) / BK, p.R != nullptr, p.swiglu_F != 0);
  if (f.pair)
    return f.width == 256 ? launch_pair<A_MN, B_MN, 256>(o, p, stream) : launch_pair<A_MN, B_MN, 128>(o, p, stream);
  if (f.width == 256) return launch_bn<A_MN, B_MN, 256>(o, p, stream);
  if (f.width == 128) return launch_bn<A_MN, B_MN, 128>(o, p, stream);
  return launch_bn<A_MN, B_MN, 64>(o, p, stream);
}

}  // namespace gemm
}  // namespace ra


// C[M,N] (ldc) = A * B^T (+ R). a_mn = 0: A is [M][lda] (K contiguous); 1: A is [K][lda] (M
// contiguous). b_mn = 0: B is [N][ldb]; 1: B is [K][ldb]. All leading dimensions in elements and
// multiples of 8; base pointers 16-byte aligned. c_fp32 selects the type of C and R (1: fp32, 0: bf16, 2: C bf16 and R fp32). R is
// an optional addend (residual or running gradient) and may alias C for in-place accumulation where their types agree.
extern "C" int ra_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N,
                            int K, long long lda, long long ldb, long long ldc, long long ldr,
                            int a_mn, int b_mn, int c_fp32, int group_m, int* status,
                            void* stream) {
  using namespace ra;
  if (M <= 0 || N <= 0 || K <= 0 || (lda % 8) || (ldb % 8) || (ldc % (c_fp32 == 1 ? 4 : 8)) ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15) || (reinterpret_cast<uintptr_t>(R) & 15) ||
      (R && (ldr % (c_fp32 ? 4 : 8)))) {
    set_error("ra_gemm_bf16: bad shape/alignment");
    return kHostBadArg;
  }
  const gemm::Operands o{A, B, lda, ldb};
  gemm::Params p{C, ldc, M, N, K, c_fp32 == 1, R, ldr, group_m > 0 ? group_m : 8, status, 0};
  p.r_fp32 = c_fp32 == 2;
  p.n_split = N;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!a_mn && !b_mn) return gemm::launch<0, 0>(o, p, s);
  if (!a_mn && b_mn) return gemm::launch<0, 1>(o, p, s);
  if (a_mn && !b_mn) return gemm::launch<1, 0>(o, p, s);
  return gemm::launch<1, 1>(o, p, s);
}


// H[M,F] (ldh) = silu(A Wg^T) * (A Wu^T) for W = [Wg ; Wu] stored as [2F][ldb] (K contiguous): the gate/up
// projection of a SwiGLU feed-forward with the activation in the GEMM epilogue, so the (M, 2F) pre-activations
// are never written. A is [M][lda], K contiguous. F must be a multiple of 8.
extern "C" int ra_gemm_bf16_swiglu(const void* A, const void* W, void* Hout, int M, int F, int K, long long lda,
                                   long long ldb, long long ldh, int group_m, int* status, void* stream) {
  using namespace ra;
  if (M <= 0 || F <= 0 || K <= 0 || (F % 8) || (lda % 8) || (ldb % 8) || (ldh % 8) ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(W) & 15) ||
      (reinterpret_cast<uintptr_t>(Hout) & 15)) {
    set_error("ra_gemm_bf16_swiglu: bad shape/alignment");
    return kHostBadArg;
  }
  gemm::Params p{Hout, ldh, M, 2 * F, K, 0, nullptr, 0, group_m > 0 ? group_m : 8, status, F};
  p.n_split = 2 * F;
  return gemm::launch<0, 0>(gemm::Operands{A, W, lda, ldb}, p, static_cast<cudaStream_t>(stream));
}


// C[M,N] = act(alpha A B^T + bias (+ R)) with the epilogues of an inference layer: `bias` is fp32 by column, padded to a
// multiple of 32 entries (null: none, and alpha is not looked at); `relu2` squares the positive part (no addend then), `C2` takes the columns [n_split, N) in fp32 (n_split a multiple of 32, N - n_split a multiple of 4). Both operands
// K-major; N a multiple of 8 (of 4 with an fp32 C); otherwise the rules of ra_gemm_bf16.
extern "C" int ra_gemm_bf16_ex(const void* A, const void* B, void* C, const void* R, float* C2, int M, int N, int K,
                               long long lda, long long ldb, long long ldc, long long ldr, long long ldc2, int n_split,
                               int relu2, int c_fp32, const float* bias, float alpha, int group_m, int* status,
                               void* stream) {
  using namespace ra;
  if (M <= 0 || N <= 0 || K <= 0 || (N % (c_fp32 ? 4 : 8)) || (lda % 8) || (ldb % 8) || (ldc % (c_fp32 ? 4 : 8)) ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15) || (reinterpret_cast<uintptr_t>(R) & 15) ||
      (reinterpret_cast<uintptr_t>(C2) & 15) || (reinterpret_cast<uintptr_t>(bias) & 15) || (R && (ldr % (c_fp32 ? 4 : 8))) || (R && relu2) ||
      (C2 && (n_split % 32 || n_split < 0 || n_split >= N || ldc2 % 4 || ldc2 < N - n_split))) {
    set_error("ra_gemm_bf16_ex: bad shape/alignment");
    return kHostBadArg;
  }
  gemm::Params p{C, ldc, M, N, K, c_fp32, R, ldr, group_m > 0 ? group_m : 8, status, 0, relu2, C2, ldc2, C2 ? n_split : N,
                 bias, alpha};
  return gemm::launch<0, 0>(gemm::Operands{A, B, lda, ldb}, p, static_cast<cudaStream_t>(stream));
}

// The form that a product gets (`addend`: there is one; with SwiGLU N counts gate and up): its tiles' columns, negative on pairs of CTAs.
extern "C" int ra_gemm_form(int M, int N, int K, int addend, int swiglu) {
  const ra::gemm::Form& f = ra::gemm::choose_form(M, N, (K + ra::gemm::BK - 1) / ra::gemm::BK, addend != 0, swiglu != 0);
  return f.pair ? -f.width : f.width;
}

RA_PACKED(ra_gemm_bf16)
RA_PACKED(ra_gemm_bf16_swiglu)
RA_PACKED(ra_gemm_bf16_ex)
