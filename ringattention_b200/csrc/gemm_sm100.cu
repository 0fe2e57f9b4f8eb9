// Persistent warp-specialised bf16 GEMM for sm_100a: C[M,N] = A[M,K] * B[N,K]^T (+ C).
//
//   warp 0      TMA producer: 128x64 A tile + BNx64 B tile per stage, mbarrier ring of 192 KiB
//   warp 1      tcgen05.mma issuer (one thread), two 128xBN fp32 accumulators in TMEM
//   warps 2..5  epilogue: tcgen05.ld -> bf16/fp32 -> global, overlapped with the next tile's MMAs
//
// Each operand is either K-major (contiguous along the reduction dim) or MN-major (contiguous
// along M resp. N); both are loaded with 128-byte-swizzled TMA boxes and described to the tensor
// core by shared-memory descriptors, so the forward (x W^T), dgrad (dy W) and wgrad (dy^T x)
// products of a linear layer all run through this one kernel without any transposes in memory.
#include "gemm_kernel.cuh"

RA_BOUNDS_TRANSLATION_UNIT()

namespace ra {
namespace gemm {

// Width of the tiles for a product of tiles_m row tiles, n columns (of the accumulator) and num_kb k-blocks: the one with the
// shortest estimated time. Wide tiles move the fewest bytes per column, which decides once every SM has several of them;
// below that a launch takes as long as one SM's tiles, and narrower ones spread over more SMs and have a shorter epilogue.
// Clocks per k-block, per 32 columns of epilogue (more with an fp32 addend) and per tile were fitted to 130 products with 128
// to 4096 rows timed on B200 at each width; the choice is within 5 % of the best of the three for all of them, 0.2 % on average.
// With 256 columns throughout, 512 x 1024 x 1024 took 10.8 us (64: 7.7), 1024 x 1024 from 4096 rows with fp32
// accumulation 36 (64: 21), 2048 x 1024 x 2816 21.6 (128: 16.6); 8192 x 4096 x 4096 takes 194 (128: 244).
inline int choose_bn(int tiles_m, int n, int num_kb, bool addend32) {
  const int width[3] = {256, 128, 64}, kb_clk[3] = {790, 487, 312};
  const int epi_clk = addend32 ? 815 : 690;
  constexpr int tile_clk = 380;
  int best = 0;
  long long best_clk = 0;
  for (int i = 0; i < 3; ++i) {
    const long long tiles = static_cast<long long>(tiles_m) * ((n + width[i] - 1) / width[i]);
    const long long waves = (tiles + sm_count() - 1) / sm_count();
    const long long main = static_cast<long long>(num_kb) * kb_clk[i], epi = width[i] / 32 * epi_clk;
    const long long clk = waves * ((main > epi ? main : epi) + tile_clk) + epi;
    if (i == 0 || clk < best_clk) {
      best = width[i];
      best_clk = clk;
    }
  }
  return best;
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

template <int A_MN, int B_MN>
int launch(const Operands& o, const Params& p, cudaStream_t stream) {
  const int bn = choose_bn((p.M + BM - 1) / BM, p.N, (p.K + BK - 1) / BK, (p.c_fp32 || p.r_fp32) && p.R);
  if (bn == 256) return launch_bn<A_MN, B_MN, 256>(o, p, stream);
  if (bn == 128) return launch_bn<A_MN, B_MN, 128>(o, p, stream);
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
  gemm::Params p{C, ldc, M, N, K, c_fp32, R, ldr, group_m > 0 ? group_m : 8, status, 0, relu2, C2, ldc2, n_split,
                 bias, alpha};
  return gemm::launch<0, 0>(gemm::Operands{A, B, lda, ldb}, p, static_cast<cudaStream_t>(stream));
}
