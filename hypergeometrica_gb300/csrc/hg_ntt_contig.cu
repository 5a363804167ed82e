// hg_ntt_contig.cu -- the contiguous NTT pass and the middle of a product.
//
// The last T <= 12 forward stages of the reference's transform (ntt-forward,
// src/number-theoretic-transform.lisp:40-90) and the first T inverse stages
// (ntt-reverse, :93-143) act on contiguous blocks of 2^T residues.  One CTA
// owns one block.  Modes:
//   kFwd  the forward stages only (spectrum hook; bit-reversed output),
//   kInv  the inverse stages only (spectrum hook),
//   kMul  both operands' forward stages, the pointwise product
//         (multiply-pointwise!, src/ntt-multiply.lisp:88-99) and the
//         inverse stages: the block is read once per operand, written once,
//   kSqr  the same for one operand squared (src/ntt-multiply.lisp:136-144),
//   kMulSpec  operand 0's forward stages, the pointwise product with a
//         finished spectrum that every product of the launch shares, and the
//         inverse stages (the chunks of an unbalanced product).
// For transforms of at most 2^12 points this is the whole product's NTT work,
// and the kernel reads the limbs and reduces them itself.
//
// The block runs in rounds of up to four stages on 16 registers per thread,
// with one trip through shared memory between rounds; the stages of the low
// row group use compile-time twiddles, and multiplications by 1 are skipped.
// Transforms below 16 points run in ntt_tiny_kernel, one thread per prime.
#include "hg_ntt_bodies.cuh"

namespace hg {
namespace {

using namespace rounds;
using namespace bodies;

template <int T, int MODE>
__global__ void __launch_bounds__(kTileThreads, kContigMinBlocks) ntt_contig_kernel(const PassArgs P) {
  extern __shared__ uint64_t smem[];
  const uint64_t bx = blockIdx.x;
  const int by = static_cast<int>(blockIdx.y);
  pdl_wait();
#include "hg_contig_body.inc"
}

// The same pass for launches that leave the GPU mostly idle (fewer CTAs of
// 4096 residues than SMs): one block of 2^T residues per CTA, so that the
// blocks spread over the SMs, and in a product the two operands' forward
// transforms side by side, each by its own half of the CTA, instead of one
// after the other.  The half of operand 1 then leaves its spectrum in shared
// memory and stops; the other half multiplies and transforms back.  Such a
// launch is bound by the chain of stages: with it a product of 2^13 points
// takes 35.9 us instead of 42.1, one of 2^16 points 47.2 instead of 51.3.
template <int T, int MODE>
__global__ void __launch_bounds__(MODE == kMul ? 2 << (T - 4) : 1 << (T - 4)) ntt_contig_small_kernel(const PassArgs P) {
  static_assert(T >= 9 && T <= kTileBits, "half a block is at least one warp");
  extern __shared__ uint64_t smem[];
  using Gr = Groups<T>;
  constexpr int ATOP = Gr::template A<Gr::G - 1>(), A0 = Gr::template A<0>();
  constexpr int LT = T - 4, NT = 1 << LT;
  constexpr bool TWO = MODE == kMul;
  const uint32_t lt = threadIdx.x & (NT - 1);
  const int op = TWO ? threadIdx.x >> LT : 0;
  const int prime = P.prime_lo + static_cast<int>(blockIdx.y);
  const uint64_t prod = blockIdx.x / P.tiles, tile = blockIdx.x % P.tiles;
  const uint64_t p = P.pc[prime].p;
  const uint32_t c = P.pc[prime].c;
  const NttTables tb = P.tb[prime];
  const uint64_t poff = prod * P.ws_stride + static_cast<uint64_t>(prime - P.prime_lo) * P.prime_stride;
  const uint64_t base = tile << T;
  uint64_t *sm = smem + (op << T);
  pdl_wait();
  uint64_t nl = 0;
  const uint64_t *limbs = MODE == kInv ? nullptr : pass_limbs(P, prod, op, nl);
  uint64_t v[16];
  uint32_t xt;
  if constexpr (MODE == kInv) {
    xt = thread_base<A0>(lt);
    load_block<A0>(v, P.data[0] + poff, nullptr, 0, base, xt, p, 2 * p);
    inverse_rounds<T>(v, through(sm), swz_table(tb, T, true), xt, lt, p, c);
    if (P.scale) scale16(v, P.scale, p, c);
    store_block<ATOP>(v, P.data[0] + poff, base, xt, 2 * p);
    return;
  } else {
    xt = thread_base<ATOP>(lt);
    load_block<ATOP>(v, (op ? P.data[1] : P.data[0]) + poff, limbs, nl, base, xt, p);
    forward_rounds<T, MODE != kFwd>(v, through(sm), swz_table(tb, T, false), xt, lt, p, c);
    if constexpr (MODE == kFwd) {
      store_block<A0>(v, P.data[0] + poff, base, xt, p);
      return;
    }
    if constexpr (TWO) {
      // The thread's words of the last exchange, read by no other thread.
      if (op) to_smem<A0, true>(sm, v, xt);
      __syncthreads();
      if (op) return;
      const SmemAt<true> sb(smem + (1u << T), xt);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = mont_mul_2p(v[i], sb[static_cast<uint32_t>(i) << A0], p, c);
    } else if constexpr (MODE == kSqr) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = mont_mul_2p(v[i], v[i], p, c);
    } else {
      const uint64_t *spec = P.data[1] + static_cast<uint64_t>(prime - P.prime_lo) * P.prime_stride + base;
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = mont_mul(v[i], spec[xt | (static_cast<uint32_t>(i) << A0)], p, c);
    }
    inverse_rounds<T, true, TWO ? NT : 0>(v, through(sm), swz_table(tb, T, true), xt, lt, p, c);
    store_block<ATOP>(v, P.data[0] + poff, base, xt, 2 * p);
  }
}

__global__ void ntt_tiny_kernel(const PassArgs P, int mode) {
  pdl_wait();
  tiny_body(P, mode, blockIdx.x, static_cast<int>(blockIdx.y));
}

// Two CTAs of 4096 residues per SM: up to there the small kernel's spread is
// faster or level (a 2^18-point square: 57.5 us without it, 53.7 with).
constexpr uint64_t kSmallTiles = 304;

template <int T, int MODE>
cudaError_t launch_tm(const PassArgs &a, uint64_t nblk, cudaStream_t st) {
  constexpr uint64_t bpc = uint64_t(1) << (kTileBits - T);
  constexpr size_t bytes = static_cast<size_t>(MODE == kMul ? 2 : 1) * (1u << kTileBits) * sizeof(uint64_t);
  const uint64_t gx = (nblk + bpc - 1) / bpc;
  if (gx == 0 || gx > 0x7fffffffull) return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(a.nprimes));
  // Raise the dynamic shared-memory limit once per instantiation (not on
  // every launch, so that launches can be captured in a CUDA graph).
  static bool raised = false;
  if (bytes > 48 * 1024 && !raised) {
    cudaError_t e = cudaFuncSetAttribute(ntt_contig_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    raised = true;
  }
  return launch_dep(ntt_contig_kernel<T, MODE>, grid, kTileThreads, bytes, st, a);
}

template <int T, int MODE>
cudaError_t launch_small(const PassArgs &a, uint64_t nblk, cudaStream_t st) {
  constexpr size_t bytes = static_cast<size_t>(MODE == kMul ? 2 : 1) * (1u << T) * sizeof(uint64_t);
  static bool raised = false;  // as in launch_tm
  if (bytes > 48 * 1024 && !raised) {
    cudaError_t e = cudaFuncSetAttribute(ntt_contig_small_kernel<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    raised = true;
  }
  return launch_dep(ntt_contig_small_kernel<T, MODE>,
                    dim3(static_cast<unsigned>(nblk), static_cast<unsigned>(a.nprimes)),
                    (MODE == kMul ? 2 : 1) << (T - 4), bytes, st, a);
}

template <int MODE>
cudaError_t launch_mode(const PassArgs &a, uint64_t nblk, cudaStream_t st) {
  if (a.logT >= 9 && ((nblk << a.logT) >> kTileBits) * a.nprimes <= kSmallTiles) {
    switch (a.logT) {
      case 9: return launch_small<9, MODE>(a, nblk, st);
      case 10: return launch_small<10, MODE>(a, nblk, st);
      case 11: return launch_small<11, MODE>(a, nblk, st);
      default: return launch_small<12, MODE>(a, nblk, st);
    }
  }
  switch (a.logT) {
    case 4: return launch_tm<4, MODE>(a, nblk, st);
    case 5: return launch_tm<5, MODE>(a, nblk, st);
    case 6: return launch_tm<6, MODE>(a, nblk, st);
    case 7: return launch_tm<7, MODE>(a, nblk, st);
    case 8: return launch_tm<8, MODE>(a, nblk, st);
    case 9: return launch_tm<9, MODE>(a, nblk, st);
    case 10: return launch_tm<10, MODE>(a, nblk, st);
    case 11: return launch_tm<11, MODE>(a, nblk, st);
    case 12: return launch_tm<12, MODE>(a, nblk, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

#if HG_CHECKED
HG_CHECKED_READER(checked_fault_contig)
#endif

cudaError_t launch_ntt_contig(const PassArgs &a, int mode, cudaStream_t st) {
  const uint64_t nblk = a.tiles * a.nprod;  // blocks per prime
  if (nblk == 0 || a.logS != 0 || a.logR != a.logT || a.nprimes < 1 || a.nprimes > kPrimes)
    return cudaErrorInvalidValue;
  if (a.logT < 4) {
    if (mode == kMulSpec || a.logT < 1 || a.logT != a.logN || a.tiles != 1 || a.nprod > 0x7fffffffull) return cudaErrorInvalidValue;
    return launch_dep(ntt_tiny_kernel, dim3(static_cast<unsigned>(a.nprod), static_cast<unsigned>(a.nprimes)), 1, 0,
                      st, a, mode);
  }
  switch (mode) {
    case kFwd: return launch_mode<kFwd>(a, nblk, st);
    case kInv: return launch_mode<kInv>(a, nblk, st);
    case kMul: return launch_mode<kMul>(a, nblk, st);
    case kSqr: return launch_mode<kSqr>(a, nblk, st);
    case kMulSpec: return launch_mode<kMulSpec>(a, nblk, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hg
