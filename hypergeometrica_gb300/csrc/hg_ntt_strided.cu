// hg_ntt_strided.cu -- strided NTT passes.
//
// The reference's forward transform is a sequence of radix-2 DIF stages
// (ntt-forward, src/number-theoretic-transform.lisp:40-90); the inverse, DIT
// stages (ntt-reverse, :93-143).  A strided pass performs the stages
// subn = M .. 2S (M = R*S, R = 2^LOGR rows, 4 <= LOGR <= 8) on every block of
// M residues.  Those stages equal an R-point transform down each of the S
// columns, bit-reversed output, with row r of column s then multiplied by
// w_M^(s * bitrev(r)); the inverse pass mirrors it.  Every residue stays
// canonical, so the pass leaves in memory exactly what the reference's
// stages leave.
//
// A CTA of 256 threads owns a tile of 4096 residues: R rows x 4096/R
// consecutive columns (>= 16 columns, so every row segment is >= 128 bytes).
// Each thread loads 16 residues straight into registers (coalesced: lanes
// run along columns), runs the stages of the top row bits, exchanges the tile
// once through shared memory, runs the stages of the low four row bits, and
// applies the inter-pass twiddle to its 16 rows of one column as a geometric
// sequence beta * gamma^k before storing from registers.
//
// Passes over residues (every pass but the first forward one, which reads and
// reduces the limbs) stage the tile through shared memory with TMA instead:
// one bulk tensor copy brings the tile's R rows of C residues in (and the
// same box of the pass's inter-pass twiddle table beside it), threads read
// their 16 residues with constant shared-memory offsets, and after the
// stages one bulk copy writes the tile back.  No thread computes a global
// address or issues a global load or store for the residues.
//
// Truncated transforms: a product of n coefficients needs n points, not the
// power of two above.  The outer pass (M = N) may keep only its first krows
// rows of outputs (krows S >= n): the passes inside then run on krows of the
// R blocks, and the outer inverse pass solves each column's krows values
// from krows outputs and the R - krows results known to be zero
// (TruncatedInverse).  krows is 9 to 15 sixteenths of R, cut by the top four
// row bits (the top three for R = 128, the top two for R = 64), which sit in
// one thread's registers in the round that ends the pass.
//
// A product's coefficients are limbs or, where that needs fewer points, digits
// of 80 bits (5 limbs hold 4 digits): the first forward pass then forms the
// digits from its limbs.
#include <algorithm>
#include <cudaTypedefs.h>
#include <mutex>

#include "hg_ntt_bodies.cuh"
#include "hg_tma.cuh"

namespace hg {
namespace {

using namespace rounds;
using namespace bodies;

// Four CTAs of 256 threads per SM (64 registers, a few spilled words): on
// the 2^25-point passes faster than three (80 registers), two (128) or five
// (48).
template <int LOGR, bool INV, bool CUT = false, bool D80 = false>
__global__ void __launch_bounds__(kTileThreads, 4) ntt_strided_kernel(const PassArgs P) {
  __shared__ ulonglong2 tw[1 << (LOGR - 1)];
  __shared__ uint64_t sm[LOGR > 4 ? (1 << kTileBits) : 1];
  pdl_wait();
  strided_ldg_body<LOGR, INV, CUT, D80, true>(P, blockIdx.x, tw, sm);
}

constexpr int kCut = 0;  // KQ of a truncated transform's outer forward pass

// Tensor maps of one TMA-staged pass: the box each CTA loads (residues, or
// the limbs of a first forward pass) and stores, per operand, and the box of
// the inter-pass twiddle table.
struct TmaMaps {
  CUtensorMap in[2];
  CUtensorMap out[2];
  CUtensorMap tw;
};

// A first forward pass's limbs per load map: the complete rows of S limbs it
// covers, the limbs of the partial row after them, and (bit k of ztop) whether
// every limb of map k lies in the lower half of the block.  Map op is operand
// op's; a long operand cut into chunks has its last chunk in map 1 and the
// others, one after another in its third dimension, in map 0.
struct TmaLimbs {
  const uint64_t *limbs[2];
  uint64_t full_rows[2];
  uint64_t tail[2];
  uint32_t ztop;
};

// A strided pass with the tile staged by TMA.  Shared memory: the tile
// [R][C] (row-major, exactly the tile position x = r C + c), then, with
// TABLE, the same box of the inter-pass twiddle table.  Three CTAs of 256
// threads per SM (66 KB of shared memory each) with the table, four
// without; 64 registers (the table variants do not spill; measured 0.3%
// faster than with 80).
//
// LIMBS (forward only): the pass reads the operand's limbs, viewed as rows
// of S limbs (a map over the rows that are complete, and over the chunks of a
// long operand; the copy fills the rows past them with zeros) and patches the partial row past the last
// complete one with plain loads before reducing every limb modulo p.  When
// the upper half of the block lies past the limbs (P.ztop bit op), the first
// stage skips its zero inputs.
//
// D80 (with LIMBS): the coefficients are 80-bit digits.  The limbs' rows have
// 5 S / 4 limbs and the tile's box 5 C / 4 of them (two boxes for R = 16, whose
// 320 limbs pass the 256 of a box); a digit lies in two words of its row.
//
// KQ < 16: the outer pass of a truncated transform.  Inverse: KQ/16 of the rows
// are known.  Forward (KQ = kCut, whatever the number): the kept rows are
// P.krows, and threads whose 16 rows are all dropped stop after the exchange
// (R > 16).  A whole transform's passes are instances of their own: taking the
// rows from P.krows there made the 2^25-point product 2% slower.
//
// SCALE (inverse only): the last pass of the spectrum entry point, which
// multiplies every residue by P.scale as it leaves (a launch and a pass over
// memory less: 2^20 points there and back 67.4 -> 61.0 us).
template <int LOGR, bool INV, bool TABLE, bool LIMBS, int KQ, bool SCALE, bool D80>
__global__ void __launch_bounds__(kTileThreads, 4)
    ntt_strided_tma_kernel(const __grid_constant__ TmaMaps maps, const PassArgs P, const TmaLimbs L) {
  constexpr int T = kTileBits;
  constexpr int LOGTC = T - LOGR;
  constexpr int ROWOFF = LOGTC;
  constexpr int A0 = ROWOFF;
  constexpr int A1 = T - 4;
  constexpr int G = (LOGR + 3) / 4;
  constexpr int NB1 = LOGR - 4;
  constexpr uint32_t kTileBytes = (1u << T) * sizeof(uint64_t);
  static_assert(LOGR >= 4 && LOGR <= 8, "strided passes have 4..8 row bits");
  static_assert(!LIMBS || !INV, "only a forward pass reads limbs");
  static_assert(KQ == 16 || (!INV && KQ == kCut && LIMBS) || (INV && truncation_ok(LOGR, KQ)),
                "rows a truncated inverse can cut");
  static_assert(!D80 || LIMBS, "digits are formed from limbs");
  constexpr int KI = INV ? KQ : 16;
  constexpr int kRows = (1 << LOGR) * KI / 16;  // inverse: known rows
  constexpr bool kCutFwd = !INV && KQ < 16;
  constexpr uint32_t kInWords = (D80 ? 5u : 4u) << (T - 2);  // words of the input box
  constexpr uint32_t kRowWords = D80 ? 5u << (LOGTC - 2) : 1u << LOGTC;  // words of an input row of the tile
  const int krows = kCutFwd ? P.krows : kRows;
  extern __shared__ __align__(128) uint64_t tile[];  // [1 << T] residues, then [1 << T] twiddles
  __shared__ ulonglong2 tw[1 << (LOGR - 1)];
  __shared__ ulonglong2 twf[INV && KQ < 16 ? 1 << (LOGR - 1) : 1];
  __shared__ __align__(8) uint64_t bar;

  const uint32_t tid = threadIdx.x;
  uint64_t bid = blockIdx.x;
  const int prime = P.prime_lo + static_cast<int>(bid % P.nprimes);
  bid /= P.nprimes;
  const int op = static_cast<int>(bid % P.nops);
  bid /= P.nops;
  const uint64_t prod = bid / P.tiles;
  const uint64_t t = P.tile_lo + bid % P.tiles;
  const uint64_t p = P.pc[prime].p;
  const uint32_t c = P.pc[prime].c;
  const NttTables tb = P.tb[prime];
  const int logS = P.logS;
  const uint64_t ncg = 1ull << (logS - LOGTC);
  const int blk = static_cast<int>(t / ncg);
  const int s0 = static_cast<int>((t % ncg) << LOGTC);
  uint64_t *twt = tile + kInWords;
  // The load map: an operand's, or the last chunk's.
  const int sel = LIMBS && P.chunk ? (prod == P.nprod - 1 ? 1 : 0) : op;

  if (tid == 0) {
    tma::mbar_init(&bar, 1);
    tma::fence_barrier_init();
  }
  __syncthreads();
  if (tid == 0) {
    const uint32_t row_bytes = kTileBytes >> LOGR;
    tma::mbar_arrive_expect_tx(&bar, (INV ? kRows * row_bytes : kInWords * 8u) +
                                         (TABLE ? static_cast<uint32_t>(krows) * row_bytes : 0u));
    if (TABLE) tma::load_3d(twt, &maps.tw, &bar, s0, 0, prime);  // no kernel of the stream writes the tables
    pdl_wait();
    const int z = sel == op ? static_cast<int>(prod) : 0;  // chunk
    if constexpr (D80 && LOGR == 4) {
      tma::load_3d(tile, &maps.in[sel], &bar, s0 / 4 * 5, blk << LOGR, z);
      tma::load_3d(tile + kInWords / 2, &maps.in[sel], &bar, s0 / 4 * 5 + static_cast<int>(kRowWords) / 2, blk << LOGR,
                   z);
    } else if constexpr (LIMBS)
      tma::load_3d(tile, &maps.in[sel], &bar, D80 ? s0 / 4 * 5 : s0, blk << LOGR, z);
    else
      tma::load_5d(tile, &maps.in[op], &bar, s0, 0, blk, prime - P.prime_lo, static_cast<int>(prod));
  }
  load_sub_twiddles(tw, INV ? tb.sub_inv : tb.sub_fwd, LOGR, tid, kTileThreads);
  if constexpr (INV && KQ < 16) load_sub_twiddles(twf, tb.sub_fwd, LOGR, tid, kTileThreads);
  if constexpr (LIMBS) pdl_wait();  // a partial row's limbs are read by every thread
  const bool landed = tma::mbar_wait_bounded(&bar, 0);
  if (!__syncthreads_and(landed)) {  // also orders the sub-twiddle table
    if (tid == 0) latch_error(P.err, kDevCopyTimeout);
    return;
  }

  // The inter-pass twiddles of the thread's 16 rows r = rhi * 16 + i of one
  // column (layout A0): from the table's box, or as a geometric sequence.
  auto inter_pass = [&](uint64_t (&v)[16], uint32_t xt, const uint64_t *hi, const uint64_t *lo) {
    if constexpr (TABLE) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (LOGR == 4 && KQ < 16 && i >= 9 && i >= krows) break;  // rows that are not kept
        v[i] = mont_mul(v[i], twt[xt | (static_cast<uint32_t>(i) << A0)], p, c);
      }
    } else {
      const uint64_t s = static_cast<uint64_t>(s0) + (xt & ((1u << LOGTC) - 1u));
      const uint32_t rhi = (xt >> (ROWOFF + 4)) & ((1u << (LOGR - 4)) - 1u);
      const int logM = LOGR + logS;
      uint32_t rrev = 0;
      if constexpr (LOGR > 4) rrev = bitrev(rhi, LOGR - 4);
      const uint64_t beta = table_twiddle(s * rrev, logM, hi, lo, p, c);
      const uint64_t gamma = table_twiddle(s << (LOGR - 4), logM, hi, lo, p, c);
      geometric_twiddle(v, beta, gamma, p, c);
    }
  };

  uint64_t v[16];
  uint32_t xt;
  if (!INV) {
    constexpr int AL = (G == 2) ? A1 : A0;
    xt = thread_base<AL>(tid);
    const bool ztop = LIMBS && ((L.ztop >> sel) & 1);
    if constexpr (LIMBS) {
      // Row tr (in the limbs' rows of S) is the partial one: limbs
      // [tr S, tr S + tail) exist past the complete rows the map covers.
      const uint64_t tr = sel ? L.full_rows[1] : L.full_rows[0];
      const uint64_t tail = sel ? L.tail[1] : L.tail[0];
      const uint64_t *lp = (op ? L.limbs[1] : L.limbs[0]) + prod * P.chunk;
      const uint64_t row0 = static_cast<uint64_t>(blk) << LOGR;
      const bool has_tail = tail != 0 && tr >= row0 && tr < row0 + (1u << LOGR);
      // Register i holds row (xt >> ROWOFF) + i 2^(AL - ROWOFF) of column col: one
      // pointer, constant offsets.
      const uint32_t row_t = xt >> ROWOFF, col = xt & ((1u << LOGTC) - 1u);
      // R = 16: columns 0 .. C/2 - 1 in the first box, the others in the second.
      const uint32_t half = D80 && LOGR == 4 ? col >> (LOGTC - 1) : 0u;
      const uint32_t lc = D80 && LOGR == 4 ? col & ((1u << (LOGTC - 1)) - 1u) : col;
      constexpr uint32_t kRow = D80 && LOGR == 4 ? kRowWords / 2 : kRowWords;
      const uint64_t *src = tile + half * (kInWords / 2) + row_t * kRow + (D80 ? 0u : col);
      const uint32_t *src32 = reinterpret_cast<const uint32_t *>(src) + ((5u * lc) >> 1);
      auto limb = [&](int i) {
        if constexpr (D80) {
          const uint32_t *w = src32 + static_cast<uint32_t>(i) * (2u * kRow << (AL - ROWOFF));
          return digit80_words(w[0], w[1], w[2], lc & 1u, P.pc[prime]);
        } else {
          return reduce64(src[static_cast<uint32_t>(i) * (kRow << (AL - ROWOFF))], p);
        }
      };
      // The partial row, where this thread holds it (whole warps do or do not),
      // after the others: a test in every register's load cost 1% of the 2^24
      // product and 3% of 2^24 x 2^16 (4545 -> 4504 us, 1669 -> 1619).
      auto patch = [&](int nreg) {
        const uint32_t d = static_cast<uint32_t>(tr - row0) - row_t;  // rows above the thread's first
        if (!has_tail || (d & ((1u << (AL - ROWOFF)) - 1u)) || (d >> (AL - ROWOFF)) >= static_cast<uint32_t>(nreg)) return;
        const uint64_t at = (tr << logS) + static_cast<uint64_t>(s0) + col;
        uint64_t w = 0;
        if constexpr (D80)
          w = coefficient<true>(lp, tr * (uint64_t(5) << (logS - 2)) + tail, at, P.pc[prime]);
        else if (s0 + col < tail)
          w = reduce64(lp[at], p);
#pragma unroll
        for (int i = 0; i < 16; ++i)
          v[i] = i < nreg && (d >> (AL - ROWOFF)) == static_cast<uint32_t>(i) ? w : v[i];
      };
      if (ztop) {
        // Registers 8..15 hold the top row bit's upper half, past the limbs:
        // zeros that the first stage (ZTOP) never reads, so neither read nor
        // reduced here.
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = limb(i);
        patch(8);
        if constexpr (G == 2) stages<NB1, 4 - NB1, A1, ROWOFF, 4, LOGR, false, false, false, true>(v, tw, xt, p, c);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = limb(i);
        patch(16);
        if constexpr (G == 2) stages<NB1, 4 - NB1, A1, ROWOFF, 4, LOGR, false, false>(v, tw, xt, p, c);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = tile[xt | (static_cast<uint32_t>(i) << AL)];
        check_below(v[i], p);  // forward input: canonical residues
      }
    }
    if constexpr (G == 2) {
      if constexpr (!LIMBS) stages<NB1, 4 - NB1, A1, ROWOFF, 4, LOGR, false, false>(v, tw, xt, p, c);
      __syncthreads();  // every thread has its values out of the tile
      to_smem<A1>(tile, v, xt);
      __syncthreads();
      xt = thread_base<A0>(tid);
      from_smem<A0>(v, tile, xt);
    }
    // A truncated transform drops the rows past krows: whole 16-row groups
    // (the thread's, warp by warp), or the last rows of the one group (R = 16).
    const bool kept = !kCutFwd || LOGR == 4 || static_cast<int>((xt >> (ROWOFF + 4)) << 4) < krows;
    if (kept) {
      if (G == 1 && ztop)
        stages<4, 0, A0, ROWOFF, 0, LOGR, false, true, true, G == 1>(v, tw, xt, p, c);
      else
        stages<4, 0, A0, ROWOFF, 0, LOGR, false, true, true>(v, tw, xt, p, c);
      inter_pass(v, xt, tb.hi_fwd, tb.lo_fwd);
    }
    __syncthreads();
    if (kept) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (!(kCutFwd && LOGR == 4 && i >= krows)) check_below(v[i], p);  // after the Montgomery inter-pass twiddle
        tile[xt | (static_cast<uint32_t>(i) << A0)] = v[i];
      }
    }
  } else {
    // Registers of the rows [0, kRows) hold the known outputs, the others nothing.
    constexpr int NK0 = LOGR == 4 ? kRows : 16;  // layout A0: registers of a thread with known rows
    constexpr int NK1 = KI;                      // the pass's last layout: register i is row bits LOGR-4 .. LOGR-1
    xt = thread_base<A0>(tid);
    const bool known = KI == 16 || LOGR == 4 || static_cast<int>((xt >> (ROWOFF + 4)) << 4) < kRows;
    if (known) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i >= NK0) {
          v[i] = 0;
          continue;
        }
        v[i] = tile[xt | (static_cast<uint32_t>(i) << A0)];
        check_below(v[i], 2 * p);  // inverse residues live in [0, 2p)
      }
      inter_pass(v, xt, tb.hi_inv, tb.lo_inv);
      if constexpr (KI == 16 || LOGR > 4) {
        stages<4, 0, A0, ROWOFF, 0, LOGR, true, true, true>(v, tw, xt, p, c);
      } else if constexpr (KI % 2 == 0) {  // the stage on row bit 0 of the known rows, then the top three bits
#pragma unroll
        for (int i = 0; i < kRows; i += 2) {
          const uint64_t u = v[i], w = v[i + 1];
          v[i] = u + w;
          v[i + 1] = u - w + p;
        }
        TruncatedInverse<LOGR, A0, ROWOFF, true>{tw, twf, xt, p, c}.template run<3, 1, KI / 2, 0, true>(v);
      } else {
        TruncatedInverse<LOGR, A0, ROWOFF, true>{tw, twf, xt, p, c}.template run<3, 0, KI, 0, true>(v);
      }
    }
    constexpr int AS = (G == 2) ? A1 : A0;
    if constexpr (G == 2) {
      __syncthreads();
      if (known) to_smem<A0>(tile, v, xt);
      __syncthreads();
      xt = thread_base<A1>(tid);
#pragma unroll
      for (int i = 0; i < NK1; ++i) v[i] = tile[xt | (static_cast<uint32_t>(i) << A1)];
      if constexpr (KI == 16) {
        stages<NB1, 4 - NB1, A1, ROWOFF, 4, LOGR, true, false>(v, tw, xt, p, c);
      } else {
        constexpr int JL = 8 - LOGR;  // register bit of the lowest row bit that this round still owes
        TruncatedInverse<LOGR, A1, ROWOFF, false>{tw, twf, xt, p, c}.template run<3, JL, (KI >> JL), 0, true>(v);
      }
    }
    if constexpr (SCALE) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = mont_mul(v[i], P.scale, p, c);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NK1; ++i) {
      check_below(v[i], 2 * p);
      tile[xt | (static_cast<uint32_t>(i) << AS)] = v[i];
    }
  }
  tma::fence_async_smem();
  __syncthreads();
  if (tid == 0) {
    tma::store_5d(&maps.out[op], tile, s0, 0, blk, prime - P.prime_lo, static_cast<int>(prod));
    tma::store_wait_read();
  }
}

// The inter-pass twiddles w_M^(s * bitrev(r)) of one (M, R, direction) in
// Montgomery form, [prime][r][s]; with scale[j] != 0 (a Montgomery-form
// factor) every entry of prime j is multiplied by it.
__global__ void pass_twiddles_kernel(uint64_t *out, int logM, int logR, bool inverse, NttTables t0, NttTables t1,
                                     NttTables t2, PrimeConst c0, PrimeConst c1, PrimeConst c2, uint64_t s0,
                                     uint64_t s1, uint64_t s2) {
  const uint64_t M = uint64_t(1) << logM;
  const int j = static_cast<int>(blockIdx.y);
  const NttTables &t = j == 0 ? t0 : (j == 1 ? t1 : t2);
  const PrimeConst &pc = j == 0 ? c0 : (j == 1 ? c1 : c2);
  const uint64_t scale = j == 0 ? s0 : (j == 1 ? s1 : s2);
  const int logS = logM - logR;
  for (uint64_t e = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; e < M;
       e += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t r = e >> logS, s = e & ((uint64_t(1) << logS) - 1);
    const uint64_t E = (s * bitrev(static_cast<uint32_t>(r), logR)) & (M - 1);
    uint64_t w = table_twiddle(E, logM, inverse ? t.hi_inv : t.hi_fwd, inverse ? t.lo_inv : t.lo_fwd, pc.p, pc.c);
    if (scale) w = mont_mul(w, scale, pc.p, pc.c);
    out[static_cast<uint64_t>(j) * M + e] = w;
  }
}

bool reads_limbs(const PassArgs &a) {
  if (a.batch) return a.read_limbs != 0;
  return a.limbs[0] != nullptr || (a.nops > 1 && a.limbs[1] != nullptr);
}

template <int LOGR>
cudaError_t launch_r(const PassArgs &a, bool inverse, unsigned grid, cudaStream_t st) {
  if (inverse && a.scale) return launch_dep(ntt_strided_kernel<LOGR, true, true>, grid, kTileThreads, 0, st, a);
  if (inverse)
    return launch_dep(ntt_strided_kernel<LOGR, true>, grid, kTileThreads, 0, st, a);
  const bool digits = a.dig80 && reads_limbs(a);
  if constexpr (LOGR != 5) {
    if (a.krows < (1 << LOGR))
      return digits ? launch_dep(ntt_strided_kernel<LOGR, false, true, true>, grid, kTileThreads, 0, st, a)
                    : launch_dep(ntt_strided_kernel<LOGR, false, true>, grid, kTileThreads, 0, st, a);
  }
  if (digits) return launch_dep(ntt_strided_kernel<LOGR, false, false, true>, grid, kTileThreads, 0, st, a);
  return launch_dep(ntt_strided_kernel<LOGR, false>, grid, kTileThreads, 0, st, a);
}

// ---- tensor maps ----------------------------------------------------------

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    else
      cudaGetLastError();
  });
  return fn;
}

cudaError_t encode(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
                   const cuuint32_t *box) {
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, static_cast<cuuint32_t>(rank), const_cast<void *>(base),
                        dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// The residue arrays of one operand as a 5-D tensor: column s (S), row r (R,
// or the kept rows of a truncated outer pass), block (points / M), prime
// (nprimes, prime_stride apart), product (nprod, ws_stride apart); the box is
// one tile, C columns by the rows.
cudaError_t residue_map(CUtensorMap *m, const uint64_t *base, const PassArgs &a) {
  const uint64_t S = uint64_t(1) << a.logS, R = uint64_t(1) << a.logR, K = static_cast<uint64_t>(a.krows);
  const uint64_t M = R * S;
  const cuuint64_t dims[5] = {S, K, K < R ? 1 : a.points / M, static_cast<cuuint64_t>(a.nprimes), a.nprod};
  const uint64_t pstride = a.nprimes > 1 ? a.prime_stride : a.points;
  const uint64_t wstride = a.nprod > 1 ? a.ws_stride : a.points * static_cast<uint64_t>(a.nprimes);
  const cuuint64_t strides[4] = {S * 8, M * 8, pstride * 8, wstride * 8};
  const cuuint32_t box[5] = {static_cast<cuuint32_t>((uint64_t(1) << kTileBits) / R), static_cast<cuuint32_t>(K), 1,
                             1, 1};
  return encode(m, base, 5, dims, strides, box);
}

// The pass's inter-pass twiddle table [prime][r][s] (M words per prime, every
// prime of the scheme) as a 3-D tensor with the same box.
cudaError_t twiddle_map(CUtensorMap *m, const uint64_t *ptw, const PassArgs &a) {
  const uint64_t S = uint64_t(1) << a.logS, R = uint64_t(1) << a.logR;
  const cuuint64_t dims[3] = {S, R, static_cast<cuuint64_t>(kPrimes)};
  const cuuint64_t strides[2] = {S * 8, R * S * 8};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>((uint64_t(1) << kTileBits) / R),
                             static_cast<cuuint32_t>(a.krows), 1};
  return encode(m, ptw, 3, dims, strides, box);
}

template <int LOGR, bool INV, bool TABLE, bool LIMBS, int KQ = 16, bool SCALE = false, bool D80 = false>
cudaError_t launch_tma_v(const TmaMaps &m, const PassArgs &a, const TmaLimbs &l, unsigned grid, cudaStream_t st) {
  constexpr size_t bytes = ((D80 ? 5 : 4) + (TABLE ? 4 : 0)) * (size_t(1) << (kTileBits - 2)) * sizeof(uint64_t);
  // Raise the dynamic shared-memory limit once per instantiation (not on
  // every launch, so that launches can be captured in a CUDA graph).
  static bool raised = false;
  if (bytes > 48 * 1024 && !raised) {
    cudaError_t e = cudaFuncSetAttribute(ntt_strided_tma_kernel<LOGR, INV, TABLE, LIMBS, KQ, SCALE, D80>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    raised = true;
  }
  return launch_dep(ntt_strided_tma_kernel<LOGR, INV, TABLE, LIMBS, KQ, SCALE, D80>, grid, kTileThreads, bytes, st, m, a,
                    l);
}

// The outer inverse pass of a truncated transform that keeps KQ sixteenths.
template <int LOGR, int KQ>
cudaError_t launch_cut(const TmaMaps &m, const PassArgs &a, const TmaLimbs &l, unsigned grid, cudaStream_t st) {
  if constexpr (truncation_ok(LOGR, KQ))
    return a.ptw ? launch_tma_v<LOGR, true, true, false, KQ>(m, a, l, grid, st)
                 : launch_tma_v<LOGR, true, false, false, KQ>(m, a, l, grid, st);
  return cudaErrorInvalidValue;
}

template <int LOGR, bool D80>
cudaError_t launch_limbs(const TmaMaps &m, const PassArgs &a, const TmaLimbs &l, unsigned grid, cudaStream_t st) {
  if constexpr (LOGR != 5) {
    if (a.krows < (1 << LOGR))
      return a.ptw ? launch_tma_v<LOGR, false, true, true, kCut, false, D80>(m, a, l, grid, st)
                   : launch_tma_v<LOGR, false, false, true, kCut, false, D80>(m, a, l, grid, st);
  }
  return a.ptw ? launch_tma_v<LOGR, false, true, true, 16, false, D80>(m, a, l, grid, st)
               : launch_tma_v<LOGR, false, false, true, 16, false, D80>(m, a, l, grid, st);
}

template <int LOGR>
cudaError_t launch_tma_r(const TmaMaps &m, const PassArgs &a, const TmaLimbs &l, bool inverse, bool limbs,
                         unsigned grid, cudaStream_t st) {
  const bool table = a.ptw != nullptr;
  if (inverse && a.krows < (1 << LOGR)) {
    switch (16 * a.krows >> LOGR) {
      case 9: return launch_cut<LOGR, 9>(m, a, l, grid, st);
      case 10: return launch_cut<LOGR, 10>(m, a, l, grid, st);
      case 11: return launch_cut<LOGR, 11>(m, a, l, grid, st);
      case 12: return launch_cut<LOGR, 12>(m, a, l, grid, st);
      case 13: return launch_cut<LOGR, 13>(m, a, l, grid, st);
      case 14: return launch_cut<LOGR, 14>(m, a, l, grid, st);
      case 15: return launch_cut<LOGR, 15>(m, a, l, grid, st);
      default: return cudaErrorInvalidValue;
    }
  }
  if (inverse && a.scale)
    return table ? launch_tma_v<LOGR, true, true, false, 16, true>(m, a, l, grid, st)
                 : launch_tma_v<LOGR, true, false, false, 16, true>(m, a, l, grid, st);
  if (inverse)
    return table ? launch_tma_v<LOGR, true, true, false>(m, a, l, grid, st)
                 : launch_tma_v<LOGR, true, false, false>(m, a, l, grid, st);
  if (limbs)
    return a.dig80 ? launch_limbs<LOGR, true>(m, a, l, grid, st) : launch_limbs<LOGR, false>(m, a, l, grid, st);
  return table ? launch_tma_v<LOGR, false, true, false>(m, a, l, grid, st)
               : launch_tma_v<LOGR, false, false, false>(m, a, l, grid, st);
}

// `count` operands of nl limbs, `stride` limbs apart, as rows of S limbs (5 S / 4
// for 80-bit digits): a 3-D map over their complete rows.
uint64_t limb_row(const PassArgs &a) { return limbs_of(uint64_t(1) << a.logS, a.dig80 != 0); }

cudaError_t limb_map(CUtensorMap *m, const uint64_t *limbs, uint64_t nl, uint64_t count, uint64_t stride,
                     const PassArgs &a) {
  const uint64_t W = limb_row(a), R = uint64_t(1) << a.logR;
  const cuuint64_t dims[3] = {W, nl / W, count};
  const cuuint64_t strides[2] = {W * 8, stride * 8};
  uint64_t cols = limbs_of((uint64_t(1) << kTileBits) / R, a.dig80 != 0);
  if (cols > 256) cols /= 2;  // R = 16: two boxes
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(cols), static_cast<cuuint32_t>(R), 1};
  return encode(m, limbs, 3, dims, strides, box);
}

// The limbs of a cut operand's last chunk.
uint64_t last_chunk(const PassArgs &a) { return a.nlimbs[0] - (a.nprod - 1) * a.chunk; }

// A first forward pass of one product (not a batch) whose block is the whole
// transform reads its limbs through TMA: each operand's limbs (each chunk's)
// fill at least one row of S, start on a 16-byte boundary and lie in the
// pass's single block.  Chunks against per-thread loads: 2^24 x 2^16 limbs
// 1709 -> 1692 us, 20000 x 500 35.8 -> 34.5, 2^22 x 2^14 439.7 -> 434.9.
bool tma_limbs_ok(const PassArgs &a) {
  if (a.batch || a.logS + a.logR != a.logN) return false;
  if (a.chunk)
    return a.nops == 1 && a.nprod > 1 && a.limbs[0] && (reinterpret_cast<uintptr_t>(a.limbs[0]) & 15u) == 0 &&
           a.chunk % 2 == 0 && a.chunk >= limb_row(a) && coefs_of(a.chunk, a.dig80 != 0) <= (uint64_t(1) << a.logN) &&
           a.nlimbs[0] > (a.nprod - 1) * a.chunk && last_chunk(a) <= a.chunk && last_chunk(a) >= limb_row(a);
  if (a.nprod != 1) return false;
  for (int op = 0; op < a.nops; ++op) {
    if (!a.limbs[op] || (reinterpret_cast<uintptr_t>(a.limbs[op]) & 15u)) return false;
    if (a.nlimbs[op] < limb_row(a) || coefs_of(a.nlimbs[op], a.dig80 != 0) > (uint64_t(1) << a.logN)) return false;
  }
  return true;
}

// TMA copies need 16-byte aligned arrays; the spectrum entry points take a
// caller's pointer, which may sit at any 8-byte offset.
bool tma_aligned(const PassArgs &a) {
  const auto al = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  return al(a.data[0]) && (a.nops < 2 || al(a.data[1])) && (!a.ptw || al(a.ptw)) && (a.prime_stride & 1) == 0 &&
         (a.ws_stride & 1) == 0;
}

}  // namespace

#if HG_CHECKED
HG_CHECKED_READER(checked_fault_strided)
#endif

cudaError_t launch_pass_twiddles(uint64_t *out, int logM, int logR, bool inverse, const NttTables *tb,
                                 const PrimeConst *pc, int nprimes, cudaStream_t st, const uint64_t *scale) {
  if (nprimes < 1 || nprimes > kPrimes || logR < 1 || logR > 8 || logM <= logR || logM > kLogNmax)
    return cudaErrorInvalidValue;
  const uint64_t M = uint64_t(1) << logM;
  const unsigned gx = static_cast<unsigned>(std::min<uint64_t>((M + 255) / 256, 152 * 64));
  const int j1 = nprimes > 1 ? 1 : 0, j2 = nprimes > 2 ? 2 : 0;
  pass_twiddles_kernel<<<dim3(gx, static_cast<unsigned>(nprimes)), 256, 0, st>>>(
      out, logM, logR, inverse, tb[0], tb[j1], tb[j2], pc[0], pc[j1], pc[j2], scale ? scale[0] : 0,
      scale ? scale[j1] : 0, scale ? scale[j2] : 0);
  return cudaGetLastError();
}

cudaError_t launch_ntt_strided(const PassArgs &a, bool inverse, cudaStream_t st) {
  const uint64_t grid = a.tiles * a.nprod * static_cast<uint64_t>(a.nops) * static_cast<uint64_t>(a.nprimes);
  if (grid == 0 || grid > 0x7fffffffull || a.logT != kTileBits || a.logS < kTileBits - a.logR)
    return cudaErrorInvalidValue;
  const unsigned g = static_cast<unsigned>(grid);
  const bool limbs = reads_limbs(a);
  const int R = 1 << a.logR;
  if (a.krows < R) {  // truncated: the outer pass, its forward side from limbs, by rows the kernels can cut
    if (a.logR + a.logS != a.logN || !truncation_ok(a.logR, 16 * a.krows >> a.logR) || (16 * a.krows) % R ||
        a.points != static_cast<uint64_t>(a.krows) << a.logS || (inverse ? !tma_aligned(a) : !limbs))
      return cudaErrorInvalidValue;
  } else if (a.krows != R || (a.points >> (a.logR + a.logS)) == 0) {
    return cudaErrorInvalidValue;
  }
  if (tma_aligned(a) && (!limbs || tma_limbs_ok(a))) {
    TmaMaps m{};
    TmaLimbs l{};
    cudaError_t e = cudaSuccess;
    for (int op = 0; op < 2 && e == cudaSuccess; ++op) {
      if (op >= a.nops && !(limbs && a.chunk)) break;  // no CTA uses map 1; an encode is 0.5 to 1 us of host time
      if (op < a.nops) e = residue_map(&m.out[op], a.data[op], a);
      if (e != cudaSuccess) break;
      if (!limbs) {
        m.in[op] = m.out[op];
        continue;
      }
      const int lo = op < a.nops ? op : 0;
      const uint64_t *p = a.limbs[lo];
      uint64_t nl = a.nlimbs[lo], count = 1, stride = limb_row(a);
      l.limbs[op] = p;
      if (a.chunk && op == 0) {
        nl = stride = a.chunk;
        count = a.nprod - 1;
      } else if (a.chunk) {
        nl = last_chunk(a);
        p += (a.nprod - 1) * a.chunk;
      }
      l.full_rows[op] = nl / limb_row(a);
      l.tail[op] = nl % limb_row(a);
      // Every limb lies in the lower half of the block: the first stage's
      // upper inputs are zero.
      if (coefs_of(nl, a.dig80 != 0) <= (uint64_t(1) << (a.logS + a.logR - 1))) l.ztop |= 1u << op;
      e = limb_map(&m.in[op], p, nl, count, stride, a);
    }
    if (e == cudaSuccess && a.ptw) e = twiddle_map(&m.tw, a.ptw, a);
    if (e != cudaSuccess) return e;
    switch (a.logR) {
      case 4: return launch_tma_r<4>(m, a, l, inverse, limbs, g, st);
      case 5: return launch_tma_r<5>(m, a, l, inverse, limbs, g, st);
      case 6: return launch_tma_r<6>(m, a, l, inverse, limbs, g, st);
      case 7: return launch_tma_r<7>(m, a, l, inverse, limbs, g, st);
      case 8: return launch_tma_r<8>(m, a, l, inverse, limbs, g, st);
      default: return cudaErrorInvalidValue;
    }
  }
  switch (a.logR) {
    case 4: return launch_r<4>(a, inverse, g, st);
    case 5: return launch_r<5>(a, inverse, g, st);
    case 6: return launch_r<6>(a, inverse, g, st);
    case 7: return launch_r<7>(a, inverse, g, st);
    case 8: return launch_r<8>(a, inverse, g, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hg
