// hg_ntt_rounds.cuh -- register rounds shared by the NTT kernels.
//
// A CTA owns a tile of 2^T residues (T <= 12).  Tile position x holds row r
// of column c: strided tiles keep the column in the low bits (x = r << ROWOFF
// | c), contiguous blocks have ROWOFF = 0.  In a round, each thread holds 16
// residues whose tile positions differ only in the four bits [A, A+4): the
// residue of register i sits at xt | (i << A), where xt deposits the thread
// index into the other bits.  Up to four radix-2 stages run on those
// registers; between rounds the tile goes through shared memory once.
//
// Every shape (A, ROWOFF, which row bits a round owns) is a template
// argument, so all index arithmetic folds to constants except one thread
// offset per stage.
#pragma once

#include "hg_internal.h"

namespace hg {
namespace rounds {

// A residue a contiguous pass reads once: not allocated in L1, which keeps
// L1 for the twiddle tables (the 2^25-point middle kernel 2.335 -> 2.319
// ms; marking the tables' loads evict-last as well measured 2.334 ms).
__device__ __forceinline__ uint64_t ld_once(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.global.L1::no_allocate.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t bitrev(uint32_t r, int bits) { return __brev(r) >> (32 - bits); }

// Thread part of the tile position for register block [A, A+4).
template <int A>
__device__ __forceinline__ uint32_t thread_base(uint32_t tid) {
  return (tid & ((1u << A) - 1u)) | ((tid >> A) << (A + 4));
}

// (w_R^e, companion), e < R/2, loaded into shared memory at entry e.  A
// strided pass's lanes run along columns, so the 8 lanes of one 16-byte
// access read the same entry.
__device__ __forceinline__ void load_sub_twiddles(ulonglong2 *tw, const ulonglong2 *src, int logR, int tid, int nthr) {
  const int half = 1 << (logR - 1);
  for (int e = tid; e < half; e += nthr) tw[e] = __ldg(src + (static_cast<uint64_t>(e) << (kTileBits - logR)));
}

// Twiddle w_M^E (E < M = 2^logM) in Montgomery form from the two-level tables
// of w_{2^30}.
__device__ __forceinline__ uint64_t table_twiddle(uint64_t E, int logM, const uint64_t *hi, const uint64_t *lo,
                                                  uint64_t p, uint32_t c) {
  const uint64_t e = E << (kLogNmax - logM);
  const uint64_t th = __ldg(hi + (e >> kTwLevelBits));
  const uint64_t tl = __ldg(lo + (e & ((1u << kTwLevelBits) - 1)));
  return mont_mul(th, tl, p, c);
}

// NB radix-2 stages on register bits [JG, JG+NB) = row bits [BLO, BLO+NB).
// The stage on row bit b multiplies by w_{2^(b+1)}^(r mod 2^b), read from the
// R/2-entry table of w_R at (r mod 2^b) << (LOGR-1-b).  r mod 2^b splits into
// the thread's row bits below b (runtime, zero when TZERO) and the register's
// (compile time).  With TZERO, butterflies whose twiddle is 1 skip the
// multiplication.
//
// Forward (DIF) butterflies keep every residue in [0, p), as ntt-forward
// does.  Inverse (DIT) butterflies take and leave [0, 2p) (2p < 2^64): u is
// folded once, v w is a corrected Shoup product (v folded when w = 1), and
// u + t, u - t + p need no correction.  Every consumer of an inverse
// residue accepts [0, 2p): the next pass's Montgomery pre-twiddle, the 1/N
// scaling and the reconstruction's Shoup products.
//
// EDGE marks the stage on row bit 0 (BLO = 0, twiddle 1) of a pass whose
// neighbour is a Montgomery product: forward, it is the last stage and its
// u + v, u - v + p go uncorrected ([0, 2p)) into the inter-pass twiddle;
// inverse, it is the first stage and its inputs are already in [0, p).
//
// ZTOP (forward only) marks a first stage whose upper inputs are all zero
// (the zero padding above an operand's limbs): u + 0 and (u - 0) w need
// neither the sum's correction nor the difference, only the product.
//
// CONTIG: the twiddle table is in a contiguous pass's padded order (tw_pos;
// its lanes have different row bits); otherwise entry e sits at e (a
// strided pass's lanes share their row bits).  Either way a twiddle's index
// is the thread's part plus a compile-time part: the thread's table pointer
// is formed once per stage, and each load takes the register's part as its
// address offset.  Dropping the XOR swizzle of the strided passes' tables
// and tiles took the forward strided pass from 0.996 to 0.980 ms and the
// inverse from 0.496 to 0.484 ms (2^25 points).
template <int NB, int JG, int A, int ROWOFF, int BLO, int LOGR, bool INV, bool TZERO, bool EDGE = false,
          bool ZTOP = false, bool CONTIG = false>
__device__ __forceinline__ void stages(uint64_t (&v)[16], const ulonglong2 *__restrict__ tw, uint32_t xt, uint64_t p,
                                       uint32_t c) {
  static_assert(!EDGE || (TZERO && BLO == 0), "the edge stage is the twiddle-free stage on row bit 0");
  static_assert(!ZTOP || !INV, "zero upper inputs only in a forward pass");
#pragma unroll
  for (int s = 0; s < NB; ++s) {
    const int jj = INV ? s : NB - 1 - s;
    const int j = JG + jj;
    const int b = BLO + jj;
    const int sh = LOGR - 1 - b;
    const uint32_t lowmask = (1u << b) - 1u;
    const uint32_t te = TZERO ? 0u : ((xt >> ROWOFF) & lowmask) << sh;
    const ulonglong2 *__restrict__ tws = tw + (CONTIG ? tw_pos(te) : te);
    auto at = [&](uint32_t k) { return CONTIG ? __ldg(tws + tw_pos(k)) : tws[k]; };
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i & (1 << j)) continue;
      const uint32_t rp = ((static_cast<uint32_t>(i) << A) >> ROWOFF) & lowmask;
      const bool trivial = TZERO && rp == 0;
      const uint64_t u = v[i], w = v[i | (1 << j)];
      if (EDGE && jj == 0) {  // twiddle 1, inputs in [0, p): outputs in [0, 2p)
        v[i] = u + w;
        v[i | (1 << j)] = u - w + p;
        continue;
      }
      if (ZTOP && s == 0) {  // w = 0: v[i] keeps u
        if (trivial) {
          v[i | (1 << j)] = u;
        } else {
          const ulonglong2 t = at(rp << sh);
          v[i | (1 << j)] = shoup_mul(u, t.x, t.y, p, c);
        }
        continue;
      }
      if (!INV) {
        v[i] = add_mod(u, w, p);
        if (trivial) {
          v[i | (1 << j)] = sub_mod(u, w, p);
        } else {
          const ulonglong2 t = at(rp << sh);
          v[i | (1 << j)] = shoup_mul(u - w + p, t.x, t.y, p, c);  // u - w + p in (0, 2p)
        }
      } else {
        const uint64_t uu = fold_p(u, p);
        uint64_t t;
        if (trivial) {
          t = fold_p(w, p);
        } else {
          const ulonglong2 tt = at(rp << sh);
          t = shoup_mul(w, tt.x, tt.y, p, c);
        }
        v[i] = uu + t;               // [0, 2p)
        v[i | (1 << j)] = uu - t + p;  // (0, 2p)
      }
    }
  }
}

// Shared-memory word of tile position x: data_swz(x) in a contiguous pass
// (its lanes may run at a stride of 16 positions), x in a strided pass
// (lanes run along columns, one position apart; the thread's word pointer
// is formed once and each register's part is the access's address offset).
template <bool CONTIG>
struct SmemAt {
  uint64_t *s;
  uint32_t sx;
  __device__ __forceinline__ SmemAt(uint64_t *sm, uint32_t xt) : s(sm + (CONTIG ? 0u : xt)), sx(data_swz(xt)) {}
  __device__ __forceinline__ uint64_t &operator[](uint32_t k) const { return CONTIG ? s[sx ^ data_swz(k)] : s[k]; }
};

// Registers <-> shared memory for register block A.
template <int A, bool CONTIG = false>
__device__ __forceinline__ void to_smem(uint64_t *sm, const uint64_t (&v)[16], uint32_t xt) {
  const SmemAt<CONTIG> s(sm, xt);
#pragma unroll
  for (int i = 0; i < 16; ++i) s[static_cast<uint32_t>(i) << A] = v[i];
}
template <int A, bool CONTIG = false>
__device__ __forceinline__ void from_smem(uint64_t (&v)[16], uint64_t *sm, uint32_t xt) {
  const SmemAt<CONTIG> s(sm, xt);
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = s[static_cast<uint32_t>(i) << A];
}

// The inverse of a truncated transform's top row bits, on registers.
//
// A truncated transform (van der Hoeven's truncated Fourier transform) keeps
// the first krows of the outer pass's R rows of outputs: krows S points
// determine a product of at most krows S coefficients.  Its inverse gets, per
// column, the R-point transform's first outputs, and knows that the rows of
// the result past krows are zero.  After the stages of the low row bits (run
// on the known rows only, as in a whole transform), each thread holds 2^JN
// values that differ in the top JN row bits (register bits J = JL .. 3):
// the first K are the transform's, the others are known results (zero at
// the top level).  run<J, JL, K, OFF, ZT> solves the n = 2^(J - JL + 1)
// values at OFF for the first K results, scaled by n as the unscaled inverse
// leaves them; results past K are already known.  With u and v the half-size
// transforms' inputs (u_h = x_h + x_(h+n/2), v_h = (x_h - x_(h+n/2)) w^h):
//   K > n/2: every u is an inverse of known outputs.  For h >= K - n/2 the
//     upper result is known, so v_h = (u_h - 2 x_(h+n/2)) w^h is too and x_h
//     = u_h - x_(h+n/2); the rest of v is the same problem at half the size,
//     and its butterflies are the inverse's own.
//   K <= n/2: u_h is known for h >= K, the rest of u is the same problem, and
//     x_h = u_h - x_(h+n/2).
// Every value is in [0, 2p) before and after.
template <int LOGR, int A, int ROWOFF, bool TZERO>
struct TruncatedInverse {
  const ulonglong2 *twi, *twf;  // (w_R^-e, companion), (w_R^e, companion), e < R / 2
  uint32_t xt;
  uint64_t p;
  uint32_t c;

  // Entry of the stage on register bit J's row bit for register i.
  template <int J>
  __device__ __forceinline__ uint32_t entry(int i) const {
    constexpr int b = J + A - ROWOFF;
    constexpr uint32_t lowmask = (1u << b) - 1u;
    constexpr int sh = LOGR - 1 - b;
    const uint32_t te = TZERO ? 0u : ((xt >> ROWOFF) & lowmask) << sh;
    return te + ((((static_cast<uint32_t>(i) << A) >> ROWOFF) & lowmask) << sh);
  }

  template <int J>
  __device__ __forceinline__ void butterfly(uint64_t (&v)[16], int i) const {
    const uint64_t u = fold_p(v[i], p), w = v[i | (1 << J)];
    uint64_t t;
    if (TZERO && entry<J>(i) == 0) {
      t = fold_p(w, p);
    } else {
      const ulonglong2 tt = twi[entry<J>(i)];
      t = shoup_mul(w, tt.x, tt.y, p, c);
    }
    v[i] = u + t;
    v[i | (1 << J)] = u - t + p;
  }

  // 2 a - b mod p in (0, 2p)
  __device__ __forceinline__ uint64_t twice_less(uint64_t a, uint64_t b) const {
    return fold_p(2 * fold_p(a, p), p) - fold_p(b, p) + p;
  }

  template <int J, int JL, int K, int OFF, bool ZT>
  __device__ __forceinline__ void run(uint64_t (&v)[16]) const {
    if constexpr (J >= JL) {
      constexpr int half = 1 << (J - JL), U = 1 << J;
      if constexpr (K == 2 * half) {
        run<J - 1, JL, half, OFF, false>(v);
        run<J - 1, JL, half, OFF | U, false>(v);
#pragma unroll
        for (int q = 0; q < (half << JL); ++q) butterfly<J>(v, OFF | q);
      } else if constexpr (K > half) {
        constexpr int K1 = K - half;
        run<J - 1, JL, half, OFF, false>(v);
#pragma unroll
        for (int q = (K1 << JL); q < (half << JL); ++q) {
          const int i = OFF | q;
          const uint64_t u = v[i], x = v[i | U];  // x: known (zero when ZT)
          const uint64_t d = ZT ? u : fold_p(u, p) - fold_p(x, p) + p;
          if (TZERO && entry<J>(i) == 0) {
            v[i | U] = d;
          } else {
            const ulonglong2 t = twf[entry<J>(i)];
            v[i | U] = shoup_mul(d, t.x, t.y, p, c);
          }
          v[i] = ZT ? 2 * fold_p(u, p) : twice_less(u, x);
        }
        run<J - 1, JL, K1, OFF | U, false>(v);
#pragma unroll
        for (int q = 0; q < (K1 << JL); ++q) butterfly<J>(v, OFF | q);
      } else {
        static_assert(!ZT, "a truncated transform keeps more than half its rows");
#pragma unroll
        for (int q = (K << JL); q < (half << JL); ++q) {  // u_h = (x_h + x_(h+n/2)) at half the scale
          const int i = OFF | q;
          const uint64_t s = add_mod(fold_p(v[i], p), fold_p(v[i | U], p), p);
          v[i] = (s + ((s & 1) ? p : 0)) >> 1;
        }
        run<J - 1, JL, K, OFF, false>(v);
#pragma unroll
        for (int q = 0; q < (K << JL); ++q) v[OFF | q] = twice_less(v[OFF | q], v[OFF | q | U]);
      }
    }
  }
};

// Multiply register i by beta * gamma^bitrev4(i) (Montgomery-form beta, gamma):
// the twiddle w_M^(s * bitrev_R(r)) of the 16 rows r = rhi*16 + i of one
// column, with beta = w_M^(s * bitrev(rhi)), gamma = w_M^(s * R/16).
__device__ __forceinline__ void geometric_twiddle(uint64_t (&v)[16], uint64_t beta, uint64_t gamma, uint64_t p,
                                                  uint32_t c) {
  uint64_t t = beta;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int i = ((k & 1) << 3) | ((k & 2) << 1) | ((k & 4) >> 1) | ((k & 8) >> 3);  // bitrev4(k)
    v[i] = mont_mul(v[i], t, p, c);
    if (k < 15) t = mont_mul(t, gamma, p, c);
  }
}

}  // namespace rounds
}  // namespace hg
