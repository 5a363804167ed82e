// hg_carry.cuh -- reconstruction and carry bodies shared by the per-launch
// carry kernels (hg_crt.cu) and the persistent batch kernel (hg_persist.cu).
//
// The reference rebuilds each convolution coefficient as a bignum
// sum_j f_j r_j mod M and adds it at limb i with a recursive carry ripple
// (src/ntt-multiply.lisp:10-51, 242-253).  CrtProducer gives each
// coefficient by Garner's mixed radix; carry_body writes one tile of limbs
// with carry-in 0 and publishes the tile's (generate, propagate) aggregate;
// fix_body, run after every tile of the product has published, composes a
// tile's carry-in from the aggregates below it and applies it.
#pragma once

#include "hg_internal.h"

namespace hg {
namespace carry {

constexpr int kCarryPer = 8;  // positions per thread (4 in short launches, hg_crt.cu)

template <int TILE>
__device__ __forceinline__ uint64_t carry_tiles_dev(uint64_t n) { return (n + TILE - 1) / TILE; }

struct V3 {
  uint64_t w0, w1, w2;
};

__device__ __forceinline__ void add128_to(V3 &acc, uint64_t lo, uint64_t hi) {
  const uint64_t s0 = acc.w0 + lo;
  const uint64_t c0 = s0 < lo;
  const uint64_t t1 = acc.w1 + hi;
  const uint64_t c1 = t1 < hi;
  const uint64_t s1 = t1 + c0;
  const uint64_t c2 = s1 < c0;
  acc.w0 = s0;
  acc.w1 = s1;
  acc.w2 += c1 + c2;
}

// acc += x y.  As one 128-bit product: a pair of 64-bit low and high products
// costs a third more (mont_mul).
__device__ __forceinline__ void add_product_to(V3 &acc, uint64_t x, uint64_t y) {
  const unsigned __int128 v = static_cast<unsigned __int128>(x) * y;
  add128_to(acc, static_cast<uint64_t>(v), static_cast<uint64_t>(v >> 64));
}

// PRESCALED: the residues are the coefficients mod p_j (CrtConst::prescaled).
// SAME_LAUNCH: an earlier phase of the same launch (the persistent batch kernel)
// wrote them, so they are read through L2 (ld.global.cg).  Else the launch
// before did: plain loads, whose L1 serves the other half of the sectors that a
// thread's 16-byte loads touch (the 4096-pair batch 2650 us through L2, 2621
// this way), and not the read-only path, since a dependent launch is resident
// before those writes are visible.
template <bool PRESCALED = false, bool SAME_LAUNCH = false>
struct CrtProducerT {
  const uint64_t *res;  // [3][N] natural-order residues from the unscaled inverse
  uint64_t n;           // N
  CrtConst k;

  // Coefficient i of the product whose residues start `off` words past res.
  __device__ __forceinline__ V3 at(uint64_t off, uint64_t i) const {
    const uint64_t *r = res + off;
    return garner(r[i], r[n + i], r[2 * n + i]);
  }

  // PER consecutive positions from i0 (a multiple of PER, 4 or 8): 16-byte loads.
  template <int PER>
  __device__ __forceinline__ void many(uint64_t off, uint64_t i0, uint64_t nproc, V3 (&v)[PER]) const {
    if (i0 + PER <= nproc) {
      uint64_t r[3][PER];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(res + off + j * n + i0);
#pragma unroll
        for (int q = 0; q < PER / 2; ++q) {
          const ulonglong2 w = SAME_LAUNCH ? __ldcg(src + q) : src[q];
          r[j][2 * q] = w.x;
          r[j][2 * q + 1] = w.y;
        }
      }
#pragma unroll
      for (int k8 = 0; k8 < PER; ++k8) v[k8] = garner(r[0][k8], r[1][k8], r[2][k8]);
    } else {
#pragma unroll
      for (int k8 = 0; k8 < PER; ++k8) v[k8] = (i0 + k8 < nproc) ? at(off, i0 + k8) : V3{0, 0, 0};
    }
  }

  __host__ __device__ __forceinline__ bool drop_top() const { return false; }

  // Residues lie in [0, 2p) (the inverse leaves them there).  Unscaled,
  // every one enters through a Shoup product that also applies N^-1 2^64.
  // Prescaled (the residues are the coefficient mod p_j), Garner's steps
  // need three Shoup products instead of six: y0 = c mod p0 is r0 folded,
  // t1 = (c - y0) / p0 mod p1 takes (r1 - y0) reduced to (0, 2 p1), and
  // t2 takes r2 - y0 + p2 in (0, 3 p2) as it is.  The host prescales only
  // where p0 < 2 p1, p0 < 2 p2 and 3 p2 < 2^64 (the reference's moduli).
  __device__ __forceinline__ V3 garner(uint64_t r0, uint64_t r1, uint64_t r2) const {
    const uint64_t p0 = k.pc[0].p, p1 = k.pc[1].p, p2 = k.pc[2].p;
    const uint32_t c0 = k.pc[0].c, c1 = k.pc[1].c, c2 = k.pc[2].c;
    check_below(r0, 2 * p0);  // inverse residues live in [0, 2p)
    check_below(r1, 2 * p1);
    check_below(r2, 2 * p2);
    uint64_t y0, t1, t2;
    if constexpr (PRESCALED) {
      y0 = fold_p(r0, p0);
      t1 = shoup_mul(fold_p(r1, p1) - fold_p(y0, p1) + p1, k.k1b.x, k.k1b.y, p1, c1);
      t2 = sub_mod_borrow(shoup_mul(r2 - fold_p(y0, p2) + p2, k.k2b.x, k.k2b.y, p2, c2),
                          shoup_mul(t1, k.k2c.x, k.k2c.y, p2, c2), p2);
    } else {
      y0 = shoup_mul(r0, k.k0.x, k.k0.y, p0, c0);
      t1 = sub_mod_borrow(shoup_mul(r1, k.k1a.x, k.k1a.y, p1, c1), shoup_mul(y0, k.k1b.x, k.k1b.y, p1, c1), p1);
      t2 = sub_mod_borrow(shoup_mul(r2, k.k2a.x, k.k2a.y, p2, c2), shoup_mul(y0, k.k2b.x, k.k2b.y, p2, c2), p2);
      t2 = sub_mod_borrow(t2, shoup_mul(t1, k.k2c.x, k.k2c.y, p2, c2), p2);
    }
    // V = y0 + p0 t1 + (p0 p1) t2 < p0 p1 p2 < 2^188
    V3 v{y0, 0, 0};
    add_product_to(v, p0, t1);
    const unsigned __int128 a = static_cast<unsigned __int128>(k.p01_lo) * t2;
    const unsigned __int128 b = static_cast<unsigned __int128>(k.p01_hi) * t2;
    const uint64_t a0 = static_cast<uint64_t>(a), a1 = static_cast<uint64_t>(a >> 64);
    const uint64_t b0 = static_cast<uint64_t>(b), b1 = static_cast<uint64_t>(b >> 64);
    // (p0p1) t2 = a0 + (a1 + b0) 2^64 + b1 2^128
    const uint64_t m1 = a1 + b0;
    const uint64_t mc = m1 < a1;
    add128_to(v, a0, m1);
    v.w2 += b1 + mc;
    return v;
  }
};

using CrtProducer = CrtProducerT<>;

// A tile's published aggregate: the launch's epoch in the high word, then
// p, g and the state bit 1 ("published").
__device__ __forceinline__ unsigned long long flag_word(uint32_t epoch, uint32_t g, uint32_t p) {
  return (static_cast<unsigned long long>(epoch) << 32) | (p << 3) | (g << 2) | 1u;
}

// One tile of NT * 8 output limbs per CTA (tile gt).  Batch (batch !=
// nullptr): tiles run product-major, tpp tiles per product; product k's
// residues are rebased by k * ws_stride and its output is
// batch[k].out[0, min(nout, n)).  The per-launch carry runs 256-thread
// CTAs (2048-limb tiles), four per SM at 64 registers, as does the
// persistent batch kernel.
//
// Each tile is written as if its carry-in were 0 and publishes its
// aggregate (g, p) once; carry_fix_kernel, launched next on the same
// stream, then adds the true carry-in.  No CTA waits on another, so the
// tiles stream at the memory and integer-pipe rate.
//
// carry_body is one CTA of NT threads on tile gt (NT * PER positions);
// s_prev holds NT * 9 words and s_warp NT / 32 pairs of shared memory.
template <class Producer, int NT, int PER = kCarryPer>
__device__ __forceinline__ void carry_body(const Producer &prod, uint64_t *__restrict__ out, uint64_t nproc,
                                           const ScanState &ss, const ProductDesc *batch, uint64_t tpp,
                                           uint64_t ws_stride, uint64_t n, uint64_t gt, uint64_t (*s_prev)[9],
                                           GP *s_warp) {
  constexpr int kCarryTile = NT * PER;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // Product k's residues are addressed through an explicit word offset.
  uint64_t tile = gt, off = 0;
  if (batch) {
    const uint64_t k = gt / tpp;
    tile = gt - k * tpp;
    off = k * ws_stride;
    out = batch[k].out;
    nproc = batch[k].nout < n ? batch[k].nout : n;
  }
  const uint64_t i0 = tile * kCarryTile + static_cast<uint64_t>(tid) * PER;

  V3 v[PER];
  prod.template many<PER>(off, i0, nproc, v);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s_prev[tid][3 * k] = v[PER - 3 + k].w0;
    s_prev[tid][3 * k + 1] = v[PER - 3 + k].w1;
    s_prev[tid][3 * k + 2] = v[PER - 3 + k].w2;
  }
  V3 pm3{0, 0, 0}, pm2{0, 0, 0}, pm1{0, 0, 0};
  if (tid == 0 && i0 >= 3) {
    pm3 = prod.at(off, i0 - 3);
    pm2 = prod.at(off, i0 - 2);
    pm1 = prod.at(off, i0 - 1);
  }
  __syncthreads();
  if (tid > 0) {
    pm3 = V3{s_prev[tid - 1][0], s_prev[tid - 1][1], s_prev[tid - 1][2]};
    pm2 = V3{s_prev[tid - 1][3], s_prev[tid - 1][4], s_prev[tid - 1][5]};
    pm1 = V3{s_prev[tid - 1][6], s_prev[tid - 1][7], s_prev[tid - 1][8]};
  }

  // W_i = v0_i + v1_(i-1) + v2_(i-2) = wl + wh 2^64 (wh <= 2); then
  // A_i = wl_i + wh_(i-1) = al + ah 2^64 (ah <= 1).
  auto wsum = [](uint64_t a, uint64_t b, uint64_t c, uint64_t &hi) {
    const uint64_t s = a + b;
    uint64_t h = s < a;
    const uint64_t t = s + c;
    h += t < s;
    hi = h;
    return t;
  };
  uint64_t whp;
  (void)wsum(pm1.w0, pm2.w1, pm3.w2, whp);  // W_(i0-1)
  uint64_t al[PER];
  uint32_t gbits = 0, pbits = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const V3 &c1 = (k >= 1) ? v[k - 1] : pm1;
    const V3 &c2 = (k >= 2) ? v[k - 2] : (k == 1 ? pm1 : pm2);
    uint64_t wh;
    const uint64_t wl = wsum(v[k].w0, c1.w1, c2.w2, wh);
    const uint64_t a = wl + whp;
    const uint32_t ah = a < wl;
    al[k] = a;
    gbits |= ah << k;
    pbits |= ((a == ~0ull) && !ah ? 1u : 0u) << k;
    whp = wh;
  }
  // Thread aggregate over its positions (position 0 least significant).
  GP t{0, 1};
#pragma unroll
  for (int k = 0; k < PER; ++k) t = gp_compose(t, GP{(gbits >> k) & 1u, (pbits >> k) & 1u});

  // Inclusive warp scan, then across warps.
  GP inc = t;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t og = __shfl_up_sync(0xffffffffu, inc.g, d);
    const uint32_t op = __shfl_up_sync(0xffffffffu, inc.p, d);
    if (lane >= d) inc = gp_compose(GP{og, op}, inc);
  }
  if (lane == 31) s_warp[wid] = inc;
  __syncthreads();
  GP wpre{0, 1};
  for (int w = 0; w < wid; ++w) wpre = gp_compose(wpre, s_warp[w]);
  GP excl;
  {
    const uint32_t og = __shfl_up_sync(0xffffffffu, inc.g, 1);
    const uint32_t op = __shfl_up_sync(0xffffffffu, inc.p, 1);
    excl = lane == 0 ? GP{0, 1} : GP{og, op};
  }
  excl = gp_compose(wpre, excl);  // runs over positions before this thread, within the tile
  if (tid == 0) {
    GP agg{0, 1};
    for (int w = 0; w < NT / 32; ++w) agg = gp_compose(agg, s_warp[w]);
    ss.flags[gt] = flag_word(ss.epoch, agg.g, agg.p);
  }
  uint32_t cin = excl.g;  // carry-in 0 at the tile's first position
  // Stage the tile's limbs in shared memory (reusing s_prev) and store them
  // with consecutive lanes on consecutive limbs: full 256-byte segments,
  // which also suits an output that lives in host memory.
  uint64_t *s_out = &s_prev[0][0];
  auto oswz = [](uint32_t w) { return w ^ ((w >> 3) & 7u); };
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const uint64_t z = al[k] + cin;
    cin = ((gbits >> k) & 1u) | (((pbits >> k) & 1u) & cin);
    s_out[oswz(static_cast<uint32_t>(tid * PER + k))] = z;
  }
  __syncthreads();
  const uint64_t tbase = tile * kCarryTile;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const uint32_t w = static_cast<uint32_t>(tid + k * NT);
    if (tbase + w < nproc) out[tbase + w] = s_out[oswz(w)];
  }
}

// carry_body for coefficients that are 80-bit digits: position i of the sum is
// worth 2^(80 i), and four positions fill five limbs.  Each coefficient splits
// into three pieces of 80 bits (the third below 2^28), the pieces that meet at
// a position add up to less than 2^82, and position i's digit before carries
// is that sum's low 80 bits plus the bits past 80 of position i - 1: at most
// one carry, as with limbs.  A tile of NT * PER positions is NT * PER * 5/4
// limbs; a thread passes its neighbour the pieces of its last positions.
// nproc is in limbs; limbs the digits fill past it must be zero.
template <class Producer, int NT, int PER>
__device__ __forceinline__ void carry80_body(const Producer &prod, uint64_t *__restrict__ out, uint64_t nproc,
                                             const ScanState &ss, const ProductDesc *batch, uint64_t tpp,
                                             uint64_t ws_stride, uint64_t n, uint64_t gt, uint64_t *s_buf, GP *s_warp) {
  constexpr int kTile = NT * PER, kOut = PER / 4 * 5;  // digits per tile, limbs per thread
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint64_t tile = gt, off = 0;
  if (batch) {
    const uint64_t k = gt / tpp;
    tile = gt - k * tpp;
    off = k * ws_stride;
    out = batch[k].out;
    nproc = batch[k].nout < limbs_of(n, true) ? batch[k].nout : limbs_of(n, true);
  }
  const uint64_t ndig = coefs_of(nproc, true);
  const uint64_t i0 = tile * kTile + static_cast<uint64_t>(tid) * PER;
  V3 v[PER];
  prod.template many<PER>(off, i0, ndig, v);
  // Pieces of a coefficient: bits 0..79 (w0 and the low 16 bits of w1), 80..159, 160...
  const auto lo1 = [](const V3 &x) { return (x.w1 >> 16) | (x.w2 << 48); };
  const auto hi1 = [](const V3 &x) { return static_cast<uint32_t>(x.w2 >> 16) & 0xffffu; };
  const auto lo2 = [](const V3 &x) { return static_cast<uint32_t>(x.w2 >> 32); };
  // The sum at a position: c0's first piece, c1's second, c2's third.
  const auto sum = [&](const V3 &c0, uint64_t b1, uint32_t b1h, uint32_t b2, uint32_t &hi) {
    uint64_t lo = c0.w0 + b1;
    hi = (static_cast<uint32_t>(c0.w1) & 0xffffu) + b1h + (lo < b1 ? 1u : 0u);
    lo += b2;
    hi += lo < b2 ? 1u : 0u;
    return lo;
  };
  // To the next thread: the last position's second piece, the third pieces of
  // the last two, and the bits past 80 of the last position's sum.
  uint64_t *s_prev = s_buf;  // [NT][3]
  {
    uint32_t h;
    (void)sum(v[PER - 1], lo1(v[PER - 2]), hi1(v[PER - 2]), lo2(v[PER - 3]), h);
    s_prev[3 * tid] = lo1(v[PER - 1]);
    s_prev[3 * tid + 1] = hi1(v[PER - 1]) | (static_cast<uint64_t>(h >> 16) << 32);
    s_prev[3 * tid + 2] = lo2(v[PER - 1]) | (static_cast<uint64_t>(lo2(v[PER - 2])) << 32);
  }
  uint64_t b1 = 0;                    // second piece of the position below
  uint32_t b1h = 0, b2 = 0, b3 = 0;   // its high bits; third pieces of the two below
  uint32_t hp = 0;                    // bits past 80 of the sum below
  if (tid == 0 && i0 >= 3) {
    const V3 q3 = prod.at(off, i0 - 3), q2 = prod.at(off, i0 - 2), q1 = prod.at(off, i0 - 1);
    uint32_t h;
    (void)sum(q1, lo1(q2), hi1(q2), lo2(q3), h);
    b1 = lo1(q1);
    b1h = hi1(q1);
    b2 = lo2(q2);
    b3 = lo2(q1);
    hp = h >> 16;
  }
  __syncthreads();
  if (tid > 0) {
    b1 = s_prev[3 * tid - 3];
    const uint64_t a = s_prev[3 * tid - 2], c = s_prev[3 * tid - 1];
    b1h = static_cast<uint32_t>(a);
    hp = static_cast<uint32_t>(a >> 32);
    b3 = static_cast<uint32_t>(c);
    b2 = static_cast<uint32_t>(c >> 32);
  }
  uint64_t al[PER];
  uint32_t ah[PER];  // the digit's bits 64..79
  uint32_t gbits = 0, pbits = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    uint32_t h;
    const uint64_t lo = sum(v[k], k ? lo1(v[k - 1]) : b1, k ? hi1(v[k - 1]) : b1h, k >= 2 ? lo2(v[k - 2]) : (k ? b3 : b2), h);
    const uint64_t a = lo + hp;
    hp = h >> 16;
    h = (h & 0xffffu) + (a < lo ? 1u : 0u);
    al[k] = a;
    ah[k] = h & 0xffffu;
    gbits |= (h >> 16) << k;
    pbits |= (a == ~0ull && h == 0xffffu ? 1u : 0u) << k;
  }
  GP t{0, 1};
#pragma unroll
  for (int k = 0; k < PER; ++k) t = gp_compose(t, GP{(gbits >> k) & 1u, (pbits >> k) & 1u});
  GP inc = t;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t og = __shfl_up_sync(0xffffffffu, inc.g, d);
    const uint32_t op = __shfl_up_sync(0xffffffffu, inc.p, d);
    if (lane >= d) inc = gp_compose(GP{og, op}, inc);
  }
  if (lane == 31) s_warp[wid] = inc;
  __syncthreads();  // also: every thread has read s_prev
  GP wpre{0, 1};
  for (int w = 0; w < wid; ++w) wpre = gp_compose(wpre, s_warp[w]);
  const uint32_t og = __shfl_up_sync(0xffffffffu, inc.g, 1);
  const uint32_t op = __shfl_up_sync(0xffffffffu, inc.p, 1);
  const GP excl = gp_compose(wpre, lane == 0 ? GP{0, 1} : GP{og, op});
  if (tid == 0) {
    GP agg{0, 1};
    for (int w = 0; w < NT / 32; ++w) agg = gp_compose(agg, s_warp[w]);
    ss.flags[gt] = flag_word(ss.epoch, agg.g, agg.p);
  }
  uint32_t cin = excl.g;
#pragma unroll
  for (int k = 0; k < PER; ++k) {  // the digits with their carries (mod 2^80)
    const uint64_t z = al[k] + cin;
    ah[k] = (ah[k] + (z < al[k] ? 1u : 0u)) & 0xffffu;
    al[k] = z;
    cin = ((gbits >> k) & 1u) | (((pbits >> k) & 1u) & cin);
  }
  uint64_t *s_out = s_buf;
#pragma unroll
  for (int q = 0; q < PER; q += 4) {
    uint64_t *o = s_out + tid * kOut + q / 4 * 5;
    o[0] = al[q];
    o[1] = ah[q] | (al[q + 1] << 16);
    o[2] = (al[q + 1] >> 48) | (static_cast<uint64_t>(ah[q + 1]) << 16) | (al[q + 2] << 32);
    o[3] = (al[q + 2] >> 32) | (static_cast<uint64_t>(ah[q + 2]) << 32) | (al[q + 3] << 48);
    o[4] = (al[q + 3] >> 16) | (static_cast<uint64_t>(ah[q + 3]) << 48);
  }
  __syncthreads();
  const uint64_t tbase = tile * (kTile / 4 * 5);
#pragma unroll
  for (int k = 0; k < kOut; ++k) {
    const uint32_t w = static_cast<uint32_t>(tid + k * NT);
    const uint64_t z = s_out[w];
    if (tbase + w < nproc)
      out[tbase + w] = z;
    else if (z)
      latch_error(ss.err, kDevCarryOverflow);
  }
}

// The second launch of a carry, one warp per tile.  Tile t's carry-in is
// the composition of the aggregates of tiles t - 1, t - 2, ... up to the
// nearest one that does not propagate (p = 0), or 0 before the product's
// first tile.  Every flag is final here (the tile launch ran to completion
// earlier on the stream), so nothing waits; a flag of another launch is an
// error.  A warp reads 128 predecessors per round, four per lane.  Batches
// (batch != nullptr) index tiles as the tile launch does.
//
// A carry-in of 1 changes only the tile's leading run of positions that
// propagate.  A position propagates exactly when its low word before
// carries, A, is 2^64 - 1: a position that generates a carry wraps to a low
// word of at most 1.  The tile launch wrote exactly A at every position of
// that run, so the run is the tile's leading limbs equal to 2^64 - 1.  They
// become 0 and the first limb after them gains 1; a tile that is one run
// becomes 0 and passes the carry on, as its p = 1 aggregate already says.
//
// With 80-bit digits a tile is TILE limbs too, all ones exactly when every
// digit is, so the same holds.
//
// fix_body is one warp on tile gt of TILE limbs; a batch's product has at most
// n limbs.
constexpr int kFixWarps = 8;

template <int TILE>
__device__ __forceinline__ void fix_body(uint64_t *out, uint64_t nproc, uint64_t tiles, const ScanState &ss,
                                         bool drop_top, const ProductDesc *batch, uint64_t tpp, uint64_t n,
                                         uint64_t gt) {
  constexpr int kCarryTile = TILE;
  const int lane = threadIdx.x & 31;
  if (gt >= tiles) return;
  uint64_t t = gt, first = 0;
  if (batch) {
    const uint64_t k = gt / tpp;
    t = gt - k * tpp;
    first = k * tpp;
    out = batch[k].out;
    nproc = batch[k].nout < n ? batch[k].nout : n;
  }
  const uint64_t ntiles = carry_tiles_dev<TILE>(nproc);  // tiles that hold positions
  if (t >= ntiles) return;
  const unsigned long long *flags = ss.flags;
  auto gp_of = [&](unsigned long long w, bool &bad) {
    if ((w >> 32) != ss.epoch || (w & 3u) != 1u) bad = true;
    return GP{static_cast<uint32_t>((w >> 2) & 1u), static_cast<uint32_t>((w >> 3) & 1u)};
  };
  GP acc{0, 1};
  bool bad = false;
  for (int64_t hi = static_cast<int64_t>(gt) - 1;; hi -= 128) {
    // Lane l composes tiles hi - 4l (most significant) down to hi - 4l - 3;
    // positions before the product's first tile emit carry 0.
    GP mine{0, 1};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t j = hi - 4 * lane - q;
      const GP f = j >= static_cast<int64_t>(first) ? gp_of(flags[j], bad) : GP{0, 0};
      mine = gp_compose(f, mine);
    }
    if (__any_sync(0xffffffffu, bad)) {
      if (lane == 0) atomicCAS(ss.err, kDevOk, kDevTicket);
      return;
    }
    // Lane 0 most significant, lane 31 least.
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t og = __shfl_down_sync(0xffffffffu, mine.g, d);
      const uint32_t op = __shfl_down_sync(0xffffffffu, mine.p, d);
      if (lane + d < 32) mine = gp_compose(GP{og, op}, mine);
    }
    const GP win{__shfl_sync(0xffffffffu, mine.g, 0), __shfl_sync(0xffffffffu, mine.p, 0)};
    acc = gp_compose(win, acc);
    if (!acc.p) break;  // decided: a window that reaches past the first tile always ends here
  }
  const uint32_t cin = acc.g;
  const uint64_t base = t * kCarryTile;
  const uint64_t end = base + kCarryTile < nproc ? base + kCarryTile : nproc;
  if (t == ntiles - 1 && lane == 0 && !drop_top) {
    bool b2 = false;
    const GP own = gp_of(flags[gt], b2);
    if (own.g | (own.p & cin)) atomicCAS(ss.err, kDevOk, kDevCarryOverflow);
  }
  if (!cin) return;
  for (uint64_t i = base; i < end; i += 32) {
    const uint64_t k = i + lane;
    const bool valid = k < end;
    const uint64_t w = valid ? out[k] : 0;
    const unsigned stop = __ballot_sync(0xffffffffu, valid && w != ~0ull);
    if (!stop) {
      if (valid) out[k] = 0;
      continue;
    }
    const int f = __ffs(stop) - 1;
    if (lane < f) out[k] = 0;
    if (lane == f) out[k] = w + 1;
    break;
  }
}

}  // namespace carry
}  // namespace hg
