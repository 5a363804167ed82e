// hg_series.cu -- the base cases of binary splitting on the device.
//
// binary-split-base-case=1 (src/binary-splitting.lisp:102-110) turns each term
// k of a series into the partial P = p(k), Q = q(k), B = b(k), R = p(k) a(k).
// For the reference's series (src/binary-splitting.lisp:147-231,
// src/pi.lisp:24-43) a, b, p and q are integer polynomials in k, with p(0) and
// q(0) replaced by 1.  One thread per term evaluates them by Horner's rule in
// 256-bit two's complement (k < 2^63, coefficients int64; the caller checks
// that every value and R fit in 255 bits) and writes sign, length without
// high zero limbs and four limbs per value.
#include "hg_host.h"
#include "hypergeometrica_gb300.h"

namespace hg {
namespace {

struct U256 {
  uint64_t w[4];
};

__device__ __forceinline__ U256 mul_small(const U256 &a, uint64_t n) {  // a * n mod 2^256
  U256 r;
  uint64_t carry = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t lo = a.w[i] * n, hi = __umul64hi(a.w[i], n);
    r.w[i] = lo + carry;
    carry = hi + (r.w[i] < lo ? 1 : 0);
  }
  return r;
}

__device__ __forceinline__ U256 add_signed(const U256 &a, int64_t c) {  // a + c mod 2^256
  const uint64_t ext = c < 0 ? ~0ull : 0ull;
  U256 r;
  uint64_t carry = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t y = i == 0 ? static_cast<uint64_t>(c) : ext;
    const uint64_t s = a.w[i] + y;
    const uint64_t t = s + carry;
    carry = (s < a.w[i] ? 1 : 0) + (t < s ? 1 : 0);
    r.w[i] = t;
  }
  return r;
}

__device__ __forceinline__ bool negative(const U256 &a) { return static_cast<int64_t>(a.w[3]) < 0; }

__device__ __forceinline__ U256 negate(const U256 &a) {
  U256 r;
  uint64_t carry = 1;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t x = ~a.w[i];
    r.w[i] = x + carry;
    carry = r.w[i] < x ? 1 : 0;
  }
  return r;
}

__device__ U256 eval_poly(const hg_poly &q, uint64_t n) {
  U256 acc{{0, 0, 0, 0}};
  if (n == 0 && q.has_zero_value) return add_signed(acc, q.zero_value);
  for (int i = q.degree; i >= 0; --i) acc = add_signed(mul_small(acc, n), q.coef[i]);
  return acc;
}

// Magnitude product mod 2^256 of two non-negative values.
__device__ U256 mul_mag(const U256 &a, const U256 &b) {
  U256 r{{0, 0, 0, 0}};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint64_t carry = 0;
#pragma unroll
    for (int j = 0; j + i < 4; ++j) {
      const uint64_t lo = a.w[i] * b.w[j], hi = __umul64hi(a.w[i], b.w[j]);
      const uint64_t s = r.w[i + j] + lo;
      const uint64_t t = s + carry;
      carry = hi + (s < lo ? 1 : 0) + (t < s ? 1 : 0);
      r.w[i + j] = t;
    }
  }
  return r;
}

__device__ void emit(const U256 &v, uint64_t *limbs, int64_t *ss) {
  const bool neg = negative(v);
  const U256 m = neg ? negate(v) : v;
  int size = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    limbs[i] = m.w[i];
    if (m.w[i]) size = i + 1;
  }
  ss[0] = (neg && size) ? -1 : 1;
  ss[1] = size;
}

__global__ void leaves_kernel(hg_poly pa, hg_poly pb, hg_poly pp, hg_poly pq, uint64_t lower, uint64_t count,
                              uint64_t *limbs, int64_t *ss) {
  const uint64_t k = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
  if (k >= count) return;
  const uint64_t n = lower + k;
  const U256 p = eval_poly(pp, n), q = eval_poly(pq, n), b = eval_poly(pb, n), a = eval_poly(pa, n);
  const bool pn = negative(p), an = negative(a);
  U256 r = mul_mag(pn ? negate(p) : p, an ? negate(a) : a);
  if (pn != an) r = negate(r);
  const U256 vals[4] = {p, q, b, r};
#pragma unroll
  for (int j = 0; j < 4; ++j) emit(vals[j], limbs + (j * count + k) * 4, ss + (j * count + k) * 2);
}

// ---- whole nodes ----------------------------------------------------------
//
// A node's partial (P, Q, B, R) over terms [lo, hi) is a function of the
// range alone: combine (src/binary-splitting.lisp:112-121) is exact integer
// arithmetic, so any split of the range gives the same four integers.  Here
// one warp folds the terms left to right: with a one-term right part t,
// combine is
//   R <- b_t q_t R + (B P) r_t,  P <- P p_t,  Q <- Q q_t,  B <- B b_t,
// where r_t = p_t a_t, so keeping BP = B P as a fifth value makes every step
// a product by a value below 2^256.  Values are sign and magnitude; the
// magnitudes live in global memory, W limbs each (a node's stay in L1).
//
// Bound by latency: a fold is a serial chain over the terms.  One lane takes
// one limb, 32 at a time: the lane's column of the product (up to four
// 64 x 64-bit products of its limb and the three below it, by shuffles), the
// columns' overlap-add, and all 32 carries at once from two ballots.  The
// terms' values are evaluated eight terms at a time, four lanes to a term.
// 2048 nodes of 44 Chudnovsky terms: 243 us, against 3838 us with one
// thread per node walking its limbs one by one.

__device__ __forceinline__ int limbs_of(const U256 &m) {
  int n = 4;
  while (n > 0 && m.w[n - 1] == 0) --n;
  return n;
}

constexpr unsigned kAll = 0xffffffffu;
constexpr int kNodeWarps = 4;   // nodes (warps) per CTA
constexpr int kNodeTerms = 8;   // terms evaluated at once

// Carry into each of 32 positions, given the lanes' generate and propagate
// bits (never both) and the carry into lane 0; `out` is the carry out of
// lane 31.  Adding the generates, moved up one, to the propagates ripples
// every carry through its run of propagating positions.
__device__ __forceinline__ uint32_t lane_carry(bool g, bool p, uint32_t cin, uint32_t &out) {
  const uint32_t G = __ballot_sync(kAll, g), P = __ballot_sync(kAll, p);
  const uint64_t sum = ((static_cast<uint64_t>(G) << 1) | cin) + P;
  const uint64_t c = sum ^ P;  // bit i: carry into position i (bit 32: out, as P has no bit 32)
  out = static_cast<uint32_t>(c >> 32) & 1u;
  return static_cast<uint32_t>(c >> (threadIdx.x & 31)) & 1u;
}

// One term's values (magnitudes; sgn bit j set: value j negative), and the
// products q b and p b with their widths where they fit in 256 bits.
struct Term {
  U256 p, q, b, r, qb, pb;
  int sgn;            // bits 0..3: p, q, b, r negative
  int np, nq, nb, nr;  // limbs
  int nqb, npb;        // limbs, or -1 when the product may pass 256 bits
};

// out[0, n + |m|) = x[0, n) * m (magnitudes); out may be x itself: a
// lane's column needs x[i - 3 .. i] only, read before the 32 columns are
// written.  Returns the trimmed size, or -1 when the product may not fit in
// cap limbs.
__device__ int mul_by(uint64_t *out, const uint64_t *x, int n, const U256 &m, int ms, int cap) {
  if (n == 0 || ms == 0) return 0;
  if (n + ms > cap) return -1;
  const int lane = threadIdx.x & 31;
  const int total = n + ms;
  uint64_t xprev = 0;             // x 32 positions below
  uint64_t h1p = 0, h2p = 0;      // the last chunk's column words 1 and 2
  uint64_t hap = 0;               // the last chunk's overlap carries
  uint32_t cin = 0;
  uint64_t top = 0;
  // x[i - t] for lane's position i: from this chunk's lane - t, or from the last chunk's.
  auto below = [&](uint64_t cur, uint64_t prev, int t) {
    const uint64_t a = __shfl_sync(kAll, cur, (lane - t) & 31), b = __shfl_sync(kAll, prev, (lane - t) & 31);
    return lane >= t ? a : b;
  };
  for (int base = 0; base < total; base += 32) {
    const int i = base + lane;
    const uint64_t xi = i < n ? x[i] : 0;
    uint64_t v0 = 0, v1 = 0, v2 = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (t >= ms) break;
      const uint64_t xt = t ? below(xi, xprev, t) : xi;
      const unsigned __int128 xm = static_cast<unsigned __int128>(xt) * m.w[t];
      const uint64_t lo = static_cast<uint64_t>(xm), hi = static_cast<uint64_t>(xm >> 64);
      v0 += lo;
      const uint64_t c0 = v0 < lo ? 1 : 0;
      const uint64_t s = v1 + hi;
      v2 += s < hi ? 1 : 0;
      v1 = s + c0;
      v2 += v1 < c0 ? 1 : 0;
    }
    xprev = xi;
    // Column i's word 0, word 1 of column i - 1, word 2 of column i - 2.
    const uint64_t u1 = below(v1, h1p, 1), u2 = below(v2, h2p, 2);
    h1p = v1;
    h2p = v2;
    uint64_t s = v0 + u1;
    uint64_t ha = s < u1 ? 1 : 0;
    s += u2;
    ha += s < u2 ? 1 : 0;
    const uint64_t hb = below(ha, hap, 1);
    hap = ha;
    const uint64_t z = s + hb;
    uint32_t cout;
    const uint32_t c = lane_carry(z < hb, z == ~0ull, cin, cout);
    cin = cout;
    __syncwarp();  // every lane has read x before any column is written
    if (i < total) out[i] = z + c;
    top = z + c;
  }
  __syncwarp();
  top = __shfl_sync(kAll, top, (total - 1) & 31);
  return total - (top == 0 ? 1 : 0);
}

// x (sign sx, size nx) += y (sign sy, size ny), in place in x.  Returns the
// trimmed size (sx updated), or -1 when the sum may not fit in cap limbs.
__device__ int add_signed_big(uint64_t *x, int nx, int &sx, const uint64_t *y, int ny, int sy, int cap) {
  const int lane = threadIdx.x & 31;
  if (ny == 0) return nx;
  if (nx == 0) {
    if (ny > cap) return -1;
    for (int i = lane; i < ny; i += 32) x[i] = y[i];
    __syncwarp();
    sx = sy;
    return ny;
  }
  const int n = nx > ny ? nx : ny;
  const bool sub = sx != sy;
  if (!sub && n + 1 > cap) return -1;
  bool swap = false;  // y is the larger magnitude
  if (sub) {
    int cmp = nx != ny ? (nx > ny ? 1 : -1) : 0;
    for (int base = (n - 1) & ~31; cmp == 0 && base >= 0; base -= 32) {
      const int i = base + lane;
      const uint64_t a = i < n ? x[i] : 0, b = i < n ? y[i] : 0;
      const unsigned ne = __ballot_sync(kAll, a != b), gt = __ballot_sync(kAll, a > b);
      if (ne) cmp = (gt >> (31 - __clz(ne))) & 1u ? 1 : -1;
    }
    if (cmp == 0) return 0;  // zero: sign is irrelevant
    swap = cmp < 0;
  }
  const int total = sub ? n : n + 1;
  uint32_t cin = 0;
  int size = 0;
  for (int base = 0; base < total; base += 32) {
    const int i = base + lane;
    const uint64_t a = i < nx ? x[i] : 0, b = i < ny ? y[i] : 0;
    const uint64_t u = swap ? b : a, v = swap ? a : b;
    const uint64_t z = sub ? u - v : u + v;
    const bool g = sub ? u < v : z < u, p = sub ? z == 0 : z == ~0ull;
    uint32_t cout;
    const uint32_t c = lane_carry(g, p, cin, cout);
    cin = cout;
    const uint64_t w = sub ? z - c : z + c;
    if (i < total) x[i] = w;
    const unsigned nz = __ballot_sync(kAll, i < total && w != 0);
    if (nz) size = base + 32 - __clz(nz);
  }
  __syncwarp();
  if (swap) sx = sy;
  return size;
}

// The terms k0 .. k0 + cnt - 1 (cnt <= kNodeTerms): four lanes to a term
// evaluate its four polynomials, then lane t of the first eight forms the
// products.
__device__ void eval_terms(Term *terms, const hg_poly *polys, uint64_t k0, int cnt) {
  const int lane = threadIdx.x & 31;
  const int t = lane >> 2, j = lane & 3;
  if (t < cnt) {
    const U256 v = eval_poly(polys[j], k0 + static_cast<uint64_t>(t));  // a, b, p, q
    const bool neg = negative(v);
    const U256 m = neg ? negate(v) : v;
    U256 &dst = j == 0 ? terms[t].r : j == 1 ? terms[t].b : j == 2 ? terms[t].p : terms[t].q;
    dst = m;
    (j == 0 ? terms[t].nr : j == 1 ? terms[t].nb : j == 2 ? terms[t].np : terms[t].nq) = neg ? 1 : 0;
  }
  __syncwarp();
  if (lane < cnt) {
    Term &e = terms[lane];
    const int an = e.nr, bn = e.nb, pn = e.np, qn = e.nq;
    e.sgn = pn | (qn << 1) | (bn << 2) | ((pn ^ an) << 3);
    e.r = mul_mag(e.p, e.r);
    e.np = limbs_of(e.p);
    e.nq = limbs_of(e.q);
    e.nb = limbs_of(e.b);
    e.nr = limbs_of(e.r);
    e.nqb = e.npb = -1;
    if (e.nq + e.nb <= 4) {
      e.qb = mul_mag(e.q, e.b);
      e.nqb = limbs_of(e.qb);
    }
    if (e.np + e.nb <= 4) {
      e.pb = mul_mag(e.p, e.b);
      e.npb = limbs_of(e.pb);
    }
  }
  __syncwarp();
}

// x <- x m0 m1, by one product with m01 where that fits (n01 >= 0).
__device__ __forceinline__ int mul_by2(uint64_t *x, int n, const U256 &m0, int n0, const U256 &m1, int n1,
                                       const U256 &m01, int n01, int cap) {
  if (n01 >= 0 && n + n0 + n1 <= cap) return mul_by(x, x, n, m01, n01, cap);
  n = mul_by(x, x, n, m0, n0, cap);
  return n < 0 ? n : mul_by(x, x, n, m1, n1, cap);
}

__device__ __forceinline__ int set_u256(uint64_t *x, const U256 &m, int n) {
  const int lane = threadIdx.x & 31;
  if (lane < 4) x[lane] = m.w[lane];
  __syncwarp();
  return n;
}

struct Polys {
  hg_poly v[4];  // a, b, p, q
};

// One warp per node: ranges[2 i], ranges[2 i + 1] = lo, hi.  Value j of
// node i: limbs[(j n + i) W ..], sign_size[(j n + i) 2 ..]; scratch holds BP
// and a temporary, 2 W limbs per node.  A size that would pass W is written
// as -1 (and the node's values are not used).
__global__ void __launch_bounds__(kNodeWarps * 32)
    nodes_kernel(const __grid_constant__ Polys polys, const uint64_t *ranges, uint64_t n, uint64_t width,
                 uint64_t *limbs, int64_t *ss, uint64_t *scratch) {
  __shared__ Term s_terms[kNodeWarps][kNodeTerms];
  __shared__ hg_poly s_polys[4];
  if (threadIdx.x < 4) s_polys[threadIdx.x] = polys.v[threadIdx.x];
  __syncthreads();
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t i = blockIdx.x * static_cast<uint64_t>(kNodeWarps) + wid;
  if (i >= n) return;
  Term *terms = s_terms[wid];
  const uint64_t lo = ranges[2 * i], hi = ranges[2 * i + 1];
  const int cap = static_cast<int>(width);
  uint64_t *P = limbs + (0 * n + i) * width, *Q = limbs + (1 * n + i) * width;
  uint64_t *B = limbs + (2 * n + i) * width, *R = limbs + (3 * n + i) * width;
  uint64_t *BP = scratch + (2 * i) * width, *T = scratch + (2 * i + 1) * width;
  int nP = 0, nQ = 0, nB = 0, nR = 0, nBP = 0, sP = 1, sQ = 1, sB = 1, sR = 1, sBP = 1;
  bool ok = true;
  for (uint64_t k0 = lo; ok && (k0 < hi || k0 == lo); k0 += kNodeTerms) {
    const int cnt = hi > k0 && hi - k0 < kNodeTerms ? static_cast<int>(hi - k0) : (hi > k0 ? kNodeTerms : 1);
    eval_terms(terms, s_polys, k0, cnt);
    for (int j = 0; ok && j < cnt; ++j) {
      const Term &t = terms[j];
      const int tp = t.sgn & 1 ? -1 : 1, tq = t.sgn & 2 ? -1 : 1, tb = t.sgn & 4 ? -1 : 1, tr = t.sgn & 8 ? -1 : 1;
      if (k0 == lo && j == 0) {
        nP = set_u256(P, t.p, t.np);
        nQ = set_u256(Q, t.q, t.nq);
        nB = set_u256(B, t.b, t.nb);
        nR = set_u256(R, t.r, t.nr);
        sP = tp;
        sQ = tq;
        sB = tb;
        sR = tr;
        nBP = mul_by(BP, B, nB, t.p, t.np, cap);
        sBP = sB * sP;
        ok = nBP >= 0;
        continue;
      }
      // R <- b q R + BP r
      nR = mul_by2(R, nR, t.q, t.nq, t.b, t.nb, t.qb, t.nqb, cap);
      sR *= tq * tb;
      const int nT = mul_by(T, BP, nBP, t.r, t.nr, cap);
      if (nR >= 0 && nT >= 0) nR = add_signed_big(R, nR, sR, T, nT, sBP * tr, cap);
      // P, Q, B, BP
      nP = mul_by(P, P, nP, t.p, t.np, cap);
      nQ = mul_by(Q, Q, nQ, t.q, t.nq, cap);
      nB = mul_by(B, B, nB, t.b, t.nb, cap);
      nBP = mul_by2(BP, nBP, t.b, t.nb, t.p, t.np, t.pb, t.npb, cap);
      sP *= tp;
      sQ *= tq;
      sB *= tb;
      sBP *= tb * tp;
      ok = nR >= 0 && nT >= 0 && nP >= 0 && nQ >= 0 && nB >= 0 && nBP >= 0;
    }
    __syncwarp();  // every lane is done with these terms
  }
  if (lane < 4) {
    const int size = lane == 0 ? nP : lane == 1 ? nQ : lane == 2 ? nB : nR;
    const int sign = lane == 0 ? sP : lane == 1 ? sQ : lane == 2 ? sB : sR;
    int64_t *o = ss + (static_cast<uint64_t>(lane) * n + i) * 2;
    o[0] = (sign < 0 && size > 0) ? -1 : 1;
    o[1] = ok ? size : -1;
  }
}

}  // namespace
#if HG_CHECKED
HG_CHECKED_READER(checked_fault_series)
#endif

}  // namespace hg

using namespace hg;

extern "C" {

int hg_series_leaves_device(const hg_poly *polys, uint64_t lower, uint64_t count, uint64_t *limbs, int64_t *sign_size,
                            void *stream) {
  if (!polys || (count && (!limbs || !sign_size))) return lib_fail(HG_ERR_ARG, "null pointer");
  if (!lib_ready()) return lib_fail(HG_ERR_NOT_INIT, "hg_series_leaves_device: call hg_init first");
  for (int j = 0; j < 4; ++j)
    if (polys[j].degree < 0 || polys[j].degree > 7)
      return lib_fail(HG_ERR_ARG, "polynomial %d: degree %d outside 0..7", j, polys[j].degree);
  if (count == 0) return HG_OK;
  if (lower + count < lower || lower + count > (uint64_t(1) << 63))
    return lib_fail(HG_ERR_ARG, "terms [%llu, %llu) out of range", (unsigned long long)lower,
                    (unsigned long long)(lower + count));
  const uint64_t blocks = (count + 255) / 256;
  if (blocks > 0x7fffffffull) return lib_fail(HG_ERR_ARG, "%llu terms exceed one launch", (unsigned long long)count);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  leaves_kernel<<<static_cast<unsigned>(blocks), 256, 0, st>>>(polys[0], polys[1], polys[2], polys[3], lower, count,
                                                               limbs, sign_size);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? HG_OK : lib_cuda_fail(e, "series leaves");
}

int hg_series_nodes_device(const hg_poly *polys, const uint64_t *ranges, uint64_t n, uint64_t width, uint64_t *limbs,
                           int64_t *sign_size, uint64_t *scratch, void *stream) {
  if (!polys || (n && (!ranges || !limbs || !sign_size || !scratch))) return lib_fail(HG_ERR_ARG, "null pointer");
  if (!lib_ready()) return lib_fail(HG_ERR_NOT_INIT, "hg_series_nodes_device: call hg_init first");
  for (int j = 0; j < 4; ++j)
    if (polys[j].degree < 0 || polys[j].degree > 7)
      return lib_fail(HG_ERR_ARG, "polynomial %d: degree %d outside 0..7", j, polys[j].degree);
  if (width < 8 || width > (1u << 30)) return lib_fail(HG_ERR_ARG, "width %llu outside 8..2^30", (unsigned long long)width);
  if (n == 0) return HG_OK;
  const uint64_t blocks = (n + kNodeWarps - 1) / kNodeWarps;
  if (blocks > 0x7fffffffull) return lib_fail(HG_ERR_ARG, "%llu nodes exceed one launch", (unsigned long long)n);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const Polys pv{{polys[0], polys[1], polys[2], polys[3]}};
  nodes_kernel<<<static_cast<unsigned>(blocks), kNodeWarps * 32, 0, st>>>(pv, ranges, n, width, limbs, sign_size,
                                                                         scratch);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? HG_OK : lib_cuda_fail(e, "series nodes");
}

}  // extern "C"
