// hg_crt.cu -- coefficient reconstruction and carry propagation.
//
// The reference rebuilds each convolution coefficient as a bignum
// sum_j f_j r_j mod M (f_j = (M/m_j) * ((M/m_j)^-1 mod m_j)) and adds it at
// limb i with a recursive carry ripple (src/ntt-multiply.lisp:10-51,
// 242-253).  The value is the unique residue mod M = m0 m1 m2, so any exact
// reconstruction gives the same limbs.  Here Garner's mixed radix
// (src/modular-arithmetic.lisp:235-267) produces each coefficient as three
// limbs V_i = y0 + p0 t1 + p0 p1 t2, the overlap-add sum_i V_i 2^(64 i) is
// formed per position, and carries are resolved by a carry-lookahead scan
// within a CTA by warp shuffles.  Across CTAs each tile is written with
// carry-in 0 and publishes its (generate, propagate) aggregate; a second
// launch composes every tile's carry-in from the aggregates below it and
// applies it (in a short launch, the CTA that finishes last does).  No kernel
// here waits on another CTA.  80-bit digits add up at 2^(80 i) the same way.
//
// The same overlap-add + scan finishes the schoolboy and by-digit products
// (src/mpz-ram.lisp:367-431), with V_i = sum_j x_(i-j) y_j.
#include "hg_carry.cuh"

namespace hg {
namespace {

using namespace carry;

// Tiles of 2048 limbs: four CTAs of 256 threads per SM (64 registers),
// 4.4% faster than two of 512 threads on 4096-limb tiles (fewer threads
// wait at each CTA barrier).
constexpr int kCarryThreads = 256;
constexpr int kCarryMinBlocks = 4;
constexpr int kCarryTile = kCarryThreads * kCarryPer;
// Launches of at most kShortCarry limbs leave SMs idle and are bound by the
// latency of one thread's positions and by the launches themselves: they run
// tiles of 1024 limbs (four positions a thread), and the CTA that finishes
// last applies the carries itself instead of a second launch (one thread per
// tile reads the aggregates, so at most 256 tiles): a product of 2^13 points
// 35.9 -> 31.8 us, of 2^16 points 47.2 -> 43.1.
constexpr int kShortPer = 4;
constexpr int kShortTile = kCarryThreads * kShortPer;
static_assert(kShortTile == kCarryMinTile && kCarryTile > kShortTile, "flag words are reserved for this tile");
constexpr uint64_t kShortCarry = static_cast<uint64_t>(kShortTile) * kCarryThreads;

// The product of a long operand cut into chunks of `chunk` coefficients (limbs
// or 80-bit digits) with a short one: chunk k's cyclic product (n > chunk +
// short - 1 points, no wrap) covers result positions k chunk .. k chunk + chunk
// + short - 2, and chunk >= short makes at most two chunks meet at a position.
// Their residues are added before the reconstruction: the sum is the product's
// own coefficient, below short * 2^160 < p0 p1 p2 (2^128 on limbs), so Garner's value of the
// summed residues is the exact sum.  The inverse leaves residues in
// [0, 2p); each is folded to [0, p) before the sum, and Garner's Shoup
// products take the sum in [0, 2p) as it is.
template <class Crt>
struct ChunkProducerT {
  Crt crt;              // res = chunk 0's residues, n = 2^logN
  uint64_t stride;      // words between consecutive chunks' residues
  uint64_t chunk, nchunks;

  __host__ __device__ __forceinline__ bool drop_top() const { return false; }

  __device__ __forceinline__ static uint64_t sum2(uint64_t a, uint64_t b, uint64_t p) {
    return fold_p(a, p) + fold_p(b, p);
  }

  __device__ __forceinline__ uint64_t sum_res(const uint64_t *r0, const uint64_t *r1, int j) const {
    const uint64_t a = r0 ? r0[j * crt.n] : 0, b = r1 ? r1[j * crt.n] : 0;
    return sum2(a, b, crt.k.pc[j].p);
  }

  // Residue pointers of position i: the chunk that starts at or below i, and
  // the one before it when position i is inside its product.
  __device__ __forceinline__ void sources(uint64_t i, const uint64_t *&r0, const uint64_t *&r1) const {
    const uint64_t k = i / chunk, o = i - k * chunk;
    r0 = k < nchunks ? crt.res + k * stride + o : nullptr;
    r1 = (k >= 1 && k - 1 < nchunks && o + chunk < crt.n) ? crt.res + (k - 1) * stride + o + chunk : nullptr;
  }

  __device__ __forceinline__ V3 at(uint64_t, uint64_t i) const {
    const uint64_t *r0, *r1;
    sources(i, r0, r1);
    return crt.garner(sum_res(r0, r1, 0), sum_res(r0, r1, 1), sum_res(r0, r1, 2));
  }

  // PER positions from i0 (a multiple of PER, as is chunk): one chunk pair.
  template <int PER>
  __device__ __forceinline__ void many(uint64_t, uint64_t i0, uint64_t nproc, V3 (&v)[PER]) const {
    if (i0 + PER > nproc) {
#pragma unroll
      for (int k8 = 0; k8 < PER; ++k8) v[k8] = (i0 + k8 < nproc) ? at(0, i0 + k8) : V3{0, 0, 0};
      return;
    }
    const uint64_t *r0, *r1;
    sources(i0, r0, r1);
    uint64_t r[3][PER];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const uint64_t p = crt.k.pc[j].p;
#pragma unroll
      for (int q = 0; q < PER / 2; ++q) {
        ulonglong2 a = make_ulonglong2(0, 0), b = make_ulonglong2(0, 0);
        if (r0) a = reinterpret_cast<const ulonglong2 *>(r0 + j * crt.n)[q];
        if (r1) b = reinterpret_cast<const ulonglong2 *>(r1 + j * crt.n)[q];
        r[j][2 * q] = sum2(a.x, b.x, p);
        r[j][2 * q + 1] = sum2(a.y, b.y, p);
      }
    }
#pragma unroll
    for (int k8 = 0; k8 < PER; ++k8) v[k8] = crt.garner(r[0][k8], r[1][k8], r[2][k8]);
  }
};

struct ConvProducer {
  const uint64_t *x;
  uint64_t nx;
  const uint64_t *y;  // null: multiply by dval
  uint64_t ny;
  uint64_t dval;

  __host__ __device__ __forceinline__ bool drop_top() const { return false; }

  template <int PER>
  __device__ __forceinline__ void many(uint64_t, uint64_t i0, uint64_t nproc, V3 (&v)[PER]) const {
#pragma unroll
    for (int k8 = 0; k8 < PER; ++k8) v[k8] = (i0 + k8 < nproc) ? at(0, i0 + k8) : V3{0, 0, 0};
  }

  __device__ __forceinline__ V3 at(uint64_t, uint64_t i) const {
    V3 v{0, 0, 0};
    if (!y) {
      if (i < nx) {
        const uint64_t a = x[i];
        v.w0 = a * dval;
        v.w1 = __umul64hi(a, dval);
      }
      return v;
    }
    const uint64_t jlo = i >= nx ? i - nx + 1 : 0;
    const uint64_t jhi = i < ny - 1 ? i : ny - 1;
    for (uint64_t j = jlo; j <= jhi; ++j) {
      const uint64_t a = x[i - j], b = y[j];
      add_product_to(v, a, b);
    }
    return v;
  }
};

// mpz-+ of two long magnitudes over the whole GPU (%add-storages/unsafe and
// %subtract-storages/unsafe, src/mpz-ram.lisp:184-274): position i holds
// x_i + y_i as (low, carry).  With opposite signs y is the smaller
// magnitude's complement over n = max(na, nb) limbs plus 1 at position 0,
// and the carry out of the top is dropped (n: the longer operand's end).  `top` is then the highest index
// where a and b differ (or -1), found before the scan; it picks the larger.
struct SumProducer {
  SumOperand a, b;
  uint64_t n;
  const long long *top;  // subtraction only

  __host__ __device__ __forceinline__ bool drop_top() const { return top != nullptr; }

  __device__ __forceinline__ bool a_larger() const {
    if (!top) return true;
    const long long t = *top;
    if (t < 0) return true;
    const uint64_t u = static_cast<uint64_t>(t);
    return a.at(u) >= b.at(u);
  }

  __device__ __forceinline__ V3 value(uint64_t i, bool ax) const {
    if (i >= n) return V3{0, 0, 0};
    const uint64_t va = a.at(i), vb = b.at(i);
    const uint64_t x = ax ? va : vb;
    uint64_t y = ax ? vb : va;
    if (top) y = ~y;
    uint64_t lo = x + y;
    uint64_t c = lo < x ? 1 : 0;
    if (top && i == 0) {
      lo += 1;
      c += lo == 0 ? 1 : 0;
    }
    return V3{lo, c, 0};
  }

  __device__ __forceinline__ V3 at(uint64_t, uint64_t i) const { return value(i, a_larger()); }

  template <int PER>
  __device__ __forceinline__ void many(uint64_t, uint64_t i0, uint64_t nproc, V3 (&v)[PER]) const {
    const bool ax = a_larger();
#pragma unroll
    for (int k8 = 0; k8 < PER; ++k8) v[k8] = (i0 + k8 < nproc) ? value(i0 + k8, ax) : V3{0, 0, 0};
  }
};

// The highest index (or -1) found by a grid: each warp's best goes to *top,
// which was -1.
__device__ __forceinline__ void grid_max(long long best, long long *top) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const long long o = __shfl_down_sync(0xffffffffu, best, d);
    best = o > best ? o : best;
  }
  if ((threadIdx.x & 31) == 0 && best >= 0) atomicMax(top, best);
}

// *top = max index i < n with a_i != b_i.
__global__ void top_diff_kernel(const SumOperand a, const SumOperand b, uint64_t n, long long *top) {
  pdl_wait();
  long long best = -1;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    if (a.at(i) != b.at(i)) best = static_cast<long long>(i);
  grid_max(best, top);
}

// result = (sign, size) of out[0, nproc): the highest nonzero limb, searched by
// the whole grid (a difference may have many zero limbs at its top: one CTA
// that searched them from the top took 24 us for 2^16-limb Newton residuals).
// The CTA that finishes last writes the result and leaves the search words
// and its own count as the next sum expects them.
__global__ void sum_finish_kernel(const uint64_t *out, uint64_t nproc, SumProducer prod, int64_t sa, int64_t sb,
                                  int64_t *result, SumWords *w) {
  __shared__ unsigned s_done;
  pdl_wait();
  long long best = -1;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < nproc; i += stride)
    if (out[i]) best = static_cast<long long>(i);
  grid_max(best, &w->top_out);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_done = atomicInc(&w->done, gridDim.x - 1);
  __syncthreads();
  if (s_done != gridDim.x - 1 || threadIdx.x != 0) return;
  __threadfence();
  const int64_t size = *static_cast<volatile long long *>(&w->top_out) + 1;
  const int64_t sign = prod.a_larger() ? sa : sb;
  result[0] = size ? sign : 1;
  result[1] = size;
  w->top_out = -1;
  w->top_diff = -1;
}

// One tile per CTA, of PER coefficients per thread (limbs, or 80-bit digits).
template <class Producer, bool D80, int PER>
__device__ __forceinline__ void carry_tile(const Producer &prod0, uint64_t *out, uint64_t nproc, const ScanState &ss,
                                           const ProductDesc *batch, uint64_t tpp, uint64_t ws_stride, uint64_t n,
                                           uint64_t *s_buf, GP *s_warp) {
  if constexpr (D80)
    carry80_body<Producer, kCarryThreads, PER>(prod0, out, nproc, ss, batch, tpp, ws_stride, n, blockIdx.x, s_buf,
                                               s_warp);
  else
    carry_body<Producer, kCarryThreads, PER>(prod0, out, nproc, ss, batch, tpp, ws_stride, n, blockIdx.x,
                                             reinterpret_cast<uint64_t(*)[9]>(s_buf), s_warp);
}

template <class Producer, bool D80>
__global__ void __launch_bounds__(kCarryThreads, kCarryMinBlocks)
    carry_kernel(const Producer prod0, uint64_t *__restrict__ out, uint64_t nproc, ScanState ss,
                 const ProductDesc *batch, uint64_t tpp, uint64_t ws_stride, uint64_t n) {
  __shared__ uint64_t s_buf[kCarryThreads * (D80 ? 10 : 9)];
  __shared__ GP s_warp[kCarryThreads / 32];
  pdl_wait();
  carry_tile<Producer, D80, kCarryPer>(prod0, out, nproc, ss, batch, tpp, ws_stride, n, s_buf, s_warp);
}

// The carries of a whole short launch, by the CTA that finished last: thread
// t composes tile t's carry-in from the aggregates of its product's tiles
// below (fix_body says why only the tile's leading limbs equal to 2^64 - 1
// and the first limb after them change).  Most tiles are done by their
// thread's first limb; the others go to whole warps.
template <int TILE>
__device__ __forceinline__ void fix_all(uint64_t *out, uint64_t nproc, uint64_t tiles, const ScanState &ss,
                                        bool drop_top, const ProductDesc *batch, uint64_t tpp, uint64_t n,
                                        GP *s_warp, uint32_t *s_long) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint64_t gt = static_cast<uint64_t>(tid);
  uint64_t t = gt;
  if (batch && gt < tiles) {
    const uint64_t k = gt / tpp;
    t = gt - k * tpp;
    out = batch[k].out;
    nproc = batch[k].nout < n ? batch[k].nout : n;
  }
  const uint64_t ntiles = carry_tiles_dev<TILE>(nproc);
  const bool live = gt < tiles && t < ntiles;
  GP own{0, 0};
  if (live) {
    const unsigned long long w = __ldcg(ss.flags + gt);
    if ((w >> 32) != ss.epoch || (w & 3u) != 1u) atomicCAS(ss.err, kDevOk, kDevTicket);
    own = GP{static_cast<uint32_t>((w >> 2) & 1u), static_cast<uint32_t>((w >> 3) & 1u)};
  }
  // Inclusive scan; a product's first tile has carry-in 0, so what is below it does not matter.
  GP inc = GP{own.g, t == 0 ? 0u : own.p};
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t og = __shfl_up_sync(0xffffffffu, inc.g, d);
    const uint32_t op = __shfl_up_sync(0xffffffffu, inc.p, d);
    if (lane >= d) inc = gp_compose(GP{og, op}, inc);
  }
  if (lane == 31) s_warp[wid] = inc;
  s_long[tid] = 0;
  __syncthreads();
  GP below{0, 0};
  for (int w = 0; w < wid; ++w) below = gp_compose(below, s_warp[w]);
  const uint32_t og = __shfl_up_sync(0xffffffffu, inc.g, 1), op = __shfl_up_sync(0xffffffffu, inc.p, 1);
  if (lane > 0) below = gp_compose(below, GP{og, op});
  const uint32_t cin = live && t > 0 ? below.g : 0;
  if (live && t == ntiles - 1 && !drop_top && (own.g | (own.p & cin))) atomicCAS(ss.err, kDevOk, kDevCarryOverflow);
  if (cin) {
    const uint64_t w = __ldcg(out + t * TILE);
    if (w != ~0ull)
      out[t * TILE] = w + 1;
    else
      s_long[tid] = 1;
  }
  __syncthreads();
  for (uint64_t k = wid; k < tiles; k += kCarryThreads / 32) {
    if (!s_long[k]) continue;
    uint64_t tile = k, np = nproc;
    uint64_t *o = out;
    if (batch) {
      const uint64_t pr = k / tpp;
      tile = k - pr * tpp;
      o = batch[pr].out;
      np = batch[pr].nout < n ? batch[pr].nout : n;
    }
    const uint64_t end = (tile + 1) * TILE < np ? (tile + 1) * TILE : np;
    for (uint64_t i = tile * TILE; i < end; i += 32) {
      const uint64_t at = i + lane;
      const uint64_t w = at < end ? __ldcg(o + at) : 0;
      const unsigned stop = __ballot_sync(0xffffffffu, at < end && w != ~0ull);
      const int f = stop ? __ffs(stop) - 1 : 32;
      if (lane < f && at < end) o[at] = 0;
      if (lane == f) o[at] = w + 1;
      if (stop) break;
    }
  }
}

// A short launch: tiles, then the carries by the CTA that finishes last.
// ss.done counts the launch's finished CTAs and wraps back to 0 with the last.
template <class Producer, bool D80>
__global__ void __launch_bounds__(kCarryThreads, kCarryMinBlocks)
    carry_short_kernel(const Producer prod0, uint64_t *out, uint64_t nproc, ScanState ss, const ProductDesc *batch,
                       uint64_t tpp, uint64_t ws_stride, uint64_t n, bool drop_top) {
  __shared__ uint64_t s_buf[kCarryThreads * 9];
  __shared__ GP s_warp[kCarryThreads / 32];
  __shared__ unsigned s_done;
  pdl_wait();
  carry_tile<Producer, D80, kShortPer>(prod0, out, nproc, ss, batch, tpp, ws_stride, n, s_buf, s_warp);
  __threadfence();  // this thread's limbs (thread 0: also the aggregate) before the count
  __syncthreads();
  if (threadIdx.x == 0) {
    s_done = atomicInc(ss.done, gridDim.x - 1);
    __threadfence();
  }
  __syncthreads();
  if (s_done != gridDim.x - 1) return;
  fix_all<D80 ? kShortTile / 4 * 5 : kShortTile>(out, nproc, gridDim.x, ss, drop_top, batch, tpp, limbs_of(n, D80),
                                                 s_warp, reinterpret_cast<uint32_t *>(s_buf));
}

template <bool D80>
__global__ void __launch_bounds__(kFixWarps * 32)
    carry_fix_kernel(uint64_t *out, uint64_t nproc, uint64_t tiles, ScanState ss, bool drop_top,
                     const ProductDesc *batch, uint64_t tpp, uint64_t n) {
  pdl_wait();
  fix_body<D80 ? kCarryTile / 4 * 5 : kCarryTile>(
      out, nproc, tiles, ss, drop_top, batch, tpp, limbs_of(n, D80), static_cast<uint64_t>(blockIdx.x) * kFixWarps + (threadIdx.x >> 5));
}

// A carry over `tiles` tiles (a batch: tpp per product): one launch where it
// is short, else the tiles and the fix.
template <bool D80 = false, class Producer>
cudaError_t launch_carry(const Producer &prod, uint64_t *out, uint64_t nproc, uint64_t tiles, bool is_short,
                         const ScanState &ss, cudaStream_t st, const ProductDesc *batch = nullptr, uint64_t tpp = 0,
                         uint64_t ws_stride = 0, uint64_t n = 0) {
  if (tiles == 0) return cudaSuccess;
  if (tiles > 0x7fffffffull || (is_short && tiles > kCarryThreads)) return cudaErrorInvalidValue;
  const dim3 grid(static_cast<unsigned>(tiles));
  if (is_short)
    return launch_dep(carry_short_kernel<Producer, D80>, grid, kCarryThreads, 0, st, prod, out, nproc, ss, batch, tpp,
                      ws_stride, n, prod.drop_top());
  cudaError_t e = launch_dep(carry_kernel<Producer, D80>, grid, kCarryThreads, 0, st, prod, out, nproc, ss, batch, tpp,
                             ws_stride, n);
  if (e != cudaSuccess) return e;
  const uint64_t blocks = (tiles + kFixWarps - 1) / kFixWarps;
  return launch_dep(carry_fix_kernel<D80>, dim3(static_cast<unsigned>(blocks)), kFixWarps * 32, 0, st, out, nproc, tiles,
                    ss, prod.drop_top(), batch, tpp, n);
}

// A schoolboy product of at most kSchoolMax limbs, whole, in one CTA: one
// thread per position, the operands in shared memory.  The general kernel
// above gives such a product a handful of threads with four positions each
// and reads the operands from global memory: 64 x 48 limbs took 25 us (eight
// positions a thread; four: the whole host call 57.5 us, with this kernel 46.9).
static_assert(kSchoolMax == 1024, "a thread per position");

__global__ void __launch_bounds__(kSchoolMax)
    school_kernel(const uint64_t *x, uint32_t nx, const uint64_t *y, uint32_t ny, uint64_t *out, uint32_t n, int *err) {
  __shared__ uint64_t s_x[kSchoolMax], s_y[kSchoolMax];  // then words 1 and 2 of the columns
  __shared__ GP s_warp[32];
  __shared__ uint32_t s_h[32];
  const uint32_t i = threadIdx.x, lane = i & 31, wid = i >> 5;
  pdl_wait();
  if (i < nx) s_x[i] = x[i];
  if (i < ny) s_y[i] = y[i];
  __syncthreads();
  V3 v{0, 0, 0};
  if (i < n) {
    const uint32_t jlo = i >= nx ? i - nx + 1 : 0, jhi = i < ny ? i + 1 : ny;
#pragma unroll 4
    for (uint32_t j = jlo; j < jhi; ++j) {
      const uint64_t a = s_x[i - j], b = s_y[j];
      add_product_to(v, a, b);
    }
  }
  __syncthreads();
  s_x[i] = v.w1;
  s_y[i] = v.w2;
  __syncthreads();
  // W_i = v0_i + v1_(i-1) + v2_(i-2) = wl + wh 2^64, A_i = wl_i + wh_(i-1), as in carry_body.
  const uint64_t u1 = i >= 1 ? s_x[i - 1] : 0, u2 = i >= 2 ? s_y[i - 2] : 0;
  uint64_t wl = v.w0 + u1;
  uint32_t wh = wl < u1;
  wl += u2;
  wh += wl < u2;
  if (lane == 31) s_h[wid] = wh;
  uint32_t whp = __shfl_up_sync(0xffffffffu, wh, 1);
  __syncthreads();
  if (lane == 0) whp = wid ? s_h[wid - 1] : 0;
  const uint64_t A = wl + whp;
  const uint32_t G = __ballot_sync(0xffffffffu, A < whp), P = __ballot_sync(0xffffffffu, A == ~0ull);
  if (lane == 0) {  // the warp's carry out: with carry-in 0, and whether it passes one on
    const uint64_t c0 = (static_cast<uint64_t>(G) << 1) + P;
    s_warp[wid] = GP{static_cast<uint32_t>(c0 >> 32), P == 0xffffffffu ? 1u : 0u};
  }
  __syncthreads();
  GP below{0, 0};
  for (uint32_t w = 0; w < wid; ++w) below = gp_compose(below, s_warp[w]);
  const uint64_t sum = ((static_cast<uint64_t>(G) << 1) | below.g) + P;
  const uint32_t c = static_cast<uint32_t>((sum ^ P) >> lane) & 1u;
  if (i < n) out[i] = A + c;
  if (i == n - 1 && ((A < whp) || (A == ~0ull && c))) latch_error(err, kDevCarryOverflow);
}

// out[N, nout) = 0 for product blockIdx.x.
__global__ void zero_tails_kernel(const ProductDesc *batch, uint64_t N) {
  const ProductDesc d = batch[blockIdx.x];
  for (uint64_t i = N + threadIdx.x; i < d.nout; i += blockDim.x) d.out[i] = 0;
}

}  // namespace

bool carry_short(uint64_t n, uint64_t nprod) { return (n + kShortTile - 1) / kShortTile * nprod <= kCarryThreads; }

uint64_t carry_tiles(uint64_t n, uint64_t nprod) {
  const uint64_t tile = carry_short(n, nprod) ? kShortTile : kCarryTile;
  return (n + tile - 1) / tile;
}

namespace {
// The carry of coefficients that `prod` reconstructs, limbs or digits.
template <class Producer>
cudaError_t launch_coefs(const Producer &prod, bool dig80, uint64_t *out, uint64_t nproc, uint64_t tiles, bool sh,
                         const ScanState &ss, cudaStream_t st, const ProductDesc *batch = nullptr, uint64_t tpp = 0,
                         uint64_t ws_stride = 0, uint64_t n = 0) {
  return dig80 ? launch_carry<true>(prod, out, nproc, tiles, sh, ss, st, batch, tpp, ws_stride, n)
               : launch_carry<false>(prod, out, nproc, tiles, sh, ss, st, batch, tpp, ws_stride, n);
}
using Prescaled = carry::CrtProducerT<true>;
}  // namespace

cudaError_t launch_crt_carry(const uint64_t *res, uint64_t n, bool dig80, const CrtConst &cc, uint64_t *out,
                             uint64_t nout, const ScanState &ss, cudaStream_t st, uint64_t *tiles_used) {
  const uint64_t nproc = nout < limbs_of(n, dig80) ? nout : limbs_of(n, dig80);
  const uint64_t ncoef = coefs_of(nproc, dig80), tiles = carry_tiles(ncoef);
  *tiles_used = tiles;
  if (tiles == 0) return cudaSuccess;
  const bool sh = carry_short(ncoef);
  if (cc.prescaled) return launch_coefs(Prescaled{res, n, cc}, dig80, out, nproc, tiles, sh, ss, st);
  return launch_coefs(CrtProducer{res, n, cc}, dig80, out, nproc, tiles, sh, ss, st);
}

cudaError_t launch_crt_carry_batch(const uint64_t *res, uint64_t ws_stride, uint64_t n, bool dig80, const CrtConst &cc,
                                   const ProductDesc *batch, uint64_t nprod, const ScanState &ss, cudaStream_t st) {
  const uint64_t tpp = carry_tiles(n, nprod);
  const uint64_t tiles = tpp * nprod;
  const bool sh = carry_short(n, nprod);
  if (tiles == 0) return cudaSuccess;
  if (tiles > 0x7fffffffull) return cudaErrorInvalidValue;
  if (cc.prescaled)
    return launch_coefs(Prescaled{res, n, cc}, dig80, nullptr, 0, tiles, sh, ss, st, batch, tpp, ws_stride, n);
  return launch_coefs(CrtProducer{res, n, cc}, dig80, nullptr, 0, tiles, sh, ss, st, batch, tpp, ws_stride, n);
}

cudaError_t launch_crt_carry_chunks(const uint64_t *res, uint64_t ws_stride, uint64_t n, bool dig80, uint64_t chunk,
                                    uint64_t nchunks, const CrtConst &cc, uint64_t *out, uint64_t nproc,
                                    const ScanState &ss, cudaStream_t st, uint64_t *tiles_used) {
  if (chunk % 8 || chunk > n || ws_stride % 2) return cudaErrorInvalidValue;
  const uint64_t ncoef = coefs_of(nproc, dig80), tiles = carry_tiles(ncoef);
  *tiles_used = tiles;
  if (tiles == 0) return cudaSuccess;
  if (tiles > 0x7fffffffull) return cudaErrorInvalidValue;
  const bool sh = carry_short(ncoef);
  if (cc.prescaled)
    return launch_coefs(ChunkProducerT<Prescaled>{{res, n, cc}, ws_stride, chunk, nchunks}, dig80, out, nproc, tiles,
                        sh, ss, st);
  return launch_coefs(ChunkProducerT<CrtProducer>{CrtProducer{res, n, cc}, ws_stride, chunk, nchunks}, dig80, out,
                      nproc, tiles, sh, ss, st);
}

cudaError_t launch_large_sum(const SumOperand &a, int64_t sa, const SumOperand &b, int64_t sb, uint64_t *out,
                             SumWords *words, int64_t *result, const ScanState &ss, cudaStream_t st) {
  const uint64_t n = a.end() > b.end() ? a.end() : b.end();
  const bool sub = sa != sb;
  const uint64_t nproc = sub ? n : n + 1;
  const uint64_t tiles = carry_tiles(nproc);
  if (tiles == 0 || tiles > 0x7fffffffull) return cudaErrorInvalidValue;
  const SumProducer prod{a, b, n, sub ? &words->top_diff : nullptr};
  const auto grid = [](uint64_t m) { return dim3(static_cast<unsigned>(m < 152 * 4 * 1024 ? (m + 1023) / 1024 : 152 * 4)); };
  cudaError_t e = cudaSuccess;
  if (sub) e = launch_dep(top_diff_kernel, grid(n), 256, 0, st, a, b, n, &words->top_diff);
  if (e == cudaSuccess) e = launch_carry(prod, out, nproc, tiles, carry_short(nproc), ss, st);
  if (e == cudaSuccess) e = launch_dep(sum_finish_kernel, grid(nproc), 256, 0, st, out, nproc, prod, sa, sb, result, words);
  if (e != cudaSuccess) {  // what was launched may have set the search words, which the next sum expects clear
    cudaMemsetAsync(words, 0xff, 2 * sizeof(long long), st);
    cudaMemsetAsync(&words->done, 0, sizeof words->done, st);
  }
  return e;
}

cudaError_t launch_zero_tails(const ProductDesc *batch, uint64_t nprod, uint64_t N, cudaStream_t st) {
  if (nprod == 0) return cudaSuccess;
  if (nprod > 0x7fffffffull) return cudaErrorInvalidValue;
  zero_tails_kernel<<<static_cast<unsigned>(nprod), 256, 0, st>>>(batch, N);
  return cudaGetLastError();
}

cudaError_t launch_schoolboy_carry(const uint64_t *x, uint64_t nx, const uint64_t *y, uint64_t ny, uint64_t *out,
                                   uint64_t nout, const ScanState &ss, cudaStream_t st, uint64_t *tiles_used) {
  const uint64_t nproc = nout < nx + ny ? nout : nx + ny;
  const uint64_t tiles = carry_tiles(nproc);
  *tiles_used = tiles;
  if (tiles == 0) return cudaSuccess;
  if (nproc == nx + ny && nproc <= kSchoolMax)
    return launch_dep(school_kernel, dim3(1), static_cast<unsigned>((nproc + 31) & ~uint64_t(31)), 0, st, x,
                      static_cast<uint32_t>(nx), y, static_cast<uint32_t>(ny), out, static_cast<uint32_t>(nproc),
                      ss.err);
  return launch_carry(ConvProducer{x, nx, y, ny, 0}, out, nproc, tiles, carry_short(nproc), ss, st);
}

cudaError_t launch_digit_carry(const uint64_t *x, uint64_t nx, uint64_t d, uint64_t *out, uint64_t nout,
                               const ScanState &ss, cudaStream_t st, uint64_t *tiles_used) {
  const uint64_t nproc = nout < nx + 1 ? nout : nx + 1;
  const uint64_t tiles = carry_tiles(nproc);
  *tiles_used = tiles;
  if (tiles == 0) return cudaSuccess;
  return launch_carry(ConvProducer{x, nx, nullptr, 1, d}, out, nproc, tiles, carry_short(nproc), ss, st);
}

#if HG_CHECKED
HG_CHECKED_READER(checked_fault_crt)
#endif

}  // namespace hg
